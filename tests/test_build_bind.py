"""The CPython module is tied to the torch it was compiled against."""
import os

import pytest

from flashquest_b200 import _lib, build


@pytest.fixture
def tree(tmp_path, monkeypatch):
    """A library folder whose module is newer than its sources; compiling only writes the output file."""
    for name, path in (("LIB_DIR", ""), ("BIND", "_fq_bind.so"), ("BIND_STAMP", "_fq_bind.built_for")):
        monkeypatch.setattr(build, name, str(tmp_path / path))
    compiled = []

    class Done:
        returncode, stdout, stderr = 0, "", ""

    def run(cmd, **kw):
        if "-shared" in cmd:
            compiled.append(cmd)
        with open(cmd[cmd.index("-o") + 1], "w") as f:
            f.write("module")
        return Done
    monkeypatch.setattr(build.subprocess, "run", run)
    build.build_bind()
    assert len(compiled) == 1 and os.path.exists(build.BIND)
    return compiled


def test_rebuilt_for_another_torch(tree, monkeypatch):
    build.build_bind()
    assert len(tree) == 1                                        # nothing changed
    import torch
    monkeypatch.setattr(torch, "__version__", "99.0")
    build.build_bind()
    assert len(tree) == 2
    build.build_bind()
    assert len(tree) == 2


def test_module_of_another_torch_is_not_loaded(tree, monkeypatch):
    monkeypatch.setattr(_lib, "_bind", None)
    monkeypatch.setattr(_lib, "BIND_PATH", build.BIND)
    with open(build.BIND_STAMP, "w") as f:
        f.write("torch 1.0 cpython-39")
    with pytest.raises(_lib.FlashQuestError, match="was built for torch 1.0"):
        _lib.bind()
