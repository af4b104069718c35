"""The CPython module over the C ABI (csrc/fq_bind.cpp) without a GPU: what it refuses before anything is launched.

Fake tensors stand in for tensors on a GPU; each test runs in a process of its own, which an exception that crosses the C
entry would abort."""
import os
import subprocess
import sys
import textwrap

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SETUP = """
    import ctypes, torch
    from torch._subclasses.fake_tensor import FakeTensorMode
    from flashquest_b200 import _lib
    mod = _lib.bind()
    B, HQ, HKV, D = 1, 4, 2, 64
    c = _lib.Int4CacheDesc(kv_dtype=_lib.FQ_F16, L=1, B=B, Hkv=HKV, D=D, page=16, max_seq_len=64)
    prm = _lib.DecodeParams(Hq=HQ)
    plan = mod.plan(4, ctypes.addressof(c), ctypes.addressof(prm), 0, 1, *[0] * 20)
    fake = FakeTensorMode()

    def calls(device):
        e = lambda *s: torch.empty(*s, dtype=torch.float16, device=device)
        with fake:
            k, v, q, cs = e(B, HKV, 1, D), e(B, HKV, 1, D), e(B, HQ, 1, D), e(1, 1, D)
            flat = [t.view(B, 1, -1) for t in (q, k, v)]
        return {"append": lambda: mod.append(4, ctypes.addressof(c), 0, 0, 0, k, v),
                "step": lambda: mod.step(plan, 0, 0, k, v, q, 0),
                "forward": lambda: mod.forward(plan, 0, 0, *flat, cs, cs, 0, None)}
"""


def _run(body):
    if not os.path.exists(os.path.join(ROOT, "flashquest_b200", "lib", "_fq_bind.so")):
        pytest.skip("library not built (python -m flashquest_b200.build)")
    r = subprocess.run([sys.executable, "-c", textwrap.dedent(SETUP) + textwrap.dedent(body)], cwd=ROOT, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]


def test_tensors_on_another_gpu_are_refused():
    _run("""
    for name, call in calls("cuda:1").items():
        assert call() == 1, name                     # the plan's and the cache's buffers are on cuda:0
    """)


def test_operators_refuse_tensors_of_two_gpus():
    _run("""
    with fake:
        a, b = torch.empty(8, device="cuda:0"), torch.empty(8, device="cuda:1")
    _lib.require_cuda(a, None, a)
    try:
        _lib.require_cuda(a, None, b)
    except _lib.FlashQuestError as e:
        assert "different GPUs" in str(e)
    else:
        raise AssertionError("accepted")
    """)


def test_tensors_without_storage_raise():
    """What torch throws below the entry point becomes a Python exception (it ended the process)."""
    _run("""
    for name, call in calls("cuda:0").items():
        try:
            call()
        except RuntimeError:
            continue
        raise AssertionError(name + ": accepted")
    """)


def test_library_symbols_stay_out_of_the_process():
    _run("""
    import ctypes
    assert not hasattr(ctypes.CDLL(None), "fq_version")
    """)
