"""The streaming score kernel's grid (csrc/fq_score_grid.cuh, compiled for the host) fills whole waves of the CTAs that fit."""
import ctypes
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "flashquest_b200", "csrc")
SMS = 148


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    d = tmp_path_factory.mktemp("score_grid")
    (d / "shim.cpp").write_text("""
#include "fq_score_grid.cuh"
extern "C" int per_sm(int nr, int ch) { return fq::score_stream_ctas_per_sm(nr, ch); }
extern "C" int ctas(int rows, int P, int resident) { return fq::score_stream_ctas(rows, P, resident); }
""")
    subprocess.run(["g++", "-O1", "-shared", "-fPIC", "-I", CSRC, str(d / "shim.cpp"), "-o", str(d / "shim.so")], check=True)
    return ctypes.CDLL(str(d / "shim.so"))


# registers a thread of each instantiation (-Xptxas -v), q heads per pass x 8-channel chunks per lane
REGISTERS = {(1, 1): 48, (2, 1): 70, (3, 1): 88, (4, 1): 108, (1, 2): 72, (2, 2): 108, (3, 2): 128, (4, 2): 168}


@pytest.mark.parametrize("nr,ch", sorted(REGISTERS))
def test_whole_waves(host, nr, ch):
    fit = 65536 // (128 * (-(-REGISTERS[nr, ch] // 8) * 8))        # 128 threads, registers in steps of 8
    assert host.per_sm(nr, ch) <= fit
    resident = host.per_sm(nr, ch) * SMS
    for rows in (8, 24, 32, 64, 96, 128, 200, 256, 512):
        for P in (2048, 8192):
            c = host.ctas(rows, P, resident)
            if rows * P < resident * 64:
                assert c == 0
                continue
            assert 1 <= c <= P // 64
            waves = -(-rows * c // resident)
            # the share of the CTA slots in use; a wave rounded up costs most with few CTAs a row
            assert rows * c / (waves * resident) >= 0.85, (rows, P, c)
