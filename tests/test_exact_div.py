"""Every input of the division-free quotients (csrc/fq_exact_div.cuh): the functions the kernels use, compiled for the host."""
import ctypes
import math
import os
import subprocess

import pytest
import torch

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "flashquest_b200", "csrc")


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    d = tmp_path_factory.mktemp("exact_div")
    (d / "shim.cpp").write_text("""
#include "fq_exact_div.cuh"
extern "C" void by_top(const float* d, float* q, int n, float top) { for (int i = 0; i < n; ++i) q[i] = fq::div_by_top(d[i], top, 1.0f / top); }
extern "C" void by_rcd(const float* x, float* q, int n) { for (int i = 0; i < n; ++i) q[i] = x[i] * fq::TURBO_RCD; }
""")
    subprocess.run(["g++", "-O1", "-ffp-contract=off", "-shared", "-fPIC", "-I", CSRC, str(d / "shim.cpp"), "-o", str(d / "shim.so")], check=True)
    return ctypes.CDLL(str(d / "shim.so"))


def _every(dtype):
    return torch.arange(65536, dtype=torch.int32).to(torch.int16).view(dtype).float().contiguous()


def _call(fn, x, *args):
    q = torch.empty_like(x)
    fn(ctypes.c_void_p(x.data_ptr()), ctypes.c_void_p(q.data_ptr()), ctypes.c_int(x.numel()), *args)
    return q


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("top", [15.0, 255.0])
def test_page_quotient(host, dtype, top):
    d = _every(dtype)
    d = d[(d >= 1e-6) | d.isnan() | (d == 0)]                # a range; quotients of smaller ones are below the least scale, 1e-6
    got, want = _call(host.by_top, d, ctypes.c_float(top)).to(dtype), (d / top).to(dtype)
    assert torch.equal(got[~d.isnan()], want[~d.isnan()]) and got[d.isnan()].isnan().all()


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_sqrt128_quotient(host, dtype):
    x = _every(dtype)
    got, want = _call(host.by_rcd, x).to(dtype), (x / torch.tensor(math.sqrt(128), dtype=torch.float32)).to(dtype)
    assert torch.equal(got[~x.isnan()], want[~x.isnan()]) and got[x.isnan()].isnan().all()
