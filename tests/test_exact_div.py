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
extern "C" void codes16(const float* d, const float* sc, const float* y, float* q, int n) { for (int i = 0; i < n; ++i) q[i] = rintf(fq::code_quotient16(d[i], sc[i], y[i])); }
extern "C" void codes32(const float* d, const float* sc, const float* y, float* q, int n) { for (int i = 0; i < n; ++i) q[i] = rintf(fq::code_quotient32(d[i], sc[i], fq::refine_rcp(sc[i], y[i]))); }
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


def _near_ties(sc, top, g):
    """fp32 numbers on, next to and between the half-integer multiples of sc, up to top."""
    h = torch.randint(0, int(top), sc.shape, generator=g) + 0.5
    d = (h.double() * sc.double()).float()
    step = torch.randint(-3, 4, sc.shape, generator=g, dtype=torch.int32)
    near = (d.view(torch.int32) + step).view(torch.float32)
    return torch.where(torch.rand(sc.shape, generator=g) < 0.9, near, torch.rand(sc.shape, generator=g) * top * sc)


def _off_by_an_ulp(y, g):
    return (y.view(torch.int32) + torch.randint(-1, 2, y.shape, generator=g, dtype=torch.int32)).view(torch.float32)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("top", [15.0, 255.0])
def test_codes_by_a_16_bit_scale(host, dtype, top):
    g = torch.Generator().manual_seed(0)
    sc = _every(dtype)
    sc = sc[(sc >= 1e-6) & (sc < 3.4e38 / top)].repeat(64)
    d = _near_ties(sc, top, g)
    got = torch.empty_like(d)
    y = _off_by_an_ulp(1 / sc, g)
    host.codes16(*(ctypes.c_void_p(t.data_ptr()) for t in (d, sc, y, got)), ctypes.c_int(d.numel()))
    assert torch.equal(got, (d / sc).round())


@pytest.mark.parametrize("top", [15.0, 255.0])
def test_codes_by_a_32_bit_scale(host, top):
    g = torch.Generator().manual_seed(1)
    fp = torch.randn(1 << 21, generator=g).abs() * torch.exp(torch.randn(1 << 21, generator=g) * 4)
    sc = torch.cat([(fp.half().float() / top).clamp_min(1e-6), (fp.bfloat16().float() / top).clamp_min(1e-6), fp.clamp(1e-6, 1e30)])
    sc = sc[torch.isfinite(sc)]
    sc[:100] = torch.tensor(0x3fffffff, dtype=torch.int32).view(torch.float32)           # a mantissa of ones: left to the caller
    d = _near_ties(sc, top, g)
    got = torch.empty_like(d)
    y = _off_by_an_ulp(1 / sc, g)
    host.codes32(*(ctypes.c_void_p(t.data_ptr()) for t in (d, sc, y, got)), ctypes.c_int(d.numel()))
    assert got[:100].isnan().all() and torch.equal(got[100:][~got[100:].isnan()], (d / sc).round()[100:][~got[100:].isnan()])
    assert got[100:].isnan().sum() < 10
