"""The eight-tokens-per-warp TurboQuant kernel (csrc/fq_turbo_quant.cu) against the warp-per-token kernel, which rows that are
not 8-byte aligned take: equal bytes for ties, signs at zero, large, tiny and constant tokens, and every remainder of a tile."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _quant(x, stride_out=None):
    from flashquest_b200._lib import check, dtype_code, lib, ptr, stream_ptr
    B, H, n, D = x.shape
    so = stride_out or 0
    m = torch.zeros(B, H, n, D // 8 + so, dtype=torch.uint8, device="cuda")
    l = torch.zeros(B, H, n, D // 4 + so, dtype=torch.uint8, device="cuda")
    s = torch.zeros(B, H, n, dtype=torch.bfloat16, device="cuda")
    check(lib().fq_quantize_turbo(None, 0, 0, 0, 0, ptr(x), x.stride(0), x.stride(1), x.stride(2), n, dtype_code(x), B, H, D, n,
                                  ptr(m), *m.stride()[:3], ptr(l), *l.stride()[:3], ptr(s), *s.stride(), stream_ptr(x.device)))
    return m[..., :D // 8], l[..., :D // 4], s


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("n,offset,stride_out", [(1, 0, 0), (8, 4, 0), (31, 0, 4), (33, 4, 0), (40000, 0, 0)])
def test_equals_warp_per_token(dtype, n, offset, stride_out):
    g = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randn(1, 2, n, 128, device="cuda", generator=g)
    kind = torch.arange(n, device="cuda") % 8
    k = kind.view(1, 1, n, 1)
    x = torch.where(k == 1, (x * 2).round(), x)                        # few distinct values: ties
    x = torch.where(k == 2, x.sign() * 4, x)                           # a rotation of signs: multiples of one step
    x = torch.where(k == 3, x * 3000 / (6 if dtype == torch.float16 else 1), x)
    x = torch.where(k == 4, x * 1e-6, x)
    x = torch.where(k == 5, x * 0, x)
    x = torch.where(k == 6, x[..., :1].expand_as(x), x)                # one coefficient holds everything
    x = x.to(dtype)
    wide = torch.empty(1, 2, n, 128 + 8, dtype=dtype, device="cuda")
    fast = wide[..., offset:offset + 128]
    fast.copy_(x)
    odd = torch.empty(1, 2, n, 128 + 1, dtype=dtype, device="cuda")[..., 1:]
    odd.copy_(x)
    for a, b in zip(_quant(fast, stride_out), _quant(odd)):
        assert torch.equal(a, b)
