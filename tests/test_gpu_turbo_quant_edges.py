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


@pytest.mark.parametrize("page", [16, 32])
@pytest.mark.parametrize("pieces", [(1, 15, 16, 1), (5, 30, 300), (20, 12, 3, 2049)])
def test_append_pieces(page, pieces):
    """The one-launch append (planes, page metadata, staging), piece by piece, against the whole stream through the general kernels."""
    from flashquest_b200.cache.persistent_turbo import PersistentTurboKVCache
    from flashquest_b200.kernel.kv_quant import quantize_k_turbo
    g = torch.Generator(device="cuda").manual_seed(sum(pieces))
    c = PersistentTurboKVCache(batch_size=2, num_layers=2, num_kv_heads=3, head_dim=128, max_seq_len=4096, page_size=page, dtype=torch.float16)
    K, V = (torch.randn(2, 3, sum(pieces), 128, device="cuda", generator=g).half() for _ in range(2))
    at = 0
    for n in pieces:
        c.update_quantized(K[:, :, at:at + n], V[:, :, at:at + n], 1)
        at += n
        done = at // page * page
        w = c.get_views(1)
        assert torch.equal(w["K_partial"], K[:, :, done:at]) and torch.equal(w["V_partial"], V[:, :, done:at])
        if not done:
            continue
        odd = torch.empty(2, 2, 3, done, 129, dtype=torch.float16, device="cuda")[..., 1:]
        odd[0].copy_(K[:, :, :done]), odd[1].copy_(V[:, :, :done])
        for name, x in (("K", odd[0]), ("V", odd[1])):
            m, l, sc = _quant(x)
            assert torch.equal(w[name + "_msb"], m) and torch.equal(w[name + "_lsb"], l) and torch.equal(w[name + "_scale_turbo"][..., 0], sc)
        _, _, _, sr, mr = quantize_k_turbo(K[:, :, :done].contiguous(), page)
        assert torch.equal(w["K_scale_raw"], sr) and torch.equal(w["K_mn_raw"], mr)
