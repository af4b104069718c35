"""Bulk packing kernel (csrc/fq_quant_pages.cu) against the CPU oracle, bit for bit: every page size, head dimension and code
width it takes, staged heads, left-over tokens, values on rounding ties, constant and extreme rows."""
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu


def _data(B, H, S, D, dtype, seed):
    g = torch.Generator().manual_seed(seed)
    x = torch.randn(B, H, S, D, generator=g)
    x[..., 5:: D // 4] *= 8
    x[:, :, 3] = 0.25                                                     # a constant row
    x[:, :, : S // 2, 7] = torch.arange(S // 2) % 16 * 0.5 - 2             # quotients on and next to half-integers
    x[:, :, 6] = torch.linspace(-7.5, 7.5, D)
    x[:, :, 9] *= 1e-6
    x[:, :, 11] *= 3e3
    return x.to(dtype)


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("page", [16, 32, 64])
@pytest.mark.parametrize("D,dtype,B,S,first", [(128, torch.float16, 2, 64 * 3 + 5, 0), (128, torch.bfloat16, 1, 64 * 5, 13),
                                              (64, torch.bfloat16, 2, 64 * 2 + 63, 7), (64, torch.float16, 1, 64, 15)])
def test_bulk_append_matches_oracle(bits, page, D, dtype, B, S, first):
    from flashquest_b200.cache.persistent_int4 import PersistentInt4KVCache
    from flashquest_b200.cache.persistent_int8 import PersistentInt8KVCache
    H = 3
    K, V = _data(B, H, S, D, dtype, 1), _data(B, H, S, D, dtype, 2)
    cache = (PersistentInt4KVCache if bits == 4 else PersistentInt8KVCache)(
        batch_size=B, num_layers=2, num_kv_heads=H, head_dim=D, max_seq_len=S + page, page_size=page, dtype=dtype)
    if first:                                                              # a staged head in front of the bulk
        cache.update_quantized(K[:, :, :first].cuda(), V[:, :, :first].cuda(), 1)
    cache.update_quantized(K[:, :, first:].cuda(), V[:, :, first:].cuda(), 1)
    n = S // page * page
    views = cache.get_views(1)
    qk, qv = (oracle.quantize_k_int4, oracle.quantize_v_int4) if bits == 4 else (oracle.quantize_k, oracle.quantize_v)
    names = ("K_packed", "V_packed") if bits == 4 else ("K_uint8", "V_uint8")
    for got, want in zip((views[names[0]], views["K_scale"], views["K_mn"]), qk(K[:, :, :n], page)):
        assert torch.equal(got.cpu(), want)
    for got, want in zip((views[names[1]], views["V_scale"], views["V_mn"]), qv(V[:, :, :n])):
        assert torch.equal(got.cpu(), want)
    assert torch.equal(views["K_partial"].cpu(), K[:, :, n:]) and torch.equal(views["V_partial"].cpu(), V[:, :, n:])
    if bits == 8:
        assert not cache.K_partial[1, :, :, S - n:].any() and not cache.V_partial[1, :, :, S - n:].any()


@pytest.mark.parametrize("bits", [3, 4, 8])
@pytest.mark.parametrize("page", [16, 64])
def test_page_range_at_the_top_of_bf16(bits, page):
    """Ranges of 3.0e38 up to the largest finite bf16 value and beyond it: the scale is the rounded quotient, not the range."""
    from flashquest_b200.cache.persistent_int4 import PersistentInt4KVCache
    from flashquest_b200.cache.persistent_int8 import PersistentInt8KVCache
    from flashquest_b200.cache.persistent_turbo import PersistentTurboKVCache
    D, S = 128, 2 * page
    K = _data(1, 2, S, D, torch.bfloat16, 3).float()
    top = torch.linspace(2.9e38, 3.38e38, 64)                               # every range that the old limit of 3.0e38 cut off
    K[:, :, 0::2, 64:], K[:, :, 1::2, 64:] = top / 2, -top / 2
    K[:, :, :page, 0], K[:, :, page - 1, 0] = 3.3e38, -3.3e38               # an infinite range
    K = K.bfloat16()
    V = _data(1, 2, S, D, torch.bfloat16, 4)
    cache = {3: PersistentTurboKVCache, 4: PersistentInt4KVCache, 8: PersistentInt8KVCache}[bits](
        batch_size=1, num_layers=1, num_kv_heads=2, head_dim=D, max_seq_len=S, page_size=page, dtype=torch.bfloat16)
    cache.update_quantized(K.cuda(), V.cuda(), 0)
    views = cache.get_views(0)
    if bits == 8:
        want = oracle.quantize_k(K, page)
        got = views["K_uint8"], views["K_scale"], views["K_mn"]
    else:
        want = oracle.quantize_k_int4(K, page)
        got = (views["K_packed"], views["K_scale"], views["K_mn"]) if bits == 4 else (None, views["K_scale_raw"], views["K_mn_raw"])
    assert torch.isfinite(want[1][..., 64:].float()).all() and want[1][..., 64:].float().max() < 3e37
    assert torch.equal(got[1].cpu(), want[1]) and torch.equal(got[2].cpu(), want[2])
    if bits != 3:
        assert torch.equal(got[0].cpu()[..., (bits * 64) // 8:], want[0][..., (bits * 64) // 8:])       # the channels of finite range


@pytest.mark.parametrize("model,stage", [(torch.bfloat16, torch.bfloat16), (torch.float16, torch.bfloat16), (torch.float16, torch.float16)])
@pytest.mark.parametrize("D", [64, 128])
def test_rope_of_the_patched_forward_matches_hugging_face(model, stage, D):
    """q, k, v that go into the cache: the bits of apply_rotary_pos_emb followed by the cast."""
    from transformers.models.llama.modeling_llama import apply_rotary_pos_emb

    from flashquest_b200.cache.persistent_int8 import PersistentInt8KVCache
    from flashquest_b200.eager.decode_step import QuestDecodeInt8
    B, Hq, Hkv = 3, 6, 2
    g = torch.Generator(device="cuda").manual_seed(3)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g).to(model)
    cache = PersistentInt8KVCache(batch_size=B, num_layers=1, num_kv_heads=Hkv, head_dim=D, max_seq_len=64, page_size=16, dtype=stage)
    engine = QuestDecodeInt8(cache, num_q_heads=Hq, q_dtype=stage)
    q, k, v, cos, sin = r(B, 1, Hq * D), r(B, 1, Hkv * D), r(B, 1, Hkv * D), r(B, 1, D), r(B, 1, D)
    O = engine.forward_token(q, k, v, cos, sin, 0)
    want_q, want_k = apply_rotary_pos_emb(q.view(B, 1, Hq, D).transpose(1, 2), k.view(B, 1, Hkv, D).transpose(1, 2), cos, sin)
    assert torch.equal(engine.q_rot, want_q.to(stage)) and torch.equal(engine.k_rot, want_k.to(stage))
    want_v = v.view(B, 1, Hkv, D).transpose(1, 2).to(stage)
    assert torch.equal(cache.K_partial[0, :, :, :1], want_k.to(stage)) and torch.equal(cache.V_partial[0, :, :, :1], want_v)
    # one staged token: its value is the output
    assert torch.allclose(O.float(), want_v.float().repeat_interleave(Hq // Hkv, 1), atol=1e-3)
    assert cache.get_seq_length() == 1


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_values_that_are_not_numbers(bits, dtype):
    """Infinities and NaNs in K and V: the codes of the channels and tokens that have them, and of their neighbours."""
    from flashquest_b200.cache.persistent_int4 import PersistentInt4KVCache
    from flashquest_b200.cache.persistent_int8 import PersistentInt8KVCache
    D, S, page = 128, 64, 16
    outs = []
    for first in (0, 1):                        # whole pages at once, and (one token first) the general kernel's last pages
        K, V = _data(1, 2, S, D, dtype, 5), _data(1, 2, S, D, dtype, 6)
        for x in (K, V):
            x[0, 0, 17, 5], x[0, 0, 33, 70], x[0, 1, 18, 9] = float("inf"), float("-inf"), float("nan")
        cache = (PersistentInt4KVCache if bits == 4 else PersistentInt8KVCache)(
            batch_size=1, num_layers=1, num_kv_heads=2, head_dim=D, max_seq_len=S, page_size=page, dtype=dtype)
        if first:
            for t in range(S):
                cache.update_quantized(K[:, :, t:t + 1].cuda(), V[:, :, t:t + 1].cuda(), 0)
        else:
            cache.update_quantized(K.cuda(), V.cuda(), 0)
        outs.append(cache)
    for name in (("K_packed", "V_packed") if bits == 4 else ("K_uint8", "V_uint8")):
        assert torch.equal(getattr(outs[0], name), getattr(outs[1], name)), name
