"""step_all on layers of equal length (one batch over all layers) against step layer by layer."""
import pytest
import torch

from ._util import bit_equal, make_kv, make_q

pytestmark = pytest.mark.gpu


def _engine(B, Ln, Hq, Hkv, D, page, seen, n_split):
    from flashquest_b200.cache.persistent_int4 import PersistentInt4KVCache
    from flashquest_b200.eager.decode_step import QuestDecodeInt4
    cache = PersistentInt4KVCache(batch_size=B, num_layers=Ln, num_kv_heads=Hkv, head_dim=D, max_seq_len=(seen // page + 2) * page,
                                  page_size=page, device="cuda", dtype=torch.float16)
    for li in range(Ln):
        if seen:
            cache.update_quantized(make_kv(10 + li, (B, Hkv, seen, D), torch.float16).cuda(), make_kv(20 + li, (B, Hkv, seen, D), torch.float16, outliers=()).cuda(), li)
    return cache, QuestDecodeInt4(cache, num_q_heads=Hq, retention=0.5, num_sinks=1, window_pages=1, q_dtype=torch.float16, n_split=n_split)


def _inputs(t, form, Ln, B, Hq, Hkv, n, D):
    k, v = (make_kv(30 + 10 * t + i, (Ln, B, Hkv, n, D), torch.float16).cuda() for i in range(2))
    q = make_q(50 + t, (Ln, B, Hq, 1, D), torch.float16).cuda()
    if form == "strided":          # q's and k's layers, sequences and heads apart from each other, in the parents' order
        q = torch.cat([q, q], dim=2)[:, :, :Hq]
        k, v = (torch.cat([x, x], dim=3)[:, :, :, :n] for x in (k, v))
    elif form == "sequence_major":  # layers inside the sequences: no stride covers both when B > 1
        q, k, v = (x.transpose(0, 1).contiguous().transpose(0, 1) for x in (q, k, v))
    elif form == "shared":          # one layer's tensors for all layers
        q, k, v = (x[:1].expand(Ln, *x.shape[1:]) for x in (q, k, v))
    return k, v, q


@pytest.mark.parametrize("B,Ln,Hq,Hkv,D,page,seen,n", [
    (1, 3, 24, 8, 128, 16, 0, 1),          # an empty cache: the staged token alone
    (1, 28, 24, 8, 128, 16, 515, 1),
    (2, 3, 6, 2, 64, 16, 127, 1),          # the append completes a page
    (3, 2, 8, 8, 128, 64, 300, 5),
    (1, 5, 32, 8, 128, 8, 1023, 1),
])
@pytest.mark.parametrize("form", ["dense", "strided", "sequence_major", "shared"])
@pytest.mark.parametrize("n_split", [1, 4, None])
def test_layers_together_equal_layers_alone(B, Ln, Hq, Hkv, D, page, seen, n, form, n_split):
    (ca, ea), (cb, eb) = (_engine(B, Ln, Hq, Hkv, D, page, seen, n_split) for _ in range(2))
    for t in range(2):
        k, v, q = _inputs(t, form, Ln, B, Hq, Hkv, n, D)
        Oa, la = (x.clone() for x in ea.step_all(k, v, q))
        each = [tuple(x.clone() for x in eb.step(k[li], v[li], q[li], li)) for li in range(Ln)]
        Ob, lb = (torch.stack(x) for x in zip(*each))
        if n_split == 1:
            assert bit_equal(Oa, Ob) and bit_equal(la, lb)
        else:
            # the same products, merged from another number of parts: an fp16 output can round to its neighbour (2^-10 of its
            # value, or of the 2^-14 below which fp16 has no finer steps), an fp32 logarithm moves by a few of its own roundings
            assert ((Oa.float() - Ob.float()).abs() <= Ob.float().abs() * 2 ** -10 + 2 ** -14).all()
            assert torch.allclose(la, lb, rtol=2e-6, atol=2e-6)
        # the scratch of every layer is ready for a step of that layer alone, and the other way round
        k1, v1, q1 = _inputs(t + 5, "dense", Ln, B, Hq, Hkv, 1, D)
        if max(ca._seen_tokens) + 1 + n <= ca.max_seq_len:
            for li in range(Ln):
                ra, rb = ea.step(k1[li], v1[li], q1[li], li), eb.step(k1[li], v1[li], q1[li], li)
                assert bit_equal(ra[0], rb[0]) and bit_equal(ra[1], rb[1])
    for name in ("K_packed", "V_packed", "K_scale", "K_mn", "V_scale", "V_mn", "K_partial", "V_partial"):
        a, b = getattr(ca, name), getattr(cb, name)
        done = ca._seen_tokens[0] // page * page
        if name in ("K_packed", "V_packed", "V_scale", "V_mn"):
            a, b = a[:, :, :, :done], b[:, :, :, :done]
        elif name in ("K_scale", "K_mn"):
            a, b = a[:, :, :, :done // page], b[:, :, :, :done // page]
        else:
            a, b = a[:, :, :, :ca._seen_tokens[0] - done], b[:, :, :, :ca._seen_tokens[0] - done]
        assert bit_equal(a, b), name


@pytest.mark.parametrize("bits", [3, 4, 8])
@pytest.mark.parametrize("B,Hq,Hkv,D,page,seen,n", [(1, 24, 8, 128, 16, 40, 1), (2, 32, 8, 64, 64, 130, 1), (3, 6, 2, 128, 16, 160, 15),
                                                    (1, 12, 2, 128, 32, 66, 7), (2, 8, 8, 64, 16, 31, 1), (1, 24, 8, 128, 64, 127, 64)])
def test_rows_staged_with_the_scores(bits, B, Hq, Hkv, D, page, seen, n):
    """A step whose tokens complete no page stages them in the launch of the scores (the last two complete one, in a launch of
    their own): the staged rows, and what the same step gives after an append by itself."""
    from flashquest_b200.cache.persistent_int4 import PersistentInt4KVCache
    from flashquest_b200.cache.persistent_int8 import PersistentInt8KVCache
    from flashquest_b200.cache.persistent_turbo import PersistentTurboKVCache
    from flashquest_b200.eager.decode_step import QuestDecodeInt4, QuestDecodeInt8, QuestDecodeTurbo
    C, E = {3: (PersistentTurboKVCache, QuestDecodeTurbo), 4: (PersistentInt4KVCache, QuestDecodeInt4), 8: (PersistentInt8KVCache, QuestDecodeInt8)}[bits]
    k0, v0 = (make_kv(i, (B, Hkv, seen, D), torch.float16).cuda() for i in (1, 2))
    k, v = (make_kv(i, (B, Hkv, 2 * n, D), torch.float16).cuda()[:, :, ::2] for i in (3, 4))
    q = make_q(5, (B, Hq, 1, D), torch.float16).cuda()
    outs = []
    for along in (True, False):
        cache = C(batch_size=B, num_layers=2, num_kv_heads=Hkv, head_dim=D, max_seq_len=(seen + n) // page * page + 2 * page, page_size=page,
                  device="cuda", dtype=torch.float16)
        step = E(cache, num_q_heads=Hq, retention=0.5, num_sinks=1, window_pages=1, q_dtype=torch.float16)
        cache.update_quantized(k0, v0, 1)
        if along:
            O, lse = step.step(k, v, q, 1)
        else:
            cache.update_quantized(k, v, 1)
            O, lse = step.step(k[:, :, :0], v[:, :, :0], q, 1)
        left = (seen + n) % page
        outs.append((O.clone(), lse.clone(), cache.K_partial[1, :, :, :left].clone(), cache.V_partial[1, :, :, :left].clone()))
        if left and left >= n:
            assert bit_equal(outs[-1][2][:, :, left - n:], k) and bit_equal(outs[-1][3][:, :, left - n:], v)
    assert all(bit_equal(a, b) for a, b in zip(*outs))
