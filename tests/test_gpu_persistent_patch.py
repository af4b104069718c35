"""patch_llama_for_quest_persistent on a random-init tiny Hugging Face LlamaModel: prefill, then
teacher-forced decode steps across page boundaries, for the INT4 cache (bool-mask path against
compact path) and the TurboQuant cache, every attention call checked against the oracle chain on the
very q / k / v that went into it (reference test: tests/test_persistent_patch_compact.py:10-66)."""
import math

import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu


def _tiny_llama():
    from transformers import AutoConfig
    from transformers.models.llama.modeling_llama import LlamaModel
    cfg = AutoConfig.for_model("llama", hidden_size=256, num_attention_heads=4, num_key_value_heads=2, num_hidden_layers=2,
                               intermediate_size=256, max_position_embeddings=512, vocab_size=128)
    cfg.head_dim = 64
    torch.manual_seed(42)
    return cfg, LlamaModel(cfg).cuda().to(torch.bfloat16).eval()


def _dense_causal(q, K, V):
    """fp32 reference of the prefill branch: query i sees keys 0..i, grouped-query heads."""
    B, Hq, Sq, D = q.shape
    n_rep = Hq // K.shape[1]
    Kf, Vf = K.float().repeat_interleave(n_rep, 1), V.float().repeat_interleave(n_rep, 1)
    s = q.float() @ Kf.transpose(-1, -2) / math.sqrt(D)
    i, j = torch.arange(Sq)[:, None], torch.arange(K.shape[2])[None, :]
    s = s.masked_fill(j > i, float("-inf"))
    return torch.softmax(s, -1) @ Vf


class _OracleCheck:
    """Replays every traced attention call on the CPU oracle."""

    def __init__(self, kv_bits, page, n_layers, H_q, retention_rows, sinks, window, k_max_static, fused_tail):
        self.bits, self.page, self.sinks, self.window, self.kms, self.fused = kv_bits, page, sinks, window, k_max_static, fused_tail
        self.K, self.V = [None] * n_layers, [None] * n_layers
        self.ret = retention_rows                       # per layer: (H_q,) fp32 retention per query head
        self.worst = {"prefill": 0.0, "decode": 0.0}
        self.calls = 0

    def __call__(self, li, q, k, v, attn):
        q, k, v, attn = q.cpu(), k.cpu(), v.cpu(), attn.float().cpu()
        self.K[li] = k if self.K[li] is None else torch.cat([self.K[li], k], 2)
        self.V[li] = v if self.V[li] is None else torch.cat([self.V[li], v], 2)
        K, V, page = self.K[li], self.V[li], self.page
        S = K.shape[2]
        nq = S - S % page
        self.calls += 1
        if q.shape[2] > 1:
            if self.bits == 4:
                kq, vq = oracle.quantize_k_int4(K[:, :, :nq], page), oracle.quantize_v_int4(V[:, :, :nq])
                Kd, Vd = oracle.dequantize_k_int4(*kq, page), oracle.dequantize_v_int4(*vq)
            elif self.bits == 8:
                kq, vq = oracle.quantize_k(K[:, :, :nq], page), oracle.quantize_v(V[:, :, :nq])
                Kd, Vd = oracle.dequantize_k(*kq, page), oracle.dequantize_v(*vq)
            else:
                kq, vq = oracle.quantize_k_turbo(K[:, :, :nq], page), oracle.quantize_v_turbo(V[:, :, :nq])
                Kd = oracle.dequantize_k_turbo(kq[0], kq[1], kq[2], head_dim=K.shape[-1])
                Vd = oracle.dequantize_v_turbo(vq[0], vq[1], vq[2], head_dim=K.shape[-1])
            want = _dense_causal(q, torch.cat([Kd.to(K.dtype), K[:, :, nq:]], 2), torch.cat([Vd.to(V.dtype), V[:, :, nq:]], 2))
            err = (attn - want).abs().max().item()
            self.worst["prefill"] = max(self.worst["prefill"], err)
            assert err <= 8e-3, ("prefill", li, err)          # bf16 probabilities and output: two bf16 ulps at |O| ~ 1
            return
        Kt, Vt = K[:, :, nq:], V[:, :, nq:]
        r = self.ret[li]
        if self.bits in (4, 8):
            qk, qv, sc, at = ((oracle.quantize_k_int4, oracle.quantize_v_int4, oracle.page_scores_int4_fast, oracle.sparse_attn_int4)
                              if self.bits == 4 else
                              (oracle.quantize_k, oracle.quantize_v, oracle.page_scores_int8_fast, oracle.sparse_attn_int8))
            kv = qk(K[:, :, :nq], page) + qv(V[:, :, :nq])
            if nq:
                mask = oracle.select_pages_vectorized(sc(q, kv[1], kv[2]), r, self.sinks, self.window, k_max_static=self.kms)
            else:
                mask = torch.zeros(q.shape[0], q.shape[1], 1, 0, dtype=torch.bool)
            want, _ = at(q, *kv, selection_mask=mask, page_size=page, K_partial=Kt, V_partial=Vt)
            tol = 2e-3 + 2 ** -8 * want.abs() * (1 if self.fused else 3)   # separate bf16 partials + merge: two more roundings
        else:
            kq, vq = oracle.quantize_k_turbo(K[:, :, :nq], page), oracle.quantize_v_turbo(V[:, :, :nq])
            parts_O, parts_l = [], []
            if nq:
                mask = oracle.select_pages_vectorized(oracle.page_scores_int4_fast(q, kq[3], kq[4]), r, self.sinks, self.window,
                                                      k_max_static=self.kms)
                O1, l1 = oracle.sparse_attn_turbo(q, kq[0], kq[1], kq[2], vq[0], vq[1], vq[2], selection_mask=mask, page_size=page)
                parts_O.append(O1); parts_l.append(l1)
            if S > nq or not nq:
                e8 = torch.empty(q.shape[0], K.shape[1], 0, K.shape[-1] // 2, dtype=torch.uint8)
                em = torch.empty(q.shape[0], K.shape[1], 0, K.shape[-1], dtype=torch.bfloat16)
                ev = torch.empty(q.shape[0], K.shape[1], 0, 1, dtype=torch.bfloat16)
                O2, l2 = oracle.sparse_attn_int4(q, e8, em, em, e8, ev, ev, selected_page_ids=torch.full((q.shape[0], q.shape[1], 1, 1), -1, dtype=torch.int32),
                                                 page_size=page, K_partial=Kt, V_partial=Vt)
                parts_O.append(O2); parts_l.append(l2)
            want, _ = oracle.lse_merge(torch.stack(parts_O), torch.stack(parts_l))
            tol = 2e-2 + 0 * want                   # q and O pass through bf16 rotations (the reference's own test bound is 5e-2)
        err = (attn - want).abs()
        self.worst["decode"] = max(self.worst["decode"], float((err / tol).max()))
        assert (err <= tol).all(), ("decode", li, S, float(err.max()))


def _run(model, cache, ids_prompt, ids_steps):
    outs = []
    with torch.no_grad():
        outs.append(model(ids_prompt, past_key_values=cache).last_hidden_state)
        for t in range(ids_steps.shape[1]):
            outs.append(model(ids_steps[:, t:t + 1], past_key_values=cache).last_hidden_state)
    return torch.cat(outs, 1)


@pytest.mark.parametrize("kv_bits,page", [(4, 8), (4, 16), (3, 16), (8, 16)])
def test_patched_forward_paths_and_oracle(kv_bits, page):
    from flashquest_b200.cache.persistent_int4 import PersistentInt4KVCache
    from flashquest_b200.cache.persistent_int8 import PersistentInt8KVCache
    from flashquest_b200.cache.persistent_turbo import PersistentTurboKVCache
    from flashquest_b200.eager import llama_persistent_patch as lpp
    from transformers.cache_utils import Cache
    cfg, model_a = _tiny_llama()
    Cls = {4: PersistentInt4KVCache, 8: PersistentInt8KVCache, 3: PersistentTurboKVCache}[kv_bits]
    mk = lambda: Cls(num_layers=2, batch_size=1, num_kv_heads=2, head_dim=64, page_size=page, max_seq_len=128)
    cache_a = mk()
    assert isinstance(cache_a, Cache) and cache_a.kv_bits == kv_bits
    head_pattern = torch.tensor([[True, True], [True, False]])          # one streaming KV head in layer 1
    retention, sinks, window = 0.5, 2, 1
    kw = dict(head_pattern=head_pattern, retention=retention, num_sinks=sinks, window_pages=window, page_size=page)
    torch.manual_seed(0)
    prompt = torch.randint(0, 128, (1, 37), device="cuda")
    steps = torch.randint(0, 128, (1, 30), device="cuda")            # crosses page boundaries at either page size
    k_max_static = math.ceil(retention * (128 // page))
    rows = [torch.where(head_pattern[l].repeat_interleave(2), torch.tensor(retention), torch.tensor(0.0)).float() for l in range(2)]

    lpp.patch_llama_for_quest_persistent(model_a, cache=cache_a, use_compact_kernel=False, **kw)
    chk_a = _OracleCheck(kv_bits, page, 2, 4, rows, sinks, window, k_max_static, fused_tail=False)
    lpp.TRACE = chk_a
    try:
        out_a = _run(model_a, cache_a, prompt, steps)
    finally:
        lpp.TRACE = None
    assert chk_a.calls == 2 * 31 and cache_a.get_seq_length() == 67
    print(f"kv_bits={kv_bits} page={page} worst prefill error {chk_a.worst['prefill']:.2e}, decode {chk_a.worst['decode']:.2f} of the bound")
    if kv_bits != 4:
        with pytest.raises(NotImplementedError, match="kv_bits=4"):
            lpp.make_quest_persistent_forward(cache=cache_a, head_pattern_layer=head_pattern[0], retention=0.5, num_sinks=2,
                                              window_pages=1, page_size=page, use_compact_kernel=True)
        return
    # path B: compact kernel, same weights (reference test: both paths agree within 5e-2)
    _, model_b = _tiny_llama()
    model_b.load_state_dict(model_a.state_dict())
    cache_b = mk()
    lpp.patch_llama_for_quest_persistent(model_b, cache=cache_b, use_compact_kernel=True, **kw)
    chk_b = _OracleCheck(kv_bits, page, 2, 4, rows, sinks, window, k_max_static, fused_tail=True)
    lpp.TRACE = chk_b
    try:
        out_b = _run(model_b, cache_b, prompt, steps)
    finally:
        lpp.TRACE = None
    # The reference's own test compares the two paths after a prefill only, at 5e-2.  Here 30 free-running
    # decode steps follow: a last-bit difference in one layer's output can move a 4-bit code of the next
    # layer's k / v by one step, so a few elements drift further; both paths are held to the oracle call by
    # call above, here the prefill must agree at the reference's bound and the decode steps in bulk.
    torch.testing.assert_close(out_b[:, :37], out_a[:, :37], atol=5e-2, rtol=5e-2)
    diff = (out_b.float() - out_a.float()).abs()
    assert (diff > 5e-2 + 5e-2 * out_a.float().abs()).float().mean().item() < 0.02 and diff.max().item() < 1.0, diff.max().item()
    for name in ("K_packed", "V_packed", "K_scale", "K_mn", "V_scale", "V_mn"):
        va, vb = cache_a.get_views(1)[name], cache_b.get_views(1)[name]
        assert va.shape == vb.shape


def test_patch_argument_errors():
    from flashquest_b200.cache.persistent_int4 import PersistentInt4KVCache
    from flashquest_b200.eager import llama_persistent_patch as lpp
    cfg, model = _tiny_llama()
    cache = PersistentInt4KVCache(num_layers=2, batch_size=1, num_kv_heads=2, head_dim=64, page_size=16, max_seq_len=64)
    with pytest.raises(ValueError, match="2D"):
        lpp.patch_llama_for_quest_persistent(model, cache=cache, head_pattern=torch.ones(2, dtype=torch.bool))
    with pytest.raises(ValueError, match="head_pattern has 1 layers"):
        lpp.patch_llama_for_quest_persistent(model, cache=cache, head_pattern=torch.ones(1, 2, dtype=torch.bool), page_size=16)
    with pytest.raises(RuntimeError, match="no LlamaAttention"):
        lpp.patch_llama_for_quest_persistent(torch.nn.Linear(2, 2), cache=cache, head_pattern=torch.ones(2, 2, dtype=torch.bool))

    class Fake:
        kv_bits, head_dim, max_seq_len, page_size = 8, 64, 64, 16
    with pytest.raises(NotImplementedError, match="kv_bits=4"):
        lpp.make_quest_persistent_forward(cache=Fake(), head_pattern_layer=torch.ones(2, dtype=torch.bool), retention=0.5,
                                          num_sinks=2, window_pages=1, page_size=16, use_compact_kernel=True)


def _oracle_checked_run(kv_bits, page, head_dim=64, model_dtype=torch.bfloat16, compact=False, n_steps=None, fused=True):
    """Prefill and decode steps across a page end, every attention call replayed on the oracle; returns (cache, patched model)."""
    from flashquest_b200.cache.persistent_int4 import PersistentInt4KVCache
    from flashquest_b200.cache.persistent_int8 import PersistentInt8KVCache
    from flashquest_b200.cache.persistent_turbo import PersistentTurboKVCache
    from flashquest_b200.eager import llama_persistent_patch as lpp
    from transformers import AutoConfig
    from transformers.models.llama.modeling_llama import LlamaModel
    cfg = AutoConfig.for_model("llama", hidden_size=256, num_attention_heads=4, num_key_value_heads=2, num_hidden_layers=2,
                               intermediate_size=256, max_position_embeddings=512, vocab_size=128, head_dim=head_dim)
    torch.manual_seed(7)
    model = LlamaModel(cfg).cuda().to(model_dtype).eval()
    S, n_steps = 4 * page - 3, n_steps or 7
    cache = {3: PersistentTurboKVCache, 4: PersistentInt4KVCache, 8: PersistentInt8KVCache}[kv_bits](
        num_layers=2, batch_size=1, num_kv_heads=2, head_dim=head_dim, page_size=page, max_seq_len=8 * page)
    pattern = torch.tensor([[True, True], [True, False]])
    retention, sinks, window = 0.5, 2, 1
    lpp.patch_llama_for_quest_persistent(model, cache=cache, head_pattern=pattern, retention=retention, num_sinks=sinks, window_pages=window,
                                         page_size=page, use_compact_kernel=compact)
    rows = [torch.where(pattern[l].repeat_interleave(2), torch.tensor(retention), torch.tensor(0.0)).float() for l in range(2)]
    g = torch.Generator(device="cuda").manual_seed(8)
    ids = torch.randint(0, 128, (1, S + n_steps), device="cuda", generator=g)
    check = _OracleCheck(kv_bits, page, 2, 4, rows, sinks, window, math.ceil(retention * 8), fused_tail=fused)
    lpp.TRACE = check
    try:
        _run(model, cache, ids[:, :S], ids[:, S:])
    finally:
        lpp.TRACE = None
    assert check.calls == 2 * (1 + n_steps) and cache.get_seq_length() == S + n_steps
    return cache, model


@pytest.mark.parametrize("kv_bits,compact", [(3, False), (4, False), (4, True), (8, False)])
def test_fp32_model_on_a_16_bit_cache(kv_bits, compact):
    """Outside the dtypes of the one-call route: Hugging Face's rotary embedding, then the native step."""
    _oracle_checked_run(kv_bits, 16, model_dtype=torch.float32, compact=compact)


@pytest.mark.parametrize("kv_bits,page,compact,model_dtype,where", [
    (4, 16, False, torch.bfloat16, "cuda"), (4, 16, True, torch.bfloat16, "cuda"), (8, 16, False, torch.bfloat16, "cuda"),
    (8, 8, False, torch.bfloat16, "cuda"), (3, 16, False, torch.bfloat16, "cuda"), (4, 16, False, torch.float32, "cuda"),
    (4, 16, False, torch.bfloat16, "cpu"), (4, 16, False, torch.bfloat16, "column")])
def test_head_pattern_changed_between_tokens(kv_bits, page, compact, model_dtype, where):
    """head_pattern_layer is read at every call: changed in place between two requests it gives what a forward made with the
    new pattern gives."""
    from types import SimpleNamespace

    from flashquest_b200.cache.persistent_int4 import PersistentInt4KVCache
    from flashquest_b200.cache.persistent_int8 import PersistentInt8KVCache
    from flashquest_b200.cache.persistent_turbo import PersistentTurboKVCache
    from flashquest_b200.eager.llama_persistent_patch import make_quest_persistent_forward
    Hq, Hkv, D, n = 4, 2, 64, 20 * page + 3
    g = torch.Generator(device="cuda").manual_seed(10)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)
    cache = {3: PersistentTurboKVCache, 4: PersistentInt4KVCache, 8: PersistentInt8KVCache}[kv_bits](
        batch_size=1, num_layers=1, num_kv_heads=Hkv, head_dim=D, max_seq_len=24 * page, page_size=page)
    cache.update_quantized(r(1, Hkv, n, D).bfloat16(), r(1, Hkv, n, D).bfloat16(), 0)
    linear = lambda w: lambda x: torch.nn.functional.linear(x, w)
    module = SimpleNamespace(head_dim=D, layer_idx=0, q_proj=linear(r(Hq * D, 32).to(model_dtype)), k_proj=linear(r(Hkv * D, 32).to(model_dtype)),
                             v_proj=linear(r(Hkv * D, 32).to(model_dtype)), o_proj=linear(torch.eye(Hq * D, device="cuda").to(model_dtype)))
    hidden, angle = r(1, 1, 32).to(model_dtype), r(1, 1, D)
    rope = (angle.cos().to(model_dtype), angle.sin().to(model_dtype))

    def pattern(*rows):
        t = torch.tensor(rows, device="cpu" if where == "cpu" else "cuda")
        return torch.stack([t, ~t], 1)[:, 0] if where == "column" else t

    def make(p):
        f = make_quest_persistent_forward(cache=cache, head_pattern_layer=p, retention=0.5, num_sinks=1, window_pages=1, page_size=page,
                                          use_compact_kernel=compact)

        def call():
            cache._seen_tokens[0] = n
            return f(module, hidden, rope, past_key_values=cache)[0].clone()
        return call
    live = pattern(True, False)
    call = make(live)
    first = call()
    assert torch.equal(first, make(pattern(True, False))())
    for rows in ((False, True), (True, True), (False, False), (True, False)):
        live.copy_(torch.tensor(rows))
        want = make(pattern(*rows))()
        assert torch.equal(call(), want)
        assert rows == (True, False) or not torch.equal(want, first)


def _small(kv_bits, page, D=64, dtype=torch.bfloat16, **kw):
    """A layer with a few pages cached and its patched forward: (call, cache)."""
    from types import SimpleNamespace

    from flashquest_b200.cache.persistent_int4 import PersistentInt4KVCache
    from flashquest_b200.cache.persistent_int8 import PersistentInt8KVCache
    from flashquest_b200.cache.persistent_turbo import PersistentTurboKVCache
    from flashquest_b200.eager.llama_persistent_patch import make_quest_persistent_forward
    g = torch.Generator(device="cuda").manual_seed(11)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()
    Hq, Hkv, n = 4, 2, 9 * page + 3
    cache = {3: PersistentTurboKVCache, 4: PersistentInt4KVCache, 8: PersistentInt8KVCache}[kv_bits](
        batch_size=1, num_layers=1, num_kv_heads=Hkv, head_dim=D, max_seq_len=12 * page, page_size=page, dtype=dtype)
    cache.update_quantized(r(1, Hkv, n, D).to(dtype), r(1, Hkv, n, D).to(dtype), 0)
    linear = lambda w: lambda x: torch.nn.functional.linear(x, w)
    module = SimpleNamespace(head_dim=D, layer_idx=0, q_proj=linear(r(Hq * D, 32)), k_proj=linear(r(Hkv * D, 32)), v_proj=linear(r(Hkv * D, 32)),
                             o_proj=linear(r(32, Hq * D)))
    hidden, rope = r(1, 1, 32), (r(1, 1, D), r(1, 1, D))
    kw = dict(dict(head_pattern_layer=torch.tensor([True, False], device="cuda"), retention=0.5, num_sinks=1, window_pages=1, page_size=page), **kw)
    forward = make_quest_persistent_forward(cache=cache, **kw)

    def call():
        cache._seen_tokens[0] = n
        return forward(module, hidden, rope, past_key_values=cache)[0].clone()
    return call, cache


@pytest.mark.parametrize("kv_bits,page", [(4, 16), (8, 16), (8, 8)])
def test_mask_route_keeps_every_page_for_a_retention_above_one(kv_bits, page):
    assert torch.equal(_small(kv_bits, page, retention=1.5)[0](), _small(kv_bits, page, retention=1.0)[0]())


@pytest.mark.parametrize("kv_bits,compact", [(4, True), (3, False)])
def test_other_routes_refuse_a_retention_above_one(kv_bits, compact):
    with pytest.raises(ValueError, match="retention must be in"):
        _small(kv_bits, 16, retention=1.5, use_compact_kernel=compact)[0]()


@pytest.mark.parametrize("dtype", [torch.int64, torch.float32])
def test_pattern_dtypes(dtype):
    """torch.where takes a boolean pattern in the mask sequence; the other routes convert theirs."""
    pattern = torch.tensor([1, 0], device="cuda", dtype=dtype)
    for kv_bits, page in ((4, 16), (8, 16), (8, 8)):
        call, cache = _small(kv_bits, page, head_pattern_layer=pattern)
        with pytest.raises(RuntimeError, match="boolean tensor"):
            call()
    for kw in (dict(kv_bits=4, use_compact_kernel=True), dict(kv_bits=3)):
        assert torch.equal(_small(page=16, head_pattern_layer=pattern, **kw)[0](), _small(page=16, **kw)[0]())
    assert torch.equal(_small(4, 16, head_pattern_layer=pattern.to(torch.uint8))[0](), _small(4, 16)[0]())


@pytest.mark.parametrize("kv_bits,compact", [(3, False), (4, False), (4, True)])
def test_unsupported_forms_raise_what_the_kernels_say(kv_bits, compact):
    """head_dim 256 and fp32 caches: the attention's own errors, not those of the rotary launch in front of it."""
    with pytest.raises(NotImplementedError, match="head_dim=256 not in"):
        _small(kv_bits, 16, D=256, use_compact_kernel=compact)[0]()
    with pytest.raises(RuntimeError, match="cache dtype code 0"):
        _small(kv_bits, 16, dtype=torch.float32, use_compact_kernel=compact)[0]()


@pytest.mark.parametrize("kv_bits,page,compact", [(3, 16, False), (4, 16, False), (4, 16, True), (8, 16, False), (8, 8, False)])
def test_storage_replaced_between_tokens(kv_bits, page, compact):
    """A cache whose tensors have been replaced (restored from a file, say) is read where it is now."""
    call, cache = _small(kv_bits, page, use_compact_kernel=compact)
    want = call()
    old = {n: t for n, t in vars(cache).items() if torch.is_tensor(t)}
    for n, t in old.items():
        setattr(cache, n, t.clone())
        t.zero_()
    assert torch.equal(call(), want)
    assert not any(t.any() for t in old.values())                    # and nothing is written to what it was


@pytest.mark.parametrize("kv_bits,page,head_dim,compact", [(4, 64, 64, False), (4, 64, 128, True), (4, 16, 128, False), (8, 64, 128, False), (8, 32, 64, False),
                                                           (3, 64, 128, False), (3, 16, 128, False), (8, 8, 64, False), (8, 128, 128, False)])
def test_pages_and_head_dims(kv_bits, page, head_dim, compact):
    """The default page of 64, head_dim 128, and the INT8 pages that keep the reference's own sequence (8 and 128)."""
    _oracle_checked_run(kv_bits, page, head_dim, compact=compact, fused=not (kv_bits == 8 and page in (8, 128)))
