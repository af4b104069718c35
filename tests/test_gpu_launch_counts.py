"""`launches` of the decode engines against the kernel nodes of a graph captured from the same calls."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _kernel_nodes(fn):
    from cuda.bindings import driver as cu
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph, capture_error_mode="thread_local"):
        fn()
    raw = cu.CUgraph(graph.raw_cuda_graph())
    rc, _, n = cu.cuGraphGetNodes(raw)
    assert rc == cu.CUresult.CUDA_SUCCESS
    rc, nodes, n = cu.cuGraphGetNodes(raw, n)
    assert rc == cu.CUresult.CUDA_SUCCESS
    return sum(cu.cuGraphNodeGetType(x)[1] == cu.CUgraphNodeType.CU_GRAPH_NODE_TYPE_KERNEL for x in nodes[:n])


@pytest.mark.parametrize("bits", [3, 4, 8])
@pytest.mark.parametrize("Hq,seen", [(4, 3), (4, 15), (4, 40), (16, 40), (16, 47)])   # no page, the first, staged, two passes of scores, a page completed
def test_step_and_step_all(bits, Hq, seen):
    from flashquest_b200.cache.persistent_int4 import PersistentInt4KVCache
    from flashquest_b200.cache.persistent_int8 import PersistentInt8KVCache
    from flashquest_b200.cache.persistent_turbo import PersistentTurboKVCache
    from flashquest_b200.eager.decode_step import QuestDecodeInt4, QuestDecodeInt8, QuestDecodeTurbo
    Cache, Engine = {3: (PersistentTurboKVCache, QuestDecodeTurbo), 4: (PersistentInt4KVCache, QuestDecodeInt4), 8: (PersistentInt8KVCache, QuestDecodeInt8)}[bits]
    kv = lambda *s: torch.randn(*s, device="cuda", dtype=torch.float16)
    cache = Cache(batch_size=1, num_layers=2, num_kv_heads=2, head_dim=128, max_seq_len=128, page_size=16, device="cuda", dtype=torch.float16)
    for li in range(2):
        cache.update_quantized(kv(1, 2, seen, 128), kv(1, 2, seen, 128), li)
    eng = Engine(cache, num_q_heads=Hq, retention=0.5, num_sinks=1, window_pages=1, q_dtype=torch.float16)
    k, v, q = kv(2, 1, 2, 1, 128), kv(2, 1, 2, 1, 128), kv(2, 1, Hq, 1, 128)

    def both(fn):
        torch.cuda.synchronize()
        for times in range(2):                              # the first call outside a capture: it sets kernel attributes
            cache._seen_tokens[:] = [seen, seen]
            before = eng.launches
            nodes = _kernel_nodes(fn) if times else fn()
        assert nodes == eng.launches - before > 0

    both(lambda: [eng.step(k[0], v[0], q[0], 0)])
    if bits == 4:
        both(lambda: [eng.step_all(k, v, q)])
        cache.update_quantized(kv(1, 2, 2, 128), kv(1, 2, 2, 128), 1)                    # unequal lengths: layer by layer
        before = eng.launches
        eng.step_all(k, v, q)
        assert eng.launches - before >= 4


def test_llama_step():
    from flashquest_b200.eager.llama_decode import LlamaConfig, LlamaInt4Decoder, random_llama_weights
    cfg = LlamaConfig(hidden=256, layers=2, q_heads=4, kv_heads=2, head_dim=64, ffn=512, vocab=512)
    w = random_llama_weights(cfg, "cuda", seed=2)
    for B in (1, 3):                                        # three sequences: norms of their own
        dec = LlamaInt4Decoder(cfg, w, batch_size=B, max_seq_len=64, page_size=16, retention=0.5, num_sinks=1, window_pages=1)
        ids = torch.arange(B, dtype=torch.int32, device="cuda")
        for _ in range(18):
            dec.decode_step(ids)
        before = dec.launches
        nodes = _kernel_nodes(lambda: [dec.decode_step(ids)])
        extra = _kernel_nodes(lambda: [dec.w.embed[ids.long()] + 0])                       # the caller's gather, and one to capture
        assert nodes - (extra - 1) == dec.launches - before
