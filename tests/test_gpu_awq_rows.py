"""The AWQ GEMM at the edges of its row tiles (csrc/fq_awq_skinny.cu, csrc/fq_awq_gemm.cu; the two give equal bits), and the GEMV
over its K splits and rows (csrc/fq_awq_gemv.cu), against a plain
PyTorch product of the fp16-rounded weights, and equal to itself over repeated launches."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _linear(K, N, group, interleaved, bias, g):
    from flashquest_b200.quant import AWQLinear
    ri = lambda *s: torch.randint(-2 ** 31, 2 ** 31 - 1, s, dtype=torch.int32, device="cuda", generator=g)
    sc = (torch.rand(K // group, N, device="cuda", generator=g) * 0.019 + 0.001).half()
    b = torch.randn(N, device="cuda", generator=g).half() if bias else None
    return AWQLinear(ri(K, N // 8), sc, ri(K // group, N // 8), b, group_size=group, interleaved=interleaved)


def _weights(lin):
    order = [0, 2, 4, 6, 1, 3, 5, 7] if lin.interleaved else list(range(8))

    def unpack(q):
        out = torch.empty(q.shape[0], q.shape[1] * 8, device=q.device)
        for i in range(8):
            out[:, order[i]::8] = ((q >> (4 * i)) & 15).float()
        return out
    rep = lambda t: t.repeat_interleave(lin.group_size, 0)
    return ((unpack(lin.qweight) - rep(unpack(lin.qzeros))) * rep(lin.scales.float())).half().float()


@pytest.mark.parametrize("M", [9, 16, 17, 33, 64, 65, 128, 129, 300])
@pytest.mark.parametrize("K,Ns,group,interleaved,bias", [(512, (128, 384), 128, True, False), (3072, (256, 128, 128), 128, True, True),
                                                         (1536, (256,), 256, False, True)])
def test_rows_and_splits(M, K, Ns, group, interleaved, bias):
    from flashquest_b200.kernel.fused_proj import awq_gemm_fused
    g = torch.Generator(device="cuda").manual_seed(M + K)
    lins = [_linear(K, N, group, interleaved, bias, g) for N in Ns]
    x = torch.randn(M, K, device="cuda", generator=g).half()
    got = awq_gemm_fused(x, lins)
    for y, lin in zip(got, lins):
        want = x.float() @ _weights(lin) + (lin.bias.float() if bias else 0)
        assert (y.float() - want).abs().max().item() <= 2e-3 * want.abs().max().item() + 1e-3
    for _ in range(5):
        assert all(torch.equal(a, b) for a, b in zip(got, awq_gemm_fused(x, lins)))


@pytest.mark.parametrize("K,N,group,interleaved,bias", [(512, 512, 128, True, False), (3072, 512, 128, True, True), (1536, 512, 256, False, True)])
def test_few_row_kernel_gives_the_bits_of_the_large_gemm(K, N, group, interleaved, bias):
    """A row's result does not depend on the kernel that the number of rows picks: the first rows of a product of 20 000 rows
    (256-row tiles) and of 14 336 (128-row tiles, above three waves of the few-row kernel's), alone."""
    from flashquest_b200.kernel.fused_proj import awq_gemm_fused
    g = torch.Generator(device="cuda").manual_seed(K)
    lin = _linear(K, N, group, interleaved, bias, g)
    x = torch.randn(20000, K, device="cuda", generator=g).half()
    (large,) = awq_gemm_fused(x, (lin,))
    assert torch.equal(awq_gemm_fused(x[:14336], (lin,))[0], large[:14336])
    for M in (9, 16, 17, 32, 33, 64, 65, 128, 129, 300, 1000, 14000):
        assert torch.equal(awq_gemm_fused(x[:M], (lin,))[0], large[:M]), M


@pytest.mark.parametrize("M", [129, 255, 256, 257, 385, 1025])
@pytest.mark.parametrize("K,Ns,group,interleaved,bias", [(64, (9600, 128), 64, True, True), (320, (9728,), 64, False, False), (256, (128, 9600, 384, 128), 256, True, False),
                                                         (1152, (19200,), 128, True, False)])
def test_pair_tiles(M, K, Ns, group, interleaved, bias):
    """Tiles of a CTA pair at their edges: rows that end in the first or the second CTA's half, projections that end in the first
    half of their last tile, 1 to 18 k blocks, one to five tiles per pair."""
    from flashquest_b200.kernel.fused_proj import awq_gemm_fused
    g = torch.Generator(device="cuda").manual_seed(M + K)
    lins = [_linear(K, N, group, interleaved, bias, g) for N in Ns]
    x = torch.randn(M, K, device="cuda", generator=g).half()
    got = awq_gemm_fused(x, lins)
    for y, lin in zip(got, lins):
        want = x.float() @ _weights(lin) + (lin.bias.float() if bias else 0)
        assert (y.float() - want).abs().max().item() <= 2e-3 * want.abs().max().item() + 1e-3
    assert all(torch.equal(a, b) for a, b in zip(got, awq_gemm_fused(x, lins)))


@pytest.mark.parametrize("M", [1, 100, 257, 1025])
@pytest.mark.parametrize("K,N,group,interleaved,bias", [(128, 9600, 64, True, True), (1152, 4992, 128, False, False), (256, 19200, 256, True, False)])
def test_gate_up_with_swiglu_equals_its_parts(M, K, N, group, interleaved, bias):
    """One launch (and, at few rows, two) gives the bits of the projections followed by fq_swiglu."""
    import ctypes
    from flashquest_b200._lib import check, lib, ptr, stream_ptr
    from flashquest_b200.kernel.fused_proj import awq_gemm_fused
    g = torch.Generator(device="cuda").manual_seed(M + K)
    lins = [_linear(K, N, group, interleaved, bias, g) for _ in range(2)]
    x = torch.randn(M, K, device="cuda", generator=g).half()
    gate, up = awq_gemm_fused(x, lins)
    want, got = torch.empty_like(gate), torch.empty_like(gate)
    check(lib().fq_swiglu(ptr(gate), ptr(up), gate.numel(), ptr(want), stream_ptr(x.device)))
    VP = ctypes.c_void_p * 2
    arr = lambda name: VP(*[ptr(getattr(lin, name)) for lin in lins])
    buf = [torch.empty_like(gate) for _ in range(2)]
    check(lib().fq_awq_gate_up_swiglu(ptr(x), M, K, group, arr("qweight"), arr("scales"), arr("qzeros"), arr("bias") if bias else None, N,
                                      ptr(buf[0]), ptr(buf[1]), ptr(got), int(interleaved), stream_ptr(x.device)))
    assert torch.equal(got.view(torch.int16), want.view(torch.int16))


@pytest.mark.parametrize("M", [1100, 2048])
def test_large_tiles_repeat(M):
    """More tiles than SMs: a CTA's second tile overlaps the epilogue of its first."""
    from flashquest_b200.kernel.fused_proj import awq_gemm_fused
    g = torch.Generator(device="cuda").manual_seed(M)
    lin = _linear(3072, 5120, 128, True, False, g)
    x = torch.randn(M, 3072, device="cuda", generator=g).half()
    (first,) = awq_gemm_fused(x, (lin,))
    want = x.float() @ _weights(lin)
    assert (first.float() - want).abs().max().item() <= 2e-3 * want.abs().max().item() + 1e-3
    for _ in range(30):
        assert torch.equal(first, awq_gemm_fused(x, (lin,))[0])


@pytest.mark.parametrize("M", [1, 3, 8])
@pytest.mark.parametrize("K,Ns,interleaved,bias", [(128, (128,), True, True), (1152, (384, 128), False, False), (8320, (256,), True, False),
                                                   (4096, (9600, 128), True, True)])
def test_gemv_splits_and_tiles(M, K, Ns, interleaved, bias):
    from flashquest_b200.kernel.fused_proj import awq_gemv_fused
    g = torch.Generator(device="cuda").manual_seed(M + K)
    lins = [_linear(K, N, 128, interleaved, bias, g) for N in Ns]
    x = torch.randn(M, K, device="cuda", generator=g).half()
    got = awq_gemv_fused(x, lins)
    for y, lin in zip(got, lins):
        want = x.float() @ _weights(lin) + (lin.bias.float() if bias else 0)
        assert (y.float() - want).abs().max().item() <= 2e-3 * want.abs().max().item() + 1e-3
    assert all(torch.equal(a, b) for a, b in zip(got, awq_gemv_fused(x, lins)))


@pytest.mark.parametrize("M", [1, 2, 3, 5, 8])
@pytest.mark.parametrize("K,Ns", [(128, (32,)), (1152, (384, 96)), (8192, (512,)), (3072, (9600, 1024))])
def test_gemv_of_known_layout_gives_the_bits_of_the_general_one(M, K, Ns):
    """Groups of 128 in AutoAWQ's order on 16-byte rows take loops that the compiler knows the sizes of; the same weights four
    bytes off take the general ones."""
    from flashquest_b200.kernel.fused_proj import awq_gemv_fused
    from flashquest_b200.quant import AWQLinear
    g = torch.Generator(device="cuda").manual_seed(M + K)
    lins = [_linear(K, N, 128, True, True, g) for N in Ns]

    def shifted(t):
        buf = torch.empty(t.numel() + 1, dtype=t.dtype, device="cuda")[1:].view_as(t)
        return buf.copy_(t)
    odd = [AWQLinear(shifted(lin.qweight), lin.scales, lin.qzeros, lin.bias, group_size=128, interleaved=True) for lin in lins]
    assert all(lin.qweight.data_ptr() % 16 == 4 for lin in odd)
    x, u = (torch.randn(M, K, device="cuda", generator=g).half() for _ in range(2))
    for kw in ({}, dict(swiglu_up=u), dict(add=u, norm_weight=u[0], return_sum=True)):
        for a, b in zip(awq_gemv_fused(x, lins, **kw), awq_gemv_fused(x, odd, **kw)):
            assert torch.equal(a.view(torch.int16), b.view(torch.int16))


@pytest.mark.parametrize("M", [1, 2, 4, 7, 8])
@pytest.mark.parametrize("K,N,group,interleaved,bias", [(128, 128, 128, True, True), (3072, 8192, 128, True, False), (1152, 352, 128, True, True),
                                                        (320, 264, 64, False, True), (1024, 1000, 32, True, False)])
def test_gemv_with_swiglu_behind_equals_its_parts(M, K, N, group, interleaved, bias):
    """Tiles of gate and up columns side by side give the bits of the two projections followed by fq_swiglu, with and without
    the norm in front, at every split."""
    import ctypes
    from flashquest_b200._lib import GEMV_ADD_RMSNORM, GemvPrologue, check, lib, ptr, stream_ptr
    from flashquest_b200.kernel.fused_proj import awq_gemv_fused
    g = torch.Generator(device="cuda").manual_seed(M + K)
    lins = [_linear(K, N, group, interleaved, bias, g) for _ in range(2)]
    x, b = (torch.randn(M, K, device="cuda", generator=g).half() for _ in range(2))
    w = torch.rand(K, device="cuda", generator=g).half()
    VP = ctypes.c_void_p * 2
    arr = lambda name: VP(*[ptr(getattr(lin, name)) for lin in lins])
    for k_split in (1, 2, 8, lib().fq_awq_gemv_default_splits(K, 2 * N, group)):
        for norm in (False, True):
            gate, up = awq_gemv_fused(x, lins, k_split=k_split, **(dict(add=b, norm_weight=w, return_sum=True) if norm else {}))[:2]
            want, got, total = torch.empty_like(gate), torch.empty_like(gate), torch.empty_like(x)
            check(lib().fq_swiglu(ptr(gate), ptr(up), gate.numel(), ptr(want), stream_ptr(x.device)))
            pro = GemvPrologue(GEMV_ADD_RMSNORM, ptr(b), ptr(w), 1e-5, ptr(total)) if norm else None
            check(lib().fq_awq_gemv_swiglu(ptr(x), M, K, group, arr("qweight"), arr("scales"), arr("qzeros"), arr("bias") if bias else None, N,
                                           ptr(got), int(interleaved), ctypes.byref(pro) if norm else None, k_split, stream_ptr(x.device)))
            assert torch.equal(got.view(torch.int16), want.view(torch.int16)), (k_split, norm)
            assert not norm or torch.equal(total, x + b)


@pytest.mark.parametrize("rows,H", [(1, 8), (3, 264), (8, 3072), (2, 8192)])
def test_norm_equals_general_kernel(rows, H):
    """Rows 16 bytes at a time give the bits of the value-by-value kernel, which unaligned rows take."""
    from flashquest_b200._lib import check, lib, ptr, stream_ptr
    g = torch.Generator(device="cuda").manual_seed(H)
    x, d = (torch.randn(rows, H, device="cuda", generator=g).half() for _ in range(2))
    w = torch.rand(H, device="cuda", generator=g).half()
    odd = torch.empty(rows * H + 1, dtype=torch.float16, device="cuda")[1:].view(rows, H)
    odd.copy_(x)
    out = []
    for a in (x, odd):
        normed, total = torch.empty_like(x), torch.empty_like(x)
        check(lib().fq_add_rmsnorm(ptr(a), ptr(d), ptr(w), 1e-5, rows, H, ptr(total), ptr(normed), stream_ptr(x.device)))
        out.append((normed, total))
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])
