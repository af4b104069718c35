"""The fp16 head GEMV (csrc/fq_llama_ops.cu) at the edges of its row tiles, k steps and register slots."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 5, 8])
@pytest.mark.parametrize("K,N", [(32, 1), (288, 17), (2080, 5000), (3072, 16 * 148 * 4 + 3), (40, 33)])
def test_gemv_f16(M, K, N):
    from flashquest_b200._lib import check, lib, ptr, stream_ptr
    g = torch.Generator(device="cuda").manual_seed(M + K + N)
    x = torch.randn(M, K, device="cuda", generator=g).half()
    W = torch.randn(N, K, device="cuda", generator=g).half()
    y = torch.full((M, N), float("nan"), dtype=torch.float16, device="cuda")
    check(lib().fq_gemv_f16(ptr(x), ptr(W), M, K, N, ptr(y), stream_ptr(x.device)))
    want = x.double() @ W.double().T
    assert (y.double() - want).abs().max().item() <= 1e-3 * want.abs().max().item() + 1e-3
