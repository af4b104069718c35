"""The streaming page-score kernel (csrc/fq_scores.cu), which large batches take, against the same rows scored one at a time."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_rep,D,P", [(1, 128, 1200), (3, 128, 1199), (5, 64, 1201), (4, 128, 1202)])
def test_equals_short_kernel(n_rep, D, P):
    from flashquest_b200._lib import check, dtype_code, lib, ptr, stream_ptr
    B, Hkv = 16, 2
    g = torch.Generator(device="cuda").manual_seed(P)
    q = torch.randn(B, Hkv * n_rep, D, device="cuda", generator=g).half()
    ks, km = (torch.randn(B, Hkv, P, D, device="cuda", generator=g).bfloat16() for _ in range(2))

    def run(i0, n):
        sc = torch.full((n, Hkv * n_rep, P), float("nan"), device="cuda")
        qq, a, m = q[i0:i0 + n], ks[i0:i0 + n], km[i0:i0 + n]
        check(lib().fq_page_scores_int4(ptr(qq), dtype_code(qq), *qq.stride()[:2], ptr(a), ptr(m), *a.stride()[:3], n, Hkv * n_rep, Hkv, P, D,
                                        ptr(sc), *sc.stride()[:2], stream_ptr(q.device)))
        return sc
    assert torch.equal(run(0, B), torch.cat([run(i, 1) for i in range(B)]))
