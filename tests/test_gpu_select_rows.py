"""The register selection kernel (csrc/fq_select.cu) at the edges of its rows per thread, with ties, infinities and clustered
scores, against an ordering by (score descending, page ascending)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B", [1, 32])
@pytest.mark.parametrize("P", [1, 33, 257, 1024, 2047, 4097, 8192, 8193])
@pytest.mark.parametrize("kind", ["normal", "ties", "inf", "clustered"])
def test_rows(B, P, kind):
    from flashquest_b200._lib import check, lib, ptr, stream_ptr
    H, sinks, window, r = 5, 2, 1, 0.2
    g = torch.Generator(device="cuda").manual_seed(P)
    x = torch.randn(B, H, P, device="cuda", generator=g)
    if kind == "ties":
        x = x.round()
    elif kind == "inf":
        x[..., ::7] = float("inf")
    elif kind == "clustered":
        x = torch.where(x > 2, x * 1e6, x * 1e-3)
    bucket = P + 4
    mask = torch.zeros(B, H, P, dtype=torch.uint8, device="cuda")
    comp = torch.zeros(B, H, bucket, dtype=torch.int32, device="cuda")
    cnt = torch.zeros(B, H, dtype=torch.int32, device="cuda")
    check(lib().fq_select_pages(ptr(x), *x.stride()[:2], B, H, P, None, r, P, sinks, window, ptr(mask), *mask.stride()[:2],
                                ptr(comp), *comp.stride()[:2], bucket, ptr(cnt), stream_ptr(x.device)))
    k = min(P, int(torch.ceil(torch.tensor(r, dtype=torch.float32) * P)))
    want = torch.zeros(B, H, P, dtype=torch.bool, device="cuda")
    want.scatter_(2, torch.sort(x, dim=2, descending=True, stable=True).indices[..., :k], True)
    want[..., :sinks] = True
    want[..., max(P - window, 0):] = True
    assert torch.equal(mask.bool(), want)
    assert torch.equal(cnt.long(), want.sum(2))
    ids = torch.where(want, torch.arange(P, device="cuda"), -1).sort(2, descending=True).values
    assert torch.equal(comp[..., :P].long(), ids) and (comp[..., P:] == -1).all()
