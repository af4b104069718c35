"""Scratch of a TurboQuant step: what its kernels hand over, the 16-bit O of the pages in the rotated basis and its lse."""
import pytest


@pytest.mark.parametrize("B,Hq,D", [(1, 1, 64), (1, 24, 128), (3, 7, 64), (16, 32, 128)])
def test_holds_one_part(B, Hq, D):
    from flashquest_b200._lib import lib
    rows = B * Hq
    assert lib().fq_decode_layer_turbo_scratch_bytes(B, Hq, D) == -(-rows * D * 2 // 256) * 256 + rows * 4
    assert lib().fq_decode_layer_turbo_scratch_bytes(0, Hq, D) == 0
