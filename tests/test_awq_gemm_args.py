"""fq_awq_gemm says what is wrong with its arguments before it chooses a kernel: at every number of rows, and without a GPU."""
import ctypes

import pytest

VP, I32 = ctypes.c_void_p * 1, ctypes.c_int * 1


@pytest.mark.parametrize("M", [9, 300, 100000])
@pytest.mark.parametrize("change,want", [(dict(scales=0), "null tensor"), (dict(qweight=0), "null tensor"), (dict(qzeros=0), "null tensor"),
                                         (dict(y=0), "null tensor"), (dict(N=0), "multiple of 128"), (dict(N=192), "multiple of 128"),
                                         (dict(N=-128), "multiple of 128"), (dict(y=4096 + 8), "aligned"), (dict(qzeros=4096 + 2), "aligned")])
def test_bad_arguments(M, change, want):
    from flashquest_b200._lib import lib
    a = dict(dict(qweight=4096, scales=4096, qzeros=4096, y=4096, N=256), **change)           # addresses: nothing is read
    arr = lambda name: VP(a[name] or None)
    rc = lib().fq_awq_gemm(ctypes.c_void_p(4096), M, 256, 128, 1, arr("qweight"), arr("scales"), arr("qzeros"), None, I32(a["N"]), arr("y"), 1, None)
    assert rc < 0 and want in lib().fq_last_error_string().decode()
