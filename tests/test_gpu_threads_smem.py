"""Calls of several threads on a kernel whose shared memory depends on the call: the limit that a kernel may ask for belongs to
the function, so a call must not lower it between another thread's setting and its launch."""
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu


def test_selection_of_several_lengths_from_several_threads():
    from flashquest_b200._lib import lib, ptr
    select, rcs = lib().fq_select_pages, []

    def work(pages):
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            scores = torch.randn(1, 1, pages, device="cuda")
            compact = torch.empty(1, 1, 16, dtype=torch.int32, device="cuda")
        args = (ptr(scores), pages, pages, 1, 1, pages, None, 0.0, 4, 1, 1, None, 0, 0, ptr(compact), 16, 16, 16, None, stream.cuda_stream)
        rcs.append([rc for rc in (select(*args) for _ in range(5000)) if rc])
        stream.synchronize()

    threads = [threading.Thread(target=work, args=(p,)) for p in (48000, 12000, 25000, 9500)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert rcs == [[]] * 4, [len(r) for r in rcs]
