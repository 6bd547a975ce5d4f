"""The status of work queued before a change of stream.

A program may queue on the default stream, give the solver another stream and ask for the
status there: it is the queued work's, not what the control block held while that work still
ran.  The tip's pivot fails, the last of the factorization, and the default stream is held
for ~10 ms first (a bounded spin kernel), so that an early look sees nothing.
"""
import pytest

from oracle import bta_oracle as orc

pytestmark = pytest.mark.gpu


def test_failure_queued_on_the_default_stream():
    import torch

    from pyinla_gb300 import _lib
    from pyinla_gb300.device import BtaHandle
    b, nt, a = 64, 8, 2
    D, L, R, T, _ = orc.make_bta_c1(5, nt=nt, b=b, a=a)
    T[1, 1] = -1.0
    Q = [torch.from_numpy(x).cuda() for x in (D, L, R, T)]
    side = torch.cuda.Stream()
    h = BtaHandle(b, nt, a)
    try:
        for _ in range(3):
            W = [q.clone() for q in Q]
            torch.cuda.synchronize()
            h.set_stream(0)
            torch.cuda._sleep(20_000_000)
            assert h.lib.gbta_pobtaf_async(h.ptr, *[w.data_ptr() for w in W]) == 0
            h.set_stream(side.cuda_stream)
            assert h.lib.gbta_status(h.ptr) == nt * b + 2, _lib.last_error()
            assert h.lib.gbta_status(h.ptr) == 0     # (reported once)
    finally:
        torch.cuda.synchronize()
        h.close()
