"""Sweeps of several columns on wide blocks: one CTA per SM up to wider blocks than one column.

A second CTA per SM, which one column is faster with from 1280 rows on, costs two to four
columns up to 27 % there.  The results do not depend on the number of CTAs, so the default
equals launches pinned to one and to two per SM bit for bit on both sides of the lines, and a
column of several equals the same column alone; and where one per SM stays the default is not
slower than it (medians of calls in turn; 1.1 leaves room for noise, two per SM take 1.2 and
more).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _setup(b, nt, nrhs, twist=True):
    import torch

    from pyinla_gb300.device import BtaHandle, current_stream_ptr
    from pyinla_gb300.synthetic import random_bta
    Q = random_bta(nt, b, 3, seed=b)
    h = BtaHandle(b, nt, 3, twist)
    h.set_stream(current_stream_ptr())
    p = [q.data_ptr() for q in Q]
    assert h.lib.gbta_pobtaf(h.ptr, *p) == 0
    x = torch.randn((nt * b + 3, nrhs), dtype=torch.float64, device="cuda",
                    generator=torch.Generator("cuda").manual_seed(1))
    return h, Q, p, x


@pytest.mark.parametrize("b,nt,twist", [(1280, 4, True), (2016, 3, True), (2017, 3, True), (2208, 3, True),
                                        (2209, 3, True), (2656, 4, True), (2657, 4, True), (3488, 2, False),
                                        (3489, 2, False)])
@pytest.mark.parametrize("nrhs", [2, 5])
def test_any_number_of_ctas(b, nt, twist, nrhs):
    import torch
    h, Q, p, x0 = _setup(b, nt, nrhs, twist)
    try:
        for trans in (0, 1, 2):
            out = []
            for ctas in (0, 1, 2):
                h.set_ctas_per_sm(ctas)
                x = x0.clone()
                assert h.lib.gbta_pobtas(h.ptr, *p, x.data_ptr(), nrhs, trans) == 0
                out.append(x)
            assert torch.equal(out[0], out[1]) and torch.equal(out[0], out[2])
            one = x0[:, nrhs - 1].contiguous()
            assert h.lib.gbta_pobtas(h.ptr, *p, one.data_ptr(), 1, trans) == 0
            assert torch.equal(out[0][:, nrhs - 1], one)
    finally:
        h.close()


@pytest.mark.parametrize("nrhs", [2, 4])
def test_default_is_not_slower_than_one(nrhs):
    import torch
    h, Q, p, x0 = _setup(1280, 12, nrhs)
    try:
        ms = {0: [], 1: []}
        for _ in range(12):
            for ctas in ms:
                h.set_ctas_per_sm(ctas)
                x = x0.clone()
                e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                e0.record()
                assert h.lib.gbta_pobtas_async(h.ptr, *p, x.data_ptr(), nrhs, 2) == 0
                e1.record()
                assert h.lib.gbta_status(h.ptr) == 0
                ms[ctas].append(e0.elapsed_time(e1))
        assert np.median(ms[0]) <= 1.1 * np.median(ms[1]), ms
    finally:
        h.close()
