"""Narrow blocks: the factorization and the selected inversion run fewer CTAs per SM below a
block width (two chains: 14 tiles for the factorization, 11 and 15 for the inversion on 152
SMs; one chain: 20, 15 and 21), later with banded couplings, whose live tiles the kernels
count themselves.

The results do not depend on the number of CTAs (every sum has a fixed order), so on both
sides of each line the default is equal, bit for bit, to a launch pinned to two per SM; both
are held against the oracle at the suite's 1e-10.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("twist", [True, False])
@pytest.mark.parametrize("b,banded", [(b, False) for b in (20, 352, 353, 448, 449, 480, 481, 640, 673)] +
                         [(b, True) for b in (448, 481, 576, 609, 640, 704)])
def test_any_number_of_ctas(b, banded, twist):
    import torch

    from oracle import bta_oracle as oracle
    from pyinla_gb300.device import BtaHandle, current_stream_ptr
    from pyinla_gb300.synthetic import random_bta
    nt, a = 4, 3
    Q = random_bta(nt, b, a, seed=b)
    if banded:
        Q = [q.clone() for q in Q]
        Q[1].copy_(torch.tril(torch.triu(Q[1], -20), 20))
    h = BtaHandle.get(b, nt, a, True)
    h.set_stream(current_stream_ptr())
    h.set_selinv_overlap(False)
    out = {}
    h.lib.gbta_set_twist(h.ptr, int(twist))
    try:
        for ctas in (0, 2):
            h.set_ctas_per_sm(ctas)
            W = [q.clone() for q in Q]
            p = [w.data_ptr() for w in W]
            assert h.lib.gbta_pobtaf(h.ptr, *p) == 0
            F = [w.clone() for w in W]
            assert h.lib.gbta_pobtasi(h.ptr, *p) == 0
            out[ctas] = F + W
    finally:
        h.set_ctas_per_sm(0)
        h.lib.gbta_set_twist(h.ptr, 1)
    for x, y in zip(out[0], out[2]):
        assert torch.equal(x, y)
    R = [q.cpu().numpy().copy() for q in Q]
    oracle.pobtaf(*R)
    oracle.pobtasi(*R)
    for x, y in zip(out[0][4:], R):
        assert np.abs(x.cpu().numpy() - y).max() <= 1e-10 * np.abs(y).max()
