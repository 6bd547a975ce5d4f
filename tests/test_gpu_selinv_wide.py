"""Selected inversion of blocks above 4096 rows: a task's product loop then has more steps than
one round of descriptors (256) and goes on from the tile it left.

The columns of the selected inverse on the pattern are held against solves with unit vectors
(the sweeps): both carry a few thousand roundings of 1.1e-16 on a matrix whose condition is
below 10, so 1e-11 of the largest entry.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("b", [4096, 4130])
def test_columns_match_solves(b):
    import torch

    from pyinla_gb300 import algs
    from pyinla_gb300.synthetic import random_bta
    nt = 2
    D, L, _, _ = random_bta(nt, b, 0, seed=3)
    algs.pobtf(D, L)
    ks = [0, b - 1, b, 2 * b - 1]
    rhs = torch.zeros((nt * b, len(ks)), dtype=torch.float64, device="cuda")
    for q, k in enumerate(ks):
        rhs[k, q] = 1.0
    algs.pobts(D, L, rhs, trans="N")
    algs.pobts(D, L, rhs, trans="C")
    algs.pobtsi(D, L)
    for q, k in enumerate(ks):
        x = rhs[:, q]
        i, c = k // b, k % b
        tol = 1e-11 * float(x.abs().max())
        assert float((D[i][:, c] - x[i * b:(i + 1) * b]).abs().max()) <= tol
        if i == 0:
            assert float((L[0][:, c] - x[b:]).abs().max()) <= tol
        else:
            assert float((L[0][c, :] - x[:b]).abs().max()) <= tol
    assert np.isfinite(float(D.abs().max()))
