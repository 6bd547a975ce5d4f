"""Tile Cholesky with pivots at the ends of the exponent range.

A block s (tridiag(1/4, 1, 1/4) 2^e) with even e has 2^(e/2) times the factor of the unscaled
block, and both are exact powers apart, so the factor is held against numpy's of the unscaled
block.  From 2^1022 on a pivot's reciprocal is subnormal and has at least 50 bits; it enters
the updates only, by a quarter or less of a pivot: 1e-13 of the largest entry is some hundred
times the rounding of such a factor.  (From one tile to the next the digit products take the
low end to about 2^-989 only.)  A subnormal pivot has no reciprocal: the pivots after it in its
tile are NaN and the matrix is refused at the next row.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _block(b):
    return np.eye(b) + 0.25 * (np.eye(b, k=1) + np.eye(b, k=-1))


@pytest.mark.parametrize("b,e", [(b, e) for b in (2, 3, 32, 33) for e in (-1010, 1018, 1020, 1022) if b < 33 or e > 0])
@pytest.mark.parametrize("s", [1.0, 1.0 + 2.0 ** -52, 1.25, 2.0 - 2.0 ** -52, 2.0, 3.75])
def test_factor_at_both_ends(b, e, s):
    from pyinla_gb300 import algs
    D = (s * _block(b))[None]
    ref = np.linalg.cholesky(D[0])
    got = np.ldexp(D, e)
    algs.pobtf(got, np.zeros((0, b, b)))
    assert np.abs(np.ldexp(got[0], -e // 2) - ref).max() <= 1e-13 * np.abs(ref).max()


@pytest.mark.parametrize("row", [0, 1, 17, 30])
def test_subnormal_pivot_is_refused_at_the_next_row(row):
    from pyinla_gb300 import algs
    b = 40
    D = _block(b)[None]
    D[0, row, :] = D[0, :, row] = 0.0
    D[0, row, row] = np.ldexp(1.0, -1030)
    with pytest.raises(np.linalg.LinAlgError, match=f"row {row + 2}\\)"):
        algs.pobtf(D, np.zeros((0, b, b)))
