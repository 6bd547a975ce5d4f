"""The tile Cholesky over the exponent range of its pivots.

The pivots' reciprocals come from the integer pipe while d and 1/d are normal numbers and
from FP64 otherwise.  Scaling a matrix by 4^k scales its factor by 2^k exactly and leaves
every significand alone, so the factor of the scaled matrix is held against the oracle's
factor of the unscaled one: 1e-13 of the largest entry, a few hundred roundings.
"""
import numpy as np
import pytest

from oracle import bta_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("b", [1, 31, 32, 33, 65])
@pytest.mark.parametrize("k", [-470, -250, 0, 250, 505])
def test_factor_of_scaled_matrix(b, k):
    from pyinla_gb300 import algs
    D, L, R, T, _ = orc.make_bta_c1(7, nt=3, b=b, a=2)
    ref = [x.copy() for x in (D, L, R, T)]
    orc.pobtaf(*ref)
    got = [np.ldexp(x, 2 * k) for x in (D, L, R, T)]
    algs.pobtaf(*got)
    for g, r in zip(got, ref):
        assert np.abs(np.ldexp(g, -k) - r).max() <= 1e-13 * np.abs(r).max()


@pytest.mark.parametrize("value", [-1.0, 0.0, np.nan, np.inf])
@pytest.mark.parametrize("row", [0, 1, 30, 31, 32])
def test_bad_pivot_is_refused(row, value):
    """A non-positive or NaN pivot is reported at its row; an infinite one makes the next
    pivots NaN (rows after it)."""
    from pyinla_gb300 import algs
    D, L, R, T, _ = orc.make_bta_c1(7, nt=2, b=40, a=2)
    D[0, row, row] = value
    with pytest.raises(np.linalg.LinAlgError) as e:
        algs.pobtaf(D, L, R, T)
    if not np.isinf(value):
        assert f"row {row + 1})" in str(e.value)


@pytest.mark.parametrize("b", [20, 33, 64, 97])
def test_factor_again_after_failure_and_with_new_values(b):
    """The pivot words that the solves follow are emptied before every factorization: a
    handle gives each matrix its own factor, also right after a refused one."""
    from pyinla_gb300 import algs
    for seed in (1, 2, 3):
        D, L, R, T, _ = orc.make_bta_c1(seed, nt=4, b=b, a=3)
        bad = [x.copy() for x in (D, L, R, T)]
        bad[0][1, b // 2, b // 2] = -1.0
        with pytest.raises(np.linalg.LinAlgError):
            algs.pobtaf(*bad)
        ref = [x.copy() for x in (D, L, R, T)]
        orc.pobtaf(*ref)
        algs.pobtaf(D, L, R, T)
        for g, r in zip((D, L, R, T), ref):
            assert np.abs(g - r).max() <= 1e-12 * np.abs(r).max()
