"""CPU replay of the tile Cholesky's update schedule (csrc/bta_common.cuh, potrf_schedule).

The pivot warp of smem_potrf keeps every pivot's multipliers w in a 32 x 32 scratch (Wt), and
the update warps apply them by a compile-time schedule: at step j everything so far to the
look-ahead slot (column j + 2), then up to POTRF_BUDGET more pivots a warp, the slots needed
first coming first.  The schedule is restated here from the constants and slot maps of the
source; the tests hold its invariants and replay the order of operations, lane by lane, against
numpy's Cholesky, with the garbage that the kernel leaves above the diagonal.
"""
import re

import numpy as np
import pytest

from tests.test_tile_schedules import FULL, SLOTS, SRC, TS, _const, column_owner, slot_col, slot_last, slot_owner

BUDGET = _const("POTRF_BUDGET")


def schedule():
    done = np.zeros((TS - 2, SLOTS), dtype=int)
    for j in range(TS - 2):
        done[j] = done[j - 1] if j else 0
        for w in range(3):
            left = BUDGET
            for s in range(SLOTS):
                if slot_owner(s) != w or slot_last(s) < j + 2:
                    continue
                while done[j, s] <= j and (slot_col(s) <= j + 2 or left > 0):
                    done[j, s] += 1
                    left -= 1
    return done


def test_schedule_restates_the_kernel():
    body = re.sub(r"\s+", " ", SRC[SRC.index("constexpr PotrfSchedule potrf_schedule()"):])
    body = body[:body.index("return t;")]
    for line in ("for (int j = 0; j < TS - 2; ++j)", "t.done[j][s] = j ? t.done[j - 1][s] : 0;",
                 "int left = POTRF_BUDGET;", "if (potrf_slot_owner(s) != w || potrf_slot_last(s) < j + 2) continue;",
                 "while (t.done[j][s] <= j && (potrf_slot_col(s) <= j + 2 || left > 0)) { ++t.done[j][s]; --left; }"):
        assert line in body, line


def test_columns_are_complete_when_handed_over():
    """No step uses a pivot that is not published yet; the slot of column j + 2 has pivots 0 .. j
    when step j hands that column to the pivot warp; a slot's pivots only grow."""
    done = schedule()
    for j in range(TS - 2):
        assert (done[j] <= j + 1).all()
        handed = [s for s in range(SLOTS) if slot_col(s) <= j + 2 <= slot_last(s)]
        assert len(handed) == 1 and done[j, handed[0]] == j + 1
    assert (np.diff(done, axis=0) >= 0).all()


def test_barrier_ids_are_free_when_they_come_round():
    """Look-ahead column p is consumed (ids rotate over four) before the pivot that column p + 4
    needs can be published, and of seven consecutive columns each update warp hands one over, so
    each has passed pivot p when pivot p + 8 takes its id."""
    for p in range(TS - 2 - 8):
        assert {column_owner(c) for c in range(p + 2, p + 9)} == {0, 1, 2}
    assert "POTRF_BAR_L + (k & 7)" in SRC and "POTRF_BAR_C + ((k - 1) & 3)" in SRC


@pytest.mark.parametrize("seed", [0, 1, 2])
def test_replay_is_cholesky(seed):
    rng = np.random.default_rng(seed)
    M = rng.standard_normal((TS, TS))
    A = M @ M.T + TS * np.eye(TS)
    S = A.copy()
    done = schedule()
    lanes = np.arange(TS)
    prow, half = 16 + (lanes & 15), lanes >> 4
    acc = [S[lanes, slot_col(s)].copy() if s < FULL else S[prow, slot_col(s) + half].copy() for s in range(SLOTS)]
    Wt = np.full((TS, TS), np.nan)

    def update_warps(j):
        for w in range(3):
            for s in range(SLOTS):
                if slot_owner(s) != w or slot_last(s) < j + 2:
                    continue
                for p in range(done[j - 1, s] if j else 0, done[j, s]):
                    if s < FULL:
                        acc[s] -= Wt[p, lanes] * S[slot_col(s), p]
                    else:
                        acc[s] -= Wt[p, prow] * S[slot_col(s) + half, p]
                if slot_col(s) == j + 2 or slot_last(s) == j + 2:
                    if s < FULL:
                        S[lanes, slot_col(s)] = acc[s]
                    else:
                        m = slot_col(s) + half == j + 2
                        S[prow[m], j + 2] = acc[s][m]

    a, an = S[:, 0].copy(), S[:, 1].copy()
    d = np.zeros(TS)
    for k in range(TS):
        d[k], ub = a[k], a[(k + 1) % TS]
        if 1 <= k < TS - 1:
            an = S[:, k + 1].copy()
        S[:, k] = a
        w = a / d[k]
        a = an - w * ub
        if k < TS - 2:
            Wt[k] = w
            update_warps(k)
    L = np.tril(S / np.sqrt(d)[None, :])
    np.testing.assert_allclose(L, np.linalg.cholesky(A), rtol=0, atol=1e-12 * np.abs(A).max())
