"""A refused factorization: the reported row, and the blocks it leaves.

Nothing that depends on a diagonal tile is formed from that tile's failing pivot or from
the ones after it: the tiles of its column and every tile behind them keep what they held.
So the row that is reported is the first failing one of its chain, whatever the timing, and
of finite blocks only finite ones are left (a solve with a non-positive pivot would leave
NaN).  The pivot made non-positive is the first, a middle and the last one of the first,
a middle and the last tile of a block.
"""
import numpy as np
import pytest

from oracle import bta_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("value", [-1.0, 0.0])
@pytest.mark.parametrize("method", [0, 1])
@pytest.mark.parametrize("twist", [True, False])
@pytest.mark.parametrize("b,block,rows", [(20, 1, (0, 19)), (97, 0, (0, 17, 31, 32, 63, 96)),
                                          (97, 2, (0, 31, 64, 95)), (160, 1, (30, 31, 80, 159))])
def test_nothing_behind_the_failing_pivot(b, block, rows, twist, method, value):
    import torch

    from pyinla_gb300.device import BtaHandle, current_stream_ptr
    nt, a = 5, 3
    D, L, R, T, _ = orc.make_bta_c1(b, nt=nt, b=b, a=a)
    h = BtaHandle(b, nt, a, twist)
    try:
        h.set_method(method)
        h.set_stream(current_stream_ptr())
        for row in rows:
            Q = [torch.from_numpy(x.copy()).cuda() for x in (D, L, R, T)]
            Q[0][block, row, row] = value
            for _ in range(5):
                W = [q.clone() for q in Q]
                assert h.lib.gbta_pobtaf(h.ptr, *[w.data_ptr() for w in W]) == block * b + row + 1
                assert all(bool(torch.isfinite(w).all()) for w in W)
    finally:
        h.close()


def test_batch_nothing_behind_the_failing_pivot():
    import torch

    from pyinla_gb300.batch import BtaBatch
    shapes = [(97, 4, 2), (64, 3, 1)]
    batch = BtaBatch(shapes)
    for row in (0, 31, 40, 96):
        for k, (b, nt, a) in enumerate(shapes):
            D, L, R, T, rhs = orc.make_bta_c1(k, nt=nt, b=b, a=a)
            if k == 0:
                D[0, row, row] = -1.0
            batch.load(k, D, L, R, T, rhs)
        with pytest.raises(np.linalg.LinAlgError, match=f"row {row + 1}\\)"):
            batch.run(1)
        for x in (batch.D, batch.L, batch.R, batch.T):
            assert all(bool(torch.isfinite(v).all()) for v in x)
