"""CPU check of unsynchronised shared-memory accesses in the tile kernels.

The selected inversion's diagonal task mirrors the lower triangle of its tile into the upper
one in place: each thread loads its elements, then stores the mirror images of those below the
diagonal, with no barrier between.  The test reads both conditions from the CUDA source, gives
every thread of the CTA its elements, and checks that no element is loaded by one thread and
stored by another, and that the stores complete the symmetric tile.
"""
import re

from tests.conftest import REPO

CSRC = REPO / "pyinla_gb300" / "csrc"
TS, NT = 32, 128


def _elements():
    """(thread, row, column) of the product loops' accumulator layout, from the source."""
    src = (CSRC / "bta_ozaki.cuh").read_text()
    row = re.search(r"int oz_row\(int nt_, int j\) \{.*?return (.*?);", src, re.S).group(1)
    col = re.search(r"int oz_col\(int nt_, int j\) \{.*?return (.*?);", src, re.S).group(1)
    out = []
    for t in range(NT):
        for nt_ in range(2):
            for j in range(4):
                names = dict(lane=t & 31, w=t >> 5, nt_=nt_, j=j)
                out.append((t, eval(row, names), eval(col, names)))
    assert sorted(e[1:] for e in out) == [(r, c) for r in range(TS) for c in range(TS)]
    return out


def test_symmetrisation_loads_no_element_that_another_thread_stores():
    src = (CSRC / "bta_selinv_task.cuh").read_text()
    load = re.search(r"sv\[n\]\[q\] = type != ST_DIAG \|\| (r >= cc) \? X\[r \* LDS \+ cc\] : 0\.0;", src)
    store = re.search(r"if \((r > cc)\) X\[cc \* LDS \+ r\] = sv\[n\]\[q\];", src)
    assert load and store and "__syncthreads" not in src[load.end():src.index("if (type == ST_OFF)", load.end())]
    elements = _elements()
    loads = {(r, c): t for t, r, c in elements if eval(load.group(1), dict(r=r, cc=c))}
    stores = {(c, r): t for t, r, c in elements if eval(store.group(1), dict(r=r, cc=c))}
    assert all(loads.get(e, t) == t for e, t in stores.items())
    assert set(loads) | set(stores) == {(r, c) for r in range(TS) for c in range(TS)}
    # a stored value is one that its thread loaded
    assert all(loads.get((c, r)) == t for (r, c), t in stores.items())
