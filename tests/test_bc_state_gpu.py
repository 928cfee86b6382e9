"""Betweenness of a source does not depend on what earlier sources left in its
arrays.  Float weights that a sum absorbs (1e8 + 1 = 1e8) make the edges of a
pair tight in both directions: the pair and what only it leads to join no
level, and their in-degrees are not counted down."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _absorbing(wtype, far):
    """0 reaches the pair 1, 2 over `far`; 5 reaches it over short edges."""
    e = [(0, 1, far), (0, 2, far), (0, 6, 1.0), (6, 1, far), (1, 2, 1.0), (2, 1, 1.0), (1, 3, 64.0), (2, 3, 64.0),
         (3, 4, 64.0), (5, 1, 1.0), (5, 2, 3.0), (5, 6, 2.0), (6, 7, 1.0)]
    e.sort()
    row = np.zeros(9, dtype=np.uint64)
    for u, _, _ in e:
        row[u + 1] += 1
    return (np.cumsum(row).astype(np.uint64), np.array([v for _, v, _ in e], dtype=np.uint32),
            np.array([w for _, _, w in e], dtype=wtype))


@pytest.mark.parametrize("wtype,far", [(np.float32, 1e8), (np.float64, 1e17)])
@pytest.mark.parametrize("single", [False, True])
def test_bc_after_cycles_of_tight_edges(wtype, far, single, gb, orc):
    row, col, w = _absorbing(wtype, far)
    kw = {"flags": gb.F_BC_SINGLE} if single else {}
    with gb.Graph(row, col, w) as g:
        alone, _ = g.betweenness([5], **kw)
    assert np.array_equal(alone, orc.betweenness(row, col, w, [5]))      # no cycle of tight edges from here
    with gb.Graph(row, col, w) as g:
        cyc, _ = g.betweenness([0], **kw)                                # leaves in-degrees of the pair
        assert np.array_equal(g.betweenness([5], **kw)[0], alone)
        assert np.array_equal(g.betweenness([0], **kw)[0], cyc)
        for srcs in ([0, 5], [5, 0], [0, 0, 5], [5, 5, 0]):
            want = np.zeros(8)
            for s in srcs:
                want = want + (alone if s == 5 else cyc)
            assert np.array_equal(g.betweenness(srcs, **kw)[0], want), srcs


@pytest.mark.parametrize("scale", [None, 17])
def test_bc_of_more_sources_than_groups(scale, gb, orc):
    """64 sources of one batched launch whose arrays do not fit in L2 together:
    their passes take several launches, the last of fewer groups."""
    a = gb.gen_grid(265, 266, 3, "u32", 1, 4) if scale is None else gb.gen_rmat(scale, 2, 3, "u32", 1, 3)
    assert a.n > 66000
    srcs = [int(s) for s in gb.sample_sources(a, 65 if scale is None else 40, 7)]
    with gb.Graph.from_host(a) as g:
        bc, st = g.betweenness(srcs)
        again, _ = g.betweenness(srcs[:3])
    assert st["sources"] == len(srcs)
    assert np.array_equal(bc, orc.betweenness(a.row, a.col, a.w, srcs))
    assert np.array_equal(again, orc.betweenness(a.row, a.col, a.w, srcs[:3]))
