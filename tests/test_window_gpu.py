"""Widths at which a merged bucket's targets only just pass the ring window, so
that a vertex can be pushed beyond it and, in the same phase, into it: the
window must never move back (distances were wrong in one of ten such runs)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wtype", ["u32", "f32"])
def test_window_edge(wtype, gb, orc):
    kws = ({}, {"flags": gb.F_NO_FUSE}, {"flags": gb.F_NO_SOLO}, {"full_items": 1},
           {"solo_entries": 1 << 30, "solo_descs": 1 << 30})
    for seed in (205, 208, 210):
        a = gb.gen_grid(47, 71, seed, wtype, 1, 1000)
        with gb.Graph.from_host(a) as g:
            for src in [int(x) for x in gb.sample_sources(a, 2, 5)]:
                ref = orc.dijkstra(a.row, a.col, a.w, src)
                pred = orc.min_tight_pred(a.row, a.col, a.w, src, ref)
                for delta in (17.0, 19.0, 20.0, 21.0):
                    for kw in kws:
                        for _ in range(6):
                            d, p, _ = g.sssp(src, delta=delta, **kw)
                            assert np.array_equal(d, ref) and np.array_equal(p, pred), (seed, src, delta, kw)
