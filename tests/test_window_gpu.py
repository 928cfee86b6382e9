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


def _dense(n, m, seed, wtype):
    rng = np.random.default_rng(seed)
    u, v = np.sort(rng.integers(0, n, m)), rng.integers(0, n, m).astype(np.uint32)
    row = np.zeros(n + 1, dtype=np.uint64)
    row[1:] = np.cumsum(np.bincount(u, minlength=n))
    w = rng.integers(0, 2000, m)
    return row, v, (w / 7.0).astype(np.float32 if wtype == "f32" else np.float64) if wtype != "u32" else w.astype(np.uint32)


@pytest.mark.parametrize("wtype", ["u32", "f32", "f64"])
@pytest.mark.parametrize("n,m", [(5, 40), (70, 900), (900, 9000)])
def test_each_vertex_once_a_bucket(n, m, wtype, gb, orc):
    """Vertices whose distance drops through many buckets, from beyond the window
    into it and inside it: a list holds a vertex of a bucket once, by the bucket
    of its old distance, and no list overflows or loses one."""
    for seed in (1, 2, 3):
        row, col, w = _dense(n, m, seed, wtype)
        with gb.Graph(row, col, w) as g:
            ref = orc.dijkstra(row, col, w, 0)
            pred = orc.min_tight_pred(row, col, w, 0, ref)
            for delta in (1.0, 3.0, 11.0, 40.0):
                for kw in ({}, {"flags": gb.F_NO_SOLO}, {"flags": gb.F_NO_SOLO | gb.F_NO_FUSE}, {"full_items": 1},
                           {"solo_entries": 1 << 30, "solo_descs": 1 << 30, "inline_edges": 1}):
                    d, p, _ = g.sssp(0, delta=delta, **kw)
                    assert np.array_equal(d, ref) and np.array_equal(p, pred), (seed, delta, kw)


@pytest.mark.parametrize("wtype", ["u32", "f32"])
def test_window_edge_in_plans(wtype, gb, orc):
    """Merged buckets and the pending list in plans, whose groups share a launch."""
    graphs = [gb.gen_grid(47, 71, 205, wtype, 1, 1000), gb.gen_grid(60, 90, 208, wtype, 1, 1000), gb.gen_rmat(11, 8, 5, wtype),
              gb.gen_grid(1, 700, 210, wtype, 1, 1000)]
    src = np.array([h.n // 3 for h in graphs], dtype=np.uint32)
    refs = [orc.dijkstra(h.row, h.col, h.w, int(s)) for h, s in zip(graphs, src)]
    with gb.Pack(graphs) as pk:
        for delta in (1.0, 17.0, 20.0, 21.0):
            for kw in ({"group_ctas": 1}, {"group_ctas": 3}, {"group_ctas": 38, "flags": gb.F_NO_SOLO}, {"light": delta / 2}):
                with gb.Plan(pk, src, delta=delta, **kw) as plan:
                    for _ in range(3):
                        plan.run()
                        dist, pred = plan.results()
                        for h, s, r, d, p in zip(graphs, src, refs, dist, pred):
                            assert np.array_equal(d, r), (delta, kw)
                            assert np.array_equal(p, orc.min_tight_pred(h.row, h.col, h.w, int(s), r)), (delta, kw)
