"""Buckets merged over several base widths give the oracle's result, and a
uint32 graph whose path sums could pass 2^32 - 1 keeps one base width a bucket."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _uniform(n, deg, seed):
    """A random graph of about that degree with rows of at most 32 edges."""
    rng = np.random.default_rng(seed)
    u, v = rng.integers(0, n, n * deg // 2), rng.integers(0, n, n * deg // 2)
    key = np.unique(np.concatenate([u * n + v, v * n + u]))
    s, d = key // n, key % n
    row = np.zeros(n + 1, dtype=np.uint64)
    row[1:] = np.cumsum(np.bincount(s, minlength=n))
    w = (1 + (np.minimum(s, d) * 31 + np.maximum(s, d) * 17) % 255).astype(np.uint32)
    return row, d.astype(np.uint32), w


def _graph(gb, kind):
    if kind == "grid":
        a = gb.gen_grid(150, 161, 4, "f32")
        return a.row, a.col, a.w
    if kind == "uniform":
        return _uniform(20000, 6, 7)
    if kind == "rmat_f64":
        a = gb.gen_rmat(14, 16, 9)
        return a.row, a.col, a.w / 37.0
    a = gb.gen_rmat(15, 16, 5)
    return a.row, a.col, a.w * np.uint32(600 if kind == "rmat_heavy" else 1)


@pytest.mark.parametrize("kind,merges", [("grid", True), ("uniform", True), ("rmat", True), ("rmat_f64", True),
                                         ("rmat_heavy", False)])
def test_merged_buckets_same_result(kind, merges, gb, orc):
    row, col, w = _graph(gb, kind)
    srcs = [int(np.argmax(np.diff(row.astype(np.int64)))), 1]
    d0 = float(w.max()) / (len(col) / (len(row) - 1))
    with gb.Graph(row, col, w) as g:
        for src in srcs:
            ref = orc.dijkstra(row, col, w, src)
            pred = orc.min_tight_pred(row, col, w, src, ref)
            # the default width, one that sends most vertices past the window, and the split schedule
            for kw in ({}, {"delta": max(d0 / 24, 1.0) if w.dtype == np.uint32 else d0 / 24}, {"full_items": 1},
                       {"flags": gb.F_NO_SOLO}):
                kw = {**kw, "flags": kw.get("flags", 0) | gb.F_TRACE}
                d, p, _ = g.sssp(src, **kw)
                spans = {r["span"] for r in g.trace()}
                assert np.array_equal(d, ref) and np.array_equal(p, pred), kw
                if src == srcs[0]:
                    assert (max(spans) > 1) == merges, (kw, spans)
        if g.wtype != gb.W_F64:
            with gb.Plan(g, np.array(srcs, dtype=np.uint32), group_ctas=3) as plan:
                plan.run()
                dist, _ = plan.results()
            for i, src in enumerate(srcs):
                assert np.array_equal(dist[i], orc.dijkstra(row, col, w, src))


def _starts(trace):
    return [r for r in trace if r["kind"] == "scan_bucket"]


def test_merges_widen_with_the_distance_on_graphs_that_spread(gb, orc):
    """Until the run drains, bucket b of a graph with rows of more than four edges
    takes in b / 4 base buckets; a grid's takes in up to 16 from the start."""
    row, col, w = _uniform(20000, 6, 7)
    grid = gb.gen_grid(150, 161, 4, "u32")
    for r, c, x, ramp in ((row, col, w, True), (grid.row, grid.col, grid.w, False)):
        n, done, wide = len(r) - 1, 0, False
        with gb.Graph(r, c, x) as g:
            d, _, _ = g.sssp(1, flags=gb.F_TRACE)
            for rec in _starts(g.trace()):
                if done < n // 16:
                    wide |= rec["span"] > rec["bucket"] // 4 + 1
                done += rec["items"]
        assert wide != ramp
        assert np.array_equal(d, orc.dijkstra(r, c, x, 1))


@pytest.mark.parametrize("wtype", ["u32", "f32", "f64"])
def test_no_merge_splits_a_bucket(wtype, gb, orc):
    """Thin buckets merge up to full_items entries, which relax whole rows: only a
    drain (of at most four base buckets), and only where the first list alone
    holds more, merges buckets that are split."""
    a = gb.gen_grid(300, 320, 4, "f32" if wtype == "f32" else "u32")
    w = a.w / 3.0 if wtype == "f64" else a.w
    with gb.Graph(a.row, a.col, w) as g:
        d, _, _ = g.sssp(1, full_items=700, flags=gb.F_TRACE)
        starts = _starts(g.trace())
        assert all(r["full"] and r["items"] <= 700 for r in starts if r["span"] > 4)
        assert max(r["span"] for r in starts) > 4
        assert np.array_equal(d, orc.dijkstra(a.row, a.col, w, 1))
