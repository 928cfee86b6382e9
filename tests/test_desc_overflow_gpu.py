"""Graphs on which fusion scans long rows again and again (average degree above
the inline limit, weights so skewed that one bucket holds most of a run): the
descriptors of a scan do not fit their list, and the rows that found no room
wait for the next scan."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DT = {"f32": np.float32, "f64": np.float64}


def _skewed(n, m, seed, wtype):
    rng = np.random.default_rng(seed)
    u, v = np.sort(rng.integers(0, n, m)), rng.integers(0, n, m)
    row = np.zeros(n + 1, dtype=np.uint64)
    row[1:] = np.cumsum(np.bincount(u, minlength=n))
    w = rng.lognormal(0, 2, m)
    return row, v.astype(np.uint32), (1 + w * 100).astype(np.uint32) if wtype == "u32" else w.astype(DT[wtype])


@pytest.mark.parametrize("wtype", ["u32", "f32", "f64"])
@pytest.mark.parametrize("n,m", [(4096, 160000), (32768, 1 << 20)])
def test_more_descriptors_than_room(n, m, wtype, gb, orc):
    row, col, w = _skewed(n, m, 1, wtype)
    with gb.Graph(row, col, w) as g:
        for src in (0, n // 3):
            ref = orc.dijkstra(row, col, w, src)
            pred = orc.min_tight_pred(row, col, w, src, ref)
            for kw in ({"solo_entries": 1024}, {"fuse_rounds": 8}, {"solo_entries": 1 << 30, "solo_descs": 1 << 30},
                       {"inline_edges": 1}):
                for _ in range(3):
                    d, p, _ = g.sssp(src, **kw)
                    assert np.array_equal(d, ref) and np.array_equal(p, pred), (src, kw)


@pytest.mark.parametrize("wtype", ["u32", "f32"])
def test_more_descriptors_than_room_in_plans(wtype, gb, orc):
    n = 40000
    row, col, w = _skewed(n, 1 << 20, 2, wtype)
    src = np.arange(5, dtype=np.uint32) * 77
    with gb.Graph(row, col, w) as g, gb.Plan(g, src, fuse_rounds=8) as plan:
        for _ in range(3):
            plan.run()
            dist, pred = plan.results()
        for i, s in enumerate(src):
            ref = orc.dijkstra(row, col, w, int(s))
            assert np.array_equal(dist[i], ref)
            assert np.array_equal(pred[i], orc.min_tight_pred(row, col, w, int(s), ref))
