"""Small graphs, solved by one CTA with their state in shared memory (a call
with every knob of the schedule at its default): distances and predecessors
are the oracle's, through every kind of output and in plans, and the calls
that do not qualify agree with them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _csr(n, edges, dtype):
    """edges: (u, v, w) triples."""
    e = sorted(edges)
    row = np.zeros(n + 1, dtype=np.uint64)
    for u, _, _ in e:
        row[u + 1] += 1
    return (np.cumsum(row).astype(np.uint64), np.array([v for _, v, _ in e], dtype=np.uint32),
            np.array([w for _, _, w in e], dtype=dtype))


def _star(n, hub_deg, dtype):
    """A hub of hub_deg edges (piece boundaries), chained leaves, one unreached tail."""
    edges = [(0, 1 + i % (n - 3), 5 + i % 7) for i in range(hub_deg)]
    edges += [(i, i + 1, 1 + i % 3) for i in range(1, n - 3)] + [(n - 2, n - 1, 4)]
    return _csr(n, edges, dtype)


def _graphs(gb):
    yield "one", _csr(1, [], np.uint32)
    yield "no edges", _csr(5, [], np.float32)
    yield "loops and zeros", _csr(4, [(0, 0, 0), (0, 1, 0), (1, 0, 0), (1, 1, 0), (1, 2, 3), (0, 2, 3), (2, 3, 0)], np.uint32)
    yield "infinite sums", _csr(4, [(0, 1, 3e38), (1, 2, 3e38), (2, 3, 1.0), (0, 3, 3.2e38)], np.float32)
    for n in (31, 32, 33, 1025):
        for d in (127, 128, 129, 256, 257):
            yield f"star {n} {d}", _star(n, d, np.uint32 if d % 2 else np.float32)
    for a in (gb.gen_rmat(10, 16, 3), gb.gen_rmat(13, 16, 4, "f32"), gb.gen_rmat(14, 4, 5), gb.gen_grid(33, 31, 2),
              gb.gen_grid(128, 128, 3), gb.gen_grid(1, 900, 4, "u32")):
        yield f"{a.n} {a.m}", (a.row, a.col, a.w)


def test_small_graphs_match_oracle(gb, orc):
    for name, (row, col, w) in _graphs(gb):
        n = len(row) - 1
        with gb.Graph(row, col, w) as g:
            for src in {0, n // 2, n - 1}:
                ref = orc.dijkstra(row, col, w, src)
                pred = orc.min_tight_pred(row, col, w, src, ref)
                d, p, st = g.sssp(src)
                assert np.array_equal(d, ref) and np.array_equal(p, pred), (name, src)
                assert st["blocks"] == 1, name
                d2, p2, s2 = g.sssp(src, solo_entries=512)   # a knob set: the persistent kernel
                assert s2["blocks"] > 1 and np.array_equal(d2, ref) and np.array_equal(p2, pred), (name, src)
                assert (st["reached"], st["edges_reached"]) == (s2["reached"], s2["edges_reached"]), (name, src)


@pytest.mark.parametrize("n,wmax,one", [(16384, 1, True), (16385, 1, False), (8192, 524287, True), (8192, 524288, False)])
def test_small_limits(n, wmax, one, gb, orc):
    """The vertex limit, and uint32 sums: n x the largest weight below 2^32 - 1."""
    edges = [(i, (i * 7 + 1) % n, wmax if i % 5 == 0 else 1) for i in range(n)]
    row, col, w = _csr(n, edges, np.uint32)
    with gb.Graph(row, col, w) as g:
        d, p, st = g.sssp(3)
    ref = orc.dijkstra(row, col, w, 3)
    assert (st["blocks"] == 1) == one
    assert np.array_equal(d, ref) and np.array_equal(p, orc.min_tight_pred(row, col, w, 3, ref))


def test_small_outputs(gb, orc):
    torch = pytest.importorskip("torch")
    a = gb.gen_rmat(9, 16, 8)
    ref = orc.dijkstra(a.row, a.col, a.w, 5)
    pred = orc.min_tight_pred(a.row, a.col, a.w, 5, ref)
    with gb.Graph.from_host(a) as g:
        dd, pd = (torch.empty(a.n, dtype=torch.int32, device="cuda") for _ in range(2))
        g.sssp_device(5, dd.data_ptr(), None)
        g.sssp_device(5, None, pd.data_ptr(), flags=gb.F_NO_STATS)
        assert np.array_equal(dd.cpu().numpy().view(np.uint32), ref) and np.array_equal(pd.cpu().numpy(), pred)
        hd, hp = gb.PinnedBuffer(a.n, np.uint32), np.empty(a.n, np.int32)
        g.sssp(5, out_dist=hd.array, out_pred=hp)
        assert np.array_equal(hd.array, ref) and np.array_equal(hp, pred)
        d, p, _ = g.sssp(5, want_pred=False)
        assert np.array_equal(d, ref) and p is None
        b1, _ = g.betweenness([5, 6, 7])                              # reads the workspace's state words
        b2, _ = g.betweenness([5, 6, 7], flags=gb.F_BC_SINGLE)
        assert np.array_equal(b1, b2)
        hd.free()


@pytest.mark.parametrize("wtype", ["u32", "f32"])
def test_small_plans(wtype, gb, orc):
    """More instances than SMs, of mixed sizes; a plan with a larger graph goes another way."""
    graphs = [gb.gen_rmat(5 + i % 6, 8, 40 + i, wtype) for i in range(330)] + [gb.gen_grid(40, 37, 3, wtype)]
    src = np.array([h.n // 3 for h in graphs], dtype=np.uint32)
    for extra in ([], [gb.gen_rmat(15, 16, 2, wtype)]):
        gs, sr = graphs + extra, np.concatenate([src, [7] * len(extra)]).astype(np.uint32)
        with gb.Pack(gs) as pk, gb.Plan(pk, sr) as plan:
            for _ in range(2):
                st = plan.run(per_instance=True)
            dist, pred = plan.results()
        assert st["completed"] == len(gs)
        for i in range(0, len(gs), 11 if extra else 1):
            h = gs[i]
            ref = orc.dijkstra(h.row, h.col, h.w, int(sr[i]))
            assert np.array_equal(dist[i], ref), i
            assert np.array_equal(pred[i], orc.min_tight_pred(h.row, h.col, h.w, int(sr[i]), ref)), i
            assert st["per_instance"][i]["reached"] == int(np.sum(pred[i] >= 0))


@pytest.mark.parametrize("wtype", ["u32", "f32"])
def test_small_light_bound(wtype, gb, orc):
    """A light bound alone keeps the one-CTA path (no run without full_items
    splits) and is reported as the persistent kernel reports it."""
    a = gb.gen_rmat(9, 16, 8, wtype)
    ref = orc.dijkstra(a.row, a.col, a.w, 5)
    with gb.Graph.from_host(a) as g:
        for light in (None, 0.0, 3.5, float("inf")):
            d, _, st = g.sssp(5, light=light)
            _, _, s2 = g.sssp(5, light=light, solo_entries=512)
            assert st["blocks"] == 1 and s2["blocks"] > 1 and np.array_equal(d, ref)
            assert st["light_used"] == s2["light_used"], light


@pytest.mark.parametrize("wtype", ["u32", "f32"])
def test_small_delta_used(wtype, gb):
    """The width reported is the one that ran: 64 default widths on graphs of at
    most 8 edges a vertex, 8 on others, and never past the uint32 range."""
    cases = [(gb.gen_grid(20, 30, 3, wtype), 64), (gb.gen_rmat(9, 16, 8, wtype), 8)]
    for a, scale in cases:
        with gb.Graph.from_host(a) as g:
            base = g.sssp(5, solo_entries=512)[2]["delta_used"]
            assert g.sssp(5)[2]["delta_used"] == scale * base
            assert g.sssp(5, delta=base)[2]["delta_used"] == scale * base
    if wtype == "u32":
        row, col, w = _csr(2, [(0, 1, 2**31 - 1)], np.uint32)
        with gb.Graph(row, col, w) as g:
            d, _, st = g.sssp(0)
            assert st["delta_used"] == 2**32 - 1 and d.tolist() == [0, 2**31 - 1]


@pytest.mark.parametrize("wtype,weights,m,one", [
    ("u32", "unit", 131072, True), ("u32", "unit", 131073, False), ("f32", "unit", 262144, True),
    ("u32", "uniform", 262144, True), ("u32", "uniform", 262145, False),
    ("f32", "skewed", 131072, True), ("f32", "skewed", 131073, False), ("u32", "zero", 131073, False)])
def test_small_limit_of_edges(wtype, weights, m, one, gb, orc):
    """The edge limit, half as large where the default width is a large part of
    the mean weight (unit float weights have a width of one sixteenth)."""
    n = 16384
    rng = np.random.default_rng(m)
    u, v = np.sort(rng.integers(0, n, m)), rng.integers(0, n, m).astype(np.uint32)
    row = np.zeros(n + 1, dtype=np.uint64)
    row[1:] = np.cumsum(np.bincount(u, minlength=n))
    w = {"unit": np.ones(m), "zero": np.zeros(m), "uniform": rng.integers(1, 256, m), "skewed": rng.lognormal(0, 2, m)}[weights]
    w = w.astype(np.uint32 if wtype == "u32" else np.float32)
    with gb.Graph(row, v, w) as g:
        d, p, st = g.sssp(3)
    ref = orc.dijkstra(row, v, w, 3)
    assert (st["blocks"] == 1) == one
    assert np.array_equal(d, ref) and np.array_equal(p, orc.min_tight_pred(row, v, w, 3, ref))


@pytest.mark.parametrize("weights,m,one", [
    ("unit", 131072, {1: True}), ("unit", 131073, {63: False, 64: True}), ("unit", 262145, {64: False}),
    ("skewed", 131073, {31: False, 32: True}), ("skewed", 262145, {63: False, 64: True}),
    ("uniform", 524288, {1: True, 2: True})])
def test_small_plan_limit(weights, m, one, gb, orc):
    """Instances from which on a plan gives each one CTA (the groups of the other
    kernel have at least two at these counts)."""
    n = 8192
    rng = np.random.default_rng(m)
    u, v = np.sort(rng.integers(0, n, m)), rng.integers(0, n, m).astype(np.uint32)
    row = np.zeros(n + 1, dtype=np.uint64)
    row[1:] = np.cumsum(np.bincount(u, minlength=n))
    w = {"unit": np.ones(m, np.uint32), "uniform": rng.integers(1, 256, m).astype(np.uint32),
         "skewed": rng.lognormal(0, 2, m).astype(np.float32)}[weights]
    with gb.Graph(row, v, w) as g:
        for k, expect in one.items():
            src = (np.arange(k, dtype=np.uint32) * 83) % n
            with gb.Plan(g, src) as plan:
                st = plan.run()
                dist, pred = plan.results()
            assert (st["group_ctas"] == 1) == expect, (k, st)
            for i in (0, k - 1):
                ref = orc.dijkstra(row, v, w, int(src[i]))
                assert np.array_equal(dist[i], ref)
                assert np.array_equal(pred[i], orc.min_tight_pred(row, v, w, int(src[i]), ref))


def test_small_pack_limit(gb, orc):
    """A pack goes by its number of graphs and every graph's weights."""
    rng = np.random.default_rng(4)
    n, m = 4096, 140000
    u, v = np.sort(rng.integers(0, n, m)), rng.integers(0, n, m).astype(np.uint32)
    row = np.zeros(n + 1, dtype=np.uint64)
    row[1:] = np.cumsum(np.bincount(u, minlength=n))
    wide = gb.HostGraph(row, v, np.ones(m, np.uint32))
    for graphs, one in (([gb.gen_rmat(8, 8, i) for i in range(40)] + [wide], False),
                        ([gb.gen_rmat(8, 8, i) for i in range(63)] + [wide], True),
                        ([gb.HostGraph(row, v, rng.integers(1, 256, m).astype(np.uint32))] * 2, True)):
        src = np.zeros(len(graphs), np.uint32)
        with gb.Pack(graphs) as pk, gb.Plan(pk, src) as plan:
            st = plan.run()
            dist, _ = plan.results()
        assert (st["group_ctas"] == 1) == one
        for i in (0, len(graphs) - 1):
            h = graphs[i]
            assert np.array_equal(dist[i], orc.dijkstra(h.row, h.col, h.w, 0))
