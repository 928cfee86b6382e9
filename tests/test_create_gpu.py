"""gbs_graph_create checks and sorts on the device: graphs with unsorted rows,
parallel edges and -0 weights give the oracle's results in every weight type,
the resident rows are the same whatever order the edges come in, and every
malformed input is refused with its reason."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DT = {"u32": np.uint32, "f32": np.float32, "f64": np.float64}


def _random_csr(n, m, seed, dtype):
    rng = np.random.default_rng(seed)
    deg = np.bincount(rng.integers(0, n, m) ** 2 // n, minlength=n)       # skewed rows, empty ones among them
    row = np.zeros(n + 1, dtype=np.uint64)
    row[1:] = np.cumsum(deg)
    col = rng.integers(0, n, m).astype(np.uint32)
    w = rng.integers(0, 9, m).astype(dtype)
    if dtype != np.uint32:
        w = w / dtype(3)
        w[w == 0] = dtype(-0.0)
    return row, col, w


def _sorted_rows(row, col, w, by_col_only=False):
    r = np.repeat(np.arange(len(row) - 1), np.diff(row.astype(np.int64)))
    o = np.lexsort((col, r) if by_col_only else (col, np.abs(w), r))
    return col[o], w[o]


@pytest.mark.parametrize("wtype", ["u32", "f32", "f64"])
@pytest.mark.parametrize("n,m", [(1, 0), (1, 3), (5, 31), (33, 1023), (40, 1024), (700, 1025), (3000, 40000)])
def test_create_orders(wtype, n, m, gb, orc):
    row, col, w = _random_csr(n, m, n + m, DT[wtype])
    src = n // 2
    ref = orc.dijkstra(row, col, np.abs(w) if wtype != "u32" else w, src)
    pred = orc.min_tight_pred(row, col, np.abs(w) if wtype != "u32" else w, src, ref)
    for c, x in ((col, w), _sorted_rows(row, col, w, True), _sorted_rows(row, col, w)):
        with gb.Graph(row, c, x) as g:
            info = g.info()
            assert (info["n"], info["m"]) == (n, m)
            assert info["max_weight"] == (float(np.abs(w).max()) if m else 0.0)
            for kw in ({}, {"full_items": 1, "delta": 1.0}):           # the split needs sorted rows
                d, p, _ = g.sssp(src, **kw)
                assert np.array_equal(d, ref) and np.array_equal(p, pred)


@pytest.mark.parametrize("what", ["offsets end", "offsets decrease", "column", "negative", "nan", "inf", "first bad wins"])
def test_create_refuses(what, gb):
    row, col, w = _random_csr(300, 5000, 3, np.float64)
    want = "weights must be finite"
    if what == "offsets end":
        row = row.copy()
        row[-1] += 1
        want = "start at 0 and end at m"
    elif what == "offsets decrease":
        row = row.copy()
        row[150] = row[-1] + 7
        col[4999] = 1 << 31                 # the offsets are reported first
        want = "row_offsets decrease"
    elif what == "column":
        col[4321] = 300
        want = "column index out of range"
    elif what == "first bad wins":
        col[4000] = 300
        w[3999] = -1.0
    else:
        w[17] = {"negative": -1.0, "nan": np.nan, "inf": np.inf}[what]
    for dtype in (np.float64, np.float32):
        with pytest.raises(gb.GbsError) as e:
            gb.Graph(row, col, w.astype(dtype))
        assert e.value.name == "INVALID_ARG" and want in str(e.value)


def test_mean_weight_is_reproducible(gb):
    """Builds of one graph agree in the controller input that holds the mean
    weight, here half way between two float32 values: the last bit of the sum
    decides which."""
    import math
    n, m = 1 << 12, 1 << 20
    rng = np.random.default_rng(5)
    row = np.arange(0, m + 1, m // n, dtype=np.uint64)
    col = rng.integers(0, n, m).astype(np.uint32)
    w = rng.random(m)
    w[0] = 1.0
    half = m * (0.5 + 2.0 ** -25)                  # float32 values near one half are 2^-24 apart
    for i in range(1, m):                          # weights moved until the exact sum is m times that
        gap = half - math.fsum(w)
        if gap == 0.0:
            break
        w[i] = min(max(w[i] + gap, 2.0 ** -20), 1.0 - 2.0 ** -20)
    assert math.fsum(w) == half
    seen = set()
    for _ in range(24):
        with gb.Graph(row, col, w) as g:
            g.sssp(1, flags=gb.F_FEATURES)
            seen.add(float(g.features()[0, 14]))
    assert len(seen) == 1 and seen <= {0.5, 0.5 + 2.0 ** -24}


@pytest.mark.parametrize("wtype", ["u32", "f64"])
def test_long_runs_of_empty_rows(wtype, gb, orc):
    """Few edges among many vertices: a build and a float64 solve search past
    empty rows instead of walking them (they took 400 times as long)."""
    import time
    n, m = 1 << 22, 4096
    rng = np.random.default_rng(8)
    best = []
    for most in (n, 64):                          # rows anywhere, rows of 64 edges at the front
        u, v = np.sort(rng.integers(0, most, m)), rng.integers(0, most, m).astype(np.uint32)
        row = np.zeros(n + 1, dtype=np.uint64)
        row[1:] = np.cumsum(np.bincount(u, minlength=n))
        w = rng.integers(1, 99, m).astype(DT[wtype])
        times = []
        for _ in range(4):
            t = time.perf_counter()
            with gb.Graph(row, v, w) as g:
                d, p, _ = g.sssp(int(u[0]))
            times.append(time.perf_counter() - t)
        best.append(min(times))
        ref = orc.dijkstra(row, v, w, int(u[0]))
        assert np.array_equal(d, ref) and np.array_equal(p, orc.min_tight_pred(row, v, w, int(u[0]), ref))
    assert best[0] < 3 * best[1], best
