"""A graph whose device build runs out of memory is built on the host, and the
failed allocation leaves nothing behind: the first solve succeeds."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture
def limit(gb):
    f = gb.lib.gbs_test_buffer_limit
    f.restype, f.argtypes = None, [ctypes.c_size_t, ctypes.c_int]
    yield lambda most, memory=1: f(most, memory)
    f(0, 1)


@pytest.mark.parametrize("wtype", ["u32", "f32", "f64"])
@pytest.mark.parametrize("scale", [8, 15])          # one CTA, persistent kernel
def test_host_build_after_a_failed_device_build(wtype, scale, limit, gb, orc):
    a = gb.gen_rmat(scale, 16, 3, "f32" if wtype == "f32" else "u32")
    w = a.w / 3.0 if wtype == "f64" else a.w
    src = int(np.argmax(np.diff(a.row.astype(np.int64))))
    ref = orc.dijkstra(a.row, a.col, w, src)
    pred = orc.min_tight_pred(a.row, a.col, w, src, ref)
    for most in (1, 8 * a.n + 300, 9 * a.m):         # fails at the first buffer, at the columns, in the sort
        limit(most)
        with gb.Graph(a.row, a.col, w) as g:
            limit(0)
            d, p, _ = g.sssp(src)
            assert np.array_equal(d, ref) and np.array_equal(p, pred), most


def test_other_calls_after_a_failed_build(limit, gb, orc):
    a = gb.gen_rmat(9, 16, 5)
    with gb.DeviceCsr.from_arrays(a.row, a.col) as c, gb.Graph.from_host(a) as g:
        limit(1)
        with pytest.raises(gb.GbsError) as e:
            c.graph(gb.W_F32)
        assert e.value.name == "NO_MEMORY"
        with pytest.raises(gb.GbsError) as e:
            gb.DeviceCsr.from_arrays(a.row, a.col)
        assert e.value.name == "NO_MEMORY"
        limit(0)
        d, _, _ = g.sssp(7)
        assert np.array_equal(d, orc.dijkstra(a.row, a.col, a.w, 7))


def test_other_failures_are_reported(limit, gb, orc):
    """Only a full device, or none, sends a build to the host."""
    a = gb.gen_rmat(9, 16, 5)
    for most in (1, 9 * a.m):
        limit(most, 0)
        with pytest.raises(gb.GbsError) as e:
            gb.Graph.from_host(a)
        assert e.value.name == "CUDA"
    limit(0)
    with gb.Graph.from_host(a) as g:
        assert np.array_equal(g.sssp(7)[0], orc.dijkstra(a.row, a.col, a.w, 7))


@pytest.mark.parametrize("wtype", ["f32", "f64"])
@pytest.mark.parametrize("shuffled", [False, True])
def test_build_memory(wtype, shuffled, limit, gb, orc):
    """A build from a device CSR holds at most 40 bytes an edge and the sort's
    12, whatever the order of the columns."""
    a = gb.gen_rmat(15, 16, 7)
    col = a.col
    if shuffled:
        rows = np.repeat(np.arange(a.n), np.diff(a.row.astype(np.int64)))
        col = col[np.lexsort((np.random.default_rng(1).random(a.m), rows))]
    with gb.DeviceCsr.from_arrays(a.row, col) as c:
        row, col, w = c.export()
        limit(52 * a.m + (3 << 20))
        with c.graph(gb.W_F64 if wtype == "f64" else gb.W_F32) as g:
            limit(0)
            d, _, _ = g.sssp(7)
    assert np.array_equal(d, orc.dijkstra(row, col, w if wtype == "f64" else w.astype(np.float32), 7))
