"""PageRank on rows at the edges of its classes (degrees around 32, 8 and 32
words, a partly filled last word, column counts not divisible by four) and
stops at the edges of an iteration batch: ranks and iteration counts are the
oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rows(lengths, n, seed):
    rng = np.random.default_rng(seed)
    row = np.zeros(n + 1, dtype=np.uint64)
    deg = np.zeros(n, dtype=np.int64)
    deg[: len(lengths)] = lengths
    rng.shuffle(deg)
    row[1:] = np.cumsum(deg)
    return row, rng.integers(0, n, int(row[-1])).astype(np.uint32)


@pytest.mark.parametrize("lengths", [
    [0, 1, 2, 31, 32, 33, 34, 63, 64, 65] * 3,
    [225, 226, 255, 256, 257, 258, 287, 288] * 2 + [1],
    [993, 994, 1023, 1024, 1025, 1026, 1055, 1056, 1057, 3] * 2,
    [5000, 70000, 3, 32],
    [1],
    [0],
])
def test_row_classes(lengths, gb, orc):
    for n in (max(64, len(lengths)), 700):
        row, col = _rows(lengths, n, len(lengths) + n)
        with gb.DeviceCsr.from_arrays(row, col) as c:
            pr, st = c.pagerank(max_iters=60)
        ref, it = orc.pagerank(row, col, 0.3, 1e-6, 60)
        assert st["iterations"] == it
        assert np.array_equal(pr, ref, equal_nan=True)


@pytest.mark.parametrize("iters", [1, 7, 8, 9, 16, 17])
def test_stops_inside_and_between_batches(iters, gb, orc):
    a = gb.gen_rmat(9, 8, 5)
    with gb.DeviceCsr.from_arrays(a.row, a.col) as c:
        pr, st = c.pagerank(max_iters=iters)
        ref, it = orc.pagerank(a.row, a.col, 0.3, 1e-6, iters)
        assert st["iterations"] == it == iters and st["converged"] == 0 and np.array_equal(pr, ref)
        for th in (0.3, 0.05, 0.01, 1e-3, 1e-4):       # converge after different numbers of iterations
            pr, st = c.pagerank(threshold=th)
            ref, it = orc.pagerank(a.row, a.col, 0.3, th)
            assert st["iterations"] == it and st["converged"] == 1 and np.array_equal(pr, ref)
