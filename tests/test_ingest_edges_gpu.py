"""Device readers at the edges of their chunks and of the id ranges: records that
start on and around 512-byte chunk boundaries, blanks, comments, missing final
newline, files in and out of row order, ids with many and few bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _expect_text(n, recs, send=True):
    row = np.array([(a if send else b) - 1 for a, b in recs], dtype=np.int64)
    col = np.array([(b if send else a) - 1 for a, b in recs], dtype=np.int64)
    o = np.argsort(row, kind="stable")
    off = np.zeros(n + 1, dtype=np.uint64)
    off[1:] = np.cumsum(np.bincount(row, minlength=n))
    return off, col[o].astype(np.uint32), np.array([b for _, b in recs]) / n


@pytest.mark.parametrize("order", ["sorted", "shuffled"])
@pytest.mark.parametrize("pad", [0, 1, 7, 15, 16, 17, 479, 480, 481, 497, 511, 512, 513])
def test_text_chunk_edges(pad, order, gb):
    rng = np.random.default_rng(pad)
    n = 97
    recs = [(int(a), int(b)) for a, b in rng.integers(1, n + 1, (700, 2))]
    recs.sort() if order == "sorted" else rng.shuffle(recs)
    recs = [tuple(r) for r in recs]
    lines = []
    for i, (a, b) in enumerate(recs):
        lines.append(f"{' ' * (i % 3)}a{' ' if i % 2 else chr(9)}{a} {b} {i}")
        if i % 11 == 0:
            lines.append("c" + " a" * (i % 5))          # comments whose later tokens are "a"
        if i % 13 == 0:
            lines.append("")
    head = "c" + "x" * max(0, pad - 2) + "\n" if pad else ""
    for tail in ("", "\n", "\n\n"):
        text = (head + f"p sp {n} {len(recs)} 1 {n}\n" + "\n".join(lines) + tail).encode()
        for direction in (gb.DIR_SEND, gb.DIR_RECV):
            with gb.DeviceCsr.parse_text(text, direction) as c:
                row, col, w = c.export()
                assert c.info["records"] == c.info["edges"] == len(recs)
            off, ecol, ew = _expect_text(n, recs, direction == gb.DIR_SEND)
            assert np.array_equal(row, off) and np.array_equal(col, ecol) and np.array_equal(w, ew)


def test_text_stops_at_e_num_and_refuses_short_lines(gb):
    recs = [(1 + i % 9, 1 + i % 7) for i in range(50)]
    body = "".join(f"a {a} {b} 1\n" for a, b in recs)
    with gb.DeviceCsr.parse_text(f"p sp 9 20 1 9\n{body}".encode()) as c:
        assert c.info["records"] == 50 and c.m == 20
        row, col, _ = c.export()
    off, ecol, _ = _expect_text(9, recs[:20])
    assert np.array_equal(row, off) and np.array_equal(col, ecol)
    for bad in ("a \n" * 60, "a 1 2\n" * 10, body + "a 1 x 1\n", body + "a 10 1 1\n", body + "a 1 0 1\n"):
        with pytest.raises(gb.GbsError) as e:
            gb.DeviceCsr.parse_text(f"p sp 9 1000 1 9\n{bad}".encode())
        assert e.value.name == "INVALID_ARG"


@pytest.mark.parametrize("dedup", [False, True])
@pytest.mark.parametrize("n,m", [(1, 0), (1, 5), (2, 33), (255, 3000), (256, 3000), (257, 3000), (70000, 5000)])
def test_bin_ids_and_order(n, m, dedup, gb):
    rng = np.random.default_rng(n + m)
    for kind in ("random", "sorted", "last row"):
        p = rng.integers(1, min(n, 40) + 1, (m, 2)).astype("<i8")
        p[m // 2:] = rng.integers(1, n + 1, (m - m // 2, 2))
        if kind == "sorted":
            p = p[np.argsort(p[:, 0], kind="stable")]
        elif kind == "last row":
            p[:, 0] = n
        data = np.array([n, m, 1, n], dtype="<i8").tobytes() + p.tobytes()
        q = p
        if dedup and m:
            _, first = np.unique(p[:, 0] * (n + 1) + p[:, 1], return_index=True)
            q = p[np.sort(first)]
        with gb.DeviceCsr.parse_bin(data, dedup=dedup) as c:
            row, col, w = c.export()
            assert c.info["duplicates"] == m - len(q)
        o = np.argsort(q[:, 0], kind="stable")
        off = np.zeros(n + 1, dtype=np.uint64)
        off[1:] = np.cumsum(np.bincount(q[:, 0] - 1, minlength=n))
        assert np.array_equal(row, off) and np.array_equal(col, (q[o, 1] - 1).astype(np.uint32))
        assert np.array_equal(w, np.where(np.arange(len(q)) % 2, 0.2, 0.1))


def test_bin_large_ids_are_refused_after_duplicates_go(gb):
    """Raw ids up to 2^32 - 1 take part in duplicate removal; beyond [0, v_num) they are refused."""
    p = np.array([[1, 1], [2**32 - 1, 2**32 - 1], [1, 1]], dtype="<i8")
    data = np.array([4, 3, 1, 4], dtype="<i8").tobytes() + p.tobytes()
    with pytest.raises(gb.GbsError) as e:
        gb.DeviceCsr.parse_bin(data, dedup=True)
    assert "edge 1" in str(e.value)
    p[1] = (2**32, 1)
    with pytest.raises(gb.GbsError) as e:
        gb.DeviceCsr.parse_bin(np.array([4, 3, 1, 4], dtype="<i8").tobytes() + p.tobytes(), dedup=True)
    assert "outside [0, 2^32)" in str(e.value)
