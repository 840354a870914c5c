"""Long rows whose columns are crowded: runs of consecutive columns inside one
thread's part of the bitmap (1,664 columns), across its edges, in the first and
the last of several passes, beside scattered columns, and around the number
from which a warp writes them; against numpy."""
import numpy as np
import pytest

import pico_gb300 as pg
from test_gpu_build_rows import expected

pytestmark = pytest.mark.gpu

OWN = 52 * 32


def runs(n, length, scattered, rng):
    """About `length` distinct columns: `scattered` anywhere, the rest in runs."""
    cols = [rng.integers(50, n, scattered)]
    left = length - scattered
    for at, most in ((50, 70), (3 * OWN, OWN), (7 * OWN - 5, 10), (n - 2000, 2000), (n // 2, 82), (n // 3, left)):
        k = min(left, most)
        cols.append(np.arange(at, min(n, at + k)))
        left -= k
    return np.unique(np.concatenate(cols))


@pytest.mark.parametrize("n", [40000, 1703936, 1703937, 4000000])
def test_crowded_columns(n):
    rng = np.random.default_rng(n)
    src, dst = [], []
    for row, (length, scattered) in enumerate([(4097, 0), (4200, 10), (5000, 2500), (4608, 4500), (12000, 300), (30000, 0), (20000, 20000)]):
        c = runs(n, length, scattered, rng)
        c = np.concatenate([c, rng.choice(c, max(300, 4200 - c.size))])  # repeated lines
        src.append(np.full(c.size, row))
        dst.append(c)
    src, dst = np.concatenate(src), np.concatenate(dst)
    at = rng.permutation(src.size)
    src, dst = src[at].astype(np.uint32), dst[at].astype(np.uint32)
    for how in ("dedup", "sort"):
        g = pg.Graph.from_edges(src, dst, n, dedup=how == "dedup", sort_rows=how == "sort")
        rowptr, col = g.csr()
        want = expected(n, src, dst, how)
        assert np.array_equal(rowptr, want[0]) and np.array_equal(col, want[1])
        g.free()


def test_cliques_of_consecutive_vertices():
    k, n = 4500, 12000
    i, j = np.triu_indices(k, 1)
    src = np.concatenate([i, i + 7000]).astype(np.uint32)
    dst = np.concatenate([j, j + 7000]).astype(np.uint32)
    g = pg.Graph.from_edges(src, dst, n, dedup=True)
    rowptr, col = g.csr()
    deg = np.diff(rowptr)
    assert (deg[:k] == k - 1).all() and (deg[7000:7000 + k] == k - 1).all() and rowptr[-1] == 2 * k * (k - 1)
    rows = col.reshape(2, k, k - 1)
    want = np.array([np.delete(np.arange(k), v) for v in range(k)])
    assert np.array_equal(rows[0], want) and np.array_equal(rows[1], want + 7000)
    g.free()
