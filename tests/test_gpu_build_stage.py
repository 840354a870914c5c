"""The partitioned CSR build where its last step changes form: 4,096 rows per
bucket, the most that are sorted by tile in shared memory, and 8,192; buckets
of one tile, of several and of tiles that are exactly full; rows that fill a
tile by themselves and tiles of single-entry rows.  Against numpy."""
import numpy as np
import pytest

import pico_gb300 as pg

pytestmark = pytest.mark.gpu


def lines(kind, n, m, rng):
    if kind == "uniform":
        return rng.integers(0, n, m), rng.integers(0, n, m)
    if kind == "hub":  # row 7 in every line
        return np.full(m, 7), rng.integers(0, n, m)
    # full tiles: every line has one end in the first bucket, none in it twice,
    # so that the bucket's entries are the lines (a multiple of 32,768 of them)
    return rng.integers(0, 64, m), rng.integers(n // 2, n, m)


@pytest.mark.parametrize("kind,m", [("uniform", (1 << 20) + 12345), ("hub", 1 << 20), ("bucket", 1 << 20), ("bucket", (1 << 20) + 1)])
@pytest.mark.parametrize("n", [4194304, 8388608, 8388609])
def test_staged_and_direct_rows(n, kind, m):
    rng = np.random.default_rng(n + m)
    src, dst = lines(kind, n, m, rng)
    flip = rng.random(m) < 0.5
    a, b = np.where(flip, dst, src).astype(np.uint32), np.where(flip, src, dst).astype(np.uint32)
    on = a != b
    row = np.concatenate([a[on], b[on]]).astype(np.int64)
    other = np.concatenate([b[on], a[on]]).astype(np.int64)
    key = np.sort(row * n + other)
    for how in ("sort", "dedup"):
        want = key if how == "sort" else np.unique(key)
        g = pg.Graph.from_edges(a, b, n, dedup=how == "dedup", sort_rows=how == "sort")
        rowptr, col = g.csr()
        g.free()
        assert np.array_equal(rowptr, np.searchsorted(want // n, np.arange(n + 1)))
        assert np.array_equal(col, (want % n).astype(np.uint32))
