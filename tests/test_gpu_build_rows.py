"""The CSR build's row sorts at the lengths where they change over: one warp,
registers of one to eight warps (powers of two from 32 to 4,096 entries and
their neighbours), column bitmaps of one and of several passes, and the radix
sort of rows too short for the bitmaps of many columns; de-duplicated, sorted
and in edge-list order, against numpy."""
import numpy as np
import pytest

import pico_gb300 as pg

pytestmark = pytest.mark.gpu

EDGES = sorted({x for k in range(5, 14) for x in (2 ** k - 1, 2 ** k, 2 ** k + 1)} | {2, 3, 4097, 4607, 4608, 20000})


def hub_rows(n, lengths, seed, repeat):
    """Vertex i gets lengths[i] edges to vertices above the hubs, the first
    `repeat` part of them repeated; lines in random order, either way round."""
    rng = np.random.default_rng(seed)
    src, dst = [], []
    for i, k in enumerate(lengths):
        fresh = max(1, int(round(k * (1 - repeat))))
        t = len(lengths) + rng.choice(n - len(lengths), fresh, replace=False)
        src.append(np.full(k, i))
        dst.append(np.concatenate([t, rng.choice(t, k - fresh)]))
    src, dst = np.concatenate(src), np.concatenate(dst)
    order = rng.permutation(src.size)
    flip = rng.random(src.size) < 0.5
    src, dst = src[order], dst[order]
    return np.where(flip, dst, src).astype(np.uint32), np.where(flip, src, dst).astype(np.uint32)


def expected(n, src, dst, how):
    row = np.stack([src, dst], 1).reshape(-1).astype(np.int64)
    other = np.stack([dst, src], 1).reshape(-1).astype(np.int64)
    if how == "keep":
        at = np.argsort(row, kind="stable")
        row, col = row[at], other[at]
    else:
        key = np.sort(row * n + other)
        if how == "dedup":
            key = np.unique(key)
        row, col = key // n, key % n
    return np.searchsorted(row, np.arange(n + 1)).astype(np.int64), col.astype(np.uint32)


# columns: one bitmap, three, nine (rows below 9 * 512 = 4,608 entries keep the radix sort)
@pytest.mark.parametrize("how", ["dedup", "sort", "keep"])
@pytest.mark.parametrize("n", [40000, 1572864, 1572865, 4000000, 14155777])
def test_row_sorts(n, how):
    for seed, repeat in ((1, 0.0), (2, 0.3)):
        src, dst = hub_rows(n, EDGES, seed, repeat)
        g = pg.Graph.from_edges(src, dst, n, dedup=how == "dedup", sort_rows=how == "sort")
        rowptr, col = g.csr()
        want_rowptr, want_col = expected(n, src, dst, how)
        assert np.array_equal(rowptr, want_rowptr)
        assert np.array_equal(col, want_col)
        g.free()
