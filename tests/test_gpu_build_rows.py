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
@pytest.mark.parametrize("n", [40000, 1703936, 1703937, 4000000, 14155777])
def test_row_sorts(n, how):
    for seed, repeat in ((1, 0.0), (2, 0.3)):
        src, dst = hub_rows(n, EDGES, seed, repeat)
        g = pg.Graph.from_edges(src, dst, n, dedup=how == "dedup", sort_rows=how == "sort")
        rowptr, col = g.csr()
        want_rowptr, want_col = expected(n, src, dst, how)
        assert np.array_equal(rowptr, want_rowptr)
        assert np.array_equal(col, want_col)
        g.free()


def skewed(n, m, seed):
    """m lines with repeated edges, self-loops and columns crowded at low ids."""
    rng = np.random.default_rng(seed)
    src = (n * rng.random(m) ** 3).astype(np.uint32)
    dst = rng.integers(0, n, m).astype(np.uint32)
    dst[::97] = src[::97]
    src[1::3], dst[1::3] = src[: src[1::3].size], dst[: src[1::3].size]
    return src, dst


# around the line count from which edges are partitioned, and over bucket
# widths: one bucket, a last bucket cut by n, few rows with many tiles each,
# 2,048 and 4,096 buckets (16,384 rows each), and more rows than buckets cover
@pytest.mark.parametrize("how", ["dedup", "sort"])
@pytest.mark.parametrize("n,m", [(50, 1 << 20), (64, (1 << 20) - 1), (65, (1 << 20) + 1), (131073, 1 << 20), (262143, 1300001),
                                 (262145, 2000003), (33554433, 1 << 20), (67108864, 1 << 20), (67108865, 1 << 20)])
def test_partitioned_build(n, m, how):
    src, dst = skewed(n, m, n)
    g = pg.Graph.from_edges(src, dst, n, dedup=how == "dedup", sort_rows=how == "sort")
    rowptr, col = g.csr()
    keep = src != dst
    want_rowptr, want_col = expected(n, src[keep], dst[keep], how)
    assert np.array_equal(rowptr, want_rowptr)
    assert np.array_equal(col, want_col)
    g.free()


def test_partitioned_build_of_one_hub_and_bad_ids():
    n, m = 3000000, 1500000
    src, dst = np.zeros(m, np.uint32), np.arange(1, m + 1, dtype=np.uint32)  # every line meets row 0
    g = pg.Graph.from_edges(src, dst, n, dedup=True)
    rowptr, col = g.csr()
    assert rowptr[1] == m and np.array_equal(col[:m], dst) and not col[m:].any()
    g.free()
    for at in (0, m - 1):
        bad = dst.copy()
        bad[at] = n
        with pytest.raises(pg.KCoreError) as e:
            pg.Graph.from_edges(src, bad, n, dedup=True)
        assert e.value.code == pg.KC_ERR_INVALID


# row counts around the digit widths of one, two and three passes, and line
# counts around a tile (4,096 lines) and a stretch of tiles
@pytest.mark.parametrize("n,m", [(1, 5), (2, 1), (2, 4095), (3, 4096), (2048, 4097), (2049, 20000), (5000, 2500001), (65537, 999),
                                 (4194304, 300000), (4194305, 300000), (70000000, 5000), (100000, 1245185)])
def test_rows_in_edge_list_order(n, m):
    src, dst = skewed(n, m, n + m)
    g = pg.Graph.from_edges(src, dst, n)
    rowptr, col = g.csr()
    keep = src != dst
    want_rowptr, want_col = expected(n, src[keep], dst[keep], "keep")
    assert np.array_equal(rowptr, want_rowptr)
    assert np.array_equal(col, want_col)
    g.free()
