"""Partitioned builds of few edges over many rows: rows per edge below, at and
above the line from which the edges are not partitioned, with the narrowest and
the widest buckets; against numpy."""
import numpy as np
import pytest

import pico_gb300 as pg
from test_gpu_build_rows import expected, skewed

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("how", ["dedup", "sort"])
@pytest.mark.parametrize("n,m", [(16 << 20, 1 << 20), ((16 << 20) + 1, 1 << 20), (33554433, 2097151), (33554433, 2097153),
                                 (67108864, 4194304), (67108864, 4194303)])
def test_sparse_builds(n, m, how):
    src, dst = skewed(n, m, n % 1000 + m)
    g = pg.Graph.from_edges(src, dst, n, dedup=how == "dedup", sort_rows=how == "sort")
    rowptr, col = g.csr()
    keep = src != dst
    want = expected(n, src[keep], dst[keep], how)
    assert np.array_equal(rowptr, want[0]) and np.array_equal(col, want[1])
    g.free()
