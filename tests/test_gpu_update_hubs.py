"""Insertions whose subcore search crosses hub rows, of lengths around the
chunks in which such rows are searched: trees of hubs and leaves (every core 1),
closed into cycles a few edges at a time."""
import numpy as np
import pytest

import oracle
import pico_gb300 as pg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("leaves", [(1022, 1023, 1024), (1025, 2047, 2048), (2049, 3071, 40000)])
def test_insertions_through_hub_rows(leaves):
    k = len(leaves)
    src, dst, n = [np.arange(k - 1)], [np.arange(1, k)], k  # the hubs form a path
    for hub, count in enumerate(leaves):
        src.append(np.full(count, hub))
        dst.append(np.arange(n, n + count))
        n += count
    g = pg.Graph.from_edges(np.concatenate(src).astype(np.uint32), np.concatenate(dst).astype(np.uint32), n, dedup=True)
    g.decompose("peelone_dyn")
    rng = np.random.default_rng(k + n)
    first = k
    steps = [([0], [k - 1]),  # the hubs' cycle
             ([first], [n - 1]),  # leaves of the first and the last hub
             (rng.integers(k, n, 40), rng.integers(k, n, 40)),
             (np.zeros(200, int), rng.integers(k, n, 200))]  # many edges at one hub: one round each
    for a, b in steps:
        core, st = g.update((np.asarray(a, np.uint32), np.asarray(b, np.uint32)), None)
        rp, col = g.csr()
        assert st["recomputed"] == 0
        assert np.array_equal(core, oracle.bz(rp, col)[0])
