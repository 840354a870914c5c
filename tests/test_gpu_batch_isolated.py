"""Batch graphs with isolated vertices: none, some and all of a graph, at the
sizes of the scan's groups and of every degree class; a first level above zero
and one at zero with rows behind it."""
import numpy as np
import pytest

import oracle
import pico_gb300 as pg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("config", [{}, {"batch.large_shared": 0, "batch.small_n": 32}], ids=["default", "global"])
def test_isolated_vertices(config):
    rng = np.random.default_rng(3)
    src, dst, sizes = [], [], []
    for n in (1, 7, 8, 9, 33, 1000, 12289, 30000, 54000, 110000):
        for share in (0.0, 0.5, 1.0):
            v = np.arange(n) + sum(sizes)
            ids = rng.permutation(v)[: int(n * (1 - share))]
            src.append(ids)
            dst.append(np.roll(ids, 1))
            src.append(rng.choice(ids, 2 * ids.size) if ids.size else ids)
            dst.append(rng.choice(ids, 2 * ids.size) if ids.size else ids)
            sizes.append(n)
    vbase = np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint32)
    g = pg.Graph.from_edges(np.concatenate(src).astype(np.uint32), np.concatenate(dst).astype(np.uint32), int(vbase[-1]), dedup=True)
    b = pg.Batch(g, vbase)
    for name, value in config.items():
        b.set_param(name, value)
    want = oracle.bz(*g.csr())[0]
    g.decompose("gppeel")  # leaves ones where the batch has to write zeros
    for _ in range(2):
        assert np.array_equal(b.decompose()[0], want)
    b.free()
    g.free()
