"""Batch graphs whose largest degree is at the limits of the 15- and 16-bit
classes, too large for 32-bit degrees in shared memory and at the edge of what
16-bit ones take, with deep cores and edgeless vertices beside the hub."""
import numpy as np
import pytest

import oracle
import pico_gb300 as pg

pytestmark = pytest.mark.gpu


def hub_graph(n, degree, seed):
    """Vertex 0 with exactly `degree` neighbours, a clique of 200, sparse rest;
    the last vertices have no edge."""
    rng = np.random.default_rng(seed)
    nb = rng.permutation(np.arange(1, n))[:degree]
    a, b = np.triu_indices(200, 1)
    who = rng.permutation(np.arange(1, n))[:200]
    s, d = rng.integers(1, n - 9, (2, n // 2))
    return n, np.concatenate([np.zeros(degree, int), who[a], s]), np.concatenate([nb, who[b], d])


SIZES = [(53000, 32768), (54000, 32767), (54000, 32768), (70000, 65534), (70000, 65535), (108544, 40000), (108545, 40000),
         (108544, 65534), (66000, 65999)]


@pytest.mark.parametrize("config", [{}, {"batch.large_threads": 128, "batch.chunk": 128}], ids=["default", "small"])
def test_hubs_at_the_class_limits(config):
    parts = [hub_graph(n, degree, i) for i, (n, degree) in enumerate(SIZES)]
    vbase = np.concatenate([[0], np.cumsum([p[0] for p in parts])]).astype(np.uint32)
    src = np.concatenate([p[1] + vbase[i] for i, p in enumerate(parts)]).astype(np.uint32)
    dst = np.concatenate([p[2] + vbase[i] for i, p in enumerate(parts)]).astype(np.uint32)
    g = pg.Graph.from_edges(src, dst, int(vbase[-1]), dedup=True)
    rowptr, col = g.csr()
    assert [int(np.diff(rowptr[lo:hi + 1]).max()) for lo, hi in zip(vbase[:-1], vbase[1:])] == [x[1] for x in SIZES]
    b = pg.Batch(g, vbase)
    for name, value in config.items():
        b.set_param(name, value)
    want = oracle.bz(rowptr, col)[0]
    for _ in range(2):
        assert np.array_equal(b.decompose()[0], want)
    b.free()
    g.free()
