"""Rounds of about one item per warp: bands (vertex v joined to the k after it)
peel from their ends, so a batch graph of c bands has about 2 c items a round,
below, at and above the warps of a CTA, with rows of one window of 32 entries
and of one more, and rows cut into ranges; in every degree class."""
import ctypes

import numpy as np
import pytest

import oracle
import pico_gb300 as pg

pytestmark = pytest.mark.gpu


def bands(n, k, c):
    v = np.repeat(np.arange(n), k)
    d = v + np.tile(np.arange(1, k + 1), n)
    v, d = v[d < n], d[d < n]
    off = (np.arange(c) * n)[:, None]
    return n * c, (v + off).ravel().astype(np.uint32), (d + off).ravel().astype(np.uint32)


BANDS = [(300, 1), (200, 4), (120, 16), (120, 17), (150, 64), (200, 65), (300, 130)]
CONFIGS = [{}, {"batch.chunk": 128, "batch.small_threads": 64}, {"batch.large_shared": 0, "batch.small_n": 32}]


@pytest.mark.parametrize("config", CONFIGS, ids=["default", "chunks", "global"])
@pytest.mark.parametrize("c", [1, 2, 4, 5, 16, 17])
def test_chains(c, config):
    parts = [bands(n, k, c) for n, k in BANDS]
    vbase = np.concatenate([[0], np.cumsum([p[0] for p in parts])]).astype(np.uint32)
    src = np.concatenate([p[1] + vbase[i] for i, p in enumerate(parts)])
    dst = np.concatenate([p[2] + vbase[i] for i, p in enumerate(parts)])
    g = pg.Graph.from_edges(src, dst, int(vbase[-1]), dedup=True)
    b = pg.Batch(g, vbase)
    for name, value in config.items():
        b.set_param(name, value)
    assert np.array_equal(b.decompose()[0], oracle.bz(*g.csr())[0])
    b.free()
    g.free()


@pytest.mark.parametrize("n, k", BANDS)
def test_chain_without_allocation(n, k):
    total, src, dst = bands(n, k, 16)
    g = pg.Graph.from_edges(src, dst, total, dedup=True)
    rowptr, col = g.device_csr()
    out = pg.DeviceBuffer(4 * total)
    pg.check(pg.lib().kc_decompose_noalloc(ctypes.c_void_p(rowptr), ctypes.c_void_p(col), total, ctypes.c_void_p(out.ptr), None))
    assert np.array_equal(out.download(np.uint32, total), oracle.bz(*g.csr())[0])
    out.free()
    g.free()
