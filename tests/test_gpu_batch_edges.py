"""The batched kernel at the sizes where its scan, queues and size classes
change over: 8-vertex scan groups and 32-bit bitmap words, more claims in one
scan than the id list holds, more row ranges in a round than the ring holds,
rows longer than one range, and the largest graph of each shared-memory class;
every result equals Batagelj-Zaversnik."""
import ctypes

import numpy as np
import pytest

import oracle
import pico_gb300 as pg

pytestmark = pytest.mark.gpu


def ring(n):
    """A cycle: every vertex is claimed by the same scan."""
    v = np.arange(n, dtype=np.uint32)
    return n, v, ((v + 1) % n).astype(np.uint32)


def random_graph(n, m, seed):
    rng = np.random.default_rng(seed)
    return n, rng.integers(0, n, m).astype(np.uint32), rng.integers(0, n, m).astype(np.uint32)


def hubs(n, k, seed):
    """k vertices joined to every other one: rows of n - 1 entries, cascades
    whose claims all queue at once."""
    s, d = np.meshgrid(np.arange(k), np.arange(n), indexing="ij")
    n, s2, d2 = random_graph(n, 2 * n, seed)
    return n, np.concatenate([s.ravel().astype(np.uint32), s2]), np.concatenate([d.ravel().astype(np.uint32), d2])


def pack(parts):
    vbase = np.concatenate([[0], np.cumsum([p[0] for p in parts])]).astype(np.uint32)
    src = np.concatenate([p[1] + vbase[i] for i, p in enumerate(parts)])
    dst = np.concatenate([p[2] + vbase[i] for i, p in enumerate(parts)])
    return pg.Graph.from_edges(src, dst, int(vbase[-1]), dedup=True), vbase


CASES = {
    "groups_and_words": [random_graph(n, 3 * n, n) for n in (1, 2, 7, 8, 9, 15, 16, 17, 31, 32, 33, 63, 64, 65, 255, 257)],
    "claims_beyond_the_lists": [ring(n) for n in (127, 1024, 1025, 5000, 12289, 30000, 60000, 105000)],
    "long_rows": [hubs(n, k, n) for n, k in ((300, 3), (5000, 9), (20000, 5), (40000, 6), (70000, 12))],
    "class_limits": [random_graph(n, 4 * n, n) for n in (12288, 12289, 24576, 25600, 26625, 49152, 51200, 53249, 98304, 107520,
                                                         108545)],
}


@pytest.mark.parametrize("config", [{}, {"batch.chunk": 128, "batch.small_threads": 64, "batch.large_threads": 128},
                                    {"batch.large_shared": 0, "batch.small_n": 1000, "batch.chunk": 1024}])
@pytest.mark.parametrize("name", sorted(CASES))
def test_batch_kernel_edges(name, config):
    g, vbase = pack(CASES[name])
    want = oracle.bz(*g.csr())[0]
    b = pg.Batch(g, vbase)
    for key, value in config.items():
        b.set_param(key, value)
    for _ in range(2):
        assert np.array_equal(b.decompose()[0], want)
    b.free()
    g.free()


@pytest.mark.parametrize("part", [ring(50000), ring(1), hubs(20000, 5, 3), random_graph(49999, 1000000, 4), random_graph(33, 90, 5)])
def test_noalloc_edges(part):
    g = pg.Graph.from_edges(part[1], part[2], part[0], dedup=True)
    rowptr, col = g.device_csr()
    out = pg.DeviceBuffer(4 * g.n)
    pg.check(pg.lib().kc_decompose_noalloc(ctypes.c_void_p(rowptr), ctypes.c_void_p(col), g.n, ctypes.c_void_p(out.ptr), None))
    assert np.array_equal(out.download(np.uint32, g.n), oracle.bz(*g.csr())[0])
    out.free()
    g.free()


def test_batch_plan_over_empty_graphs_and_tiles():
    """Segments of 0, 1 and up to 9,000 vertices (tiles of 4,096 vertices and
    entries end inside, at and between graphs), with edgeless ones first and
    last; then one vertex moved to its neighbour's segment is refused."""
    rng = np.random.default_rng(5)
    sizes = [0, 1, 0, 0, 3, 4095, 1, 4096, 0, 2, 9000, 31, 0, 5000, 64, 1, 0]
    parts = [random_graph(n, 3 * n, n) if n > 2 else (n, np.zeros(0, np.uint32), np.zeros(0, np.uint32)) for n in sizes]
    g, vbase = pack(parts)
    want = oracle.bz(*g.csr())[0]
    b = pg.Batch(g, vbase)
    assert np.array_equal(b.decompose()[0], want)
    b.free()
    for i in (5, 7, 10, 13):  # the first vertex of a connected segment into the one before
        moved = vbase.copy()
        moved[i] += 1
        for j in range(i - 1, 0, -1):
            moved[j] = min(moved[j], moved[i])
        with pytest.raises(pg.KCoreError):
            pg.Batch(g, moved)
    g.free()
