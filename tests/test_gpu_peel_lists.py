"""The peel's per-CTA vertex lists at the sizes where they change place:
graphs with fewer 32-vertex groups than CTAs, vertex counts around a group's
edge, lists of about one entry per thread and of about the shared-memory
capacity per CTA, and levels that empty a list; every result equals
Batagelj-Zaversnik, with the default grid and with one CTA per SM."""
import numpy as np
import pytest

import oracle
import pico_gb300 as pg

pytestmark = pytest.mark.gpu


def graph(n, deg, seed):
    """A ring (so that no vertex is isolated) and n * deg / 2 random edges."""
    rng = np.random.default_rng(seed)
    v = np.arange(n, dtype=np.uint32)
    m = n * deg // 2
    src = np.concatenate([v, rng.integers(0, n, m).astype(np.uint32)])
    dst = np.concatenate([((v + 1) % n).astype(np.uint32), (n * rng.random(m) ** 3).astype(np.uint32)])
    return pg.Graph.from_edges(src, dst, n, dedup=True)


# 304 or 152 CTAs of 512 threads: 32 n-groups per CTA at 311,296 vertices (512
# entries with 304 CTAs), LIST_CAP = 2,048 entries at 622,592
SIZES = [1, 2, 31, 32, 33, 63, 65, 4095, 4864, 9727, 9728, 9729, 155647, 155649, 311296, 311297, 622591, 622593, 700001]


@pytest.mark.parametrize("ctas_per_sm", [0, 1])
@pytest.mark.parametrize("n", SIZES)
def test_peel_lists(n, ctas_per_sm):
    g = graph(n, 8, n)
    want = oracle.bz(*g.csr())[0]
    g.set_param("peel.ctas_per_sm", ctas_per_sm)
    for _ in range(2):
        got, st = g.decompose("peelone_dyn")
        assert np.array_equal(got, want)
        assert st.levels == np.unique(want).size
    g.free()


@pytest.mark.parametrize("setting", [{"peel.threads": 256}, {"peel.scan_unroll": 8}, {"peel.balanced": 0}, {"peel.queues": 8}])
def test_peel_lists_in_every_variant(setting):
    g = graph(400001, 12, 3)
    want = oracle.bz(*g.csr())[0]
    for name, value in setting.items():
        g.set_param(name, value)
    for grid in (1, 0):  # a larger grid after a smaller one regrows the lists
        g.set_param("peel.ctas_per_sm", grid)
        assert np.array_equal(g.decompose("peelone")[0], want)
    g.free()
