"""Plans and builds that start with a short upload, made while other threads
upload large graphs: the kernels behind the upload read what this call wrote.
Batches change their graphs' sizes and order from one to the next, edge lists
their lines, so that what an earlier call left behind is another result."""
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

import oracle
import pico_gb300 as pg

pytestmark = pytest.mark.gpu


def lists(seed):
    rng = np.random.default_rng(seed)
    n = int(rng.integers(50, 3000))
    m = int(n * rng.uniform(1, 8))
    return n, rng.integers(0, n, m).astype(np.uint32), rng.integers(0, n, m).astype(np.uint32)


def test_short_uploads_beside_long_ones():
    rng = np.random.default_rng(1)
    n = 1 << 20
    big = oracle.csr_dedup(n, rng.integers(0, n, 8 << 20).astype(np.uint32), rng.integers(0, n, 8 << 20).astype(np.uint32))
    parts = [lists(seed) for seed in range(24)]
    cores = [oracle.bz(*oracle.csr_dedup(*p))[0] for p in parts]

    def uploads(_):
        for _ in range(30):
            pg.Graph.from_csr(*big).free()
        return True

    def builds(k):
        for i in range(60):
            j = (5 * i + k) % len(parts)
            n, s, d = parts[j]
            g = pg.Graph.from_edges(s, d, n, dedup=True)
            ok = np.array_equal(g.decompose("peelone")[0], cores[j])
            g.free()
            if not ok:
                return False
        return True

    def batches(k):
        for i in range(30):
            take = np.random.default_rng(100 * k + i).permutation(len(parts))[: 3 + i % 20]
            vbase = np.concatenate([[0], np.cumsum([parts[j][0] for j in take])]).astype(np.uint32)
            src = np.concatenate([parts[j][1] + vbase[q] for q, j in enumerate(take)])
            dst = np.concatenate([parts[j][2] + vbase[q] for q, j in enumerate(take)])
            g = pg.Graph.from_edges(src, dst, int(vbase[-1]), dedup=True)
            b = pg.Batch(g, vbase)
            ok = np.array_equal(b.decompose()[0], np.concatenate([cores[j] for j in take]))
            b.free()
            g.free()
            if not ok:
                return False
        return True

    with ThreadPoolExecutor(6) as ex:
        jobs = [ex.submit(f, k) for k in range(2) for f in (uploads, builds, batches)]
        assert all(j.result() for j in jobs)
