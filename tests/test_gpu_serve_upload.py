"""Requests that the submitting call sends to the device, those that stay in
host memory, and groups of both: sizes around the 256 KB line, lane memory that
holds all, some or none of them, large graphs that run alone, several
submitting threads.  Every core array against Batagelj-Zaversnik."""
import threading

import numpy as np
import pytest

import oracle
import pico_gb300 as pg

pytestmark = pytest.mark.gpu


def csr(n, m, seed):
    """A random graph of exactly 2 * m entries."""
    rng = np.random.default_rng(seed)
    keys = np.empty(0, np.int64)
    while keys.size < m:
        a, b = rng.integers(0, n, (2, 2 * m))
        keys = np.union1d(keys, (np.minimum(a, b) * n + np.maximum(a, b))[a != b])
    keys = rng.permutation(keys)[:m]
    lo, hi = keys // n, keys % n
    both = np.sort(np.concatenate([lo * n + hi, hi * n + lo]))
    return np.searchsorted(both // n, np.arange(n + 1)).astype(np.int64), (both % n).astype(np.uint32)


# 8 (n + 1) + 8 m bytes: 262,136, 262,144 and 262,152 are the line and its neighbours
SIZES = [(50, 100), (2000, 30766), (2000, 30767), (2000, 30768), (20000, 60000), (3, 3), (60000, 200000), (1, 0),
         (250000, 300000), (40000, 90000)]


@pytest.mark.parametrize("slots,max_bytes,max_graphs", [(2, 256 << 20, 64), (1, 256 << 20, 3), (2, 4 << 20, 64),
                                                        (3, 1 << 20, 64), (1, 1, 1)])
def test_uploaded_and_held_requests(slots, max_bytes, max_graphs):
    reqs = [csr(n, m, 7 * i) for i, (n, m) in enumerate(SIZES)] * 2
    want = [oracle.bz(rp, col)[0] for rp, col in reqs[:len(SIZES)]] * 2
    g = pg.rmat_graph(12, 8, seed=3)
    s = pg.Server(g, decompose_slots=slots, max_batch_bytes=max_bytes, max_batch_graphs=max_graphs)
    got = [None] * len(reqs)

    def client(k):
        tickets = []
        for i in range(k, len(reqs), 2):
            rp, col = reqs[i][0].copy(), reqs[i][1].copy()
            tickets.append((i, s.submit_decompose(rp, col)))
            rp[:] = -1  # the server keeps nothing of the caller's arrays
            col[:] = 0xffffffff
        for i, t in tickets:
            got[i] = s.wait(t, core_cap=reqs[i][0].size - 1)["core"]

    threads = [threading.Thread(target=client, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    st = s.stats()
    s.close()
    assert st["completed_decompositions"] == len(reqs) and st["failed"] == 0
    for a, b in zip(got, want):
        assert np.array_equal(a, b)
