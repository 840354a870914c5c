"""Requests at the size from which the submitting call sends the graph to the
device, alone, together and among smaller and larger ones, with lane memory for
all, some or none; against Batagelj-Zaversnik."""
import numpy as np
import pytest

import oracle
import pico_gb300 as pg
from test_gpu_serve_upload import csr

pytestmark = pytest.mark.gpu

# 8 (n + 1) + 8 m bytes: 786,424, 786,432 and 786,440 are the line and its neighbours
SIZES = [(2000, 96302), (2000, 96303), (2000, 96304), (50, 100), (30000, 200000), (2000, 96303)]


@pytest.mark.parametrize("slots,max_bytes", [(2, 256 << 20), (1, 8 << 20), (2, 1)])
def test_requests_at_the_upload_line(slots, max_bytes):
    reqs = [csr(n, m, 11 * i) for i, (n, m) in enumerate(SIZES)]
    want = [oracle.bz(rp, col)[0] for rp, col in reqs]
    s = pg.Server(pg.rmat_graph(12, 8, seed=3), decompose_slots=slots, max_batch_bytes=max_bytes)
    for (rp, col), w in zip(reqs, want):
        assert np.array_equal(s.wait(s.submit_decompose(rp, col), core_cap=w.size)["core"], w)
    tickets = [s.submit_decompose(rp, col) for rp, col in reqs]
    for t, w in zip(tickets, want):
        assert np.array_equal(s.wait(t, core_cap=w.size)["core"], w)
    st = s.stats()
    s.close()
    assert st["completed_decompositions"] == 2 * len(reqs) and st["failed"] == 0
