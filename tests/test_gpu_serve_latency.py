"""What the submitting call does with a request is part of its latency: a graph
of 120 MB, whose copy is most of the call, to the device and to host memory."""
import time

import numpy as np
import pytest

import pico_gb300 as pg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("max_bytes", [1 << 30, 1], ids=["device", "host"])
def test_latency_covers_the_submitting_call(max_bytes):
    n, k = 300000, 50  # every vertex joined to the k before and the k after it
    step = np.concatenate([np.arange(-k, 0), np.arange(1, k + 1)])
    col = ((np.arange(n)[:, None] + step) % n).astype(np.uint32).ravel()
    rowptr = np.arange(n + 1, dtype=np.int64) * (2 * k)
    s = pg.Server(pg.rmat_graph(12, 8, seed=3), decompose_slots=1, max_batch_bytes=max_bytes)
    for _ in range(3):
        t0 = time.perf_counter()
        ticket = s.submit_decompose(rowptr, col)
        call_ms = 1e3 * (time.perf_counter() - t0)
        res = s.wait(ticket, core_cap=n)
        wall_ms = 1e3 * (time.perf_counter() - t0)
        assert (res["core"] == 2 * k).all()
        # a lane may take the request while the call returns; the copy comes before that
        assert res["queue_ms"] > 0.5 * call_ms, (res["queue_ms"], call_ms)
        assert res["queue_ms"] < res["latency_ms"] <= wall_ms
    s.close()
