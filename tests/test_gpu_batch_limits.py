"""Plans whose shared memory is about the 48 KB that a kernel gets without
opting in to more, dynamic and static variables together; each in a process of
its own, since the limit, once raised, stays."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

RUN = """
import sys
sys.path.insert(0, %r)
import numpy as np
import oracle
import pico_gb300 as pg
n, parallel = int(sys.argv[1]), int(sys.argv[2])
v = np.arange(n)
rows = [np.array([u - 1, u + 1]) %% n for u in v]
for a, b in ((0, 1), (1, 0)):
    rows[a] = np.concatenate([rows[a], np.full(parallel, b)])
rowptr = np.concatenate([[0], np.cumsum([r.size for r in rows])]).astype(np.int64)
g = pg.Graph.from_csr(rowptr, np.concatenate(rows).astype(np.uint32))
b = pg.Batch(g, np.array([0, n], np.uint32))
for kv in sys.argv[3:]:
    name, value = kv.split("=")
    b.set_param(name, int(value))
assert np.array_equal(b.decompose()[0], oracle.bz(*g.csr())[0])
print("exact")
""" % ROOT


# dynamic shared memory of 48 KB less 32 bytes in the classes of 256 and 512
# threads and of 32-bit degrees (an edge repeated 70,000 times), and one step
# of 32 vertices below and above it
@pytest.mark.parametrize("n, parallel, params", [
    (21632, 0, []), (21664, 0, []), (21665, 0, []), (21664, 0, ["batch.small_n=24576"]),
    (20224, 0, ["batch.small_n=24576", "batch.small_threads=512"]), (8928, 70000, [])])
def test_plan_at_the_default_shared_memory_limit(n, parallel, params):
    r = subprocess.run([sys.executable, "-c", RUN, str(n), str(parallel)] + params, capture_output=True, text=True)
    assert r.returncode == 0 and "exact" in r.stdout, r.stderr[-2000:]
