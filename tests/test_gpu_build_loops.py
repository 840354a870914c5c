"""Edge lists that hold no entry: self-loops alone, at vertex counts that take
one, two and three radix passes, in every row order."""
import numpy as np
import pytest

import pico_gb300 as pg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flags", [{}, {"sort_rows": True}, {"dedup": True}], ids=["keep", "sort", "dedup"])
@pytest.mark.parametrize("n", [1, 2, 2048, 2049, 5000, 5000000])
def test_self_loops_alone(n, flags):
    v = np.random.default_rng(n).integers(0, n, 3000).astype(np.uint32)
    g = pg.Graph.from_edges(v, v, n, **flags)
    rowptr, col = g.csr()
    assert rowptr.shape == (n + 1,) and not rowptr.any() and col.size == 0
    assert not g.decompose("peelone_dyn")[0].any()
    g.free()
