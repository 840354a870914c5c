"""Where a cascade starts in few places, the claims go to the shared queues as
long as CTAs are idle, however few row entries a CTA holds: on grids the waves
from the corners are a few hundred short rows, less than a CTA may keep."""
import numpy as np
import pytest

import pico_gb300 as pg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("setting", [{}, {"peel.threads": 256}, {"peel.balanced": 0}, {"peel.ctas_per_sm": 1}])
def test_waves_of_short_rows_are_shared(setting):
    k = 400
    v = np.arange(k * k, dtype=np.uint32).reshape(k, k)
    src = np.concatenate([v[:, :-1].ravel(), v[:-1].ravel()])
    dst = np.concatenate([v[:, 1:].ravel(), v[1:].ravel()])
    g = pg.Graph.from_edges(src, dst, k * k, dedup=True)
    g.set_param("trace", 1)
    for name, value in setting.items():
        g.set_param(name, value)
    core, _ = g.decompose("peelone")
    assert (core == 2).all()  # each corner goes first, then the diagonals behind it
    assert sum(t["spilled"] for t in g.trace()) > 100
    g.free()
