"""The spill tunable goes back to its default: explicit values and -1 on one
graph, before and after the autotuner, which may set one of its own."""
import numpy as np
import pytest

import oracle
import pico_gb300 as pg

pytestmark = pytest.mark.gpu


def test_spill_by_row_length_after_explicit_values():
    g = pg.rmat_graph(16, 16, seed=5)
    want = oracle.bz(*g.csr())[0]
    g.set_param("trace", 1)

    def spilled(value):
        g.set_param("peel.spill", value)
        assert np.array_equal(g.decompose("peelone")[0], want)
        return sum(t["spilled"] for t in g.trace())

    everything = spilled(0)
    by_rule = spilled(-1)
    kept = spilled(3072)
    assert kept < by_rule < everything
    g.autotune()
    assert kept < spilled(-1) < everything
    for value in (-2, 3073):
        with pytest.raises(pg.KCoreError) as e:
            g.set_param("peel.spill", value)
        assert e.value.code == pg.KC_ERR_INVALID
    g.free()
