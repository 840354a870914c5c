"""The CSR rewrite of an update where its pieces change over: change lists of
one tile, of several and of too many entries for the tiled sort; row and column
arrays around their tiles; edits at the first and last entry, into empty rows
and of whole rows; repeated, reversed and self-loop lines, edges both deleted
and inserted, and entries that change nothing.  Against numpy, exactly."""
import numpy as np
import pytest

import oracle
import pico_gb300 as pg

pytestmark = pytest.mark.gpu


def keys_of(s, d):
    s, d = np.asarray(s, np.int64), np.asarray(d, np.int64)
    on = s != d
    return np.unique(np.minimum(s, d)[on] << 32 | np.maximum(s, d)[on])


def split(keys):
    return (keys >> 32).astype(np.uint32), (keys & 0xffffffff).astype(np.uint32)


def csr_of(n, keys):
    lo, hi = keys >> 32, keys & 0xffffffff
    both = np.sort(np.concatenate([lo << 32 | hi, hi << 32 | lo]))
    return np.searchsorted(both >> 32, np.arange(n + 1)).astype(np.int64), (both & 0xffffffff).astype(np.uint32)


def apply_and_check(g, n, keys, ins, dels, full):
    """One update and the numpy one; returns the new keys."""
    ik, dk = keys_of(*ins), keys_of(*dels)
    gone = np.setdiff1d(np.intersect1d(keys, dk), ik)
    come = np.setdiff1d(ik, keys)
    want = np.union1d(np.setdiff1d(keys, gone), come)
    core, st = g.update(ins if len(ins[0]) else None, dels if len(dels[0]) else None)
    rp, col = g.csr()
    rp2, col2 = csr_of(n, want)
    assert np.array_equal(rp, rp2) and np.array_equal(col, col2)
    assert g.max_degree == int(np.diff(rp2).max(initial=0))
    if full:
        assert (st["deleted"], st["inserted"]) == (gone.size, come.size)
    assert np.array_equal(core, oracle.bz(rp2, col2)[0])
    return want


def graph(n, keys, full):
    g = pg.Graph.from_edges(*split(keys), n, dedup=True)
    big = 0 if full else 1 << 30
    g.set_param("update.incremental_max", big)
    g.set_param("update.deletion_incremental_max", big)
    g.decompose("peelone_dyn")
    return g


# listed edges: a tile holds 1,024, the tiled sort 65,536
@pytest.mark.parametrize("m", [1, 127, 128, 129, 1023, 1024, 1025, 2048, 9000, 65535, 65536, 65537])
def test_list_lengths(m):
    n = 5000
    rng = np.random.default_rng(m)
    keys = keys_of(rng.integers(0, n, 120000), rng.integers(0, n, 120000))
    g = graph(n, keys, True)
    for n_ins, n_del in ((m, 0), (0, m), (m, m)):
        a, b = rng.integers(0, n, (2, n_ins))
        lines = rng.permutation(keys)[:n_del]
        s, d = split(lines)
        pad = n_del - s.size  # more lines than edges: absent ones
        s = np.concatenate([s, rng.integers(0, n, pad, dtype=np.uint32)])
        d = np.concatenate([d, rng.integers(0, n, pad, dtype=np.uint32)])
        flip = rng.random(n_del) < 0.5
        dels = (np.where(flip, d, s), np.where(flip, s, d))
        keys = apply_and_check(g, n, keys, (a.astype(np.uint32), b.astype(np.uint32)), dels, True)


# rows around the row tile, entries around the column tile
@pytest.mark.parametrize("full", [True, False])
@pytest.mark.parametrize("n,entries", [(2, 0), (2, 2), (2047, 8190), (2048, 8192), (2049, 8194), (4097, 512),
                                       (40000, 16384)])
def test_array_edges(n, entries, full):
    rng = np.random.default_rng(n + entries)
    keys = np.empty(0, np.int64)
    while keys.size < entries // 2:
        keys = np.union1d(keys, keys_of(rng.integers(0, n, entries), rng.integers(0, n, entries)))
    keys = np.sort(rng.permutation(keys)[:entries // 2])
    g = graph(n, keys, full)
    none = (np.empty(0, np.uint32),) * 2
    ends = keys[[0, -1]] if keys.size else keys
    corner = np.array([1, (n - 2) << 32 | (n - 1)], np.int64)  # edges (0, 1) and (n-2, n-1)
    steps = [(split(corner), none), (none, split(ends)), (split(ends), split(corner)),  # put back, taken out
             (none, split(keys)), (split(np.union1d(keys, corner)), none),          # emptied, filled
             (([0, 1, 0], [1, 0, 0]), ([0, 0], [1, 0])), (none, none)]              # repeats, self-loops, kept
    for ins, dels in steps:
        ins, dels = (tuple(np.asarray(x, np.uint32) for x in e) for e in (ins, dels))
        keys = apply_and_check(g, n, keys, ins, dels, full)


@pytest.mark.parametrize("m", [3, 70000])
def test_bad_ids_leave_the_graph(m):
    n = 3000
    rng = np.random.default_rng(5)
    keys = keys_of(rng.integers(0, n, 20000), rng.integers(0, n, 20000))
    g = graph(n, keys, True)
    good = rng.integers(0, n, (2, m)).astype(np.uint32)
    bad = good.copy()
    bad[1, m // 2] = n
    for ins, dels in ((bad, None), (None, bad), (good, bad), (bad, good), (good[:, :3], bad), (bad[:, m // 2:], good)):
        with pytest.raises(pg.KCoreError) as e:
            g.update(tuple(ins) if ins is not None else None, tuple(dels) if dels is not None else None)
        assert e.value.code == pg.KC_ERR_INVALID
    rp, col = g.csr()
    rp2, col2 = csr_of(n, keys)
    assert np.array_equal(rp, rp2) and np.array_equal(col, col2)
