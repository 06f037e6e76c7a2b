"""GPU: the seeds of the standalone eikonal solve.  The bit-exact build with
every seed given the oracle's way (one redistance from those seeds over the
whole mesh is covered elsewhere); here the argument forms: a vertex given
more than once counts with its last value, the order of distinct seeds does
not matter, values at and above LARGENUM seed nothing closer, more seeds in a
later call than in the first, all vertices as seeds, and none."""
import numpy as np
import pytest

import lsgb300
import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,n,flags", [(2, 13, 0), (3, 9, 0), (3, 9, lsgb300.HOST_STAGING)])
def test_seed_forms(dim, n, flags):
    w = synth.workload("c1" if dim == 2 else "c2", n=n)
    # a length unit that is a power of two: the FIM frame scales exactly
    ls = lsgb300.from_workload(w, bit_exact=True, flags=flags, length_scale=0.125)
    nv = len(w["xyz"])
    rng = np.random.default_rng(n)
    seeds = rng.choice(nv, 7, replace=False).astype(np.int32)
    values = rng.uniform(0, 0.2, 7).astype(np.float32)
    d = ls.eikonal(seeds, values)
    # a seed is never visited
    assert np.array_equal(d[seeds], values) and np.all(d < 1e9)
    order = rng.permutation(7)
    np.testing.assert_array_equal(ls.eikonal(seeds[order], values[order]), d)
    # duplicates: the last value of each vertex
    twice = np.concatenate([seeds, seeds]), np.concatenate([values + 0.3, values])
    np.testing.assert_array_equal(ls.eikonal(*twice), d)
    # a seed at LARGENUM holds that value and starts no front
    far = np.setdiff1d(np.arange(nv, dtype=np.int32), seeds)[:1]
    e = ls.eikonal(np.concatenate([seeds, far]), np.concatenate([values, [2e9]]).astype(np.float32))
    keep = np.ones(nv, bool)
    keep[far] = False
    assert e[far[0]] == 1e9 and np.all(e[keep] >= d[keep])
    # every vertex a seed; none
    allv = rng.uniform(0, 1, nv).astype(np.float32)
    np.testing.assert_array_equal(ls.eikonal(np.arange(nv, dtype=np.int32), allv), allv)
    assert np.all(ls.eikonal(np.zeros(0, np.int32), np.zeros(0, np.float32)) == 1e9)
    np.testing.assert_array_equal(ls.eikonal(seeds, values), d)
