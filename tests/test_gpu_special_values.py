"""GPU: inputs with NaN, infinite and out-of-range values, and meshes with
collapsed elements (whose updates divide by zero).  The two-copies sweep leaves
solves out that cannot lower a value; the one-copy kernel of the bit-exact
build runs every one, that of the fast build lists them by its own test.  The
kernels must agree, to the bit, on such inputs too."""
import numpy as np
import pytest

import lsgb300
import synth

pytestmark = pytest.mark.gpu


def _workload(name, n, seed, kind):
    w = synth.workload(name, n=n, seed=seed)
    rng = np.random.default_rng(seed)
    x, p = w["xyz"].copy(), w["phi0"].copy()
    nv = len(p)
    if kind == "collapsed":
        # some vertices moved onto another vertex of the mesh
        k = rng.integers(0, nv, nv // 15)
        x[k] = x[w["elems"][rng.integers(0, len(w["elems"]), len(k)), 0]]
    if kind == "nan":
        p[rng.integers(0, nv, 5)] = np.nan
    if kind == "inf":
        p[rng.integers(0, nv, 5)] = np.inf
        p[rng.integers(0, nv, 3)] = -np.inf
    if kind == "beyond":  # interface values above LARGENUM
        p = np.where(p > 0, np.float32(1e10), np.float32(-1e10))
        p[rng.integers(0, nv, 9)] = -0.0
    if kind == "scattered":  # the same, and patches that are not connected
        p = np.where(p > 0, np.float32(1e10), np.float32(-1e10))
        p[rng.integers(0, nv, 9)] = -0.0
        w["npart"], w["nparts"] = (rng.permutation(nv) % 40).astype(np.int32), 40
    w["xyz"], w["phi0"] = x.astype(np.float32), p.astype(np.float32)
    if w["update"] == "curvature":
        w["dt"] = 0.2 * w["h"] ** 2
    return w


KINDS = ["plain", "collapsed", "nan", "inf", "beyond", "scattered"]


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("name,n", [("c2", 8), ("c2", 5), ("c3", 7)])
@pytest.mark.parametrize("kw", [dict(), dict(largenum=0.3), dict(length_scale=7.0), dict(ref_compat=True)])
@pytest.mark.parametrize("bit_exact", [False, True])
def test_kernels_agree(kind, name, n, kw, bit_exact):
    for seed in (0, 1, 2, 3, 7):
        w = _workload(name, n, seed, kind)
        out = []
        for ctas in (3, 5, 6, 7):
            ls = lsgb300.from_workload(w, bit_exact=bit_exact, fim_ctas_per_sm=ctas, max_fim_iters=150, **kw)
            try:
                hist, done = ls.solve(3)
            except lsgb300.LevelSetError as e:
                hist, done = ls.phi(), -e.code
            out.append((done, hist))
        for done, hist in out[1:]:
            assert done == out[0][0]
            assert np.array_equal(hist, out[0][1], equal_nan=True)


@pytest.mark.parametrize("stretch", [1, 2, 5, 50])
@pytest.mark.parametrize("largenum", [0.05, 0.1, 0.3])
def test_exact_kernels_agree_where_candidates_pass_largenum(stretch, largenum):
    # interface values between LARGENUM and the heights of their tets: the
    # solver's result is capped at LARGENUM, though its candidates lie above
    for seed in range(12):
        w = dict(_workload("c2", 8, seed, "plain"), update="none")
        w["xyz"] = w["xyz"] * np.array([stretch, 1, 1], np.float32)
        w["phi0"] = np.random.default_rng(seed).normal(size=len(w["phi0"])).astype(np.float32) * np.float32(w["h"])
        hist = [lsgb300.from_workload(w, bit_exact=True, fim_ctas_per_sm=c, largenum=largenum, max_fim_iters=150).solve(2)[0]
                for c in (3, 5, 7)]
        assert np.array_equal(hist[0], hist[1], equal_nan=True) and np.array_equal(hist[0], hist[2], equal_nan=True)
