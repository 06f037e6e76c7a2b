"""Cases that measure this framework's paths as its users run them.

A case is one call sequence of the public Python interface (the ctypes mirror
of the C ABI): a narrowband time step through host buffers, a run of steps
with its history, a batch of meshes, a standalone eikonal solve, and the
learned warm start's network in training and in inference.  Sizes, meshes and
parameters are those of the package's own workloads (synth.py): jittered unit
squares and cubes, CFL 0.5 advection by a rotation or a constant wind,
mean-curvature flow at dt = 0.5 h^2, narrowbands of 5 h and 6 h.

The mesh of a case is fixed by its size; the seed draws the interface, the
velocity and the data.  The handle (mesh, partition, device layout) is the
plan that a program keeps; `run` is the call that it repeats.
"""
import functools
import os
import sys

import numpy as np

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
for _p in (os.path.join(ROOT, "sci-solver_level-set_gb300"),):
    if _p not in sys.path:
        sys.path.insert(0, _p)

import lsgb300  # noqa: E402
import synth  # noqa: E402

# bytes of one narrowband vertex-update: the vertex's values and its share of
# the elements' connectivity, coordinates and velocity, each once
UPDATE_BYTES = {(3, "curvature"): 113.8, (3, "advect"): 173.2, (2, "advect"): 54.8, (2, "curvature"): 46.8}


def listed():
    return [
        # the smallest call: a short 2D advection run with the history of
        # every step, as the reference's solveLevelSet returns it
        dict(name="run2d-64", kind="run", dim=2, n=64, update="advect", part="blocks", build="fast", steps=20),
        # a large triangle mesh with the default graph partition (16-vertex patches)
        dict(name="step2d-graph-403", kind="step", dim=2, n=403, update="curvature", part="graph", build="fast"),
        # the small 3D advection workload, several steps per call
        dict(name="run3d-32", kind="run", dim=3, n=32, update="advect", part="blocks", build="fast", steps=10),
        # an unstructured mesh: shuffled numbering, default graph partition, odd size
        dict(name="step3d-graph-45", kind="step", dim=3, n=45, update="advect", part="graph", build="fast"),
        # the headline workload, one step through host buffers
        dict(name="step3d-128", kind="step", dim=3, n=128, update="curvature", part="blocks", build="fast"),
        # the bit-exact build and the precision form, options that users take for parity and accuracy
        dict(name="step3d-exact-48", kind="step", dim=3, n=48, update="curvature", part="blocks", build="exact"),
        dict(name="step3d-fp64-33", kind="step", dim=3, n=33, update="curvature", part="blocks", build="fp64"),
        # many small and ordinary meshes stepped together
        dict(name="batch3d-12", kind="batch", dim=3, nmin=16, nmax=48, meshes=12, steps=2),
        # distances from a few sources over a whole mesh
        dict(name="eikonal2d-150", kind="eikonal", dim=2, n=150, part="graph", sources=5),
        dict(name="eikonal3d-64", kind="eikonal", dim=3, n=64, part="blocks", sources=3),
        # the network of the learned warm start: training (forward, backward,
        # optimiser) and inference on a held-out set, host arrays in and out
        dict(name="mlp-train-50000", kind="train", n=50000, batch=8192, epochs=2),
        dict(name="mlp-predict-40001", kind="predict", n=40001),
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["run", "run", "step", "step", "step", "step", "batch", "eikonal", "eikonal", "train", "predict"])
    if kind in ("run", "step"):
        dim = rng.choice([2, 3, 3])
        part = rng.choice(["blocks", "blocks", "graph"])
        build = "fast" if dim == 2 else rng.choice(["fast", "fast", "fast", "exact", "fp64"])
        hi = 420 if dim == 2 else (96 if build == "fast" and part == "blocks" else 48)
        c = dict(kind=kind, dim=dim, n=_log(rng, 48 if dim == 2 else 16, hi), update=rng.choice(["advect", "curvature"]),
                 part=part, build=build)
        if kind == "run":
            # the histories of large runs come in fewer steps
            c["n"] = min(c["n"], 200 if dim == 2 else 40)
            c["steps"] = rng.randint(2, 12)
        return c
    if kind == "batch":
        lo = rng.randint(10, 20)
        return dict(kind=kind, dim=3, nmin=lo, nmax=lo + rng.randint(4, 24), meshes=rng.randint(3, 14),
                    steps=rng.randint(1, 3))
    if kind == "eikonal":
        dim = rng.choice([2, 3])
        return dict(kind=kind, dim=dim, n=_log(rng, 40, 300) if dim == 2 else _log(rng, 12, 64),
                    part=rng.choice(["blocks", "graph"]), sources=rng.randint(1, 9))
    if kind == "train":
        return dict(kind=kind, n=_log(rng, 3000, 50000), batch=rng.choice([1024, 3000, 8192, 16384]),
                    epochs=rng.randint(1, 2))
    return dict(kind=kind, n=_log(rng, 100, 60000))


# ---------------------------------------------------------------- inputs
@functools.lru_cache(maxsize=4)
def _mesh(dim, n, shuffled):
    """Jittered unit square or cube; shuffled: random vertex and element
    numbering, as a mesh generator's output."""
    xyz, el = synth.square_mesh(n, 0.2, 0) if dim == 2 else synth.cube_mesh(n, 0.15, 0)
    if shuffled:
        rng = np.random.default_rng(n)
        perm = rng.permutation(len(xyz))
        new = np.empty(len(xyz), np.int64)
        new[perm] = np.arange(len(xyz))
        xyz = np.ascontiguousarray(xyz[perm])
        el = np.ascontiguousarray(new[el][rng.permutation(len(el))].astype(np.int32))
    return xyz, el


def _interface(dim, xyz, rng):
    """Signed distance to a union of one to three circles or spheres."""
    k = int(rng.integers(1, 4))
    centers = rng.uniform(0.3, 0.7, size=(k, dim))
    radii = rng.uniform(0.1, 0.25, size=k)
    d = np.full(len(xyz), np.inf, np.float32)
    p = xyz[:, :dim]
    for c, r in zip(centers.astype(np.float32), radii.astype(np.float32)):
        q = p - c
        d = np.minimum(d, np.sqrt(np.einsum("ij,ij->i", q, q)) - r)
    return d


def _velocity(dim, xyz, el, rng):
    """Constant wind (2D) or a rigid rotation about the centre (3D), one
    vector per element, and its largest speed."""
    if dim == 2:
        a = rng.uniform(0, 2 * np.pi)
        v = np.zeros((len(el), 3), np.float32)
        v[:, 0], v[:, 1] = np.cos(a), np.sin(a)
        return v, 1.0
    axis = rng.normal(size=3)
    v = synth.velocity_rotation(xyz, el, 2 * np.pi, axis=axis)
    return v, float(np.sqrt(np.einsum("ij,ij->i", v, v).max()))


def _partition(ls, dim, n, part):
    if part == "blocks":
        ls.set_partition(*synth.structured_partition(dim, n + 1, 5 if dim == 2 else 3))
    # otherwise the library's default partitioner (graph, 16-vertex patches)


def _handle(case, rng, setup=True):
    dim, n = case["dim"], case["n"]
    xyz, el = _mesh(dim, n, case["part"] == "graph")
    h = 1.0 / n
    kw = {}
    if case["update"] == "curvature":
        kw = dict(update_kind=lsgb300.UPDATE_CURVATURE, time_step=0.5 * h * h, bandwidth=6 * h)
        vel = None
    else:
        vel, speed = _velocity(dim, xyz, el, rng)
        kw = dict(update_kind=lsgb300.UPDATE_ADVECT, time_step=0.5 * h / speed * case.get("cfl", 1.0), bandwidth=5 * h)
    flags = {"fast": 0, "exact": lsgb300.BITEXACT, "fp64": lsgb300.FP64_FLAGGED}[case["build"]]
    ls = lsgb300.LevelSet(dim == 2, lsgb300.default_params(flags=flags, **kw))
    ls.set_mesh(xyz, el)
    _partition(ls, dim, n, case["part"])
    phi = _interface(dim, xyz, rng)
    ls.set_phi(phi)
    if vel is not None:
        ls.set_velocity(vel)
    if setup:
        ls.setup()
    return ls, phi


def _samples(n, rng):
    """Rows of network input as the warm start makes them: 32 slots of
    (dx, dy, dz, phi) / h, the first the vertex itself, some of the last
    empty; the target is the vertex's distance."""
    x = rng.standard_normal((n, 32, 4), dtype=np.float32)
    x[:, :, :3] *= 0.6
    normal = rng.standard_normal((n, 3), dtype=np.float32)
    normal /= np.linalg.norm(normal, axis=1, keepdims=True)
    t = rng.uniform(-5, 5, n).astype(np.float32)
    x[:, 0, :3] = 0
    x[:, :, 3] = t[:, None] + np.einsum("nsk,nk->ns", x[:, :, :3], normal) + 0.02 * x[:, :, 3]
    ring = rng.integers(10, 32, n)
    x[np.arange(32)[None, :] >= ring[:, None]] = 0
    return np.ascontiguousarray(x.reshape(n, 128)), t


def _weights(rng):
    f = 128
    w = rng.uniform(-np.sqrt(6 / f), np.sqrt(6 / f), 3 * f * f)
    w4 = rng.uniform(-np.sqrt(3 / f), np.sqrt(3 / f), f)
    return np.concatenate([w, rng.uniform(-0.05, 0.05, 3 * f), w4, [0.0]]).astype(np.float32)


def _batch_members(case, rng):
    sizes = np.linspace(case["nmin"], case["nmax"], case["meshes"]).round().astype(int)
    for n in sizes:
        # a small step: the interfaces keep their shape over a long series of calls
        yield dict(kind="step", dim=3, n=int(n), update="advect", part="blocks", build="fast", cfl=1e-3)


def _seeds(case, nv, rng):
    seeds = np.sort(rng.choice(nv, size=case["sources"], replace=False)).astype(np.int32)
    values = rng.uniform(0, 0.1, case["sources"]).astype(np.float32)
    return seeds, values


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind in ("run", "step"):
        ls, phi = _handle(case, rng)
        return dict(case=case, ls=ls, phi=phi, out=np.zeros_like(phi))
    if kind == "batch":
        b = lsgb300.LevelSetBatch()
        for c in _batch_members(case, rng):
            ls, _ = _handle(c, rng, setup=False)
            b.add(ls)
            ls.close()
        b.setup()
        return dict(case=case, batch=b)
    if kind == "eikonal":
        dim, n = case["dim"], case["n"]
        xyz, el = _mesh(dim, n, case["part"] == "graph")
        ls = lsgb300.LevelSet(dim == 2, lsgb300.default_params())
        ls.set_mesh(xyz, el)
        _partition(ls, dim, n, case["part"])
        ls.setup()
        seeds, values = _seeds(case, len(xyz), rng)
        return dict(case=case, ls=ls, seeds=seeds, values=values)
    net = lsgb300.MLP(0)
    w = _weights(rng)
    x, t = _samples(case["n"], rng)
    net.set_params(w)
    return dict(case=case, net=net, w=w, x=x, t=t)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "step":
        state["ls"].step_host(state["phi"], state["out"])
        return state["out"]
    if kind == "run":
        state["ls"].set_phi(state["phi"])
        return state["ls"].solve(case["steps"])[0]
    if kind == "batch":
        b = state["batch"]
        b.solve(case["steps"])
        return [b.phi(i) for i in range(case["meshes"])]
    if kind == "eikonal":
        return state["ls"].eikonal(state["seeds"], state["values"])
    net = state["net"]
    if kind == "train":
        # from the start's weights: set_params restarts the optimiser too
        net.set_params(state["w"])
        loss = net.train(state["x"], state["t"], epochs=case["epochs"], batch=case["batch"])
        return {"params": net.params(), "loss": loss}
    return net.predict(state["x"])


# ---------------------------------------------------------------- work
def _step_work(dim, n, update, xyz, rng):
    """Bytes and operations of one step: phi in and out, and the narrowband's
    vertex-updates, each with its elements' local solves once."""
    width = (6.0 if update == "curvature" else 5.0) / n
    band = float(np.count_nonzero(np.abs(_interface(dim, xyz, rng)) <= width))
    per = 5.5 * 4 * 100 if dim == 3 else 2 * 3 * 40
    return 8.0 * len(xyz) + band * UPDATE_BYTES[(dim, update)], band * per


def work(case):
    rng = np.random.default_rng(0)
    kind = case["kind"]
    f = 128
    if kind in ("run", "step"):
        xyz, _ = _mesh(case["dim"], case["n"], False)
        b, fl = _step_work(case["dim"], case["n"], case["update"], xyz, rng)
        k = case.get("steps", 1)
        return {"bytes": k * b, "flops": k * fl}
    if kind == "batch":
        b = fl = 0.0
        for c in _batch_members(case, rng):
            x = _step_work(3, c["n"], "advect", _mesh(3, c["n"], False)[0], rng)
            b, fl = b + x[0] * case["steps"], fl + x[1] * case["steps"]
        return {"bytes": b, "flops": fl}
    if kind == "eikonal":
        xyz, el = _mesh(case["dim"], case["n"], False)
        d1 = case["dim"] + 1
        return {"bytes": len(xyz) * 16.0 + len(el) * 4.0 * d1, "flops": len(el) * d1 * (100.0 if d1 == 4 else 40.0)}
    if kind == "train":
        return {"bytes": case["n"] * 4.0 * (f + 1) + 16.0 * 3 * f * f, "flops": case["epochs"] * case["n"] * 3 * 6.0 * f * f}
    return {"bytes": case["n"] * 4.0 * (f + 1) + 4.0 * 3 * f * f, "flops": case["n"] * 3 * 2.0 * f * f}


# ---------------------------------------------------------------- exact
def _torch():
    import torch

    return torch, torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _local(torch, P, T, X):
    """Least T_lin(y) + |y - X| over the simplex with vertices P (lists of
    [n, 3]) and values T: the vertices, the edges' stationary points and, for a
    triangle, the interior ones."""
    best = T[0] + (P[0] - X).norm(dim=1)
    for a in range(1, len(P)):
        best = torch.minimum(best, T[a] + (P[a] - X).norm(dim=1))
    for a in range(len(P)):
        for b in range(a + 1, len(P)):
            f, w, u = P[b] - P[a], X - P[a], T[b] - T[a]
            ff, fw, ww = (f * f).sum(1), (f * w).sum(1), (w * w).sum(1)
            q = ff - u * u
            r = torch.sqrt(torch.clamp(ff * ww - fw * fw, min=0)) / torch.sqrt(torch.where(q > 0, q, torch.ones_like(q)))
            lam = (fw - u * r) / ff
            ok = (q > 0) & (lam >= 0) & (lam <= 1)
            best = torch.where(ok, torch.minimum(best, T[a] + lam * u + r), best)
    if len(P) == 3:
        e1, e2, w = P[0] - P[2], P[1] - P[2], X - P[2]
        a, b, c = (e1 * e1).sum(1), (e1 * e2).sum(1), (e2 * e2).sum(1)
        u1, u2 = T[0] - T[2], T[1] - T[2]
        det = a * c - b * b
        g1, g2 = (c * u1 - b * u2) / det, (a * u2 - b * u1) / det
        d1, d2 = (e1 * w).sum(1), (e2 * w).sum(1)
        f1, f2 = (c * d1 - b * d2) / det, (a * d2 - b * d1) / det
        height2 = (w * w).sum(1) - (f1 * d1 + f2 * d2)
        gg = g1 * u1 + g2 * u2
        k = torch.sqrt(torch.clamp(height2, min=0)) / torch.sqrt(torch.where(gg < 1, 1 - gg, torch.ones_like(gg)))
        l1, l2 = f1 - k * g1, f2 - k * g2
        y = l1[:, None] * e1 + l2[:, None] * e2 - w
        ok = (gg < 1) & (l1 >= 0) & (l2 >= 0) & (l1 + l2 <= 1)
        best = torch.where(ok, torch.minimum(best, T[2] + l1 * u1 + l2 * u2 + y.norm(dim=1)), best)
    return best


def _eikonal_exact(case, seed):
    torch, dev = _torch()
    xyz, el = _mesh(case["dim"], case["n"], case["part"] == "graph")
    seeds, values = _seeds(case, len(xyz), np.random.default_rng(seed))
    X = torch.from_numpy(xyz.astype(np.float64)).to(dev)
    E = torch.from_numpy(el.astype(np.int64)).to(dev)
    sd = torch.from_numpy(seeds.astype(np.int64)).to(dev)
    sv = torch.from_numpy(values.astype(np.float64)).to(dev)
    far = 1e9
    T = torch.full((len(xyz),), far, dtype=torch.float64, device=dev)
    T[sd] = sv
    d1 = E.shape[1]
    for _ in range(100000):
        new = T.clone()
        live = (T[E] < far).any(1)
        L = E[live]
        for k in range(d1):
            face = [j for j in range(d1) if j != k]
            r = _local(torch, [X[L[:, j]] for j in face], [T[L[:, j]] for j in face], X[L[:, k]])
            new.scatter_reduce_(0, L[:, k], r, "amin")
        new[sd] = sv
        moved = float((T - new).max())
        T = new
        if moved < 1e-13:
            break
    return T.cpu().numpy()


def _mlp_split(w):
    f = 128
    W = [w[i * f * f:(i + 1) * f * f].reshape(f, f) for i in range(3)]
    o = 3 * f * f
    return W, [w[o + i * f:o + (i + 1) * f] for i in range(3)], w[o + 3 * f:o + 4 * f], w[o + 4 * f]


def _mlp_forward(w, x):
    W, b, w4, b4 = _mlp_split(w)
    acts = [x]
    for i in range(3):
        acts.append(np.maximum(acts[-1] @ W[i].T + b[i], 0.0))
    return acts, acts[-1] @ w4 + b4


def _train_exact(case, seed):
    rng = np.random.default_rng(seed)
    w = _weights(rng).astype(np.float64)
    x, t = (a.astype(np.float64) for a in _samples(case["n"], rng))
    m1, m2 = np.zeros_like(w), np.zeros_like(w)
    step, losses = 0, []
    for _ in range(case["epochs"]):
        losses = []
        for s in range(0, case["n"], case["batch"]):
            xb, tb = x[s:s + case["batch"]], t[s:s + case["batch"]]
            acts, y = _mlp_forward(w, xb)
            W, _, w4, _ = _mlp_split(w)
            e = y - tb
            losses.append(0.5 * float(np.mean(e * e)))
            dy = e / len(tb)
            gW, gb = [None] * 3, [None] * 3
            d = dy[:, None] * w4[None, :] * (acts[3] > 0)
            for i in (2, 1, 0):
                gW[i], gb[i] = d.T @ acts[i], d.sum(0)
                if i:
                    d = (d @ W[i]) * (acts[i] > 0)
            g = np.concatenate([a.ravel() for a in gW] + gb + [acts[3].T @ dy, [dy.sum()]])
            step += 1
            m1 = 0.9 * m1 + 0.1 * g
            m2 = 0.999 * m2 + 0.001 * g * g
            w = w - 1e-3 * (m1 / (1 - 0.9 ** step)) / (np.sqrt(m2 / (1 - 0.999 ** step)) + 1e-8)
    return {"params": w, "loss": float(np.mean(losses))}


def exact(case, seed):
    kind = case["kind"]
    if kind == "eikonal":
        return _eikonal_exact(case, seed)
    if kind == "predict":
        rng = np.random.default_rng(seed)
        w = _weights(rng).astype(np.float64)
        return _mlp_forward(w, _samples(case["n"], rng)[0].astype(np.float64))[1]
    if kind == "train":
        return _train_exact(case, seed)
    # time steps: where the redistance stops (the sentinel beyond the last
    # patch that the front reaches) is the patch schedule's, not arithmetic's
    return None
