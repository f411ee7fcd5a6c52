"""The work this framework is used for, as measurable cases over its public entry points.

Families (``kind``):

* ``force``      one force evaluation on device tensors by an order-p FMM handle (update_tree_device +
                 solve_device, or the captured step): the inner call of every N-body and t-SNE driver.
* ``reference``  the same two calls on a handle of the reference's expansion order (the class's defaults),
                 symmetric or non-symmetric, FP32 or FP64.
* ``dropin``     updateTree + solveNbody on host ``Points``, the reference's own interface.
* ``leapfrog``   N-body time steps with energy and momentum read back.
* ``tsne``       t-SNE iterations of one embedding, then the embedding read back for display.
* ``batch``      one lockstep iteration of several embeddings in CUDA graphs, embeddings read back.
* ``bh``         the Barnes-Hut solver (monopole, or with quadrupoles) on host arrays.
* ``pm``         the particle-mesh t-SNE repulsion on host arrays.
* ``affinity``   the t-SNE affinity matrix from input points (exact kNN, perplexities, symmetric CSR).

FP32 handles write forces of FP32 accuracy into FP64 words; where the caller of such a handle keeps forces,
energies or embeddings, it keeps them as FP32 (what an FP32 integrator or a vertex buffer takes).
"""
import ctypes
import math

import numpy as np
import torch

from masterthesislucas_gb300 import (NBodySolverFMM_MORTON, NBodySolverFMM_SYM_MORTON, Points, affinity, get_depth)
from masterthesislucas_gb300._lib import check, lib, ptr
from masterthesislucas_gb300.nbody import LeapfrogNBody
from masterthesislucas_gb300.solver import barnes_hut, particle_mesh
from masterthesislucas_gb300.tsne import TSNE, TSNEBatch

EPS = 1e-3    # gravity softening of every configuration here
NEIGH = 90    # 3 x perplexity 30


def listed():
    return [
        # the smallest embedding of the batched t-SNE range: launches and round trips are all of it
        dict(name="force_embedding_2k", kind="force", n=2000, kernel="tsne", order=8, leaf=16, deeper=0, theta=0.5,
             mac="cell", p2p=0, captured=False),
        # a middle-sized clustered gravity system at a low order
        dict(name="force_mixture_65k", kind="force", n=65537, kernel="gravity", order=4, leaf=64, deeper=0, theta=0.5,
             mac="cell", p2p=0, captured=False),
        # the fixed order-12 configuration of the two-disk system, plain calls
        dict(name="force_disks_1m", kind="force", n=1048576, kernel="gravity", order=12, leaf=64, deeper=2,
             theta=0.95, mac="bmax", p2p=64, captured=False),
        # the benchmark's force step: 4M two-disk particles, autotuned order 8, one captured graph per step
        dict(name="force_disks_4m", kind="force", n=4194304, kernel="gravity", order=8, leaf=64, deeper=2,
             theta=0.75, mac="bmax", p2p=64, captured=True),
        # the class's defaults (the reference's expansion) on a large odd-sized system
        dict(name="reference_200k", kind="reference", n=200003, kernel="gravity", leaf=64, theta=0.5,
             precision="fp32", variant="sym"),
        # a user of the reference's solver interface: host points in, sorted points and forces out
        dict(name="dropin_20k", kind="dropin", n=20011, kernel="tsne", leaf=16, theta=0.5),
        # an N-body run of ordinary size, energies logged every second step
        dict(name="leapfrog_200k", kind="leapfrog", n=200001, order=8, leaf=64, theta=1.0, steps=2),
        # the 70,000-point t-SNE benchmark, display refreshed every fifth iteration
        dict(name="tsne_70k", kind="tsne", n=70000, order=8, leaf=16, theta=0.5, iters=5),
        # many small uneven embeddings in lockstep
        dict(name="batch_16", kind="batch", systems=16, n_min=2000, n_max=30000, order=8, leaf=16, theta=0.5),
        # the plain Barnes-Hut benchmark
        dict(name="bh_mixture_65k", kind="bh", n=65536, kernel="gravity", leaf=16, theta=0.5, multipole=False),
        # the particle-mesh benchmark at the reference's settings (4 nodes, cells of 1, at least 4 cells)
        dict(name="pm_embedding_70k", kind="pm", n=70000, scale=25.0, cell=1.0),
        # affinities of image-like inputs (8-bit pixels, 784 of them)
        dict(name="affinity_20k", kind="affinity", n=20000, dim=784, clusters=10),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["force", "force", "force", "reference", "dropin", "leapfrog", "tsne", "batch", "bh", "pm",
                       "affinity"])
    kernel = rng.choice(["tsne", "gravity"])
    leaf = 16 if kernel == "tsne" else 64
    if kind == "force":
        mac = rng.choice(["cell", "bmax"])
        return dict(kind=kind, n=size(2000, 2000000), kernel=kernel, order=rng.choice([4, 6, 8, 10, 12]), leaf=leaf,
                    deeper=rng.choice([0, 1, 2]), theta=round(rng.uniform(0.5, 0.95 if mac == "bmax" else 1.0), 2),
                    mac=mac, p2p=rng.choice([0, 64]), captured=rng.random() < 0.3)
    if kind == "reference":
        precision = rng.choice(["fp32", "fp32", "fp64"])
        return dict(kind=kind, n=size(2000, 200000 if precision == "fp32" else 30000), kernel=kernel, leaf=leaf,
                    theta=round(rng.uniform(0.4, 0.8), 2), precision=precision, variant=rng.choice(["sym", "morton"]))
    if kind == "dropin":
        return dict(kind=kind, n=size(1000, 200000), kernel=kernel, leaf=leaf, theta=round(rng.uniform(0.4, 0.8), 2))
    if kind == "leapfrog":
        return dict(kind=kind, n=size(5000, 1000000), order=rng.choice([4, 8, 12]), leaf=64,
                    theta=round(rng.uniform(0.6, 1.0), 2), steps=rng.choice([1, 2, 4]))
    if kind == "tsne":
        return dict(kind=kind, n=size(2000, 100000), order=rng.choice([0, 4, 8, 8]), leaf=16,
                    theta=round(rng.uniform(0.4, 0.8), 2), iters=rng.choice([1, 5, 10]))
    if kind == "batch":
        return dict(kind=kind, systems=rng.randint(4, 16), n_min=2000, n_max=size(4000, 30000),
                    order=rng.choice([4, 8, 12]), leaf=16, theta=0.5)
    if kind == "bh":
        return dict(kind=kind, n=size(2000, 65536), kernel=kernel, leaf=rng.choice([8, 16, 32]),
                    theta=round(rng.uniform(0.4, 0.8), 2), multipole=rng.random() < 0.5)
    if kind == "pm":
        return dict(kind=kind, n=size(2000, 200000), scale=round(rng.uniform(5.0, 30.0), 1),
                    cell=rng.choice([1.0, 1.0, 2.0]))
    return dict(kind=kind, n=size(2000, 20000), dim=size(32, 784), clusters=rng.randint(5, 20))


# ---------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64)


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float64)


def _mixture(g, n, k, scale=1.0):
    """Equal-weight 2D Gaussian clusters: centres in [-1, 1]^2, sigmas in [0.02, 0.2]."""
    centres = 2.0 * _rand(g, k, 2) - 1.0
    sigmas = 0.02 + 0.18 * _rand(g, k)
    lab = torch.randint(0, k, (n,), generator=g, device="cuda")
    return scale * (centres[lab] + _randn(g, n, 2) * sigmas[lab, None])


def _disks(g, n):
    """Two exponential disks (scale lengths 0.1 and 0.05, centres 0.6 apart) and their owners."""
    own = torch.arange(n, device="cuda") >= n // 2
    r = -torch.log((1.0 - _rand(g, n)) * (1.0 - _rand(g, n))) * torch.where(own, 0.05, 0.1).double()
    phi = 2.0 * math.pi * _rand(g, n)
    cx = torch.where(own, 0.3, -0.3).double()
    return torch.stack([cx + r * torch.cos(phi), r * torch.sin(phi)], 1), cx, r


def _positions(case, seed):
    g = _gen(seed)
    if case["kernel"] == "tsne":
        return _mixture(g, case["n"], 10, 20.0)  # a developed embedding of ten clusters
    if case["kind"] == "bh" or case.get("order") == 4:
        return _mixture(g, case["n"], 8)
    return _disks(g, case["n"])[0]


def _embedding(seed, n):
    """A developed embedding of ten clusters and a symmetric affinity matrix over its clusters, about 2 x NEIGH
    entries a row as the symmetrised kNN graph has, as CSR."""
    g = _gen(seed)
    k = 10
    size = n // k
    # point i belongs to cluster i mod k; its neighbours are random members of that cluster
    i = torch.arange(n, device="cuda")
    j = torch.randint(0, size, (n, NEIGH), generator=g, device="cuda") * k + (i % k)[:, None]
    w = torch.exp(-3.0 * _rand(g, n, NEIGH))
    w /= w.sum(1, keepdim=True)
    row = i[:, None].expand(n, NEIGH).reshape(-1)
    col = j.reshape(-1)
    keep = row != col
    row, col, w = row[keep], col[keep], w.reshape(-1)[keep] / (2.0 * n)
    key = torch.cat([row * n + col, col * n + row])
    key, order = torch.sort(key)
    val = torch.cat([w, w])[order]
    key, inv = torch.unique_consecutive(key, return_inverse=True)
    val = torch.zeros(key.numel(), dtype=torch.float64, device="cuda").scatter_add_(0, inv, val)
    rows = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    rows[1:] = torch.cumsum(torch.bincount(key // n, minlength=n), 0)
    centres = 2.0 * _rand(g, k, 2) - 1.0
    sigmas = 0.02 + 0.18 * _rand(g, k)
    y = 20.0 * (centres[i % k] + _randn(g, n, 2) * sigmas[i % k, None])
    return rows, key % n, val, y


def _batch_sizes(case):
    """Sizes spread over the logarithm of the range, in no order."""
    k = case["systems"]
    lo, hi = math.log(case["n_min"]), math.log(case["n_max"])
    return [int(math.exp(lo + (hi - lo) * ((7 * i + 3) % k + 0.5) / k)) for i in range(k)]


def _tsne(case, seed, n, **kw):
    rows, col, val, y = _embedding(seed, n)
    return TSNE(rows.cpu().numpy(), col.cpu().numpy(), val.cpu().numpy(), y.cpu().numpy(), min_theta=case["theta"],
                max_theta=case["theta"], max_children=case["leaf"], order=case["order"], **kw)


def _velocities(pos, cx, r):
    """Rotation about each disk's centre at the speed its enclosed mass gives."""
    s = torch.where(cx > 0, 0.05, 0.1).double()
    inside = 0.5 * (1.0 - (1.0 + r / s) * torch.exp(-r / s))
    v = torch.sqrt(inside * r * r / (r * r + EPS * EPS) ** 1.5) / torch.clamp(r, min=1e-12)
    return torch.stack([-v * pos[:, 1], v * (pos[:, 0] - cx)], 1)


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case)
    if kind in ("force", "reference"):
        n = case["n"]
        pos = _positions(case, seed)
        s["stream"] = torch.cuda.Stream()
        kw = dict(max_children=case["leaf"], theta=case["theta"], softening=EPS, stream=s["stream"].cuda_stream)
        if kind == "force":
            depth = get_depth(case["leaf"], n) + case["deeper"]
            solver = NBodySolverFMM_SYM_MORTON(case["kernel"], tree_depth=depth, order=case["order"],
                                               mac=case["mac"], leaf_p2p=case["p2p"], **kw)
        else:
            cls = NBodySolverFMM_SYM_MORTON if case["variant"] == "sym" else NBodySolverFMM_MORTON
            solver = cls(case["kernel"], precision=case["precision"], **kw)
        # forces and the pair sum side by side, so that one conversion hands both on
        buf = torch.zeros(2 * n + 1, dtype=torch.float64, device="cuda")
        s.update(pos=pos, solver=solver, buf=buf, grad=buf[:2 * n].view(n, 2), total=buf[2 * n:])
        if case.get("precision") != "fp64":
            s["out"] = torch.empty(2 * n + 1, dtype=torch.float32, device="cuda")
        if case.get("captured"):
            torch.cuda.synchronize()
            solver.update_tree_device(pos)
            solver.capture_step(pos, s["grad"], s["total"])
    elif kind == "dropin":
        pos = _positions(case, seed).cpu().numpy()
        s["points"] = Points.from_positions(pos)
        s["box"] = pos.min(0), pos.max(0)
        s["solver"] = NBodySolverFMM_SYM_MORTON(case["kernel"], max_children=case["leaf"], theta=case["theta"],
                                                softening=EPS)
        s["forces"] = np.empty((case["n"], 2), np.float32)
    elif kind == "leapfrog":
        pos, cx, r = _disks(_gen(seed), case["n"])
        s["sim"] = LeapfrogNBody(pos.cpu().numpy(), _velocities(pos, cx, r).cpu().numpy(), dt=1e-4, softening=EPS,
                                 max_children=case["leaf"], theta=case["theta"], order=case["order"])
    elif kind == "tsne":
        # late iterations with short steps: the embedding keeps its shape however often it is stepped
        s["system"] = _tsne(case, seed, case["n"], learn_rate=1.0)
        s["system"].iteration_counter = 300
    elif kind == "batch":
        systems = [_tsne(case, seed * 1000 + k, n) for k, n in enumerate(_batch_sizes(case))]
        for t in systems:
            t.iteration_counter = 300
        s["batch"] = TSNEBatch(systems)
        for _ in range(2):  # the first iteration sizes the buffers, the second captures the graphs
            s["batch"].time_step()
    elif kind == "bh":
        s["pos"] = _positions(case, seed).cpu().numpy()
    elif kind == "pm":
        s["pos"] = _mixture(_gen(seed), case["n"], 10, case["scale"]).cpu().numpy()
    else:
        n = case["n"]
        s["x"] = _pixels(case, seed)
        s["rows"] = torch.zeros(n + 1, dtype=torch.int32, device="cuda")
        s["col"] = torch.zeros(2 * n * NEIGH, dtype=torch.int32, device="cuda")
        s["val"] = torch.zeros(2 * n * NEIGH, dtype=torch.float64, device="cuda")
    return s


def _pixels(case, seed):
    """Clustered inputs clipped to [0, 1] in steps of 1/256, as 8-bit images are."""
    g = _gen(seed)
    centres = 0.2 + 0.6 * _rand(g, case["clusters"], case["dim"])
    lab = torch.randint(0, case["clusters"], (case["n"],), generator=g, device="cuda")
    x = centres[lab] + 0.15 * _randn(g, case["n"], case["dim"])
    return (torch.round(x.clamp(0.0, 1.0) * 256.0) / 256.0).float()


# ---------------------------------------------------------------- one pass
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("force", "reference"):
        solver, n2 = state["solver"], 2 * case["n"]
        if case.get("captured"):
            solver.launch_step()
        else:
            with torch.cuda.stream(state["stream"]):
                state["total"].zero_()
            solver.update_tree_device(state["pos"])
            solver.solve_device(state["grad"], state["total"])
        if "out" not in state:
            return state["grad"], state["total"]
        with torch.cuda.stream(state["stream"]):
            state["out"].copy_(state["buf"])
        return state["out"][:n2], state["out"][n2:]
    if kind == "dropin":
        pts, solver = state["points"], state["solver"]
        pts.derivative[...] = 0.0
        solver.updateTree(pts, *state["box"])
        z = solver.solveNbody(0.0, pts)
        state["forces"][pts.ID] = pts.derivative  # back to the callers' order, as the t-SNE driver does
        return state["forces"], z, pts.ID
    if kind == "leapfrog":
        sim = state["sim"]
        sim.step(case["steps"])
        d = sim.diagnostics()
        return sim.x, sim.v, d["kinetic"], d["potential"]
    if kind == "tsne":
        t = state["system"]
        for _ in range(case["iters"]):
            t.time_step()
        y, _, g = t.embedding()
        return y.astype(np.float32), g.astype(np.float32)
    if kind == "batch":
        b = state["batch"]
        b.time_step()
        return [t.embedding()[0].astype(np.float32) for t in b.systems]
    if kind == "bh":
        g, z = barnes_hut(state["pos"], kernel=case["kernel"], softening=EPS, max_children=case["leaf"],
                          theta=case["theta"], multipole=case["multipole"])
        return g.astype(np.float32), z
    if kind == "pm":
        return particle_mesh(state["pos"], n_interp=4, cell_size=case["cell"], min_intervals=4)
    d, i = affinity.knn(state["x"], NEIGH)
    p = affinity.perplexity_rows(d, 30.0)
    # the matrix stays on the device, in buffers of its largest size
    rows, col, val, nnz = state["rows"], state["col"], state["val"], ctypes.c_int64(0)
    check(lib().tc_symmetrize_device(ptr(i), ptr(p), case["n"], NEIGH, ptr(rows), ptr(col), ptr(val),
                                     ctypes.byref(nnz), None))
    return d, i, p, rows, col, val, nnz.value


# ---------------------------------------------------------------- what a pass cannot do without
def work(case):
    """Positions (16 bytes a particle) in and forces (16) out; an FMM force of these accuracies takes some 500
    particle pairs of 20 flops a particle, Barnes-Hut as much."""
    kind, n = case["kind"], case.get("n", 0)
    if kind in ("force", "reference", "dropin", "bh"):
        return dict(bytes=32 * n, flops=1e4 * n)
    if kind == "leapfrog":
        return dict(bytes=case["steps"] * 64 * n, flops=case["steps"] * 1e4 * n)
    if kind in ("tsne", "batch"):
        if kind == "batch":  # the mean of the log-uniform sizes
            n = case["systems"] * (case["n_max"] - case["n_min"]) / math.log(case["n_max"] / case["n_min"])
        it = case.get("iters", 1)
        return dict(bytes=it * n * (2 * NEIGH * 8 + 64), flops=it * n * (1e4 + 2 * NEIGH * 12))
    if kind == "pm":
        nf = 8.0 * 2.6 * case["scale"] / case["cell"]  # the padded grid of 4 nodes a cell
        return dict(bytes=32 * n + 9 * 8 * nf * nf, flops=9 * 2.5 * nf * nf * 2 * math.log2(nf) + 400 * n)
    return dict(bytes=4 * n * case["dim"] + 2 * NEIGH * 12 * n, flops=1.5 * n * n * case["dim"])


# ---------------------------------------------------------------- the same in 64 bits
def _direct(kernel, p):
    """The force on every point and the pair sum, by the direct sum over all others."""
    n = p.shape[0]
    f = torch.empty_like(p)
    z = 0.0
    rows = max(1, (1 << 27) // n)
    c = 1.0 if kernel == "tsne" else EPS * EPS
    for r in range(0, n, rows):
        q = p[r:r + rows]
        dx = q[:, None, 0] - p[None, :, 0]
        dy = q[:, None, 1] - p[None, :, 1]
        u = dx * dx
        u.addcmul_(dy, dy).add_(c)
        u = u.reciprocal_() if kernel == "tsne" else u.rsqrt_()
        z += float(u.sum())
        w = u.square() if kernel == "tsne" else u.pow_(3).neg_()
        f[r:r + rows, 0] = (w * dx).sum(1)
        f[r:r + rows, 1] = (w * dy).sum(1)
    return (f, z - n) if kernel == "tsne" else (f, n / EPS - z)


def _tsne_steps(rows, col, val, y, iters, lr):
    n = y.shape[0]
    row = torch.repeat_interleave(torch.arange(n, device="cuda"), rows[1:] - rows[:-1])
    prev = y.clone()
    for _ in range(iters):
        rep, z = _direct("tsne", y)
        d = y[col] - y[row]
        w = (val / (1.0 + (d * d).sum(1)))[:, None] * d
        att = torch.zeros_like(y).index_add_(0, row, w)
        g = 4.0 / z * rep + 4.0 * att  # late iterations: no exaggeration, momentum 0.8
        y, prev = y + lr * g + 0.8 * (y - prev), y
    return y, g


def _affinity(x):
    """Exact neighbours (ties by index), perplexities and symmetrisation. Distances of 8-bit pixels are sums of
    multiples of 2^-16, exact in 32 bits too, so the neighbours are the same in any precision."""
    n = x.shape[0]
    x = x.double()
    sq = (x * x).sum(1)
    d = torch.empty(n, NEIGH, dtype=torch.float64, device="cuda")
    j = torch.empty(n, NEIGH, dtype=torch.int64, device="cuda")
    cols = torch.arange(n, device="cuda")
    for r in range(0, n, 2048):
        q = x[r:r + 2048]
        k = torch.round((sq[r:r + 2048, None] + sq[None, :] - 2.0 * (q @ x.T)) * 65536.0).to(torch.int64)
        k = k * n + cols[None, :]
        k[torch.arange(len(q), device="cuda"), cols[r:r + 2048]] = 1 << 62
        k = torch.topk(k, NEIGH, dim=1, largest=False, sorted=True).values
        d[r:r + 2048] = (k // n).double() / 65536.0
        j[r:r + 2048] = k % n
    dist, d = d, d - d[:, :1]
    beta, lo, hi = torch.ones(n, 1, dtype=torch.float64, device="cuda"), 0.0 * d[:, :1], d[:, :1] + math.inf
    live = torch.ones(n, 1, dtype=torch.bool, device="cuda")
    for _ in range(100):
        w = torch.exp(-d * beta)
        s = w.sum(1, keepdim=True)
        diff = torch.log(s) + beta * (d * w).sum(1, keepdim=True) / s - math.log(30.0)
        live = live & (diff.abs() >= 1e-5)
        up = diff > 0
        lo, hi = torch.where(live & up, beta, lo), torch.where(live & ~up, beta, hi)
        beta = torch.where(live, torch.where(torch.isinf(hi), beta * 2.0, 0.5 * (lo + hi)), beta)
    w = torch.exp(-d * beta)
    rows_p = w / w.sum(1, keepdim=True)
    p = (rows_p / (2.0 * n)).reshape(-1)
    row = cols[:, None].expand(n, NEIGH).reshape(-1)
    key, order = torch.sort(torch.cat([row * n + j.reshape(-1), j.reshape(-1) * n + row]))
    p = torch.cat([p, p])[order]
    key, inv = torch.unique_consecutive(key, return_inverse=True)
    val = torch.zeros(2 * n * NEIGH, dtype=torch.float64, device="cuda").scatter_add_(0, inv, p)
    return dist, None, rows_p, None, None, val, None


def exact(case, seed):
    kind = case["kind"]
    if kind in ("force", "reference", "dropin", "bh"):
        if case["n"] > 250000:
            return None
        f, z = _direct(case["kernel"], _positions(case, seed))
        if kind in ("force", "reference"):
            z = torch.tensor([z], dtype=torch.float64)
            return (f.reshape(-1) if case.get("precision") != "fp64" else f), z
        return (f, z, None) if kind == "dropin" else (f, z)
    if kind == "pm":
        return _direct("tsne", _mixture(_gen(seed), case["n"], 10, case["scale"]))
    if kind == "leapfrog":
        if case["n"] * case["steps"] > 500000:
            return None
        x, cx, r = _disks(_gen(seed), case["n"])
        v, m, dt = _velocities(x, cx, r), 1.0 / case["n"], 1e-4
        a, z = _direct("gravity", x)
        for _ in range(case["steps"]):
            v = v + 0.5 * dt * m * a
            x = x + dt * v
            a, z = _direct("gravity", x)
            v = v + 0.5 * dt * m * a
        return x, v, 0.5 * m * float((v * v).sum()), 0.5 * m * m * z
    if kind == "tsne":
        if case["n"] * case["iters"] > 500000:
            return None
        return _tsne_steps(*_embedding(seed, case["n"]), case["iters"], 1.0)
    if kind == "batch":
        # two iterations in prepare, one in the pass
        return [_tsne_steps(*_embedding(seed * 1000 + k, n), 3, n / 15.0)[0]
                for k, n in enumerate(_batch_sizes(case))]
    return _affinity(_pixels(case, seed))
