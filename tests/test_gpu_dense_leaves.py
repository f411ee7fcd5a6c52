"""Leaves of many particles beside small ones, where the leaf passes change the way they split the work.

* order p: leaves around the split line of the near field (512 particles) and around whole runs of its staged
  sources (2,048), and around the line above which a leaf's P2M takes a block;
* the reference's expansion order: leaves around a lane's, a warp's and a block's share of the moments, the P2L and
  the point stage.
"""
import numpy as np
import pytest

import oracle
from masterthesislucas_gb300 import NBodySolverFMM_MORTON, NBodySolverFMM_SYM_MORTON, Points

pytestmark = pytest.mark.gpu

EPS = 1e-3


def cells(sizes, depth, seed=0):
    """sizes[i] random points in cell i (row-major) of the 2^depth grid over [0, 1)^2, and the box."""
    rng = np.random.default_rng(seed)
    w = 1 << depth
    pts = [(np.array([i % w, i // w]) + 0.01 + 0.98 * rng.random((c, 2))) / w for i, c in enumerate(sizes) if c]
    return np.concatenate(pts), np.zeros(2), np.ones(2)


def rel_err(a, b):
    return np.linalg.norm(a - b, axis=1) / np.maximum(np.linalg.norm(b, axis=1), 1e-300)


@pytest.mark.parametrize("kernel", ["tsne", "gravity"])
@pytest.mark.parametrize("sizes", [(512, 0, 0, 1), (513, 7, 0, 33), (1023, 1, 512, 514), (2047, 0, 0, 0),
                                   (2048, 1, 0, 0), (4097, 513, 0, 2), (5000, 600, 545, 40)])
def test_order_p_near_field_of_dense_leaves(kernel, sizes):
    pos, mn, mx = cells(sizes, 1)
    pos *= 10.0
    s = NBodySolverFMM_SYM_MORTON(kernel, tree_depth=1, order=8, theta=0.1, softening=EPS)  # all pairs direct
    pts = Points.from_positions(pos)
    s.updateTree(pts, mn, 10.0 * mx)
    total = s.solveNbody(0.0, pts)
    k = oracle.KERNEL_TSNE if kernel == "tsne" else oracle.KERNEL_GRAVITY
    ref, ref_total = oracle.naive(pts.position, kernel=k, eps=EPS)
    # An FP32 sum of m terms is off by at most (longest chain) 2^-24 sum |f|: chains of 1,024 terms a run and one
    # term a run, and some 64 roundings of coordinates and of the kernel a term (cancellation in R included: cells
    # of 5, separations above 5e-6 of them enter with their full weight, so bound the term's error by its largest
    # derivative times 2^-22 of the cell as well)
    d = pts.position[:, None, :] - pts.position[None, :, :]
    r2 = (d * d).sum(-1)
    w = 1.0 / (1.0 + r2) ** 2 if kernel == "tsne" else (r2 + EPS * EPS) ** -1.5
    chain = (1024 + len(pos) / 2048 + 64) * 2.0 ** -24 * (w * np.sqrt(r2)).sum(1)
    shift = 5.0 * 2.0 ** -22 * 3.0 * w.sum(1)
    assert np.all(np.linalg.norm(pts.derivative - ref, axis=1) <= chain + shift)
    assert total == pytest.approx(ref_total, rel=1e-4 if kernel == "tsne" else 1e-3)


REF_SIZES = [0, 1, 7, 8, 9, 31, 32, 33, 63, 64, 65, 129, 300, 0, 2, 700]


@pytest.mark.parametrize("kernel", ["tsne", "gravity"])
@pytest.mark.parametrize("theta", [0.3, 1.0])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("symmetric", [True, False])
def test_reference_order_dense_leaves(kernel, theta, precision, symmetric):
    pos, mn, mx = cells(REF_SIZES, 2)
    k = oracle.KERNEL_TSNE if kernel == "tsne" else oracle.KERNEL_GRAVITY
    cls = NBodySolverFMM_SYM_MORTON if symmetric else NBodySolverFMM_MORTON
    s = cls(kernel, tree_depth=2, theta=theta, softening=EPS, precision=precision)
    pts = Points.from_positions(pos)
    s.updateTree(pts, mn, mx)
    total = s.solveNbody(0.0, pts)
    ref = oracle.sym_fmm(pos, kernel=k, eps=EPS, depth=2, theta=theta, mn=mn, mx=mx, symmetric=symmetric)
    np.testing.assert_array_equal(pts.ID, ref["ids"])
    nodes = s.tree_dump()["nodes"]  # ..., count at 5, centre of mass at 6, M0 at 8, M2 at 9
    np.testing.assert_array_equal(nodes[:, 5], ref["nodes"]["count"])
    np.testing.assert_array_equal(nodes[:, 6:8], ref["nodes"]["com"])
    np.testing.assert_array_equal(nodes[:, 9:13], ref["nodes"]["m2"])
    err = rel_err(pts.derivative, ref["grad"])
    if precision == "fp64":
        assert err.max() < 1e-10
        assert total == pytest.approx(ref["total"], rel=1e-10)
    else:
        assert np.median(err) <= 2e-6 and err.max() <= 1e-3
        assert total == pytest.approx(ref["total"], rel=2e-6)


@pytest.mark.parametrize("order", [None, 8])
@pytest.mark.parametrize("scale", [1.0, 1e12])
@pytest.mark.parametrize("sizes", [(1, 1, 1, 1), (3, 33, 0, 1)])
def test_pair_sum_in_any_units(order, scale, sizes):
    """Sources that fill up a group's share add nothing to the pair sum, also where every term is 1e-12."""
    pos, mn, mx = cells(sizes, 1)
    pos *= scale
    s = NBodySolverFMM_SYM_MORTON("gravity", tree_depth=1, theta=0.1, softening=0.1 * scale,
                                  **({} if order is None else {"order": order}))  # all pairs direct
    pts = Points.from_positions(pos)
    s.updateTree(pts, mn, mx * scale)
    total = s.solveNbody(0.0, pts)
    _, ref_total = oracle.naive(pts.position, kernel=oracle.KERNEL_GRAVITY, eps=0.1 * scale)
    # up to 38 terms a sink, each to 3 2^-23 (coordinates, square, reciprocal root), the sum to 38 2^-24; the order-p
    # path adds and takes out the sink's own term, up to ten times the others'
    assert total == pytest.approx(ref_total, rel=(3 * 2 + 38) * 10 * 2.0 ** -24, abs=0.0)


@pytest.mark.parametrize("symmetric", [True, False])
@pytest.mark.parametrize("theta", [0.4, 0.5, 0.7])
@pytest.mark.parametrize("scale", [1.0, 2.0 ** -61, 2.0 ** -62, 2.0 ** -63, 2.0 ** -75, 2.0 ** 61])
def test_point_criteria_at_any_scale(symmetric, theta, scale):
    """The points' criteria decide as in FP64 where their FP32 squares leave the normal range."""
    pos, mn, mx = cells(REF_SIZES, 2)
    cls = NBodySolverFMM_SYM_MORTON if symmetric else NBodySolverFMM_MORTON
    counts = []
    for p, c in (("fp64", 1.0), ("fp32", scale)):
        s = cls("tsne", tree_depth=2, theta=theta, precision=p)
        pts = Points.from_positions(pos * c)
        s.updateTree(pts, mn * c, mx * c)
        s.solveNbody(0.0, pts)
        counts.append(s.counters())
    assert counts[0] == counts[1]


@pytest.mark.parametrize("symmetric", [True, False])
@pytest.mark.parametrize("offset", [0.0, 2.0 ** 30 / 3, 2.0 ** 38 / 3, 2.0 ** 46 / 3])
def test_point_criteria_far_from_the_origin(symmetric, offset):
    """The points' criteria decide as in FP64 where the cells' centres are rounded by much of a cell."""
    pos, mn, mx = cells(REF_SIZES, 2)
    pos, mn, mx = pos + offset, mn + offset, mx + offset
    cls = NBodySolverFMM_SYM_MORTON if symmetric else NBodySolverFMM_MORTON
    counts = []
    for p in ("fp64", "fp32"):
        s = cls("tsne", tree_depth=2, theta=0.4, precision=p)
        pts = Points.from_positions(pos)
        s.updateTree(pts, mn - 0.0137, mx + 0.0171)
        s.solveNbody(0.0, pts)
        counts.append(s.counters())
    assert counts[0] == counts[1]
