"""Barnes-Hut trees of every shape against the oracle, FP64: the sorted build, the level-by-level one, and the line between.

Few points and one (no split), leaves of one point (long chains of nodes), equal points within a leaf, the longest
leaves of the sorted build, inputs far from the origin, and clusters that need more levels than its keys hold.
"""
import numpy as np
import pytest

import oracle
from masterthesislucas_gb300 import datasets
from masterthesislucas_gb300.solver import barnes_hut

pytestmark = pytest.mark.gpu

EPS = 1e-3


def rel_err(a, b):
    return np.linalg.norm(a - b, axis=1) / np.maximum(np.linalg.norm(b, axis=1), 1e-300)


def points(shape, n, seed=3):
    rng = np.random.default_rng(seed)
    if shape == "uniform":
        return rng.random((n, 2))
    if shape == "mixture":
        return datasets.gaussian_mixture(n, seed=seed).astype(np.float64)
    if shape == "equal":  # every point eight times
        return np.repeat(rng.normal(size=((n + 7) // 8, 2)), 8, axis=0)[:n][rng.permutation(n)]
    if shape == "far":
        return 1.0e5 + 20.0 * rng.normal(size=(n, 2))
    pos = rng.normal(size=(n, 2))  # deep: a tenth of the points within 1e-7 of one place
    pos[: n // 10] = 0.3 + 1e-7 * rng.normal(size=(n // 10, 2))
    return pos


@pytest.mark.parametrize("multipole", [False, True])
@pytest.mark.parametrize("shape,n,leaf", [("uniform", 1, 16), ("uniform", 2, 1), ("uniform", 17, 16), ("uniform", 33, 1),
                                          ("mixture", 3001, 1), ("mixture", 4096, 16), ("mixture", 5003, 256),
                                          ("mixture", 5003, 257), ("equal", 2000, 8), ("far", 3000, 16),
                                          ("deep", 3000, 8)])
@pytest.mark.parametrize("kernel", ["tsne", "gravity"])
def test_tree_shapes(kernel, shape, n, leaf, multipole):
    pos = points(shape, n)
    k = oracle.KERNEL_TSNE if kernel == "tsne" else oracle.KERNEL_GRAVITY
    f = oracle.bhmp if multipole else oracle.bh
    ref, ref_total = f(pos, kernel=k, eps=EPS, max_children=leaf, theta=0.5)
    g, total = barnes_hut(pos, kernel=kernel, softening=EPS, max_children=leaf, theta=0.5, precision="fp64",
                          multipole=multipole)
    assert rel_err(g, ref).max() < 1e-11
    assert total == pytest.approx(ref_total, rel=1e-11)
    # FP32 on the same tree: single sums of up to n terms
    g32, total32 = barnes_hut(pos, kernel=kernel, softening=EPS, max_children=leaf, theta=0.5, multipole=multipole)
    err = rel_err(g32, ref)
    assert np.median(err) < 1e-5 and err.max() < 1e-3
    assert total32 == pytest.approx(ref_total, rel=1e-5)


@pytest.mark.parametrize("multipole", [False, True])
@pytest.mark.parametrize("kernel", ["gravity", "tsne"])
@pytest.mark.parametrize("shift", [10, 20, 30, 40])
def test_close_pairs_in_fp32(shift, kernel, multipole):
    """Points with a partner 2^-shift away: the FP32 forces of the FP64 offsets."""
    rng = np.random.default_rng(shift)
    a = rng.random((64, 2))
    pos = np.concatenate([a, a + 2.0 ** -shift * (1.0 + rng.random((64, 2)))])
    kw = dict(kernel=kernel, softening=0.0 if kernel == "gravity" else EPS, max_children=16, theta=0.5,
              multipole=multipole)
    ref, ref_total = barnes_hut(pos, precision="fp64", **kw)
    g, total = barnes_hut(pos, **kw)
    # sums of up to 128 terms; a term takes some 16 roundings of 2^-24 (offset, square, reciprocal root to two ulps and
    # its cube), an accepted node's quadrupole twice that
    d = pos[:, None, :] - pos[None, :, :]
    r2 = (d * d).sum(-1) + np.eye(len(pos)) * 1e300
    size = (np.sqrt(r2) * ((1.0 + r2) ** -2 if kernel == "tsne" else r2 ** -1.5)).sum(1)
    assert np.all(np.linalg.norm(g - ref, axis=1) <= (32 + 40) * 2.0 ** -24 * size)
    assert total == pytest.approx(ref_total, rel=2e-6)
