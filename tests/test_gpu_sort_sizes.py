"""The Morton sort's permutation against the oracle's stable sort, where its kernels and tiles change: one block up to
4,096 keys, tiles of 2,048, one and many tiles to look back over, tiles with scanned counts; equal codes keep their input order."""
import numpy as np
import pytest

import oracle
from masterthesislucas_gb300 import NBodySolverFMM_SYM_MORTON, Points

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 31, 2047, 4095, 4096, 4097, 6143, 6145, 100003, 1 << 20, (1 << 20) + 1])
@pytest.mark.parametrize("ties", [False, True])
def test_permutation(n, ties):
    rng = np.random.default_rng(n)
    pos = rng.integers(0, 40, (n, 2)) / 40.0 if ties else rng.normal(size=(n, 2))
    mn, mx = np.full(2, pos.min() - 1.0), np.full(2, pos.max() + 1.0)
    codes = oracle.morton_codes(pos, mn, mx)
    s = NBodySolverFMM_SYM_MORTON("tsne", tree_depth=3, theta=0.9, order=4)
    pts = Points.from_positions(pos)
    s.updateTree(pts, mn, mx)
    np.testing.assert_array_equal(pts.ID, oracle.sort_perm(codes))
