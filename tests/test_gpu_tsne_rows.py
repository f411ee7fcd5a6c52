"""The attraction's rows (a block takes 32, a lane up to four entries at a time) against the oracle's step.

Numbers of points around whole blocks of rows; rows of no entry, of one, around 32 and 128, and of hundreds.
"""
import numpy as np
import pytest

import oracle
from masterthesislucas_gb300.tsne import TSNE

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 31, 33, 641])
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_rows_of_every_length(n, precision):
    rng = np.random.default_rng(n)
    y = rng.normal(0, 3, (n, 2))
    lengths = np.resize([0, 1, 31, 32, 33, 127, 128, 129, 200, 500], n)
    row_ptr = np.concatenate([[0], np.cumsum(lengths)]).astype(np.uint32)
    col = rng.integers(0, n, row_ptr[-1]).astype(np.uint32)
    val = rng.random(len(col)) / max(len(col), 1)
    t = TSNE(row_ptr, col, val, y, min_theta=0.5, max_theta=0.5, max_children=16, precision=precision)
    t.time_step()
    got, _, grad = t.embedding()
    yn, gref, _ = oracle.tsne_step(y, y, row_ptr, col, val, theta=0.5)  # early iterations: factor 16, momentum 0.5
    # FP32: the reference-order forces agree to 1e-5 of the largest, the attraction's sums of 500 terms to 500 2^-24
    tol = 5e-5 if precision == "fp32" else 1e-10
    assert np.abs(grad - gref).max() <= tol * np.abs(gref).max()
    assert np.abs(got - yn).max() <= tol * (np.abs(gref).max() * n / 15.0 + np.abs(y).max())
