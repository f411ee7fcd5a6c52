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


@pytest.mark.parametrize("offset", [0.0] + [2.0 ** e + 0.4 * 2.0 ** (e - 23) for e in (20, 30, 40)])
def test_attraction_far_from_the_origin(offset):
    """FP32 products of differences that are as good as the FP64 positions', wherever the embedding lies."""
    rng = np.random.default_rng(7)
    n = 300
    y = offset + rng.normal(0, 1, (n, 2))
    lengths = np.resize([0, 1, 2, 90, 200], n)
    row_ptr = np.concatenate([[0], np.cumsum(lengths)]).astype(np.uint32)
    rows, col = np.repeat(np.arange(n), lengths), rng.integers(0, n, row_ptr[-1]).astype(np.uint32)
    val = 1e6 * rng.random(len(col)) / len(col)  # an attraction far above the repulsion
    t = TSNE(row_ptr, col, val, y, min_theta=0.5, max_theta=0.5, max_children=16)
    t.time_step()
    _, _, grad = t.embedding()
    _, gref, _ = oracle.tsne_step(y, y, row_ptr, col, val, theta=0.5)
    d = y[col] - y[rows]
    w = 16.0 * val / (1.0 + (d * d).sum(1))
    attr, size = np.zeros((n, 2)), np.zeros((n, 2))
    np.add.at(attr, rows, w[:, None] * d)
    np.add.at(size, rows, w[:, None] * np.abs(d).max(1)[:, None])
    # a term is off by at most 12 roundings of 2^-24 (differences, square, reciprocal to two ulps, products), a sum of
    # 200 terms by 7 in a lane and 5 across; the repulsion (positions and cells rounded at the offset) by a tenth
    assert np.all(np.abs(grad - gref) <= 24 * 2.0 ** -24 * size + 0.1 * np.abs(gref - attr).max())
