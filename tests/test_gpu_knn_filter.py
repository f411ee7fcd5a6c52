"""The kNN with its tensor-core candidate filter against the oracle, bit for bit.

Sizes around the filter's smallest, its tiles (128 x 256) and its K steps and stages (16, 64), one that takes two
chunks of the approximate distances; inputs that are BF16 numbers and that are not; and inputs that the filter gives
up on, all of their rows or some: many equal points, distances small against the norms, tiny, huge and non-finite
values.
"""
import numpy as np
import pytest

import oracle
from masterthesislucas_gb300 import affinity

pytestmark = pytest.mark.gpu


def check(x, k):
    import torch
    d, i = affinity.knn(torch.from_numpy(x).cuda(), k)
    rd, ri = oracle.knn(x, k)
    np.testing.assert_array_equal(i.cpu().numpy(), ri)
    np.testing.assert_array_equal(d.cpu().numpy(), rd)


@pytest.mark.parametrize("n,dim,k", [(1024, 1, 1), (1025, 15, 90), (1151, 16, 128), (1153, 17, 90), (1279, 63, 2),
                                     (1281, 64, 90), (1536, 65, 90), (2049, 100, 127), (3000, 784, 90),
                                     (9001, 8, 90)])
@pytest.mark.parametrize("values", ["pixels", "normal"])
def test_sizes(n, dim, k, values):
    rng = np.random.default_rng(n + dim)
    centres = rng.random((7, dim))
    x = centres[rng.integers(0, 7, n)] + 0.15 * rng.normal(size=(n, dim))
    if values == "pixels":
        x = np.round(np.clip(x, 0, 1) * 256) / 256
    check(x.astype(np.float32), k)


@pytest.mark.parametrize("n", [1024 + 1, 1024 + 31, 1024 + 33, 1024 + 97, 2048 + 127])
def test_last_rows_within_a_warp(n):
    """The last row block ends inside a warp's 32 rows, several column tiles each."""
    rng = np.random.default_rng(n)
    check(rng.normal(size=(n, 40)).astype(np.float32), 30)


@pytest.mark.parametrize("kind", ["equal", "some_equal", "offset", "tiny", "huge", "outlier", "infinite"])
def test_rows_that_the_filter_gives_up_on(kind):
    rng = np.random.default_rng(5)
    x = rng.normal(size=(2000, 24)).astype(np.float32)
    if kind == "equal":
        x[:] = x[rng.integers(0, 3, 2000)]
    elif kind == "some_equal":
        x[100:700] = x[100]
    elif kind == "offset":
        x += 1000.0
    elif kind == "tiny":
        x *= np.float32(1e-24)
    elif kind == "huge":
        x *= np.float32(1e17)
    elif kind == "outlier":
        x[77] *= np.float32(1e6)
    else:
        x[77, 3] = np.inf
    check(x, 90)
