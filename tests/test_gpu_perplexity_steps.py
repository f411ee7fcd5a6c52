"""k_perplexity, whose bisection steps FP32 decides where it can, against the oracle's all-FP64 rows, bit for bit.

Short rows, the longest rows of the FP32 screen and longer ones, perplexities that no bandwidth reaches, equal
distances, distances near both ends of the FP32 range, and rows that do not start with their smallest.
"""
import numpy as np
import pytest

import oracle
from masterthesislucas_gb300 import affinity

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 2, 31, 90, 128, 129, 300])
@pytest.mark.parametrize("scale", [1.0, 1e-30, 1e-42, 1e30, "equal", "wide", "unordered"])
@pytest.mark.parametrize("perplexity", [1.5, 30.0])
def test_rows_match_the_oracle(k, scale, perplexity):
    import torch
    rng = np.random.default_rng(k)
    d = np.sort(rng.gamma(8.0, 1.0, (193, k)), axis=1)
    if scale == "equal":
        d[:] = d[:, :1]
    elif scale == "wide":
        d = np.sort(10.0 ** rng.uniform(-35, 35, (193, k)), axis=1)
    elif scale == "unordered":
        d = d[:, ::-1].copy()
    else:
        d *= scale
    d = d.astype(np.float32)
    p = affinity.perplexity_rows(torch.from_numpy(d).cuda(), perplexity)
    np.testing.assert_array_equal(p.cpu().numpy(), oracle.perplexity_rows(d, perplexity))
