"""k_knn's tiles and run boundaries against the oracle, bit for bit.

Sizes around a query block (64 rows) and a candidate tile (128), around one and several runs of units, dimensions
that end inside a staged chunk, rows off a 16-byte boundary, and list lengths up to the longest; one input has many
equal distances (ties go by index).
"""
import numpy as np
import pytest

import oracle
from masterthesislucas_gb300 import affinity

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,dim,k", [(2, 1, 1), (63, 3, 62), (65, 16, 64), (129, 17, 128), (257, 4, 90), (1000, 8, 90),
                                     (1700, 33, 31), (3001, 20, 128)])
@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("ties", [False, True])
def test_knn_matches_the_oracle(n, dim, k, offset, ties):
    import torch
    rng = np.random.default_rng(n + dim)
    x = rng.integers(0, 3, (n, dim)).astype(np.float32) if ties else rng.normal(size=(n, dim)).astype(np.float32)
    flat = torch.zeros(n * dim + offset, device="cuda")
    xd = flat[offset:].view(n, dim)  # off the boundary by one float when offset is 1
    xd.copy_(torch.from_numpy(x))
    d, i = affinity.knn(xd, k)
    rd, ri = oracle.knn(x, k)
    np.testing.assert_array_equal(d.cpu().numpy(), rd)
    np.testing.assert_array_equal(i.cpu().numpy(), ri)


def test_threads_of_different_k():
    """Calls of different list lengths from several threads at once, each on its own stream."""
    import threading

    import torch
    rng = np.random.default_rng(11)
    x = torch.from_numpy(rng.random((1500, 24)).astype(np.float32)).cuda()
    refs = {k: oracle.knn(x.cpu().numpy(), k) for k in (1, 100, 128)}
    torch.cuda.synchronize()
    errors = []

    def work(k):
        try:
            st = torch.cuda.Stream()
            for _ in range(60):
                with torch.cuda.stream(st):
                    d, i = affinity.knn(x, k, stream=st.cuda_stream)
                st.synchronize()
                np.testing.assert_array_equal(i.cpu().numpy(), refs[k][1])
                np.testing.assert_array_equal(d.cpu().numpy(), refs[k][0])
        except BaseException as e:  # reported by the main thread
            errors.append((k, e))

    threads = [threading.Thread(target=work, args=(k,)) for k in refs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]
