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


@pytest.mark.parametrize("n", [127, 128, 129])
@pytest.mark.parametrize("k", [1, 126])
def test_one_candidate_tile(n, k):
    """Up to 128 points the lists are whole and written at once; above, they are joined."""
    import torch
    x = np.random.default_rng(n).normal(size=(n, 7)).astype(np.float32)
    d, i = affinity.knn(torch.from_numpy(x).cuda(), k)
    rd, ri = oracle.knn(x, k)
    np.testing.assert_array_equal(d.cpu().numpy(), rd)
    np.testing.assert_array_equal(i.cpu().numpy(), ri)


def test_scratch_kept_between_calls():
    """Calls at the ends of the range whose launches are sized to what is kept, and a large one, which is given back."""
    import gc

    import torch
    gc.collect()  # handles of tests before this one give their memory back now, not meanwhile
    rng = np.random.default_rng(13)
    free = []
    for n in (1500, 9000, 12288, 12289, 20000, 1500):
        x = torch.from_numpy(rng.random((n, 3)).astype(np.float32)).cuda()
        d, i = affinity.knn(x, 5)
        torch.cuda.synchronize()
        dist = ((x[:200, None, :] - x[None, :, :]) ** 2).sum(-1)
        dist[torch.arange(200), torch.arange(200)] = np.inf
        ref = torch.topk(dist, 5, largest=False).values.sort(1).values
        np.testing.assert_allclose(d[:200].cpu().numpy(), ref.cpu().numpy(), rtol=1e-5, atol=1e-12)
        del x, d, i, dist, ref
        torch.cuda.empty_cache()
        free.append(torch.cuda.mem_get_info()[0])
    assert max(free) - min(free) <= 96 << 20


CAPTURED_FIRST_CALL = """
import sys
import torch
from masterthesislucas_gb300 import affinity
x = torch.rand(int(sys.argv[1]), 8, device="cuda")
torch.cuda.synchronize()
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph, stream=torch.cuda.Stream()):
    d, i = affinity.knn(x, 5, stream=torch.cuda.current_stream().cuda_stream)
for _ in range(3):
    x.copy_(torch.rand_like(x))
    graph.replay()
    torch.cuda.synchronize()
    d2, i2 = affinity.knn(x, 5)
    torch.cuda.synchronize()
    assert torch.equal(d, d2) and torch.equal(i, i2)
"""


@pytest.mark.parametrize("n", [100, 900, 3000])
def test_first_call_inside_a_capture(n):
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", CAPTURED_FIRST_CALL, str(n)], capture_output=True, text=True, cwd=root)
    assert r.returncode == 0, r.stderr
