"""The kNN filter's approximate distances against FP64: within the bound that makes the neighbours exact, with room.

The bound allots 2^-15 |x_i| |x_j| to the parts dropped (three quarters of it at worst), 2^-20 of it to each MMA step
and 2^-21 (|x_i|^2 + |x_j|^2) to the norms and the last sum, each at least four thirds of what the arithmetic can lose.
Inputs of either sign, inputs whose dropped parts all have one sign, and BF16 numbers; few dimensions and the most.
"""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from masterthesislucas_gb300 import build

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def native(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("gram") / "knn_gram.so")
    cmd = [build.nvcc(), "-shared", "-o", so, os.path.join(HERE, "native", "knn_gram.cu")]
    r = subprocess.run(cmd + build._flags("affinity.cu"), capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    lib = ctypes.CDLL(so)
    lib.gram.argtypes = [ctypes.c_void_p, ctypes.c_longlong, ctypes.c_int] + [ctypes.c_void_p] * 6
    return lib


@pytest.mark.parametrize("dim", [1, 16, 784, 4096])
@pytest.mark.parametrize("values", ["normal", "one_sided", "pixels"])
def test_error_of_the_approximate_distances(native, dim, values):
    import torch
    n, npad, rblocks = 700, 768, 6
    rng = np.random.default_rng(dim)
    if values == "normal":
        x = rng.normal(size=(n, dim))
    elif values == "pixels":
        x = rng.integers(0, 257, (n, dim)) / 256.0
    else:  # above a BF16 number by a little less than half a step, by a little less than half a step of the rest
        x = (1.0 + rng.integers(0, 128, (n, dim)) / 128.0) + 2.0 ** -9 * (1.0 + 2.0 ** -7 * rng.integers(0, 64, (n, dim))) \
            + 0.49 * 2.0 ** -16
        x -= 2.0 ** -9
    x = x.astype(np.float32)
    dimp = (dim + 15) // 16 * 16
    dev = dict(device="cuda")
    xd = torch.from_numpy(x).cuda()
    hi, lo = (torch.empty(npad * dimp, dtype=torch.int16, **dev) for _ in range(2))
    s, a = torch.empty(npad, **dev), torch.empty(npad * 128 * rblocks, **dev)
    gmin, stat = torch.empty(npad * 128 * rblocks // 4, **dev), torch.zeros(4, dtype=torch.int32, **dev)
    torch.cuda.synchronize()
    assert native.gram(xd.data_ptr(), n, dim, hi.data_ptr(), lo.data_ptr(), s.data_ptr(), a.data_ptr(), gmin.data_ptr(),
                       stat.data_ptr()) == 0
    bad, any_lo = stat.cpu().numpy()[:2]
    assert bad == 0 and (any_lo == 0) == (values == "pixels")
    a = a.cpu().numpy().reshape(npad // 256, rblocks, 256, 128).transpose(1, 3, 0, 2).reshape(rblocks * 128, npad)[:n, :n]
    x64 = x.astype(np.float64)
    nu = np.sqrt((x64 * x64).sum(1))
    d = nu[:, None] ** 2 + nu[None, :] ** 2 - 2.0 * x64 @ x64.T  # good to 4096 2^-53 of the norms
    num = nu.max()
    steps = (3 if any_lo else 1) * (dimp // 16) + 8
    e = (nu * num * (2.1 * steps * 2.0 ** -20 + (2.0 ** -15 if any_lo else 0.0)) + 2.0 ** -21 * (nu ** 2 + num ** 2))
    assert np.all(np.abs(a - d) <= 0.75 * e[:, None])
