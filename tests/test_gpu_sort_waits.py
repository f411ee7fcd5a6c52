"""The sort's bounded waits, run out: every tile that looks back before its predecessor is there counts for itself.

The sort is compiled with a limit of no polls at all, so that this happens to most tiles of a pass; the order has to be
the stable one all the same, from one tile to look back over up to the most keys whose tiles look back, with even and
odd numbers of passes, spread keys and few different ones.
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
def sort(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("sort") / "sort_waits.so")
    cmd = [build.nvcc(), "-shared", "-o", so, os.path.join(HERE, "native", "sort_waits.cu"), "-DTC_SORT_POLLS=0"]
    r = subprocess.run(cmd + build._flags("sort.cu"), capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    lib = ctypes.CDLL(so)
    lib.sort_tmp_words.restype = ctypes.c_longlong
    lib.sort_tmp_words.argtypes = [ctypes.c_longlong]
    lib.sort_u32.argtypes = [ctypes.c_void_p] * 4 + [ctypes.c_longlong, ctypes.c_void_p, ctypes.c_int, ctypes.c_void_p]
    return lib


@pytest.mark.parametrize("n", [4097, 6145, 100003, 1 << 20])
@pytest.mark.parametrize("lo_bit", [0, 8])
@pytest.mark.parametrize("values", [1 << 32, 5])
def test_order_without_waiting(sort, n, lo_bit, values):
    import torch
    rng = np.random.default_rng(n + lo_bit)
    k = rng.integers(0, values, n, dtype=np.uint64).astype(np.uint32) << (0 if values > 5 else 28)
    keys, vals, ak, av = (torch.zeros(n, dtype=torch.int32, device="cuda") for _ in range(4))
    odd = (32 - lo_bit + 7) // 8 % 2
    (ak if odd else keys).copy_(torch.from_numpy(k.view(np.int32)))
    tmp = torch.empty(sort.sort_tmp_words(n), dtype=torch.int32, device="cuda")
    assert sort.sort_u32(keys.data_ptr(), vals.data_ptr(), ak.data_ptr(), av.data_ptr(), n, tmp.data_ptr(), lo_bit,
                         torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    order = np.argsort(k >> lo_bit, kind="stable")
    np.testing.assert_array_equal(vals.cpu().numpy().view(np.uint32), order)
    np.testing.assert_array_equal(keys.cpu().numpy().view(np.uint32), k[order])
