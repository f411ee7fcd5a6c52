"""The host entries of Barnes-Hut and the particle mesh, whose device copies are kept for later calls: several threads and
sizes at once, and nothing kept of a large call."""
import ctypes
import threading

import numpy as np
import pytest

from masterthesislucas_gb300._lib import check, lib
from masterthesislucas_gb300.solver import barnes_hut, particle_mesh

pytestmark = pytest.mark.gpu


def test_threads_of_different_sizes():
    rng = np.random.default_rng(2)
    jobs = [(f, rng.normal(0, 3, (n, 2))) for n in (40, 1500, 20011) for f in (barnes_hut, particle_mesh)]
    refs = [f(p) for f, p in jobs]
    errors = []

    def work(k):
        try:
            for _ in range(8):
                f, p = jobs[k]
                g, total = f(p)
                np.testing.assert_allclose(g, refs[k][0], rtol=0, atol=1e-12 * np.abs(refs[k][0]).max())
                assert total == pytest.approx(refs[k][1], rel=1e-12)
        except BaseException as e:  # reported by the main thread
            errors.append((k, e))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]


def test_a_large_call_keeps_no_copies():
    import gc

    import torch
    gc.collect()  # handles of tests before this one give their memory back now, not meanwhile
    n = 3_000_000  # 48 MB in, 48 MB out
    pos = np.random.default_rng(0).random((n, 2))
    d = torch.from_numpy(pos).cuda()
    g, total = torch.empty_like(d), torch.empty(1, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    # the workspace grows to its size by the device entry
    check(lib().tc_bh_solve_device(1, 1e-3, 64, 2.0, 0, ctypes.c_void_p(d.data_ptr()), n, ctypes.c_void_p(g.data_ptr()),
                                   ctypes.c_void_p(total.data_ptr()), None))
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    gh, _ = barnes_hut(pos, kernel="gravity", softening=1e-3, max_children=64, theta=2.0)
    np.testing.assert_array_equal(gh, g.cpu().numpy())
    assert before - torch.cuda.mem_get_info()[0] < 64 << 20
