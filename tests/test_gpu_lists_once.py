"""Interaction lists built in one pass per level (a handle's later builds) against the counted, scanned and filled ones
(its first build): the same lists, entry for entry.

Candidates within one batch of 128, several, and more than the outcomes kept for the writing (2,048); empty cells;
every MAC and both precisions of the records; leaf pairs sent to P2P.
"""
import ctypes

import numpy as np
import pytest

from masterthesislucas_gb300 import NBodySolverFMM_MORTON, NBodySolverFMM_SYM_MORTON, Points, datasets
from masterthesislucas_gb300._lib import check, lib, ptr

pytestmark = pytest.mark.gpu


def lists(solver, depth):
    out = []
    for level in range(depth + 1):
        for kind in (0, 1):
            p, tot = np.zeros((1 << (2 * level)) + 1, np.uint32), ctypes.c_int64(0)
            check(lib().tc_get_list(solver._h, level, kind, ptr(p), None, ctypes.byref(tot)))
            idx = np.zeros(max(tot.value, 1), np.uint32)
            check(lib().tc_get_list(solver._h, level, kind, ptr(p), ptr(idx), ctypes.byref(tot)))
            assert p[-1] == tot.value
            out += [p, idx[:tot.value]]
    return out


@pytest.mark.parametrize("depth,theta", [(0, 0.5), (1, 0.5), (4, 0.9), (5, 0.05), (6, 0.5), (9, 0.8)])
@pytest.mark.parametrize("kind", ["sym", "sym64", "morton", "order_cell", "order_bmax", "order_p2p"])
def test_one_pass_lists_equal_counted_ones(depth, theta, kind):
    cls = NBodySolverFMM_MORTON if kind == "morton" else NBodySolverFMM_SYM_MORTON
    kw = dict(order_cell=dict(order=4, mac="cell"), order_bmax=dict(order=4, mac="bmax"),
              order_p2p=dict(order=8, mac="bmax", leaf_p2p=64), sym64=dict(precision="fp64")).get(kind, {})
    pos = datasets.gaussian_mixture(3000, seed=depth).astype(np.float64)
    s = cls("gravity", tree_depth=depth, theta=theta, softening=1e-3, **kw)
    pts = Points.from_positions(pos)
    s.updateTree(pts, pos.min(0), pos.max(0))
    counted = lists(s, depth)
    pts = Points.from_positions(pos)
    s.updateTree(pts, pos.min(0), pos.max(0))
    for a, b in zip(counted, lists(s, depth)):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("depth", [4, 5, 6])
def test_kept_outcomes_of_several_batches(depth):
    """Every pair near (256, 1,024 and 4,096 candidates a node, of which 2,048 are kept), built over and over."""
    pos = np.random.default_rng(depth).random((4000, 2))
    mn, mx = np.zeros(2), np.ones(2)
    s = NBodySolverFMM_SYM_MORTON("tsne", tree_depth=depth, theta=0.01, order=4)
    s.updateTree(Points.from_positions(pos), mn, mx)
    counted = lists(s, depth)
    for _ in range(10):
        s.updateTree(Points.from_positions(pos), mn, mx)
        for a, b in zip(counted, lists(s, depth)):
            np.testing.assert_array_equal(a, b)


def test_lists_after_replays_of_a_captured_step():
    """The pointers of the last replay; entries only as far as the captured step's total, which the caller has room for."""
    import torch
    rng = np.random.default_rng(4)
    pos = rng.random((20000, 2))
    box, depth = np.array([0.0, 0.0, 1.0, 1.0]), 5
    pd = torch.from_numpy(pos).cuda()
    g, t = torch.zeros_like(pd), torch.zeros(1, dtype=torch.float64, device="cuda")
    s, fresh = (NBodySolverFMM_SYM_MORTON("tsne", tree_depth=depth, theta=0.8, order=4, mac="bmax") for _ in range(2))
    s.update_tree_device(pd, box[:2], box[2:])
    s.capture_step(pd, g, t, box=box)
    more = 0
    for f in (0.99, 0.97, 0.95, 0.93):
        pd.copy_(torch.from_numpy(pos * f))
        s.launch_step()
        torch.cuda.synchronize()
        assert s.async_status() == 0
        fresh.update_tree_device(pd, box[:2], box[2:])
        for level in range(depth + 1):
            for kind in (0, 1):
                words, tots = [], []
                for h in (s, fresh):
                    p, tot = np.zeros((1 << (2 * level)) + 1, np.uint32), ctypes.c_int64(0)
                    check(lib().tc_get_list(h._h, level, kind, ptr(p), None, ctypes.byref(tot)))
                    idx = np.full(2 * tot.value + 100000, 0xFFFFFFFF, np.uint32)
                    check(lib().tc_get_list(h._h, level, kind, ptr(p), ptr(idx), ctypes.byref(tot)))
                    assert np.all(idx[tot.value:] == 0xFFFFFFFF)
                    words.append((p, idx))
                    tots.append(tot.value)
                np.testing.assert_array_equal(words[0][0], words[1][0])
                m = min(tots)
                np.testing.assert_array_equal(words[0][1][:m], words[1][1][:m])
                more += words[1][0][-1] > tots[0]
    assert more > 0  # some lists had outgrown the captured total
