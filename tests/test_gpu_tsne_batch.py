"""Batched t-SNE: the graph-captured batch step against the same steps
enqueued uncaptured (bit-identical embeddings), against independent
single-system steps (close), and the input checks."""
import numpy as np
import pytest

from masterthesislucas_gb300 import affinity, datasets
from masterthesislucas_gb300.tsne import TSNE, TSNEBatch

pytestmark = pytest.mark.gpu


def make_systems(sizes, seed=0):
    out = []
    for k, n in enumerate(sizes):
        x, _ = datasets.cluster_data(n, 16, k=5 + k, seed=seed + k)
        rp, col, val = affinity.build_p_csr(x, perplexity=10.0, device="cuda")
        y0 = np.random.default_rng(seed + 100 + k).normal(0.0, 1e-2, (n, 2))
        out.append((rp, col, val, y0))
    return out


def build(data, order=8):
    return [TSNE(rp, col, val, y0, early_exaggeration=12.0, max_children=16, order=order)
            for rp, col, val, y0 in data]


def test_graph_replay_matches_uncaptured_batch_steps():
    data = make_systems([2100, 3500, 7000])
    a, b = build(data), build(data)
    ba = TSNEBatch(a, margin=0.3, capture=True)
    bb = TSNEBatch(b, margin=0.3, capture=False)
    for _ in range(40):
        ba.time_step()
        bb.time_step()
    st = ba.stats()
    assert st["graph_launches"] >= 30 and st["captures"] >= 3 and st["graph_nodes"] > 100
    for sa, sb in zip(a, b):
        ya, _, ga = sa.embedding()
        yb, _, gb = sb.embedding()
        assert np.array_equal(ya, yb)
        assert np.array_equal(ga, gb)
    ba.close()
    bb.close()


def test_batch_tracks_independent_systems():
    data = make_systems([2500, 6000], seed=3)
    a, b = build(data), build(data)
    batch = TSNEBatch(a, margin=0.5)
    for _ in range(25):
        batch.time_step()
        for s in b:
            s.time_step()
    for sa, sb in zip(a, b):
        ya = sa.embedding()[0]
        yb = sb.embedding()[0]
        # the batch builds trees over enlarged boxes: the FMM approximation
        # differs, not the step; early exaggeration amplifies the difference
        # for a few points, so the bound is on the distribution
        scale = np.abs(yb).max()
        d = np.linalg.norm(ya - yb, axis=1)
        assert np.median(d) < 5e-3 * scale and np.percentile(d, 90) < 2e-2 * scale, (np.median(d), scale)
    batch.close()


def test_batch_rejects_systems_out_of_step():
    from masterthesislucas_gb300._lib import TreecodeError
    data = make_systems([2000, 2200], seed=5)
    s = build(data)
    s[0].time_step()  # out of step with s[1]
    with pytest.raises(TreecodeError):
        TSNEBatch(s)


@pytest.mark.parametrize("sizes", [[2049, 2600], [513, 5000, 40]])
def test_dense_leaves_in_a_batch(sizes):
    """Leaves of more than 512 points, whose near-field items a batch does not split, against single systems, which do."""
    rng = np.random.default_rng(8)
    data = []
    for n in sizes:
        rp = (4 * np.arange(n + 1)).astype(np.uint32)
        data.append((rp, rng.integers(0, n, 4 * n).astype(np.uint32), np.full(4 * n, 0.25 / n), rng.normal(0, 3, (n, 2))))

    def systems():  # four leaves, all pairs direct whatever the box
        return [TSNE(rp, col, val, y0, max_children=16, order=8, depth=1, min_theta=0.1, max_theta=0.1)
                for rp, col, val, y0 in data]

    a, b = systems(), systems()
    batch = TSNEBatch(a, margin=0.5)
    for _ in range(3):  # the first uncaptured, then replays
        batch.time_step()
        for sa, sb in zip(a, b):
            sb.time_step()
            ga, gb = sa.embedding()[2], sb.embedding()[2]
            # FP32 sums of up to 5,000 terms on either side, runs of 2,048 with 64 lanes' partial sums a run
            assert np.abs(ga - gb).max() <= 2e-5 * np.abs(gb).max()
    batch.close()
