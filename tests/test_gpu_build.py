"""The tree build at the sizes where its single-pass kernels can go wrong: one
and two visible splats, the edges of tiles of splats (2048) and nodes (128),
culled splats between the visible ones, equal keys, a pool of coefficients
that runs out, more views than a launch covers, and wait words of many tiles.
Every array equals the CPU oracle's bit for bit."""
import numpy as np
import pytest
import torch

import oracle
from test_gpu_descent_tables import T, cloud, smp  # noqa: F401

pytestmark = pytest.mark.gpu
W, H, F = 60, 50, 64.0


def check(smp, pts, nrm, sd, pool=0):
    tree = smp.build_tree(W, H, F, T(pts[None]), T(nrm[None]), T(sd[None]), 8, 0.0, 0.01, coef_pool=pool)
    assert tree["h"] == np.float32(oracle.view_bandwidth(W, H, F, pts, nrm, sd, 0.0))
    t = oracle.Tree(W, H, F, pts, tree["h"], tree["radius"], 0.01, coef_pool=pool if pool else -1)
    e, n = t.export(), t.n
    assert tree["n_visible"] == n and tree["n_coefs"] == t.num_coefs
    np.testing.assert_array_equal(tree["keys"].numpy().view(np.uint32), e["keys"])
    for k in ("ids", "parent", "count", "degree", "centre", "box"):
        np.testing.assert_array_equal(tree[k].numpy(), e[k])
    for k in ("left", "right"):
        np.testing.assert_array_equal(tree[k].numpy()[: n - 1], e[k][: n - 1])
    if n:
        rng = np.random.default_rng(n)
        nodes = rng.integers(0, 2 * n - 1, size=200).astype(np.int32)
        q = rng.uniform(0, H, size=(200, 2)).astype(np.float32)
        got = smp.fgt_eval(tree, torch.as_tensor(nodes).cuda(), T(q)).cpu().numpy()
        np.testing.assert_array_equal(got, np.array([t.node_weight(int(v), q[i]) for i, v in enumerate(nodes)],
                                                    np.float32))
    return n


@pytest.mark.parametrize("n", [0, 1, 2, 3, 33, 128, 129, 130, 2047, 2048, 2049, 4097, 70_000])
def test_sizes(smp, n):
    N = n + n // 3 + 5  # the others behind the camera, in between
    pts, nrm, sd = cloud(n, N, W, H, F, 0.02)
    hidden = np.random.default_rng(n).permutation(N)[n:]
    pts[hidden, 2] *= -1
    assert check(smp, pts, nrm, sd) == n


def test_equal_keys(smp):
    pts, nrm, sd = cloud(1, 5000, W, H, F, 0.02)
    pts[:] = pts[0]
    check(smp, pts, nrm, sd)


@pytest.mark.parametrize("pool", [500, 20_000])
def test_pool_runs_out(smp, pool):
    pts, nrm, sd = cloud(2, 3000, W, H, F, 0.02)
    check(smp, pts, nrm, sd, pool)


def test_more_views_than_a_launch(smp):
    B, K, w, h = 35, 4, 20, 17
    parts = [cloud(b, 300, w, h, F, 0.05) for b in range(B)]
    p, n, s = (np.stack([q[k] for q in parts]) for k in range(3))
    idx, st = smp.sample(w, h, F, T(p), T(n), None, T(s), K, 0.0, 0.01, seed=5, return_stats=True)
    many = smp.sample_views([(w, h, F)] * B, T(p), T(n), None, T(s), K, 0.0, 0.01, seed=5)
    for b in (0, 1, 31, 32, 34):
        ref, _ = oracle.sample_view(w, h, F, *parts[b], K, 0.0, 0.01, h=float(st["h"][b]), seed=5, view=b)
        np.testing.assert_array_equal(idx[b].cpu().numpy(), ref)
        np.testing.assert_array_equal(many[b][0].cpu().numpy(), ref)
    assert torch.equal(torch.cat(list(many)), idx)
