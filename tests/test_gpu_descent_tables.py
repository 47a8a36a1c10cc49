"""The descent's shared tables at the sizes where they can go wrong: unions
too large for a warp's tables (half the lanes at a time), masses past the
rows in shared memory, sample lists of every storage (registers, shared
memory), image edges, pixels whose capacity is used up.  Sampled indices and
path probabilities equal the CPU oracle's bit for bit."""
import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def T(a):
    return torch.as_tensor(np.ascontiguousarray(a)).to(device=DEV, dtype=torch.float32)


@pytest.fixture(scope="module")
def smp():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from unbiased_differentiable_splatting_gb300 import _lib
    from unbiased_differentiable_splatting_gb300.cudaExtensions import sampling
    _lib.load()
    return sampling


def cloud(seed, N, W, H, f, sd, spots=0):
    """Splats over the whole view, or (spots > 0) in that many tight spots."""
    rng = np.random.default_rng(seed)
    z = rng.uniform(-2.4, -1.6, N)
    if spots:
        c = rng.uniform(0.1, 0.9, size=(spots, 2))[rng.integers(0, spots, N)]
        u = c + rng.normal(0.0, 0.002, size=(N, 2))
    else:
        u = rng.uniform(0.0, 1.0, size=(N, 2))
    pts = np.stack([(u[:, 0] - 0.5) * -z * W / f, (u[:, 1] - 0.5) * -z * H / f, z], 1)
    n = rng.normal(size=(N, 3))
    n[:, 2] = np.abs(n[:, 2]) + 0.5
    n /= np.linalg.norm(n, axis=1, keepdims=True)
    return pts.astype(np.float32), n.astype(np.float32), np.full((N, 2), sd, np.float32)


@pytest.mark.parametrize("W,H,N,sd,precision,K,spots,tile", [
    (24, 20, 20_000, 0.002, 0.01, 8, 0, 8),    # h far below a pixel: the lanes' trees hardly overlap
    (24, 20, 20_000, 0.002, 0.01, 8, 0, 4),
    (33, 18, 30_000, 0.02, 1e-4, 8, 0, 16),    # long lists of expansions of high degree
    (9, 5, 4_000, 0.01, 0.01, 9, 0, 32),       # K = 9: first size with 16 keys
    (31, 7, 3_000, 0.02, 0.01, 17, 0, 8),      # K = 17: first size with lists in shared memory
    (17, 9, 3_000, 0.02, 0.01, 64, 0, 4),      # largest K
    (1, 1, 500, 0.02, 0.01, 8, 0, 8),
    (40, 24, 60, 0.004, 0.01, 8, 0, 8),        # a splat or two per pixel: rounds after the capacity is used up
    (40, 24, 900, 0.004, 0.01, 4, 6, 8),       # tight spots: deep stems
])
def test_indices_match_oracle(smp, W, H, N, sd, precision, K, spots, tile):
    f = 1.1 * W
    pts, nrm, s = cloud(N + K, N, W, H, f, sd, spots)
    idx, st = smp.sample(W, H, f, T(pts[None]), T(nrm[None]), None, T(s[None]), K, 0.0, precision, seed=21,
                         tile_x=tile, return_stats=True)
    ref, _ = oracle.sample_view(W, H, f, pts, nrm, s, K, 0.0, precision, h=float(st["h"][0]), seed=21)
    got = idx.cpu().numpy()[0]
    assert (got >= 0).any()
    np.testing.assert_array_equal(got, ref)


@pytest.mark.parametrize("W,H,N,sd,K,spots", [(24, 20, 20_000, 0.002, 4, 0), (33, 18, 6_000, 0.02, 8, 0),
                                              (40, 24, 900, 0.004, 5, 6)])
def test_stochastic_matches_oracle(smp, W, H, N, sd, K, spots):
    f = 1.1 * W
    pts, nrm, s = cloud(N + K, N, W, H, f, sd, spots)
    idx, prob, st = smp.sample_stochastic(W, H, f, T(pts[None]), T(nrm[None]), T(s[None]), K, 0.0, 0.01, seed=22,
                                          return_stats=True)
    ri, rp = oracle.sample_view_stochastic(W, H, f, pts, nrm, s, K, 0.0, 0.01, h=float(st["h"][0]), seed=22)
    np.testing.assert_array_equal(idx.cpu().numpy()[0], ri)
    np.testing.assert_array_equal(prob.cpu().numpy()[0], rp)
    assert (ri >= 0).any()
