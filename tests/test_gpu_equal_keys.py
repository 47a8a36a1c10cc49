"""Order sampling where many keys are equal: coincident splats and uniforms of
few values, for sample lists of every storage.  Which of equal keys stays, and
in which order, follows the swaps of the reference's list: equal bits with the
oracle, also where the list is full."""
import math

import numpy as np
import pytest

import oracle
from test_gpu_descent_tables import T, cloud, smp  # noqa: F401


pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [3, 8, 16, 17, 24, 40, 64])
def test_equal_keys(smp, K):
    W, H, N = 12, 9, 900
    f = 1.1 * W
    pts, nrm, sd = cloud(K, N, W, H, f, 0.05)
    rng = np.random.default_rng(K)
    pts[:] = pts[rng.integers(0, 30, N)]
    R = math.ceil(math.sqrt(K))
    u = rng.integers(1, 4, size=(1, W, H, R, K)).astype(np.float32) * 0.25
    idx, st = smp.sample(W, H, f, T(pts[None]), T(nrm[None]), None, T(sd[None]), K, 0.0, 0.01, uniforms=T(u),
                         return_stats=True)
    ref, _ = oracle.sample_view(W, H, f, pts, nrm, sd, K, 0.0, 0.01, h=float(st["h"][0]), uniforms=u[0])
    assert (ref >= 0).mean() > 0.5
    np.testing.assert_array_equal(idx.cpu().numpy()[0], ref)
