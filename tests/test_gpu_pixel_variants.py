"""scatter and deterministic gather at the edges of their kernels: one to five
and eight channels, rows that start off a 16-byte boundary, views whose number
of samples is no multiple of four, and samples and splats at the edges of the
packing's (8192) and the sort's (4096) tiles, of none and of all valid, and of
one to three passes.  Copies and sums in sample order: equal bits."""
import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("unaligned", [False, True])
@pytest.mark.parametrize("B,W,H,K,N,C,valid", [
    (1, 1, 1, 1, 1, 1, 1.0), (2, 5, 3, 1, 7, 2, 0.5), (2, 6, 4, 3, 9, 3, 0.5), (3, 4, 4, 2, 2000, 4, 0.0),
    (1, 64, 64, 1, 1, 1, 1.0), (1, 4097, 1, 1, 5, 3, 1.0), (1, 64, 128, 1, 1024, 5, 1.0), (1, 8193, 1, 1, 1025, 8, 1.0),
    (2, 90, 70, 8, 700_000, 3, 0.3)])
def test_equal_bits(B, W, H, K, N, C, valid, unaligned):
    from unbiased_differentiable_splatting_gb300.cudaExtensions import pixelgather as pg
    rng = np.random.default_rng(N + C)
    idx = rng.integers(0, N, size=(B, W, H, K)).astype(np.int32)
    idx[rng.random(idx.shape) >= valid] = -1
    v = rng.normal(size=(B, N, C)).astype(np.float32)
    g = rng.normal(size=(B, W, H, K, C)).astype(np.float32)

    def t(a):
        a = torch.as_tensor(a).cuda()
        return torch.cat([a.new_zeros(1), a.flatten()])[1:].view(a.shape) if unaligned else a

    np.testing.assert_array_equal(pg.scatter(t(idx), t(v)).cpu().numpy(), oracle.pixel_scatter(idx, v))
    np.testing.assert_array_equal(pg.gather(t(idx), t(g), N, deterministic=True).cpu().numpy(),
                                  oracle.pixel_gather(idx, g, N))
