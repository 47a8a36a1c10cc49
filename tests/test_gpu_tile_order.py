"""The order in which the descent takes an image's tiles covers every pixel:
images of less than a cell, of ragged and of single rows and columns of cells,
and of more pixels than cells of the smallest size reach, in every block
shape, for one view, several equal ones and different ones in one call."""
import pytest
import torch

from test_gpu_descent_tables import T, cloud, smp  # noqa: F401

pytestmark = pytest.mark.gpu


def scene(W, H, seed=0):
    f = 1.1 * max(W, H)
    p, n, s = cloud(seed, 2 * W * H + 500, W, H, f, 3.0 / f)  # two splats per pixel, a pixel wide or more
    n[:] = (0.0, 0.0, 1.0)
    return f, T(p[None]), T(n[None]), T(s[None])


@pytest.mark.parametrize("W,H,K,tile", [(1, 1, 8, 8), (16, 16, 8, 4), (17, 33, 8, 8), (33, 17, 20, 4), (255, 31, 13, 8),
                                        (1, 3000, 8, 8), (3000, 1, 20, 8), (3, 66000, 4, 8), (66000, 2, 8, 4),
                                        (1030, 1100, 4, 8)])
def test_every_pixel(smp, W, H, K, tile):
    f, p, n, s = scene(W, H)
    idx = smp.sample(W, H, f, p, n, None, s, K, 0.0, 0.01, seed=1, tile_x=tile)
    assert (idx[..., 0] >= 0).all()
    idx, prob = smp.sample_stochastic(W, H, f, p, n, s, 4, 0.0, 0.01, seed=1)[:2]
    assert (idx[..., 0] >= 0).all() and (prob[..., 0] > 0).all()


def test_views(smp):
    sizes = [(40, 33), (17, 90), (1, 5), (200, 16)]
    # every view sees the scene of its own size: the splats of the others are spare
    parts = [scene(w, h, b) for b, (w, h) in enumerate(sizes)]
    N = max(q[1].shape[1] for q in parts)
    pad = lambda t: torch.cat([t, t[:, :1].expand(1, N - t.shape[1], t.shape[2])], 1)  # noqa: E731
    p, n, s = (torch.cat([pad(q[k]) for q in parts]).contiguous() for k in (1, 2, 3))
    out = smp.sample_views([(w, h, q[0]) for (w, h), q in zip(sizes, parts)], p, n, None, s, 8, 0.0, 0.01, seed=1)
    for o in out:
        assert (o[..., 0] >= 0).all()
    w, h = sizes[0]
    f, p, n, s = parts[0]
    rep = lambda t: t.expand(3, -1, -1).contiguous()  # noqa: E731
    many = smp.sample(w, h, f, rep(p), rep(n), None, rep(s), 8, 0.0, 0.01, seed=1)
    one = smp.sample(w, h, f, p, n, None, s, 8, 0.0, 0.01, seed=1)
    assert torch.equal(many[:1], one) and (many[..., 0] >= 0).all()


def test_descent_of_another_size(smp):
    """A tree built for one image, descended for images of other sizes: every
    pixel that the descent for the tree's own size takes, and as it does."""
    W, H = 70, 90
    f, p, n, s = scene(W, H)
    prm = smp.params(W, H, f, p, s, 8, 0.0, 0.01, 1)
    L = smp.load()
    ws = torch.empty(L.uds_sample_workspace_size(prm), dtype=torch.uint8, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    assert L.uds_tree_build(prm, 0, p.data_ptr(), n.data_ptr(), s.data_ptr(), None, None, None, None, None, None, None,
                            None, None, None, None, ws.data_ptr(), ws.numel(), stream) == 0

    def descend(w, h):
        q = smp.params(w, h, f, p, s, 8, 0.0, 0.01, 1)
        idx = torch.full((w, h, 8), -1, dtype=torch.int32, device="cuda")
        assert L.uds_sample_descent(q, 0, None, idx.data_ptr(), ws.data_ptr(), ws.numel(), stream) == 0
        return idx

    own = descend(W, H)
    assert torch.equal(own, smp.sample(W, H, f, p, n, None, s, 8, 0.0, 0.01, seed=1)[0])
    assert torch.equal(descend(33, H), own[:33])  # (the same pixel numbers, hence uniforms)
    assert (descend(200, 40)[:W, :, 0] >= 0).all()
