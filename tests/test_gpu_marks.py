"""The marks of sampled (view, splat) pairs in their forms: bit maps of one
range and of several, ranges that end off a word, sample by sample for few
samples or very many splats, aligned and not.  Reference: the same samples on
the sampled splats alone, renumbered.  No two samples of a view share a splat,
so weights and gradients have equal bits; splats that no pixel samples get
zero gradients."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("unaligned", [False, True])
@pytest.mark.parametrize("N,side", [(40_000, 96), (1 << 20, 96), ((1 << 20) + 1, 96), (2_500_033, 97), (4_194_305, 96),
                                    (5_001, 20)])
def test_marked_pairs(N, side, unaligned):
    from unbiased_differentiable_splatting_gb300 import library  # noqa: F401
    o = torch.ops.uds
    B, W, H, K, f = 2, side, side + 1, 4, 0.9 * side
    g = torch.Generator(device=DEV).manual_seed(N)
    rand = lambda *s: torch.rand(s, device=DEV, generator=g)  # noqa: E731
    S = W * H * K
    idx = torch.stack([torch.randperm(N, device=DEV, generator=g)[:S] for _ in range(B)]).view(B, W, H, K)
    idx[:, :, :, 0] = torch.where(rand(B, W, H) < 0.5, idx[:, :, :, 0], N)  # out of range
    idx[idx == N - 1] = -1
    idx[:, 0, 0, 1] = N - 1  # the last one, by one pixel
    pts = torch.stack([(rand(B, N) - 0.5) * 2, (rand(B, N) - 0.5) * 2, -2 - rand(B, N)], -1).contiguous()
    nrm = torch.nn.functional.normalize(rand(B, N, 3) - torch.tensor([0.5, 0.5, -0.5], device=DEV), dim=-1)
    sd = 0.05 + rand(1, N, 2)
    some = idx[(idx >= 0) & (idx < N)].unique()
    to = torch.full((N + 1,), -1, dtype=torch.int64, device=DEV)
    to[some] = torch.arange(some.shape[0], device=DEV)
    small = torch.where((idx >= 0) & (idx < N), to[idx.clamp(0, N)], -1).int()
    idx = idx.int()
    if unaligned:
        idx = torch.cat([idx.new_zeros(1), idx.flatten()])[1:].view(idx.shape)
    part = [t[:, some].contiguous() for t in (pts, nrm, sd)]
    w = o.splat_forward(W, H, f, idx, pts, nrm, sd, 0.1)
    assert torch.equal(w, o.splat_forward(W, H, f, small, *part, 0.1))
    grad = rand(B, W, H, K) - 0.5
    gp, gn, gs = o.splat_backward(W, H, f, grad, idx, pts, nrm, sd, 0.1)
    hp, hn, hs = o.splat_backward(W, H, f, grad, small, *part, 0.1)
    for a, b in ((gp, hp), (gn, hn), (gs, hs)):
        assert torch.equal(a[:, some], b)
        a[:, some] = 0
        assert not a.any()
