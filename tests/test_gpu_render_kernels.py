"""The per-pixel render kernels over their variants: numbers of samples at
the edges of the unrolled and rolled forms, odd image sizes, numbers of
channels around the vector widths, rows that start off a 16-byte boundary,
and the gradient ops against the raw gradients with the reference's
post-processing.  No two samples of a view share a splat, so that no sum
depends on the order of atomic additions: everything is bit-identical to the
separate ops, but for the post-processing's norms, whose roundings differ by
a few units in the last place (1e-6)."""
import pytest
import torch

from test_gpu_fused_render import DEV, _inputs, mods  # noqa: F401

pytestmark = pytest.mark.gpu


def off(t):
    """The same tensor, contiguous, one element off its allocation's start."""
    return torch.cat([t.new_zeros(1), t.flatten()])[1:].view(t.shape)


def post(g):
    g = g / torch.clamp(g.norm(dim=-1, keepdim=True) + 1e-4, 1.0)
    return torch.nan_to_num(g, nan=0.0, posinf=float("inf"), neginf=float("-inf"))


@pytest.mark.parametrize("unaligned", [False, True])
@pytest.mark.parametrize("K,C,aB,sB", [(1, 1, 1, 1), (3, 2, 2, 2), (8, 4, 1, 1), (9, 5, 2, 1), (12, 8, 1, 2),
                                       (16, 3, 1, 1), (17, 7, 2, 1), (33, 3, 1, 2), (64, 4, 1, 1)])
def test_variants(mods, K, C, aB, sB, unaligned):
    splatting, filtering, interpolation = mods
    o = torch.ops.uds
    B, W, H = 2, 19, 23
    N = W * H * K + 3
    idx, pts, nrm, sd, attr, f = _inputs(K, B, N, W, H, K, C, aB, 20.0)
    sd = sd.expand(sB, N, 2).contiguous()
    idx = torch.stack([torch.randperm(N, device=DEV)[:W * H * K].view(W, H, K).int() for _ in range(B)])
    idx[torch.rand(idx.shape, device=DEV) < 0.3] = -1
    idx[:, :5] = -1  # pixels without a sample
    idx[:, 7, 0] += 2 * N  # out of range: no sample
    if unaligned:
        idx, attr = off(idx), off(attr)
    img, dw, w = o.render_splats(W, H, f, idx, pts, nrm, sd, 0.1, attr)
    w_ref = splatting.forward(W, H, f, idx, pts, nrm, sd, 0.1)
    dw_ref = filtering.forward(idx, w_ref, W, H, f, pts, nrm)
    assert torch.equal(w, w_ref) and torch.equal(dw, dw_ref)
    assert torch.equal(img, interpolation.forward(idx, dw_ref, attr))
    g, gd, gw = torch.randn_like(img), torch.randn_like(dw), torch.randn_like(w)
    for gdepth, gweights in ((None, None), (gd, None), (gd, gw)):
        args = (W, H, f, g, gdepth, gweights, idx, w, pts, nrm, sd, 0.1, attr)
        gp, gn, gs, ga = o.render_splats_backward(*args)
        ge_in, ga_ref = interpolation.backward(g, idx, dw_ref, attr)
        ge = filtering.backward(idx, w_ref, ge_in if gdepth is None else ge_in + gd, W, H, f, pts, nrm)
        ge = ge if gweights is None else ge + gw
        raw = splatting.backward(W, H, f, ge, idx, pts, nrm, sd, 0.1)
        for got, ref in zip((gp, gn, gs, ga), (*raw, ga_ref)):
            assert torch.equal(got, ref)
        for got, ref in zip((*o.render_splats_gradients(*args), *o.splat_gradients(W, H, f, ge, idx, pts, nrm, sd, 0.1)),
                            (post(gp), post(gs), ga, post(gp), post(gs))):
            torch.testing.assert_close(got, ref, rtol=1e-6, atol=0)


def test_opcheck_gradients(mods):
    idx, pts, nrm, sd, attr, f = _inputs(5, 2, 300, 20, 16, 4, 3, 1, 30.0)
    img, dw, w = torch.ops.uds.render_splats(20, 16, f, idx, pts, nrm, sd, 0.0, attr)
    tests = ("test_schema", "test_faketensor")  # sums of atomic additions: no bit-equal second run
    torch.library.opcheck(torch.ops.uds.splat_gradients.default, (20, 16, f, w, idx, pts, nrm, sd, 0.0),
                          test_utils=tests)
    torch.library.opcheck(torch.ops.uds.render_splats_gradients.default,
                          (20, 16, f, img, dw, None, idx, w, pts, nrm, sd, 0.0, attr), test_utils=tests)
