"""Gradient sums over splats of the transform and of the per-splat Lambert
shading where a thread takes four splats and where it takes one: sizes at the
edge of the two and off their blocks, more views than a block sums at a time.
Sums of N float32 products against float64: 1e-5 of the sum of magnitudes (a
tree of at most 2^9 sequential additions of 2^-24 each)."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def close(got, exact, scale):
    assert float(((got.double() - exact).abs() / scale.clamp_min(1e-30)).max()) < 1e-5


@pytest.mark.parametrize("affine", [True, False])
@pytest.mark.parametrize("B,N", [(1, 5), (1, 310_272), (2, 310_273), (3, 311_296), (35, 1000), (33, 311_001)])
def test_transform(affine, B, N):
    from unbiased_differentiable_splatting_gb300 import library  # noqa: F401
    g = torch.Generator(device=DEV).manual_seed(N + B)
    M, v = torch.randn(B, 4, 4, device=DEV, generator=g), torch.randn(1, N, 3, device=DEV, generator=g)
    go = torch.randn(B, N, 3, device=DEV, generator=g)
    gM, gv = (torch.ops.uds.affine_backward if affine else torch.ops.uds.linear_backward)(go, M, v)
    vd, gd, Md = v[0].double(), go.double(), M.double()
    h = torch.cat([vd, (torch.ones if affine else torch.zeros)(N, 1, dtype=torch.float64, device=DEV)], 1)
    for b in range(B):
        close(gM[b, :3], gd[b].t() @ h, gd[b].abs().t() @ h.abs())
    assert not gM[:, 3].any()
    close(gv[0], torch.einsum("bni,bij->nj", gd, Md[:, :3, :3]),
          torch.einsum("bni,bij->nj", gd.abs(), Md[:, :3, :3].abs()))


@pytest.mark.parametrize("B,N,L,aB,IB,dB", [(1, 155_136, 1, 1, 1, 1), (2, 155_137, 2, 2, 1, 1),
                                            (2, 156_001, 4, 1, 2, 2), (3, 77, 3, 3, 3, 1)])
def test_lambert(B, N, L, aB, IB, dB):
    from unbiased_differentiable_splatting_gb300 import library  # noqa: F401
    g = torch.Generator(device=DEV).manual_seed(N + L)
    r = lambda *s: torch.randn(s, device=DEV, generator=g)  # noqa: E731
    amb, dirs, inten = r(aB, 1, 3).abs(), r(B, L, 3), r(IB, L, 3).abs()
    nrm, dif, go = r(B, N, 3), r(dB, N, 3).abs(), r(B, N, 3)
    got = torch.ops.uds.lambert_backward(go, amb, dirs, inten, nrm, dif)
    ins = [t.double().requires_grad_(True) for t in (amb, dirs, inten, nrm, dif)]
    a, d, i, n, f = ins

    def shade():
        s = torch.einsum("blk,bnk->bln", d, n)
        c = s.clamp(0.0, 1.0)
        out = a * f
        for k in range(L):
            out = out + i[:, k:k + 1] * c[:, k, :, None] * f / torch.pi
        return out

    exact = torch.autograd.grad(shade(), ins, go.double(), allow_unused=True)
    for q, (x, e) in enumerate(zip(got, exact)):
        if e is None or e.numel() == 0:
            continue
        if q < 3:  # sums over the splats (and views, where shared) of terms of order one
            assert float((x.double() - e).abs().max()) < 1e-5 * N * B
        else:
            torch.testing.assert_close(x, e.float(), rtol=1e-4, atol=1e-4)
