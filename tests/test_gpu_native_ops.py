"""The native CUDA implementations of torch.ops.uds: opcheck of the ops that
only they and the Python definitions share, gradients equal to the Python
formulas', and the refusals (devices, types, layouts, sizes) of the Python
wrappers with the same exception types."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def ops():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from unbiased_differentiable_splatting_gb300 import library  # noqa: F401
    return torch.ops.uds


def rand(*shape, grad=False):
    return torch.rand(shape, device=DEV).requires_grad_(grad)


@pytest.mark.parametrize("kind", [0, 1])
def test_image_loss(ops, kind):
    x, y = rand(2, 5, 3, 3, grad=True), rand(2, 5, 3, 3)
    torch.library.opcheck(ops.image_loss.default, (x, y, kind, 0.25))
    loss, _ = ops.image_loss(x, y, kind, 0.25)
    (g,) = torch.autograd.grad(3.0 * loss, x)
    ref = 0.25 * ((x - y).abs() if kind == 0 else (x - y) ** 2).sum()
    (gr,) = torch.autograd.grad(3.0 * ref, x)
    torch.testing.assert_close(loss, ref, rtol=1e-6, atol=0)  # 90 terms in another order
    torch.testing.assert_close(g, gr, rtol=1e-6, atol=0)


def test_nearest_losses(ops):
    N, M = 40, 5
    pts, nrm = rand(1, N, 3, grad=True), torch.nn.functional.normalize(rand(1, N, 3), dim=-1).requires_grad_(True)
    near = torch.randint(-1, N, (1, N, M), dtype=torch.int32, device=DEV)
    torch.library.opcheck(ops.nearest_losses.default, (pts, nrm, near, 0.5, True))
    a, b, gp, gn = ops.nearest_losses(pts, nrm, near, 0.5, True)
    losses, gp2, gn2 = ops.nearest_regularizer(near, pts.detach(), nrm.detach(), 0.5, True)
    assert torch.equal(torch.stack([a, b]), losses) and torch.equal(gp, gp2) and torch.equal(gn, gn2)
    g1, g2 = torch.autograd.grad(2.0 * a + 3.0 * b, (pts, nrm))
    assert torch.equal(g1, 3.0 * gp) and torch.equal(g2, 2.0 * gn)
    only = torch.autograd.grad(ops.nearest_losses(pts, nrm, near, 0.5, True)[0], (pts, nrm))
    assert not only[0].any() and torch.equal(only[1], gn)


def test_unused_outputs_and_undefined_gradients(ops):
    """Gradients that reach only some outputs of a multi-output op."""
    idx = torch.zeros(1, 4, 4, 2, dtype=torch.int32, device=DEV)
    p = torch.tensor([[[0.0, 0.0, -2.0]]], device=DEV, requires_grad=True)
    n = torch.tensor([[[0.0, 0.0, -1.0]]], device=DEV)
    s, a = torch.full((1, 1, 2), 0.5, device=DEV, requires_grad=True), rand(1, 1, 3, grad=True)
    img, depth, w = ops.render_splats(4, 4, 4.0, idx, p, n, s, 0.0, a)
    both = torch.autograd.grad(depth.sum() + w.sum(), (p, s, a), retain_graph=True)
    zero = torch.zeros_like(img)
    full = torch.autograd.grad((img * zero).sum() + depth.sum() + w.sum(), (p, s, a))
    for x, y in zip(both, full):
        torch.testing.assert_close(x, y, rtol=1e-6, atol=0)
    cam, nrm = rand(2, 6, 3, grad=True), rand(1, 6, 3, grad=True)
    fc, fw = ops.backface(cam, nrm)
    assert torch.autograd.grad(fw.sum(), nrm)[0].shape == nrm.shape


def test_refusals(ops):
    from unbiased_differentiable_splatting_gb300._lib import UdsError
    M, v = rand(2, 4, 4, grad=True), rand(1, 9, 3)
    with pytest.raises(ValueError, match="must be a CUDA tensor"):
        ops.affine_forward(M.cpu(), v.cpu())
    with pytest.raises(ValueError, match="must be a CUDA tensor"):
        ops.affine_forward(M, v.cpu())
    with pytest.raises(TypeError, match="must be torch.float32"):
        ops.affine_forward(M.double(), v)
    with pytest.raises(ValueError, match="must be contiguous"):
        ops.affine_forward(M.transpose(1, 2), v)
    with pytest.raises(ValueError, match="expected transformation"):
        ops.affine_forward(M[:, :3].contiguous(), v)
    idx, w = torch.zeros(1, 2, 2, 70, dtype=torch.int32, device=DEV), rand(1, 2, 2, 70)
    with pytest.raises(UdsError, match="invalid argument"):
        ops.filter_forward(idx, w, 2, 2, 1.0, v, v)
    with pytest.raises(TypeError):
        ops.lambert_forward(rand(3), rand(1, 9, 3), rand(1, 9, 3), v, v)  # nine lights
    with pytest.raises(RuntimeError):  # no second derivatives
        (g,) = torch.autograd.grad(ops.affine_forward(M, v).sum(), M, create_graph=True)
        g.sum().backward()
        (g,) = torch.autograd.grad((ops.affine_forward(M, v) ** 2).sum(), M, create_graph=True)
        g.sum().backward()
