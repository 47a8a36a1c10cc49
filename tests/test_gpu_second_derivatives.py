"""No second derivatives: the backward ops have no formula of their own,
whether the first gradient depends on the differentiated input or not."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("outer", [lambda y: y.sum(), lambda y: (y ** 2).sum(), lambda y: y.exp().sum()])
@pytest.mark.parametrize("at", [0, 1])
def test_refused(outer, at):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from unbiased_differentiable_splatting_gb300 import library  # noqa: F401
    inputs = [torch.rand(s, device=DEV).requires_grad_(True) for s in ((2, 4, 4), (1, 9, 3))]
    (g,) = torch.autograd.grad(outer(torch.ops.uds.affine_forward(*inputs)), inputs[at], create_graph=True)
    with pytest.raises(RuntimeError):
        g.sum().backward()
