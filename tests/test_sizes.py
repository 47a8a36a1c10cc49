"""Arrays that the kernels index by other arrays' sizes: one of another size
is refused with a ValueError before anything is enqueued, by the Python
wrappers (here without a GPU: device checks and the library are stubbed) and by
the native CUDA implementations of torch.ops.uds."""
import pytest
import torch

from unbiased_differentiable_splatting_gb300 import library, training  # noqa: F401  (registers torch.ops.uds)
from unbiased_differentiable_splatting_gb300.cudaExtensions import (filtering, interpolation, shading, splatting,
                                                                    transform)

B, W, H, K, N, C, L = 2, 4, 3, 2, 5, 3, 2


def arrays(device):
    z = lambda *s: torch.zeros(s, device=device)  # noqa: E731
    return dict(idx=torch.zeros((B, W, H, K), dtype=torch.int32, device=device), w=z(B, W, H, K), pts=z(B, N, 3),
                sd=z(1, N, 2), attr=z(1, N, C), img=z(B, W, H, C), M=z(B, 4, 4), v=z(1, N, 3), dirs=z(B, L, 3),
                power=z(1, L, 3), coef=z(1, 9, 3), px=z(B, W, H, 3), pos=z(B, 3), quat=z(B, 4), g16=z(B, 1, 4, 4))


# name of the call, (op of torch.ops.uds, its arguments in order, Python wrapper), then the argument
# that is replaced and by what shape
def calls(a):
    u = torch.ops.uds
    geo = (a["idx"], a["pts"], a["pts"], a["sd"], 0.0)
    return {
        "image_loss": (u.image_loss, training.image_loss, (a["px"], a["px"], 1, 1.0)),
        "splat_forward": (u.splat_forward, splatting.forward, (W, H, 4.0, *geo)),
        "splat_backward": (u.splat_backward, splatting.backward, (W, H, 4.0, a["w"], *geo)),
        "render_splats_backward": (u.render_splats_backward, splatting.renderBackward,
                                   (W, H, 4.0, a["img"], None, None, a["idx"], a["w"], a["pts"], a["pts"], a["sd"],
                                    0.0, a["attr"])),
        "filter_forward": (u.filter_forward, filtering.forward, (a["idx"], a["w"], W, H, 4.0, a["pts"], a["pts"])),
        "filter_backward": (u.filter_backward, filtering.backward,
                            (a["idx"], a["w"], a["w"], W, H, 4.0, a["pts"], a["pts"])),
        "interp_backward": (u.interp_backward, interpolation.backward, (a["img"], a["idx"], a["w"], a["attr"])),
        "affine_backward": (u.affine_backward, transform.affineBackward, (a["pts"], a["M"], a["v"])),
        "view_matrix_forward": (u.view_matrix_forward, transform.viewMatrixForward, (a["pos"], a["quat"])),
        "view_matrix_backward": (u.view_matrix_backward, transform.viewMatrixBackward, (a["g16"], a["quat"])),
        "backface_backward": (u.backface_backward, transform.backfaceBackward, (a["pts"], a["pts"], a["pts"], 1)),
        "shade_forward": (u.shade_forward, shading.forward, (a["dirs"], a["power"], a["px"], a["px"])),
        "shade_backward": (u.shade_backward, shading.backward, (a["px"], a["dirs"], a["power"], a["px"], a["px"])),
        "shade_sh_forward": (u.shade_sh_forward, shading.forwardSh, (a["coef"], a["px"], a["px"])),
        "shade_sh_backward": (u.shade_sh_backward, shading.backwardSh, (a["px"], a["coef"], a["px"], a["px"])),
    }


BAD = [("image_loss", 1, (1, W, H, 3)), ("splat_forward", (4, 5), (B, N, 2)), ("splat_forward", 6, (1, N, 1)),
       ("splat_backward", 7, (1, N, 1)), ("render_splats_backward", 12, (1, N - 1, C)),
       ("render_splats_backward", 12, (3, N, C)), ("filter_forward", (5, 6), (B, N, 2)),
       ("filter_backward", 2, (B, W, H, K - 1)), ("interp_backward", 0, (B, W, H, C - 1)),
       ("affine_backward", 2, (1, N, 2)), ("affine_backward", 1, (B, 3, 4)), ("view_matrix_forward", 0, (1, 3)),
       ("view_matrix_forward", 1, (B, 3)), ("view_matrix_backward", 0, (1, 1, 4, 4)),
       ("backface_backward", 1, (1, N, 3)), ("backface_backward", 2, (1, N, 3)), ("shade_forward", 0, (1, L, 3)),
       ("shade_forward", 1, (1, L, 2)), ("shade_backward", 0, (1, W, H, 3)), ("shade_backward", 1, (B, L - 1, 3)),
       ("shade_sh_forward", 0, (1, 9, 1)), ("shade_sh_backward", 0, (B, W, H, 2))]


def replaced(args, at, shape):
    at = at if isinstance(at, tuple) else (at,)
    dev = next(x for x in args if isinstance(x, torch.Tensor)).device
    return tuple(torch.zeros(shape, device=dev) if k in at else x for k, x in enumerate(args))


@pytest.mark.parametrize("name,at,shape", BAD)
def test_wrappers_refuse(monkeypatch, name, at, shape):
    class Enqueued(Exception):
        pass

    def load():
        raise Enqueued

    def need(t, name, dtype=torch.float32, device=None):
        return t

    _, wrapper, args = calls(arrays("cpu"))[name]
    module = __import__(wrapper.__module__, fromlist=["x"])
    monkeypatch.setattr(module, "load", load)
    monkeypatch.setattr(module, "need", need)
    with pytest.raises(Enqueued):  # the sizes as they should be
        wrapper(*args)
    with pytest.raises(ValueError):
        wrapper(*replaced(args, at, shape))


@pytest.mark.gpu
def test_native_ops_refuse():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    cases = calls(arrays("cuda:0"))
    for name, at, shape in BAD:
        op, _, args = cases[name]
        op(*args)
        with pytest.raises(ValueError):
            op(*replaced(args, at, shape))
    torch.cuda.synchronize()


@pytest.mark.gpu
def test_images_of_other_shapes():
    """As many elements in another shape are one image after the other."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from unbiased_differentiable_splatting_gb300.training import L1ImageLoss
    x, y = torch.rand((1, 6, 5, 3), device="cuda:0"), torch.rand((6, 5, 3), device="cuda:0")
    torch.testing.assert_close(L1ImageLoss()(x, y)[0], (x[0] - y).abs().mean(), rtol=1e-6, atol=0)
    with pytest.raises(ValueError):
        L1ImageLoss()(x.repeat(2, 1, 1, 1), x)
