"""The proposal network's gradient over numbered rows: the same bits as over
the rows copied out, at row counts around a tile and around a tile per SM; rows
out of range add nothing; and a workspace off a 16-byte boundary."""
import pytest
import torch

from test_gpu_mlp import DEV, L, init_params  # noqa: F401

pytestmark = pytest.mark.gpu


def run(L, P, X, target, rows=None, shift=0):
    R = X.shape[0] if rows is None else rows.shape[0]
    G, lo = torch.zeros_like(P), torch.zeros(1, device=DEV)
    err = torch.zeros(1, dtype=torch.int32, device=DEV)
    size = L.uds_mlp_grad_workspace_size(R)
    ws = torch.empty(size + shift, dtype=torch.uint8, device=DEV)
    tail = (X.data_ptr(), target.data_ptr(), P.data_ptr(), G.data_ptr(), lo.data_ptr(), err.data_ptr(),
            ws.data_ptr() + shift, size, torch.cuda.current_stream().cuda_stream)
    if rows is None:
        assert L.uds_mlp_grad(R, *tail) == 0
    else:
        assert L.uds_mlp_grad_rows(R, rows.data_ptr(), X.shape[0], *tail) == 0
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    return G, lo


@pytest.mark.parametrize("R", [1, 127, 129, 19456, 20001])
def test_rows(L, R):  # noqa: F811
    g = torch.Generator(device=DEV).manual_seed(R)
    P = init_params(L.uds_mlp_param_count(), seed=R).to(DEV)
    X = torch.randn(3000, 16, device=DEV, generator=g)
    target = torch.rand(3000, device=DEV, generator=g)
    rows = torch.randint(0, 3000, (R,), device=DEV, generator=g)
    a = run(L, P, X, target, rows)
    b = run(L, P, X[rows].contiguous(), target[rows].contiguous(), shift=4)
    assert torch.equal(a[0], b[0]) and torch.equal(a[1], b[1]) and a[0].abs().sum() > 0
    # rows out of range: the other rows' sums, divided by all R
    if R > 1:
        rows[R // 2:] = 3000
        c = run(L, P, X, target, rows)
        n = R // 2
        d = run(L, P, X[rows[:n]].contiguous(), target[rows[:n]].contiguous())
        # scale / R enters before the operands' rounding to bf16 (2^-9 relative)
        assert float((c[0] * (R / n) - d[0]).norm() / d[0].norm()) < 2 ** -8
        torch.testing.assert_close(c[1] * (R / n), d[1], rtol=1e-5, atol=0)
