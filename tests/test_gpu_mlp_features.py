"""Feature rows and targets as ProposalNet takes them: rows whose storage does
not start on 16 bytes (copied), targets of other lengths, and what is refused
before a launch."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def proposal():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from unbiased_differentiable_splatting_gb300 import _lib, proposal
    _lib.load()
    return proposal


def _rows(n):
    g = torch.Generator(device=DEV).manual_seed(n)
    return torch.randn(n, 16, device=DEV, generator=g), torch.rand(n, device=DEV, generator=g)


def _moved(t, by):
    """The same values with their storage `by` floats further on."""
    out = torch.empty(t.numel() + by, device=DEV)[by:].view(t.shape)
    out.copy_(t)
    return out


@pytest.mark.parametrize("by", [1, 2, 3, 5])
def test_rows_off_a_boundary(proposal, by):
    X, t = _rows(700)
    a, b = (proposal.ProposalNet(DEV, seed=3) for _ in range(2))
    moved = _moved(X, by)
    assert moved.data_ptr() % 16 and moved.is_contiguous()
    la = a.train(X, t, steps=3, batch=256)
    lb = b.train(moved, _moved(t, by), steps=3, batch=256)
    assert torch.equal(la, lb) and torch.equal(a.params, b.params)
    assert torch.equal(a.logits(X), b.logits(moved)) and not b.failed()


def test_targets(proposal):
    X, t = _rows(300)
    nets = [proposal.ProposalNet(DEV, seed=4) for _ in range(4)]
    longer = torch.cat([t, torch.full((50,), float("nan"), device=DEV)])  # never read
    losses = [n.train(X, y, steps=2, batch=128) for n, y in zip(nets, (t, longer, t[:, None].contiguous()))]
    assert torch.equal(losses[0], losses[1]) and torch.equal(losses[0], losses[2])
    for bad in (t[:-1], torch.stack([t, t], 1), t[0]):
        with pytest.raises(ValueError):
            nets[3].train(X, bad.contiguous(), steps=1)


@pytest.mark.parametrize("cols", [8, 15, 17])
def test_other_widths_are_refused(proposal, cols):
    net = proposal.ProposalNet(DEV, seed=5)
    X = torch.zeros(64, cols, device=DEV)
    with pytest.raises(ValueError):
        net.logits(X)
    with pytest.raises(ValueError):
        net.train(X, torch.zeros(64, device=DEV), steps=1)


def test_entry_points_refuse_misaligned_rows(proposal):
    from unbiased_differentiable_splatting_gb300 import _lib
    L = _lib.load()
    X, t = _rows(64)
    net = proposal.ProposalNet(DEV, seed=6)
    at, out = _moved(X, 1).data_ptr(), torch.empty(64, 2, device=DEV)
    rows = torch.arange(64, device=DEV)
    ws = torch.empty(L.uds_mlp_grad_workspace_size(64), dtype=torch.uint8, device=DEV)
    loss, err = torch.zeros(1, device=DEV), net._err.data_ptr()
    s = torch.cuda.current_stream().cuda_stream
    tail = (t.data_ptr(), net.params.data_ptr(), net.grad.data_ptr(), loss.data_ptr(), err, ws.data_ptr(), ws.numel(), s)
    assert L.uds_mlp_forward(64, at, net.params.data_ptr(), out.data_ptr(), err, s) == 1
    assert L.uds_mlp_forward_dev(64, rows.data_ptr(), at, net.params.data_ptr(), out.data_ptr(), err, s) == 1
    assert L.uds_mlp_grad(64, at, *tail) == 1
    assert L.uds_mlp_grad_rows(64, rows.data_ptr(), 64, at, *tail) == 1
