"""Scratch buffers of the Python wrappers: calls that may run at the same time
(two streams, two threads) have buffers of their own, since the kernels keep
tickets and look-back words in them; and the results of such calls."""
import threading

import numpy as np
import pytest
import torch

from unbiased_differentiable_splatting_gb300 import _lib

DEV = "cuda:0"


def test_no_two_calls_share_a_buffer():
    cpu = torch.device("cpu")
    held = [_lib.Workspace.get(cpu, 1000, "sample") for _ in range(2)]
    threads = [threading.Thread(target=lambda: held.append(_lib.Workspace.get(cpu, 1000, "sample")))
               for _ in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    spans = sorted((b.data_ptr(), b.data_ptr() + b.numel()) for b in held)
    assert len(spans) == 4 and all(b.numel() >= 1000 for b in held)
    assert all(a[1] <= b[0] for a, b in zip(spans, spans[1:]))


def _scene(seed, N=40_000, W=96, H=80):
    rng = np.random.default_rng(seed)
    z = rng.uniform(-2.4, -1.6, N)
    p = np.stack([rng.uniform(-0.5, 0.5, N) * -z, rng.uniform(-0.5, 0.5, N) * -z, z], 1).astype(np.float32)
    n = rng.normal(size=(N, 3))
    n[:, 2] = np.abs(n[:, 2]) + 0.5
    n = (n / np.linalg.norm(n, axis=1, keepdims=True)).astype(np.float32)
    t = lambda a: torch.as_tensor(a).to(DEV)  # noqa: E731
    return W, H, float(W), t(p[None]), t(n[None]), t(np.full((1, N, 2), 0.01, np.float32))


@pytest.mark.gpu
@pytest.mark.parametrize("threads", [False, True])
def test_calls_side_by_side(threads):
    """Trees, descents and gathers of different scenes enqueued on four
    streams, from one thread or four, give what they give alone."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from unbiased_differentiable_splatting_gb300.cudaExtensions import pixelgather, sampling
    scenes = [_scene(s, N) for s, N in enumerate((40_000, 9_000, 70_000, 25_000))]

    def work(k):
        W, H, f, p, n, sd = scenes[k]
        idx = sampling.sample(W, H, f, p, n, None, sd, 8, 0.0, 0.01, seed=k)
        si, sp = sampling.sample_stochastic(W, H, f, p, n, sd, 4, 0.0, 0.01, seed=k)
        g = pixelgather.gather(idx, sp.repeat(1, 1, 1, 2)[..., None].contiguous(), p.shape[1], deterministic=True)
        return idx, si, sp, g

    alone = [work(k) for k in range(4)]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(4)]
    got = [[] for _ in range(4)]

    def many(k):
        with torch.cuda.stream(streams[k]):
            for _ in range(6):
                got[k].append(work(k))

    if threads:
        ts = [threading.Thread(target=many, args=(k,)) for k in range(4)]
        for t in ts:
            t.start()
        for t in ts:
            t.join()
    else:
        for _ in range(6):
            for k in range(4):
                with torch.cuda.stream(streams[k]):
                    got[k].append(work(k))
    torch.cuda.synchronize()
    for k in range(4):
        for out in got[k]:
            for a, b in zip(out, alone[k]):
                assert torch.equal(a, b)


@pytest.mark.gpu
def test_tree_freed_before_its_evaluation_has_run():
    """A tree's memory is not given out again while a side stream reads it."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from unbiased_differentiable_splatting_gb300.cudaExtensions import sampling
    W, H, f, p, n, sd = _scene(5, 20_000)
    nodes = torch.arange(64, dtype=torch.int32, device=DEV)
    queries = torch.rand((64, 2), device=DEV) * torch.tensor([W, H], device=DEV)
    tree = sampling.build_tree(W, H, f, p, n, sd, 8, 0.0, 0.01)
    expected = sampling.fgt_eval(tree, nodes, queries)
    bytes_, at = tree["_ws"].numel(), tree["_ws"].data_ptr()
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        torch.cuda._sleep(50_000_000)  # clock cycles: some 25 ms
        got = sampling.fgt_eval(tree, nodes, queries)
    del tree
    other = torch.empty(bytes_, dtype=torch.uint8, device=DEV)
    assert other.data_ptr() != at  # still held for the side stream
    torch.cuda.synchronize()
    assert torch.equal(got, expected) and bool((expected > 0).any())
