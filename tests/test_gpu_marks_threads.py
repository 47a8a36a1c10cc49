"""EWA weights of scenes of different sizes from several host threads: the
marks' bit maps ask for more than 48 KB of shared memory from 393,216 splats
on, which is an attribute of the kernel and not of the launch."""
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def test_launches_of_different_sizes():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from unbiased_differentiable_splatting_gb300 import _lib
    L = _lib.load()
    W, H, K, f = 128, 32, 8, 100.0
    failed = []

    def run(N, seed):
        g = torch.Generator(device=DEV).manual_seed(seed)
        p = torch.rand((1, N, 3), generator=g, device=DEV) - torch.tensor([0.5, 0.5, 2.0], device=DEV)
        n = torch.tensor([0.0, 0.0, -1.0], device=DEV).repeat(1, N, 1)
        sd = torch.full((1, N, 2), 0.5, device=DEV)
        idx = torch.randint(-1, N, (1, W, H, K), generator=g, device=DEV, dtype=torch.int32)
        ws = torch.empty(L.uds_splat_workspace_size(1, N), dtype=torch.uint8, device=DEV)
        stream = torch.cuda.Stream()
        outs = [torch.empty((1, W, H, K), device=DEV) for _ in range(2)]
        torch.cuda.synchronize()
        ready.wait()
        for k in range(3000):
            st = L.uds_splat_forward(1, W, H, K, f, idx.data_ptr(), p.data_ptr(), n.data_ptr(), 1, N, sd.data_ptr(),
                                     0.0, outs[min(k, 1)].data_ptr(), ws.data_ptr(), ws.numel(), stream.cuda_stream)
            if st:
                failed.append((N, k, st, L.uds_last_error()))
                return
            if k % 100 == 99:
                stream.synchronize()
        stream.synchronize()
        if not torch.equal(*outs):
            failed.append((N, "values"))

    sizes = (1 << 20, 400_000, 1_000_000, 450_000)
    ready = threading.Barrier(len(sizes))
    threads = [threading.Thread(target=run, args=(N, s)) for s, N in enumerate(sizes)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed
