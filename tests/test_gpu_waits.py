"""Waits of one block for another that run out (tests/wait_check.cu, with a
short limit and a tile that never publishes): the block gives up, all of its
threads agree on it, nothing is written out of place, and the failure is
reported (gathers of NaNs, a counter, an error where a view's statistics are
read)."""
import ctypes
import os
import subprocess

import pytest
import torch

DEV = "cuda:0"
HERE = os.path.dirname(os.path.abspath(__file__))
TILE = 16 * 256  # pairs per block of the gather's sort


def test_statistics_of_a_failed_view_raise():
    from unbiased_differentiable_splatting_gb300 import _lib
    from unbiased_differentiable_splatting_gb300.cudaExtensions import sampling
    stats = torch.zeros((3, 8), dtype=torch.float32)
    assert sampling.view_stats(stats)["n_visible"].tolist() == [0, 0, 0]
    stats.view(torch.int32)[1, 6] = 1
    with pytest.raises(_lib.UdsError, match=r"views \[1\]"):
        sampling.view_stats(stats)


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from unbiased_differentiable_splatting_gb300 import _build
    out = str(tmp_path_factory.mktemp("waits") / "libwaits.so")
    subprocess.run([_build._nvcc(), *_build.FLAGS, *_build.ARCH, "-shared", "-cudart", "shared", "-o", out,
                    os.path.join(HERE, "wait_check.cu")], check=True, capture_output=True)
    return ctypes.CDLL(out)


def p(t):
    return ctypes.c_void_p(t.data_ptr())


def stream():
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


def failures(lib):
    n = ctypes.c_uint()
    assert lib.check_failures(ctypes.byref(n)) == 0
    return n.value


@pytest.mark.gpu
@pytest.mark.parametrize("missing", [0, 1, 2, None])
def test_look_back(lib, missing):
    ready, prefix = 1 << 62, -(1 << 63)  # state 2 in the top bits
    words = torch.tensor([prefix | 5, ready | 6, ready | 8, 0], dtype=torch.int64, device=DEV)
    if missing is not None:
        words[missing] = 0
    flag, bad = torch.zeros(1, dtype=torch.int32, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
    count = failures(lib)
    assert lib.check_look_back(p(words), p(flag), p(bad), stream()) == 0
    torch.cuda.synchronize()
    lost = missing is not None
    assert int(flag) == lost and int(bad) == 32 * lost and failures(lib) == count + lost
    if not lost:
        assert int(words[3]) == (prefix | (5 + 6 + 8 + 7))


@pytest.mark.gpu
@pytest.mark.parametrize("value", [0, 1])
def test_flag_is_the_same_for_a_block(lib, value):
    flag = torch.full((1,), value, dtype=torch.int32, device=DEV)
    seen = torch.full((256,), 7, dtype=torch.int32, device=DEV)
    assert lib.check_flag(p(flag), p(seen), stream()) == 0
    assert seen.tolist() == [value] * 256


@pytest.mark.gpu
@pytest.mark.parametrize("first,failed", [(0, 0), (1, 0), (0, 1)])
def test_gather(lib, first, failed):
    """first = 1: the first tile's block never starts, those behind it wait for
    it in vain; failed = 1: an earlier kernel has failed."""
    n, M, C = 3 * TILE + 17, 600, 2
    g = torch.Generator(device=DEV).manual_seed(1)
    keys = torch.randint(0, M, (n,), generator=g, device=DEV, dtype=torch.int32)
    samples = torch.arange(n, device=DEV, dtype=torch.int32)
    hist = torch.bincount(keys, minlength=1024).to(torch.int32)
    words = torch.zeros(4 * 1024, dtype=torch.int32, device=DEV)
    ko, so = (torch.full((n,), -1, dtype=torch.int32, device=DEV) for _ in range(2))
    bounds = torch.zeros((M, 2), dtype=torch.int32, device=DEV)
    values = torch.rand((n, C), generator=g, device=DEV)
    out = torch.zeros((M, C), device=DEV)
    state = torch.zeros(64, dtype=torch.uint8, device=DEV)
    count = failures(lib)
    assert lib.check_gather(n, first, failed, p(hist), p(words), p(keys), p(samples), p(ko), p(so), p(bounds), M, C,
                            p(values), p(out), p(state), stream()) == 0
    torch.cuda.synchronize()
    if first or failed:
        assert torch.isnan(out).all() and not bounds.any()
        assert bool((ko == -1).all()) and failures(lib) == count + (3 if first else 0)
    else:
        order = torch.sort(keys.long(), stable=True).indices
        assert torch.equal(so.long(), order) and torch.equal(ko, keys[order]) and failures(lib) == count
        torch.testing.assert_close(out, torch.zeros_like(out).index_add_(0, keys.long(), values), rtol=1e-5, atol=0)


@pytest.mark.gpu
def test_none_ran_out():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from unbiased_differentiable_splatting_gb300 import _lib
    assert _lib.wait_failures() == 0 == _lib.wait_failures(torch.device(DEV))
