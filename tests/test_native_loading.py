"""When the native implementations of torch.ops.uds are built and loaded:
importing the package and tracing its ops need neither compiled library; one
built for another torch or Python is rebuilt; and what happens where it cannot
be."""
import os
import shutil
import subprocess
import sys

import pytest
import torch

from unbiased_differentiable_splatting_gb300 import _build, _lib

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PACKAGE = "unbiased_differentiable_splatting_gb300"

IMPORTS = f"""
import torch
from {PACKAGE} import _build
def build(*a, **k):
    raise SystemExit("a compiler was called")
_build.build = build
from {PACKAGE} import extensions, library, regularizers, render, scenes, training
training.L1ImageLoss()
regularizers.NearestSamplesRegularizer(sigma=1.0)
m = lambda *s: torch.empty(s, device="meta")
assert torch.ops.uds.affine_forward(m(2, 4, 4), m(1, 7, 3)).shape == (2, 7, 3)
assert torch.ops.uds.image_loss(m(2, 3), m(2, 3), 0, 1.0)[1].shape == (2, 3)
print([l for l in open("/proc/self/maps") if "libuds" in l])
"""


def test_imports_without_the_libraries(tmp_path):
    shutil.copytree(os.path.join(ROOT, PACKAGE), tmp_path / PACKAGE,
                    ignore=shutil.ignore_patterns("*.so", "_build", "__pycache__"))
    r = subprocess.run([sys.executable, "-c", IMPORTS], cwd=tmp_path, capture_output=True, text=True,
                       env={**os.environ, "PYTHONPATH": str(tmp_path)})
    assert r.returncode == 0, r.stderr
    assert r.stdout.strip() == "[]"


@pytest.fixture
def loads(monkeypatch, tmp_path):
    """load_ops with the build and the loading replaced; returns their calls."""
    calls = []
    monkeypatch.setattr(_build, "OPS_STAMP", str(tmp_path / "stamp"))
    monkeypatch.setattr(_build, "OPS_LIB", str(tmp_path / "libuds_torch.so"))
    monkeypatch.setattr(_build, "build", lambda *a, **k: calls.append("build"))
    monkeypatch.setattr(torch.ops, "load_library", lambda path: calls.append("load"))
    monkeypatch.setattr(_lib, "_ops_loaded", False)
    monkeypatch.setattr(_lib, "_lib", object())
    (tmp_path / "libuds_torch.so").write_bytes(b"")
    return calls


@pytest.mark.parametrize("stamp,expected", [(None, ["build", "load"]), ("torch 1.0, cpython-30\n", ["build", "load"]),
                                            ("this", ["load"])])
def test_rebuilt_for_another_torch(loads, stamp, expected):
    if stamp is not None:
        with open(_build.OPS_STAMP, "w") as f:
            f.write(_build._ops_target() if stamp == "this" else stamp)
    assert _build.ops_built() == (stamp == "this")
    _lib.load_ops()
    _lib.load_ops()
    assert loads == expected


def test_python_definitions_stay_where_it_cannot_be_built(loads, monkeypatch):
    def build(*a, **k):
        raise RuntimeError("no compiler")

    monkeypatch.setattr(_build, "build", build)
    with pytest.warns(RuntimeWarning, match="no compiler"):
        _lib.load_ops()
    assert loads == []


def test_build_is_up_to_date():
    _build.build()
    assert _build.ops_built() and _build._ops_up_to_date() and _build.up_to_date()


@pytest.mark.gpu
def test_native_after_the_first_call():
    """The native code is what runs on a GPU (no silent fallback)."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from unbiased_differentiable_splatting_gb300 import library  # noqa: F401
    x = torch.rand((1, 2, 2, 3), device="cuda:0")
    torch.ops.uds.image_loss(x, x, 0, 1.0)
    assert any("libuds_torch.so" in line for line in open("/proc/self/maps"))
    for key in ("CUDA", "AutogradCUDA"):
        assert torch._C._dispatch_has_kernel_for_dispatch_key("uds::image_loss", key)
