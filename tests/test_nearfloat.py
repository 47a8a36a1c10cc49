"""The float evaluation of the reference's two double expressions
(csrc/uds_nearfloat.cuh) against the double formulas, bit for bit, on random
and edge-case inputs (host build of the header the kernels use)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "unbiased_differentiable_splatting_gb300", "csrc")


def test_matches_double(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    exe = str(tmp_path / "nearfloat_check")
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I", CSRC,
                    os.path.join(HERE, "nearfloat_check.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe, "2000000"], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
    n_rem, fast_rem, bad_rem, n_q, fast_q, bad_q = (int(v) for v in out.stdout.split()[-6:])
    assert bad_rem == 0 and bad_q == 0
    assert n_rem > 8_000_000 and n_q > 8_000_000
    # the exact paths stay rare (products and quotients with few significant
    # bits, which end on the boundary, are a fifth of the inputs here)
    assert fast_rem > 0.9 * n_rem and fast_q > 0.9 * n_q
