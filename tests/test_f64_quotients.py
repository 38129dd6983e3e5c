"""Exactness of the FP64 face quotients (csrc/fv_f64.cuh) for every denominator
their guard lets pass: the kernel's arithmetic on the host, next to midpoints of
two doubles, and the error of the reciprocal seed on the GPU over all its inputs
against what the arithmetic asks for."""
import os
import shutil
import subprocess

import pytest

from drnum_b200 import build

HERE = os.path.dirname(os.path.abspath(__file__))


def run(cmd, **kw):
    res = subprocess.run(cmd, capture_output=True, text=True, **kw)
    return res.returncode, res.stdout + res.stderr


def test_guarded_quotients_next_to_midpoints(tmp_path):
    exe = str(tmp_path / "f64_quotients")
    rc, out = run([shutil.which("g++"), "-O2", "-march=native", "-ffp-contract=off", "-std=c++17", "-Wno-unknown-pragmas",
                   "-I", build.CSRC, "-o", exe, os.path.join(HERE, "f64_quotients.cpp")])
    assert rc == 0, out
    rc, out = run([exe, "300000"])
    assert rc == 0, out


@pytest.mark.gpu
def test_reciprocal_seed_error(tmp_path):
    exe = str(tmp_path / "f64_seed")
    rc, out = run([build.nvcc(), *build.ARCH, "-O2", "-std=c++17", "--expt-relaxed-constexpr", "-I", build.CSRC, "-o",
                   exe, os.path.join(HERE, "f64_seed.cu")])
    assert rc == 0, out
    rc, out = run([exe])
    assert rc == 0, out
    e, room = map(float, out.split())
    assert e < 2.0 ** -19.9 and room > 1.0, out
