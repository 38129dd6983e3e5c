"""AUSM+, VanLeer and Roe in the fused FP64 stage: their fast fluxes against the
plain expressions at the edges of every guard, and every launch form of a grid
(per patch, batched tile shapes, schedules, tuned) against one another."""
import os
import subprocess

import numpy as np
import pytest

from drnum_b200 import build, cases
from drnum_b200._lib import DN_FP64, DN_OPT_BATCH_MIN_PLANES, DN_OPT_BATCHED, DN_OPT_GRAPH
from drnum_b200.api import AusmPlus, Roe, VanLeer
from test_gpu_grid import make_grid

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


def test_guarded_fluxes_equal_the_plain_ones(tmp_path):
    exe = str(tmp_path / "f64_schemes")
    cmd = [build.nvcc(), *build.ARCH, "-O3", "-std=c++17", "-fmad=false", "--expt-relaxed-constexpr", "-I", build.CSRC,
           "-I", build.INCLUDE, "-o", exe, os.path.join(HERE, "f64_schemes.cu")]
    res = subprocess.run(cmd, capture_output=True, text=True)
    assert res.returncode == 0, res.stderr
    res = subprocess.run([exe], capture_output=True, text=True)
    assert res.returncode == 0, res.stdout + res.stderr
    passed = {tuple(line.split()[:2]): int(line.split()[2]) for line in res.stdout.splitlines()}
    assert len(passed) == 27 and min(passed.values()) > 0, passed


def states(name, scheme, batched=1, shapes=None, min_planes=None, tune=False, graph=0):
    it, objs, _, dt, _ = make_grid(name, DN_FP64, op=scheme())
    it.setOption(DN_OPT_BATCHED, batched)
    it.setOption(DN_OPT_GRAPH, graph)
    if min_planes:
        it.setOption(DN_OPT_BATCH_MIN_PLANES, min_planes)
    if shapes:
        for q in range(len(objs)):
            it.setTile(q, shapes[q % len(shapes)])
    if tune:
        it.autotune()
    for _ in range(3):
        it.rkStep(dt, cases.RK3_ALPHA)
    it.updateHost(fields=(0,))
    it.close()
    return [cp.getField(0).copy() for cp in objs]


@pytest.mark.parametrize("scheme", [AusmPlus, VanLeer, Roe])
@pytest.mark.parametrize("name", ["octants_jet", "sphere_pair", "octants_ragged"])
def test_launch_forms_give_the_same_bits(name, scheme):
    ref = states(name, scheme, batched=0)
    for kw in (dict(), dict(shapes=[0]), dict(shapes=[1]), dict(shapes=[2]), dict(shapes=[2, 0, 1], min_planes=1),
               dict(min_planes=24), dict(tune=True), dict(tune=True, graph=1), dict(batched=0, tune=True)):
        for a, b in zip(ref, states(name, scheme, **kw)):
            assert np.array_equal(a, b), (name, scheme.__name__, kw)
