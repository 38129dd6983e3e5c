"""What the autotuner spends and what it changes, with given tile shape costs (a
cache file), so that nothing of its trials depends on a clock."""
import time

import numpy as np
import pytest

from drnum_b200 import cases
from drnum_b200._lib import DN_FP32, DN_FP64, DN_OPT_BATCH_MIN_PLANES
from drnum_b200.api import AusmPlus, B200CartesianIterator, CartesianPatch, Roe, VanLeer

pytestmark = pytest.mark.gpu


def iterator(extents, precision, scheme=AusmPlus):
    it = B200CartesianIterator(scheme(), 0, precision)
    for n in extents:
        p = CartesianPatch(*n, spacing=(0.1,) * 3, periodic=(True,) * 3)
        p.setField(0, cases.random_state(*n, seed=1, amp=0.01, mach=0.2))
        it.addPatch(p)
    it.updateDevice(fields=(0,))
    return it


@pytest.fixture
def equal_costs(tmp_path):
    """A cache file with the same cost for every tile shape."""
    def make(precision):
        path = tmp_path / "tune.txt"
        it = iterator([(8, 8, 32), (8, 8, 32)], precision)
        cost = it.autotune(path)
        it.close()
        line = path.read_text().strip().split("|")
        path.write_text("|".join(line[:-len(cost)] + ["1"] * len(cost)) + "\n")
        return path
    return make


def test_trials_of_a_grid(equal_costs):
    # an 8 x 32 and a 16 x 16 cross-section: per-patch shapes differ, so every
    # uniform shape is tried as well; eight trials of five stages, two launches each
    path = equal_costs(DN_FP32)
    it = iterator([(16, 8, 32), (16, 16, 16)], DN_FP32)
    before = it.launchCount()
    assert np.array_equal(it.autotune(path), np.ones(3))
    assert 0 < it.launchCount() - before <= 8 * 5 * 2
    it.close()


@pytest.mark.parametrize("precision", [DN_FP64, DN_FP32])
def test_trials_of_a_patch(equal_costs, precision):
    # a lone patch: its plane ranges, six of seven stages at most
    path = equal_costs(precision)
    it = iterator([(64, 32, 32)], precision)
    before = it.launchCount()
    assert np.array_equal(it.autotune(path), np.ones(3))
    assert 0 < it.launchCount() - before <= 6 * 7
    it.close()


def test_default_range_comes_back():
    # FP64 patches of few columns: the default takes ranges of a plane or two,
    # 32 planes are many times slower, and setting the default again is the default
    it = iterator([(64, 16, 32), (64, 16, 32)], DN_FP64)

    def step():
        best = 1e9
        for _ in range(20):
            it.sync()
            t = time.perf_counter()
            it.rkStep(1e-9, cases.RK3_ALPHA)
            it.sync()
            best = min(best, time.perf_counter() - t)
        return best

    default = step()
    it.setOption(DN_OPT_BATCH_MIN_PLANES, 32)
    assert step() > 3 * default
    it.setOption(DN_OPT_BATCH_MIN_PLANES, 8)
    assert step() < 1.5 * default
    it.close()


def test_cache_keeps_schemes_apart(tmp_path):
    # each scheme reads its own costs, none those of another or of a line without a scheme
    path = tmp_path / "tune.txt"
    costs = {}
    for scheme in (AusmPlus, VanLeer, Roe):
        it = iterator([(16, 8, 32), (16, 16, 16)], DN_FP64, scheme)
        costs[scheme] = it.autotune(path)
        it.close()
    lines = path.read_text().splitlines()
    assert len(lines) == 3
    device, precision = lines[0].split("|")[:2]
    path.write_text("%s|%s|3|1|1|1\n" % (device, precision) + "\n".join(lines) + "\n")
    for scheme, cost in costs.items():
        it = iterator([(16, 8, 32), (16, 16, 16)], DN_FP64, scheme)
        assert np.array_equal(it.autotune(path), cost)
        it.close()
    assert len(path.read_text().splitlines()) == 4
