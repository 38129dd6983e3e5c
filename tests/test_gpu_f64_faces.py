"""FP64 faces at the edges of their fast evaluation (fv_f64.cuh): operands the
guard sends to the plain expressions, zero and tiny differences, all at sizes
around the tile edges, equal to the oracle restatement (as numbers: only the
sign of a zero may differ)."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle"))
import pyoracle  # noqa: E402
from drnum_b200 import cases  # noqa: E402
from drnum_b200._lib import DN_FP64  # noqa: E402
from drnum_b200.api import AusmPlus, B200CartesianIterator, CartesianPatch  # noqa: E402

pytestmark = pytest.mark.gpu


def ones_mantissa(U, rng):
    """Every third cell's values with the upper significand bits all ones."""
    b = U.view(np.uint64).copy()
    sel = rng.random(U.shape) < 0.33
    b[sel] |= np.uint64(0x000FFFFF00000000)
    return b.view(np.float64)


def state(kind, n, seed=5):
    rng = np.random.default_rng(seed)
    U = cases.random_state(*n, seed=seed, amp=0.01, mach=0.3)
    if kind == "uniform":                       # zero differences everywhere but in a few cells
        V = cases.uniform_state([dict(n=n)], mach=0.3)[0]
        V[:, n[0] // 2, n[1] // 2] = U[:, n[0] // 2, n[1] // 2]
        return V
    if kind == "tiny":                          # momenta down to subnormals, both zeros
        for q in (2, 3):
            U[q] = np.ldexp(rng.uniform(-1, 1, n), rng.integers(-1080, -200, n))
            U[q][rng.random(n) < 0.2] = 0.0
            U[q][rng.random(n) < 0.2] = -0.0
        return U
    if kind == "ones":
        return ones_mantissa(U, rng)
    if kind == "supersonic":                    # |M| around and beyond 1, both directions
        p, T, u, v, w = cases.cons_to_prim(U)
        a = cases.A_INF
        return cases.prim_to_cons(p, T, u + rng.choice([-2.0, -1.0, 0.7, 1.5], n) * a, v + a, w - 1.2 * a)
    if kind == "small_scale":                   # outside the guarded range: every face by the plain expressions
        return U * 1e-100
    return U * 1e95                             # large_scale


@pytest.mark.parametrize("kind", ["uniform", "tiny", "ones", "supersonic", "small_scale", "large_scale"])
@pytest.mark.parametrize("n,periodic", [((5, 4, 32), (True, True, True)), ((4, 9, 33), (False, False, False)),
                                        ((3, 5, 66), (True, False, True)), ((9, 3, 7), (False, True, False))])
def test_guarded_faces_equal_the_oracle(kind, n, periodic):
    U = state(kind, n)
    h = 1.0 / 16
    dt = 0.05 * h / (4.0 * cases.A_INF)
    steps = 2
    patch = CartesianPatch(*n, spacing=(h, h, h), periodic=periodic)
    patch.setField(0, U)
    it = B200CartesianIterator(AusmPlus(), 0, DN_FP64)
    it.addPatch(patch)
    it.updateDevice(fields=(0,))
    for _ in range(steps):
        it.rkStep(dt, cases.RK3_ALPHA)
    it.updateHost(fields=(0,))
    it.close()
    ref = pyoracle.oracle_run(U, h, dt, steps, periodic=periodic)
    assert np.isfinite(ref).all()
    out = patch.getField(0)
    assert np.array_equal(out, ref), np.abs(out - ref).max() / np.abs(ref).max()
