"""Patch-face fluxes of FP32-bulk tiles at sizes around the tile edges: full,
inside and edge tiles place them in the slots of the missing faces, so the
single-patch kernel and the batched tile shapes (which cut the same patch
into different forms) must agree bit for bit, and all with the FP64 path
within the FP32-bulk bounds (2 steps: L2 1e-5, maximum 1e-4 of each
variable's scale)."""
import numpy as np
import pytest

from drnum_b200 import _lib, cases
from drnum_b200._lib import DN_FP32, DN_FP64
from drnum_b200.api import AusmPlus, B200CartesianIterator, CartesianPatch

pytestmark = pytest.mark.gpu
STEPS = 2


def run(n, periodic, U, h, precision, shape=None):
    it = B200CartesianIterator(AusmPlus(), 0, precision)
    patches = []
    for q in range(1 if shape is None else 2):      # two equal patches: the batched launches
        p = CartesianPatch(*n, spacing=(h, h, h), periodic=periodic)
        p.setField(0, U)
        far = (cases.P_INF, cases.T_INF, 0.3 * cases.A_INF, 10.0, -5.0)
        inflow = cases.jet_table(dict(n=n, length=tuple(m * h for m in n)), 120.0, 310.0, 4 * h, noise=1e-3, p_jet=1.01e5)
        kinds = [(3, None, inflow), (1, far, None), (2, None, None), (1, far, None), (1, far, None), (2, None, None)]
        for side, bc in enumerate(kinds):
            if not periodic[side // 2]:
                p.setBoundary(side, *bc)
        it.addPatch(p)
        patches.append(p)
    it.updateDevice(fields=(0,))
    for q in range(len(patches)):
        if shape is not None:
            it.setTile(q, shape)
    dt = cases.cfl_dt(U, h, 0.2)
    for _ in range(STEPS):
        it.rkStep(dt, cases.RK3_ALPHA)
    it.updateHost(fields=(0,))
    it.close()
    for p in patches[1:]:
        assert np.array_equal(p.getField(0), patches[0].getField(0))
    return patches[0].getField(0).copy()


@pytest.mark.parametrize("n", [(5, 16, 32), (4, 17, 33), (7, 15, 31), (3, 33, 35), (6, 31, 64), (3, 3, 3)])
@pytest.mark.parametrize("periodic", [(False, False, False), (True, False, False), (False, True, False)])
def test_patch_faces_in_every_tile_form(n, periodic):
    h = 1.0 / 32
    U = cases.random_state(*n, seed=3, amp=0.01, mach=0.2)
    ref = run(n, periodic, U, h, DN_FP64)
    one = run(n, periodic, U, h, DN_FP32)
    scale = np.abs(ref).reshape(5, -1).max(axis=1)[:, None, None, None]
    err = (one - ref) / scale
    assert np.sqrt((err ** 2).mean()) < 1e-5 and np.abs(err).max() < 1e-4, (n, periodic, np.abs(err).max())
    for shape in range(_lib.DN_NUM_TILE_SHAPES):
        assert np.array_equal(run(n, periodic, U, h, DN_FP32, shape), one), (n, periodic, shape)
