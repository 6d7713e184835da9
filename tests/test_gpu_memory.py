"""FP64 calls where device memory is nearly used up: the digit planes and
descriptors only make a call faster, so they may not take the room that its
scratch, or an operator created later, needs.  Memory is held down by one large
allocation that nothing touches."""
import numpy as np
import pytest

import imsrg_gb300 as ig
from modelspace_ref import RefModelSpace

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

MB = 1 << 20


def hold(leave):
    """An allocation that leaves about that many bytes free, or None."""
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    return torch.empty(free - leave, dtype=torch.uint8, device="cuda") if free > leave else None


def operators(space, n):
    return [ig.DeviceOperator(space, 1 if k != 1 else -1) for k in range(n)]


def test_scratch_comes_before_planes():
    """At emax 8 a commutator's scratch is some 150 MB, its descriptors 140 and its
    planes 450.  From the scratch upwards (and 250 MB for the runtime, which takes
    memory in pieces) every amount has to do, down each step of what else fits."""
    ms = RefModelSpace(8, 16, 8)
    X, Y = ms.random_operator(1, True), ms.random_operator(2, False)
    want = None
    for leave in [None] + [400 * MB + 60 * MB * k for k in range(14)]:
        space = ig.ModelSpace(8, "O16", "O16")
        dX, dY, dZ = operators(space, 3)
        dX.upload(X)
        dY.upload(Y)
        held = None if leave is None else hold(leave)
        try:
            ig.Commutator.device_commutator(dX, dY, dZ, "fp64")
            Z = dZ.download()
        finally:
            del held
            torch.cuda.empty_cache()
        want = Z if want is None else want
        assert np.max(abs(Z - want)) <= 1e-13 * np.max(abs(want)), leave


def test_planes_make_room_for_operators():
    space = ig.ModelSpace(8, "O16", "O16")
    dX, dY, dZ = operators(space, 3)
    dX.fill_random(1)
    dY.fill_random(2)
    ig.Commutator.device_commutator(dX, dY, dZ, "fp64")
    want = dZ.download()
    held = hold(30 * MB)  # an operator takes 56
    try:
        more = operators(space, 2)
        ig.Commutator.device_commutator(dX, dY, more[0], "fp64")
        Z = more[0].download()
    finally:
        del held
        torch.cuda.empty_cache()
    assert np.max(abs(Z - want)) <= 1e-13 * np.max(abs(want))
    ig.Commutator.device_commutator(dX, dY, dZ, "fp64")  # and the planes come back
    assert np.max(abs(dZ.download() - want)) <= 1e-13 * np.max(abs(want))


def test_captured_planes_stay():
    """A graph holds on to the planes it was captured with: they are not given up."""
    space = ig.ModelSpace(8, "O16", "O16")
    dX, dY, dZ = operators(space, 3)
    dX.fill_random(1)
    dY.fill_random(2)
    batch = ig.CommutatorBatch([(dX, dY, dZ), (dX, dY, ig.DeviceOperator(space, 1))], "fp64")
    want = dZ.download()
    held = hold(30 * MB)
    try:
        with pytest.raises(ig.IMSRGError):
            operators(space, 2)
        dZ.zero()
        batch.launch()
        batch.sync()
        Z = dZ.download()
    finally:
        del held
        torch.cuda.empty_cache()
    assert np.array_equal(Z[32:], want[32:])
