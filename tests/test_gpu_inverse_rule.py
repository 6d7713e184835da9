"""The inverse Pandya kernel a commutator takes where neither a call nor the
tuning file chose one (the descriptors), against the channel tiles and
quadruple blocks it takes when told so.  FP64: the same sums in another order,
a dozen terms an element: 1e-14 of the largest.  Split: the same products'
Z bar, double-float sums good to 2^-44 = 6e-14 a term: 1e-12."""
import numpy as np
import pytest

import imsrg_gb300 as ig
from modelspace_ref import RefModelSpace

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,key,tol", [("fp64", b"inverse.fp64", 1e-14), ("split", b"inverse.split", 1e-12)])
@pytest.mark.parametrize("emax,nucleus,herms", [(1, "O16", (1, -1)), (2, "O16", (1, 1)), (4, "O18", (1, -1)), (7, "O16", (-1, 1))])
def test_default_inverse_vs_explicit(emax, nucleus, herms, prec, key, tol, monkeypatch):
    monkeypatch.setenv("IMSRG_GB300_TUNING", "off")
    ref = RefModelSpace(emax, *{"O16": (16, 8), "O18": (18, 8)}[nucleus])
    arenas = [ref.random_operator(40 + k, h == 1) for k, h in enumerate(herms)]
    space = ig.ModelSpace(emax, nucleus, nucleus)
    hz = -1 if herms[0] == herms[1] else 1
    with ig.DeviceOperator(space, herms[0]) as dX, ig.DeviceOperator(space, herms[1]) as dY, ig.DeviceOperator(space, hz) as dZ:
        dX.upload(arenas[0])
        dY.upload(arenas[1])
        assert space.tuning()[key.decode()] == 0
        ig.Commutator.device_commutator(dX, dY, dZ, prec)
        got = dZ.download()
        assert ig.lib().imsrg_space_set_tuning(space._h, key, 0) == 0
        ig.Commutator.device_commutator(dX, dY, dZ, prec)
        want = dZ.download()
    assert np.linalg.norm(want) > 0
    assert np.max(abs(got - want)) <= tol * np.max(abs(want))
