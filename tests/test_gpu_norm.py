"""Operator::Norm on the device against the sum written out, and the same sum
beside the BCH update: sqrt(sum (2 j_p + 1) O_pq^2 + sum (2 J + 1)^2 V^2), in
pieces of 8192 two-body and 512 one-body elements.  A sum of positive terms is
off by at most (its longest chain of additions + 2) 2^-53 of itself, here a
few thousand partial sums: 4e-13 / 2 after the root."""
import numpy as np
import pytest

import imsrg_gb300 as ig
from modelspace_ref import RefModelSpace

pytestmark = pytest.mark.gpu


def norm(ms, a):
    one = ms.onebody(a)
    j = np.array(ms.j2)
    same = np.array([[(ms.l[p], ms.j2[p], ms.tz2[p]) == (ms.l[q], ms.j2[q], ms.tz2[q]) for q in range(ms.norb)]
                     for p in range(ms.norb)])
    s = float(np.sum(np.where(same, one**2 * (j + 1)[:, None], 0.0)))
    for ch in range(ms.nch):
        s += float(np.sum(ms.block(a, ch)**2)) * (2 * ms.channels[ch][0] + 1)**2
    return np.sqrt(s)


@pytest.mark.parametrize("emax", [0, 1, 4, 7])
def test_norm(emax):
    ms = RefModelSpace(emax, 4, 2) if emax == 0 else RefModelSpace(emax, 16, 8)
    X = ms.random_operator(3, True)
    space = ig.ModelSpace(emax, *(("He4",) * 2 if emax == 0 else ("O16",) * 2))
    with ig.DeviceOperator(space, 1) as d:
        d.upload(X)
        got = d.norm()
    want = norm(ms, X)
    assert abs(got - want) <= 2e-13 * want


@pytest.mark.parametrize("emax", [1, 3])
def test_bch_update_and_norm(emax):
    """The transform against its loop in separate launches: as many nested
    commutators, the same sum (each of its up to 40 additions off by 2^-53)."""
    ms = RefModelSpace(emax, 16, 8)
    H, om = ms.random_operator(4, True), ms.random_operator(5, False)
    om *= 0.05 / norm(ms, om)
    space = ig.ModelSpace(emax, "O16", "O16")
    with ig.DeviceOperator(space, 1) as dH, ig.DeviceOperator(space, -1) as dO, ig.DeviceOperator(space, 1) as dZ, \
            ig.DeviceOperator(space, 1) as a, ig.DeviceOperator(space, 1) as b:
        dH.upload(H)
        dO.upload(om)
        taken = ig.BCH.device_transform(dH, dO, dZ, "fp64")
        # the reference's rule (src/BCH.cc:87-201) with norms of their own launches
        nx, ny = dH.norm(), dO.norm()
        eps = nx * np.exp(-2 * ny) * ig.BCH.bch_transform_threshold / (2 * ny)
        a.upload(H)
        out, f, want = H.copy(), 1.0, 0
        for i in range(1, 41):
            ig.Commutator.device_commutator(dO, a, b, "fp64")
            a, b = b, a
            f /= i
            out += f * a.download()
            eps *= i + 1
            want = i
            if a.norm() < eps:
                break
        assert taken == want
        Z = dZ.download()
    assert np.max(abs(Z - out)) <= 1e-13 * np.max(abs(out))
