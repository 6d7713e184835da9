"""FP64 products on the tensor cores: comm222_pp_hhss in the FP64 form against
extended-precision sums, element by element, within the classical bound of an
FP64 sum of K terms, (K + 5) 2^-53 sum |x||w||y| (plus the update's rounding),
which holds for the digit products (sqrt(K) 2^-53 where their guard accepts
them) and for the elements evaluated with FP64 FMAs alike.

Sizes: K from 1 to two chunks (20 blocks of 32), channels from one row over
tile edges (32, 128); weights +-1 and fractional.  Values: the benchmark's,
rows of falling magnitude (elements the digits cannot vouch for), products of
far-off-diagonal elements, zero rows, a channel far below the others, an
infinity."""
import numpy as np
import pytest

import imsrg_gb300 as ig
from modelspace_ref import RefModelSpace

pytestmark = pytest.mark.gpu

U = 2.0**-53
SPACES = {"He4": (4, 2), "O16": (16, 8), "O18": (18, 8), "Ca40": (40, 20)}


def shaped(ms, a, kind, rng):
    N = 2 * ms.n + ms.l
    for ch in range(ms.nch):
        kets = ms.channels[ch][3]
        if not kets:
            continue
        e = np.array([N[p] + N[q] for p, q in kets], dtype=float)
        b = ms.block(a, ch)
        if kind == "graded":
            b *= np.exp2(-1.5 * (e[:, None] + e))
        elif kind == "steep":
            b *= np.exp2(-6.0 * (e[:, None] + e))
        elif kind == "offdiag":
            b *= np.exp2(-4.0 * abs(e[:, None] - e))
        elif kind == "zeros":
            z = rng.random(len(kets)) < 0.4
            b[z, :] = 0
            b[:, z] = 0
            if ch % 3 == 0:
                b *= 2.0**-500  # rows outside the digits' exponent range
        elif kind == "inf" and ch % 4 == 0:
            b[0, -1] = b[-1, 0] = np.inf
    return a


@pytest.mark.parametrize("emax,ref,kind", [(1, "O16", "plain"), (2, "He4", "plain"), (3, "O18", "plain"), (5, "Ca40", "plain"),
                                           (8, "O16", "plain"), (4, "O18", "graded"), (8, "O16", "graded"), (4, "O16", "steep"),
                                           (5, "O18", "offdiag"), (4, "O18", "zeros"), (3, "O16", "inf")])
def test_ladder_elementwise(emax, ref, kind):
    ms = RefModelSpace(emax, *SPACES[ref])
    rng = np.random.default_rng(emax)
    X = shaped(ms, ms.random_operator(11, True), kind, rng)
    Y = shaped(ms, ms.random_operator(12, False), kind, rng)
    Z0 = ms.random_operator(13, True)
    space = ig.ModelSpace(emax, ref, ref)
    with ig.DeviceOperator(space, 1) as dX, ig.DeviceOperator(space, -1) as dY, ig.DeviceOperator(space, 1) as dZ:
        dX.upload(X)
        dY.upload(Y)
        dZ.upload(Z0)
        ig.Commutator.device_term("comm222_pp_hhss", dX, dY, dZ, "fp64")
        Z = dZ.download()
    Q = np.longdouble
    for ch in range(ms.nch):
        kets = ms.channels[ch][3]
        if not kets:
            continue
        # X P Y - X (nn) Y over the kets with a weight (ph kets of full shells have none)
        w = np.array([(1 - ms.occ[p]) * (1 - ms.occ[q]) - ms.occ[p] * ms.occ[q] for p, q in kets])
        k = np.nonzero(w)[0]
        n = len(kets)
        rows = np.arange(n) if n <= 140 else np.sort(rng.choice(n, 10, replace=False))
        x, y, z, z0 = (ms.block(a, ch) for a in (X, Y, Z, Z0))
        with np.errstate(invalid="ignore"):
            wy = (w[k, None] * y[k]).astype(Q)
            wyr = (w[k, None] * y[np.ix_(k, rows)]).astype(Q)
            R = x[np.ix_(rows, k)].astype(Q) @ wy
            T = (x[:, k].astype(Q) @ wyr).T
            S = abs(x[np.ix_(rows, k)]) @ abs(wy) + (abs(x[:, k]) @ abs(wyr)).T
            M = R + T + z0[rows]
            if not np.isfinite(S).all():
                fine = np.isfinite(M)
                assert np.array_equal(fine, np.isfinite(z[rows]))
            else:
                fine = np.ones(M.shape, dtype=bool)
            err = abs(z[rows] - M)
        bound = (len(k) + 5) * U * S + 2 * U * (abs(z[rows]) + abs(z0[rows]))
        worst = float(np.max(err[fine] - bound[fine], initial=-1.0))
        assert worst <= 0, (ch, n, len(k), worst)
