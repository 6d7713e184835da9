"""comm222_pp_hhss in the split form where five 8-bit digits in chunks are taken
(a reduction above 339), element by element.  With 2^a_i the common power of
two above a row's entries of X and, c apart, of the weighted Y, every product
of the doubled reduction is off by at most 2^(a_i + a_j + c) times

  2^-38           the two operands' last digit rounded to 38 bits
  2^-36 x 1.01    the digit products left out (four of the first dropped weight:
                  4 x 2^14 x 2^24 / 2^76, and less below)
  2^-37           the two lowest kept groups' FP32 sums, where they pass 2^24

which is below 2^-35; the leading groups' sums and the chunks' are exact."""
import numpy as np
import pytest

import imsrg_gb300 as ig
from modelspace_ref import RefModelSpace

pytestmark = pytest.mark.gpu


def shaped(ms, a, kind, rng, anti):
    for ch in range(ms.nch):
        if not ms.channels[ch][3]:
            continue
        b = ms.block(a, ch)
        n = b.shape[0]
        if kind == "coherent":  # every digit near its largest, all of one sign (Y: of its triangle's)
            q = 63 * 2.0**32 + 127 * (2.0**24 + 2.0**16 + 2.0**8 + 1)
            b[:] = q * 2.0**-38
            if anti:
                b *= np.sign(np.subtract.outer(np.arange(n), np.arange(n)))
        elif kind == "halves":  # alternating extremes, rows far apart
            g = np.exp2(-(np.arange(n) % 7) * 3.0)
            b *= np.minimum.outer(g, g)
    return a


@pytest.mark.parametrize("emax,nucleus,kind", [(8, "O16", "plain"), (8, "O18", "coherent"), (9, "O16", "coherent"),
                                               (8, "O16", "halves")])
def test_ladder_five_digits_elementwise(emax, nucleus, kind):
    ms = RefModelSpace(emax, *{"O16": (16, 8), "O18": (18, 8)}[nucleus])
    rng = np.random.default_rng(emax)
    X = shaped(ms, ms.random_operator(21, True), kind, rng, False)
    Y = shaped(ms, ms.random_operator(22, False), kind, rng, True)
    space = ig.ModelSpace(emax, nucleus, nucleus)
    with ig.DeviceOperator(space, 1) as dX, ig.DeviceOperator(space, -1) as dY, ig.DeviceOperator(space, 1) as dZ:
        dX.upload(X)
        dY.upload(Y)
        ig.Commutator.device_term("comm222_pp_hhss", dX, dY, dZ, "split")
        Z = dZ.download()
    longest = 0
    for ch in range(ms.nch):
        kets = ms.channels[ch][3]
        if not kets:
            continue
        w = np.array([(1 - ms.occ[p]) * (1 - ms.occ[q]) - ms.occ[p] * ms.occ[q] for p, q in kets])
        k = np.nonzero(w)[0]
        if not len(k):
            continue
        longest = max(longest, len(k))
        x, y, z = (ms.block(a, ch) for a in (X, Y, Z))
        A, B = x[:, k], y[:, k] * w[k]
        P = (x[:, k] * w[k]) @ y[k]
        R = P + P.T
        # |v| < 2^e, rows with a zero maximum far below
        eA, eB = (np.where(m > 0, np.frexp(m)[1], -100000) for m in (abs(A).max(1), abs(B).max(1)))
        c = eB.max() - eA.max() if eB.max() > -1000 and eA.max() > -1000 else 0
        a = np.maximum(eA, eB - c).astype(float)
        S = abs(A) @ abs(B).T
        bound = 2 * len(k) * np.exp2(a[:, None] + a[None, :] + c - 35) + (len(k) + 5) * 2.0**-52 * (S + S.T)
        worst = float(np.max(abs(z - R) - bound))
        assert worst <= 0, (ch, len(kets), len(k), worst)
    assert longest > 339
