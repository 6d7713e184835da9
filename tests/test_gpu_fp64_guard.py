"""Operands for which the FP64 products' guard lists many elements or none by
their zeros: one operand a generator (nonzero between pp and hh kets only), a
Hamiltonian with its energies on the diagonal, both falling off from it, rows
with one to three elements far apart.  Element by element against
extended-precision sums, within the classical bound of an FP64 sum,
(K + 5) 2^-53 sum |x||w||y| (plus the update's rounding): the digits' error is
below it wherever the guard lets them pass, the listed elements' by its proof.
Sizes: one row to several tiles, K from 1 to two chunks (above 640 at emax 9);
symmetrised jobs (scalar ladder) and plain ones with m != n (tensor ladder)."""
import numpy as np
import pytest

import imsrg_gb300 as ig
from modelspace_ref import RefModelSpace

pytestmark = pytest.mark.gpu

U = 2.0**-53
Q = np.longdouble
SPACES = {"He4": (4, 2), "O16": (16, 8), "O18": (18, 8), "Ca40": (40, 20)}


def energies(ms, ch):
    N = 2 * ms.n + ms.l
    return np.array([N[p] + N[q] for p, q in ms.channels[ch][3]], dtype=float)


def holes(ms, ch):
    return np.array([int(ms.occ[p] > 1e-6) + int(ms.occ[q] > 1e-6) for p, q in ms.channels[ch][3]])


def weights(ms, ch):
    return np.array([(1 - ms.occ[p]) * (1 - ms.occ[q]) - ms.occ[p] * ms.occ[q] for p, q in ms.channels[ch][3]])


def shape(ms, b, cb, ck, kind, role, rng):
    """Gives block (cb, ck) of the X or Y (role) the kind's form."""
    if not b.size:
        return
    eb, ek = energies(ms, cb), energies(ms, ck)
    if kind == "generator" and role == "Y":
        b *= abs(holes(ms, cb)[:, None] - holes(ms, ck)) == 2
    elif kind == "diagonal" and role == "X":
        b *= 0.02
        if cb == ck:
            b[np.diag_indices(len(eb))] += eb + 3
    elif kind == "decay":
        b *= np.exp2(-1.5 * abs(eb[:, None] - ek))
    elif kind == "sparse":
        keep = rng.random(b.shape) < 1.5 / max(b.shape)
        if cb == ck:
            keep = np.triu(keep) | np.triu(keep).T
        far = np.exp2(-rng.integers(0, 40, b.shape).astype(float))
        b *= keep * (np.minimum(far, far.T) if cb == ck else far)


@pytest.mark.parametrize("emax,ref,kind", [(2, "He4", "generator"), (4, "O18", "generator"), (8, "O16", "generator"),
                                           (3, "O16", "diagonal"), (6, "O18", "diagonal"), (9, "O16", "diagonal"),
                                           (5, "Ca40", "decay"), (9, "O16", "decay"), (1, "O16", "sparse"), (4, "O18", "sparse"),
                                           (8, "O16", "sparse")])
def test_scalar_ladder(emax, ref, kind):
    ms = RefModelSpace(emax, *SPACES[ref])
    rng = np.random.default_rng(emax)
    X, Y, Z0 = ms.random_operator(11, True), ms.random_operator(12, False), ms.random_operator(13, True)
    for ch in range(ms.nch):
        shape(ms, ms.block(X, ch), ch, ch, kind, "X", rng)
        shape(ms, ms.block(Y, ch), ch, ch, kind, "Y", rng)
    space = ig.ModelSpace(emax, ref, ref)
    with ig.DeviceOperator(space, 1) as dX, ig.DeviceOperator(space, -1) as dY, ig.DeviceOperator(space, 1) as dZ:
        dX.upload(X)
        dY.upload(Y)
        dZ.upload(Z0)
        ig.Commutator.device_term("comm222_pp_hhss", dX, dY, dZ, "fp64")
        Z = dZ.download()
    for ch in range(ms.nch):
        n = len(ms.channels[ch][3])
        w = weights(ms, ch)
        k = np.nonzero(w)[0]
        rows = np.arange(n) if n <= 140 else np.sort(rng.choice(n, 8, replace=False))
        x, y, z, z0 = (ms.block(a, ch) for a in (X, Y, Z, Z0))
        wy, wyr = w[k, None] * y[k], w[k, None] * y[np.ix_(k, rows)]
        M = x[np.ix_(rows, k)].astype(Q) @ wy.astype(Q) + (x[:, k].astype(Q) @ wyr.astype(Q)).T + z0[rows]
        S = abs(x[np.ix_(rows, k)]) @ abs(wy) + (abs(x[:, k]) @ abs(wyr)).T
        bound = (len(k) + 5) * U * S + 2 * U * (abs(z[rows]) + abs(z0[rows]))
        worst = float(np.max(abs(z[rows] - M) - bound, initial=-1.0))
        assert worst <= 0, (ch, n, len(k), worst)


@pytest.mark.parametrize("emax,ref,rank,kind", [(2, "O16", (1, 0, 1), "plain"), (5, "O18", (2, 0, 0), "plain"),
                                                (6, "O16", (1, 1, 0), "diagonal"), (6, "O16", (2, 0, 0), "decay"),
                                                (4, "Ca40", (3, 1, 1), "decay"), (5, "O16", (2, 1, 1), "generator"),
                                                (5, "O18", (0, 1, 0), "sparse")])
def test_tensor_ladder(emax, ref, rank, kind):
    """Z2 += X w Y - Y w X for a tensor Y: two plain products, two additions."""
    ms = RefModelSpace(emax, *SPACES[ref])
    rng = np.random.default_rng(emax)
    X, Y, Z0 = ms.random_operator(21, True), ms.random_tensor(22, *rank), ms.random_tensor(23, *rank)
    blocks, offs, _ = ms.tensor_layout(*rank)

    def block(a, cb, ck, o):
        nb, nk = len(ms.channels[cb][3]), len(ms.channels[ck][3])
        return a[o:o + nb * nk].reshape(nb, nk, order="F")

    for ch in range(ms.nch):
        shape(ms, ms.block(X, ch), ch, ch, kind, "X", rng)
    for (cb, ck), o in zip(blocks, offs):
        shape(ms, block(Y, cb, ck, o), cb, ck, kind, "Y", rng)
    space = ig.ModelSpace(emax, ref, ref)
    with ig.DeviceOperator(space, 1) as dX, ig.DeviceOperator(space, 1, rank) as dY, ig.DeviceOperator(space, 1, rank) as dZ:
        dX.upload(X)
        dY.upload(Y)
        dZ.upload(Z0)
        ig.Commutator.device_tensor_term("comm222_pp_hh_221st", dX, dY, dZ, "fp64")
        Z = dZ.download()
    for (cb, ck), o in zip(blocks, offs):
        y, z, z0 = (block(a, cb, ck, o) for a in (Y, Z, Z0))
        if not z.size:
            continue
        wb, wk = weights(ms, cb), weights(ms, ck)
        kb, kk = np.nonzero(wb)[0], np.nonzero(wk)[0]
        rows = np.arange(len(z)) if len(z) <= 60 else np.sort(rng.choice(len(z), 6, replace=False))
        xb, xk = ms.block(X, cb)[np.ix_(rows, kb)] * wb[kb], (wk[:, None] * ms.block(X, ck))[kk]
        yr, z, z0 = y[np.ix_(rows, kk)], z[rows], z0[rows]
        M1, M2 = xb.astype(Q) @ y[kb].astype(Q), yr.astype(Q) @ xk.astype(Q)
        S = abs(xb) @ abs(y[kb]) + abs(yr) @ abs(xk)
        bound = (max(len(kb), len(kk)) + 5) * U * S + 2 * U * (abs(z) + abs(z0) + abs(M1 - M2).astype(float) + abs(M1).astype(float))
        worst = float(np.max(abs(z - (M1 - M2 + z0)) - bound))
        assert worst <= 0, (cb, ck, z.shape, worst)


def test_generator_is_not_slow():
    """A commutator with a generator lists a percent of the FP64 work: it may not
    take twice as long as one of random operators (3.8 times as long where the
    zeros counted as products and whole tiles were listed)."""
    torch = pytest.importorskip("torch")
    ms = RefModelSpace(8, 16, 8)
    space = ig.ModelSpace(8, "O16", "O16")
    X, Y = ms.random_operator(1, True), ms.random_operator(2, False)
    G = Y.copy()
    for ch in range(ms.nch):
        shape(ms, ms.block(G, ch), ch, ch, "generator", "Y", None)
    best = []
    with ig.DeviceOperator(space, 1) as dX, ig.DeviceOperator(space, -1) as dY, ig.DeviceOperator(space, 1) as dZ:
        dX.upload(X)
        for y in (Y, G):
            dY.upload(y)
            times = []
            for _ in range(8):
                a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
                a.record()
                ig.Commutator.device_commutator(dX, dY, dZ, "fp64")
                b.record()
                b.synchronize()
                times.append(a.elapsed_time(b))
            best.append(min(times[3:]))
    assert best[1] < 2 * best[0], best
