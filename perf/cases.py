"""What the performance of this framework is measured on: the work that a user
has it do through the public Python API, from the smallest model space to the
largest configuration (64-pair batches, a Magnus flow step at emax 12).

A case names its kind, the model space (emax, reference nucleus), the
precision form and the hermiticities.  Operators are seeded random ones of the
benchmark's distribution: uniform [-1, 1] entries on the symmetry-allowed
elements, (anti)symmetrised, the one-body matrix and every two-body channel
block scaled to unit Frobenius norm; Hamiltonians carry oscillator energies on
the one-body diagonal.
"""
import functools
import math

import numpy as np
import torch

import imsrg_gb300 as ig

DEV = "cuda" if torch.cuda.is_available() else "cpu"
NUCLEI = {"He4": (4, 2), "C12": (12, 6), "O16": (16, 8), "O18": (18, 8), "Ca40": (40, 20)}


def listed():
    return [
        # the smallest space in use: one commutator on resident operators; launches and host calls count
        dict(name="commutator emax2 fp64", kind="commutator", emax=2, reference="O16", precision="fp64", hx=1, hy=-1),
        # a small space with a partly filled shell (fractional occupations), both operators anti-hermitian as in BCH_Product
        dict(name="commutator emax4 O18 split", kind="commutator", emax=4, reference="O18", precision="split", hx=-1, hy=-1),
        # the ordinary FP64 commutator of a developer's run (28 orbits per isospin); fp64 is the default form
        dict(name="commutator emax6 fp64", kind="commutator", emax=6, reference="O16", precision="fp64", hx=1, hy=-1),
        # a heavier reference: more holes, other ragged pp / hh / ph extents
        dict(name="commutator emax7 Ca40 fp64", kind="commutator", emax=7, reference="Ca40", precision="fp64", hx=-1, hy=1),
        # the headline benchmark: split form at emax 10 (66 orbits per isospin)
        dict(name="commutator emax10 split", kind="commutator", emax=10, reference="O16", precision="split", hx=1, hy=-1),
        # the same commutator in the FP64 form it is compared with
        dict(name="commutator emax10 fp64", kind="commutator", emax=10, reference="O16", precision="fp64", hx=1, hy=-1),
        # many independent uneven commutators replayed as one graph
        dict(name="batch 64 pairs split", kind="batch", emax_min=2, emax_max=6, pairs=64, reference="O16", precision="split", hx=1, hy=-1),
        # the similarity transform of a Hamiltonian (about ten nested commutators)
        dict(name="bch emax8 split", kind="bch", emax=8, reference="O16", precision="split", omega=8.0),
        # one Magnus-Euler step of the largest flow: generator, BCH_Product, BCH_Transform
        dict(name="flow step emax12 split", kind="flow", emax=12, reference="O16", precision="split", omega=2.0, ds=0.5),
        # an electric quadrupole observable evolved with the flow: scalar-tensor commutator
        dict(name="tensor E2 emax8 split", kind="tensor", emax=8, reference="O16", precision="split", lam=2, trank=0, parity=0, hy=1),
        # a Gamow-Teller transition operator in the FP64 form
        dict(name="tensor GT emax6 fp64", kind="tensor", emax=6, reference="O16", precision="fp64", lam=1, trank=1, parity=0, hy=1),
        # the drop-in call: host operators in, host operator out
        dict(name="host commutator emax5 fp64", kind="host", emax=5, reference="O16", precision="fp64", hx=1, hy=-1),
    ]


def draw(rng):
    kind = rng.choice(["commutator", "commutator", "commutator", "batch", "bch", "flow", "tensor", "host"])
    prec = rng.choice(["fp64", "split"])
    refs = ["He4", "C12", "O16", "O18", "Ca40"]
    if kind in ("commutator", "host"):
        top = 6 if kind == "host" else 11 if prec == "split" else 9
        emax = rng.randint(2, top)
        ref = rng.choice(refs[:4] if emax < 3 else refs)
        if emax < 2 + (ref == "O18"):
            ref = "O16"
        return dict(kind=kind, emax=emax, reference=ref, precision=prec, hx=rng.choice([1, -1]), hy=rng.choice([1, -1]))
    if kind == "batch":
        lo = rng.randint(2, 5)
        pairs = int(round(2 ** rng.uniform(1, 6)))
        return dict(kind=kind, emax_min=lo, emax_max=rng.randint(lo, 6), pairs=pairs, reference=rng.choice(refs[:3]), precision=prec, hx=1, hy=rng.choice([1, -1]))
    if kind == "bch":
        return dict(kind=kind, emax=rng.randint(3, 9 if prec == "split" else 6), reference=rng.choice(refs[1:]), precision=prec, omega=round(rng.uniform(1.0, 10.0), 2))
    if kind == "flow":
        return dict(kind=kind, emax=rng.randint(8, 11), reference=rng.choice(refs[1:]), precision="split", omega=round(rng.uniform(0.5, 4.0), 2), ds=rng.choice([0.25, 0.5, 1.0]))
    lam, trank, parity = rng.choice([(0, 1, 0), (1, 0, 1), (1, 1, 0), (2, 0, 0), (2, 1, 1), (3, 0, 1)])
    return dict(kind=kind, emax=rng.randint(4, 8 if prec == "split" else 7), reference=rng.choice(refs), precision=prec, lam=lam, trank=trank, parity=parity, hy=rng.choice([1, -1]))


# --------------------------------------------------------------- model space
def _round32(x):
    return (x + 31) // 32 * 32


class Basis:
    """Orbits, two-body channels and the arena layout of a model space."""

    def __init__(self, emax, reference):
        A, Z = NUCLEI[reference]
        orb = []
        for N in range(emax + 1):
            for l in range(N, -1, -2):
                for j2 in (2 * l + 1, 2 * l - 1):
                    if j2 > 0:
                        orb += [((N - l) // 2, l, j2, -1), ((N - l) // 2, l, j2, 1)]
        self.n, self.l, self.j2, self.tz2 = (np.array(c) for c in zip(*orb))
        self.norb = N = len(orb)
        # shells fill in order of N, then j descending in steps of the reference's g = 2N+1, 2N-3, ...
        self.occ = np.zeros(N)
        left = {-1: float(Z), 1: float(A - Z)}
        for shell in range(emax + 1):
            for g in range(2 * shell + 1, -2 * shell - 1, -4):
                j2 = abs(g)
                l = (j2 + 1) // 2 if g < 0 else (j2 - 1) // 2
                for tz in (-1, 1):
                    put = min(left[tz], j2 + 1.0)
                    left[tz] -= put
                    at = [i for i, o in enumerate(orb) if o == ((shell - l) // 2, l, j2, tz)]
                    self.occ[at[0]] = put / (j2 + 1.0)
        p, q = np.triu_indices(N)
        self.nch = 6 * (int(self.j2.max()) + 1)
        self.channels, self.off = [], []
        cur = _round32(32 + N * N)
        for ch in range(self.nch):
            J, par, Tz = ch // 6, ch % 2, (ch % 6) // 2 - 1
            ok = ((self.l[p] + self.l[q]) % 2 == par) & (self.tz2[p] + self.tz2[q] == 2 * Tz)
            ok &= (self.j2[p] + self.j2[q] >= 2 * J) & (abs(self.j2[p] - self.j2[q]) <= 2 * J) & ~((p == q) & (J % 2 == 1))
            self.channels.append((J, par, Tz, p[ok], q[ok]))
            self.off.append(cur)
            cur = _round32(cur + int(ok.sum()) ** 2)
        self.size = cur
        self.same = (self.l[:, None] == self.l) & (self.j2[:, None] == self.j2) & (self.tz2[:, None] == self.tz2)

    def tensor_blocks(self, lam, trank, parity):
        """[(ch_bra, ch_ket, offset)] and the arena length of a tensor of that rank."""
        out, cur = [], _round32(32 + self.norb**2)
        for cb in range(self.nch):
            for ck in range(cb, self.nch):
                (Jb, pb, Tb, b, _), (Jk, pk, Tk, k, _) = self.channels[cb], self.channels[ck]
                if abs(Jb - Jk) <= lam <= Jb + Jk and abs(Tb - Tk) == trank and (pb + pk + parity) % 2 == 0:
                    out.append((cb, ck, cur))
                    cur = _round32(cur + len(b) * len(k))
        return out, cur


@functools.lru_cache(maxsize=None)
def basis(emax, reference):
    return Basis(emax, reference)


@functools.lru_cache(maxsize=None)
def space(emax, reference, copy=0):
    """The model space a user's program keeps (one per pair in a batch)."""
    return ig.ModelSpace(emax, reference, reference)


def _gen(seed, salt):
    return torch.Generator(device=DEV).manual_seed((int(seed) * 1000003 + salt) % (1 << 62))


def _uniform(gen, *shape):
    return torch.rand(*shape, generator=gen, dtype=torch.float64, device=DEV) * 2 - 1


def scalar_arena(b, seed, salt, herm, hamiltonian=False):
    """A random scalar operator of the benchmark's distribution, as an arena."""
    g, N = _gen(seed, salt), b.norb
    a = torch.zeros(b.size, dtype=torch.float64, device=DEV)
    r = _uniform(g, N, N) * torch.from_numpy(b.same).to(DEV)
    one = (r + herm * r.T) / 2
    if hamiltonian:
        energy = torch.from_numpy(2 * b.n + b.l + 1.5).to(DEV)
        one = 0.1 * one.triu(1) + 0.1 * one.triu(1).T + torch.diag(energy)
    else:
        one = one / one.norm()
        a[0] = _uniform(g, 1)[0] if herm == 1 else 0.0
    a[32 : 32 + N * N] = one.T.reshape(-1)
    for (J, par, Tz, p, q), o in zip(b.channels, b.off):
        n = len(p)
        if n:
            m = _uniform(g, n, n)
            m = (m + herm * m.T) / 2
            f = m.norm()
            a[o : o + n * n] = (m / torch.where(f > 0, f, torch.ones_like(f))).T.reshape(-1)
    return a


def tensor_arena(b, seed, salt, lam, trank, parity, herm):
    """A random reduced tensor operator, as an arena of its rank."""
    blocks, size = b.tensor_blocks(lam, trank, parity)
    g, N = _gen(seed, salt), b.norb
    a = torch.zeros(size, dtype=torch.float64, device=DEV)
    ok = ((b.l[:, None] + b.l + parity) % 2 == 0) & (abs(b.j2[:, None] - b.j2) <= 2 * lam) & (b.j2[:, None] + b.j2 >= 2 * lam)
    ok &= abs(b.tz2[:, None] - b.tz2) == 2 * trank
    ph = np.where((b.j2[:, None] - b.j2) // 2 % 2, -1.0, 1.0) * herm
    one = (_uniform(g, N, N) * torch.from_numpy(ok).to(DEV)).triu()
    one = one * torch.from_numpy(np.where(np.eye(N, dtype=bool) & (ph < 0), 0.0, 1.0)).to(DEV)
    one = one + (one * torch.from_numpy(ph).to(DEV)).triu(1).T
    a[32 : 32 + N * N] = (one / one.norm().clamp_min(1e-300)).T.reshape(-1)
    for cb, ck, o in blocks:
        nb, nk = len(b.channels[cb][3]), len(b.channels[ck][3])
        if nb and nk:
            m = _uniform(g, nb, nk)
            if cb == ck:
                m = (m + herm * m.T) / 2
            f = m.norm()
            a[o : o + nb * nk] = (m / torch.where(f > 0, f, torch.ones_like(f))).T.reshape(-1)
    return a


def norm(b, a):
    """Operator::Norm of a scalar arena: the weights of the BCH stopping rule."""
    one = a[32 : 32 + b.norb**2].reshape(b.norb, b.norb)
    n2 = float((one**2 * torch.from_numpy(b.j2 + 1.0).to(DEV)).sum())
    for (J, _, _, p, _), o in zip(b.channels, b.off):
        if len(p):
            n2 += float((a[o : o + len(p) ** 2] ** 2).sum()) * (2 * J + 1) ** 2
    return math.sqrt(n2)


# ------------------------------------------------------------------- prepare
class _View:
    """The operator's device arena for torch, which holds on to this object and so to the operator."""

    def __init__(self, op):
        self.op = op
        self.__cuda_array_interface__ = dict(shape=(op.size,), typestr="<f8", data=(op.device_ptr(), False), version=3)


def _tensor(op):
    """The operator's arena as a tensor (no copy)."""
    return torch.as_tensor(_View(op), device=DEV)


def _device_op(ms, herm, values=None, rank=(0, 0, 0)):
    op = ig.DeviceOperator(ms, herm, rank)
    if values is not None:
        _tensor(op).copy_(values)
    return op


def _batch_emax(case):
    """The model spaces of a batch: emax spread evenly over the range, in a fixed uneven order."""
    span = case["emax_max"] - case["emax_min"] + 1
    return [case["emax_min"] + (7 * k + k // 3) % span for k in range(case["pairs"])]


def _inputs(case, seed):
    """The input arenas of a case, in the order its call takes them."""
    if case["kind"] == "batch":
        return [[scalar_arena(basis(e, case["reference"]), seed, 2 * k + s, h) for s, h in ((0, case["hx"]), (1, case["hy"]))]
                for k, e in enumerate(_batch_emax(case))]
    b = basis(case["emax"], case["reference"])
    if case["kind"] == "tensor":
        return [scalar_arena(b, seed, 1, 1), tensor_arena(b, seed, 2, case["lam"], case["trank"], case["parity"], case["hy"])]
    if case["kind"] in ("bch", "flow"):
        H, om = scalar_arena(b, seed, 1, 1, hamiltonian=True), scalar_arena(b, seed, 2, -1)
        om *= case["omega"] / norm(b, om)
        return [H, om] if case["kind"] == "bch" else [H, om, scalar_arena(b, seed, 3, 1, hamiltonian=True)]
    return [scalar_arena(b, seed, 1, case["hx"]), scalar_arena(b, seed, 2, case["hy"])]


def prepare(case, seed):
    inp, kind, prec = _inputs(case, seed), case["kind"], case["precision"]
    s = dict(kind=kind, precision=prec)
    if kind == "batch":
        pairs = []
        for k, (e, (x, y)) in enumerate(zip(_batch_emax(case), inp)):
            ms = space(e, case["reference"], k)
            pairs.append((_device_op(ms, case["hx"], x), _device_op(ms, case["hy"], y), _device_op(ms, 1)))
        s.update(batch=ig.CommutatorBatch(pairs, prec), out=[_tensor(z) for _, _, z in pairs])
        return s
    ms = space(case["emax"], case["reference"])
    if kind == "host":
        s["X"], s["Y"] = (ig.Operator(ms, arena=a.cpu().numpy(), hermitian=h == 1) for a, h in zip(inp, (case["hx"], case["hy"])))
        return s
    if kind == "tensor":
        rank = (case["lam"], case["trank"], case["parity"])
        s.update(X=_device_op(ms, 1, inp[0]), Y=_device_op(ms, case["hy"], inp[1], rank), Z=_device_op(ms, 1, None, rank))
    elif kind == "bch":
        s.update(X=_device_op(ms, 1, inp[0]), Y=_device_op(ms, -1, inp[1]), Z=_device_op(ms, 1))
    elif kind == "flow":
        s.update(H0=_device_op(ms, 1, inp[0]), omega=_device_op(ms, -1, inp[1]), H=_device_op(ms, 1, inp[2]), ds=case["ds"],
                 eta=_device_op(ms, -1), step=_device_op(ms, -1), new=_device_op(ms, -1), Z=_device_op(ms, 1), generator=ig.Generator())
        s["out"] = [_tensor(s[k]) for k in ("eta", "new", "Z")]
        return s
    else:
        s.update(X=_device_op(ms, case["hx"], inp[0]), Y=_device_op(ms, case["hy"], inp[1]), Z=_device_op(ms, 1))
    s["out"] = [_tensor(s["Z"])]
    return s


def run(s):
    kind, prec = s["kind"], s["precision"]
    if kind == "commutator":
        ig.Commutator.device_commutator(s["X"], s["Y"], s["Z"], prec)
    elif kind == "batch":
        s["batch"].launch()
    elif kind == "bch":
        ig.BCH.device_transform(s["X"], s["Y"], s["Z"], prec)
    elif kind == "tensor":
        ig.Commutator.device_scalar_tensor(s["X"], s["Y"], s["Z"], prec)
    elif kind == "host":
        return [ig.Commutator.Commutator(s["X"], s["Y"], prec).arena]
    else:
        s["generator"].device_update(s["H"], s["eta"])
        s["step"].copy_from(s["eta"])
        s["step"].scale(s["ds"])
        ig.BCH.device_product(s["step"], s["omega"], s["new"], prec)
        ig.BCH.device_transform(s["H0"], s["new"], s["Z"], prec)
    return s["out"]


# ---------------------------------------------------------------------- work
def _commutator_flops(b):
    """The two dense contractions, each over the shorter set of its factors."""
    hole = b.occ > 1e-6
    fl = 0.0
    for J, par, Tz, p, q in b.channels:
        n = len(p)
        k = int((~hole[p] & ~hole[q]).sum() + (hole[p] & hole[q]).sum())
        fl += 2.0 * n * n * k
    p, q = np.triu_indices(b.norb)
    for ch in range(b.nch):
        J, par, Tz = ch // 6, ch % 2, (ch % 6) // 2 - 1
        ok = ((b.l[p] + b.l[q]) % 2 == par) & (abs(b.tz2[p] - b.tz2[q]) == 2 * Tz)
        ok &= (b.j2[p] + b.j2[q] >= 2 * J) & (abs(b.j2[p] - b.j2[q]) <= 2 * J)
        fl += 8.0 * float(ok.sum()) ** 2 * float((ok & (hole[p] != hole[q])).sum())
    return fl


def work(case):
    kind = case["kind"]
    if kind == "batch":
        bs = [basis(e, case["reference"]) for e in _batch_emax(case)]
        return dict(bytes=sum(24.0 * b.size for b in bs), flops=sum(_commutator_flops(b) for b in bs))
    b = basis(case["emax"], case["reference"])
    if kind == "tensor":
        blocks, size = b.tensor_blocks(case["lam"], case["trank"], case["parity"])
        hole, fl = b.occ > 1e-6, 0.0
        k = [int((~hole[p] & ~hole[q]).sum() + (hole[p] & hole[q]).sum()) for _, _, _, p, q in b.channels]
        for cb, ck, _ in blocks:
            fl += 2.0 * len(b.channels[cb][3]) * len(b.channels[ck][3]) * (k[cb] + k[ck])
        return dict(bytes=8.0 * (b.size + 2 * size), flops=fl)
    # series: the commutators that the norms ask for in practice
    times = dict(bch=max(4, round(4 + 0.7 * case.get("omega", 0))), flow=9).get(kind, 1)
    arenas = dict(bch=3, flow=6).get(kind, 3)
    return dict(bytes=8.0 * arenas * b.size, flops=times * _commutator_flops(b))


# --------------------------------------------------------------------- exact
# The commutator in 64 bits from its textbook form: unnormalised J-coupled
# elements over ordered orbit pairs, every sum written out, no occupation
# classes and no folded symmetries.
@functools.lru_cache(maxsize=None)
def _sixj_exact(a, b, c, d, e, f):
    """{a b c; d e f} of doubled angular momenta, by Racah's sum in integers."""
    tri = ((a, b, c), (a, e, f), (d, b, f), (d, e, c))
    if any(x + y < z or abs(x - y) > z or (x + y + z) % 2 for x, y, z in tri):
        return 0.0
    fac = math.factorial
    num = den = 1
    for x, y, z in tri:
        num *= fac((x + y - z) // 2) * fac((x - y + z) // 2) * fac((-x + y + z) // 2)
        den *= fac((x + y + z) // 2 + 1)
    lo = max((x + y + z) // 2 for x, y, z in tri)
    four = ((a + b + d + e) // 2, (b + c + e + f) // 2, (c + a + f + d) // 2)
    hi = min(four)
    scale = math.prod(fac(hi - (x + y + z) // 2) for x, y, z in tri) * math.prod(fac(s - lo) for s in four)
    total = 0
    for t in range(lo, hi + 1):
        total += (-1) ** t * fac(t + 1) * (scale // (math.prod(fac(t - (x + y + z) // 2) for x, y, z in tri) * math.prod(fac(s - t) for s in four)))
    return math.copysign(math.sqrt((total * total * num) / (scale * scale * den)), total)


class Exact:
    """Tables of a model space for exact()."""

    def __init__(self, b):
        self.b, N = b, b.norb
        cu = lambda x: torch.from_numpy(np.ascontiguousarray(x)).to(DEV)  # noqa: E731
        self.j2, self.l, self.tz2, self.occ = cu(b.j2), cu(b.l), cu(b.tz2), cu(b.occ)
        nj, self.NJ = int(b.j2.max() + 1) // 2, int(b.j2.max()) + 1
        six = np.zeros((nj, nj, self.NJ, nj, nj, self.NJ))
        for a in range(nj):
            for c in range(nj):
                for d in range(nj):
                    for e in range(nj):
                        for J in range(abs(a - c), a + c + 2):
                            if J < abs(d - e) or J > d + e + 1:
                                continue
                            for K in range(max(abs(a - e), abs(d - c)), min(a + e, d + c) + 2):
                                # columns 1, 2 swap and pairs of columns flip: one value for each orbit of these
                                key = min((a, c, J, d, e, K), (c, a, J, e, d, K), (d, e, J, a, c, K), (e, d, J, c, a, K),
                                          (a, e, K, d, c, J), (e, a, K, c, d, J), (d, c, K, a, e, J), (c, d, K, e, a, J))
                                six[a, c, J, d, e, K] = _sixj_exact(2 * key[0] + 1, 2 * key[1] + 1, 2 * key[2], 2 * key[3] + 1, 2 * key[4] + 1, 2 * key[5])
        self.six, self.nj = cu(six).reshape(-1), nj
        self.jx = (self.j2 - 1) // 2  # half-integer j as an index
        # ordered pairs of each two-body channel, and the p <= q ket and factor each is made of
        self.pairs = []
        for J, par, Tz, p, q in b.channels:
            n, odd = len(p), p != q
            ph = np.where(((b.j2[p] + b.j2[q]) // 2 - J) % 2, 1.0, -1.0)  # -(-1)^(jp + jq - J)
            P, Q = np.concatenate([p, q[odd]]), np.concatenate([q, p[odd]])
            ket = np.concatenate([np.arange(n), np.arange(n)[odd]])
            f = np.concatenate([np.where(odd, 1.0, math.sqrt(2.0)), ph[odd]])
            self.pairs.append((cu(P), cu(Q), cu(ket), cu(f)))
        # ordered particle-hole pairs (a, b) of each (J, parity, tz_a - tz_b), all blocks in one buffer
        A, B = np.divmod(np.arange(N * N), N)
        self.cc, self.pos, self.base, self.width = [], np.zeros((self.NJ, N * N), np.int64), np.zeros((self.NJ, N * N), np.int64), np.zeros((self.NJ, N * N), np.int64)
        cur = 0
        for J in range(self.NJ):
            tri = (b.j2[A] + b.j2[B] >= 2 * J) & (abs(b.j2[A] - b.j2[B]) <= 2 * J)
            for par in (0, 1):
                for dt in (-1, 0, 1):
                    at = np.nonzero(tri & ((b.l[A] + b.l[B]) % 2 == par) & (b.tz2[A] - b.tz2[B] == 2 * dt))[0]
                    self.pos[J, at], self.base[J, at], self.width[J, at] = np.arange(len(at)), cur, len(at)
                    self.cc.append((J, cu(A[at]), cu(B[at]), cur))
                    cur += len(at) ** 2
        self.cc_size = cur
        self.pos, self.base, self.width = cu(self.pos), cu(self.base), cu(self.width)
        # position of an ordered pair in its two-body channel; each channel's unnormalised matrix in one buffer
        self.at2, self.base2, self.width2 = (torch.full((self.NJ, N * N), -1, dtype=torch.int64, device=DEV) for _ in range(3))
        cur = 0
        for (J, par, Tz, p, q), (P, Q, ket, f) in zip(b.channels, self.pairs):
            m = len(P)
            k = P * N + Q
            self.at2[J, k], self.base2[J, k], self.width2[J, k] = torch.arange(m, device=DEV), cur, m
            cur += m * m
        self.full_size = cur

    def sixj(self, a, b, J, c, d, K):
        """{j_a j_b J; j_c j_d K} of orbit index tensors; J, K numbers."""
        i = ((self.jx[a] * self.nj + self.jx[b]) * self.NJ + J) * self.nj + self.jx[c]
        return self.six[(i * self.nj + self.jx[d]) * self.NJ + K]

    def unpack(self, a):
        """(one-body, {channel: matrix over ordered pairs}, all of them in one buffer)"""
        b, N, two = self.b, self.b.norb, []
        flat = torch.zeros(self.full_size, dtype=torch.float64, device=DEV)
        cur = 0
        for (J, par, Tz, p, q), o, (P, Q, ket, f) in zip(b.channels, b.off, self.pairs):
            n, m = len(p), len(P)
            M = flat[cur : cur + m * m].view(m, m)
            if n:
                B = a[o : o + n * n].view(n, n).T
                M.copy_(B[ket][:, ket] * f[:, None] * f)
            two.append(M)
            cur += m * m
        return a[32 : 32 + N * N].view(N, N).T, two, flat

    def pandya(self, flat, J, a, b_, c, d):
        """-sum_K (2K+1) {a b J; c d K} X^K(ad, cb) over rows (a, b) and columns (c, d)."""
        N = self.b.norb
        a, b_, c, d = a[:, None], b_[:, None], c[None, :], d[None, :]
        r, s = a * N + d, c * N + b_
        out = torch.zeros(r.shape, dtype=torch.float64, device=DEV)
        if not out.numel():
            return out
        for K in range(self.NJ):
            six = self.sixj(a, b_, J, c, d, K)
            i, k = self.at2[K][r], self.at2[K][s]
            ok = (i >= 0) & (k >= 0) & (six != 0)
            v = flat[torch.where(ok, self.base2[K][r] + i * self.width2[K][r] + k, 0)]
            out -= torch.where(ok, (2 * K + 1) * six * v, 0.0)
        return out

    def commutator(self, X, Y):
        b, N, occ = self.b, self.b.norb, self.occ
        (X1, X2, Xf), (Y1, Y2, Yf) = self.unpack(X), self.unpack(Y)
        Z = torch.zeros_like(X)
        deg = (self.j2 + 1).double()
        C1 = X1 @ Y1 - Y1 @ X1
        z0, Z1 = (C1.diagonal() * occ * deg).sum(), C1.clone()
        # Z-bar(ab, cd) = sum_ef (n_e - n_f) X-bar(ab, ef) Y-bar(ef, cd)
        zb = torch.zeros(self.cc_size, dtype=torch.float64, device=DEV)
        for J, A, B, o in self.cc:
            w = occ[A] - occ[B]
            k = torch.nonzero(w).reshape(-1)
            if len(k):
                left = self.pandya(Xf, J, A, B, A[k], B[k]) * w[k]
                zb[o : o + len(A) ** 2] = (left @ self.pandya(Yf, J, A[k], B[k], A, B)).reshape(-1)
        mono = torch.zeros(2, N, N, dtype=torch.float64, device=DEV)
        for c, ((J, par, Tz, p, q), off, (P, Q, ket, f)) in enumerate(zip(b.channels, b.off, self.pairs)):
            n, m = len(p), len(P)
            if not n:
                continue
            x, y = X2[c], Y2[c]
            nP, nQ = occ[P], occ[Q]
            hh, pp = nP * nQ, (1 - nP) * (1 - nQ)
            z0 = z0 + (2 * J + 1) * 0.25 * torch.einsum("a,ab,ba,b->", hh, x, y, pp) - (2 * J + 1) * 0.25 * torch.einsum("a,ab,ba,b->", hh, y, x, pp)
            Mhh = 0.5 * (x @ (hh[:, None] * y) - y @ (hh[:, None] * x))
            Mpp = 0.5 * (x @ (pp[:, None] * y) - y @ (pp[:, None] * x))
            z = Mpp - Mhh
            # one-body operators in the pair basis: (E_X Y - Y E_X) - (E_Y X - X E_Y)
            for one, two, s in ((X1, y, 1.0), (Y1, x, -1.0)):
                E = one[P][:, P] * (Q[:, None] == Q) + one[Q][:, Q] * (P[:, None] == P)
                z = z + s * (E @ two - two @ E)
            # exchange-antisymmetrised inverse Pandya transform
            T = torch.zeros(m, m, dtype=torch.float64, device=DEV)
            i, j, k, l = P[:, None], Q[:, None], P[None, :], Q[None, :]
            r, s = i * N + l, k * N + j
            for K in range(self.NJ):
                six = self.sixj(i, j, J, k, l, K)
                ok = (six != 0) & (self.width[K][r] > 0)
                v = zb[torch.where(ok, self.base[K][r] + self.pos[K][r] * self.width[K][r] + self.pos[K][s], 0)]
                T += torch.where(ok, (2 * K + 1) * six * v, 0.0)
            swap = self.at2[J][Q * N + P]
            ph = torch.where(((self.j2[P] + self.j2[Q]) // 2 - J) % 2 == 0, -1.0, 1.0).double()
            T = T + ph[:, None] * T[swap]
            z = z + T + T[:, swap] * ph
            # one-body part: sum over c of (2J+1) [n_c Mpp + (1 - n_c) Mhh](ci, cj), and the monopoles of comm121
            for M, w in ((Mpp, occ), (Mhh, 1 - occ)):
                r, s = torch.nonzero(P[:, None] == P[None, :], as_tuple=True)
                Z1.index_put_((Q[r], Q[s]), (2 * J + 1) * w[P[r]] * M[r, s] / deg[Q[r]], accumulate=True)
            for one, two, s_ in ((X1, y, 1.0), (Y1, x, -1.0)):
                # sum_ab (n_a - n_b) one(a, b) two(bi, aj)
                g = ((occ[:, None] - occ) * one)[P[None, :], P[:, None]] * two
                r, s = torch.nonzero(g, as_tuple=True)
                Z1.index_put_((Q[r], Q[s]), s_ * (2 * J + 1) * g[r, s] / deg[Q[r]], accumulate=True)
            first = torch.arange(n, device=DEV)
            Z[off : off + n * n] = (z[first][:, first] / f[:n][:, None] / f[:n]).T.reshape(-1)
        Z[0] = z0
        Z[32 : 32 + N * N] = (Z1 * torch.from_numpy(b.same).to(DEV)).T.reshape(-1)
        return Z


@functools.lru_cache(maxsize=2)
def tables(emax, reference):
    return Exact(basis(emax, reference))


def exact(case, seed):
    kind = case["kind"]
    # the scalar-tensor sums over 9j symbols and whole flow steps take minutes written out like this
    if kind in ("tensor", "flow") or case.get("emax", 0) > 10:
        return None
    inp = _inputs(case, seed)
    if kind == "batch":
        return [tables(e, case["reference"]).commutator(x, y) for e, (x, y) in zip(_batch_emax(case), inp)]
    t = tables(case["emax"], case["reference"])
    if kind != "bch":
        return [t.commutator(*inp)]
    H, om = inp
    ny, out, nested, fden = norm(t.b, om), H.clone(), H, 1.0
    eps = norm(t.b, H) * math.exp(-2 * ny) * 1e-9 / (2 * ny)
    for i in range(1, 41):  # nested commutators until the reference's rule stops them
        nested, fden = t.commutator(om, nested), fden / i
        out += fden * nested
        eps *= i + 1
        if norm(t.b, nested) < eps:
            break
    return [out]
