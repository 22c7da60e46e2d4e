"""Performance cases of the IMSRG(2) commutator engine.

Each case is one call that a program using the library makes: single [L, R]
commutators in every precision, the packed host-operand call, a batch of
independent commutators, the reverse-mode commutator, and Magnus flow steps.
Bases are harmonic-oscillator j-orbits with 2n + l <= emax whose lowest
`filled` shells are holes (1: 4He, 2: 16O), emax 2 to 6.  Operators are seeded
synthetic ones: H has the oscillator spectrum hw (2n + l + 3/2), N(0, 0.5) MeV
off-diagonals and N(0, sigma) MeV Hermitian two-body elements; an
anti-Hermitian operator has N(0, 0.05) elements.

A program keeps a basis (device tables, workspace, the split engine's plan)
for all the Hamiltonians it treats in it, so bases are kept here too; every
state has its own operators.
"""
from __future__ import annotations

import functools
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "eom-imsrg_full_gb300")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

SQUARE = (True, False, False, True, True, False)  # gam 1..6: pppp ppph pphh phph hhhh phhh
ROWCAT = (0, 0, 0, 1, 2, 1)
COLCAT = (0, 1, 2, 1, 2, 2)


# --- the cases ---------------------------------------------------------------
def _comm(name, emax, filled, precision, digits=6, herm_L=-1, herm_R=1, with_e0=True, hw=20.0, sigma=1.0):
    return dict(name=name, op="commutator", emax=emax, filled=filled, precision=precision, digits=digits,
                herm_L=herm_L, herm_R=herm_R, with_e0=with_e0, hw=hw, sigma=sigma)


def listed():
    return [
        # the smallest bases (tests, parameter scans): launches and their latency
        _comm("comm_e2_fp64", 2, 1, "fp64"),
        _comm("comm_e2_split6", 2, 1, "ozaki", 6),
        # a term of the Magnus series, [Omega, Omega'] without E0, in plain FP64
        _comm("comm_e4_fp64_magnus", 4, 2, "fp64", 6, -1, -1, False),
        # an odd emax with a small hole space, library-default digits
        _comm("comm_e5_split6", 5, 1, "ozaki", 6),
        # the headline workload: [Omega, H] at emax 6, five digits
        _comm("comm_e6_split5", 6, 2, "ozaki", 5),
        # the same in plain FP64
        _comm("comm_e6_fp64", 6, 2, "fp64"),
        # host-resident operators in the packed (vectorize) layout, page-locked:
        # what a host driver without resident operators pays per commutator
        dict(name="host_e6_split5", op="host_packed", emax=6, filled=2, precision="ozaki", digits=5, herm_L=-1,
             herm_R=1, with_e0=True, hw=20.0, sigma=1.0),
        # a scan over oscillator frequencies and couplings: independent
        # commutators of mixed emax in one call
        dict(name="batch12_split5", op="batch", n=12, precision="ozaki", digits=5, hw=20.0, sigma=1.0),
        # backward direction: d<C, [X, Y]>/dY of the gradient sweep
        dict(name="adjoint_e4", op="adjoint", emax=4, filled=2, herm_L=-1, herm_R=1, with_e0=True, hw=20.0,
             sigma=1.0),
        dict(name="adjoint_e6", op="adjoint", emax=6, filled=2, herm_L=-1, herm_R=1, with_e0=True, hw=20.0,
             sigma=1.0),
        # whole calls: graph-captured Magnus steps (generator, both series, E0)
        dict(name="flow_e4_split6", op="flow", emax=4, filled=2, precision="ozaki", digits=6, steps=3, hw=20.0,
             sigma=1.0),
        dict(name="flow_e6_split5", op="flow", emax=6, filled=2, precision="ozaki", digits=5, steps=2, hw=20.0,
             sigma=1.0),
    ]


def draw(rng):
    op = rng.choice(["commutator"] * 4 + ["host_packed", "batch", "adjoint", "flow"])
    c = dict(op=op, hw=round(rng.uniform(12.0, 28.0), 3), sigma=round(rng.uniform(0.5, 2.0), 3))
    c["precision"], c["digits"] = rng.choice([("fp64", 6), ("ozaki", 5), ("ozaki", 6), ("ozaki", 8)])
    if op == "batch":
        c["n"] = rng.randint(3, 12)
        return c
    c["emax"] = rng.randint(2, 6)
    c["filled"] = rng.randint(1, 2)
    if op == "flow":
        c["steps"] = rng.randint(1, 3 if c["emax"] < 5 else 1)
        return c
    c["herm_L"], c["herm_R"], c["with_e0"] = rng.choice([(-1, 1, True), (-1, 1, True), (-1, -1, False), (1, 1, True)])
    if op == "adjoint":
        del c["precision"], c["digits"]
    return c


# --- single-particle space and block layout ------------------------------------
class Space:
    """Orbits, (2J, Tz, parity) blocks and the flat operator layout
    [E0 | fhh | fph | fpp | per block gam 1..6], all matrices column-major."""

    def __init__(self, emax, filled):
        orb = [(n, l, j, t) for e in range(emax + 1) for l in range(e, -1, -2) for n in [(e - l) // 2]
               for j in (2 * l - 1, 2 * l + 1) if j > 0 for t in (-1, 1)]
        self.nn, self.ll, self.jj, self.tz = (np.array(x) for x in zip(*orb))
        self.con = (2 * self.nn + self.ll < filled).astype(np.int64)
        N = self.N = len(orb)
        self.holes, self.parts = np.flatnonzero(self.con == 1), np.flatnonzero(self.con == 0)
        A, P = self.A, self.P = len(self.holes), len(self.parts)
        self.pos = np.zeros(N, np.int64)
        self.pos[self.holes], self.pos[self.parts] = np.arange(A), np.arange(P)
        self.jtm = int(self.jj.max())
        self.o_hh, self.o_ph, self.o_pp = 1, 1 + A * A, 1 + A * A + P * A
        self.o_two = off = self.o_pp + P * P
        same = lambda x: x[:, None] == x[None, :]  # noqa: E731
        self.allowed = same(self.jj) & same(self.ll) & same(self.tz)
        self.blocks, self.row = [], np.full((self.jtm + 1, N, N), -1)
        ia, ib = np.triu_indices(N)
        for J2 in range(0, 2 * self.jtm + 1, 2):
            ok = (abs(self.jj[ia] - self.jj[ib]) <= J2) & (J2 <= self.jj[ia] + self.jj[ib])
            for t in (-1, 0, 1):
                for par in (0, 1):
                    m = ok & (self.tz[ia] + self.tz[ib] == 2 * t) & ((self.ll[ia] + self.ll[ib]) % 2 == par)
                    pairs = []
                    for cat in range(3):
                        k = m & (self.con[ia] + self.con[ib] == cat)
                        pairs.append(np.stack([ia[k], ib[k]], 1))
                        self.row[J2 // 2, ia[k], ib[k]] = np.arange(k.sum())
                    n = [len(p) for p in pairs]
                    offs, dims = [], []
                    for g in range(6):
                        offs.append(off)
                        dims.append((n[ROWCAT[g]], n[COLCAT[g]]))
                        off += dims[-1][0] * dims[-1][1]
                    self.blocks.append((J2, pairs, n, offs, dims))
        self.nfull = off
        self.goff = np.array([b[3] for b in self.blocks])
        self.gn1 = np.array([[d[0] for d in b[4]] for b in self.blocks])

    def packed_index(self):
        """Flat index of each packed (vectorize) element: E0, fhh, fpp, fph,
        then per block and array the lower triangle (square) or everything, by
        columns."""
        out = [[0], np.arange(self.o_hh, self.o_ph), np.arange(self.o_pp, self.o_two),
               np.arange(self.o_ph, self.o_pp)]
        for _, _, _, offs, dims in self.blocks:
            for g in range(6):
                n1, n2 = dims[g]
                r, c = np.arange(n1)[None, :], np.arange(n2)[:, None]
                k = offs[g] + r + c * n1
                out.append(k[(r >= c)] if SQUARE[g] else k.ravel())
        return np.concatenate(out)

    def random(self, rng, herm, sigma, sigma1, spectrum=None):
        """A seeded operator; identical-orbit pairs vanish at odd J."""
        x = np.zeros(self.nfull)
        A, P = self.A, self.P
        for o, rows, cols in ((self.o_hh, self.holes, self.holes), (self.o_ph, self.parts, self.holes),
                              (self.o_pp, self.parts, self.parts)):
            m = rng.normal(0.0, sigma1, (len(rows), len(cols)))
            if rows is cols:
                m = np.triu(m, 1)
                m = m + herm * m.T
                if spectrum is not None:
                    m[np.diag_indices(len(rows))] = spectrum[rows]
                elif herm < 0:
                    m[:] = 0.0
            m = m * self.allowed[np.ix_(rows, cols)]
            x[o:o + m.size] = m.T.ravel()
        for J2, pairs, _, offs, dims in self.blocks:
            live = [1.0 - ((p[:, 0] == p[:, 1]) & (J2 // 2 % 2 == 1)) for p in pairs]
            for g in range(6):
                if dims[g][0] * dims[g][1] == 0:
                    continue
                m = rng.normal(0.0, sigma, dims[g])
                if SQUARE[g]:
                    m = np.triu(m) + herm * np.triu(m, 1).T
                    if herm < 0:
                        m[np.diag_indices(len(m))] = 0.0
                m = m * live[ROWCAT[g]][:, None] * live[COLCAT[g]][None, :]
                x[offs[g]:offs[g] + m.size] = m.T.ravel()
        return x


@functools.lru_cache(maxsize=None)
def space(emax, filled):
    return Space(emax, filled)


def _operator(sp, rng, herm, case):
    if herm > 0:
        return sp.random(rng, 1, case["sigma"], 0.5, case["hw"] * (2 * sp.nn + sp.ll + 1.5))
    return sp.random(rng, -1, 0.05, 0.05)


def _inputs(case, seed):
    """The operators of a case in the flat layout, as numpy arrays."""
    rng = np.random.Generator(np.random.Philox(key=int(seed)))
    if case["op"] == "batch":
        out = []
        for k in range(case["n"]):
            sp = _batch_space(k)
            c = dict(hw=case["hw"] * rng.uniform(0.8, 1.2), sigma=case["sigma"] * rng.uniform(0.7, 1.4))
            out.append((_operator(sp, rng, -1, c), _operator(sp, rng, 1, c)))
        return out
    sp = space(case["emax"], case["filled"])
    if case["op"] == "flow":
        return [_operator(sp, rng, 1, case)]
    second = -case["herm_L"] * case["herm_R"] if case["op"] == "adjoint" else case["herm_R"]
    pair = [_operator(sp, rng, case["herm_L"], case), _operator(sp, rng, second, case)]
    if case["op"] == "adjoint":
        pair[1][0] = 1.0  # the E0 component of the incoming gradient
    return pair


def _batch_space(k):
    return space((2, 4, 6)[k % 3], (1, 2, 2)[k % 3])


# --- states and passes ---------------------------------------------------------
@functools.lru_cache(maxsize=None)
def basis(emax, filled, digits, k=0):
    from imsrg_gpu import api
    sp = space(emax, filled)
    b = api.Basis(sp.nn, sp.ll, sp.jj, sp.tz, sp.con)
    b.set_split_digits(digits)
    return b


@functools.lru_cache(maxsize=None)
def _batch(n, digits):
    from imsrg_gpu import api
    bases = [basis((2, 4, 6)[k % 3], (1, 2, 2)[k % 3], digits, k // 3 + 1) for k in range(n)]
    return api.Batch(bases)


@functools.lru_cache(maxsize=None)
def _flow_ops(b):
    """The evolving H and Omega of a basis: a program that flows several
    Hamiltonians loads each into the same pair."""
    from imsrg_gpu import api
    return api.Operator(b, 1), api.Operator(b, -1)


class _View:
    """Zero-copy description of an operator's flat device buffer; a tensor made
    from it holds it, and so the operator, for as long as it lives."""

    def __init__(self, op):
        self.op = op
        self.__cuda_array_interface__ = dict(shape=(op.basis.nfull,), typestr="<f8", data=(op.device_ptr(), False),
                                             version=3)


def _tensor(op):
    return torch.as_tensor(_View(op), device="cuda")


def prepare(case, seed):
    from imsrg_gpu import api
    x = _inputs(case, seed)
    op = case["op"]
    if op == "batch":
        bt = _batch(case["n"], case["digits"])
        L = [api.Operator(b, -1, p[0]) for b, p in zip(bt.bases, x)]
        R = [api.Operator(b, 1, p[1]) for b, p in zip(bt.bases, x)]
        RES = [api.Operator(b, 1) for b in bt.bases]
        return dict(case=case, batch=bt, L=L, R=R, RES=RES, out=[_tensor(r) for r in RES])
    b = basis(case["emax"], case["filled"], case.get("digits", 6))
    if op == "flow":
        HS, G = _flow_ops(b)
        return dict(case=case, H0=api.Operator(b, 1, x[0]), HS=HS, G=G, out=[_tensor(HS), _tensor(G)])
    if op == "host_packed":
        k = space(case["emax"], case["filled"]).packed_index()
        bufs = [torch.from_numpy(v[k]).pin_memory() for v in x] + [torch.zeros(len(k), dtype=torch.float64).pin_memory()]
        return dict(case=case, basis=b, keep=bufs, arrays=[t.numpy() for t in bufs])
    hL, hR = case["herm_L"], case["herm_R"]
    L = api.Operator(b, hL, x[0])
    R = api.Operator(b, -hL * hR if op == "adjoint" else hR, x[1])
    RES = api.Operator(b, 1)
    return dict(case=case, L=L, R=R, RES=RES, out=_tensor(RES))


def run(state):
    from imsrg_gpu import api
    c = state["case"]
    op = c["op"]
    if op == "commutator":
        api.commutator(state["L"], state["R"], state["RES"], c["precision"], c["with_e0"])
        return state["out"]
    if op == "host_packed":
        L, R, RES = state["arrays"]
        api.commutator_host_packed(state["basis"], L, c["herm_L"], R, c["herm_R"], RES, c["precision"], c["with_e0"])
        return RES
    if op == "batch":
        state["batch"].commutator(state["L"], state["R"], state["RES"], c["precision"])
        return state["out"]
    if op == "adjoint":
        api.commutator_adjoint(state["L"], state["R"], c["herm_R"], state["RES"], c["with_e0"])
        return state["out"]
    api.copy_sq_op(state["H0"], state["HS"])
    r = api.magnus_decouple_graph(state["HS"], state["G"], s_max=50.0, ds=0.5, max_steps=c["steps"],
                                  precision=c["precision"])
    return state["out"] + [r["trace"]]


# --- the work a pass cannot do without -----------------------------------------
@functools.lru_cache(maxsize=None)
def _flops(emax, filled):
    """Multiply-adds (x 2) of one commutator's dense contractions: twelve
    ladder products per block and the particle-hole product per cross-coupled
    block, pairs of one isospin projection at a time."""
    sp = space(emax, filled)
    f = 0
    for _, _, (p, x, h), _, _ in sp.blocks:
        f += p**3 + h**3 + h * h * p + p * p * h + 2 * (p * h * p + p * h * h) + x * x * h + x * x * p
        f += 2 * (x * h * h + p * x * p + x * h * p + p * x * h)
    d = (sp.tz[:, None] - sp.tz[None, :]) // 2
    par = (sp.ll[:, None] + sp.ll[None, :]) % 2
    ph = (sp.con[:, None] == 0) & (sp.con[None, :] == 1)
    for J2 in range(0, 2 * sp.jtm + 1, 2):
        tri = (abs(sp.jj[:, None] - sp.jj[None, :]) <= J2) & (J2 <= sp.jj[:, None] + sp.jj[None, :])
        for t in (-1, 0, 1):
            for q in (0, 1):
                m = tri & (d == t) & (par == q)
                f += int(m.sum()) ** 2 * int((m & ph).sum())
    return 2.0 * f


def work(case):
    if case["op"] == "batch":
        spaces = [(2, 4, 6)[k % 3] for k in range(case["n"])]
        return dict(bytes=sum(24.0 * _batch_space(k).nfull for k in range(case["n"])),
                    flops=sum(_flops(e, 1 if e == 2 else 2) for e in spaces))
    sp = space(case["emax"], case["filled"])
    f = _flops(case["emax"], case["filled"])
    if case["op"] == "flow":  # two series of about twelve terms in all per step
        return dict(bytes=24.0 * sp.nfull * 12 * case["steps"], flops=12 * case["steps"] * f)
    if case["op"] == "host_packed":
        return dict(bytes=24.0 * len(sp.packed_index()), flops=f)
    return dict(bytes=24.0 * sp.nfull, flops=f)


# --- the same results in plain 64-bit torch on the CPU ---------------------------
def _sixj(j1, j2, J3, j4, j5, J6):
    """{j1 j2 J3; j4 j5 J6} for integer arrays of doubled arguments (Racah's
    single sum in extended precision)."""
    a, b, c, d, e, f = (np.asarray(x) for x in np.broadcast_arrays(j1, j2, J3, j4, j5, J6))
    fact = np.concatenate([[np.longdouble(1)], np.cumprod(np.arange(1, 120, dtype=np.longdouble))])
    ok = np.ones(a.shape, bool)
    for x, y, z in ((a, b, c), (a, e, f), (d, b, f), (d, e, c)):
        ok &= (abs(x - y) <= z) & (z <= x + y) & ((x + y + z) % 2 == 0)
    out = np.zeros(a.shape, np.longdouble)
    a, b, c, d, e, f = (x[ok] for x in (a, b, c, d, e, f))
    s = [(a + b + c) // 2, (a + e + f) // 2, (d + b + f) // 2, (d + e + c) // 2]
    p = [(a + b + d + e) // 2, (b + c + e + f) // 2, (c + a + f + d) // 2]
    lo, hi = np.maximum.reduce(s), np.minimum.reduce(p)
    tot = np.zeros(a.shape, np.longdouble)
    for k in range(int((hi - lo).max()) + 1 if len(a) else 0):
        t = lo + k
        m = t <= hi
        term = fact[t[m] + 1]
        for x in s:
            term = term / fact[(t - x)[m]]
        for x in p:
            term = term / fact[(x - t)[m]]
        tot[m] += np.where(t[m] % 2, -1, 1) * term
    for x, y, z in ((a, b, c), (a, e, f), (d, b, f), (d, e, c)):
        tot = tot * np.sqrt(fact[(x + y - z) // 2] * fact[(x - y + z) // 2] * fact[(-x + y + z) // 2] /
                            fact[(x + y + z) // 2 + 1])
    out[ok] = tot
    return out.astype(np.float64)


def _t(x):
    return torch.from_numpy(np.ascontiguousarray(x))


class Exact:
    """The J-coupled IMSRG(2) commutator, White generator and Magnus flow on
    flat 64-bit torch vectors."""

    def __init__(self, sp):
        self.sp = sp
        N, jtm = sp.N, sp.jtm
        h = np.arange((jtm + 1) // 2)
        J = np.arange(jtm + 1)
        g = np.meshgrid(h, h, h, h, J, J, indexing="ij")
        self.six = _sixj(2 * g[0] + 1, 2 * g[1] + 1, 2 * g[4], 2 * g[2] + 1, 2 * g[3] + 1, 2 * g[5])
        # f(a, b) over all orbits: flat index, and whether it takes herm (hole-particle)
        c, pos = sp.con, sp.pos
        a, b = np.meshgrid(np.arange(N), np.arange(N), indexing="ij")
        s = c[a] + c[b]
        self.fidx = np.where(s == 0, sp.o_pp + pos[a] + pos[b] * sp.P,
                             np.where(s == 2, sp.o_hh + pos[a] + pos[b] * sp.A,
                                      np.where(c[a] > c[b], sp.o_ph + pos[b] + pos[a] * sp.P,
                                               sp.o_ph + pos[a] + pos[b] * sp.P)))
        self.ftrans = _t((c[a] > c[b]).astype(np.float64))
        self.fidx = _t(self.fidx)
        self._one_body()
        self._pairs()
        self._cross()
        self._elements()

    def loc(self, a, b, c, d, J2):
        """<a b|V|c d>_J: flat index (-1: zero), factor, read transposed."""
        sp = self.sp
        a, b, c, d, J2 = np.broadcast_arrays(a, b, c, d, J2)
        j, t, l = sp.jj, sp.tz, sp.ll
        ok = (abs(j[a] - j[b]) <= J2) & (J2 <= j[a] + j[b]) & (abs(j[c] - j[d]) <= J2) & (J2 <= j[c] + j[d])
        ok = ok & (t[a] + t[b] == t[c] + t[d]) & ((l[a] + l[b] + l[c] + l[d]) % 2 == 0) & (J2 <= 2 * sp.jtm)
        Jc = np.where(ok, J2, 0)
        q = 3 * Jc + (t[a] + t[b]) + 2 + (l[a] + l[b]) % 2
        fac = np.ones(a.shape)
        rows = []
        for x, y in ((a, b), (c, d)):
            fac = fac * np.where((x > y) & ((1 + (j[x] + j[y] - J2) // 2) % 2 == 1), -1.0, 1.0)
            fac = fac * np.where(x == y, np.sqrt(2.0), 1.0)
            rows.append(sp.row[Jc // 2, np.minimum(x, y), np.maximum(x, y)])
        C1, C2 = sp.con[a] + sp.con[b], sp.con[c] + sp.con[d]
        gam = np.array([[0, 1, 2], [1, 3, 5], [2, 5, 4]])[C1, C2]
        tr = C1 > C2
        r, s = np.where(tr, rows[1], rows[0]), np.where(tr, rows[0], rows[1])
        idx = np.where(ok, sp.goff[q, gam] + r + s * sp.gn1[q, gam], -1)
        return idx, np.where(ok, fac, 0.0), tr

    def read(self, x, herm, loc):
        idx, fac, tr = loc
        return x[_t(np.maximum(idx, 0))] * _t(fac * np.where(tr, float(herm), 1.0))

    def f(self, x, herm):
        return x[self.fidx] * (1.0 + (herm - 1.0) * self.ftrans)

    def _one_body(self):
        """Gather lists of the 121 and 221 sums of the (l,j,tz)-allowed one-body
        elements (rows p <= q of square arrays)."""
        sp = self.sp
        p, q = np.nonzero(sp.allowed & ((sp.con[:, None] != sp.con[None, :]) | (np.arange(sp.N)[:, None] <= np.arange(sp.N)[None, :])) &
                          ~((sp.con[:, None] == 1) & (sp.con[None, :] == 0)))
        self.ob = (p, q)
        J = np.arange(0, 2 * sp.jtm + 1, 2)
        i, k = np.nonzero(sp.allowed & (sp.con[:, None] == 0) & (sp.con[None, :] == 1))  # (particle, hole)
        e, m, JJ = np.meshgrid(np.arange(len(p)), np.arange(len(i)), J, indexing="ij")
        self.l121 = [self.loc(i[m], p[e], k[m], q[e], JJ), self.loc(k[m], p[e], i[m], q[e], JJ)]
        self.l121_ph = (i, k)
        self.l121_w = (JJ + 1.0) / (sp.jj[p[e]] + 1.0)
        e, m, JJ = np.meshgrid(np.arange(len(p)), np.arange(sp.N), J, indexing="ij")
        self.l221 = [self.loc(m, p[e], m, q[e], JJ), self.loc(m, q[e], m, p[e], JJ)]
        self.l221_w = (JJ + 1.0) / (sp.jj[p[e]] + 1.0)
        self.l221_hole = sp.con[m] == 1
        self.l221_square = (sp.con[p] == sp.con[q])[:, None, None]
        self.l221_diag = (p == q)[:, None, None]

    def _pairs(self):
        """Per block: the one-body insertion matrices of the 122 sums as
        (row, column, f index, factor) lists, and 1/sqrt(1 + delta)."""
        sp = self.sp
        self.ins = []
        for J2, pairs, n, _, _ in sp.blocks:
            u = np.concatenate(pairs)
            nu = len(u)
            base = np.concatenate([[0], np.cumsum(n)])
            D = np.where(u[:, 0] == u[:, 1], np.sqrt(0.5), 1.0) if nu else np.zeros(0)
            lst = []
            for leg in (0, 1):
                r, x = np.nonzero(sp.allowed[u[:, leg]]) if nu else (np.zeros(0, int),) * 2
                a, b = (x, u[r, 1]) if leg == 0 else (u[r, 0], x)
                lo, hi = np.minimum(a, b), np.maximum(a, b)
                col = base[sp.con[lo] + sp.con[hi]] + sp.row[J2 // 2, lo, hi]
                fac = np.where((a > b) & ((1 + (sp.jj[a] + sp.jj[b] - J2) // 2) % 2 == 1), -1.0, 1.0)
                fac = fac * np.where(a == b, np.sqrt(2.0), 1.0) * D[r]
                lst.append((r, col, u[r, leg], x, fac))
            r, col, o, x, fac = (np.concatenate(z) for z in zip(*lst))
            self.ins.append((nu, _t(r * nu + col), _t(o * sp.N + x), _t(col * nu + r), _t(x * sp.N + o), _t(fac)))

    def _cross(self):
        """Cross-coupled blocks (J', |Tz|, parity): rows all ordered pairs,
        columns (particle, hole), with the transform's gather list."""
        sp = self.sp
        N, jtm = sp.N, sp.jtm
        a, b = (x.ravel() for x in np.meshgrid(np.arange(N), np.arange(N), indexing="ij"))
        self.ccrow = np.full((4 * (jtm + 1), N, N), -1)
        self.cc, el, ix, cf, tr = [], [], [], [], []
        off = woff = 0
        for q1 in range(4 * (jtm + 1)):
            JC, PAR, TZ = q1 % (jtm + 1) * 2, q1 // (2 * jtm + 2), q1 % (2 * jtm + 2) // (jtm + 1)
            m = (abs(sp.jj[a] - sp.jj[b]) <= JC) & (JC <= sp.jj[a] + sp.jj[b]) & \
                ((sp.ll[a] + sp.ll[b]) % 2 == PAR) & (abs(sp.tz[a] - sp.tz[b]) // 2 == TZ)
            ra, rb = a[m], b[m]
            k = m & (sp.con[a] == 0) & (sp.con[b] == 1)
            p, h = a[k], b[k]
            r, c = len(ra), len(p)
            self.ccrow[q1, ra, rb] = np.arange(r)
            self.cc.append((off, woff, r, c))
            if r * c:
                e = off + np.arange(r)[:, None] + r * np.arange(c)[None, :]
                A, B, Pp, Hh = (np.broadcast_to(x, (r, c)) for x in (ra[:, None], rb[:, None], p[None, :], h[None, :]))
                outer = np.where((sp.jj[Hh] + sp.jj[B] + JC) // 2 % 2 == 1, -1.0, 1.0) * np.sqrt(JC + 1.0)
                for J2 in range(0, 2 * jtm + 1, 2):
                    idx, fac, t = self.loc(Hh, A, Pp, B, J2)
                    g = idx >= 0
                    if g.any():
                        s = self.six[sp.jj[Pp] // 2, sp.jj[Hh] // 2, sp.jj[A] // 2, sp.jj[B] // 2, JC // 2, J2 // 2]
                        w = (-1.0 if J2 // 2 % 2 else 1.0) * (J2 + 1) * s * outer * fac
                        el.append(e[g])
                        ix.append(idx[g])
                        cf.append(w[g])
                        tr.append(t[g])
            off += r * c
            woff += r * r
        self.ncc = off
        self.ccl = [np.concatenate(x) if x else np.zeros(0, int) for x in (el, ix, cf, tr)]

    def _elements(self):
        """Upper-triangle two-body elements with their recoupling gather lists."""
        sp = self.sp
        cols = [[] for _ in range(9)]
        for J2, pairs, _, offs, dims in sp.blocks:
            for g in range(6):
                n1, n2 = dims[g]
                if n1 * n2 == 0:
                    continue
                I, K = (x.ravel() for x in np.meshgrid(np.arange(n1), np.arange(n2), indexing="ij"))
                if SQUARE[g]:
                    I, K = I[I <= K], K[I <= K]
                pr, pc = pairs[ROWCAT[g]], pairs[COLCAT[g]]
                e = offs[g] + I + K * n1
                em = offs[g] + K + I * n1 if SQUARE[g] else e
                for lst, v in zip(cols, (e, em, pr[I, 0], pr[I, 1], pc[K, 0], pc[K, 1], np.full(len(e), J2),
                                         np.full(len(e), SQUARE[g]), (I == K) & SQUARE[g])):
                    lst.append(v)
        e, em, i, j, k, l, J2, sq, dg = (np.concatenate(x) for x in cols)
        self.e, self.em, self.sq, self.dg = e, em, sq, dg
        jj, JT = sp.jj, sp.jtm + 1
        nd = (i == j).astype(int) + (k == l)
        lit = .70710678118
        norm = np.where(nd == 0, 1.0, np.where(nd == 1, lit, lit * lit))
        ph = np.where((jj[i] + jj[j] + jj[k] + jj[l]) // 2 % 2 == 1, -1.0, 1.0)
        self.rec = []
        for u, v, sign in ((k, l, np.where((jj[l] + jj[k] + J2) // 2 % 2 == 0, -1.0, 1.0)), (l, k, 1.0)):
            # channel i-u, j-v: rows (u, i), (j, v), (v, j), (i, u)
            lo = np.maximum(abs(jj[j] - jj[v]), abs(jj[i] - jj[u]))
            hi = np.minimum(jj[j] + jj[v], jj[i] + jj[u])
            q0 = abs(sp.tz[i] - sp.tz[u]) // 2 * JT + 2 * JT * ((sp.ll[i] + sp.ll[u]) % 2)
            for step in range(int((hi - lo).max()) // 2 + 1):
                JP = lo + 2 * step
                m = np.flatnonzero(JP <= hi)
                if not len(m):
                    continue
                q1 = q0[m] + JP[m] // 2
                rows = [self.ccrow[q1, x[m], y[m]] for x, y in ((u, i), (j, v), (v, j), (i, u))]
                w0 = np.array([c[1] for c in self.cc])[q1]
                r = np.array([c[2] for c in self.cc])[q1]
                at = [w0 + x + y * r for x, y in ((rows[0], rows[1]), (rows[2], rows[3]), (rows[3], rows[2]),
                                                  (rows[1], rows[0]))]
                s6 = self.six[jj[i][m] // 2, jj[j][m] // 2, jj[v][m] // 2, jj[u][m] // 2, J2[m] // 2, JP[m] // 2]
                coef = s6 * norm[m] * (sign[m] if np.ndim(sign) else sign)
                self.rec.append((_t(m), [_t(x) for x in at], _t(coef), _t(ph[m])))

    def full(self, x, herm, blk):
        _, _, (p, b, h), offs, dims = blk
        g = [x[o:o + n1 * n2].reshape(n2, n1).T for o, (n1, n2) in zip(offs, dims)]
        return torch.cat([torch.cat([g[0], g[1], g[2]], 1), torch.cat([herm * g[1].T, g[3], g[5]], 1),
                          torch.cat([herm * g[2].T, herm * g[5].T, g[4]], 1)], 0)

    def commutator(self, L, hL, R, hR, with_e0=True):
        sp = self.sp
        hS = -hL * hR
        A, P = sp.A, sp.P
        fL, fR = self.f(L, hL), self.f(R, hR)
        two = torch.zeros(sp.nfull, dtype=torch.float64)
        # 122 sums, ladder products and W1, W2 for the 221 sums, block by block
        c122, lad, W1, W2 = [torch.zeros(sp.o_two, dtype=torch.float64)], [torch.zeros(sp.o_two, dtype=torch.float64)], \
            [torch.zeros(sp.o_two, dtype=torch.float64)], [torch.zeros(sp.o_two, dtype=torch.float64)]
        for blk, (nu, lin, fi, linT, fiT, fac) in zip(sp.blocks, self.ins):
            if nu == 0:
                continue
            VL, VR = self.full(L, hL, blk), self.full(R, hR, blk)
            ins = lambda f: (torch.zeros(nu * nu, dtype=torch.float64).index_add(0, lin, fac * f.reshape(-1)[fi]).view(nu, nu),  # noqa: E731
                             torch.zeros(nu * nu, dtype=torch.float64).index_add(0, linT, fac * f.reshape(-1)[fiT]).view(nu, nu))
            aL, bL = ins(fL)
            aR, bR = ins(fR)
            T = aL @ VR - VR @ bL - aR @ VL + VL @ bR
            p, b, h = blk[2]
            w = [VL[:, :p] @ VR[:p], VL[:, p + b:] @ VR[p + b:]]
            v = [VR[:, :p] @ VL[:p], VR[:, p + b:] @ VL[p + b:]]
            cut = [slice(0, p), slice(p, p + b), slice(p + b, nu)]
            for g in range(6):
                rc = (cut[ROWCAT[g]], cut[COLCAT[g]])
                flat = lambda m: m.T.reshape(-1)  # noqa: E731
                c122.append(flat(T[rc]))
                x1, x2 = (w[0][rc], w[1][rc]) if SQUARE[g] else (w[0][rc] - v[0][rc], w[1][rc] - v[1][rc])
                W1.append(flat(x1))
                W2.append(flat(x2))
                d = x1 - x2
                lad.append(flat(d - (hL * hR) * d.T if SQUARE[g] else d))
        c122, lad, W1, W2 = (torch.cat(x) for x in (c122, lad, W1, W2))
        # particle-hole products and their recoupling
        el, ix, cf, tr = self.ccl
        cc = [torch.zeros(self.ncc, dtype=torch.float64).index_add(0, _t(el), x[_t(ix)] * _t(cf * np.where(tr, float(hx), 1.0)))
              for x, hx in ((L, hL), (R, hR))]
        wcc = []
        for o, _, r, c in self.cc:
            X, Y = (z[o:o + r * c].reshape(c, r) for z in cc)
            wcc.append((Y.T @ X).reshape(-1))  # column-major W(x, y) = sum X(x) Y(y)
        wcc = torch.cat(wcc)
        rec = torch.zeros(len(self.e), dtype=torch.float64)
        for m, at, coef, ph in self.rec:
            w = [wcc[x] for x in at]
            z = hL * (w[0] + ph * w[1]) - hR * (ph * w[2] + w[3])
            rec = rec.index_add(0, m, coef * z)
        e, em = _t(self.e), _t(self.em)
        rest = lad[e] + rec
        t = c122[e] + torch.where(_t(self.dg), hS * rest, rest)
        off = _t(np.flatnonzero(self.sq & ~self.dg))
        two = two.index_copy(0, e, t).index_copy(0, em[off], hS * t[off])
        # one-body part
        one = fL @ fR - fR @ fL
        p, q = self.ob
        i, k = self.l121_ph
        w = _t(self.l121_w)
        x = 0.0
        for f, g, hg in ((fL, R, hR), (fR, L, hL)):
            up = f[_t(k), _t(i)][None, :, None] * self.read(g, hg, self.l121[0])
            dn = f[_t(i), _t(k)][None, :, None] * self.read(g, hg, self.l121[1])
            x = (up - dn) if f is fL else x - (up - dn)
        s121 = (w * x).sum((1, 2))
        hole = _t(self.l221_hole)
        y = torch.where(hole, self.read(W1, 1, self.l221[0]), self.read(W2, 1, self.l221[0]))
        y2 = torch.where(hole, self.read(W1, 1, self.l221[1]), self.read(W2, 1, self.l221[1]))
        y = y - (hL * hR) * torch.where(_t(self.l221_square), y2, torch.zeros_like(y2))
        y = torch.where(_t(self.l221_diag), hS * y, y)
        s221 = (_t(self.l221_w) * y).sum((1, 2))
        val = one[_t(p), _t(q)] + s121 + s221
        one = one.index_put((_t(p), _t(q)), val)
        mir = (sp.con[p] == sp.con[q]) & (p != q)
        one = one.index_put((_t(q[mir]), _t(p[mir])), hS * val[_t(np.flatnonzero(mir))])
        H, Pt = _t(sp.holes), _t(sp.parts)
        parts = [one[H][:, H].T.reshape(-1), one[Pt][:, H].T.reshape(-1), one[Pt][:, Pt].T.reshape(-1)]
        e0 = torch.zeros(1, dtype=torch.float64)
        if with_e0:
            lp, rp = (z[sp.o_ph:sp.o_pp].reshape(A, P) for z in (L, R))
            e0 = e0 + (hL - hR) * ((lp * rp).sum(1) * _t(sp.jj[sp.holes] + 1.0)).sum()
            for J2, _, _, offs, dims in sp.blocks:
                n = dims[2][0] * dims[2][1]
                if n and hL * hR == -1:
                    e0 = e0 - 2.0 * hR * (J2 + 1) * (L[offs[2]:offs[2] + n] * R[offs[2]:offs[2] + n]).sum()
        return torch.cat([e0] + parts + [two[sp.o_two:]])

    # --- the Magnus flow ---
    def white(self, H):
        sp = self.sp
        f = self.f(H, 1).numpy()
        d = np.diag(f)
        a, b = np.meshgrid(np.arange(sp.N), np.arange(sp.N), indexing="ij")
        mono = np.zeros((sp.N, sp.N))
        cross = np.zeros((sp.N, sp.N))
        for J2 in range(0, 2 * sp.jtm + 1, 2):
            v = (J2 + 1) * self.read(H, 1, self.loc(a, b, a, b, J2)).numpy()
            mono += v
            cross += np.where(J2 <= 2 * sp.jj[b], v, 0.0)
        mono = mono / (sp.jj[a] + 1.0) / (sp.jj[b] + 1.0)
        cross = cross / (sp.jj[b] + 1.0) ** 2
        eta = np.zeros(sp.nfull)
        p, h = np.ix_(sp.parts, sp.holes), None
        den = d[sp.parts][:, None] - d[sp.holes][None, :] - cross[p]
        ok = sp.allowed[p]
        eta[sp.o_ph:sp.o_pp] = np.where(ok, f[p] / np.where(ok, den, 1.0), 0.0).T.ravel()
        x = H.numpy()
        e2 = 0.0
        for J2, pairs, _, offs, dims in sp.blocks:
            n1, n2 = dims[2]
            if n1 * n2 == 0:
                continue
            (a, b), (i, j) = (pairs[0][:, :, None]).transpose(1, 0, 2), (pairs[2][:, :, None]).transpose(1, 2, 0)
            den = mono[a, b] + mono[i, j] - mono[a, i] - mono[a, j] - mono[i, b] - mono[j, b]
            den = den + d[a] + d[b] - d[i] - d[j]
            g = x[offs[2]:offs[2] + n1 * n2].reshape(n2, n1).T
            eta[offs[2]:offs[2] + n1 * n2] = (g / den).T.ravel()
            e2 += (J2 + 1.0) * (g * g / (d[i] + d[j] - d[a] - d[b])).sum()
        return _t(eta), float(e2)

    def norm(self, x):
        sp = self.sp
        s = float((x[sp.o_hh:] ** 2).sum()) + float((x[sp.o_ph:sp.o_pp] ** 2).sum())
        for _, _, _, offs, dims in sp.blocks:
            s += sum(float((x[offs[g]:offs[g] + dims[g][0] * dims[g][1]] ** 2).sum()) for g in (1, 2, 5))
        return np.sqrt(s)

    def flow(self, H0, ds, steps):
        cof = (1.0, -0.5, .0833333333, 0.0, -0.00138888888, 0.0, 3.306878e-5)
        G = torch.zeros_like(H0)
        HS, s = H0, 0.0
        eta, e2 = self.white(H0)
        trace = [[0.0, 0.0, float(H0[0]), float(H0[0]) + e2, abs(e2)]]
        while abs(e2) > 1e-6 and len(trace) <= steps:
            X, DG, adv, full, look = eta, eta, [0.0, self.norm(eta)] + [0.0] * 6, self.norm(G), 1
            for i in range(2, 8):
                if full < 1e-9:
                    break
                small = abs(adv[i - look] / full) < 1e-6
                look = 1 if abs(cof[i - 1]) > 1e-6 else 2
                if small:
                    break
                X = self.commutator(G, -1, X, -1, False)
                DG = DG + cof[i - 1] * X
                adv[i] = self.norm(X) * abs(cof[i - 1])
            G = G + ds * DG
            s += ds
            HS, X, coef = H0, H0, 1.0
            for n in range(2, 41):
                X = self.commutator(G, -1, X, 1)
                HS = HS + coef * X
                if self.norm(X) * coef < 1e-6:
                    break
                coef = coef / n
            eta, e2 = self.white(HS)
            trace.append([float(len(trace)), s, float(HS[0]), float(HS[0]) + e2, abs(e2)])
        return HS, G, np.array(trace)


@functools.lru_cache(maxsize=4)
def _exact(emax, filled):
    return Exact(space(emax, filled))


def exact(case, seed):
    x = _inputs(case, seed)
    op = case["op"]
    if op == "batch":
        return [_exact((2, 4, 6)[k % 3], (1, 2, 2)[k % 3]).commutator(_t(L), -1, _t(R), 1).numpy()
                for k, (L, R) in enumerate(x)]
    E = _exact(case["emax"], case["filled"])
    if op == "flow":
        HS, G, trace = E.flow(_t(x[0]), 0.5, case["steps"])
        return [HS.numpy(), G.numpy(), trace]
    hL, hR = case["herm_L"], case["herm_R"]
    if op == "adjoint":
        Y = torch.zeros(E.sp.nfull, dtype=torch.float64, requires_grad=True)
        C = E.commutator(_t(x[0]), hL, Y, hR, case["with_e0"])
        return torch.autograd.grad(C, Y, _t(x[1]))[0].numpy()
    r = E.commutator(_t(x[0]), hL, _t(x[1]), hR, case["with_e0"]).numpy()
    return r[E.sp.packed_index()] if op == "host_packed" else r
