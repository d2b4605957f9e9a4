"""The work that the performance of this framework is judged by: its public calls over the sizes they are used at.

A case is one call of the Python interface (imsrg_gb300) on a basis, a precision and seeded operators:

  commutator  Engine.commutator, [Omega, H] (or [Omega, eta], herm_r = -1): the call that every flow is made of
  step        Engine.magnus_step, one Magnus step of the flow replayed as a CUDA graph
  bch         Engine.bch_expand, H(s) = exp(Omega) H exp(-Omega) on device-resident operators
  vjp         Engine.commutator_vjp, the backward pass of the adjoint dE0/dtheta
  observable  Engine.bch_tensor, the BCH transformation of a rank-2 tensor observable, from and to host arrays
  eom         LadderSpace.matvec, one product of the EOM-IMSRG Lanczos iteration, from and to host vectors
  hf          Engine.calc_hf, Hartree-Fock and normal ordering of a bare Hamiltonian

Inputs are made here from the seed alone with torch: operators of the library's slab layout whose elements fall off
with the shell energies of their orbits, as interaction matrix elements do, with a shell gap in the one-body part.
exact() restates what the calls compute in 64 bits with torch, from the J-coupled formulas in their textbook form.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "eom-imsrg_gb300"))

DEV = "cuda" if torch.cuda.is_available() else "cpu"

# ---------------------------------------------------------------------------------------------------- the cases


def listed():
    def c(name, kind, emax, prec="fp64", A=16, **more):
        return {"name": name, "kind": kind, "emax": emax, "lmax": emax, "A": A, "prec": prec, **more}

    return [
        # the smallest call: 12 orbits, 4He, where launches and latency are all there is
        c("commutator_fp64_e2", "commutator", 2, A=4),
        # a middling basis in the default precision (development runs, the adjoint's size)
        c("commutator_fp64_e6", "commutator", 6),
        # the plain FP64 commutator at the benchmark's size, the comparator of every mixed run
        c("commutator_fp64_e10", "commutator", 10),
        # an odd basis in the headline mode, [Omega, eta] as MAGNUS_EXPAND calls it
        c("commutator_bf16x3_e7", "commutator", 7, "bf16x3", herm_r=-1),
        # the three-slice mode at the precision study's size
        c("commutator_bf16x6_e8", "commutator", 8, "bf16x6"),
        # the headline: 132 orbits in bf16x3
        c("commutator_bf16x3_e10", "commutator", 10, "bf16x3"),
        # the FP64 flow of the validation runs, a step at a time
        c("step_fp64_e4", "step", 4),
        # the transformation of H at the end of a mixed flow
        c("bch_tf32x3_e8", "bch", 8, "tf32x3"),
        # the reverse sweep of the adjoint
        c("vjp_fp64_e6", "vjp", 6),
        # a quadrupole-like observable after the flow
        c("observable_fp64_e4", "observable", 4, rank=4),
        # excited states: a 2+ product
        c("eom_fp64_e6", "eom", 6, rank=4, dpar=0),
        # the start of every calculation
        c("hf_e8", "hf", 8),
    ]


def draw(rng):
    kind = rng.choice(["commutator"] * 6 + ["step", "bch", "vjp", "observable", "eom", "hf"])
    top = {"commutator": 10, "step": 6, "bch": 8, "vjp": 7, "observable": 4, "eom": 6, "hf": 9}[kind]
    prec = rng.choice(["fp64", "fp64", "bf16x3", "bf16x3", "bf16x6", "tf32x3"])
    c = {"kind": kind, "emax": rng.randint(3, top), "A": rng.choice([4, 16, 16])}
    c["lmax"] = max(2, c["emax"] - rng.choice([0, 0, 1, 2]))  # bases cut in l are as common as full ones
    c["prec"] = "fp64" if kind in ("vjp", "hf") else prec
    if kind == "bch" and prec == "fp64":
        c["emax"] = min(c["emax"], 7)
    if kind == "commutator":
        c["herm_r"] = rng.choice([1, 1, -1])
    if kind in ("observable", "eom"):
        c["rank"] = rng.choice([0, 2, 4, 4])
    if kind == "eom":
        c["dpar"] = rng.choice([0, 2])
    return c


def work(case):
    """The least that a pass moves and computes: operators read and written once, the channel products once.  A series
    counts the nested commutators that it takes at least (three of BCH, three of MAGNUS_EXPAND)."""
    s = space(case)
    slab = 8.0 * s.slab
    kind = case["kind"]
    if kind == "commutator":
        return {"bytes": 3 * slab, "flops": s.product_flops()}
    if kind == "step":
        return {"bytes": 6 * slab, "flops": 6 * s.product_flops()}
    if kind == "bch":
        return {"bytes": 3 * slab, "flops": 3 * s.product_flops()}
    if kind == "vjp":  # two products for each product of the forward pass
        return {"bytes": 5 * slab, "flops": 2 * s.product_flops()}
    if kind == "observable":
        t = TensorSpace(s, case["rank"], 0)
        return {"bytes": 8.0 * 2 * t.slab + slab, "flops": 3 * t.ladder_flops()}
    if kind == "eom":
        t = TensorSpace(s, case["rank"], case["dpar"])
        return {"bytes": slab + 16.0 * t.n_pphh(), "flops": t.excitation_flops()}
    return {"bytes": 2 * slab, "flops": 4.0 * s.slab}


# ---------------------------------------------------------------------------------------------------- layout


def orbits(emax, lmax):
    """(n, l, 2j, 2tz, e) in the order of the reference's hk*.sps files."""
    return [((e - l) // 2, l, j, t, e) for e in range(emax + 1) for l in range(e % 2, min(e, lmax) + 1, 2)
            for j in (2 * l - 1, 2 * l + 1) if j > 0 for t in (-1, 1)]


CLASSES = [(0, 0), (0, 1), (0, 2), (1, 1), (2, 2), (1, 2)]  # (bra, ket) pair classes of gam(1..6): pp, ph, hh
T_CLASSES = [(0, 0), (0, 1), (0, 2), (1, 1), (2, 2), (1, 2), (2, 0), (1, 0), (2, 1)]  # of a tensor's nine arrays


class Space:
    """The operator slab [E0][fhh][fpp][fph][gam(1..6) of every channel (J, Tz, parity)], column-major."""

    def __init__(self, emax, lmax, A):
        o = np.array(orbits(emax, lmax))
        self.emax, self.N = emax, len(o)
        self.n, self.l, self.j, self.t, self.e = (o[:, k] for k in range(5))
        self.con = np.zeros(self.N, np.int64)
        self.con[: {4: 2, 16: 6}[A]] = 1
        self.holes, self.parts = np.flatnonzero(self.con), np.flatnonzero(self.con == 0)
        self.JM = int(self.j.max())
        nh, npar = len(self.holes), len(self.parts)
        self.o_hh = 1
        self.o_pp = self.o_hh + nh * nh
        self.o_ph = self.o_pp + npar * npar
        at = self.o_ph + npar * nh
        a, b = np.triu_indices(self.N)
        par, tz, cls = (self.l[a] + self.l[b]) % 2, (self.t[a] + self.t[b]) // 2, self.con[a] + self.con[b]
        lo, hi = abs(self.j[a] - self.j[b]), self.j[a] + self.j[b]
        self.chan = []  # (J2, tz, parity, [pairs of a class as (a, b) arrays], [offset, n1, n2 of an array])
        for J in range(0, 2 * self.JM + 1, 2):
            for t in (-1, 0, 1):
                for p in (0, 1):
                    ok = (tz == t) & (par == p) & (lo <= J) & (J <= hi)
                    pairs = [(a[ok & (cls == c)], b[ok & (cls == c)]) for c in range(3)]
                    arrays = []
                    for c1, c2 in CLASSES:
                        n1, n2 = len(pairs[c1][0]), len(pairs[c2][0])
                        arrays.append((at, n1, n2))
                        at += n1 * n2
                    self.chan.append((J, t, p, pairs, arrays))
        self.slab = at

    def block(self, a, b):
        return (self.l[a] == self.l[b]) & (self.j[a] == self.j[b]) & (self.t[a] == self.t[b])

    def weights(self, q, c):
        """The fall-off of an element with its pair's shell energies; zero for a Pauli-forbidden pair."""
        J, (a, b) = self.chan[q][0], self.chan[q][3][c]
        return torch.from_numpy(np.where((a == b) & (J // 2 % 2 == 1), 0.0, np.exp(-(self.e[a] + self.e[b]) / self.emax))).to(DEV)

    def product_flops(self):
        """2MNK of the ladder products and of one cross-coupled product for each (J, |Tz|, parity)."""
        f = 0.0
        for J, t, p, pairs, _ in self.chan:
            n = [len(x[0]) for x in pairs]
            f += 2.0 * n[0] * (n[0] ** 2 + n[2] ** 2 + 2 * n[0] * n[2] + n[1] ** 2 + 2 * n[0] * n[1] + 2 * n[1] * n[2])
        i, k = (x.ravel() for x in np.indices((self.N, self.N)))
        for J in range(0, 2 * self.JM + 1, 2):
            tri = (abs(self.j[i] - self.j[k]) <= J) & (J <= self.j[i] + self.j[k])
            for t in (0, 2):
                for p in (0, 1):
                    ok = tri & (abs(self.t[i] - self.t[k]) == t) & ((self.l[i] + self.l[k]) % 2 == p)
                    f += 2.0 * ok.sum() ** 2 * (ok & (self.con[i] == 0) & (self.con[k] == 1)).sum()
        return f


class TensorSpace:
    """The tensor slab [E0][fhh][fpp][fph][the nine arrays of every block (J1 <= J2, Tz, bra parity)]."""

    def __init__(self, s, rank, dpar):
        self.s, self.rank, self.dpar = s, rank, dpar
        at = s.chan[0][4][0][0]
        self.arrays = []  # (offset, bra channel, ket channel, bra class, ket class, n1, n2)
        for J1 in range(0, 2 * s.JM + 1, 2):
            for J2 in range(max(abs(J1 - rank), J1), J1 + rank + 1, 2):
                for t in (-1, 0, 1):
                    for p in (0, 1):
                        if J2 > 2 * s.JM:
                            continue
                        q1 = J1 // 2 * 6 + (t + 1) * 2 + p
                        q2 = J2 // 2 * 6 + (t + 1) * 2 + (p ^ (dpar // 2))
                        for c1, c2 in T_CLASSES:
                            n1, n2 = len(s.chan[q1][3][c1][0]), len(s.chan[q2][3][c2][0])
                            self.arrays.append((at, q1, q2, c1, c2, n1, n2))
                            at += n1 * n2
        self.slab = at

    def n_pphh(self):
        return sum(n1 * n2 for _, _, _, c1, c2, n1, n2 in self.arrays if {c1, c2} == {0, 2})

    def excitation_flops(self):
        return 2.0 * sum(n1 * n2 * (n1 + n2) for _, _, _, c1, c2, n1, n2 in self.arrays if {c1, c2} == {0, 2})

    def ladder_flops(self):
        pp = [len(c[3][0][0]) for c in self.s.chan]
        return sum(2.0 * n1 * n2 * (pp[q1] + pp[q2]) for _, q1, q2, _, _, n1, n2 in self.arrays)


SPACES = {}


def space(case):
    key = (case["emax"], case["lmax"], case["A"])
    if key not in SPACES:
        SPACES[key] = Space(*key)
    return SPACES[key]


# ---------------------------------------------------------------------------------------------------- inputs


def generator(seed, salt):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 1000003 + salt)


def two_body(s, slab, herm, gen, scale):
    """Random two-body arrays: scale[g] times N(0, 1) times the fall-off, symmetric or antisymmetric where square."""
    slab[s.chan[0][4][0][0]:] = torch.randn(s.slab - s.chan[0][4][0][0], dtype=torch.float64, device=DEV, generator=gen)
    for q, (_, _, _, _, arrays) in enumerate(s.chan):
        w = [s.weights(q, c) for c in range(3)]
        for g, (o, n1, n2) in enumerate(arrays):
            if n1 * n2 == 0:
                continue
            m = slab[o:o + n1 * n2].view(n2, n1)
            m *= scale[g] * w[CLASSES[g][1]][:, None] * w[CLASSES[g][0]][None, :]
            if CLASSES[g][0] == CLASSES[g][1]:
                m.copy_((m + herm * m.T) / math.sqrt(2.0))


def one_body(s, slab, F):
    """The N x N one-body matrix F into fhh, fpp and fph."""
    h, p = torch.from_numpy(s.holes).to(DEV), torch.from_numpy(s.parts).to(DEV)
    slab[s.o_hh:s.o_pp] = F[h][:, h].T.reshape(-1)
    slab[s.o_pp:s.o_ph] = F[p][:, p].T.reshape(-1)
    slab[s.o_ph:s.chan[0][4][0][0]] = F[p][:, h].T.reshape(-1)


def random_f(s, herm, gen, scale):
    i, k = np.indices((s.N, s.N))
    w = torch.from_numpy(np.where(s.block(i, k), np.exp(-(s.e[i] + s.e[k]) / (2.0 * s.emax)), 0.0)).to(DEV)
    m = torch.randn(s.N, s.N, dtype=torch.float64, device=DEV, generator=gen) * w * scale
    return (m + herm * m.T) / math.sqrt(2.0)


def hamiltonian(s, seed):
    """A normal-ordered Hamiltonian (MeV): single-particle energies with a shell gap, matrix elements of about 1 MeV."""
    gen = generator(seed, 1)
    x = torch.zeros(s.slab, dtype=torch.float64, device=DEV)
    two_body(s, x, 1, gen, [1.0] * 6)
    F = random_f(s, 1, gen, 1.0) + torch.diag(torch.from_numpy(15.0 * s.e - 25.0).to(DEV))
    one_body(s, x, F)
    x[0] = -100.0 - float(torch.rand(1, dtype=torch.float64, device=DEV, generator=gen))
    return x


def antihermitian(s, seed, salt, size):
    """Omega or eta: mostly particle-hole and pp-hh amplitudes, with the smaller parts that a flow fills in elsewhere."""
    gen = generator(seed, salt)
    x = torch.zeros(s.slab, dtype=torch.float64, device=DEV)
    two_body(s, x, -1, gen, [0.1 * size, 0.1 * size, size, 0.1 * size, 0.1 * size, 0.1 * size])
    F = random_f(s, -1, gen, 0.1 * size)
    one_body(s, x, F)
    return x


def bare(s, seed):
    """Kinetic energy in the oscillator basis (hw = 20 MeV) and a two-body interaction, not normal ordered."""
    gen = generator(seed, 5)
    x = torch.zeros(s.slab, dtype=torch.float64, device=DEV)
    two_body(s, x, 1, gen, [0.5] * 6)
    F = np.zeros((s.N, s.N))
    for a in range(s.N):
        F[a, a] = 10.0 * (s.e[a] + 1.5)
        for b in range(a):
            if s.block(a, b) and abs(s.n[a] - s.n[b]) == 1:
                m = max(s.n[a], s.n[b])
                F[a, b] = F[b, a] = 10.0 * math.sqrt(m * (m + s.l[a] + 0.5))
    one_body(s, x, torch.from_numpy(F).to(DEV))
    return x


def tensor(t, seed):
    """A hermitian tensor operator of rank t.rank: one- and two-body parts."""
    s, gen = t.s, generator(seed, 6)
    x = torch.zeros(t.slab, dtype=torch.float64, device=DEV)
    i, k = np.indices((s.N, s.N))
    ok = (abs(s.j[i] - s.j[k]) <= t.rank) & (t.rank <= s.j[i] + s.j[k]) & (s.t[i] == s.t[k]) & ((s.l[i] + s.l[k] + t.dpar // 2) % 2 == 0)
    m = torch.randn(s.N, s.N, dtype=torch.float64, device=DEV, generator=gen) * torch.from_numpy(ok * np.exp(-(s.e[i] + s.e[k]) / (2.0 * s.emax))).to(DEV)
    sign = torch.from_numpy(1.0 - (abs(s.j[i] - s.j[k]) // 2 % 2) * 2).to(DEV)
    one_body(s, x, torch.triu(m) + (sign * torch.triu(m, 1).T.contiguous()))
    for o, q1, q2, c1, c2, n1, n2 in t.arrays:
        if n1 * n2 == 0:
            continue
        m = torch.randn(n2, n1, dtype=torch.float64, device=DEV, generator=gen) * 0.1 * s.weights(q2, c2)[:, None] * s.weights(q1, c1)[None, :]
        if q1 == q2 and c1 == c2:
            m = (m + m.T) / math.sqrt(2.0)
        x[o:o + n1 * n2] = m.reshape(-1)
    lead = {a[1:5]: a for a in t.arrays}
    for o, q1, q2, c1, c2, n1, n2 in t.arrays:  # J1 == J2: the arrays below the diagonal mirror those above it
        if q1 == q2 and c1 > c2 and n1 * n2:
            src = lead[(q1, q2, c2, c1)]
            x[o:o + n1 * n2] = x[src[0]:src[0] + n1 * n2].view(n1, n2).T.reshape(-1)
    return x


# ---------------------------------------------------------------------------------------------------- the calls


class DeviceSlab:
    """An operator's device array as torch sees it; a tensor made of it keeps the operator and its engine alive."""

    def __init__(self, op):
        self.op = op
        self.__cuda_array_interface__ = {"shape": (op.eng.slab,), "typestr": "<f8", "data": (op.device_ptr(), False), "version": 3}


ENGINES = {}


def engine(case, own=False):
    """The program's engine for a basis and a precision; `own`: one that this state alone has (its captured step)."""
    from imsrg_gb300 import Engine, make_basis
    key = (case["emax"], case["lmax"], case["A"], case["prec"])
    if own or key not in ENGINES:
        Z = case["A"] // 2
        e = Engine(make_basis(case["emax"], Z, Z, lmax=case["lmax"]), device=0, precision=case["prec"])
        if own:
            return e
        ENGINES.clear()  # a state keeps its own engine alive
        ENGINES[key] = e
    return ENGINES[key]


def operator(eng, herm, slab=None):
    """An operator and its device slab as a tensor, filled with `slab`."""
    op = eng.new_op(herm)
    view = torch.as_tensor(DeviceSlab(op), device="cuda")
    if slab is not None:
        eng.synchronize()
        view.copy_(slab)
        torch.cuda.synchronize()
    return op, view


def inputs(case, seed):
    """The operators of a case as slabs on the device (exact() takes the same ones)."""
    s, kind = space(case), case["kind"]
    if kind == "commutator":
        return {"L": antihermitian(s, seed, 2, 0.05), "R": hamiltonian(s, seed) if case.get("herm_r", 1) == 1 else antihermitian(s, seed, 3, 0.3)}
    if kind == "step":
        return {"H": hamiltonian(s, seed), "G": antihermitian(s, seed, 2, 0.01), "DG": antihermitian(s, seed, 3, 0.02)}
    if kind == "bch":
        return {"H": hamiltonian(s, seed), "G": antihermitian(s, seed, 2, 0.01)}
    if kind == "vjp":
        return {"L": antihermitian(s, seed, 2, 0.05), "R": hamiltonian(s, seed), "C": hamiltonian(s, seed + 500009)}
    if kind == "observable":
        return {"G": antihermitian(s, seed, 2, 0.01), "X": tensor(TensorSpace(s, case["rank"], 0), seed).cpu().numpy()}
    if kind == "eom":
        return {"H": hamiltonian(s, seed)}
    return {"H": bare(s, seed)}


def prepare(case, seed):
    kind, x = case["kind"], inputs(case, seed)
    eng = engine(case, own=kind == "step")
    st = {"kind": kind, "eng": eng}
    if kind == "commutator":
        h = case.get("herm_r", 1)
        st["L"], st["R"] = operator(eng, -1, x["L"])[0], operator(eng, h, x["R"])[0]
        st["RES"], st["out"] = operator(eng, h)
    elif kind == "step":
        st["H"], st["G0"], st["DG0"] = operator(eng, 1, x["H"])[0], operator(eng, -1, x["G"])[0], operator(eng, -1, x["DG"])[0]
        (st["HS"], a), (st["G"], b), (st["DG"], c) = operator(eng, 1), operator(eng, -1), operator(eng, -1)
        st["out"] = [a, b, c]
    elif kind == "bch":
        st["H"], st["G"] = operator(eng, 1, x["H"])[0], operator(eng, -1, x["G"])[0]
        st["HS"], st["out"] = operator(eng, 1)
    elif kind == "vjp":
        st["L"], st["R"], st["C"] = operator(eng, -1, x["L"])[0], operator(eng, 1, x["R"])[0], operator(eng, 1, x["C"])[0]
        (st["Lb"], a), (st["Rb"], b) = operator(eng, -1), operator(eng, 1)
        st["out"] = [a, b]
    elif kind == "observable":
        st["G"], st["X"] = operator(eng, -1, x["G"])[0], x["X"]
        st["Q"] = eng.new_tensor(case["rank"], 0, 1)
    elif kind == "eom":
        from imsrg_gb300.eom import LadderSpace
        st["H"] = operator(eng, 1, x["H"])[0]
        st["space"] = LadderSpace(eng, case["rank"], case["dpar"])
        st["v"] = np.random.default_rng(seed).standard_normal(st["space"].n)
    else:
        st["bare"] = operator(eng, 1, x["H"])[0]
        st["H"], st["out"] = operator(eng, 1)
    return st


def run(st):
    kind, eng = st["kind"], st["eng"]
    if kind == "commutator":
        eng.commutator(st["L"], st["R"], st["RES"])
        return st["out"]
    if kind == "step":  # from the flow's state in hand
        eng.copy_sq_op(st["G0"], st["G"])
        eng.copy_sq_op(st["DG0"], st["DG"])
        r = eng.magnus_step(st["HS"], st["G"], st["DG"], st["H"], 0.5, max_terms=10, conv=1e-8, allow_unconverged=True)
        return {"slabs": st["out"], "E0": r["E0"], "mbpt2": r["mbpt2"], "terms": [r["magnus_terms"], r["bch_terms"]]}
    if kind == "bch":
        n = eng.bch_expand(st["HS"], st["G"], st["H"])
        return {"HS": st["out"], "terms": n}
    if kind == "vjp":  # the cotangents accumulate: cleared first, as at the start of a reverse sweep
        eng.clear_sq_op(st["Lb"])
        eng.clear_sq_op(st["Rb"])
        eng.commutator_vjp(st["L"], st["R"], st["C"], st["Lb"], st["Rb"])
        return st["out"]
    if kind == "observable":
        st["Q"].upload(st["X"])
        n = eng.bch_tensor(st["G"], st["Q"])
        return {"Q": st["Q"].download(), "terms": n}
    if kind == "eom":
        return st["space"].matvec(st["H"], st["v"])
    eng.copy_sq_op(st["bare"], st["H"])
    D, info = eng.calc_hf(st["H"])
    return {"H": st["out"], "D": D, "e_hf": info["e_hf"], "iterations": info["iterations"]}


# ---------------------------------------------------------------------------------------------------- 64-bit values


def exact(case, seed):
    """The commutator, the series made of it and Hartree-Fock.  The transposes, tensors and ladder operators have no
    short independent form: None."""
    kind = case["kind"]
    if kind in ("vjp", "observable", "eom"):
        return None
    x, m = inputs(case, seed), Reference(space(case))
    if kind == "commutator":
        h = case.get("herm_r", 1)
        return m.to_slab(m.commutator(m.from_slab(x["L"], -1), m.from_slab(x["R"], h)))
    if kind == "hf":
        return m.hartree_fock(x["H"])
    H, G = m.from_slab(x["H"], 1), m.from_slab(x["G"], -1)
    if kind == "bch":
        HS, n = m.bch(G, H, 40, float(np.float32(1e-6)))
        return {"HS": m.to_slab(HS), "terms": n}
    G, k = m.magnus(G, m.from_slab(x["DG"], -1), 0.5)
    HS, n = m.bch(G[0], H, 10, 1e-8)
    eta = m.white(HS)
    return {"slabs": [m.to_slab(HS), m.to_slab(G[0]), m.to_slab(eta)], "E0": float(HS["E0"]), "mbpt2": m.mbpt2(HS), "terms": [k, n]}


def six_j_table(JM, dev):
    """{j1 j2 J; j4 j5 K} (Racah's formula) for half-integer j <= JM / 2 and all J, K, as [j1, j2, J, j4, j5, K]."""
    nh, nJ = (JM + 1) // 2, JM + 1
    lf = torch.cat([torch.zeros(1, dtype=torch.float64), torch.log(torch.arange(1, 400, dtype=torch.float64)).cumsum(0)]).to(dev)
    h, J = 2 * torch.arange(nh, device=dev) + 1, 2 * torch.arange(nJ, device=dev)
    j1, j2, j3, j4, j5, j6 = torch.meshgrid(h, h, J, h, h, J, indexing="ij")

    def f(x):
        return lf[x.clamp(min=0)]

    ok, d = torch.ones_like(j1, dtype=torch.bool), 0.0
    for a, b, c in ((j1, j2, j3), (j1, j5, j6), (j4, j2, j6), (j4, j5, j3)):
        ok &= ((a - b).abs() <= c) & (c <= a + b)
        d = d + 0.5 * (f((a + b - c) // 2) + f((a - b + c) // 2) + f((b + c - a) // 2) - f((a + b + c) // 2 + 1))
    low = [(j1 + j2 + j3) // 2, (j1 + j5 + j6) // 2, (j4 + j2 + j6) // 2, (j4 + j5 + j3) // 2]
    high = [(j1 + j2 + j4 + j5) // 2, (j2 + j3 + j5 + j6) // 2, (j3 + j1 + j6 + j4) // 2]
    z0 = torch.maximum(torch.maximum(low[0], low[1]), torch.maximum(low[2], low[3]))
    z1 = torch.minimum(torch.minimum(high[0], high[1]), high[2])
    out = torch.zeros_like(d)
    for k in range(JM + 2):
        z = z0 + k
        term = f(z + 1) + d
        for x in low:
            term = term - f(z - x)
        for x in high:
            term = term - f(x - z)
        out += torch.where(ok & (z <= z1), (1.0 - 2.0 * (z % 2)) * torch.exp(term), 0.0)
    return out


class Reference:
    """IMSRG(2) in 64 bits on full channel matrices over the normalised pairs a <= b (class order pp, ph, hh) and an
    N x N one-body matrix: {"E0", "f", "v": [a matrix of every channel], "h": +1 or -1}."""

    def __init__(self, s):
        self.s = s

        def dev(x):
            return torch.from_numpy(np.ascontiguousarray(x)).to(DEV)

        self.j, self.l, self.t, self.con = dev(s.j), dev(s.l), dev(s.t), dev(s.con)
        N, nJ = s.N, s.JM + 1
        self.pos = np.full((N, N, nJ), -1, np.int64)
        self.size = [sum(len(x[0]) for x in c[3]) for c in s.chan]
        self.start = np.concatenate([[0], np.cumsum([n * n for n in self.size])])
        self.a, self.b = [], []
        for q, c in enumerate(s.chan):
            a, b = np.concatenate([x[0] for x in c[3]]), np.concatenate([x[1] for x in c[3]])
            self.pos[a, b, c[0] // 2] = np.arange(len(a))
            self.a.append(dev(a))
            self.b.append(dev(b))
        self.pos = dev(self.pos)
        self.d_start, self.d_size = dev(self.start), dev(np.array(self.size))
        self.six = six_j_table(s.JM, DEV)
        i, k = np.indices((N, N))
        self.same = dev(s.block(i, k))
        self.twice = self.j.double() + 1.0  # 2j + 1

    # ---- storage
    def from_slab(self, x, h):
        s = self.s
        hh, pp, ph = x[s.o_hh:s.o_pp], x[s.o_pp:s.o_ph], x[s.o_ph:s.chan[0][4][0][0]]
        A, P = len(s.holes), len(s.parts)
        H, Q = torch.from_numpy(s.holes).to(DEV), torch.from_numpy(s.parts).to(DEV)
        f = torch.zeros(s.N, s.N, dtype=torch.float64, device=DEV)
        f[H[:, None], H[None]] = hh.view(A, A).T
        f[Q[:, None], Q[None]] = pp.view(P, P).T
        f[Q[:, None], H[None]] = ph.view(A, P).T
        f[H[:, None], Q[None]] = h * ph.view(A, P)
        v = []
        for _, _, _, pairs, arrays in s.chan:
            at = np.concatenate([[0], np.cumsum([len(p[0]) for p in pairs])])
            m = torch.zeros(at[3], at[3], dtype=torch.float64, device=DEV)
            for (c1, c2), (o, n1, n2) in zip(CLASSES, arrays):
                blk = x[o:o + n1 * n2].view(n2, n1).T
                m[at[c1]:at[c1 + 1], at[c2]:at[c2 + 1]] = blk
                if c1 != c2:
                    m[at[c2]:at[c2 + 1], at[c1]:at[c1 + 1]] = h * blk.T
            v.append(m)
        return {"E0": float(x[0]), "f": f, "v": v, "h": h}

    def to_slab(self, op):
        s = self.s
        x = torch.zeros(s.slab, dtype=torch.float64, device=DEV)
        x[0] = op["E0"]
        one_body(s, x, op["f"])
        for m, (_, _, _, pairs, arrays) in zip(op["v"], s.chan):
            at = np.concatenate([[0], np.cumsum([len(p[0]) for p in pairs])])
            for (c1, c2), (o, n1, n2) in zip(CLASSES, arrays):
                x[o:o + n1 * n2] = m[at[c1]:at[c1 + 1], at[c2]:at[c2 + 1]].T.reshape(-1)
        return x

    def element(self, flat, a, b, c, d, J):
        """<ab; J| V |cd; J> of unnormalised pairs in any order, zero where a pair cannot couple to J."""
        j, t, l = self.j, self.t, self.l
        ok = ((j[a] - j[b]).abs() <= J) & (J <= j[a] + j[b]) & ((j[c] - j[d]).abs() <= J) & (J <= j[c] + j[d])
        ok = ok & (t[a] + t[b] == t[c] + t[d]) & ((l[a] + l[b] + l[c] + l[d]) % 2 == 0)
        lo1, hi1, lo2, hi2 = torch.minimum(a, b), torch.maximum(a, b), torch.minimum(c, d), torch.maximum(c, d)
        p1, p2 = self.pos[lo1, hi1, J // 2], self.pos[lo2, hi2, J // 2]
        q = (J // 2) * 6 + (t[a] + t[b] + 2) + (l[a] + l[b]) % 2
        v = flat[torch.where(ok, self.d_start[q] + p1 * self.d_size[q] + p2, 0)]
        s1 = torch.where(a > b, 1.0 - 2.0 * ((1 + (j[a] + j[b] - J) // 2) % 2), 1.0)
        s2 = torch.where(c > d, 1.0 - 2.0 * ((1 + (j[c] + j[d] - J) // 2) % 2), 1.0)
        root = torch.sqrt((1.0 + (a == b).double()) * (1.0 + (c == d).double()))
        return torch.where(ok, v * s1 * s2 * root, 0.0)

    def lifted(self, M, q, product):
        """A one-body matrix on the normalised pairs of a channel: M (x) 1 + 1 (x) M, or M (x) M with `product`."""
        a, b, J = self.a[q], self.b[q], self.s.chan[q][0]
        sign = (1.0 - 2.0 * ((1 + (self.j[a] + self.j[b] - J) // 2) % 2))[:, None]
        A, B, C, D = a[:, None], b[:, None], a[None], b[None]
        if product:
            x = M[A, C] * M[B, D] + sign * M[B, C] * M[A, D]
        else:
            x = M[A, C] * (B == D) + M[B, D] * (A == C) + sign * (M[B, C] * (A == D) + M[A, D] * (B == C))
        return x / torch.sqrt((1.0 + (A == B).double()) * (1.0 + (C == D).double()))

    def summed(self, v, p, q, x, y):
        """sum_J (2J+1) <x p; J| V |y q; J> of a flat operator."""
        tot = 0.0
        for J in range(0, 2 * self.s.JM + 1, 2):
            tot = tot + (J + 1.0) * self.element(v, x, p, y, q, J)
        return tot

    # ---- the commutator
    def commutator(self, L, R, e0=True):
        s, con = self.s, self.con
        fL, fR, n = L["f"], R["f"], con.double()
        E0 = 0.0
        if e0:
            E0 = float((((n[:, None] * (1 - n)[None]) * (fL * fR.T - fR * fL.T)) * self.twice[:, None]).sum())
        f = fL @ fR - fR @ fL
        v, w1, w2 = [], [], []
        for q, c in enumerate(s.chan):
            A, B = L["v"][q], R["v"][q]
            k = con[self.a[q]] + con[self.b[q]]
            pp, hh = (k == 0).double(), (k == 2).double()
            ladder_p = (A * pp) @ B - (B * pp) @ A
            ladder_h = (A * hh) @ B - (B * hh) @ A
            FL, FR = self.lifted(fL, q, False), self.lifted(fR, q, False)
            v.append(ladder_p - ladder_h + FL @ B - B @ FL - FR @ A + A @ FR)
            w1.append(ladder_p.reshape(-1))
            w2.append(ladder_h.reshape(-1))
            if e0:
                E0 += (c[0] + 1.0) * float(((A * pp) @ B - (B * pp) @ A).diagonal() @ hh)
        flat_l, flat_r = torch.cat([m.reshape(-1) for m in L["v"]]), torch.cat([m.reshape(-1) for m in R["v"]])
        w1, w2 = torch.cat(w1), torch.cat(w2)
        # one-body parts: pairs (p, q) of one (l, j, tz) block
        P, Q = self.same.nonzero(as_tuple=True)
        X, Y = (self.same & (con[:, None] == 0) & (con[None] == 1)).nonzero(as_tuple=True)  # (particle, hole)
        if len(X):
            p, q, x, y = P[:, None], Q[:, None], X[None], Y[None]
            r1, r2 = self.summed(flat_r, p, q, x, y), self.summed(flat_r, p, q, y, x)
            l1, l2 = self.summed(flat_l, p, q, x, y), self.summed(flat_l, p, q, y, x)
            f[P, Q] += (fL[Y, X] * r1 - fL[X, Y] * r2 - fR[Y, X] * l1 + fR[X, Y] * l2).sum(1) / self.twice[P]
        c = torch.arange(s.N, device=DEV)[None]
        from_p, from_h = self.summed(w1, P[:, None], Q[:, None], c, c), self.summed(w2, P[:, None], Q[:, None], c, c)
        f[P, Q] += (n * from_p + (1 - n) * from_h).sum(1) / self.twice[P]
        for m, x in zip(v, self.particle_hole(flat_l, flat_r)):
            m += x
        return {"E0": E0, "f": f, "v": v, "h": -L["h"] * R["h"]}

    def particle_hole(self, L, R):
        """The particle-hole part of the two-body commutator: Pandya transforms, products through the pairs with one
        orbit occupied, and the transformation back."""
        s, j, six = self.s, self.j, self.six
        N, nJ = s.N, s.JM + 1
        i, k = (torch.from_numpy(x.ravel()).to(DEV) for x in np.indices((N, N)))
        row, start, size, Z, at = torch.full((N, N, nJ), -1, device=DEV), np.zeros((nJ, 3, 2), np.int64), np.zeros((nJ, 3, 2), np.int64), [], 0
        for K in range(0, 2 * s.JM + 1, 2):
            tri = ((j[i] - j[k]).abs() <= K) & (K <= j[i] + j[k])
            for t in (-1, 0, 1):
                for p in (0, 1):
                    ok = tri & (self.t[i] - self.t[k] == 2 * t) & ((self.l[i] + self.l[k]) % 2 == p)
                    I, B = i[ok], k[ok]
                    row[I, B, K // 2] = torch.arange(len(I), device=DEV)
                    mixed = self.con[I] != self.con[B]
                    start[K // 2, t + 1, p], size[K // 2, t + 1, p] = at, len(I)
                    at += len(I) ** 2
                    C, D = I[mixed], B[mixed]

                    def bar(v, a, b, c, d):  # <a b-bar| v |c d-bar> = - sum_J (2J+1) {ja jb K; jc jd J} v(a d, c b; J)
                        tot = 0.0
                        for J in range(0, 2 * s.JM + 1, 2):
                            tot = tot - (J + 1.0) * six[j[a] // 2, j[b] // 2, K // 2, j[c] // 2, j[d] // 2, J // 2] * self.element(v, a, d, c, b, J)
                        return tot

                    if len(C) == 0:
                        Z.append(torch.zeros(len(I) ** 2, dtype=torch.float64, device=DEV))
                        continue
                    left = bar(L, I[:, None], B[:, None], C[None], D[None])
                    right = bar(R, C[:, None], D[:, None], I[None], B[None])
                    Z.append(((left * (self.con[C] - self.con[D]).double()) @ right).reshape(-1))
        Z = torch.cat(Z)
        start, size = torch.from_numpy(start).to(DEV), torch.from_numpy(size).to(DEV)

        def back(a, b, c, d, J):  # sum_K (2K+1) {ja jb J; jc jd K} Z^K(a d-bar, c b-bar)
            tot, t, p = 0.0, (self.t[a] - self.t[d]) // 2 + 1, (self.l[a] + self.l[d]) % 2
            for K in range(nJ):
                x, y = row[a, d, K], row[c, b, K]
                ok = (x >= 0) & (y >= 0)
                z = Z[torch.where(ok, start[K, t, p] + x * size[K, t, p] + y, 0)]
                tot = tot + torch.where(ok, (2 * K + 1.0) * six[j[a] // 2, j[b] // 2, J // 2, j[c] // 2, j[d] // 2, K] * z, 0.0)
            return tot

        out = []
        for q, c in enumerate(s.chan):
            J = c[0]
            a, b = self.a[q][:, None], self.b[q][:, None]
            x, y = self.a[q][None], self.b[q][None]
            s1, s2 = 1.0 - 2.0 * (((j[a] + j[b] - J) // 2) % 2), 1.0 - 2.0 * (((j[x] + j[y] - J) // 2) % 2)
            if a.numel() == 0:
                out.append(torch.zeros(0, 0, dtype=torch.float64, device=DEV))
                continue
            m = back(a, b, x, y, J) - s1 * back(b, a, x, y, J) - s2 * back(a, b, y, x, J) + s1 * s2 * back(b, a, y, x, J)
            out.append(m / torch.sqrt((1.0 + (a == b).double()) * (1.0 + (x == y).double())))
        return out

    # ---- series and generator
    def combine(self, A, x, B, with_e0=True):
        return {"E0": A["E0"] + (x * B["E0"] if with_e0 else 0.0), "f": A["f"] + x * B["f"], "v": [p + x * q for p, q in zip(A["v"], B["v"])], "h": A["h"]}

    def norm(self, A):
        return math.sqrt(float((A["f"] ** 2).sum()) + sum(float((m ** 2).sum()) for m in A["v"]))

    def bch(self, G, H, max_terms, conv):
        HS, ad, coef = H, H, 1.0
        for k in range(2, max_terms + 1):
            coef /= k - 1.0
            ad = self.commutator(G, ad)
            HS = self.combine(HS, coef, ad)
            if coef * self.norm(ad) < conv:
                return HS, k - 1
        return HS, max_terms - 1

    def magnus(self, G, DG, ds):
        """Omega after a step: MAGNUS_EXPAND with the reference's coefficients and tests, then the Euler step."""
        cof, conv = [1.0, -0.5, .0833333333, 0.0, -0.00138888888, 0.0, 3.306878e-5], float(np.float32(1e-6))
        norms, full, out, ad, qq, used = {1: self.norm(DG)}, self.norm(G), DG, DG, 1, 0
        for k in range(2, 8):
            last = norms[k - qq]
            qq = 1 if abs(cof[k - 1]) > conv else 2
            if abs(last / full) < conv:
                break
            ad = self.commutator(G, ad, False)
            used += 1
            out = self.combine(out, cof[k - 1], ad, False)
            norms[k] = self.norm(ad) * abs(cof[k - 1])
        return (self.combine(G, ds, out),), used

    def monopoles(self, H):
        flat = torch.cat([m.reshape(-1) for m in H["v"]])
        a, b = (torch.from_numpy(x).to(DEV) for x in np.indices((self.s.N, self.s.N)))
        return self.summed(flat, b, b, a, a) / (self.twice[:, None] * self.twice[None]), flat

    def white(self, H):
        """The White generator with Epstein-Nesbet denominators."""
        s, con, e = self.s, self.con, H["f"].diagonal()
        mono, flat = self.monopoles(H)
        f = torch.zeros_like(H["f"])
        X, Y = (self.same & (con[:, None] == 0) & (con[None] == 1)).nonzero(as_tuple=True)
        if len(X):
            d = sum((J + 1.0) * self.element(flat, X, Y, X, Y, J) for J in range(0, 2 * s.JM + 1, 2)) / self.twice[Y] ** 2
            f[X, Y] = H["f"][X, Y] / (e[X] - e[Y] - d)
            f[Y, X] = -f[X, Y]
        v = []
        for q, m in enumerate(H["v"]):
            a, b = self.a[q][:, None], self.b[q][:, None]
            i, k = self.a[q][None], self.b[q][None]
            ok = (con[a] + con[b] == 0) & (con[i] + con[k] == 2)
            d = mono[a, b] + mono[i, k] - mono[a, i] - mono[a, k] - mono[i, b] - mono[k, b] + e[a] + e[b] - e[i] - e[k]
            x = torch.where(ok, m / torch.where(ok, d, 1.0), 0.0)
            v.append(x - x.T)
        return {"E0": 0.0, "f": f, "v": v, "h": -1}

    def mbpt2(self, H):
        tot, e, con = 0.0, H["f"].diagonal(), self.con
        for q, m in enumerate(H["v"]):
            a, b = self.a[q][:, None], self.b[q][:, None]
            i, k = self.a[q][None], self.b[q][None]
            ok = (con[a] + con[b] == 0) & (con[i] + con[k] == 2)
            d = e[i] + e[k] - e[a] - e[b]
            tot += (self.s.chan[q][0] + 1.0) * float(torch.where(ok, m * m / torch.where(ok, d, 1.0), 0.0).sum())
        return tot

    # ---- Hartree-Fock
    def hartree_fock(self, slab):
        s = self.s
        H = self.from_slab(slab, 1)
        T, flat = H["f"], torch.cat([m.reshape(-1) for m in H["v"]])
        P, Q = self.same.nonzero(as_tuple=True)
        full = torch.zeros(s.N, dtype=torch.bool, device=DEV)
        full[(self.same & (self.con[None] == 1)).any(1)] = True
        g, h = (self.same & full[:, None]).nonzero(as_tuple=True)
        M = self.summed(flat, g[None], h[None], P[:, None], Q[:, None])

        def field(rho):  # rho(h, g) of a block, one particle in each of its 2j+1 states
            G = torch.zeros_like(T)
            G[P, Q] = (M * rho[h, g][None]).sum(1) / self.twice[P]
            return G

        D, eig, crit, n = torch.eye(s.N, dtype=torch.float64, device=DEV), torch.zeros(s.N, dtype=torch.float64, device=DEV), 10.0, 0
        occ = self.con.double()
        while crit > float(np.float32(1e-6)):
            G = field((D * occ) @ D.T)
            F, crit, new = T + G, 0.0, torch.zeros_like(D)
            for o in range(s.N):
                blk = self.same[o].nonzero()[:, 0]
                if int(blk[0]) != o:
                    continue
                w, V = torch.linalg.eigh(F[blk][:, blk])
                new[blk[:, None], blk[None]] = V
                crit += float(((eig[blk] - w) ** 2).sum().sqrt())
                eig[blk] = w
            D, n = new, n + 1
        D = torch.where(D.diagonal() < 0, -D, D)
        f = D.T @ (T + G) @ D
        e_hf = float((((D.T @ T @ D).diagonal() + 0.5 * (D.T @ G @ D).diagonal()) * occ * self.twice).sum())
        v = []
        for q, m in enumerate(H["v"]):
            U = self.lifted(D, q, True)
            v.append(U.T @ m @ U)
        return {"H": self.to_slab({"E0": e_hf, "f": f, "v": v}), "D": D.cpu().numpy(), "e_hf": e_hf, "iterations": n}
