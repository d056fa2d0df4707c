"""What a program that uses this library has it do, as measurable cases.

A case is one call sequence on one model: impurity models with a few bath
sites, Hubbard rings and plaquettes, a two-orbital impurity.  The stages are
reached as a program reaches them, through pomerol_b200.pgx.Engine or, for the
`dropin` kind, the pomerol class API:

  pair    G and chi of a solved model on a frequency list
  g2      the two-particle function of a solved model on a cube of triples
  chi3    the three-point susceptibility of a solved model on a square
  solve   new coefficients of a model -> eigensystem, weights, G and chi, as
          in every turn of a self-consistency loop or a fit
  grad    the same with the gradient of a loss on G (forward and backward)
  batch   many independent impurity models in one context
  dropin  a whole program of the class API, from the expression to G and G2

The models are drawn around this repository's configurations (plaquette,
Anderson 1+5, the 64-model batch, Kanamori, Hubbard rings): the seed moves the
couplings, the case fixes the sizes.  `exact` restates every result in plain
torch with 64-bit numbers.
"""
import math

import numpy as np
import torch

from pomerol_b200 import _pomerol as P
from pomerol_b200 import pgx

POLE_RES = 1e-8


def listed():
    return [
        # the smallest call: a band of G and a few chi of a 4-site plaquette, launches and host work count
        dict(name="pair_plaquette", kind="pair", model="ring", sites=4, nz=256, nchi=16),
        # every quadruple summed (no weight threshold) on the plaquette's 8^3 cube
        dict(name="g2_exact_plaquette", kind="g2", model="ring", sites=4, nfreq=8, form="exact"),
        # a whole small program written against the class API
        dict(name="dropin_plaquette", kind="dropin", model="ring", sites=4, nz=256, nfreq=8),
        # one turn of an impurity solver's loop: blocks up to 400 states
        dict(name="solve_anderson5", kind="solve", model="anderson", sites=6, nz=1024, nchi=32),
        # the same with a complex Hermitian Hamiltonian (a ring with a flux), ragged sizes
        dict(name="solve_flux5", kind="solve", model="flux", sites=5, nz=333, nchi=17),
        # blocks up to 1225 states: the eigensolver's and rotation's large-block paths
        dict(name="solve_ring7", kind="solve", model="ring", sites=7, nz=256, nchi=48),
        # the two-particle function of an impurity, FP64
        dict(name="g2_anderson5", kind="g2", model="anderson", sites=6, nfreq=16, form="anchored"),
        # the same on larger blocks, FP64, with an odd cube
        dict(name="g2_ring7", kind="g2", model="ring", sites=7, nfreq=7, form="anchored"),
        # the 8-site ring's largest block chain (4900 states), split products: one piece of work of a full run
        dict(name="g2_ring8_chain", kind="g2", model="ring", sites=8, nfreq=16, form="split", chains=1),
        dict(name="chi3_anderson5", kind="chi3", model="anderson", sites=6, nfreq=32),
        # gradient of a 512-frequency loss with respect to every term of a two-orbital impurity
        dict(name="grad_kanamori", kind="grad", model="kanamori", sites=6, nz=512),
        # 64 impurity models of 3 to 6 bath sites at their own temperatures
        dict(name="batch_64", kind="batch", model="anderson", models=64, nz=1024, nchi=32),
    ]


def draw(rng):
    def log(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    kind = rng.choice(["pair", "pair", "g2", "g2", "g2", "solve", "solve", "chi3", "grad", "batch", "dropin"])
    if kind == "grad":
        return dict(kind=kind, model="kanamori", sites=6, nz=log(16, 600))
    if kind == "batch":
        return dict(kind=kind, model="anderson", models=log(2, 40), nz=log(32, 1200), nchi=log(1, 48))
    if kind == "dropin":
        return dict(kind=kind, model="ring", sites=rng.choice([2, 3, 4, 5]), nz=log(8, 512), nfreq=rng.randint(2, 9))
    if kind == "pair":
        m, s = rng.choice([("ring", 2), ("ring", 4), ("ring", 6), ("anderson", 4), ("anderson", 6), ("flux", 4)])
        return dict(kind=kind, model=m, sites=s, nz=log(1, 2000), nchi=log(1, 64))
    if kind == "solve":
        m, s = rng.choice([("ring", 4), ("ring", 6), ("ring", 7), ("anderson", 4), ("anderson", 5), ("anderson", 6),
                           ("anderson", 7), ("flux", 4), ("flux", 5)])
        return dict(kind=kind, model=m, sites=s, nz=log(16, 1500), nchi=log(1, 64))
    if kind == "chi3":
        return dict(kind=kind, model=rng.choice(["ring", "anderson"]), sites=rng.choice([3, 4, 5, 6]), nfreq=log(2, 40))
    m, s, top, form = rng.choice([("ring", 3, 12, "exact"), ("ring", 4, 9, "exact"), ("anderson", 4, 10, "exact"),
                                  ("ring", 5, 16, "anchored"), ("ring", 6, 14, "anchored"), ("ring", 7, 6, "anchored"),
                                  ("anderson", 4, 20, "anchored"), ("anderson", 5, 20, "anchored"),
                                  ("anderson", 6, 18, "anchored"), ("anderson", 7, 4, "anchored"),
                                  ("flux", 4, 8, "anchored"), ("ring", 7, 7, "split")])
    return dict(kind=kind, model=m, sites=s, nfreq=rng.randint(2, top), form=form)


# ---------------------------------------------------------------- models
class Model:
    """Couplings and Fock-space tables of one model: modes 0..n-1 are the
    up spins, n..2n-1 the down spins; blocks are the (N_up, N_down) sectors."""

    def __init__(self, n, terms, beta, is_complex=False):
        self.n, self.terms, self.beta, self.is_complex = n, terms, beta, is_complex
        s = np.arange(1 << (2 * n), dtype=np.int64)
        nu, nd = (sum((s >> (k + o)) & 1 for k in range(n)) for o in (0, n))
        self.block_of = (nu * (n + 1) + nd).astype(np.int32)
        order = np.argsort(self.block_of, kind="stable")
        self.dims = np.bincount(self.block_of).astype(np.int64)
        self.first = np.concatenate([[0], np.cumsum(self.dims)])
        self.fock = s[order]
        self.inner = np.empty(len(s), dtype=np.int32)
        self.inner[order] = (np.arange(len(s)) - self.first[self.block_of[order]]).astype(np.int32)

    def block(self, b):
        return self.fock[self.first[b]:self.first[b + 1]]

    def act(self, ops, states):
        """Images of Fock states under a product of (dagger, mode) and their signs (0 where it vanishes)."""
        st, sg = states.copy(), np.ones(len(states))
        for dag, m in reversed(ops):
            occ = (st >> m) & 1
            sg = np.where(occ == (0 if dag else 1), sg, 0.0)
            below = st & ((1 << m) - 1)
            par = np.zeros(len(st), dtype=np.int64)
            for k in range(m):
                par ^= (below >> k) & 1
            sg = np.where(par == 1, -sg, sg)
            st = np.where(sg != 0, st ^ (1 << m), st)
        return st, sg

    def action(self, sums):
        """Parts (right block, left block, targets, coefficients) of a sum of monomials that all map states alike."""
        parts = []
        for b in range(len(self.dims)):
            tgt, cf, left = np.full(self.dims[b], -1), np.zeros(self.dims[b]), -1
            for ops in sums:
                st, sg = self.act(ops, self.block(b))
                ok = sg != 0
                if ok.any():
                    left = int(self.block_of[st[ok][0]])
                    tgt[ok] = self.inner[st[ok]]
                    cf += sg
            if left >= 0:
                parts.append((b, left, tgt.astype(np.int32), cf))
        return parts

    def h(self, b):
        """Dense block of the Hamiltonian."""
        d = int(self.dims[b])
        H = np.zeros((d, d), dtype=complex if self.is_complex else float)
        k = np.arange(d)
        for ops, c in self.terms:
            st, sg = self.act(ops, self.block(b))
            ok = sg != 0
            np.add.at(H, (self.inner[st[ok]], k[ok]), (c if self.is_complex else np.real(c)) * sg[ok])
        return H


def number(m):
    return ((True, m), (False, m))


def hop(i, j, t):
    return [(((True, i), (False, j)), t), (((True, j), (False, i)), np.conj(t))]


def anderson(n, rng, U=3.0, beta=20.0, lo=0.2, hi=0.8):
    eps, V = rng.uniform(-2, 2, n - 1), rng.uniform(lo, hi, n - 1)
    t = [(number(0) + number(n), U), (number(0), -U / 2), (number(n), -U / 2)]
    for k in range(1, n):
        for o in (0, n):
            t += [(number(k + o), eps[k - 1])] + hop(o, k + o, V[k - 1])
    return Model(n, t, beta)


def ring(n, rng, flux=False):
    U, amp = rng.uniform(3.5, 4.5), -rng.uniform(0.9, 1.1)
    phase = np.exp(1j * rng.uniform(0.2, 1.0)) if flux else 1.0
    t = []
    for i in range(n):
        t += [(number(i) + number(i + n), U), (number(i), -U / 2), (number(i + n), -U / 2)]
        if n > 2 or i == 0:
            for o in (0, n):
                t += hop(i + o, (i + 1) % n + o, amp * phase)
    return Model(n, t, 10.0 if n <= 5 else 5.0, flux)


def kanamori(n, rng, U=2.5, J=0.4):
    Up, ed = U - 2 * J, -(3 * U - 5 * J) / 2
    eps, V = rng.uniform(-2, 2, n - 2), rng.uniform(0.2, 0.8, n - 2)
    t = []
    for o in (0, 1):
        q = 1 - o
        t += [(number(o) + number(o + n), U), (number(o), ed), (number(o + n), ed), (number(o) + number(q + n), Up)]
        t += [(((True, o), (False, o + n), (True, q + n), (False, q)), -J),
              (((True, o), (True, o + n), (False, q + n), (False, q)), J)]
    t += [(number(s) + number(1 + s), Up - J) for s in (0, n)]
    for k in range(2, n):
        for s in (0, n):
            t += [(number(k + s), eps[k - 2])] + hop((k % 2) + s, k + s, V[k - 2])
    return Model(n, t, 30.0)


def make(case, seed):
    rng = np.random.default_rng([seed, case["sites"]])
    if case["model"] == "anderson":
        return anderson(case["sites"], rng)
    if case["model"] == "kanamori":
        return kanamori(case["sites"], rng)
    return ring(case["sites"], rng, case["model"] == "flux")


def make_batch(case, seed):
    rng = np.random.default_rng([seed, case["models"]])
    return [anderson(1 + int(nb), rng, rng.uniform(1, 6), rng.uniform(5, 50), 0.1, 1.0)
            for nb in np.resize([5, 3, 6, 4], case["models"])]


def fermi(n, beta):
    return 1j * math.pi * (2 * np.arange(n) + 1) / beta


def bose(n, beta):
    return 2j * math.pi * np.arange(n) / beta


def grid(n, dim, beta):
    k = np.arange(-(n // 2), n - n // 2)
    return 1j * math.pi * (2 * np.stack(np.meshgrid(*([k] * dim), indexing="ij"), -1).reshape(-1, dim) + 1) / beta


PERMUTATIONS = [((0, 1, 2), 1), ((0, 2, 1), -1), ((1, 0, 2), -1), ((1, 2, 0), 1), ((2, 0, 1), 1), ((2, 1, 0), -1)]


def chains(cu, cd, keep):
    """Block chains S1 <O1| S2 <O2| S3 <O3| S4 <c+_d| S1 of chi_(u,d,u,d): (positions, blocks, permutation, sign).
    cu, cd: right -> left block maps of c+_u and c+_d."""
    au, ad = {v: k for k, v in cu.items()}, {v: k for k, v in cd.items()}
    right, left = [au, ad, cu], [cu, cd, au]  # c_u, c_d, c+_u: right -> left, left -> right
    out = []
    for s1, s4 in sorted(cd.items()):
        for p, sign in PERMUTATIONS:
            s2, s3 = left[p[0]].get(s1), right[p[2]].get(s4)
            if s2 is None or s3 is None or left[p[1]].get(s2) != s3 or not any(keep[b] for b in (s1, s2, s3, s4)):
                continue
            out.append((p, (s1, s2, s3, s4), sign))
    return out


def chain_set(case, m, parts):
    """All block chains, or the `chains` largest ones (a run over several GPUs deals them out in such pieces)."""
    if "chains" not in case:
        return parts
    return sorted(parts, key=lambda c: -math.prod(int(m.dims[b]) for b in c[1]))[:case["chains"]]


def ph_parts(cu, cd):
    """Parts of the particle-hole chi3(c+_u, c_u; c+_d c_d): (blocks i, j, k, m, swapped)."""
    out = []
    for i, m in ((r, k) for k, r in cd.items()):  # c_d: i -> m, then c+_d: m -> i
        if i in {v: 0 for v in cu.values()}:
            out.append(((i, {v: k for k, v in cu.items()}[i], i, m), False))
        if i in cu:
            out.append(((i, cu[i], i, m), True))
    return sorted(out)


# ---------------------------------------------------------------- states
class State:
    pass


def mapping(parts):
    return {r: l for r, l, _, _ in parts}


def engine_of(m):
    e = pgx.Engine(0)
    e.set_blocks(m.dims, m.is_complex)
    return e


def assemble(e, m):
    e.assemble_hamiltonian(m.terms, 2 * m.n, m.fock, m.block_of, m.inner)


def solve(s):
    """Eigensystem, weights and rotated operators of the state's model; c+ operators are s.ops, density is s.dens."""
    e = s.e
    e.eigh()
    w, Z = e.weights(s.m.beta)
    for op in s.ops.values():
        e.op_rotate(op)
    if s.dens is not None:
        e.op_rotate(s.dens)
    for op in s.adj.values():
        e.op_release(op)
    s.adj = {k: e.op_adjoint(op) for k, op in s.ops.items()}
    return w, Z


def prepare(case, seed):
    kind = case["kind"]
    s = State()
    s.case = case
    if kind == "dropin":
        return prepare_dropin(s, case, seed)
    if kind == "batch":
        return prepare_batch(s, case, seed)
    m = s.m = make(case, seed)
    e = s.e = engine_of(m)
    act = {"u": m.action([((True, 0),)])}
    if kind in ("g2", "chi3"):
        act["d"] = m.action([((True, m.n),)])
    dens = m.action([number(0), number(m.n)]) if kind in ("pair", "solve") else None
    s.ops = {k: e.op_define(a) for k, a in act.items()}
    s.dens = e.op_define(dens) if dens else None
    s.adj = {}
    maps = {k: mapping(a) for k, a in act.items()}
    s.outer, s.inner = (np.array(x, dtype=np.int32) for x in zip(*sorted(maps["u"].items())))
    s.diag = np.array([p[0] for p in dens], dtype=np.int32) if dens else None
    if kind in ("pair", "solve", "grad"):
        s.z = fermi(case["nz"], m.beta)
        s.zx = bose(case.get("nchi", 0), m.beta)
    if kind == "grad":
        s.target = target(case, seed)
        return s
    if kind == "solve":
        return s
    assemble(e, m)
    solve(s)
    if kind == "g2":
        keep = e.truncate_blocks(1e-12) if case["sites"] >= 8 else np.ones(len(m.dims), dtype=bool)
        ops = [s.adj["u"], s.adj["d"], s.ops["u"], s.ops["d"]]
        s.parts = [((ops[p[0]], ops[p[1]], ops[p[2]], ops[3]), b, p, sg)
                   for p, b, sg in chain_set(case, m, chains(maps["u"], maps["d"], keep))]
        s.z = grid(case["nfreq"], 3, m.beta)
        s.flags = {"exact": pgx.PGX_G2_EXACT, "anchored": pgx.PGX_G2_ANCHORED,
                   "split": pgx.PGX_G2_ANCHORED | pgx.PGX_G2_SPLIT_I8}[case["form"]]
        s.tol = 1e-13 if case["sites"] >= 8 else 1e-16
        if case["sites"] >= 8:
            e.set_g2_split_slices(5)
    elif kind == "chi3":
        cu, au, cd, ad = s.ops["u"], s.adj["u"], s.ops["d"], s.adj["d"]
        s.parts = [((au, cu) if sw else (cu, au)) + (cd, ad, b, sw) for b, sw in ph_parts(maps["u"], maps["d"])]
        s.z = grid(case["nfreq"], 2, m.beta)
    return s


def target(case, seed):
    """The function a fit aims at: a few poles."""
    rng = np.random.default_rng([seed, 77])
    z = fermi(case["nz"], 30.0)
    return (rng.dirichlet(np.ones(5))[:, None] / (z[None, :] - rng.uniform(-3, 3, 5)[:, None])).sum(0)


def prepare_batch(s, case, seed):
    s.ms = make_batch(case, seed)
    dims, blocks, cdag, dens, first = [], [], [], [], [0]
    for m in s.ms:
        o = len(dims)
        dims += list(m.dims)
        blocks += [m.h(b) for b in range(len(m.dims))]
        cdag += [(r + o, l + o, t, c) for r, l, t, c in m.action([((True, m.n),)])]
        dens += [(r + o, l + o, t, c) for r, l, t, c in m.action([number(0), number(m.n)])]
        first.append(len(dims))
    beta = np.array([m.beta for m in s.ms])
    e = s.e = pgx.Engine(0)
    e.set_blocks(dims)
    e.set_hamiltonian(blocks)
    e.set_models(first, beta)
    s.cdag, s.dens, s.c = e.op_define(cdag), e.op_define(dens), None
    s.outer, s.inner = (np.array(x, dtype=np.int32) for x in zip(*((r, l) for r, l, _, _ in cdag)))
    s.diag = np.array([r for r, _, _, _ in dens], dtype=np.int32)
    s.z = np.stack([fermi(case["nz"], b) for b in beta])
    s.zx = np.stack([bose(case["nchi"], b) for b in beta])
    return s


def prepare_dropin(s, case, seed):
    m = s.m = make(case, seed)
    n, U, t = m.n, m.terms[0][1], next(c for ops, c in m.terms if len(ops) == 2 and ops[0][1] != ops[1][1])
    L = P.LatticePresets
    s.expr = P.RealExpr()
    for i in range(n):
        s.expr += L.CoulombS("S%d" % i, float(U), float(-U / 2))
        if n > 2 or i == 0:
            s.expr += L.Hopping("S%d" % i, "S%d" % ((i + 1) % n), float(t))
    s.z = [complex(z) for z in fermi(case["nz"], m.beta)]
    s.triples = [tuple(complex(x) for x in r) for r in grid(case["nfreq"], 3, m.beta)]
    return s


# ---------------------------------------------------------------- one pass
def run(s):
    return {"pair": run_pair, "solve": run_solve, "g2": run_g2, "chi3": run_chi3, "grad": run_grad, "batch": run_batch,
            "dropin": run_dropin}[s.case["kind"]](s)


def run_pair(s):
    G = s.e.gf(s.adj["u"], s.ops["u"], s.outer, s.inner, s.z, coef_tol=0.0)
    X, zero = s.e.susc(s.dens, s.dens, s.diag, s.diag, s.zx, s.m.beta, coef_tol=0.0)
    return {"G": G, "X": X, "zero": np.array([zero])}


def run_solve(s):
    assemble(s.e, s.m)
    w, Z = solve(s)
    return dict(run_pair(s), w=np.concatenate(w), Z=Z)


def run_g2(s):
    return {"G2": s.e.g2(s.parts, s.z, pole_res=POLE_RES, coef_tol=s.tol if s.flags else 1e-16, flags=s.flags)}


def run_chi3(s):
    return {"chi3": s.e.chi3(pgx.PGX_PH, s.parts, s.z, POLE_RES)}


def run_grad(s):
    assemble(s.e, s.m)
    solve(s)
    a, b = s.adj["u"], s.ops["u"]
    G = s.e.gf(a, b, s.outer, s.inner, s.z, coef_tol=0.0)
    dterm, dE = s.e.gf_vjp(a, b, s.outer, s.inner, s.z, 2 * np.conj(G - s.target))
    return {"G": G, "dterm": dterm, "dE": dE}


def run_batch(s):
    e = s.e
    e.eigh()
    w, _, Z = e.weights_models()
    e.op_rotate(s.cdag)
    e.op_rotate(s.dens)
    if s.c is not None:
        e.op_release(s.c)
    s.c = e.op_adjoint(s.cdag)
    G = e.gf_models(s.c, s.cdag, s.outer, s.inner, s.z, coef_tol=0.0)
    X, zero = e.susc_models(s.dens, s.dens, s.diag, s.diag, s.zx, coef_tol=0.0)
    return {"G": G, "X": X, "zero": zero, "w": np.concatenate(w), "Z": Z}


def run_dropin(s):
    ii = P.MakeIndexClassification(s.expr)
    hs = P.MakeHilbertSpace(ii, s.expr)
    hs.compute()
    S = P.StatesClassification()
    S.compute(hs)
    H = P.Hamiltonian(S)
    H.prepare(s.expr, hs)
    H.compute()
    rho = P.DensityMatrix(S, H, s.m.beta)
    rho.prepare()
    rho.compute()
    u, d = ii.getIndex("S0", 0, P.up), ii.getIndex("S0", 0, P.down)
    ops = P.FieldOperatorContainer(ii, hs, S, H, {u, d})
    ops.prepareAll(hs)
    ops.computeAll()
    g = P.GreensFunction(S, H, ops.getAnnihilationOperator(u), ops.getCreationOperator(u), rho)
    g.CoefficientTolerance = 0.0
    g.prepare()
    g.compute()
    chi = P.TwoParticleGFContainer(ii, S, H, rho, ops)
    chi.prepareAll([(u, d, u, d)])
    return {"G": np.asarray(g.values(s.z)), "G2": np.asarray(chi.computeAll(True, s.triples)[(u, d, u, d)])}


# ---------------------------------------------------------------- the work of a pass
def sector_dims(n):
    c = [math.comb(n, k) for k in range(n + 1)]
    return {(a, b): c[a] * c[b] for a in range(n + 1) for b in range(n + 1)}


#: share of a model's states whose Boltzmann weight is over the anchored sum's threshold
ANCHORS = {"anderson": 0.015, "ring": 0.2, "flux": 0.3, "kanamori": 0.02}


def work(case):
    """Estimates from the block sizes: each matrix read or written once, 64-bit multiply-adds of the chain."""
    if case["kind"] == "batch":
        w = [work(dict(case, kind="solve", sites=1 + int(nb))) for nb in np.resize([5, 3, 6, 4], case["models"])]
        return {k: sum(x[k] for x in w) for k in ("bytes", "flops")}
    n, cx = case["sites"], 4 if case["model"] == "flux" else 1
    d = sector_dims(n)
    up = [(v, d[(a + 1, b)]) for (a, b), v in d.items() if a < n]
    sq = sum(v * v for v in d.values())
    pair = sum(a * b for a, b in up)
    g = {"bytes": 8 * cx * (pair + sq), "flops": 12 * (pair * case.get("nz", 0) + sq * case.get("nchi", 0))}
    eig = {"bytes": 8 * cx * 2 * sq, "flops": cx * (14 / 3 * sum(v ** 3 for v in d.values())
                                                      + 2 * sum(a * b * (a + b) / 2 for a, b in up))}
    nf = case.get("nfreq", 0)
    if case["kind"] == "pair":
        return g
    if case["kind"] in ("solve", "grad"):
        more = 2 if case["kind"] == "grad" else 1
        return {k: eig[k] * more + g[k] * more for k in g}
    r = 1.0 if case.get("form") == "exact" else 0.05 if n >= 8 else ANCHORS[case["model"]]
    keys = sorted(d)
    pos = {k: i for i, k in enumerate(keys)}
    size = [d[k] for k in keys]
    cu = {pos[k]: pos[(k[0] + 1, k[1])] for k in keys if k[0] < n}
    cd = {pos[k]: pos[(k[0], k[1] + 1)] for k in keys if k[1] < n}
    if case["kind"] == "chi3":
        blocks = [b for b, _ in ph_parts(cu, cd)]
        return {"bytes": 8 * sum(size[i] * (2 * size[j] + size[m]) for i, j, _, m in blocks) + 48 * nf ** 2,
                "flops": sum(4 * size[i] * size[j] * size[k] * nf + 8 * size[i] * size[k] * nf ** 2
                             for i, j, k, _ in blocks)}
    every = [b for _, b, _ in chains(cu, cd, [True] * len(size))]
    if "chains" in case:
        every = sorted(every, key=lambda b: -math.prod(size[x] for x in b))[:case["chains"]]
    flops = nbytes = 0.0
    for b in every:
        d1, d2, d3, d4 = (size[x] for x in b)
        # per (z1, z3): the anchors' rows or columns of two products through the middle; per triple: their contractions
        flops += r * nf ** 2 * 8 * (2 * d2 * d3 * d4 + 2 * d1 * d3 * d4)
        flops += r * nf ** 3 * 8 * (d1 * d4 + d2 * d3 + d1 * d3 + d2 * d4)
        nbytes += 8 * cx * (d1 * d2 + d2 * d3 + d3 * d4 + d4 * d1)
    out = {"bytes": nbytes + 64 * nf ** 3, "flops": cx * flops}
    return out if case["kind"] == "g2" else {k: out[k] + eig[k] + g[k] for k in out}


# ---------------------------------------------------------------- the same in plain torch, 64 bits
def on():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


class Solved:
    """Eigensystem, weights and rotated operators of a Model by torch.linalg."""

    def __init__(self, m):
        self.m = m
        dev = on()
        self.E, self.U = [], []
        for b in range(len(m.dims)):
            E, U = torch.linalg.eigh(torch.from_numpy(m.h(b)).to(dev))
            self.E.append(E)
            self.U.append(U)
        e0 = min(float(E.min()) for E in self.E)
        raw = [torch.exp(-m.beta * (E - e0)) for E in self.E]
        self.Z = sum(float(x.sum()) for x in raw)
        self.w = [x / self.Z for x in raw]

    def rotate(self, action):
        """{right block: (left block, matrix)}"""
        out = {}
        for r, l, t, c in action:
            t, c = torch.from_numpy(np.asarray(t)).long().to(on()), torch.from_numpy(c).to(on())
            k = torch.nonzero(t >= 0)[:, 0]
            out[r] = (l, self.U[l].conj()[t[k]].T @ (c[k, None] * self.U[r][k]))
        return out


def tz(z):
    return torch.from_numpy(np.asarray(z, dtype=complex)).to(on())


def poles(R, Q, z):
    """sum R / (z - Q) over all pairs, in pieces."""
    R, Q = R.reshape(-1), Q.reshape(-1)
    return torch.stack([(R / (x - Q)).sum() for x in z]) if R.numel() * len(z) > 1 << 26 else \
        (R[None, :] / (z[:, None] - Q[None, :])).sum(1)


def exact_pair(q, case, cu, dens, z, zx):
    G = torch.zeros(len(z), dtype=torch.complex128, device=on())
    for r, (l, C) in q.rotate(cu).items():
        G += poles((C.abs() ** 2).T * (q.w[r][:, None] + q.w[l][None, :]), q.E[l][None, :] - q.E[r][:, None], z)
    X, zero = torch.zeros(len(zx), dtype=torch.complex128, device=on()), 0.0
    for b, (_, N) in q.rotate(dens).items():
        A, Q = N.abs() ** 2, q.E[b][None, :] - q.E[b][:, None]
        near = Q.abs() < POLE_RES
        zero = zero + float((A * q.w[b][:, None])[near].sum())
        X -= poles(torch.where(near, 0.0, A * (q.w[b][:, None] - q.w[b][None, :])), torch.where(near, 1e300, Q), zx)
    X = X + (zx.abs() <= 2.3e-16).double() * (zero * q.m.beta)
    return {"G": G, "X": X, "zero": torch.tensor([zero], dtype=torch.complex128)}


def exact_g2(q, case, cu, cd):
    m = q.m
    nf, beta = case["nfreq"], m.beta
    u, d = q.rotate(cu), q.rotate(cd)
    adj = {0: {l: (r, C.conj().T) for r, (l, C) in u.items()}, 1: {l: (r, C.conj().T) for r, (l, C) in d.items()}, 2: u}
    lefts = [{l: (r, C) for r, (l, C) in adj[k].items()} for k in range(3)]
    axis = tz(1j * math.pi * (2 * np.arange(-(nf // 2), nf - nf // 2) + 1) / beta)
    out = torch.zeros(nf, nf, nf, dtype=torch.complex128, device=on())
    for p, blocks, sign in chain_set(case, m, chains(mapping(cu), mapping(cd), [True] * len(m.dims))):
        b1, b2, b3, b4 = blocks
        O1, O2 = lefts[p[0]][b1][1].to(torch.complex128), lefts[p[1]][b2][1].to(torch.complex128)
        O3, X4 = adj[p[2]][b4][1].to(torch.complex128), d[b1][1].to(torch.complex128)
        E1, E2, E3, E4 = (q.E[b] for b in blocks)
        w1, w2, w3, w4 = (q.w[b] for b in blocks)
        z = [(-axis if k == 2 else axis) for k in p]  # permuted (a, b, c) of {z1, z2, -z3}
        A = O1 / (z[0][:, None, None] - (E2[None, :] - E1[:, None]))
        C = O3 / (z[2][:, None, None] - (E4[None, :] - E3[:, None]))
        B = O2 / (z[1][:, None, None] - (E3[None, :] - E2[:, None])) * (w2[:, None] + w3[None, :])
        AO, CX, OC, XA = A @ O2, C @ X4, O2 @ C, X4 @ A
        got = torch.zeros(nf, nf, nf, dtype=torch.complex128, device=on())  # [a, b, c]
        Bf = B.reshape(nf, -1).T
        sums, at = torch.unique(torch.round((z[1][:, None] + z[2][None, :]).imag * beta / math.pi), return_inverse=True)
        sums = 1j * math.pi / beta * sums
        for i in range(nf):
            G = CX @ A[i]                                            # c: S3 x S2
            got[i] -= (G.transpose(1, 2).reshape(nf, -1) @ Bf).T
            Y = X4.T * (AO[i] @ C)                                   # c: S1 x S4
            K = (w1[:, None] + w4[None, :]) / ((z[0][i] + sums)[:, None, None] - (E4[None, :] - E1[:, None]))
            got[i] += torch.gather(K.reshape(len(sums), -1) @ Y.reshape(nf, -1).T, 0, at)
            D = (z[0][i] + z[1])[:, None, None] - (E3[None, :] - E1[:, None])
            hit = D.abs() <= POLE_RES
            F = torch.where(hit, beta * w1[:, None], (w3[None, :] - w1[:, None]) / torch.where(hit, 1.0, D))
            got[i] += (AO[i] * F).reshape(nf, -1) @ CX.transpose(1, 2).reshape(nf, -1).T
        for k in range(nf):
            D = (z[1] + z[2][k])[:, None, None] - (E4[None, :] - E2[:, None])
            hit = D.abs() <= POLE_RES
            F = torch.where(hit, -beta * w2[:, None], (w2[:, None] - w4[None, :]) / torch.where(hit, 1.0, D))
            got[:, :, k] += XA.transpose(1, 2).reshape(nf, -1) @ (OC[k] * F).reshape(nf, -1).T
        back = [p.index(k) for k in range(3)]
        out += sign * got.permute(back)
    return {"G2": out.reshape(-1)}


def exact_chi3(q, case, cu, cd):
    nf, beta = case["nfreq"], q.m.beta
    u, d = q.rotate(cu), q.rotate(cd)
    axis = tz(1j * math.pi * (2 * np.arange(-(nf // 2), nf - nf // 2) + 1) / beta)
    out = torch.zeros(nf, nf, dtype=torch.complex128, device=on())
    au = {l: (r, C.conj().T) for r, (l, C) in u.items()}
    for (i, j, k, m), sw in ph_parts(mapping(cu), mapping(cd)):
        F1 = (au[j][1] if sw else u[j][1]).to(torch.complex128)      # <i|F1|j>
        F2 = (u[k][1] if sw else au[k][1]).to(torch.complex128)      # <j|F2|k>
        B = (d[m][1] @ d[m][1].conj().T).to(torch.complex128)        # <k|c+_d c_d|i>, k = i
        Ei, Ej, Ek, wi, wj, wk = q.E[i], q.E[j], q.E[k], q.w[i], q.w[j], q.w[k]
        pf = 1.0 if sw else -1.0
        Eij, Ejk, Eik = Ei[:, None] - Ej[None, :], Ej[:, None] - Ek[None, :], Ei[:, None] - Ek[None, :]
        far = Eik.abs() > POLE_RES
        each = axis[:, None, None]
        for a in range(nf):
            z1, near = axis[a], torch.where(far.T, 0.0, B * wi[None, :])
            FB = torch.where(far.T, B * (wk[:, None] - wi[None, :]) / torch.where(far.T, z1 - each - Eik.T, 1.0), 0.0)
            if sw:
                D1, D2 = F1 / (each + Eij), F2 / (z1 - Ejk)
                v = ((B * wi[None, :]).T * (D1 @ D2) + B.T * ((D1 * wj[None, :]) @ D2)).sum((1, 2))
                v = pf * v - pf * (FB.transpose(1, 2) * (F1 @ D2)).sum((1, 2))
                v[a] += beta * pf * (near.T * (F1 @ D2)).sum()
            else:
                D1, D2 = F1 / (z1 - Eij), F2 / (each + Ejk)
                W = torch.where(far, wk[None, :], wi[:, None])
                v = (B.T * W * (D1 @ D2) + B.T * ((D1 * wj[None, :]) @ D2)).sum((1, 2))
                v = pf * v + pf * (FB.transpose(1, 2) * (D1 @ F2)).sum((1, 2))
                v[a] -= beta * pf * (near.T * (F1 @ (F2 / (z1 + Ejk)))).sum()
            out[a] += v
    return {"chi3": out.reshape(-1)}


def exact_grad(q, case, seed, cu):
    """G, and the reverse pass through the Lehmann sum, the weights, the rotation and the eigensystem."""
    m, z = q.m, tz(fermi(case["nz"], q.m.beta))
    rot = q.rotate(cu)
    G = exact_pair(q, case, cu, [], z, z[:0])["G"]
    lam = 2 * (G - tz(target(case, seed))).conj()
    Eb, wb = ([torch.zeros_like(E) for E in q.E] for _ in (0, 1))
    Ub = [torch.zeros_like(U) for U in q.U]
    for r, l, t, c in cu:
        C = rot[r][1]                                                # l x r
        pole = q.E[l][:, None] - q.E[r][None, :]
        Px, Qx = torch.zeros_like(pole), torch.zeros_like(pole)
        for x, y in zip(z, lam):
            inv = 1.0 / (x - pole)
            Px += (y * inv).real
            Qx += (y * inv * inv).real
        s = q.w[l][:, None] + q.w[r][None, :]
        wb[l] += (C * C * Px).sum(1)
        wb[r] += (C * C * Px).sum(0)
        de = C * C * s * Qx
        Eb[l] += de.sum(1)
        Eb[r] -= de.sum(0)
        Cb = 2 * C * s * Px
        t, c = torch.from_numpy(np.asarray(t)).long().to(on()), torch.from_numpy(c).to(on())
        k = torch.nonzero(t >= 0)[:, 0]
        Ub[l].index_add_(0, t[k], c[k, None] * (q.U[r] @ Cb.T)[k])
        Ub[r].index_add_(0, k, c[k, None] * (q.U[l] @ Cb)[t[k]])
    S = sum(float(a @ b) for a, b in zip(q.w, wb))
    top = max(1.0, max(float(E.abs().max()) for E in q.E))
    dterm = [0.0] * len(m.terms)
    for b in range(len(q.E)):
        Eb[b] -= m.beta * q.w[b] * (wb[b] - S)
        gap = q.E[b][None, :] - q.E[b][:, None]
        keep = gap.abs() > 1e-10 * top
        X = torch.where(keep, 1.0 / torch.where(keep, gap, 1.0), 0.0) * (q.U[b].T @ Ub[b]) + torch.diag(Eb[b])
        H = q.U[b] @ X @ q.U[b].T
        H = (0.5 * (H + H.T)).cpu().numpy()
        for i, (ops, _) in enumerate(m.terms):
            st, sg = m.act(ops, m.block(b))
            k = np.nonzero(sg)[0]
            dterm[i] += float((sg[k] * H[m.inner[st[k]], k]).sum())
    return {"G": G, "dterm": torch.tensor(dterm, dtype=torch.float64), "dE": torch.cat(Eb)}


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return exact_batch(case, seed) if case["models"] <= 12 else None
    nf = case.get("nfreq", 0)
    if kind == "g2" and (case["sites"] >= 8 or sum(v ** 3 for v in sector_dims(case["sites"]).values()) * nf ** 2 > 1e12):
        return None  # minutes, or hours, in this form
    m = make(case, seed)
    q = Solved(m)
    cu, dens = m.action([((True, 0),)]), m.action([number(0), number(m.n)])
    if kind == "grad":
        return exact_grad(q, case, seed, cu)
    if kind == "chi3":
        return exact_chi3(q, case, cu, m.action([((True, m.n),)]))
    out = {}
    if kind != "g2":
        out = exact_pair(q, case, cu, dens, tz(fermi(case["nz"], m.beta)), tz(bose(case.get("nchi", 0), m.beta)))
    if kind in ("g2", "dropin"):
        out.update(exact_g2(q, case, cu, m.action([((True, m.n),)])))
    if kind == "dropin":
        return {k: out[k] for k in ("G", "G2")}
    if kind == "solve":
        out.update(w=torch.cat(q.w), Z=q.Z)
    return out


def exact_batch(case, seed):
    got = []
    for m in make_batch(case, seed):
        q = Solved(m)
        o = exact_pair(q, case, m.action([((True, m.n),)]), m.action([number(0), number(m.n)]),
                       tz(fermi(case["nz"], m.beta)), tz(bose(case["nchi"], m.beta)))
        got.append(dict(o, w=torch.cat(q.w), Z=torch.tensor([q.Z], dtype=torch.float64)))
    return {"G": torch.stack([o["G"] for o in got]), "X": torch.stack([o["X"] for o in got]),
            "zero": torch.cat([o["zero"] for o in got]), "w": torch.cat([o["w"] for o in got]),
            "Z": torch.cat([o["Z"] for o in got])}
