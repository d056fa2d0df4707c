"""The two forms of the exact G2 sum, each against the oracle and against one
another: full matrices part by part (PGX_G2_FULL_MATRICES) and all parts
together with every state an anchor."""
import numpy as np
import pytest

from oracle import ed as EDm
from oracle import lehmann as L
from oracle import model as M
from tests.test_g2_plans import solved, with_odd_values
from tests.test_gpu_kernels import FORMS, engine, freq_list, small_model, symmetric

pytestmark = pytest.mark.gpu


def batched(eng, *args, **kw):
    """The sum, and whether the batched form's contractions ran."""
    eng.profile_begin()
    v = eng.g2(*args, **kw)
    return v, any("contract_gemm" in k["name"] for k in eng.profile_end())


# The bound of the other G2 tests over these lists: 1e-12 of the largest value,
# that of both operator choices (with equal operators the sum at z1 = z2 is zero,
# its terms are not).
@pytest.mark.parametrize("kind", ["real", "complex"])
@pytest.mark.parametrize("form", FORMS)
def test_full_matrices_over_forms_of_frequency_lists(form, kind):
    from pomerol_b200.pgx import PGX_G2_EXACT, PGX_G2_FULL_MATRICES
    g, u, d = solved(kind)
    ed = EDm.ED(small_model(kind), 7.0)
    z = freq_list(form, 3, 7.0, np.random.default_rng(5))
    sel = np.unique(np.linspace(0, len(z) - 1, 24).astype(int))
    ref, full, exact = [], [], []
    for i, j in ((u, d), (u, u)):
        parts = g.g2_parts(g.c(i), g.c(j), g.cdag(i), g.cdag(j))
        oparts = L.g2_parts(ed, ed.c(i), ed.c(j), ed.cdag(i), ed.cdag(j))
        assert len({p[2] for p in parts}) == 6
        ref.append(L.g2_exact(ed, oparts, [tuple(z[t]) for t in sel]))
        v, b = batched(g.eng, parts, z, flags=PGX_G2_FULL_MATRICES)
        assert not b
        full.append(v)
        exact.append(g.eng.g2(parts, z, flags=PGX_G2_EXACT))
    ref, full, exact = np.array(ref), np.array(full), np.array(exact)
    scale = max(np.abs(ref).max(), np.abs(full).max())
    assert np.abs(full[:, sel] - ref).max() < 1e-12 * scale
    assert np.abs(exact - full).max() < 1e-12 * scale


# 36-state blocks with exact degeneracies, so the delta branches count at zero
# bosonic transfer.
@pytest.mark.parametrize("beta", [2.0, 10.0])
def test_both_forms_of_the_plaquette_against_the_oracle(beta):
    from pomerol_b200.pgx import PGX_G2_EXACT, PGX_G2_FULL_MATRICES
    from tests.pgx_harness import GpuED
    m = M.make_model(M.plaquette())
    g, ed = GpuED(m, beta), EDm.ED(m, beta)
    u, d = m.info.getIndex("A", 0, 1), m.info.getIndex("A", 0, 0)
    fz = L.fermionic(np.array([(a, b, x) for a in range(-3, 3) for b in range(-3, 3) for x in range(-3, 3)]), beta)
    parts = g.g2_parts(g.c(u), g.c(d), g.cdag(u), g.cdag(d))
    oparts = L.g2_parts(ed, ed.c(u), ed.c(d), ed.cdag(u), ed.cdag(d))
    sel = list(range(0, len(fz), 9))
    ref = L.g2_exact(ed, oparts, [tuple(fz[t]) for t in sel])
    full, b1 = batched(g.eng, parts, fz, flags=PGX_G2_FULL_MATRICES)
    exact, b2 = batched(g.eng, parts, fz, flags=PGX_G2_EXACT)
    assert b2 and not b1
    for v in (full, exact):
        assert np.abs(v[sel] - ref).max() < 1e-10 * np.abs(ref).max()
    assert np.abs(full - exact).max() < 1e-10 * np.abs(full).max()


def test_anderson_a5_in_full_matrices():
    """Anderson 1+5 (blocks to 400 states): the full-matrix sum over every
    quadruple on a 4^3 part of the 16^3 cube against the oracle (ordinary and
    resonant triples), the batched form and the anchored sum."""
    from pomerol_b200.pgx import PGX_G2_ANCHORED, PGX_G2_EXACT, PGX_G2_FULL_MATRICES
    from tests.pgx_harness import GpuED
    U, epsd, eps, V, beta = M.anderson_a5_params(0)
    m = M.make_model(M.anderson(U, epsd, eps, V))
    g, ed = GpuED(m, beta), EDm.ED(m, beta)
    u, d = m.info.getIndex("C", 0, 1), m.info.getIndex("C", 0, 0)
    S = (-8, -1, 0, 7)
    trip = np.array([(a, b, x) for a in S for b in S for x in S])
    fz = L.fermionic(trip, beta)
    parts = g.g2_parts(g.c(u), g.c(d), g.cdag(u), g.cdag(d))
    full, b = batched(g.eng, parts, fz, flags=PGX_G2_FULL_MATRICES)
    assert not b
    for flags, tol in ((PGX_G2_EXACT, 0.0), (PGX_G2_ANCHORED, 1e-16)):
        v = g.eng.g2(parts, fz, coef_tol=tol, flags=flags)
        assert np.abs(v - full).max() < 1e-9 * np.abs(full).max()
    oparts = L.g2_parts(ed, ed.c(u), ed.c(d), ed.cdag(u), ed.cdag(d))
    pick = [(-8, -8, -8), (7, 0, -8), (-1, 0, -1), (7, -1, -1)]
    sel = [int(np.flatnonzero((trip == np.array(t)).all(1))[0]) for t in pick]
    ref = L.g2_exact(ed, oparts, [tuple(fz[t]) for t in sel])
    assert np.abs(full[sel] - ref).max() < 1e-9 * np.abs(ref).max()


def test_rule_of_the_exact_sum():
    """Scattered triples of one chain of 70 to 126 states take full matrices, a
    grid of it the batched form; both forms give the same sums."""
    from pomerol_b200.pgx import PGX_G2_EXACT, PGX_G2_FULL_MATRICES
    rng = np.random.default_rng(9)
    dims = [70, 96, 126, 84]
    e = engine([symmetric(rng, n) / 4 for n in dims])
    e.eigh()
    e.weights(2.0)
    ops = []
    for q in range(4):
        left, right = q, (q + 1) % 4
        tgt = np.full(dims[right], -1)
        k = min(dims[left], dims[right])
        tgt[:k] = rng.permutation(dims[left])[:k]
        ops.append(e.op_define([(right, left, tgt, np.where(tgt >= 0, 1.0, 0.0))]))
        e.op_rotate(ops[-1])
    k = 1j * np.pi * (2 * np.arange(-2, 2) + 1) / 2.0
    lists = {False: 1j * rng.uniform(0.5, 9, (150, 3)) * rng.choice([-1, 1], (150, 3)),
             True: np.stack(np.meshgrid(k, k, k, indexing="ij"), -1).reshape(-1, 3)}
    for perm, sign in (((0, 1, 2), 1), ((2, 0, 1), 1), ((1, 0, 2), -1)):
        parts = [(tuple(ops), (0, 1, 2, 3), perm, sign)]
        for grid, z in lists.items():
            v, b = batched(e, parts, z, flags=PGX_G2_EXACT)
            full, bf = batched(e, parts, z, flags=PGX_G2_FULL_MATRICES)
            assert b == grid and not bf
            assert np.abs(v - full).max() < 1e-12 * np.abs(full).max()


# Nearly equal levels at zero bosonic transfer: (w3 - w1)/D is of the order of
# beta w however small D is, and both forms take it from the same weights and
# energies, so they differ by the rounding of the products around it only.  A
# form that divides w3 and w1 by D apart enlarges that rounding by 1 / (beta D).
@pytest.mark.parametrize("kind", ["real", "complex"])
@pytest.mark.parametrize("split", [1e-7, 1e-6, 1e-5])
def test_nearly_equal_levels(split, kind):
    from pomerol_b200.pgx import PGX_G2_EXACT, PGX_G2_FULL_MATRICES
    from tests.pgx_harness import GpuED
    if kind == "real":
        e = M.plaquette()
    else:
        e = M.CoulombS("A", 2.0, -1.2) + M.CoulombS("B", 2.5, -0.9) + M.CoulombS("C", 1.5, -0.8)
        for a, b, t in (("A", "B", 0.7 * np.exp(0.4j)), ("B", "C", 0.5j), ("C", "A", -0.6)):
            for s in (M.UP, M.DOWN):
                e += M.HoppingS(a, b, t, 0, 0, s, s)
    e += M.Level1("A", split, 0, M.DOWN)
    m = M.make_model(e)
    g = GpuED(m, 10.0)
    u, d = m.info.getIndex("A", 0, 1), m.info.getIndex("A", 0, 0)
    fz = L.fermionic(np.array([(a, b, x) for a in range(-2, 2) for b in range(-2, 2) for x in range(-2, 2)]), 10.0)
    parts = g.g2_parts(g.c(u), g.c(d), g.cdag(u), g.cdag(d))
    full = g.eng.g2(parts, fz, flags=PGX_G2_FULL_MATRICES)
    exact, b = batched(g.eng, parts, fz, flags=PGX_G2_EXACT)
    assert b
    assert np.abs(exact - full).max() < 1e-13 * np.abs(full).max()


@pytest.mark.parametrize("kind", ["real", "complex"])
def test_neighbouring_frequencies_keep_their_own_values(kind):
    """z2 a few units apart, 1e-9 from a pole, where 40 units are 1e-6 of the sum or more:
    each triple's value is that of a call of its own.  A difference z - E is the
    same number in both calls, so the values agree to rounding."""
    from pomerol_b200.pgx import PGX_G2_ANCHORED, PGX_G2_EXACT
    g, u, d = solved(kind)
    parts = g.g2_parts(g.c(u), g.c(d), g.cdag(u), g.cdag(d))
    ops, b, _, _ = next(p for p in parts if p[2] == (0, 1, 2) and min(len(g.E[x]) for x in p[1]) > 2)
    left = [l for _, l in g.eng.op_info(ops[1])].index(b[1])
    i, j = np.unravel_index(np.abs(g.eng.op_read(ops[1], left)).argmax(), (len(g.E[b[1]]), len(g.E[b[2]])))
    pole = g.E[b[2]][j] - g.E[b[1]][i]
    z = np.array([(0.7j, pole + 1e-9 + k * 40 * np.spacing(abs(pole)), 0.3 - 1.1j) for k in range(8)])
    for flags in (PGX_G2_EXACT, PGX_G2_ANCHORED):
        v = g.eng.g2(parts, z, coef_tol=0.0, flags=flags)
        one = np.array([g.eng.g2(parts, t[None], coef_tol=0.0, flags=flags)[0] for t in z])
        assert np.abs(np.diff(one)).max() > 1e-7 * np.abs(one).max()  # the pole is felt
        assert np.all(np.abs(v - one) < 1e-9 * np.abs(one))


@pytest.mark.parametrize("kind", ["real", "complex"])
def test_negative_pole_resolution(kind):
    """|D| <= pole_res holds nowhere then, also for bosonic sums nearer to a pole
    than its modulus."""
    from pomerol_b200.pgx import PGX_G2_ANCHORED, PGX_G2_EXACT, PGX_G2_FULL_MATRICES
    g, u, d = solved(kind)
    ed = EDm.ED(small_model(kind), 7.0)
    rng = np.random.default_rng(8)
    z = 1j * rng.uniform(0.4, 3, (12, 3)) * rng.choice([-1, 1], (12, 3))
    z[::2, 1] = -z[::2, 0] + 0.2j
    z[1::2, 2] = z[1::2, 1] - 0.15j
    parts = g.g2_parts(g.c(u), g.c(d), g.cdag(u), g.cdag(d))
    oparts = L.g2_parts(ed, ed.c(u), ed.c(d), ed.cdag(u), ed.cdag(d))
    ref = L.g2_exact(ed, oparts, [tuple(t) for t in z], res=-0.5)
    for flags in (PGX_G2_EXACT, PGX_G2_FULL_MATRICES, PGX_G2_ANCHORED):
        v = g.eng.g2(parts, z, pole_res=-0.5, coef_tol=0.0, flags=flags)
        assert np.abs(v - ref).max() < 1e-12 * np.abs(ref).max()


@pytest.mark.parametrize("dims,n", [([300, 2, 310, 1], 25), ([1, 7, 2, 9], 60)])
def test_scattered_triples_of_one_chain_stay_in_full_matrices(dims, n):
    """Few states in some blocks, so the batched form's products are mostly the
    padding of their tiles, or few operations in all, so that its planning counts:
    it took 1.3 to 1.9 times as long here."""
    from pomerol_b200.pgx import PGX_G2_ANCHORED, PGX_G2_EXACT
    rng = np.random.default_rng(5)
    e = engine([symmetric(rng, k) / 4 for k in dims])
    e.eigh()
    e.weights(3.0)
    ops = []
    for q in range(4):
        left, right = q, (q + 1) % 4
        tgt = np.full(dims[right], -1)
        k = min(dims[left], dims[right])
        tgt[:k] = rng.permutation(dims[left])[:k]
        ops.append(e.op_define([(right, left, tgt, np.where(tgt >= 0, 1.0, 0.0))]))
        e.op_rotate(ops[-1])
    parts = [(tuple(ops), (0, 1, 2, 3), (0, 1, 2), 1)]
    z = rng.uniform(-2, 2, (n, 3)) + 1j * rng.uniform(0.2, 2, (n, 3))
    v, b = batched(e, parts, z, flags=PGX_G2_EXACT)
    assert not b
    anchored = e.g2(parts, z, coef_tol=0.0, flags=PGX_G2_ANCHORED)
    assert np.abs(v - anchored).max() < 1e-12 * np.abs(v).max()


@pytest.mark.parametrize("kind", ["real", "complex"])
@pytest.mark.parametrize("place", [0, 1, 2])
def test_full_matrices_beside_undefined_frequencies(place, kind):
    from pomerol_b200.pgx import PGX_G2_FULL_MATRICES
    g, u, d = solved(kind)
    z = freq_list("odd", 3, 7.0, np.random.default_rng(5))
    y, keep = with_odd_values(z, place, np.random.default_rng(place))
    parts = g.g2_parts(g.c(u), g.c(d), g.cdag(u), g.cdag(d))
    ref = g.eng.g2(parts, z, flags=PGX_G2_FULL_MATRICES)
    got = g.eng.g2(parts, y, flags=PGX_G2_FULL_MATRICES)
    assert np.abs(got[keep] - ref[keep]).max() < 1e-12 * np.abs(ref).max()
