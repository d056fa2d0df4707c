"""Kernels at the sizes where they can go wrong (edges of tiles, remainders,
both sides of a dispatch), on random blocks through the C ABI, against numpy."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
EPS = np.finfo(float).eps


def engine(blocks, is_complex=False):
    from pomerol_b200.pgx import Engine
    e = Engine(0)
    e.set_blocks([len(b) for b in blocks], is_complex)
    e.set_hamiltonian(blocks)
    return e


def symmetric(rng, n, kind="dense"):
    """dense: random; pieces: exact degeneracies and splits (a block-diagonal
    matrix of equal 5 x 5 blocks and a constant diagonal tail)."""
    if kind == "dense":
        a = rng.standard_normal((n, n))
        return (a + a.T) / 2
    a = np.zeros((n, n))
    s = rng.standard_normal((5, 5))
    for k in range(0, n // 2 - 5, 5):
        a[k:k + 5, k:k + 5] = s + s.T
    a[np.arange(n // 2, n), np.arange(n // 2, n)] = 0.25
    return a


# Reduction to tridiagonal form and the reflectors' application carry a
# backward error of a few n eps ||H||; vectors of eigenvalues further apart than
# 1e-4 ||H|| are left as inverse iteration gives them, orthogonal to eps / 1e-4.
@pytest.mark.parametrize("kind", ["dense", "pieces"])
@pytest.mark.parametrize("dims", [[1, 2, 3, 4, 31, 32, 33, 34, 35, 66, 67, 127], [463, 464, 465, 513, 514, 679, 680],
                                  [1273, 1274, 600], [697, 698, 1489, 1490], [3073, 3074], [1025] + [900] * 16,
                                  [3] * 400, [7, 5] * 150])
def test_eigensolve_at_the_edges_of_its_paths(dims, kind):
    rng = np.random.default_rng(sum(dims))
    H = [symmetric(rng, n, kind) for n in dims]
    e = engine(H)
    e.eigh()
    E, U = e.eigensystem()
    for h, w, u in zip(H, E, U):
        n, norm = len(h), max(1.0, np.abs(np.linalg.eigvalsh(h)).max())
        assert np.all(np.diff(w) >= 0)
        assert np.abs(w - np.linalg.eigvalsh(h)).max() < 10 * (n + 10) * EPS * norm
        assert np.abs(h @ u - u * w).max() < 10 * (n + 10) * EPS * norm
        assert np.abs(u.T @ u - np.eye(n)).max() < 10 * EPS / 1e-4


# lanes per eigenvalue: 32, 8, 2, 1
@pytest.mark.parametrize("count", [3, 90, 300, 1200])
def test_eigenvalues_of_many_blocks(count):
    rng = np.random.default_rng(count)
    H = [symmetric(rng, 130 if k % 3 else 97, "dense" if k % 5 else "pieces") for k in range(count)]
    e = engine(H)
    e.eigh()
    E, _ = e.eigensystem()
    for h, w in zip(H, E):
        ref = np.linalg.eigvalsh(h)
        assert np.abs(w - ref).max() < 10 * (len(h) + 10) * EPS * np.abs(ref).max()


def pair_setup(rng, dims, is_complex):
    H = []
    for n in dims:
        a = rng.standard_normal((n, n)) + (1j * rng.standard_normal((n, n)) if is_complex else 0)
        H.append((a + a.conj().T) / 2)
    e = engine(H, is_complex)
    e.eigh()
    E, U = e.eigensystem()
    w, _ = e.weights(1.3)
    k = min(dims)
    tgt = np.full(dims[0], -1)
    tgt[:k] = rng.permutation(dims[1])[:k]
    cf = np.where(tgt >= 0, rng.choice([-1.0, 1.0], dims[0]), 0.0)
    op = e.op_define([(0, 1, tgt, cf)])
    e.op_rotate(op)
    C = np.zeros((dims[1], dims[0]))
    C[tgt[tgt >= 0], np.nonzero(tgt >= 0)[0]] = cf[tgt >= 0]
    ref = U[1].conj().T @ C @ U[0]
    # products of K terms of at most one in modulus, K eps each
    assert np.abs(e.op_read(op, 0) - ref).max() < 4 * (max(dims) + 4) * EPS
    return e, E, w, op, e.op_adjoint(op), ref


# Parts of every tile shape in one batch: few tiles of each, which share a
# launch, and many.  Products of K terms of at most one in modulus, K eps each.
@pytest.mark.parametrize("is_complex", [False, True])
@pytest.mark.parametrize("copies", [1, 40])
def test_rotation_of_parts_of_many_sizes(copies, is_complex):
    rng = np.random.default_rng(copies)
    dims = [1, 9, 130, 17, 200, 33, 70, 3, 90] * copies
    H = []
    for n in dims:
        a = rng.standard_normal((n, n)) + (1j * rng.standard_normal((n, n)) if is_complex else 0)
        H.append((a + a.conj().T) / 2)
    e = engine(H, is_complex)
    e.eigh()
    _, U = e.eigensystem()
    acts = []
    for q in range(0, len(dims) - 1):
        tgt = np.full(dims[q], -1)
        k = min(dims[q], dims[q + 1])
        tgt[rng.permutation(dims[q])[:k]] = rng.permutation(dims[q + 1])[:k]
        acts.append((q, q + 1, tgt, np.where(tgt >= 0, rng.choice([-1.0, 0.5], dims[q]), 0.0)))
    op = e.op_define(acts)
    e.op_rotate(op)
    for p, (q, r, tgt, cf) in enumerate(acts):
        C = np.zeros((dims[r], dims[q]))
        C[tgt[tgt >= 0], np.nonzero(tgt >= 0)[0]] = cf[tgt >= 0]
        assert np.abs(e.op_read(op, p) - U[r].conj().T @ C @ U[q]).max() < 4 * (max(dims) + 4) * EPS


# The sums' error is a few eps of the sum of the terms' moduli: ten or so
# rounded operations per term, and up to a thousand additions per partial sum.
@pytest.mark.parametrize("is_complex", [False, True])
@pytest.mark.parametrize("dims", [(1, 1), (3, 5), (17, 31), (70, 45)])
@pytest.mark.parametrize("nz", [1, 2, 5, 31, 33, 129, 300])
def test_pair_sums(dims, nz, is_complex):
    rng = np.random.default_rng(100 * nz + dims[0])
    e, E, w, cd, c, M = pair_setup(rng, dims, is_complex)
    axis = 1j * rng.uniform(0.3, 40, nz)
    off = axis + rng.uniform(-3, 3, nz)
    far = np.where(np.arange(nz) % 2, axis, 1e40j)  # one value out of the shared range
    for z in (axis, off, far):
        every = np.abs(M) ** 2 * (w[0][None, :] + w[1][:, None])
        mid = np.sort(np.append(every, 0.0))[every.size // 2:][:2]  # a threshold between two residues, not one of them
        for tol in (0.0, mid.mean()):
            R = np.where(every > tol, every, 0.0)
            t = R / (z[:, None, None] - (E[1][:, None] - E[0][None, :]))
            got = e.gf(c, cd, [0], [1], z, coef_tol=tol)
            assert np.all(np.abs(got - t.sum((1, 2))) <= 40 * EPS * np.abs(t).sum((1, 2)) + 1e-300)
    # chi: zero poles on the diagonal, z = 0 among the frequencies
    d = e.op_define([(b, b, np.arange(dims[b]), np.arange(1, dims[b] + 1.0)) for b in (0, 1)])
    e.op_rotate(d)
    z = 1j * np.concatenate([[0.0], rng.uniform(0.3, 40, nz)])
    got, zero = e.susc(d, d, [0, 1], [0, 1], z, 1.3, coef_tol=0.0)
    ref, size, w0 = np.zeros(nz + 1, complex), np.zeros(nz + 1), 0.0
    for b in (0, 1):
        A = np.abs(e.op_read(d, b)) ** 2
        P = E[b][None, :] - E[b][:, None]
        near = np.abs(P) < 1e-8
        w0 += (A * w[b][:, None])[near].sum()
        R = np.where(near, 0.0, A * (w[b][:, None] - w[b][None, :]))
        t = -R / (z[:, None, None] - np.where(near, 1.0, P))
        ref += t.sum((1, 2))
        size += np.abs(t).sum((1, 2))
    ref[0] += 1.3 * w0
    assert abs(zero - w0) <= 40 * EPS * w0
    assert np.all(np.abs(got - ref) <= 40 * EPS * (size + 1.3 * w0))


# ---------------------------------------------------------------- G2 and chi3
def small_model(kind):
    from oracle import model as M
    if kind == "complex":
        e = M.CoulombS("A", 2.0, -1.2) + M.CoulombS("B", 2.5, -0.9) + M.CoulombS("C", 1.5, -0.8)
        for a, b, t in (("A", "B", 0.7 * np.exp(0.4j)), ("B", "C", 0.5j), ("C", "A", -0.6)):
            for s in (M.UP, M.DOWN):
                e += M.HoppingS(a, b, t, 0, 0, s, s)
        return M.make_model(e)
    e = M.CoulombS("C", 2.0, -0.7)
    for k, (ek, vk) in enumerate([(-0.7, 0.4), (0.2, 0.3), (0.9, 0.5)]):
        e += M.Level(f"b{k}", ek)
        e += M.Hopping("C", f"b{k}", vk)
    return M.make_model(e)


def freq_list(form, dim, beta, rng):
    """Forms of frequency lists: cubes that hold all, some or none of their
    conjugates, shuffled lists with repeats, general points off the axis."""
    def cube(ns):
        k = np.stack(np.meshgrid(*[np.asarray(n) for n in ns], indexing="ij"), -1).reshape(-1, dim)
        return 1j * np.pi * (2 * k + 1) / beta
    if form == "even":
        return cube([range(-2, 2)] * dim)
    if form == "odd":
        return cube([range(-1, 2)] * dim)
    if form == "above":
        return cube([range(0, 3)] * dim)
    if form == "ragged":
        return cube([range(-3, 2), range(-1, 1), range(0, 4)][:dim])
    if form == "repeats":
        z = cube([range(-2, 2)] * dim)
        z = np.concatenate([z, z[::3], z.conj()[::2], z[5:6], z[5:6].conj()])
        return z[rng.permutation(len(z))]
    if form == "one":
        return cube([[1]] * dim)
    if form == "far":           # values far beyond the others do not blur them
        z = cube([range(-2, 2)] * dim)
        z[::5, 0] = 1e14j
        z[1::7, -1] = -3e13j
        return z
    z = rng.uniform(-2, 2, (40, dim)) + 1j * rng.uniform(0.2, 3, (40, dim)) * rng.choice([-1, 1], (40, dim))
    z[::4] = z[1::4].conj()     # some conjugate pairs
    z[2, 0] = 0.123 + 0.0j      # on the real axis, off every pole
    z[3, :] = z[2, :].conj()
    return z


FORMS = ["even", "odd", "above", "ragged", "repeats", "one", "far", "general"]


# A sum over at most 3e5 quadruples of terms that the resolvents bound: errors
# stay below 1e-12 of the largest value, the bound the other parity tests use.
@pytest.mark.parametrize("kind", ["real", "complex"])
@pytest.mark.parametrize("form", FORMS)
def test_g2_over_forms_of_frequency_lists(form, kind):
    from oracle import ed as EDm
    from oracle import lehmann as L
    from pomerol_b200.pgx import PGX_G2_ANCHORED, PGX_G2_EXACT
    from tests.pgx_harness import GpuED
    m, beta = small_model(kind), 7.0
    lab = "A" if kind == "complex" else "C"
    u, d = m.info.getIndex(lab, 0, 1), m.info.getIndex(lab, 0, 0)
    g, ed = GpuED(m, beta), EDm.ED(m, beta)
    z = freq_list(form, 3, beta, np.random.default_rng(5))
    parts = g.g2_parts(g.c(u), g.c(d), g.cdag(u), g.cdag(d))
    oparts = L.g2_parts(ed, ed.c(u), ed.c(d), ed.cdag(u), ed.cdag(d))
    sel = np.unique(np.linspace(0, len(z) - 1, 24).astype(int))
    ref = L.g2_exact(ed, oparts, [tuple(z[t]) for t in sel])
    exact = g.eng.g2(parts, z, flags=PGX_G2_EXACT)
    anchored = g.eng.g2(parts, z, coef_tol=0.0, flags=PGX_G2_ANCHORED)
    scale = max(np.abs(ref).max(), np.abs(exact).max())
    assert np.abs(exact[sel] - ref).max() < 1e-12 * scale
    assert np.abs(anchored - exact).max() < 1e-12 * scale
    # tiles of the (z1, z3) plane, and one part at a time
    g.eng.set_g2_workspace(0, 1 << 15)
    tiled = g.eng.g2(parts, z, coef_tol=0.0, flags=PGX_G2_ANCHORED)
    assert np.abs(tiled - exact).max() < 1e-12 * scale


# Six balanced digits hold an operand to 254^-6 = 4e-15 of its row's or column's
# largest entry; products along a chain of four operators bring that to no more
# than 1e-9 of the largest value, the bound the other split tests use.
@pytest.mark.parametrize("pair", [False, True])
@pytest.mark.parametrize("kind", ["real", "complex"])
@pytest.mark.parametrize("form", ["even", "odd", "ragged", "far", "general"])
def test_split_g2_over_forms_of_frequency_lists(form, kind, pair):
    from pomerol_b200.pgx import PGX_G2_ANCHORED, PGX_G2_SPLIT_I8
    from tests.pgx_harness import GpuED
    m, beta = small_model(kind), 7.0
    lab = "A" if kind == "complex" else "C"
    u, d = m.info.getIndex(lab, 0, 1), m.info.getIndex(lab, 0, 0)
    g = GpuED(m, beta)
    z = freq_list(form, 3, beta, np.random.default_rng(5))
    parts = g.g2_parts(g.c(u), g.c(d), g.cdag(u), g.cdag(d))
    fp64 = g.eng.g2(parts, z, coef_tol=0.0, flags=PGX_G2_ANCHORED)
    g.eng.set_split_cta_pair(pair)
    g.eng.set_g2_split_threshold(0.0)
    split = g.eng.g2(parts, z, coef_tol=0.0, flags=PGX_G2_ANCHORED | PGX_G2_SPLIT_I8)
    assert np.abs(split - fp64).max() < 1e-9 * np.abs(fp64).max()


def test_exact_g2_on_both_sides_of_its_rule():
    """Scattered triples of one chain of 70 to 126 states: the plane of their
    z1 and z3 holds far more pairs than occur, so the full-matrix form runs;
    a small grid of the same chain goes to the batched form."""
    from pomerol_b200.pgx import PGX_G2_ANCHORED, PGX_G2_EXACT
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
    parts = [(tuple(ops), (0, 1, 2, 3), (0, 1, 2), 1)]
    scattered = 1j * rng.uniform(0.5, 9, (150, 3)) * rng.choice([-1, 1], (150, 3))
    k = 1j * np.pi * (2 * np.arange(-2, 2) + 1) / 2.0
    grid = np.stack(np.meshgrid(k, k, k, indexing="ij"), -1).reshape(-1, 3)
    for z in (scattered, grid):
        a = e.g2(parts, z, flags=PGX_G2_EXACT)
        t = e.g2_timing()
        assert t["total_ms"] > 0 and t["gemm_ms"] > 0 and t["gemm_flops"] > 0
        b = e.g2(parts, z, coef_tol=0.0, flags=PGX_G2_ANCHORED)
        assert np.abs(a - b).max() < 1e-12 * np.abs(a).max()


@pytest.mark.parametrize("kind", ["real", "complex"])
@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("channel", [0, 1, 2])
def test_chi3_over_forms_of_frequency_lists(channel, form, kind):
    from oracle import chi3 as X3
    from oracle import ed as EDm
    from tests.pgx_harness import GpuED
    m, beta = small_model(kind), 7.0
    lab = "A" if kind == "complex" else "C"
    u, d = m.info.getIndex(lab, 0, 1), m.info.getIndex(lab, 0, 0)
    g, ed = GpuED(m, beta), EDm.ED(m, beta)
    z = freq_list(form, 2, beta, np.random.default_rng(6))
    got, _ = g.chi3(channel, (u, u, d, d), z)
    parts = X3.chi3_parts(ed, channel, ed.cdag(u), ed.c(u), ed.cdag(d), ed.c(d))
    sel = np.unique(np.linspace(0, len(z) - 1, 24).astype(int))
    ref = X3.chi3_exact(ed, parts, channel, [tuple(z[t]) for t in sel])
    assert np.abs(got[sel] - ref).max() < 1e-12 * max(1.0, np.abs(ref).max())
