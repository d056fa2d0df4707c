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
                                  [1273, 1274, 600], [3] * 400, [7, 5] * 150])
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
