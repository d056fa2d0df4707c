"""The eigensolver at the limits of its cluster sizes and lane counts, and its
large-block launches, each started while the one before drains, under capture."""
import numpy as np
import pytest

from tests.test_gpu_kernels import EPS, engine, symmetric

pytestmark = pytest.mark.gpu


def check(H, E, U):
    """Backward error of a few n eps ||H||; vectors of eigenvalues further apart
    than 1e-4 ||H|| are orthogonal to eps / 1e-4."""
    for h, w, u in zip(H, E, U):
        n, ref = len(h), np.linalg.eigvalsh(h)
        norm = max(1.0, np.abs(ref).max())
        assert np.all(np.diff(w) >= 0)
        assert np.abs(w - ref).max() < 10 * (n + 10) * EPS * norm
        assert np.abs(h @ u - u * w).max() < 10 * (n + 10) * EPS * norm
        assert np.abs(u.T @ u - np.eye(n)).max() < 10 * EPS / 1e-4


# the largest block of 1, 2, 4 and 8 CTAs and the next, which takes the next cluster size
@pytest.mark.parametrize("kind", ["dense", "pieces"])
@pytest.mark.parametrize("dims", [[166, 167], [233, 234], [325, 326], [452, 453, 464],
                                  [513, 452, 325, 233, 166, 1]])
def test_limits_of_the_cluster_sizes(dims, kind):
    rng = np.random.default_rng(sum(dims))
    H = [symmetric(rng, n, kind) for n in dims]
    e = engine(H)
    e.eigh()
    check(H, *e.eigensystem())


# eigenvalues in all: 4760 and 9450 (16 lanes each), 18900 (8), 37800 (4), 59500 (2)
@pytest.mark.parametrize("n,count", [(119, 40), (105, 90), (105, 180), (105, 360), (119, 500)])
def test_eigenvalues_at_every_lane_count(n, count):
    rng = np.random.default_rng(count)
    H = [symmetric(rng, n, "dense" if k % 5 else "pieces") for k in range(count)]
    e = engine(H)
    e.eigh()
    for h, w in zip(H, e.eigensystem()[0]):
        ref = np.linalg.eigvalsh(h)
        assert np.abs(w - ref).max() < 10 * (n + 10) * EPS * np.abs(ref).max()


# The reduction's products grow with the square of the matrix, which stays in
# range between 1e-135 and 1e150; its third power does not.
@pytest.mark.parametrize("scale", [1e-130, 1e-105, 1e120, 1e150])
@pytest.mark.parametrize("dims", [[600, 520, 200, 40], [1130] * 10])
def test_matrices_of_any_scale(dims, scale):
    rng = np.random.default_rng(sum(dims))
    H = [symmetric(rng, n) for n in dims]
    e = engine([h * scale for h in H])
    e.eigh()
    E, U = e.eigensystem()
    check(H, [w / scale for w in E], U)


# above 513 states, and above 100 MB of matrices (one triangle read) down to below it
@pytest.mark.parametrize("dims", [[600, 520, 40], [1130] * 10])
def test_captured_large_blocks(dims):
    rng = np.random.default_rng(sum(dims))
    H = [symmetric(rng, n) for n in dims]
    e = engine(H)
    e.eigh()
    e.graph_begin()
    e.eigh()
    gid = e.graph_end()
    for _ in range(2):
        H = [symmetric(rng, n) for n in dims]
        e.set_hamiltonian(H)
        e.graph_replay(gid)
        check(H, *e.eigensystem())
    e.graph_destroy(gid)
