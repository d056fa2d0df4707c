"""Pair sums beside undefined and infinite frequencies."""
import numpy as np
import pytest

from oracle import lehmann as L
from tests.test_g2_plans import ODD, solved

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["real", "complex"])
def test_sums_at_undefined_frequencies(kind):
    """A sum without terms is zero at any frequency; with terms the other
    frequencies keep their values to rounding (40 eps of the terms' moduli, here
    of sums of at most one in modulus over |z| >= 0.4)."""
    g, u, _ = solved(kind)
    c, cd = g.c(u), g.cdag(u)
    z = np.concatenate([L.fermionic(np.arange(40), 7.0), 0.3 + 0.2j * np.arange(1, 20)])
    y = z.copy()
    odd = np.arange(3, len(z), 5)
    y[odd] = [ODD[i % len(ODD)] for i in range(len(odd))]
    assert np.all(g.gf(c, cd, y, coef_tol=10.0) == 0.0)
    keep = np.setdiff1d(np.arange(len(z)), odd)
    ref, got = g.gf(c, cd, z, coef_tol=0.0), g.gf(c, cd, y, coef_tol=0.0)
    assert np.abs(got[keep] - ref[keep]).max() < 40 * np.finfo(float).eps / 0.2
    assert not np.isfinite(got[odd]).any()
