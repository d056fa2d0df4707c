"""The frequency plans of G2 and chi3: undefined and infinite frequencies among
ordinary ones.  tests/cpp/plan_g2.cpp and plan_chi3.cpp check the
plans themselves without a GPU."""
import subprocess
from pathlib import Path

import numpy as np
import pytest

from tests.test_gpu_kernels import freq_list, small_model

ROOT = Path(__file__).resolve().parents[1]
NAN, INF = float("nan"), float("inf")
ODD = [complex(NAN, NAN), complex(NAN, 1.0), complex(0.0, NAN), complex(0.0, INF), complex(-INF, 1.0)]


@pytest.mark.parametrize("program", ["plan_g2", "plan_chi3"])
def test_plan_of_undefined_frequencies(program, tmp_path):
    exe = tmp_path / program
    r = subprocess.run(["g++", "-O1", "-std=c++17", "-Wall", "-D_GLIBCXX_ASSERTIONS", "-I",
                        str(ROOT / "pomerol_b200" / "csrc"), "-I", "/usr/local/cuda/include",
                        str(ROOT / "tests" / "cpp" / f"{program}.cpp"), "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr


def solved(kind):
    from tests.pgx_harness import GpuED
    m = small_model(kind)
    g = GpuED(m, 7.0)
    lab = "A" if kind == "complex" else "C"
    return g, m.info.getIndex(lab, 0, 1), m.info.getIndex(lab, 0, 0)


def with_odd_values(z, place, rng):
    """Some entries of one place undefined or infinite, and the rows left alone."""
    y = z.copy()
    rows = rng.permutation(len(z))[:max(1, len(z) // 5)]
    for i, t in enumerate(rows):
        y[t, place] = ODD[i % len(ODD)]
        if i % 3 == 0:
            y[t, (place + 1) % z.shape[1]] = ODD[(i + 1) % len(ODD)]
    return y, np.setdiff1d(np.arange(len(z)), rows)


# Rounding: the other rows' sums are the same ones, in another order (1e-12 of
# the largest value, 1e-9 with split products, the bounds of the parity tests).
@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["real", "complex"])
@pytest.mark.parametrize("form", ["even", "odd", "general"])
@pytest.mark.parametrize("place", [0, 1, 2])
def test_g2_beside_undefined_frequencies(place, form, kind):
    from pomerol_b200.pgx import PGX_G2_ANCHORED, PGX_G2_EXACT, PGX_G2_SPLIT_I8
    g, u, d = solved(kind)
    z = freq_list(form, 3, 7.0, np.random.default_rng(5))
    y, keep = with_odd_values(z, place, np.random.default_rng(place))
    parts = g.g2_parts(g.c(u), g.c(d), g.cdag(u), g.cdag(d))
    g.eng.set_g2_split_threshold(0.0)
    for flags, tol in ((PGX_G2_EXACT, 1e-12), (PGX_G2_ANCHORED, 1e-12), (PGX_G2_ANCHORED | PGX_G2_SPLIT_I8, 1e-9)):
        ref = g.eng.g2(parts, z, coef_tol=0.0, flags=flags)
        got = g.eng.g2(parts, y, coef_tol=0.0, flags=flags)
        assert np.abs(got[keep] - ref[keep]).max() < tol * np.abs(ref).max()
    g.eng.set_g2_workspace(0, 1 << 15)  # tiles of the (z1, z3) plane
    got = g.eng.g2(parts, y, coef_tol=0.0, flags=PGX_G2_ANCHORED)
    assert np.abs(got[keep] - ref[keep]).max() < 1e-9 * np.abs(ref).max()


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["real", "complex"])
@pytest.mark.parametrize("form", ["even", "odd", "general"])
@pytest.mark.parametrize("channel", [0, 1, 2])
def test_chi3_beside_undefined_frequencies(channel, form, kind):
    g, u, d = solved(kind)
    z = freq_list(form, 2, 7.0, np.random.default_rng(6))
    for place in (0, 1):
        y, keep = with_odd_values(z, place, np.random.default_rng(place))
        ref, _ = g.chi3(channel, (u, u, d, d), z)
        got, _ = g.chi3(channel, (u, u, d, d), y)
        assert np.abs(got[keep] - ref[keep]).max() < 1e-12 * np.abs(ref).max()
