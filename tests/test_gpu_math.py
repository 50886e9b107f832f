"""Device functions that stand in for divisions, pow and erff (quotients.cuh, the GELU of act_layout.h), swept on
their own: tests/cpp/math_sweep.cu compares them with the functions they stand in for and with long double."""
import math
import os
import subprocess

import pytest

from gpreempt_b200 import build as gpx_build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _compile(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("math") / "math_sweep")
    res = subprocess.run([gpx_build.nvcc(), *[f for f in gpx_build.NVCC_FLAGS if f != "-lineinfo"],
                          "-I", os.path.join(ROOT, "gpreempt_b200", "csrc"),
                          os.path.join(ROOT, "tests", "cpp", "math_sweep.cu"), "-o", exe], capture_output=True, text=True)
    assert res.returncode == 0, res.stderr
    return exe


def test_sweep_compiles(tmp_path_factory):
    _compile(tmp_path_factory)


@pytest.fixture(scope="module")
def sweep(gpx, tmp_path_factory):
    res = subprocess.run([_compile(tmp_path_factory)], capture_output=True, text=True, timeout=300)
    assert res.returncode == 0, res.stdout
    rows = [line.split() for line in res.stdout.splitlines()]
    return lambda name: [[float(v) for v in r[1:]] for r in rows if r[0] == name]


@pytest.mark.gpu
def test_reciprocals_are_correctly_rounded(sweep):
    """Every mantissa at nine exponents in float; in double within two ulps' product."""
    assert sweep("reciprocal") == [[0.0, 0.0]]


@pytest.mark.gpu
def test_quotients_are_those_of_the_division(sweep):
    """Every float over eight divisors, and 2^32 pairs with extremes among them: bit-identical to the division, except
    that infinities and NaN are the caller's business and a numerator below 2^-100 may miss by one or two in the last place."""
    rows = sweep("numerators")
    assert len(rows) == 16
    for same, left, near, wrong in rows:
        # (of 256 exponents one is infinities and NaN, a divisor of 0.3 overflows over two more, and the residuals
        # of the lowest 24 round to fewer bits: they decide in few of the quotients)
        assert wrong == 0 and left <= 2 ** 32 * 3 / 256 and near <= 2 ** 32 * 4e-3 and same + left + near == 2 ** 32
    (same, left, near, wrong), = sweep("pairs")
    # (24 of 256 exponents overflow over the smallest divisors: 12 on average, and the extremes)
    assert wrong == 0 and left <= 2 ** 32 * 0.15 and near <= 2 ** 32 * 2e-2


@pytest.mark.gpu
def test_power_gives_the_float_pressures_of_pow(sweep):
    rows = sweep("power")
    assert len(rows) == 5
    for mine, cuda, differ in rows:
        assert mine <= 3.2 and differ == 0, (mine, cuda)  # units of 1e-16: an ulp and a half at most
    assert sweep("power_outside") == [[0.0]]


@pytest.mark.gpu
def test_gelu_is_as_accurate_as_the_form_with_erff(sweep):
    rows = sweep("gelu")
    assert len(rows) == 18
    for lo, hi, worst, worst_erff, rms, rms_erff, rel in rows:
        # (an ulp of the smallest results: both forms round the same product there)
        assert worst <= worst_erff * 1.001 + 1e-12 and rms <= rms_erff * 1.001 + 1e-12, (lo, hi)
        if lo >= -6:
            assert rel <= 1e-5, (lo, hi)
    inf, ninf, nan, big, nbig, zero, nzero, tiny, ntiny, edge, nedge = sweep("gelu_odd")[0]
    assert inf == math.inf and abs(ninf) < 1e-30 and math.isnan(nan)
    assert big == pytest.approx(3e38, rel=1e-6) and abs(nbig) < 1e-30 and zero == 0 and nzero == 0
    assert tiny == pytest.approx(5e-41, rel=1e-3) and ntiny == pytest.approx(-5e-41, rel=1e-3)
    assert edge == pytest.approx(1.25 * 0.8943502263331446, rel=2e-7) and nedge == pytest.approx(-1.25 * 0.10564977366685535, rel=1e-6)
