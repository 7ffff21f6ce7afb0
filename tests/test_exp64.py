"""The FP64 exponential as mantissa and exponent, the quotient by kT with its
rest, and the rate of a pair from its factors (kmc_exp64.cuh), compiled for the
host, against exact arithmetic."""
import math
import os
import shutil
import subprocess
from fractions import Fraction

import numpy as np
import pytest

from conftest import REPO
from test_host_threads import CSRC, HERE, _cuda_include, _host_source

mpmath = pytest.importorskip("mpmath")


@pytest.fixture(scope="module")
def exp64(tmp_path_factory):
    if not shutil.which("g++"):
        pytest.skip("no g++")
    folder = tmp_path_factory.mktemp("exp64")
    with open(os.path.join(CSRC, "kmc_exp64.cuh")) as f:
        (folder / "kmc_exp64.cuh").write_text(_host_source(f.read()))
    r = subprocess.run(["g++", "-std=c++20", "-O1", "-ffp-contract=off", "-w", "-pthread", "-I", str(folder), "-I", HERE,
                        "-I", _cuda_include(), os.path.join(HERE, "exp64.cpp"), "-o", str(folder / "exp64")],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]

    def call(function, *columns):
        rec = np.zeros((len(columns[0]), 3))
        for k, c in enumerate(columns):
            rec[:, k] = c
        r = subprocess.run([str(folder / "exp64"), str(function)], input=rec.tobytes(), capture_output=True, check=True)
        return np.frombuffer(r.stdout).reshape(-1, 2)

    return call


def _split_ulps(out, x, y):
    """Error of the mantissas in their last place."""
    worst = 0.0
    with mpmath.workprec(160):
        for (m, k), a, b in zip(out, x, y):
            assert 2.0 ** (-1 / 256) * (1 - 1e-15) <= m < 2.0     # table entry 0 with r < 0: below 1
            exact = mpmath.exp(mpmath.mpf(a) + mpmath.mpf(b)) * mpmath.mpf(2) ** -int(k)
            worst = max(worst, float(abs(mpmath.mpf(m) - exact) / mpmath.mpf(np.spacing(m))))
    return worst


def test_exp_split_is_within_half_an_ulp_and_a_bit(exp64):
    """0.51 units in the last place: half for the last add, the table's and
    the polynomial's (|r|^6/720 of 1 at |r| = ln2/256: 5e-19) below 0.01; an
    argument up to 2^17 is reduced without loss, its correction of up to half
    its last place added."""
    rng = np.random.default_rng(0)
    x = np.concatenate([-708 * rng.random(6000), 40 * rng.standard_normal(4000), rng.uniform(-2.0**17, 2.0**17, 6000),
                        np.arange(-1000, 1000) * math.log(2) / 256, [0.0, -0.0, 5e-324, 1e-20, np.nextafter(2.0**17, 0)]])
    assert np.all(exp64(2, x)[:, 1] == 1)          # splittable
    assert not np.any(exp64(2, [2.0**17, -2.0**17, np.inf, -np.inf, np.nan, 1e300])[:, 1])
    zero = np.zeros_like(x)
    assert _split_ulps(exp64(0, x, zero), x, zero) <= 0.51
    rest = np.where(rng.random(x.size) < 0.5, 1, -1) * rng.random(x.size) * np.spacing(np.abs(x)) / 2
    assert _split_ulps(exp64(0, x, rest), x, rest) <= 0.515


def test_quotient_by_kT_and_its_rest(exp64):
    rng = np.random.default_rng(1)
    x = np.concatenate([rng.standard_normal(4000) * 10.0 ** rng.uniform(-6, 6, 4000), [0.0, 1.0, -3.0]])
    kT = 10.0 ** rng.uniform(-4, 4, x.size)
    kT[:100] = 1.0
    for (y, rest), a, t in zip(exp64(1, x, kT), x, kT):
        exact = Fraction(a) / Fraction(t)
        assert y == float(exact)                   # correctly rounded
        missing = exact - Fraction(y)
        assert abs(Fraction(rest) - missing) <= abs(missing) * Fraction(1, 2**50)


def test_rate_of_factors_over_the_whole_exponent_range(exp64):
    """min(cap, g 2^ex) rounded once: normal and subnormal results and
    factors, exponents beyond either end, pairs without a constant."""
    rng = np.random.default_rng(2)
    n = 6000
    g = (1 + rng.random(n)) * 2.0 ** rng.integers(-60, 8, n)
    g[:1500] = np.ldexp(1 + rng.random(1500), rng.integers(-1074, -1000, 1500))
    g[1500:1600] = 0.0
    ex = np.concatenate([rng.integers(-60, 60, 2000), rng.integers(-1150, -960, 2000), rng.integers(950, 1100, 1000),
                         rng.integers(-10**6, 10**6, 1000)])
    cap = np.where(rng.random(n) < 0.3, np.ldexp(g, rng.integers(-30, 30, n)), 10.0 ** rng.uniform(-320, 300, n))
    cap[1500:1600] = 0.0
    for (r, _), a, e, c in zip(exp64(2, g, ex, cap), g, ex, cap):
        try:
            want = math.ldexp(a, int(e))
        except OverflowError:
            want = math.inf
        assert r == min(c, want)
