"""The shortened division and arctangent of the weight generation
(helm-project_gb300/csrc/geom.cuh) against the full operations, on random
operands and on both sides of every line between the short and the full form."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "helm-project_gb300", "csrc")


@pytest.fixture(scope="module")
def geom(gpu, tmp_path_factory):
    nvcc = shutil.which("nvcc") or os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    out = str(tmp_path_factory.mktemp("geom") / "libgeom.so")
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++20", "--fmad=false", "-shared",
                    "-Xcompiler", "-fPIC", "-I", CSRC, os.path.join(HERE, "native", "geom_harness.cu"), "-o", out], check=True)
    lib = C.CDLL(out)

    def run(a, b, what):
        a, b = (np.ascontiguousarray(v, np.float64) for v in np.broadcast_arrays(a, b))
        r = np.empty_like(a)
        assert lib.geom_eval(*(v.ctypes.data_as(C.c_void_p) for v in (a, b, r)), a.size, what) == 0
        return a, b, r

    return run


def _around(values, steps=3):
    """The values and their neighbours, a few ulps to either side."""
    out = []
    for v in values:
        lo = hi = np.float64(v)
        out.append(lo)
        for _ in range(steps):
            lo, hi = np.nextafter(lo, -np.inf), np.nextafter(hi, np.inf)
            out += [lo, hi]
    return np.array(out)


def test_division_by_a_reciprocal_is_correctly_rounded(geom):
    """Bit for bit IEEE division: mantissas of every kind, exponents on both sides of
    2^+-500 and far outside, zeros, infinities and NaN."""
    rng = np.random.default_rng(1)
    n = 1_000_000
    m = 1.0 + rng.random(n)
    m[: n // 4] = _around([1.0, 1.5, 2.0 - 2.0**-52])[rng.integers(0, 21, n // 4)]
    ea = rng.choice([-1000, -501, -500, -499, -1, 0, 1, 499, 500, 501, 1000], n) + rng.integers(-2, 3, n)
    a = np.ldexp(m, ea) * rng.choice([-1.0, 1.0], n)
    b = np.ldexp(m[rng.permutation(n)], ea[rng.permutation(n)])
    edge = np.concatenate([_around([2.0**-500, 2.0**500, 1.0, 3.0]), [0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, 1.7e308]])
    a = np.concatenate([a, np.repeat(edge, len(edge)), rng.random(n)])
    b = np.concatenate([b, np.tile(edge, len(edge)), rng.random(n) * 1e-4])
    a, b, r = geom(a, b, 0)
    with np.errstate(all="ignore"):
        want = a / b
    assert np.array_equal(r, want, equal_nan=True)
    assert np.array_equal(np.signbit(r[~np.isnan(want)]), np.signbit(want[~np.isnan(want)]))


def test_twice_the_arctangent(geom):
    """2 atan2(num, den). The series' error: the quotient's (one ulp), the next term
    (2^-73) and the last addition's (half an ulp); CUDA's atan2 is within 2 ulp and
    the host's within 1, doubling is exact: 3 ulp in all."""
    rng = np.random.default_rng(2)
    n = 500_000
    den = np.concatenate([rng.uniform(0.4, 17.0, n), rng.choice(_around([0.5, 1.0, 4.0, 8.0, 16.0]), n),
                          rng.uniform(-2.0, 0.5, n // 5)])
    t = np.concatenate([2.0 ** rng.uniform(-60, -5, n), rng.choice(_around([2.0**-7, 2.0**-8, 2.0**-6]), n),
                        2.0 ** rng.uniform(-20, 3, n // 5)]) * rng.choice([-1.0, 1.0], den.size)
    num, den, r = geom(t * np.abs(den), den, 1)
    want = 2.0 * np.arctan2(num, den)
    assert np.all(np.abs(r - want) <= 3.0 * np.spacing(np.abs(want)))
    zero = geom(np.array([0.0, -0.0]), np.array([4.0, 4.0]), 1)[2]
    assert np.all(zero == 0.0)
