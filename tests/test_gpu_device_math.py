"""The engine's FP64 reciprocal square root and quotient (sph_device.cuh: a hardware seed and one
third-order step) against 80-bit values, over all exponents of normal numbers and random mantissas,
with the largest, the smallest and the powers of two among them.

Bounds, with u = 2^-53 and seeds good to 20 bits (the tests print what they are):
  inv_sqrt   y (1 + e (1/2 + 3/8 e)), e = 1 - x y^2.  x y is rounded, which moves e by u and the
             result by u / 2; the series leaves 5/16 e^3 < u / 50 (e < 2^-19); the last operation
             rounds once.  Half an ulp and 0.53 u: 1.03 ulp at most.
  length_of  x times that: 1.53 u of it and its own rounding, 2.6 u.
  quotient   a times y (1 + e + e^2), e = 1 - b y: the series leaves e^3 < u / 128, two operations
             round: 2.02 u.
Where the seed has no value (0 and below the smallest normal number) neither result is finite:
length_of gives 0 there, and the quotient's NaN is taken as above every limit, so that a ghost
velocity's factor is then its largest."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import PKG, ROOT

pytestmark = pytest.mark.gpu
LD, U = np.longdouble, 2.0 ** -53
INV_SQRT, INV_SQRT_SEED, QUOTIENT, RCP_SEED, LENGTH = range(5)


@pytest.fixture(scope="module")
def ev(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("math") / "libdevice_math.so")
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    subprocess.run([nvcc, "-O3", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a",
                    "--expt-relaxed-constexpr", "-shared", "-Xcompiler", "-fPIC",
                    "-I" + os.path.join(PKG, "csrc"), "-I" + os.path.join(ROOT, "include"),
                    os.path.join(ROOT, "tests", "device_math.cu"), "-o", so], check=True)
    lib = ctypes.CDLL(so)
    P = ctypes.POINTER(ctypes.c_double)

    def call(op, a, b=None):
        a = np.ascontiguousarray(a, dtype=np.float64)
        b = np.ones_like(a) if b is None else np.ascontiguousarray(b, dtype=np.float64)
        out = np.empty_like(a)
        assert lib.eval_host(op, a.ctypes.data_as(P), b.ctypes.data_as(P), out.ctypes.data_as(P),
                             a.size) == 0
        return out

    return call


def _numbers(lo, hi, per=256, seed=0):
    """Positive numbers of binary exponents lo .. hi: random mantissas, 1, the one after it and
    the last."""
    rng = np.random.default_rng(seed)
    e = np.repeat(np.arange(lo, hi + 1), per)
    m = rng.uniform(1.0, 2.0, e.size)
    m[::per], m[1::per], m[2::per] = 1.0, 1.0 + 2.0 ** -52, 2.0 - 2.0 ** -52
    return np.ldexp(m, e)


def _relative(got, want):
    return np.abs((got.astype(LD) - want) / want).astype(float)


def test_inverse_square_root(ev):
    x = _numbers(-1022, 1023)
    want = LD(1) / np.sqrt(x.astype(LD))
    seed = _relative(ev(INV_SQRT_SEED, x), want)
    got = ev(INV_SQRT, x)
    ulp = np.abs((got.astype(LD) - want) / np.spacing(want.astype(np.float64))).astype(float)
    print("inv_sqrt: seed within 2^%.1f, result within %.3f ulp" % (np.log2(seed.max()), ulp.max()))
    assert ulp.max() <= 1.03
    length = _relative(ev(LENGTH, x), np.sqrt(x.astype(LD)))
    print("length_of: within %.3f u" % (length.max() / U))
    assert length.max() <= 2.6 * U


def test_quotient(ev):
    b = _numbers(-1000, 1000, seed=1)
    rng = np.random.default_rng(2)
    b *= rng.choice([-1.0, 1.0], b.size)
    seed = _relative(ev(RCP_SEED, b, b), LD(1) / b.astype(LD))
    # quotients of exponents -20 .. 20, as of two distances near a boundary
    a = np.ldexp(np.frexp(rng.permutation(np.abs(b)))[0], np.frexp(b)[1] + rng.integers(-20, 21, b.size))
    a *= rng.choice([-1.0, 1.0], b.size)
    err = _relative(ev(QUOTIENT, a, b), a.astype(LD) / b.astype(LD))
    print("quotient: seed within 2^%.1f, result within %.3f u" % (np.log2(seed.max()), err.max() / U))
    assert err.max() <= 2.02 * U


def test_arguments_without_a_value(ev):
    tiny = np.array([0.0, 5e-324, 1e-310, np.nextafter(2.0 ** -1022, 0.0)])
    assert not np.isfinite(ev(INV_SQRT, tiny)).any()
    assert np.array_equal(ev(LENGTH, tiny), np.zeros(4))
    assert ev(LENGTH, np.array([2.0 ** -1022]))[0] == 2.0 ** -511
    # a fluid particle on a boundary: 1 + ds / dq has to end at its limit, `b <= max ? b : max`
    for ds in (0.25, -0.25, 0.0, 1e300):
        beta = 1.0 + ev(QUOTIENT, np.full(4, ds), tiny)
        assert not (beta <= 1.5).any()
    beta = 1.0 + ev(QUOTIENT, np.full(2, 0.25), np.array([2.0 ** -1022, 2.0 ** -1000]))
    assert (beta > 1.5).all()
