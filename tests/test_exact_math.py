"""Integer-pipe division and square root and the FP32 forms of the float solver's double expressions
(csrc/exact_math.cuh), compiled for the host and compared bit for bit with the processor's correctly rounded
IEEE operations, on operands of the whole range with the special values and the hard cases (significands of
few and of nearly all ones, results next to half-way points) among them."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "shll-sve-cfd_gb300")
CUDA = os.path.dirname(os.path.dirname(os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")))

SOURCE = r"""
#include "exact_math.cuh"
using namespace exact_math;
typedef double D;
extern "C" {
#define LOOP for (long i = 0; i < n; i++)
void t_divide(const D* a, const D* b, D* o, long n) { LOOP o[i] = divide(a[i], divisor(b[i])); }
void t_divide_plain(const D* a, const D* b, D* o, long n) { LOOP o[i] = divide_plain(a[i], divisor(b[i])); }
void t_sqrt(const D* a, D* o, long n) { LOOP o[i] = square_root(a[i]); }
// a / sqrt(b) with the root's reciprocal as it comes from the root
void t_root_divisor(const D* a, const D* b, D* o, long n) { LOOP { Divisor r; square_root_plain(b[i], &r); o[i] = divide_plain(a[i], r); } }
void t_scale(const D* a, D* o, long n, int k, D p) { LOOP o[i] = scale_pow2(a[i], k, p); }
void t_minmod(const D* l, const D* r, D* o, long n) {
    LOOP { bool s = false; const D m = minmod_plain(l[i], r[i], &s); o[i] = s ? minmod_general(l[i], r[i], 1.0) : m; }
}
void t_fdivide(const float* a, const float* b, float* o, long n) {
    LOOP o[i] = divide_plain(a[i], b[i], reciprocal_plain(b[i], em_rcp(b[i])));
}
void t_fsqrt(const float* a, float* o, long n) { LOOP { float y; o[i] = square_root_plain(a[i], &y); } }
void t_temperature(const float* e, const float* p, float* o, long n, float c) {
    LOOP { const float kh = p[i] * p[i]; o[i] = temperature_ref(e[i], 0.5f * kh, 0.5f * fmaf(p[i], p[i], -kh), c, 1.0f / c); }
}
void t_z2(const float* a, const float* t, float* o, long n) { LOOP o[i] = z2_ref(a[i], t[i]); }
void t_sub_product(const float* u, const float* s, float* o, long n, float c) { LOOP o[i] = sub_product_ref(u[i], c, s[i]); }
}
"""


@pytest.fixture(scope="module")
def em(tmp_path_factory):
    d = tmp_path_factory.mktemp("exact_math")
    (d / "t.cpp").write_text(SOURCE)
    so = str(d / "t.so")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-I", os.path.join(PKG, "csrc"),
                    "-I", os.path.join(CUDA, "include"), str(d / "t.cpp"), "-o", so], check=True)
    return ctypes.CDLL(so)


def call(f, *arrays, extra=()):
    out = np.empty_like(arrays[0])
    p = ctypes.c_void_p
    f(*[p(a.ctypes.data) for a in arrays], p(out.ctypes.data), ctypes.c_long(out.size), *extra)
    return out


def same(a, b):
    """the same bits, any NaN for a NaN"""
    i = np.uint64 if a.dtype == np.float64 else np.uint32
    return np.all((a.view(i) == b.view(i)) | (np.isnan(a) & np.isnan(b)))


def doubles(rng, n, lo, hi):
    """signed values of exponents lo..hi, a third each with random, sparse and nearly full significands"""
    m = rng.integers(0, 1 << 52, n, dtype=np.uint64)
    few = np.uint64(1) << rng.integers(0, 52, n, dtype=np.uint64)
    kind = rng.integers(0, 3, n)
    m = np.where(kind == 1, few, np.where(kind == 2, np.uint64((1 << 52) - 1) ^ few, m))
    e = rng.integers(lo + 1023, hi + 1024, n).astype(np.uint64)
    return (m | (e << np.uint64(52)) | (rng.integers(0, 2, n).astype(np.uint64) << np.uint64(63))).view(np.float64)


def floats(rng, n, lo, hi):
    m = rng.integers(0, 1 << 23, n, dtype=np.uint32)
    few = np.uint32(1) << rng.integers(0, 23, n, dtype=np.uint32)
    kind = rng.integers(0, 3, n)
    m = np.where(kind == 1, few, np.where(kind == 2, np.uint32((1 << 23) - 1) ^ few, m)).astype(np.uint32)
    return (m | (rng.integers(lo + 127, hi + 128, n).astype(np.uint32) << np.uint32(23))).view(np.float32)


SPECIAL = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, -5e-324, 2.2250738585072014e-308, 2.225073858507201e-308,
                    1.7976931348623157e308, 1.0, -1.0, 3.0, 0.1])
N = 400000


@pytest.fixture(autouse=True)
def quiet():
    with np.errstate(all="ignore"):
        yield


def test_division(em):
    rng = np.random.default_rng(1)
    a, b = doubles(rng, N, -1022, 1023), doubles(rng, N, -1022, 1023)
    s, t = [x.ravel().copy() for x in np.meshgrid(SPECIAL, SPECIAL)]
    sub = (a / 2.0**1000) / 2.0**60   # subnormals among them
    for x, y in ((a, b), (s, t), (sub, b), (b, sub), (a, np.full(N, 2.5))):
        assert same(call(em.t_divide, x, y), x / y)
    a, b = doubles(rng, N, -400, 400), np.abs(doubles(rng, N, -400, 400))
    assert same(call(em.t_divide_plain, a, b), a / b)
    # quotients next to half-way points: a = b (q + half an ulp), rounded either way
    q = 1.0 + rng.integers(0, 1 << 52, N) * 2.0**-52
    a = b * q
    for x in (a, np.nextafter(a, np.inf), np.nextafter(a, 0), b, np.nextafter(b, np.inf)):
        assert same(call(em.t_divide_plain, x, b), x / b)


def test_square_root(em):
    rng = np.random.default_rng(2)
    a = np.abs(doubles(rng, N, -1022, 1023))
    assert same(call(em.t_sqrt, a), np.sqrt(a))
    assert same(call(em.t_sqrt, SPECIAL), np.sqrt(SPECIAL))
    r = np.abs(doubles(rng, N, -500, 500))
    for x in (r * r, np.nextafter(r * r, np.inf), np.nextafter(r * r, 0)):   # next to exact squares
        assert same(call(em.t_sqrt, x), np.sqrt(x))
    m, x = doubles(rng, N, -300, 300), np.abs(doubles(rng, N, -600, 600))
    assert same(call(em.t_root_divisor, m, x), m / np.sqrt(x))


@pytest.mark.parametrize("k", [-1, 1, -2])
def test_scaling(em, k):
    a = np.concatenate([doubles(np.random.default_rng(3), N, -1022, 1023), SPECIAL])
    assert same(call(em.t_scale, a, extra=(ctypes.c_int(k), ctypes.c_double(2.0**k))), a * 2.0**k)


def test_minmod(em):
    rng = np.random.default_rng(4)
    l, r = doubles(rng, N, -1022, 1023), doubles(rng, N, -1022, 1023)
    l2, r2 = doubles(rng, N, -540, -500), doubles(rng, N, -580, -500)   # products that underflow
    s, t = [x.ravel().copy() for x in np.meshgrid(SPECIAL, SPECIAL)]
    for x, y in ((l, r), (l2, r2), (s, t), (l, l.copy()), (l, -l)):
        ref = np.where(x * y < 0.0, 0.0, np.where(np.abs(x) < np.abs(y), x, y))
        assert same(call(em.t_minmod, x, y), ref)


def test_float_division_and_root(em):
    rng = np.random.default_rng(5)
    a, b = floats(rng, N, -30, 30), floats(rng, N, -30, 30)
    b = np.where(b.view(np.uint32) & 0x7FFFFF == 0x7FFFFF, np.float32(1.5), b)   # (the residual step's exception)
    assert same(call(em.t_fdivide, a, b), a / b)
    assert same(call(em.t_fdivide, np.zeros(N, np.float32), b), np.zeros(N, np.float32))
    assert same(call(em.t_fsqrt, a), np.sqrt(a))


def test_float_expressions(em):
    """against the double expressions that they stand for, rounded to float"""
    rng = np.random.default_rng(6)
    d = np.float64
    for c in (2.5, 3.0, 1.7):
        c = np.float32(c)
        p = floats(rng, N, -8, 6) * np.where(rng.integers(0, 2, N), 1, -1).astype(np.float32)
        for e in (floats(rng, N, -4, 8), (d(0.5) * d(p) * d(p) * (1 + rng.uniform(0, 1e-4, N))).astype(np.float32)):
            ref = ((d(e) - 0.5 * d(p) * d(p)) / d(c)).astype(np.float32)
            assert same(call(em.t_temperature, e, p, extra=(ctypes.c_float(c),)), ref)
    a, t = floats(rng, N, -10, 10), np.concatenate([rng.uniform(0, 3, N // 2), 1 + rng.uniform(-1e-3, 1e-3, N // 2)]).astype(np.float32)
    assert same(call(em.t_z2, a, t), (0.5 * d(a) * (1.0 - d(t))).astype(np.float32))
    for c in (0.125, 0.0625, 0.1, 0.3):
        c = np.float32(c)
        u, s = floats(rng, N, -10, 10), floats(rng, N, -40, 10) * np.where(rng.integers(0, 2, N), 1, -1).astype(np.float32)
        for x in (u, (d(c) * d(s) * (1 + rng.uniform(-1e-6, 1e-6, N))).astype(np.float32)):
            ref = (d(x) - d(c) * d(s)).astype(np.float32)
            assert same(call(em.t_sub_product, x, s, extra=(ctypes.c_float(c),)), ref)
