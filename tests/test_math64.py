"""
The functions of the double precision kernels (csrc/mkg_math64.h, integer
arithmetic) compiled for the host: division and square root equal to the
processor's bit for bit, exp, log, powers and roots of cubics within 0.6
units in the last place of the result in longer arithmetic, also at the
edges of the ranges and where the library's function takes over. The
device's approximations (some units in the last place) are taken as exact,
low and high.
"""
import ctypes
import os
import subprocess

import numpy as np
import pytest

import myokit_gb300
from myokit_gb300 import exporter

CSRC = os.path.join(os.path.dirname(myokit_gb300.__file__), 'csrc')

HOST = r'''
#include <cmath>
#include <cstring>
typedef unsigned int mkg_u32;
typedef unsigned long long mkg_u64;
#define __device__
@TABLE@
#define MKG_M64 static inline
#define MKG_M64_SLOW static inline
#define MKG_M64_FN static inline
static int ulp = 0;
MKG_M64 mkg_u32 mkg_mulhi(mkg_u32 a, mkg_u32 b)
{ return (mkg_u32)(((mkg_u64)a * b) >> 32); }
MKG_M64 mkg_u32 mkg_shl(mkg_u32 lo, mkg_u32 hi, mkg_u32 s)
{ return s ? (hi << s) | (lo >> (32 - s)) : hi; }
MKG_M64 mkg_u32 mkg_shr(mkg_u32 lo, mkg_u32 hi, mkg_u32 s)
{ return s ? (lo >> s) | (hi << (32 - s)) : lo; }
MKG_M64 mkg_u32 mkg_rcp_bits(mkg_u32 b)
{
    float x; memcpy(&x, &b, 4);
    float y = 1.0f / x; mkg_u32 r; memcpy(&r, &y, 4);
    r += ulp;
    return r < 0x3f000000u ? 0x3f000000u : r;
}
MKG_M64 mkg_u64 bits(double x) { mkg_u64 u; memcpy(&u, &x, 8); return u; }
MKG_M64 mkg_u32 mkg_hi(double x) { return (mkg_u32)(bits(x) >> 32); }
MKG_M64 mkg_u32 mkg_lo(double x) { return (mkg_u32)bits(x); }
MKG_M64 double mkg_make(mkg_u32 h, mkg_u32 l)
{ mkg_u64 u = ((mkg_u64)h << 32) | l; double d; memcpy(&d, &u, 8); return d; }
MKG_M64 mkg_u64 mkg_exp_entry(mkg_u32 j)
{ return j < sizeof(mkg_exp_tab) / 8 ? mkg_exp_tab[j] : 0; }
MKG_M64 mkg_u64 mkg_log_entry(int k, mkg_u32 j)
{ return j < 256 ? mkg_log_tab[2 * j + k] : 0; }
MKG_M64 mkg_u32 mkg_clz(mkg_u32 x) { return x ? __builtin_clz(x) : 32; }
static float off(float y, int n)
{ mkg_u32 u; memcpy(&u, &y, 4); u += n; memcpy(&y, &u, 4); return y; }
MKG_M64 mkg_u32 mkg_rsqrt_fixed(mkg_u32 b)
{
    float x; memcpy(&x, &b, 4);
    return (mkg_u32)(off((float)(1 / std::sqrt((double)x)), 2 * ulp) *
                     2147483648.0f);
}
MKG_M64 mkg_u64 mkg_cos_third_start(long long z)
{
    float c = std::cos(std::acos((float)(int)(z >> 32) * 1.862645149e-9f) *
                       0.33333334f);
    c = std::fmin(off(c, 4 * ulp), 1.0f);
    return (mkg_u64)(mkg_u32)(c * 2147483648.0f) << 32;
}
MKG_M64 mkg_u32 mkg_slope_inverse(mkg_u32 c2)
{
    return (mkg_u32)(off(1 / ((float)(int)(c2 - 0x10000000u) *
                              1.117587090e-8f), ulp) * 268435456.0f);
}
#include "mkg_math64.h"
extern "C" void divide(const double *a, const double *b, double *q, long n,
                       int u)
{ ulp = u; for (long i = 0; i < n; ++i) q[i] = mkg_div(a[i], b[i]); }
extern "C" void divide_by(const double *a, double b, unsigned y, double *q,
                          long n)
{ for (long i = 0; i < n; ++i) q[i] = mkg_div_by(a[i], b, y); }
extern "C" void roots(const double *x, double *y, long n, int u)
{ ulp = u; for (long i = 0; i < n; ++i) y[i] = mkg_sqrt(x[i]); }
static double units(double y, long double e)
{
    return (double)(fabsl((long double)y - e) /
                    ldexpl(1.0L, ilogbl(e) - 52));
}
extern "C" void exps(const double *x, double *y, double *ulps, long n)
{
    for (long i = 0; i < n; ++i) {
        y[i] = mkg_exp(x[i]);
        ulps[i] = units(y[i], expl((long double)x[i]));
    }
}
extern "C" void logs(const double *x, double *y, double *ulps, long n)
{
    for (long i = 0; i < n; ++i) {
        y[i] = mkg_log(x[i]);
        ulps[i] = units(y[i], logl((long double)x[i]));
    }
}
extern "C" void powers(const double *x, double p, mkg_u64 P, double *y,
                       double *ulps, long n)
{
    for (long i = 0; i < n; ++i) {
        y[i] = mkg_pow_literal(x[i], p, P, p < 0 ? ~0u : 0u);
        ulps[i] = units(y[i], powl((long double)x[i], (long double)p));
    }
}
extern "C" void thirds(const double *z, double *y, double *ulps, long n,
                       int u)
{
    ulp = u;
    for (long i = 0; i < n; ++i) {
        y[i] = mkg_cos_third(z[i]);
        ulps[i] = units(y[i], cosl(acosl((long double)z[i]) / 3));
    }
}
'''


@pytest.fixture(scope='module')
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp('math64')
    src = d / 'm.cpp'
    src.write_text(HOST.replace('@TABLE@', exporter._math_tables()))
    so = d / 'm.so'
    subprocess.run(['g++', '-O2', '-shared', '-fPIC', '-ffp-contract=off',
                    '-I', CSRC, '-o', str(so), str(src)], check=True)
    return ctypes.CDLL(str(so))


def _ptr(a):
    return a.ctypes.data_as(ctypes.c_void_p)


def _doubles(rng, n, spread):
    """Random significands (some short, some all ones), exponents within
    ``spread`` of 0 and random signs."""
    m = rng.integers(0, 1 << 52, n, dtype=np.uint64)
    k = n // 8
    m[:k] &= np.uint64(0xfffff00000000)
    m[k:2 * k] |= np.uint64(0xfffffffff0000)
    m[2 * k:3 * k] = rng.integers(0, 4, k)
    e = (rng.integers(-spread, spread + 1, n) + 1023).astype(np.uint64)
    s = rng.integers(0, 2, n, dtype=np.uint64)
    x = (m | (e << np.uint64(52)) | (s << np.uint64(63))).view(np.float64)
    return rng.permutation(x)


@pytest.mark.parametrize('ulp', [-1, 0, 1])
@pytest.mark.parametrize('spread', [3, 60, 1022])
def test_division_is_correctly_rounded(lib, ulp, spread):
    rng = np.random.default_rng(spread + ulp)
    n = 400000
    a, b = _doubles(rng, n, spread), _doubles(rng, n, spread)
    edge = np.array([0.0, -0.0, 1.0, -3.0, np.inf, -np.inf, np.nan, 5e-324,
                     1e-310, 2.3e-308, 1.7e308])
    a[:121], b[:121] = np.repeat(edge, 11), np.tile(edge, 11)
    q = np.empty(n)
    lib.divide(_ptr(a), _ptr(b), _ptr(q), ctypes.c_long(n), ulp)
    with np.errstate(all='ignore'):
        r = a / b
    same = (q.view(np.uint64) == r.view(np.uint64)) | (
        np.isnan(q) & np.isnan(r))
    assert same.all(), (a[~same][:3], b[~same][:3])


@pytest.mark.parametrize('b', [1.0, -6.8, 5.98, 10.0, 1 / 3, 4.0,
                               1.9999999999999998, 2.0 ** -1022])
def test_division_by_a_literal(lib, b):
    y = exporter._reciprocal_digits(b)
    a = _doubles(np.random.default_rng(1), 200000, 40)
    q = np.empty(len(a))
    lib.divide_by(_ptr(a), ctypes.c_double(b), ctypes.c_uint(y), _ptr(q),
                  ctypes.c_long(len(a)))
    with np.errstate(all='ignore'):
        assert np.array_equal(q.view(np.uint64), (a / b).view(np.uint64))


def test_division_by_literals_without_digits():
    assert [exporter._reciprocal_digits(x) for x in (
        0.0, np.inf, np.nan, 1e-310)] == [None] * 4


@pytest.mark.parametrize('size', [1e-17, 1e-12, 1e-6, 2e-3, 0.1, 1.0, 5.0,
                                  40.0, 708.0])
def test_exp(lib, size):
    rng = np.random.default_rng(int(size * 1e6) % 1000)
    x = rng.uniform(-size, size, 300000)
    # Around the multiples of ln(2) (and 1/256), where k and j change
    k = np.arange(-60, 61)
    x[:121] = k * np.log(2)
    x[121:242] = np.nextafter(k / 256, 1)
    y, u = np.empty(len(x)), np.empty(len(x))
    lib.exps(_ptr(x), _ptr(y), _ptr(u), ctypes.c_long(len(x)))
    assert u.max() < 0.57


def test_exp_outside_the_fast_range(lib):
    x = np.array([0.0, -0.0, 1e-300, 5e-17, 708.0, 709.7, 710.0, -708.5,
                  -745.0, -746.0, np.inf, -np.inf, np.nan])
    y, u = np.empty(len(x)), np.empty(len(x))
    lib.exps(_ptr(x), _ptr(y), _ptr(u), ctypes.c_long(len(x)))
    with np.errstate(all='ignore'):
        r = np.exp(x)
    assert np.array_equal(np.isnan(y), np.isnan(r))
    assert np.array_equal(np.isinf(y), np.isinf(r))
    ok = np.isfinite(r)
    assert np.all(np.abs(y[ok] - r[ok]) <= np.spacing(r[ok]))


@pytest.mark.parametrize('ulp', [-1, 0, 1])
@pytest.mark.parametrize('spread', [2, 60, 1022])
def test_square_root_is_correctly_rounded(lib, ulp, spread):
    rng = np.random.default_rng(7 * spread + ulp)
    x = np.abs(_doubles(rng, 400000, spread))
    # Squares of numbers with few bits, and their neighbours
    k = np.arange(1, 50001, dtype=float) ** 2
    x[:50000], x[50000:100000] = k, np.nextafter(k, 0)
    x[100000:150000] = np.nextafter(k, np.inf)
    x[150000:150010] = [0.0, -0.0, np.inf, np.nan, 5e-324, 1e-310, 1.7e308,
                        -1.0, np.nextafter(4, 0), 2.0 ** -1022]
    y = np.empty(len(x))
    lib.roots(_ptr(x), _ptr(y), ctypes.c_long(len(x)), ulp)
    with np.errstate(all='ignore'):
        r = np.sqrt(x)
    same = (y.view(np.uint64) == r.view(np.uint64)) | (
        np.isnan(y) & np.isnan(r))
    assert same.all(), x[~same][:3]


@pytest.mark.parametrize('size', [1e-4, 0.01, 0.3, 3.0, 20.0, 700.0])
def test_log(lib, size):
    rng = np.random.default_rng(int(size * 1e4))
    x = np.exp(rng.uniform(-size, size, 300000))
    # Where the leading bits, the exponent or the branch change
    e = np.concatenate([1 + np.arange(256) / 256, 2.0 ** np.arange(-40, 41),
                        np.exp([-2.0 ** -7, 2.0 ** -7])])
    e = np.concatenate([e, np.nextafter(e, 0), np.nextafter(e, 9e99)])
    x[:len(e)] = e
    x = x[x != 1]
    y, u = np.empty(len(x)), np.empty(len(x))
    lib.logs(_ptr(x), _ptr(y), _ptr(u), ctypes.c_long(len(x)))
    assert u.max() < 0.6


@pytest.mark.parametrize('p', [1.4, -1.4, 0.7, 2.5, 1 / 3, 2.0 ** -8, -3.7,
                               15.999999999999998])
def test_literal_power(lib, p):
    rng = np.random.default_rng(int(abs(p) * 100))
    x = np.exp(rng.uniform(-1, 1, 200000) * rng.choice([1e-3, 1, 30], 200000))
    y, u = np.empty(len(x)), np.empty(len(x))
    lib.powers(_ptr(x), ctypes.c_double(p), ctypes.c_ulonglong(
        int(abs(p) * 2 ** 60)), _ptr(y), _ptr(u), ctypes.c_long(len(x)))
    assert u.max() < 0.6
    x = np.array([0.0, 1.0, np.inf, np.nan, -2.0, 1e-310, 1e300, 1e-300,
                  5e-324])
    y, u = np.empty(len(x)), np.empty(len(x))
    lib.powers(_ptr(x), ctypes.c_double(p), ctypes.c_ulonglong(
        int(abs(p) * 2 ** 60)), _ptr(y), _ptr(u), ctypes.c_long(len(x)))
    with np.errstate(all='ignore'):
        r = x ** p
        ok = (y == r) | (np.isnan(y) & np.isnan(r)) | (
            np.abs(y - r) <= 1e-15 * np.abs(r))
    assert ok.all(), (x[~ok], y[~ok], r[~ok])


@pytest.mark.parametrize('ulp', [-1, 0, 1])
@pytest.mark.parametrize('a,b', [(-0.9995, 1.0), (-0.99951, -0.999),
                                 (0.999, 1.0), (-1e-9, 1e-9)])
def test_root_of_a_cubic(lib, ulp, a, b):
    z = np.random.default_rng(5).uniform(a, b, 200000)
    y, u = np.empty(len(z)), np.empty(len(z))
    lib.thirds(_ptr(z), _ptr(y), _ptr(u), ctypes.c_long(len(z)), ulp)
    assert u.max() < 0.6
    # Near -1 (a double root) and from 1 on: the library's functions
    z = np.array([-1.0, -0.9999, 1.0, 1.1, -1.1, np.nan, np.inf, 0.0, -0.0,
                  1e-300])
    y, u = np.empty(len(z)), np.empty(len(z))
    lib.thirds(_ptr(z), _ptr(y), _ptr(u), ctypes.c_long(len(z)), ulp)
    with np.errstate(all='ignore'):
        r = np.cos(np.arccos(z) / 3)
    ok = (np.abs(y - r) <= 1e-15) | (np.isnan(y) & np.isnan(r))
    assert ok.all(), z[~ok]


def test_where_the_functions_are_written(decker):
    from conftest import myokit
    w = exporter.CudaExpressionWriter(False, soft=True, fuse=True)
    w.set_lhs_function(lambda x: 'x')
    x, n = myokit.Name(decker.get('membrane.V')), myokit.Number
    third = myokit.Divide(myokit.ACos(x), n(3))
    for e, text in (
            (myokit.Sqrt(x), 'mkg_sqrt(x)'), (myokit.Log(x), 'mkg_log(x)'),
            (myokit.Power(x, n(0.5)), 'mkg_sqrt(x)'),
            (myokit.Power(x, n(-1.5)),
             'mkg_pow_literal(x, -1.5, 1729382256910270464ull, ~0u)'),
            (myokit.Power(x, n(17.5)), 'pow(x, 17.5)'),
            (myokit.Power(x, n(-0.001)), 'pow(x, -0.001)'),
            (myokit.Cos(third), 'mkg_cos_third(x)'),
            (myokit.Cos(x), 'cos(x)'),
            (myokit.Divide(x, n(1)), 'x'),
            (myokit.Divide(x, n(-0.25)), '(x * -4.0)')):
        assert w.ex(e) == text
