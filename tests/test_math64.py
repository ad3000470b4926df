"""
exp and division of the double precision kernels (csrc/mkg_math64.h, integer
arithmetic) compiled for the host: division equal to the processor's bit for
bit, exp within 0.57 units in the last place of the 64-bit-significand
result, also at the edges of the ranges and where the library's function
takes over. The device's reciprocal approximation (one unit in the last
place) is taken as exact, one unit low and one unit high.
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
#include "mkg_math64.h"
extern "C" void divide(const double *a, const double *b, double *q, long n,
                       int u)
{ ulp = u; for (long i = 0; i < n; ++i) q[i] = mkg_div(a[i], b[i]); }
extern "C" void divide_by(const double *a, double b, unsigned y, double *q,
                          long n)
{ for (long i = 0; i < n; ++i) q[i] = mkg_div_by(a[i], b, y); }
extern "C" void exps(const double *x, double *y, double *ulps, long n)
{
    for (long i = 0; i < n; ++i) {
        y[i] = mkg_exp(x[i]);
        const long double e = expl((long double)x[i]);
        ulps[i] = (double)(fabsl((long double)y[i] - e) /
                           ldexpl(1.0L, ilogbl(e) - 52));
    }
}
'''


@pytest.fixture(scope='module')
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp('math64')
    src = d / 'm.cpp'
    src.write_text(HOST.replace('@TABLE@', exporter._exp_table()))
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
