"""
The functions of the double precision kernels (csrc/mkg_math64.h) on the
device, whose approximations they start from: division and square root equal
to the processor's bit for bit, the others within the bounds that the header
states, in units in the last place against longer arithmetic; zeros,
denormals, infinities and NaN as CUDA's functions have them.
"""
import ctypes

import numpy as np
import pytest

from myokit_gb300 import _lib, exporter

POWERS = [1.4, -1.4, 0.7, 1 / 3, -3.7, 2.0 ** -8]
SOURCE = 'typedef double Real;\n@HELPERS@\n' + ''.join(
    'extern "C" __global__ void %s(const double *x, const double *z,'
    ' double *y, int n)\n{ const int i = blockIdx.x * 256 + threadIdx.x;\n'
    '  if (i < n) y[i] = %s; }\n' % f for f in [
        ('f_exp', 'mkg_exp(x[i])'), ('f_log', 'mkg_log(x[i])'),
        ('f_sqrt', 'mkg_sqrt(x[i])'), ('f_div', 'mkg_div(x[i], z[i])'),
        ('f_third', 'mkg_cos_third(x[i])')] + [
        ('f_pow%d' % q, 'mkg_pow_literal(x[i], %r, %dull, %s)' % (
            p, int(abs(p) * 2 ** 60), '~0u' if p < 0 else '0u'))
        for q, p in enumerate(POWERS)])


@pytest.fixture(scope='module', params=[False, True],
                ids=['inlined', 'called'])
def device(request):
    """name, x[, z] -> the function's values on the GPU."""
    torch = pytest.importorskip('torch')
    cubin, _ = _lib.compile_source(
        SOURCE.replace('@HELPERS@',
                       exporter._pow_helpers(False, request.param)),
        ['--gpu-architecture=sm_103a', '--std=c++17', '--fmad=false'])
    torch.zeros(1, device='cuda')
    cuda = ctypes.CDLL('libcuda.so.1')
    module, kernel = ctypes.c_void_p(), ctypes.c_void_p()
    assert cuda.cuModuleLoadData(ctypes.byref(module), cubin) == 0

    def call(name, x, z=None):
        assert cuda.cuModuleGetFunction(
            ctypes.byref(kernel), module, name.encode()) == 0
        n = len(x)
        t = [torch.from_numpy(np.ascontiguousarray(v)).cuda()
             for v in (x, x if z is None else z, np.empty(n))]
        args = [ctypes.c_void_p(v.data_ptr()) for v in t] + [
            ctypes.c_int(n)]
        torch.cuda.synchronize()
        assert cuda.cuLaunchKernel(
            kernel, -(-n // 256), 1, 1, 256, 1, 1, 0, None,
            (ctypes.c_void_p * 4)(*[
                ctypes.cast(ctypes.byref(a), ctypes.c_void_p)
                for a in args]), None) == 0
        torch.cuda.synchronize()
        return t[2].cpu().numpy()
    return call


def _same(y, r):
    ok = (y.view(np.uint64) == r.view(np.uint64)) | (
        np.isnan(y) & np.isnan(r))
    assert ok.all(), (y[~ok][:3], r[~ok][:3])


def _units(y, e):
    """|y - e| in units in the last place of e (longer arithmetic)."""
    one = np.spacing(np.abs(e.astype(np.float64)))
    return float(np.max(np.abs(y.astype(np.longdouble) - e) / one))


def _doubles(rng, n, spread):
    return rng.choice([-1.0, 1.0], n) * rng.uniform(1, 2, n) * np.exp2(
        rng.integers(-spread, spread, n).astype(float))


EDGES = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, 1e-310, 1.0,
                  2.0 ** -1022, 1.7976931348623157e308, -1.0, -1e-310, 0.5,
                  np.nextafter(1, 0), np.nextafter(1, 2), -708.0, 709.9])


@pytest.mark.gpu
def test_division_and_square_root(device):
    rng = np.random.default_rng(1)
    with np.errstate(all='ignore'):
        for spread in (2, 60, 1022):
            x, z = (_doubles(rng, 1 << 20, spread) for _ in range(2))
            x[:len(EDGES) ** 2] = np.repeat(EDGES, len(EDGES))
            z[:len(EDGES) ** 2] = np.tile(EDGES, len(EDGES))
            _same(device('f_div', x, z), x / z)
            x = np.abs(x)
            k = np.arange(1, 50001, dtype=float) ** 2
            x[:150000] = np.concatenate(
                [k, np.nextafter(k, 0), np.nextafter(k, np.inf)])
            x[150000:150000 + len(EDGES)] = EDGES
            _same(device('f_sqrt', x), np.sqrt(x))


@pytest.mark.gpu
def test_exponential_and_logarithm(device):
    rng = np.random.default_rng(2)
    for size in (1e-9, 0.01, 1.0, 30.0, 708.0):
        x = rng.uniform(-size, size, 1 << 18)
        # (the library's function, to an ulp, for tiny arguments)
        assert _units(device('f_exp', x), np.exp(
            x.astype(np.longdouble))) <= (0.58 if size > 1e-3 else 1.0)
    for size in (0.3, 3.0, 700.0):
        x = np.exp(rng.uniform(-size, size, 1 << 18))
        far = np.abs(np.log(x)) > 0.008
        y, e = device('f_log', x), np.log(x.astype(np.longdouble))
        assert _units(y[far], e[far]) <= 0.53
        near = (x != 1) & ~far
        assert not near.any() or _units(y[near], e[near]) <= 1.0
    with np.errstate(all='ignore'):
        for name, f in (('f_exp', np.exp), ('f_log', np.log)):
            y, r = device(name, EDGES), f(EDGES)
            ok = np.isfinite(r)
            assert np.array_equal(y[~ok], r[~ok], equal_nan=True)
            assert np.all(np.abs(y - r)[ok] <= np.spacing(np.abs(r[ok])))


@pytest.mark.gpu
def test_powers_and_cubic_roots(device):
    rng = np.random.default_rng(3)
    for q, p in enumerate(POWERS):
        x = np.exp(rng.uniform(-1, 1, 1 << 18) *
                   rng.choice([1e-3, 1, 30], 1 << 18))
        e = np.power(x.astype(np.longdouble), np.longdouble(p))
        # (the library's pow, to two ulps, near 1)
        near = np.abs(np.log(x)) < 1e-9
        assert _units(device('f_pow%d' % q, x)[~near], e[~near]) <= 0.61
        with np.errstate(all='ignore'):
            y, r = device('f_pow%d' % q, EDGES), EDGES ** p
            ok = (y == r) | (np.isnan(y) & np.isnan(r)) | (
                np.abs(y - r) <= 2 * np.spacing(np.abs(r)))
        assert ok.all(), (EDGES[~ok], y[~ok], r[~ok])
    for a, b in ((-0.9995, 1.0), (0.999, 1.0), (-1e-9, 1e-9)):
        z = rng.uniform(a, b, 1 << 18)
        e = np.cos(np.arccos(z.astype(np.longdouble)) / 3)
        assert _units(device('f_third', z), e) <= 0.61
    z = np.array([-1.0, -0.9999, 1.0, 1.1, -1.1, np.nan, np.inf, 0.0, -0.0,
                  1e-300])
    with np.errstate(all='ignore'):
        y, r = device('f_third', z), np.cos(np.arccos(z) / 3)
    assert np.array_equal(np.isnan(y), np.isnan(r))
    ok = ~np.isnan(r)
    assert np.all(np.abs(y - r)[ok] <= 1e-15)
