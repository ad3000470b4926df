"""
The arithmetic the exporter writes out: multiply-adds chosen from the
expression alone (kernels are compiled without the compiler's contraction),
and single precision exponentials with their scale in two parts. The text is
evaluated here in rational arithmetic, where it has to equal the expression;
on the GPU, kernels of different structure give the same bits.
"""
from fractions import Fraction

import numpy as np
import pytest

from conftest import myokit
import myokit_gb300 as mg
from myokit_gb300 import exporter

SP = myokit.SINGLE_PRECISION
DP = myokit.DOUBLE_PRECISION
f32 = np.float32


def _rational(text, **names):
    """The value of a text in exact rational arithmetic."""
    import re
    text = re.sub(r'(?<=[0-9.])[fu](?![0-9a-zA-Z_])', '', text)
    text = re.sub(r'(?<![\w.])(\d+(\.\d*)?)', r'Fraction("\1")', text)
    return eval(text, dict(
        names, Fraction=Fraction, fma=lambda a, b, c: a * b + c,
        fmaf=lambda a, b, c: a * b + c, mkg_pow2=lambda x: x * x,
        __fdividef=lambda a, b: a / b, mkg_div=lambda a, b: a / b,
        mkg_div_by=lambda a, b, y: a / b))


def _expressions(model):
    v = myokit.Name(model.get('membrane.V'))
    m = myokit.Name(model.get('ina.m'))
    n = myokit.Number
    a = myokit.Plus(v, n(47.125))
    A = lambda x, y: x + Fraction(377, 8)  # noqa: E731
    yield (myokit.Minus(myokit.Multiply(v, m), myokit.Multiply(n(3), m)),
           lambda x, y: x * y - 3 * y)
    yield (myokit.Minus(myokit.Multiply(v, m), a),
           lambda x, y: x * y - A(x, y))
    yield (myokit.Plus(myokit.PrefixMinus(myokit.Multiply(v, m)), v),
           lambda x, y: x - x * y)
    yield (myokit.Minus(v, myokit.PrefixMinus(myokit.Multiply(v, m))),
           lambda x, y: x + x * y)
    yield myokit.Minus(v, myokit.Divide(a, n(0.5))), \
        lambda x, y: x - 2 * A(x, y)
    yield myokit.Minus(myokit.Divide(a, n(-0.25)), m), \
        lambda x, y: -4 * A(x, y) - y
    yield (myokit.Plus(myokit.Power(m, n(2)), myokit.Divide(v, m)),
           lambda x, y: y * y + x / y)
    yield myokit.Minus(n(1), myokit.Power(v, n(2))), lambda x, y: 1 - x * x
    yield myokit.Minus(myokit.Minus(v, m), a), lambda x, y: x - y - A(x, y)
    yield myokit.Multiply(myokit.Plus(v, m), a), \
        lambda x, y: (x + y) * A(x, y)


@pytest.mark.parametrize('single', [True, False])
@pytest.mark.parametrize('fast', [True, False])
def test_written_out_arithmetic_is_the_expression(decker, single, fast):
    w = exporter.CudaExpressionWriter(single, fast_divide=fast, soft=True,
                                      fuse=True)
    w.set_lhs_function(lambda x: x.var().qname().split('.')[-1])
    fused = 0
    for e, f in _expressions(decker):
        if single and not fast and any(isinstance(x, myokit.Divide)
                                       for x in e.walk()):
            continue     # (written by the base class)
        text = w.ex(e)
        fused += 'fma' in text
        for V, m in ((Fraction(-169, 2), Fraction(1, 128)),
                     (Fraction(13, 4), Fraction(7, 8))):
            assert _rational(text, V=V, m=m) == f(V, m), text
    assert fused >= 5


@pytest.mark.parametrize('k', [1.0, -1.0, 0.1, 1 / 6.8, -2.0 ** -7, 1e-3, 40])
def test_scale_of_an_exponential_in_two_parts(k):
    w = exporter.CudaExpressionWriter(True, fuse=True)
    hi, lo = [f32(x.strip(' f)')) for x in
              w.scaled_exp('x', k).split(',')[1:]]
    want = k * np.log2(np.e)
    # A rest of the same sign and not zero: an infinite x stays infinite
    assert lo != 0 and np.sign(lo) == np.sign(hi) == np.sign(k)
    assert abs(float(hi) + float(lo) - want) <= 2.0 ** -46 * abs(want)


@pytest.mark.parametrize('k', [0.0, 1e-30, 1e30])
def test_scales_beyond_two_parts(k):
    w = exporter.CudaExpressionWriter(True, fuse=True)
    assert w.scaled_exp('x', k).startswith('expf((x) * ')


@pytest.mark.gpu
@pytest.mark.parametrize('precision', [SP, DP])
@pytest.mark.parametrize('shape', [(64, 20), (37, 23), 700])
def test_kernels_of_different_structure_give_the_same_bits(decker, precision,
                                                           shape):
    out = []
    for lazy, stage, block in ((0, True, 128), (1, True, 64), (0, False, 96)):
        p = myokit.pacing.blocktrain(period=1000, duration=2, level=1)
        s = mg.SimulationCUDA(decker, p, ncells=shape, rl=True,
                              precision=precision, stage_tiles=stage,
                              block=block, min_blocks=1)
        s._stage_lazy = lazy
        s.set_paced_cells(4)
        s.run(1.5, log=['engine.time'])
        out.append(s.state_array())
    assert np.array_equal(out[0], out[1])
    assert np.array_equal(out[0], out[2])
