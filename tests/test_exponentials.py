"""
Single precision exponentials: 2^t with the argument's literal factor in two
parts only where their product would be rounded; else the library's function,
which is within an ulp at any exponent. Denormals are kept in the modes that
promise to.
"""
import numpy as np
import pytest

from conftest import myokit
import myokit_gb300 as mg

SP = myokit.SINGLE_PRECISION
ARGS = ['y', '-y', '2 * y', '0.25 * y', 'y / 4', '0.1 * y', 'y / -6.8']


def _exponentials(model, args=ARGS):
    """``model`` with a state y and a variable exp(...) per argument."""
    m = model.clone()
    c = m.add_component('ex')
    y = c.add_variable('y')
    y.set_rhs('0 * membrane.V')
    y.promote(0.5)
    for q, a in enumerate(args):
        c.add_variable('e%d' % q).set_rhs(
            'exp(%s)' % a.replace('y', 'ex.y'))
    return m


def _texts(model, math):
    s = mg.SimulationCUDA(_exponentials(model), None, ncells=200,
                          fp32_math=math)
    k = s._kernel([s._model.get('ex.e%d' % q) for q in range(len(ARGS))])
    text = dict((k._name(lhs), k.rhs_code(lhs, rhs))
                for lhs, rhs in k.rhs_eqs)
    return k, [text[k._name(s._model.get('ex.e%d' % q))]
               for q in range(len(ARGS))]


@pytest.mark.parametrize('math', ['fast', 'default', 'ieee'])
def test_which_exponentials_are_scaled(br77, math):
    k, text = _texts(br77, math)
    scaled = [t.startswith('mkg_exp_scaled(') for t in text]
    assert scaled == [False] * 5 + [True] * 2
    assert all(t.startswith('expf(') for t, x in zip(text, scaled) if not x)
    # Flushing denormals in fast mode only
    flush = math == 'fast'
    assert ('ex2.approx.ftz.f32' in k.source()) == flush
    assert ('ex2.approx.f32' in k.source()) != flush
    assert ('--ftz=true' in k.options()) == flush


@pytest.mark.parametrize('math', ['fast', 'default', 'ieee'])
def test_decay_of_gates(decker, math):
    # Scaled where it saves the roundings of a reciprocal time constant
    s = mg.SimulationCUDA(decker, None, ncells=200, rl=True, fp32_math=math)
    k = s._kernel([])
    assert k.rl_states
    for inf, tau in k.rl_states.values():
        t = k.decay(tau, k._name(tau), k.rates)
        scaled = tau in k.rates
        assert t.startswith('mkg_exp_scaled(' if scaled else 'expf(-(')


@pytest.mark.gpu
@pytest.mark.parametrize('math', ['fast', 'default', 'ieee'])
def test_errors_against_64_bits(br77, math):
    # Within 2 ulps of the exact exponential of the argument, of which the
    # product with a factor that is not a power of two may be rounded, and
    # the factor with it
    m = _exponentials(br77)
    n = 4096
    rng = np.random.default_rng(1)
    y = np.float32(np.concatenate([
        rng.uniform(-85, 85, n // 2), rng.uniform(-2, 2, n // 4),
        rng.uniform(-100, -88, n // 4)]))
    s = mg.SimulationCUDA(m, None, ncells=n, diffusion=False, fp32_math=math)
    st = s.state_array().reshape(n, -1).copy()
    st[:, s._model.get('ex.y').index()] = y
    s.set_state(st.reshape(-1))
    keys = ['%d.ex.e%d' % (c, q) for q in range(len(ARGS)) for c in range(n)]
    d = s.run(s.step_size(), log=keys, log_interval=s.step_size())
    y = y.astype(float)
    for q, (arg, k) in enumerate(zip(ARGS, (1, -1, 2, 0.25, 0.25, 0.1,
                                            -1 / 6.8))):
        got = np.array([d['%d.ex.e%d' % (c, q)][0] for c in range(n)], float)
        with np.errstate(over='ignore'):
            want = np.exp(k * y)
        ok = want < 3.4e38
        assert np.all(np.isinf(got[~ok]))
        product = 0 if k in (1, -1, 2, 0.25) else 2 * 2.0 ** -24 * abs(k * y)
        bound = want * (2 * 2.0 ** -23 + product)
        # Denormals flush to zero in fast mode, and are whole units of the
        # smallest in the others
        bound = np.maximum(bound, 1.18e-38 if math == 'fast' else 2.9e-45)
        err = np.abs(got - want)
        assert np.all(err[ok] <= bound[ok]), (arg, np.max(
            (err / bound)[ok]))
        if math != 'fast':
            small = (want < 1e-38) & (want > 1e-43)
            assert np.all(got[small] > 0)
