"""
Resident kernels of models whose diffusion current enters several equations,
as in ion balances that conserve charge: no warp of a team reads the tile's V
or its neighbours' words once the first warp may have stored those of the
next step, and no warp tests a stop word that another may be setting.
"""
import itertools
import re

import numpy as np
import pytest

from conftest import myokit
import myokit_gb300 as mg
from test_resident import _check_plan, _kernel, _run, _same

DP = myokit.DOUBLE_PRECISION
SP = myokit.SINGLE_PRECISION


def _balances(model, n):
    """``model`` with ``n`` more states that the diffusion current changes."""
    m = model.clone()
    i = m.binding('diffusion_current').qname()
    c = m.add_component('balance')
    for q in range(n):
        v = c.add_variable('x%d' % q)
        v.set_rhs('-0.001 * (%s + %d * balance.x%d)' % (i, q + 1, q))
        v.promote(1.0)
    return m


def _through(model):
    """``model`` with two states that the current reaches through others."""
    m = model.clone()
    i = m.binding('diffusion_current').qname()
    c = m.add_component('through')
    x = [c.add_variable('x%d' % q) for q in range(2)]
    for v in x:
        v.set_rhs('0')
        v.promote(1.0)
    c.add_variable('t').set_rhs('%s + 0.5 * through.x0' % i)
    c.add_variable('e').set_rhs('exp(-0.0001 * through.t * through.t)')
    x[0].set_rhs('-0.001 * (through.t + through.e)')
    x[1].set_rhs('-0.01 * through.e * through.x1')
    return m


def _parts(k):
    """Each warp's code of a step, cut where the team meets."""
    body = re.split(r'\n *(?:else )?if \(part_ == \d+\) \{\n',
                    '\n' + k.team_body)[1:]
    assert len(body) == k.team
    return [b.split('mkg_team_sync();') for b in body]


def _check_current(k):
    """The last read of V and of the neighbours' words stands in front of a
    meeting of the team, or in the warp that stores V, in front of that."""
    parts = _parts(k)
    assert len(set(len(p) for p in parts)) == 1
    stored = [(w, f) for w, p in enumerate(parts) for f, x in enumerate(p)
              if re.search(r'\bvs\[lane\] = ', x)]
    assert len(stored) == 1
    w0, f0 = stored[0]
    takers = 0
    for w, p in enumerate(parts):
        for f, x in enumerate(p):
            takers += 'MKG_HALO(id_)' in x
            if 'MKG_HALO(' in x or 'MKG_HALO_ASK(' in x:
                assert f < f0 or (w, f) == (w0, f0), (w, f)
        assert w == w0 or 'mkg_word_store' not in ''.join(p)
    x = parts[w0][f0]
    assert x.rfind('MKG_HALO') < x.index('vs[lane] = ')
    return takers


@pytest.mark.parametrize('precision,kw', [
    (SP, {}), (DP, {}), (SP, {'accumulate': 'kahan'}),
    (SP, {'accumulate': 'double'})])
@pytest.mark.parametrize('n', [0, 1, 2])
@pytest.mark.parametrize('team', [1, 2, 4, 8])
def test_current_is_read_before_it_changes(decker, br77, team, n, precision,
                                           kw):
    for m, rl in ((decker, True), (br77, False), (br77, True)):
        k = _kernel(_balances(m, n), precision, team, rl, **kw)
        _check_plan(k)
        assert _check_current(k) >= 1


@pytest.mark.parametrize('precision', [SP, DP])
@pytest.mark.parametrize('team', [2, 4, 8])
def test_current_through_other_variables(decker, br77, team, precision):
    for m, rl in ((decker, True), (br77, False)):
        k = _kernel(_through(m), precision, team, rl)
        _check_plan(k)
        _check_current(k)
        _check_stop(k)


def test_current_of_default_launch_shapes(decker, br77):
    for m, rl in ((decker, True), (br77, False)):
        for n in (200, 4000, 20000, (128, 128), (200, 150)):
            for precision in (SP, DP):
                k = mg.SimulationCUDA(_balances(m, 1), None, ncells=n,
                                      precision=precision, rl=rl)._kernel([])
                if k.team:
                    _check_current(k)


def _check_stop(k):
    """A word that says to leave is not set in an interval between two
    meetings in which another warp tests it: that warp could leave a step
    before the others, which would wait for it at the next meeting. (Words
    by the step's parity: 0 is the step's, 1 the next step's.)"""
    sets, tests = {}, {}
    for w, p in enumerate(_parts(k)):
        word = 0
        for f, x in enumerate(p):
            for t in re.findall(r'MKG_HALO\(id_\)|MKG_CHECK_HALT\(\)|'
                                r'if \(s_stop|stop_ \^= 1', x):
                if t.startswith('stop_'):
                    word ^= 1
                else:
                    (tests if t.startswith('if') else sets).setdefault(
                        (f, word), set()).add(w)
    assert set(tests) == {(1, 0)} and len(tests[1, 0]) == k.team
    assert not set(sets) & set(tests)
    # What is set before the test is tested in this step, else in the next
    assert all(word == min(f, 1) for f, word in sets)
    loop = k.source().split('for (; k < nsteps; ++k) {')[1]
    assert set(re.findall(r's_stop\W?\w*\W?', loop)) == {'s_stop[stop_]'}
    assert 'int stop_ = k & 1;' in loop


@pytest.mark.parametrize('precision', [SP, DP])
@pytest.mark.parametrize('team', [1, 2, 4, 8])
def test_stop_word_is_not_tested_while_it_may_be_set(decker, br77, team,
                                                     precision):
    for m, rl, n in ((br77, False, 0), (br77, False, 2), (br77, True, 0),
                     (decker, True, 0), (decker, True, 1)):
        _check_stop(_kernel(_balances(m, n), precision, team, rl))


# ---------------------------------------------------------------------------
# GPU
# ---------------------------------------------------------------------------

@pytest.mark.gpu
@pytest.mark.parametrize('precision,kw', [
    (SP, {}), (DP, {}), (SP, {'accumulate': 'double'})],
    ids=['fp32', 'fp64', 'double'])
def test_several_balances_equal_undivided(decker, br77, precision, kw):
    # Grids, per-edge conductances and connections with more than four
    # neighbours, several times
    near = [(i, j, 0.5 + (i * j) % 3) for i, j in itertools.combinations(
        range(150), 2) if j - i in (1, 2, 31, 33, 64)]
    for m, rl, shape, more in (
            (br77, False, 200, {}), (br77, False, (40, 9), {}),
            (br77, False, 150, dict(conn=near)),
            (br77, False, (41, 7), dict(hetero=True)),
            (decker, True, (61, 5), {})):
        for m, name in ((_balances(m, 2), 'balance.x1'),
                        (_through(m), 'through.x1')):
            _check_runs(m, rl, shape, more, precision, kw, name)


def _check_runs(m, rl, shape, more, precision, kw, name):
    log = ['%s3.%s' % ('2.' if isinstance(shape, tuple) else '', name)]
    want = _run(m, 0, shape, precision, rl, log=log, **more, **kw)
    assert not np.all(want[1][log[0]] == 1.0)
    for team in (2, 4, 8, 4, 2):
        _same(want, _run(m, team, shape, precision, rl, log=log, **more,
                         **kw))
