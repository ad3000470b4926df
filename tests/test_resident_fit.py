"""
Whether a resident kernel's tiles fit on an SM: their static shared memory,
in units of 128 bytes, and the kilobyte that the device keeps per CTA. Where
they do not, the undivided kernel runs.
"""
import pytest

from conftest import myokit
import myokit_gb300 as mg

SP = myokit.SINGLE_PRECISION
TILES = 152 * 16


def _states(model, n):
    """``model`` with states that decay, ``n`` in all."""
    m = model.clone()
    c = m.add_component('more')
    for q in range(n - m.count_states()):
        v = c.add_variable('x%d' % q)
        v.set_rhs('-0.01 * more.x%d' % q)
        v.promote(1.0)
    return m


def _simulation(br77, n, tiles):
    return mg.SimulationCUDA(_states(br77, n), None, ncells=32 * tiles,
                             precision=SP)


# (104 states and sixteen CTAs fill an SM's 228 KB to the last byte)
@pytest.mark.parametrize('n,tiles,team', [
    (104, TILES, 1), (105, TILES, 0), (106, TILES, 0), (107, TILES, 0),
    (106, TILES - 152, 1), (106, TILES - 151, 0)])
def test_tiles_that_do_not_fit(br77, n, tiles, team):
    k = _simulation(br77, n, tiles)._kernel([])
    assert k.n_state == n and k.team == team


@pytest.mark.gpu
@pytest.mark.parametrize('n', [104, 105, 106])
def test_runs_where_tiles_just_fit(br77, n):
    s = _simulation(br77, n, TILES)
    s.set_paced_cells(5)
    d = s.run(2 * s.step_size(), log=['engine.time', '7.membrane.V'],
              log_interval=s.step_size())
    assert len(d['7.membrane.V']) == 2
    assert s._last_kernel.team == (1 if n == 104 else 0)
