"""
Connections beyond a cell's first four, whose words resident tiles ask for in
groups: every number of them, inside and outside a tile, gives the undivided
kernel's bits.
"""
import itertools

import numpy as np
import pytest

from conftest import myokit
import myokit_gb300 as mg
from myokit_gb300 import _lib
from test_resident import _run, _same

DP = myokit.DOUBLE_PRECISION
SP = myokit.SINGLE_PRECISION
NEAR = (1, 2, 31, 33, 64, 3, 5, 40, 65, 97, 7, 50, 90)


@pytest.mark.parametrize('most,precision,team', [
    (40, SP, 4), (41, SP, 0), (41, DP, 8)])
def test_many_neighbours(br77, most, precision, team):
    # Single precision: the undivided kernel from 41 neighbours of one cell
    s = mg.SimulationCUDA(br77, None, ncells=200, precision=precision)
    s.set_connections([(0, j, 1.0) for j in range(1, most + 1)])
    assert s._kernel([]).team == team
    s.set_connections([(i, i + 1, 1.0) for i in range(199)])
    assert s._kernel([]).team
    s.set_connections([])
    assert s._kernel([]).team


def test_kernel_of_few_neighbours(br77):
    # No code for more than four where no cell has them
    s = mg.SimulationCUDA(br77, None, ncells=200)
    many = []
    for most in (4, 5, 3):
        s.set_connections([(0, j, 1.0) for j in range(1, most + 1)])
        many.append(s._kernel([]))
    assert [k.many for k in many] == [False, True, False]
    assert many[0] is many[2] and '#define MANY 1' in many[1].source()
    cubin, _ = _lib.compile_source(many[0].source(), many[0].options())
    assert cubin[:4] == b'\x7fELF'


@pytest.mark.gpu
def test_connections_that_change(br77):
    few = [(i, i + 1, 2.0) for i in range(149)]
    more = few + [(i, i + 5, 0.5) for i in range(0, 145)] + [
        (i, i + 40, 0.25) for i in range(110)]
    s = mg.SimulationCUDA(br77, myokit.pacing.blocktrain(
        period=1000, duration=2, level=1), ncells=150)
    for conn in (few, more, few):
        t = mg.SimulationCUDA(br77, myokit.pacing.blocktrain(
            period=1000, duration=2, level=1), ncells=150)
        out = []
        for x in (s, t):
            x.reset()
            x.set_paced_cell_list([0, 40])
            x.set_connections(conn)
            x.run(1.0, log=['engine.time'], log_interval=0.5)
            out.append(x.state_array().copy())
        assert np.array_equal(*out)
        assert s._last_kernel.many == (conn is more)


@pytest.mark.gpu
@pytest.mark.parametrize('precision,kw', [
    (SP, {}), (DP, {}), (SP, {'accumulate': 'double'})],
    ids=['fp32', 'fp64', 'double'])
@pytest.mark.parametrize('most', [3, 4, 6, 7, 13])
def test_equals_undivided(br77, precision, kw, most):
    # (up to twice as many neighbours, fewer at the ends of the row)
    conn = [(i, j, 0.2 + 0.1 * ((i * j) % 3)) for i, j in
            itertools.combinations(range(150), 2) if j - i in NEAR[:most]]
    want = _run(br77, 0, 150, precision, False, conn=conn, paced=[0, 40],
                **kw)
    for team in (1, 2, 4, 8):
        _same(want, _run(br77, team, 150, precision, False, conn=conn,
                         paced=[0, 40], **kw))
