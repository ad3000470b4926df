"""
What simulations keep between calls: generated kernels shared by what they
are generated from, log columns and connections converted once. Every change
of the model, the options or the log has to be seen.
"""
import threading

import numpy as np
import pytest

from conftest import myokit
import myokit_gb300 as mg
from myokit_gb300 import simulation

SP = myokit.SINGLE_PRECISION
DP = myokit.DOUBLE_PRECISION


def _sim(model, **kw):
    kw.setdefault('ncells', 40)
    return mg.SimulationCUDA(model, None, **kw)


def test_one_kernel_for_equal_simulations(br77):
    a, b = _sim(br77)._kernel([]), _sim(br77)._kernel([])
    assert a is b
    # Anything the kernel depends on makes it another
    others = [
        _sim(br77, precision=DP)._kernel([]),
        _sim(br77, ncells=(8, 5))._kernel([]),
        _sim(br77, diffusion=False)._kernel([]),
        _sim(br77, accumulate='kahan')._kernel([]),
        _sim(br77, fp32_math='ieee')._kernel([]),
        _sim(br77, native_maths=True)._kernel([]),
        _sim(br77, block=64)._kernel([]),
        _sim(br77, rl=True)._kernel([]),
    ]
    s = _sim(br77)
    others.append(s._kernel([s._model.get('isi.Isi')]))
    s.set_field('isi.gsBar', np.full(40, 0.08))
    others.append(s._kernel([]))
    s = _sim(br77)
    s.set_connections([(0, 1, 2.0)])
    others.append(s._kernel([]))
    assert all(k is not a for k in others)
    assert len(set(id(k) for k in others)) == len(others)


def test_bounded_and_shared_between_threads():
    made = []

    def make(i):
        made.append(i)
        return object()
    with simulation._KERNELS_LOCK:
        saved = dict(simulation._KERNELS)
        simulation._KERNELS.clear()
    try:
        threads = [threading.Thread(target=lambda: [
            simulation.shared_kernel(i, lambda: make(i)) for i in range(50)])
            for _ in range(4)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert len(simulation._KERNELS) == 32
        k = simulation.shared_kernel('x', object)
        assert simulation.shared_kernel('x', object) is k
    finally:
        with simulation._KERNELS_LOCK:
            simulation._KERNELS.clear()
            simulation._KERNELS.update(saved)


@pytest.mark.gpu
def test_changed_logs_and_connections_are_seen(br77):
    # One simulation whose log and connections change between runs, against
    # new simulations; and two simulations that share a kernel
    def new():
        s = mg.SimulationCUDA(br77, myokit.pacing.blocktrain(
            period=1000, duration=2, level=1), ncells=70)
        s.set_paced_cell_list([0, 1])
        return s
    chain = [(i, i + 1, 8.0) for i in range(69)]
    logs = [['engine.time', '3.membrane.V'], ['3.membrane.V', '4.membrane.V'],
            ['4.membrane.V', '3.membrane.V'], ['3.ina.m', '60.isi.Isi'],
            ['3.membrane.V'], ['engine.time', 'engine.pace']]
    s = new()
    for k, log in enumerate(logs + logs[::-1]):
        conn = chain if k % 3 else [(i, j, g / 2) for i, j, g in chain[::-1]]
        out = []
        for sim in (s, new()):
            sim.reset()
            sim.set_connections(conn)
            d = sim.run(1.5, log=log, log_interval=0.25)
            out.append((sim.state_array(), {
                n: np.asarray(v) for n, v in d.items()}))
        assert list(out[0][1]) == list(out[1][1]) == log
        assert np.array_equal(out[0][0], out[1][0])
        for n in log:
            assert len(out[0][1][n]) == 6
            assert np.array_equal(out[0][1][n], out[1][1][n])


@pytest.mark.gpu
def test_appending_to_a_log(br77):
    # A log of a former run is continued, as lists or arrays
    p = myokit.pacing.blocktrain(period=1000, duration=2, level=1)
    keys = ['engine.time', '0.membrane.V', '9.membrane.V']
    s = mg.SimulationCUDA(br77, p, ncells=10)
    d = s.run(1, log=keys, log_interval=0.25)
    first = {k: list(d[k]) for k in keys}
    d2 = s.run(1, log=keys, log_interval=0.25)
    assert [len(d[k]) for k in keys] == [4] * 3
    assert d2['engine.time'][0] > first['engine.time'][-1]
    assert list(d['0.membrane.V']) == first['0.membrane.V']
