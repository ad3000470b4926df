"""
The reverse of a resident simulation: the matrices of a stretch of steps, all
at once, and a sweep over them. It differs from the general reverse kernel
only by the order of the multiply-adds, so gradients agree to rounding: a
gradient is a sum over some hundred steps of products with one rounding per
factor, and the states' sensitivities grow by less than a thousand over
them, so 1e-11 of an array's largest value in double precision (2^-53 times
1e5) and 1e-3 in single.
"""
import itertools

import numpy as np
import pytest

from conftest import myokit
import myokit_gb300 as mg
from myokit_gb300 import _lib, adjoint

DP = myokit.DOUBLE_PRECISION
SP = myokit.SINGLE_PRECISION


def _adjoint(model, precision, shape, rl, general, conn=None, hetero=False,
             fields=(), diffusion=True, probes=(0,), segment=40, spl=0,
             **kw):
    p = myokit.pacing.blocktrain(period=1000, duration=2, level=1)
    s = mg.SimulationCUDA(model, p, ncells=shape, precision=precision, rl=rl,
                          diffusion=diffusion, **kw)
    s.set_step_size(0.01)
    sh = shape[::-1] if isinstance(shape, tuple) else (shape,)
    rng = np.random.default_rng(3)
    if hetero and len(sh) == 2:
        s.set_conductance_field(rng.uniform(4, 9, (sh[0], sh[1] - 1)),
                                rng.uniform(2, 5, (sh[0] - 1, sh[1])))
    elif hetero:
        s.set_conductance_field(rng.uniform(4, 9, sh[0] - 1))
    if conn is not None:
        s.set_connections(conn)
    for f in fields:
        s.set_field(f, s._model.get(f).eval() * rng.lognormal(0, 0.2, sh))
    return adjoint.TissueAdjoint(s, probes, segment_steps=segment,
                                 threads=64 if general else None)


def _kernel(adj):
    kernel = adj.sim._kernel([])
    return adj._make(kernel, adj._tiles_per_sm(kernel))


CONN = [(i, j, 0.5 + (i * j) % 3) for i, j in itertools.combinations(
    range(150), 2) if j - i in (1, 2, 31, 33, 64)]
CASES = {
    'sheet': dict(shape=(41, 7), probes=[(0, 0), (40, 6), (32, 3)]),
    'row': dict(shape=(33, 1), probes=[(0, 0), (32, 0)]),
    'column': dict(shape=(1, 9), probes=[(0, 4)]),
    'cell': dict(shape=1),
    'cable': dict(shape=97, probes=[0, 64, 96], segment=7),
    'edges': dict(shape=(65, 3), hetero=True, probes=[(0, 0), (64, 2)]),
    'cable edges': dict(shape=64, hetero=True, probes=[31, 32]),
    'connections': dict(shape=150, conn=CONN, probes=[0, 77]),
    'apart': dict(shape=40, diffusion=False, probes=[0, 39], segment=1),
}


@pytest.mark.parametrize('case', CASES)
@pytest.mark.parametrize('precision', [SP, DP])
def test_route_and_columns(br77, decker, case, precision):
    for model, rl, fields in ((br77, False, ['isi.gsBar']),
                              (br77, True, ['ina.gNaBar']),
                              (decker, True, ['ina.Gbar'])):
        adj = _adjoint(model, precision, rl=rl, general=False,
                       fields=fields, **CASES[case])
        ak = _kernel(adj)
        if case == 'apart':
            # (no V that neighbours read: the general kernel)
            assert not ak.parts
            continue
        assert ak.parts == (4 if precision == SP else 8)
        text = ak.source()
        rows = text[text.index('mkg_adjoint_tape('):]
        # Every number is written once and read by one warp
        for t in range(ak.slots):
            want = f'tape + {t} * 32)'
            assert text.count('= __ldcg(' + want) == 3, t
        assert all(rows.count(f'tape[{t} * 32] =') <= 1
                   for t in range(ak.slots))
        assert not _kernel(_adjoint(model, precision, rl=rl, general=True,
                                    fields=fields, **CASES[case])).parts


def test_route_by_size(br77, decker):
    # Few warps per tile where many tiles share an SM, the general kernel
    # where two steps' numbers do not fit the registers and on large grids
    for model, precision, rows, parts in (
            (br77, SP, 152, 4), (br77, SP, 152 * 8, 2),
            (br77, SP, 152 * 9, 0), (br77, DP, 152 * 2, 8),
            (br77, DP, 152 * 4, 4), (br77, DP, 152 * 8, 2),
            (decker, SP, 152 * 2, 4), (decker, SP, 152 * 8, 0),
            (decker, SP, 4000, 0)):
        assert _kernel(_adjoint(model, precision, (32, rows), True, False,
                                probes=[(0, 0)])).parts == parts


def test_compiles(br77):
    ak = _kernel(_adjoint(br77, SP, (41, 7), True, False, hetero=True,
                          probes=[(0, 0)]))
    cubin, _ = _lib.compile_source(ak.source(), ak.options())
    assert ak.parts and cubin[:4] == b'\x7fELF'


@pytest.mark.gpu
@pytest.mark.parametrize('case', [c for c in CASES if c != 'apart'])
@pytest.mark.parametrize('precision,kw', [
    (DP, {}), (SP, {}), (SP, {'accumulate': 'double'})],
    ids=['fp64', 'fp32', 'double'])
def test_equals_general_kernel(br77, decker, case, precision, kw):
    models = [(br77, False, ['isi.gsBar', 'ina.gNaBar'])]
    models += [(br77, True, ['ina.gNaBar'])] if precision == DP else [
        (decker, True, ['ina.Gbar'])]
    if case == 'sheet' and precision == DP:
        models += [(decker, True, ['ina.Gbar'])]
    for model, rl, fields in models:
        out = []
        for general in (True, False):
            adj = _adjoint(model, precision, rl=rl, general=general,
                           fields=fields, **CASES[case], **kw)
            v = adj.forward(1.0, 0.13)
            w = np.cos(np.arange(v.size)).reshape(v.shape)
            out.append((v, adj.backward(w), adj.backward(w)))
        assert np.array_equal(out[0][0], out[1][0])
        for k, want in out[0][1].items():
            got = out[1][1][k]
            assert np.array_equal(got, out[1][2][k]), k
            far = np.max(np.abs(np.subtract(got, want)), initial=0)
            most = np.max(np.abs(want), initial=0)
            assert far <= (1e-11 if precision == DP else 1e-3) * most, k


@pytest.mark.gpu
def test_recorded_trajectory_is_recomputed_after_changes(br77):
    # The forward run leaves the last segment's trajectory for the backward
    # pass. Fields that a run changed in between apply to the backward pass,
    # with the general kernel and with this one
    out = []
    for general in (True, False):
        adj = _adjoint(br77, DP, 70, False, general, fields=['isi.gsBar'],
                       probes=[0, 69], segment=200)
        v = adj.forward(1.0, 0.13)
        w = np.cos(np.arange(v.size)).reshape(v.shape)
        before = adj.backward(w)['isi.gsBar']
        adj.sim.set_field('isi.gsBar', np.linspace(0.05, 0.12, 70))
        adj.sim.run(0.05)
        out.append((before, adj.backward(w)['isi.gsBar']))
    for a, b in zip(*out):
        assert np.max(np.abs(a - b)) <= 1e-11 * np.max(np.abs(a))
    assert not np.array_equal(*out[0]) and not np.array_equal(*out[1])
