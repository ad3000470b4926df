"""
Resident kernels: every warp tile is a CTA of 1 to 16 warps that keeps its
states in shared memory for a whole launch and exchanges V with its
neighbours word by word. The warps share the tile's equations without
dividing any, so the results are those of the undivided kernel bit for bit.
"""
import ctypes
import itertools

import numpy as np
import pytest

from conftest import myokit
import myokit_gb300 as mg
from myokit_gb300 import _lib, autotune, exporter

DP = myokit.DOUBLE_PRECISION
SP = myokit.SINGLE_PRECISION


# ---------------------------------------------------------------------------
# CPU: the division of the equations
# ---------------------------------------------------------------------------

def _kernel(model, precision, team, rl, **kw):
    s = mg.SimulationCUDA(model, None, ncells=(40, 3), precision=precision,
                          rl=rl, **kw)
    s._team = team
    return s._kernel([])


def _check_plan(k):
    """Every state is updated once; whatever a warp evaluates in a phase it
    has from the states, from its own earlier work or from a hand-over that
    one warp wrote in an earlier phase."""
    plan = k.team_plan
    n = k.team
    done = sorted([i for gs in plan.gates_of for g in gs for i in g] +
                  [i for g in plan.tails_of for i in g])
    assert done == list(range(k.n_state))
    lines = {}
    for lhs, rhs in k.cell_const_eqs + k.rhs_eqs:
        lines[k._name(lhs)] = set(k._name(r) for r in rhs.references())
    known = set(k._name(s) for s in k.states) | {
        't_', 'pace_', 'idiff_'} | set(k._name(f) for f in k.fields)
    have = [set(known) for _ in range(n)]
    there = {}               # hand-overs written so far
    for f in range(len(plan.work)):
        for w in range(n):
            assert all(x in there for x in plan.read[f][w])
            have[w] |= set(plan.read[f][w])
            for x in plan.work[f][w]:
                assert lines[x] <= have[w], (f, w, x)
                have[w].add(x)
            for i in plan.gates_of[f][w]:
                inf, tau = k.rl_states[k.states[i]]
                need = set(k._name(v) for v in (inf, tau)
                           if myokit.Name(v) not in k.literal_subst)
                if tau in k.rates:
                    need.discard(k._name(tau))
                    need |= set(k._name(r)
                                for r in k.rates[tau].references())
                assert need <= have[w], (f, w, i)
        for w in range(n):
            for x in plan.written[f][w]:
                assert x in have[w] and x not in there
                there[x] = w
    for w in range(n):
        for i in plan.tails_of[w]:
            assert k._name(k.states[i].lhs()) in have[w]
    assert set(there) == set(plan.slots)
    assert sorted(plan.slots.values()) == list(range(k.team_nslot))
    # V, which exchanges words with the neighbours, is the first warp's
    if k.diffusion:
        assert k.i_vm in plan.tails_of[0]


@pytest.mark.parametrize('team', [1, 2, 4, 8, 16])
@pytest.mark.parametrize('rl', [False, True])
@pytest.mark.parametrize('precision,kw', [
    (SP, {}), (DP, {}), (SP, {'accumulate': 'kahan'}),
    (SP, {'accumulate': 'double'}), (SP, {'diffusion': False})])
def test_plan(decker, br77, team, rl, precision, kw):
    for m in (decker, br77):
        k = _kernel(m, precision, team, rl, **kw)
        assert k.team == team and k.block == (32 * team, 1)
        assert k.n_state * 32 * (4 if k.single else 8) < k.resident_bytes()
        _check_plan(k)
        if team > 1 and m is decker:
            # the work is shared: no warp has more than twice its part
            whole = _kernel(m, precision, 1, rl, **kw).team_plan.cost[0][0]
            assert all(max(c) <= max(2 * whole / team, 160)
                       for c in k.team_plan.cost)


@pytest.mark.parametrize('team', [1, 2, 4])
def test_equations_that_are_alike(decker, team):
    # The three calcium buffers are one function, called with the
    # arguments of each (a single warp has its code to itself)
    k = _kernel(decker, SP, team, True)
    names = ['ca_cal', 'ca_i', 'ca_jsr']
    calls = [k.repeated.get('v_' + n) for n in names]
    if team == 1:
        assert not k.functions and not any(calls)
        return
    assert len(k.functions) == 1 and ' mkg_equation_0(' in k.functions[0]
    text = k.source()
    for n, call in zip(names, calls):
        assert call == 'mkg_equation_0(%s)' % ', '.join(
            'v_%s_%s' % (n, x) for x in 'bcd')
        assert text.count(call) >= 1


def test_when_neighbours_are_asked(decker, br77):
    # In a long first phase the words are asked for on the way and the
    # current is taken before the team meets; else they are asked for at the
    # start of a step and the current is taken in the last phase
    for m, rl, precision, team, soon in (
            (decker, True, SP, 4, True), (decker, True, SP, 1, False),
            (br77, False, SP, 4, False), (br77, False, DP, 8, True),
            (decker, True, SP, 16, False), (decker, True, DP, 16, True)):
        k = _kernel(m, precision, team, rl)
        assert k.team_plan.halo_first == soon
        body = k.team_body
        body = body[:body.index('else if (part_') if team > 1 else None]
        # (after the log row's own copy)
        rest = body[body.index('MKG_CHECK_HALT'):]
        meets = rest.index('mkg_team_sync();')
        assert rest.count('MKG_HALO(id_)') == 1
        assert rest.count('MKG_HALO_ASK()') == int(soon)
        if soon:
            assert rest.index('MKG_HALO_ASK()') < \
                rest.index('MKG_HALO(id_)') < meets
        else:
            assert body.index('MKG_HALO_ASK()') < body.index('row >= 0')
            assert team == 1 or rest.index('MKG_HALO(id_)') > meets


@pytest.mark.parametrize('precision', [SP, DP])
def test_compiles(decker, precision):
    k = _kernel(decker, precision, 16, True)
    cubin, _ = _lib.compile_source(k.source(), k.options())
    assert cubin[:4] == b'\x7fELF'


def test_shape_by_size():
    shape = autotune.resident_shape
    for single, most in ((True, 16), (False, 8)):
        for tiles in (1, 152, 153, 304, 608, 609, 912, 1216):
            team, minb = shape(tiles, 152, single)
            assert tiles <= minb * 152 and team * minb <= 16
        assert shape(152 * most, 152, single) == (1, most)
        assert shape(152 * most + 1, 152, single) is None


def test_shape_of_small_models(br77, decker):
    # Fewer than 16 states in double precision: code for many warps
    for tiles, want in ((7, (8, 1)), (152 * 4, (8, 4)), (152 * 4 + 1, (4, 5)),
                        (152 * 8, (4, 8)), (152 * 8 + 1, None)):
        assert autotune.resident_shape(tiles, 152, False, 8) == want
        k = mg.SimulationCUDA(br77, None, ncells=32 * tiles,
                              precision=DP)._kernel([])
        assert k.team == (want[0] if want else 0)
        assert not want or k.team_plan.halo_first
    k = mg.SimulationCUDA(decker, None, ncells=32 * 500, precision=DP,
                          rl=True)._kernel([])
    assert k.team == 2


def test_launch_shape_of_large_grids(decker, br77):
    for m, rl, precision, n, kw, want in (
            (decker, True, SP, (512, 512), {}, (256, 2, 0, 'barrier')),
            (decker, True, SP, (1024, 1024), {}, (512, 1, 0, 'neighbors')),
            (decker, True, SP, (800, 790), {'accumulate': 'kahan'},
             (512, 1, 0, 'neighbors')),
            (decker, True, DP, (512, 512), {}, (64, 4, 1, 'barrier')),
            (br77, False, DP, (512, 512), {}, (512, 1, 1, 'barrier')),
            (br77, False, SP, (512, 512), {}, (256, 2, 0, 'barrier'))):
        s = mg.SimulationCUDA(m, None, ncells=n, precision=precision, rl=rl,
                              **kw)
        k = s._kernel([])
        assert (k.block[0], k.min_blocks, k.stage_lazy, k.sync) == want
        assert k.layout and not k.team
        # An explicit launch shape is taken as before
        s = mg.SimulationCUDA(m, None, ncells=n, precision=precision, rl=rl,
                              block=96, min_blocks=1, **kw)
        k = s._kernel([])
        assert (k.block[0], k.min_blocks, k.stage_lazy, k.sync) == (
            96, 1, 0, 'barrier')


def test_launch_shape_between_resident_and_memory_bound(decker, br77):
    # 60 tiles per SM: many rounds of tiles per warp, planes still in L2
    for m, rl, n, want in (
            (decker, True, (640, 457), (512, 1, 0, 'neighbors')),
            (decker, True, (640, 455), (256, 2, 0, 'barrier')),
            (decker, True, 292000, (512, 1, 0, 'neighbors')),
            (br77, False, (640, 457), (256, 2, 0, 'barrier'))):
        k = mg.SimulationCUDA(m, None, ncells=n, precision=SP,
                              rl=rl)._kernel([])
        assert (k.block[0], k.min_blocks, k.stage_lazy, k.sync) == want


def test_large_models_and_launch_options_are_not_resident(br77):
    s = mg.SimulationCUDA(br77, None, ncells=64)
    assert s._kernel([]).team == 4
    s = mg.SimulationCUDA(br77, None, ncells=64, precision=DP)
    assert s._kernel([]).team == 8
    for kw in ({'block': 128}, {'min_blocks': 2}):
        assert mg.SimulationCUDA(br77, None, ncells=64,
                                 **kw)._kernel([]).team == 0
    for name, v in (('_split', 2), ('_sync', 'barrier'), ('_stage_lazy', 0)):
        s = mg.SimulationCUDA(br77, None, ncells=64)
        setattr(s, name, v)
        assert s._kernel([]).team == 0
    assert mg.SimulationCUDA(br77, None,
                             ncells=(512, 512))._kernel([]).team == 0


def test_create_validates_team():
    lib = _lib.load()
    for team, block, stage, split, ok in (
            (4, 128, 0, 1, True), (4, 256, 0, 1, False),
            (3, 96, 0, 1, False), (32, 1024, 0, 1, False),
            (4, 128, 1, 1, False), (4, 128, 0, 4, False)):
        h = ctypes.c_void_p()
        cfg = _lib.MkgConfig()
        cfg.nx, cfg.ny, cfg.real_bytes, cfg.n_state = 200, 1, 8, 8
        cfg.block_x, cfg.block_y = block, 1
        cfg.team, cfg.stage, cfg.split = team, stage, split
        code = lib.mkg_create(ctypes.byref(cfg), b'x', 1, ctypes.byref(h))
        assert code != _lib.MKG_OK
        assert (b'resident' not in lib.mkg_last_error(None)) == ok


# ---------------------------------------------------------------------------
# GPU
# ---------------------------------------------------------------------------

def _run(model, team, shape, precision, rl, conn=None, hetero=False,
         fields=(), paced=None, log=(), spl=0, diffusion=True, nan=None,
         dur=2.0, **kw):
    p = myokit.pacing.blocktrain(period=1000, duration=2, level=1)
    s = mg.SimulationCUDA(model, p, ncells=shape, precision=precision, rl=rl,
                          diffusion=diffusion, steps_per_launch=spl, **kw)
    s._team = team
    if not team:
        s._block = (64, 1)
    s.set_step_size(0.01)
    rng = np.random.default_rng(3)
    sh = shape[::-1] if isinstance(shape, tuple) else (shape,)
    if hetero and len(sh) == 2:
        s.set_conductance_field(rng.uniform(4, 9, (sh[0], sh[1] - 1)),
                                rng.uniform(2, 5, (sh[0] - 1, sh[1])))
    elif hetero:
        s.set_conductance_field(rng.uniform(4, 9, sh[0] - 1))
    if conn is not None:
        s.set_connections(conn)
    if paced is not None:
        s.set_paced_cell_list(paced)
    elif diffusion:
        s.set_paced_cells(3, sh[0])
    for f in fields:
        s.set_field(f, s._model.get(f).eval() * rng.lognormal(0, 0.2, sh))
    st = s.state_array().reshape(-1, s._nstate)
    st *= 1 + 0.01 * rng.standard_normal((len(st), 1))
    if nan is not None:
        st[nan] = np.nan
    s.set_state(st.reshape(-1))
    d = s.run(dur, log=['engine.time'] + list(log), log_interval=0.23,
              report_nan=False)
    assert s._last_kernel.team == team
    return s.state_array(), {k: np.asarray(v) for k, v in d.items()}


def _same(a, b):
    assert np.array_equal(a[0], b[0], equal_nan=True)
    assert a[1].keys() == b[1].keys()
    for k in a[1]:
        assert np.array_equal(a[1][k], b[1][k], equal_nan=True), k


@pytest.mark.gpu
@pytest.mark.parametrize('precision,kw', [
    (SP, {}), (DP, {}), (SP, {'accumulate': 'kahan'}),
    (SP, {'accumulate': 'double'})], ids=['fp32', 'fp64', 'kahan', 'double'])
@pytest.mark.parametrize('shape', [(70, 9), (33, 4), (96, 3), 1, 65, 200])
def test_equals_undivided(decker, precision, kw, shape):
    two_d = isinstance(shape, tuple)
    log = ['0.0.membrane.V', '5.2.ina.m'] if two_d else ['0.membrane.V']
    want = _run(decker, 0, shape, precision, True, log=log, **kw)
    for team in (1, 2, 4, 8, 16):
        _same(want, _run(decker, team, shape, precision, True, log=log, **kw))


@pytest.mark.gpu
@pytest.mark.parametrize('team', [1, 4, 16])
@pytest.mark.parametrize('precision', [SP, DP])
def test_modes_equal_undivided(br77, decker, team, precision):
    # Per-edge conductances, fields, paced lists, connections with more
    # than four neighbours (inside and outside a tile), no diffusion,
    # several launches, logged intermediaries and the diffusion current
    cases = [
        (decker, (41, 7), True, dict(hetero=True, fields=['ikr.Gbar'])),
        (br77, 130, False, dict(hetero=True, fields=['isi.gsBar'],
                                paced=[0, 1, 64, 129])),
        (br77, 150, False, dict(conn=[
            (i, j, 0.5 + (i * j) % 3) for i, j in itertools.combinations(
                range(150), 2) if j - i in (1, 2, 31, 33, 64)],
            paced=[0, 40])),
        (br77, 100, False, dict(diffusion=False)),
        (br77, (40, 40), False, dict(spl=7)),
        (br77, (9, 5), False, dict(log=['3.3.isi.Isi', '0.0.ina.m',
                                        '8.4.membrane.i_diff'])),
        (decker, (1, 40), True, dict(log=['0.39.membrane.V'])),
    ]
    for m, shape, rl, kw in cases:
        _same(_run(m, 0, shape, precision, rl, **kw),
              _run(m, team, shape, precision, rl, **kw))


@pytest.mark.gpu
@pytest.mark.parametrize('team', [2, 16])
@pytest.mark.parametrize('spl', [0, 7])
def test_nan_halt(br77, team, spl):
    # Cell 0 becomes NaN by diffusion from a far cell: the run halts at the
    # log point that sees it, all tiles after the same step
    log = ['0.membrane.V', '90.membrane.V']
    out = [_run(br77, t, 100, DP, False, nan=3, log=log, spl=spl, dur=1.0)
           for t in (0, team)]
    _same(*out)
    assert np.isnan(out[0][1]['0.membrane.V'][-1])
    assert len(out[0][1]['engine.time']) < 4


@pytest.mark.gpu
def test_wait_runs_out(decker):
    # A wait that nothing satisfies ends within its bound and leaves the
    # handle usable (the hook raises every target)
    p = myokit.pacing.blocktrain(period=1000, duration=2, level=1)
    s = mg.SimulationCUDA(decker, p, ncells=(64, 8), rl=True)
    ref = s.run(0.5, log=['engine.time', '0.0.membrane.V'], log_interval=0.1)
    assert s._last_kernel.team
    st = s.state_array()
    be = s._backend[1]
    s.reset()
    assert be.lib.mkg_set_wait(be.h, 20000000, 1000) == 0
    with pytest.raises(_lib.MkgError) as e:
        s.run(0.5, log=['engine.time', '0.0.membrane.V'], log_interval=0.1)
    assert e.value.code == _lib.MKG_ERR_TIMEOUT
    assert be.lib.mkg_set_wait(be.h, 2000000000, 0) == 0
    s.reset()
    d = s.run(0.5, log=['engine.time', '0.0.membrane.V'], log_interval=0.1)
    assert np.array_equal(s.state_array(), st)
    for k in ref:
        assert np.array_equal(np.asarray(ref[k]), np.asarray(d[k]))


@pytest.mark.gpu
@pytest.mark.parametrize('precision,acc', [(DP, None), (SP, 'double'),
                                           (SP, 'kahan')])
def test_adjoint_of_a_resident_simulation(decker, precision, acc):
    from myokit_gb300 import adjoint
    out = []
    for team in (0, 16):
        p = myokit.pacing.blocktrain(period=1000, duration=2, level=1)
        s = mg.SimulationCUDA(decker, p, ncells=(41, 3), rl=True,
                              precision=precision, accumulate=acc)
        s._team = team
        s.set_step_size(0.01)
        s.set_paced_cells(3, 3)
        s.set_field('ina.Gbar', np.full((3, 41),
                                        s._model.get('ina.Gbar').eval()))
        adj = adjoint.TissueAdjoint(s, [(0, 0), (40, 2)], segment_steps=30)
        v = adj.forward(0.7, 0.1)
        out.append((v, adj.backward(np.ones_like(v))))
    assert np.array_equal(out[0][0], out[1][0])
    for k in ('ina.Gbar', 'gx', 'gy'):
        assert np.array_equal(out[0][1][k], out[1][1][k]), k
