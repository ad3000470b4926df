"""
The adjoint on sheets whose rows are not whole warps: the lanes past the end
of a row hold no cell and must not record a trajectory (a staged tile is read
by every lane of the warp, and those lanes' cell numbers are the next row's).
"""
import re

import numpy as np
import pytest

from conftest import myokit
import myokit_gb300 as mg
from myokit_gb300 import adjoint, exporter


def _sim(model, shape, **kw):
    p = myokit.pacing.blocktrain(period=1000, duration=2, level=1)
    s = mg.SimulationCUDA(model, p, ncells=shape, rl=True,
                          precision=myokit.DOUBLE_PRECISION, **kw)
    s.set_step_size(0.01)
    s.set_paced_cells(3, shape[1])
    s.set_field('ina.Gbar', np.full(shape[::-1],
                                    s._model.get('ina.Gbar').eval()))
    return s


@pytest.mark.parametrize('lazy', [0, 1, 2])
def test_trajectory_is_recorded_by_live_lanes_only(decker, lazy):
    s = _sim(decker, (31, 17))
    s._stage_lazy = lazy
    k = s._kernel([])
    assert k.layout
    fwd = exporter.TissueKernel(
        s._model, s._precision, s._native_math, s._bound_variables, [],
        k.diffusion, k.two_d, list(s._fields.keys()), s._rl_states, k.block,
        traj=True, stage=k.stage, row_pad=k.row_pad, stage_lazy=lazy)
    src = fwd.source()
    stores = [m.start() for m in re.finditer(r'\(Real \*\)a\.traj', src)]
    assert len(stores) == k.n_state
    start = src.index('            if (live) {\n#if !STAGE || STAGE_LAZY')
    assert all(i > start for i in stores)


@pytest.mark.gpu
@pytest.mark.parametrize('nx', [31, 33, 64])
def test_gradients_of_ragged_rows(decker, nx):
    # Staged and direct loads, twice: the same gradients
    out = []
    for stage in (True, True, False):
        s = _sim(decker, (nx, 17), stage_tiles=stage)
        adj = adjoint.TissueAdjoint(s, [(0, 0), (5, 3), (nx - 1, 16)])
        v = adj.forward(0.4, 0.1)
        out.append(adj.backward(np.ones_like(v)))
    for a in out[:2]:
        for k in ('ina.Gbar', 'gx', 'gy'):
            r = np.asarray(out[2][k])
            # (the two kernels may contract different multiply-adds)
            assert np.max(np.abs(np.asarray(a[k]) - r)) <= \
                1e-9 * np.max(np.abs(r)), k
    assert np.array_equal(out[0]['ina.Gbar'], out[1]['ina.Gbar'])
