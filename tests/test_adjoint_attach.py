"""
An adjoint whose attachment failed is not attached: nothing runs with some of
its kernels and buffers and some of the last one's.
"""
import ctypes

import numpy as np
import pytest

from conftest import myokit
import myokit_gb300 as mg
from myokit_gb300 import _lib, adjoint
from myokit_gb300.simulation import compile_kernel

DP = myokit.DOUBLE_PRECISION


def test_order_of_calls_without_a_device():
    lib = _lib.load()
    n = ctypes.c_int64()
    assert lib.mkg_adj_forward(None, 0.0, 1.0, 0.1, 1.0,
                               ctypes.byref(n)) == _lib.MKG_ERR_ARG


@pytest.mark.gpu
def test_failed_attachment(br77):
    def new(threads):
        s = mg.SimulationCUDA(br77, myokit.pacing.blocktrain(
            period=1000, duration=2, level=1), ncells=70, precision=DP)
        s.set_step_size(0.01)
        s.set_field('isi.gsBar', np.full(70, 0.08))
        return adjoint.TissueAdjoint(s, [0, 69], threads=threads)
    sweep = new(None)
    kernel = sweep.sim._kernel([])
    ak = sweep._make(kernel, sweep._tiles_per_sm(kernel))
    assert ak.parts
    cubin = compile_kernel(ak)
    adj = new(64)
    v = adj.forward(1.0, 0.25)
    want = adj.backward(np.ones_like(v))
    be = adj.sim._backend[1]
    # (a sweep of another CTA size than its kernel's is refused)
    assert be.lib.mkg_adj_attach_map(be.h, cubin, len(cubin), 50, ak.slots,
                                     ak.parts * 2) == _lib.MKG_ERR_ARG
    for f in (lambda: adj.backward(np.ones_like(v)),
              lambda: adj.forward(1.0, 0.25)):
        with pytest.raises(_lib.MkgError) as e:
            f()
        assert e.value.code == _lib.MKG_ERR_ORDER
    # Attached again, all is as before; and a new attachment forgets the
    # forward run of the last
    adj._attached = None
    assert np.array_equal(adj.forward(1.0, 0.25), v)
    got = adj.backward(np.ones_like(v))
    assert got.keys() == want.keys()
    assert all(np.array_equal(got[k], want[k]) for k in want)
    adj._attached = None
    with pytest.raises(_lib.MkgError):
        adj.backward(np.ones_like(v))
