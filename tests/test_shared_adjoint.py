"""
Reverse kernels are shared by everything that they are generated from, the
CTA size among it.
"""
from conftest import myokit
import myokit_gb300 as mg
from myokit_gb300 import _lib, adjoint, simulation

DP = myokit.DOUBLE_PRECISION


def test_reverse_kernel_of_an_explicit_block(br77, monkeypatch):
    # Two simulations with the same forward kernel, one of them with the
    # default launch shape given: each has the reverse kernel of its own CTA
    # size, whichever was generated first
    made = []
    monkeypatch.setattr(simulation, '_KERNELS', type(simulation._KERNELS)())
    monkeypatch.setattr(simulation, 'compile_kernel',
                        lambda ak: made.append(ak) or b'')

    class Handle(object):
        lib, h = _lib.load(), None

        def check(self, code):
            return code

    def reverse(**kw):
        s = mg.SimulationCUDA(br77, None, ncells=(512, 512), precision=DP,
                              stage_tiles=False, **kw)
        monkeypatch.setattr(s, '_get_backend', lambda kernel: Handle())
        adjoint.TissueAdjoint(s, [(0, 0)])._prepare()
        return s._kernel([]).key(), made[-1].threads

    given = dict(block=512, min_blocks=1)
    for order in ((given, {}), ({}, given)):
        simulation._KERNELS.clear()
        out = [reverse(**kw) for kw in order]
        assert out[0][0] == out[1][0]
        assert [t for _, t in out] == [512 if kw else 256 for kw in order]
