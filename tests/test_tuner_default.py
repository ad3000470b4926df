"""
What the launch-shape tuner times and what it saved: never less than the
shape that a simulation takes without it.
"""
import json
import os

import pytest

from conftest import myokit
import myokit_gb300 as mg
from myokit_gb300 import autotune as at

SP = myokit.SINGLE_PRECISION
DP = myokit.DOUBLE_PRECISION


@pytest.fixture
def empty_cache(tmp_path, monkeypatch):
    monkeypatch.setenv('MYOKIT_GB300_CACHE', str(tmp_path))
    return tmp_path


@pytest.mark.parametrize('precision', [SP, DP])
def test_candidates_hold_the_default_shape(decker, br77, empty_cache,
                                           precision):
    for m, rl in ((decker, True), (br77, False)):
        for n in (200, (300, 300), (512, 512), (640, 520), (2048, 2048)):
            s = mg.SimulationCUDA(m, None, ncells=n, precision=precision,
                                  rl=rl)
            k = s._kernel([])
            timed = at._candidates(s) + at._resident_candidates(s)
            assert any(
                c[0] == k.block and c[1] == k.min_blocks and
                (c[6:] or (0,))[0] == k.team and (k.team or (
                    int(c[3]) == k.stage_lazy and c[4] == k.sync and
                    (c[5:] or (1,))[0] == 1))
                for c in timed), (n, k.block, k.min_blocks)
            assert len(set(timed)) == len(timed)
