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


@pytest.mark.parametrize('saved,team', [
    ({}, 4), ({'team': 0}, 0), ({'team': 2}, 2)])
def test_choices_saved_before_there_were_resident_tiles(br77, empty_cache,
                                                        saved, team):
    # An entry that names no team was chosen among other shapes only: it
    # does not keep a small grid off resident tiles. One that does stands
    def new():
        return mg.SimulationCUDA(br77, None, ncells=200)
    entry = dict({'block': [128, 1], 'min_blocks': 1, 'steps_per_launch': 0,
                  'stage_lazy': 0, 'sync': 'barrier', 'split': 4, 'rate': 1.0,
                  'when': 'test'}, **saved)
    if saved.get('team'):
        entry.update(block=[64, 1], split=1)
    with open(os.path.join(str(empty_cache), 'tune.json'), 'w') as f:
        json.dump({at.signature(new()): entry}, f)
    k = new()._kernel([])
    assert k.team == team
    if not team:
        assert k.block == (128, 1) and k.split == 4
    # Larger grids keep what was saved for them
    s = mg.SimulationCUDA(br77, None, ncells=(512, 512))
    with open(os.path.join(str(empty_cache), 'tune.json'), 'w') as f:
        json.dump({at.signature(s): dict(entry, block=[384, 1], split=1)}, f)
    if not saved.get('team'):
        assert s._kernel([]).block == (384, 1)
