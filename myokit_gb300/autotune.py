"""
Launch-shape autotuner for :class:`SimulationCUDA`.

The fused kernel's speed depends on the CTA size, on the register cap that
the minimum number of resident CTAs per SM implies, and on how steps are
grouped into launches (one cooperative launch per chunk with a grid barrier
between steps, or one plain launch per step replayed from a CUDA graph).
:func:`autotune` times candidates on the simulation itself -- same model,
grid, fields and precision -- and keeps the fastest. Results are cached per
configuration signature in ``<cache dir>/tune.json``; a simulation created
with ``block=None`` uses a cached result when one matches.
"""
import json
import os
import time

import numpy as np

from ._deps import myokit

# Candidate (threads per CTA, min CTAs per SM, steps per launch, tile
# staging, step synchronisation). The register cap is 64K / (threads * min
# CTAs), and a warp scheduler holds 16K registers. 576 and 640 threads trade
# registers for the 18 or 20 warps per SM that even out the warp tiles of
# mid-size sheets. Staging 0 prefetches each tile into registers; 1 and 2
# read it from shared memory where used (lazy), which keeps those kernels
# from spilling, with one or two buffers per warp (2: the copies of the
# tile after the next overlap a tile's computation). Steps are separated by
# a grid barrier or by waits on the neighbouring warps only.
_B, _N = 'barrier', 'neighbors'
_CANDIDATES = [
    ((256, 1), 2, 0, False, _B), ((128, 1), 4, 0, False, _B),
    ((512, 1), 1, 0, False, _B), ((192, 1), 3, 0, False, _B),
    ((384, 1), 1, 0, False, _B), ((640, 1), 1, 0, False, _B),
    ((128, 1), 1, 0, False, _B), ((256, 1), 2, 1, False, _B),
    ((512, 1), 1, 0, True, _B), ((576, 1), 1, 0, True, _B),
    ((640, 1), 1, 0, True, _B), ((256, 1), 2, 0, True, _B),
    ((384, 1), 1, 0, True, _B),
    ((512, 1), 1, 0, False, _N), ((384, 1), 1, 0, False, _N),
    ((256, 1), 2, 0, False, _N), ((640, 1), 1, 0, True, _N),
    ((256, 1), 2, 0, True, _N),
    ((256, 1), 2, 0, 2, _B), ((384, 1), 1, 0, 2, _N),
]
# (double precision: the shapes of default_shape among them)
_CANDIDATES_FP64 = [((128, 1), 1, 0, False, _B), ((256, 1), 1, 0, False, _B),
                    ((64, 1), 1, 0, False, _B), ((32, 1), 1, 0, False, _B),
                    ((256, 1), 1, 0, True, _B), ((256, 1), 1, 0, False, _N),
                    ((64, 1), 4, 0, True, _B), ((512, 1), 1, 0, True, _B)]
# Grids with fewer warp tiles than SMs: teams of 2 to 16 warps share each
# tile's work (a sixth entry: warps per tile): one team per CTA or two, or
# one team per cluster of 2 or 4 CTAs
_CANDIDATES_SPLIT = [((64, 1), 1, 0, False, _B, 2),
                     ((128, 1), 1, 0, False, _B, 4),
                     ((128, 1), 1, 0, False, _B, 2),
                     ((256, 1), 1, 0, False, _B, 4),
                     ((128, 1), 1, 0, False, _B, 8),
                     ((128, 1), 1, 0, False, _B, 16)]


def _cache_path():
    from .simulation import _cache_dir
    return os.path.join(_cache_dir(), 'tune.json')


def _shipped_path():
    return os.path.join(os.path.dirname(os.path.abspath(__file__)),
                        'tuned.json')


def signature(sim):
    """A string identifying what the best launch shape depends on."""
    import hashlib
    code = hashlib.sha1(sim.model_code().encode()).hexdigest()[:16]
    return '|'.join(str(x) for x in (
        sim._model.name(), code, sim._nx, sim._ny, len(sim._dims),
        sim._precision, sim._accumulate, sim._diffusion_mode(),
        ','.join(v.qname() for v in sim._fields), len(sim._rl_states),
        sim._fp32_math, sim._native_math,
        'staged' if sim._stage_tiles else 'direct'))


def _load(path):
    try:
        with open(path) as f:
            return json.load(f)
    except (OSError, ValueError):
        return {}


def lookup(sim):
    """The cached choice for this simulation's signature, or None."""
    sig = signature(sim)
    for path in (_cache_path(), _shipped_path()):
        d = _load(path)
        if sig in d:
            return d[sig]
    return None


def resident_shape(tiles, sms, single, n_state=16):
    """
    ``(warps per tile, CTAs per SM)`` of a resident kernel
    (``csrc/resident_kernel.cu.in``) for a grid of ``tiles`` warp tiles, or
    None where the tiles do not fit on ``sms`` SMs at once.

    The more warps share a tile the shorter is its own step, and the more
    code an SM has to fetch. Measured, us per step with 1 / 2 / 4 / 8 warps
    per tile and (last) the undivided kernel, by tiles on an SM:

    - 48 states, single precision: one tile 3.0 / 2.3 / 1.7 / 1.7, 5.3;
      four 3.0 / 2.2 / 1.9 / 2.8, 5.3; six 3.4 / 2.4 / 2.5, 5.3; eight
      3.5 / 2.9 / 3.3, 5.5; twelve 4.1 / 4.5, 7.2; sixteen 5.5 / 6.7, 7.4;
    - the same in double precision: one tile 73 / 36 / 21 / 15, 83; two
      73 / 36 / 23 / 51, 84; three 73 / 40 / 35 / 44, 84; four 74 / 41 / 51,
      85; six 79 / 57 / 74, 85; eight 81 / 77, 95;
    - 8 states, single precision: one 0.94 / 0.85 / 0.87 / 0.90, 2.3; eight
      1.05 / 0.88 / 1.00, 2.4; sixteen 1.3 / 2.0, 3.0;
    - the same in double precision: one 12.2 / 6.9 / 4.1 / 2.7, 13.4; two
      12.2 / 6.9 / 4.5 / 3.2, 13.4; four 12.5 / 8.4 / 6.3 / 5.3, 13.6; five
      13.6 / 8.9 / 7.0, 16.3; eight 14.3 / 11.2 / 10.3, 16.5. Its code is
      small enough for many warps (fewer than 16 states).

    Nine tiles on an SM in double precision take 100 us with the 48 states,
    the undivided kernel 94: its 8 warps per SM have the registers they need.
    """
    per = -(-tiles // sms)
    for team, most in ((4, 4), (2, 8), (1, 16)) if single else (
            (8, 4), (4, 8)) if n_state < 16 else (
            (8, 1), (4, 3), (2, 7), (1, 8)):
        if per <= most:
            return team, per
    return None


def default_shape(single, n_state, plane_bytes, tiles_per_sm):
    """
    The launch shape of a grid too large for resident tiles, where nobody
    chose one: ``(threads, CTAs per SM, lazy staging, synchronisation)``.
    ``plane_bytes``: the states and accumulation planes of all cells.

    Measured, us per step:

    - single precision, planes beyond the L2 (129 MB): 512 threads with
      neighbour waits, 48 states: 2048 x 2048 Kahan 366 against 417 with 256
      x 2 and the grid barrier, 1024 x 1024 Kahan 86 and 104, 1531 x 777 86
      and 101; 8 states 2048 x 2048 74 and 74. The many tiles of a warp
      even out what neighbours wait for, and no warp idles at a barrier
      while memory does;
    - many states, 60 tiles per SM and more, planes in the L2: the same (48
      states, 640 x 520 25.8 against 27.8, Kahan 28.5 and 29.7, per-edge
      Kahan 32.3 and 32.9, FP64 accumulation 54.6 and 54.6; 800 x 700 41.6
      and 44.6, Kahan 46.8 and 54.2);
    - else 256 x 2 with the barrier (512 x 512, 54 tiles per SM, 20.9
      against 20.7, Kahan 22.4 and 22.6, per-edge 23.1 and 23.9, FP64
      accumulation 41.4 and 43.0; 8 states 640 x 520 8.0 and 8.2, 512 x 512
      6.4 and 7.1, 290 x 290 4.0 and 4.7: their steps are too short to hide
      the neighbours' counters). With many states neither is always ahead
      there: barrier and neighbours, plain, Kahan, FP64 accumulation and
      per-edge, 256 x 256 7.3 and 7.4, 8.0 and 8.3, 13.9 and 14.1, 7.5 and
      7.7; 320 x 320 11.3 and 10.9, 12.3 and 12.1, 20.4 and 19.9, 11.7 and
      11.3; 400 x 400 16.0 and 15.5, 17.4 and 17.5, 30.3 and 30.4, 16.5 and
      16.3; 448 x 448 17.5 and 16.7, 19.1 and 18.3, 33.6 and 33.1, 18.0 and
      17.4; 512 x 512 20.9 and 20.8, 22.7 and 23.1, 42.2 and 42.6, 21.5 and
      21.7;
    - double precision, many states: 8 warps per SM of 64-thread CTAs, read
      from shared memory where used: 256 x 256 114 against 180 with 128
      threads and prefetch, 301 x 211 119 and 182, 512 x 512 491 and 676;
    - double precision, few states (registers do not limit the warps): 512
      threads, 512 x 512 with 8 states 79 against 85; 64-thread CTAs 100.
    """
    if not single:
        return (64, 4, 1, 'barrier') if n_state >= 16 else (
            512, 1, 1, 'barrier')
    if plane_bytes > 120e6 or (tiles_per_sm >= 60 and n_state >= 16):
        return 512, 1, 0, 'neighbors'
    return 256, 2, 0, 'barrier'


def _apply(sim, block, min_blocks, spl, lazy=False, sync='barrier',
           split=1, team=0):
    sim._block = tuple(block)
    sim._min_blocks = int(min_blocks)
    sim._steps_per_launch = int(spl)
    sim._stage_lazy = int(lazy)
    sim._sync = sync
    sim._split = int(split)
    sim._team = int(team)
    sim._graphs = 1


def _sm_count(device):
    """SMs of a CUDA device (152 on a GB300, taken when it cannot be
    read)."""
    try:
        import torch
        if torch.cuda.is_available():
            return int(torch.cuda.get_device_properties(
                device).multi_processor_count)
    except Exception:   # pragma: no cover
        pass
    return 152


def _few_tiles(sim):
    """True when the grid has fewer warp tiles than the device has SMs."""
    tiles = -(-sim._nx // 32) * sim._ny
    return tiles < _sm_count(sim._device)


def _candidates(sim):
    """The launch configurations the tuner times on ``sim``."""
    double = sim._precision == myokit.DOUBLE_PRECISION
    # FP64 kernels spill when registers are capped
    out = list(_CANDIDATES_FP64 if double else _CANDIDATES)
    if _few_tiles(sim) and sim._accumulate is None:
        # Cluster teams (more warps per tile than the CTA holds) pay where
        # a tile's double precision instructions bind; a single precision
        # small grid is bound by the step's latency, and its cluster
        # barrier only costs (200-cell cable: 0.074 and 0.065 against
        # 0.098e9 cell-steps/s)
        out += [c for c in _CANDIDATES_SPLIT
                if double or c[5] <= c[0][0] // 32]
    return out


def _resident_candidates(sim):
    """The resident shapes to time on ``sim``: that of its size."""
    two_d = len(sim._dims) == 2 and sim._diffusion_mode() in (1, 2)
    nx, ny = (sim._nx, sim._ny) if two_d else (sim._ntotal, 1)
    shape = resident_shape(-(-nx // 32) * ny, _sm_count(sim._device),
                           sim._precision == myokit.SINGLE_PRECISION,
                           sim._nstate)
    if shape is None:
        return []
    team, minb = shape
    return [((32 * team, 1), minb, 0, False, _N, 1, team)]


def autotune(sim, duration=None, candidates=None, store=True,
             verbose=False):
    """
    Times each candidate launch configuration on ``sim`` for ``duration``
    time units (default: about 4e8 cell-steps) without logging, restores the
    simulation's state and time, applies the fastest configuration and
    returns ``(best, results)``. ``results`` maps each candidate to its
    cell-steps per second of device time.
    """
    if candidates is None:
        candidates = _candidates(sim) + _resident_candidates(sim)
    if duration is None:
        steps = max(20, int(4e8 / sim._ntotal))
        if sim._precision == myokit.DOUBLE_PRECISION:
            steps = max(4, steps // 20)
        duration = steps * sim.step_size()
    saved = (sim._state.copy(), sim._time, sim._block, sim._min_blocks,
             sim._steps_per_launch, sim._graphs, sim._stage_lazy, sim._sync,
             sim._split, sim._team)
    results = {}
    try:
        for cand in candidates:
            _apply(sim, *cand)
            block, mb, spl = cand[:3]
            sim._state = saved[0].copy()
            sim._time = saved[1]
            try:
                sim._run(duration / 4, myokit.LOG_NONE, 1, False, None, '')
                sim._state = saved[0].copy()
                sim._run(duration, myokit.LOG_NONE, 1, False, None, '')
            except Exception as e:   # pragma: no cover
                if verbose:
                    print('autotune: %s failed: %s' % (cand, e))
                continue
            st = sim.last_run_stats()
            rate = st['cell_steps'] / (st['kernel_ms'] / 1000.0)
            results[cand] = rate
            if verbose:
                print('autotune: block=%s min_blocks=%d steps/launch=%d'
                      ' -> %.4g cell-steps/s' % (block, mb, spl, rate))
    finally:
        sim._state, sim._time = saved[0], saved[1]
        sim._block, sim._min_blocks = saved[2], saved[3]
        sim._steps_per_launch, sim._graphs = saved[4], saved[5]
        sim._stage_lazy, sim._sync = saved[6], saved[7]
        sim._split, sim._team = saved[8], saved[9]
    if not results:
        return None, results
    best = max(results, key=results.get)
    _apply(sim, *best)
    sim._tuned = True
    if store:
        path = _cache_path()
        d = _load(path)
        d[signature(sim)] = {
            'block': list(best[0]), 'min_blocks': best[1],
            'steps_per_launch': best[2],
            'stage_lazy': int(best[3]) if len(best) > 3 else 0,
            'sync': best[4] if len(best) > 4 else 'barrier',
            'split': best[5] if len(best) > 5 else 1,
            'team': best[6] if len(best) > 6 else 0,
            'rate': results[best],
            'when': time.strftime('%Y-%m-%dT%H:%M:%S')}
        try:
            os.makedirs(os.path.dirname(path), exist_ok=True)
            tmp = path + '.%d' % os.getpid()
            with open(tmp, 'w') as f:
                json.dump(d, f, indent=1, sort_keys=True)
            os.replace(tmp, path)
        except OSError:   # pragma: no cover
            pass
    return best, results
