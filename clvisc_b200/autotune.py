"""Autotuner of the fused viscous stage's launch shape for one event.

The first candidate is the library's own choice (kernel 0, chunk 0): patches on
(2+1)D grids, tiles with the x planes per block chosen from the grid where eta
has 24 cells or more, one thread per cell between. The others: the tiled kernel's
(y, eta) tiles from its compile-time set (8 x 32, 16 x 16, 8 x 16, CLV_OPT_TILE)
and x extents per block (CLV_OPT_CHUNK), the marching (2+1)D kernel, and one
thread per cell. In the exact build every variant computes the same bits; in the
tolerance build the variants differ within its tolerance (1e-5 FP32, 1e-11 FP64),
so there the choice, which hangs on timings, enters the last bits of a run.
tune_visc() times each
candidate for a few fused steps on the run's own state, saved before and
restored after each, and leaves the fastest selected for that run only: the
choice goes into the run's own clv_params (opt_* fields), so other CLVisc
objects in the process keep theirs.

    from clvisc_b200.autotune import tune_visc
    v = CLVisc(cfg); v.load_ini(ic)
    best, table = tune_visc(v)
"""
import torch

from . import _lib

DEFAULTS = {'kernel': 0, 'tile': 0, 'chunk': 32, 'blocks': 2}


def _apply(v, c):
    """Select candidate c for the run v (its clv_params opt_* fields)."""
    p = v.params
    p.opt_stage_kernel = c['kernel'] + 1
    p.opt_tile = c['tile'] + 1
    p.opt_chunk = c['chunk']
    p.opt_tiled_blocks = c['blocks']


def candidates(nz, use_float32=True, fast=False):
    """(kernel, tile, chunk, blocks) choices worth timing on a grid with nz
    cells along eta (the 16 x 32 tile exists in the FP32 tolerance build); chunk
    0 leaves the x planes per block to the library."""
    out = [dict(DEFAULTS, chunk=0), dict(DEFAULTS, kernel=1)]
    if nz == 1:
        return out + [dict(DEFAULTS, kernel=3)]
    tiles = (0, 1, 2, 3) if (fast and use_float32) else (0, 1, 2)
    blocks = 2 if use_float32 else 1
    for tile in tiles:
        for chunk in (0, 5, 8, 12, 16, 24, 32, 48):
            out.append({'kernel': 2, 'tile': tile, 'chunk': chunk, 'blocks': blocks})
    if use_float32:
        out.append({'kernel': 2, 'tile': 0, 'chunk': 32, 'blocks': 1})
    return out


def _state(v):
    ts = list(v.ideal.d_ev) + list(v.d_pi) + [v.d_src, v.d_udiff, v.d_goodcell, v._key]
    return ts


def tune_visc(v, steps=3, cands=None):
    """Time `steps` fused steps of the CLVisc v for each candidate; returns
    (the chosen candidate, {candidate key: ms per step}) and selects it."""
    cands = cands or candidates(v.cfg.NZ, v.cfg.use_float32, bool(v.params.flags & _lib.CLV_FLAG_FAST))
    tensors = _state(v)
    saved = [t.clone() for t in tensors]
    tau = v.ideal.tau
    table = {}
    for c in cands:
        _apply(v, c)
        v.step(0)  # warm-up (and one-time kernel set-up)
        torch.cuda.synchronize(v.device)
        e0 = torch.cuda.Event(enable_timing=True)
        e1 = torch.cuda.Event(enable_timing=True)
        e0.record()
        for n in range(1, steps + 1):
            v.step(n)
        e1.record()
        torch.cuda.synchronize(v.device)
        key = 'kernel%d_tile%d_chunk%d_blocks%d' % (c['kernel'], c['tile'], c['chunk'], c['blocks'])
        table[key] = e0.elapsed_time(e1) / steps
        for t, s in zip(tensors, saved):
            t.copy_(s)
        v.ideal.tau = tau
    best_key = min(table, key=table.get)
    best = next(c for c in cands if 'kernel%d_tile%d_chunk%d_blocks%d' % (c['kernel'], c['tile'], c['chunk'],
                                                                            c['blocks']) == best_key)
    _apply(v, best)
    return best, table


def reset(v=None):
    """The run v (if given) back to the process-wide launch choices, and
    those back to the library's defaults."""
    if v is not None:
        p = v.params
        p.opt_stage_kernel = p.opt_tile = p.opt_chunk = p.opt_tiled_blocks = 0
    _lib.set_option(_lib.CLV_OPT_STAGE_KERNEL, DEFAULTS['kernel'])
    _lib.set_option(_lib.CLV_OPT_TILE, DEFAULTS['tile'])
    _lib.set_option(_lib.CLV_OPT_CHUNK, DEFAULTS['chunk'])
    _lib.set_option(_lib.CLV_OPT_TILED_BLOCKS, DEFAULTS['blocks'])
