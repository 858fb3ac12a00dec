"""Cells whose next state hangs on the last bit: T^{tau i} at the 1e-7 below
which it is set to zero, or T at the ZETAOS_TMIN below which Pi is. In the FP32
tolerance build a change of rounding moves such a cell by 1e-4 to 1e-1 of its
value, so the batched (2+1)D stage must go on giving the values it always gave.

tests/golden/dilute_cells.npz holds five such cells of batched events with bulk
viscosity (the 121 x 121 to 301 x 301 events of perf/cases.py, 8 to 17 steps
into their runs): the fields of a window around the cell (it starts at a
multiple of 16 planes in x and reaches 5 cells beyond the cell, one more than a
step's stencil) and the cell's (e, v, pi, Pi) one step later as the strips of
rows - 4 = 60 rows by 16 planes gave them on a B200."""
import os

import numpy as np
import pytest

from parity_util import make_cfg

pytestmark = pytest.mark.gpu
GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), 'golden', 'dilute_cells.npz')


@pytest.mark.parametrize('n', range(5))
def test_dilute_cell_one_step(cuda_lib, n):
    import torch
    from clvisc_b200.batch import CLViscBatch
    z = np.load(GOLDEN)
    f, (i, j, k), want = z['fields%d' % n], z['cell%d' % n], z['want%d' % n]
    _, nx, ny = f.shape
    cfg = make_cfg(nx, ny, 1, dx=0.16, dz=0.15, etaos=0.16, tau0=1.0 + 0.02 * int(k), arithmetic='fast',
                   ZETAOS_MAX=0.05, ZETAOS_T0=0.18, ZETAOS_WIDTH=0.02, ZETAOS_SKEW=0.0)
    cfg.TAU0 = float(np.float32(cfg.TAU0))
    cfg.TFRZ, cfg.ntskip = 0.137, 20
    b = CLViscBatch(cfg, [(nx, ny, 1)], max_loops=1, stop_at_freezeout=False, launch=('tile', 64, 16, 64))
    ld = b.layout[0][0]
    for arena, lo, w in ((b.d_ev[1], 0, 4), (b.d_pi[1], 4, 11), (b.d_udiff, 15, 4), (b.d_ev[2], 19, 1)):
        planes = torch.zeros((w, ld), dtype=torch.float32)
        planes[:, :nx * ny] = torch.from_numpy(f[lo:lo + w].reshape(w, -1))
        arena[:w * ld].copy_(planes.reshape(-1))
    b.evolve(use_graph=False)
    at = int(i) * ny + int(j)
    got = np.concatenate([b.ev_to_host(0)[at], b.pi_to_host(0)[at], b.bulk_to_host(0)[at:at + 1]])
    # the FP32 tolerance, 1e-5 of each field's largest magnitude
    scale = np.concatenate([[f[0].max()], np.full(3, np.abs(f[1:4]).max()), np.full(10, np.abs(f[4:14]).max()),
                            [np.abs(f[14]).max()]])
    assert (np.abs(got - want) <= 1e-5 * scale).all(), np.abs(got - want) / scale
