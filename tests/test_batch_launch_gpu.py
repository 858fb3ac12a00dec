"""The tiled launch shape of a small batch: its grid counts strips, the kernel's
items are smaller patches."""
import numpy as np
import pytest

from parity_util import assert_same, make_cfg, seeded_ic

pytestmark = pytest.mark.gpu
GRIDS = [(121, 121, 1), (131, 127, 1), (141, 139, 1), (151, 149, 1)]


def _batch(launch=None):
    from clvisc_b200.batch import CLViscBatch
    cfg = make_cfg(*GRIDS[0], dx=0.16, arithmetic='fast', ntskip=20)
    b = CLViscBatch(cfg, GRIDS, max_loops=20, stop_at_freezeout=False, launch=launch)
    for e, g in enumerate(GRIDS):
        b.load_ini(e, seeded_ic(make_cfg(*g, dx=0.16), seed=e))
    return b


def _ms(b):
    import torch
    snap = [t.clone() for t in (b.d_ev[1], b.d_pi[1], b.d_udiff, b.d_ev[2])]
    times = []
    for _ in range(8):
        for dst, src in zip((b.d_ev[1], b.d_pi[1], b.d_udiff, b.d_ev[2]), snap):
            dst.copy_(src)
        t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        t0.record()
        b.evolve()
        t1.record()
        torch.cuda.synchronize()
        times.append(t0.elapsed_time(t1))
    return float(np.median(times[2:]))


def test_strip_count_fills_the_gpu(cuda_lib):
    """A shape with one block a strip runs as many patches at once as the GPU
    takes: the same values, and no slower (1.3 for the timer; 1.9 with the strips
    taken as blocks) than a grid that fills it."""
    strips = ('tile', 64, 16, _batch().tiles(64, 16))
    a, b = _batch(strips), _batch(('tile', 64, 16, 0))
    ta, tb = _ms(a), _ms(b)
    for e in range(len(GRIDS)):
        assert_same('ev %d' % e, a.ev_to_host(e), b.ev_to_host(e))
        assert_same('pi %d' % e, a.pi_to_host(e), b.pi_to_host(e))
    assert ta <= 1.3 * tb, (ta, tb)


def test_one_tiled_candidate(cuda_lib):
    """rows, chunk and the strip count give one and the same launch: timed once."""
    b = _batch()
    tiled = [c for c in b.candidates() if c[0] == 'tile']
    assert len(tiled) == 1 and tiled[0][2] == 16
