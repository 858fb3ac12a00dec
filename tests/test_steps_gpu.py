"""The library's step calls (clv_visc_steps, clv_ideal_steps) against separate
stage calls, their refusals, a stop inside an output block, and subclasses whose
own methods are called stage by stage. The exact build: the same bits."""
import ctypes

import numpy as np
import pytest

from parity_util import assert_same, make_cfg, seeded_ic

pytestmark = pytest.mark.gpu


def _visc(cls, grid=(13, 11, 1), use_float32=True, **kw):
    cfg = make_cfg(*grid, use_float32=use_float32, **kw)
    v = cls(cfg)
    v.load_ini(seeded_ic(cfg, seed=4, flow=0.2))
    v.IS_initialize()
    return v


@pytest.mark.parametrize('use_float32', [True, False])
@pytest.mark.parametrize('grid', [(13, 11, 1), (7, 9, 25), (6, 7, 5)])
@pytest.mark.parametrize('n', [0, 1, 5])
def test_visc_steps_are_stage_calls(cuda_lib, grid, use_float32, n):
    from clvisc_b200 import _lib
    from clvisc_b200.visc import CLVisc
    both = _lib.CLV_PART_IS | _lib.CLV_PART_KT
    a, b = (_visc(CLVisc, grid, use_float32) for _ in range(2))
    a._steps(0, n, edmax=True)
    for k in range(n):
        b._stage(1, both, fused=True)
        b.update_time(k)
        if k == n - 1:
            b._call('clv_max_ed_reset', _lib.ptr(b._key), b.stream)
        b._stage(2, both, fused=True, edmax=k == n - 1)
    assert a.ideal.tau == b.ideal.tau
    for x, y in zip(list(a.ideal.d_ev) + a.d_pi + [a.d_src, a.d_udiff], list(b.ideal.d_ev) + b.d_pi + [b.d_src, b.d_udiff]):
        assert_same('field', x.cpu().numpy(), y.cpu().numpy())
    if n:
        assert a.read_edmax_key() == b.read_edmax_key() == a.ideal.max_energy_density()


def test_step_calls_refuse(cuda_lib):
    from clvisc_b200 import _lib
    from clvisc_b200.ideal import CLIdeal
    from clvisc_b200.visc import CLVisc
    v = _visc(CLVisc)
    both = _lib.CLV_PART_IS | _lib.CLV_PART_KT
    b1, b2, tau = v._buffers(1, both, fused=True), v._buffers(2, both, fused=True), v.ideal.times(0, 2)
    before = [t.clone() for t in v.ideal.d_ev + v.d_pi]
    r, p, s = ctypes.byref, ctypes.byref(v.params), v.stream
    for n, t, x, y in ((-1, tau, r(b1), r(b2)), (1, None, r(b1), r(b2)), (1, tau, None, r(b2)), (1, tau, r(b1), None)):
        assert v.lib.clv_visc_steps(p, n, t, x, y, s) == -1 and b'visc_steps' in v.lib.clv_last_error()
    assert v.lib.clv_visc_steps(None, 1, tau, r(b1), r(b2), s) == -1
    assert v.lib.clv_visc_steps(p, 0, None, r(b1), r(b2), s) == 0
    i = v.ideal
    f = [_lib.ptr(t) for t in (i.d_ev[1], i.d_ev[2], i.d_Src, i._key)]
    out, done = (ctypes.c_double * 2)(), ctypes.c_int(7)
    for n, t, key, o, d in ((-1, tau, f[3], out, r(done)), (1, None, f[3], out, r(done)), (1, tau, None, out, r(done)),
                            (1, tau, f[3], None, r(done)), (1, tau, f[3], out, None)):
        assert i.lib.clv_ideal_steps(p, n, t, f[0], f[1], f[2], key, 0.0, o, d, s) == -1
        assert b'ideal_steps' in i.lib.clv_last_error()
    assert i.lib.clv_ideal_steps(p, 1, tau, None, f[1], f[2], f[3], 0.0, out, r(done), s) == -1 and done.value == 0
    assert i.lib.clv_ideal_steps(p, 0, None, f[0], f[1], f[2], f[3], 0.0, None, r(done), s) == 0 and done.value == 0
    for x, y in zip(v.ideal.d_ev + v.d_pi, before):
        assert_same('untouched', x.cpu().numpy(), y.cpu().numpy())
    assert isinstance(i, CLIdeal)


def test_a_refused_step_leaves_tau(cuda_lib):
    from clvisc_b200.visc import CLVisc
    v = _visc(CLVisc)
    tau, nx = v.ideal.tau, v.params.nx
    v.params.nx = 0
    with pytest.raises(Exception):
        v._steps(0, 3)
    assert v.ideal.tau == tau
    v.params.nx = nx
    v._steps(0, 3)
    assert v.ideal.tau == v.cfg.real(v.cfg.TAU0 + 3 * v.cfg.DT)


@pytest.mark.parametrize('name', ['update_time', '_stage', '_buffers'])
@pytest.mark.parametrize('on_object', [False, True])
def test_overridden_viscous_methods_run_between_the_stages(cuda_lib, name, on_object):
    from clvisc_b200.visc import CLVisc
    seen = []

    def wrap(v, base):
        def f(*a, **k):
            seen.append((name, float(v.ideal.tau)))
            return base(*a, **k)
        return f

    if on_object:
        v = _visc(CLVisc)
        setattr(v, name, wrap(v, getattr(v, name)))
    else:
        own = type('Own', (CLVisc,), {name: lambda self, *a, **k: wrap(self, lambda *b, **c: getattr(CLVisc, name)(
            self, *b, **c))(*a, **k)})
        v = _visc(own)
    o = _visc(CLVisc)
    seen.clear()
    for h in (v, o):
        h.evolve(max_loops=6, save_hypersf=False, force_run_to_maxloop=True)
    assert_same('ev', v.ideal.d_ev[1].cpu().numpy(), o.ideal.d_ev[1].cpu().numpy())
    assert v.ideal.history == o.ideal.history
    taus = [float(v.cfg.real(v.cfg.TAU0 + k * v.cfg.DT)) for k in range(7)]
    want = taus[:6] if name == 'update_time' else [t for k in range(6) for t in taus[k:k + 2]]
    assert [t for _, t in seen] == want


def test_overridden_surface_is_asked_for_at_every_step(cuda_lib):
    from clvisc_b200.ideal import CLIdeal
    from clvisc_b200.visc import CLVisc
    calls = []

    class Visc(CLVisc):
        def get_hypersf(self, n, ntskip, is_finished):
            calls.append(n)
            return CLVisc.get_hypersf(self, n, ntskip, is_finished)

    class Ideal(CLIdeal):
        def get_hypersf(self, n, ntskip):
            calls.append(n)
            return CLIdeal.get_hypersf(self, n, ntskip)

    v = _visc(Visc, TFRZ=0.05)
    v.evolve(max_loops=6, save_pi=False, force_run_to_maxloop=True)
    assert calls == list(range(6))
    calls.clear()
    cfg = make_cfg(13, 11, 1)
    i = Ideal(cfg)
    i.load_ini(seeded_ic(cfg))
    i.evolve(max_loops=6, save_bulk=False, plot_bulk=False, to_maxloop=True)
    assert calls == list(range(6))


@pytest.mark.parametrize('use_float32', [True, False])
@pytest.mark.parametrize('to_maxloop', [False, True])
@pytest.mark.parametrize('grid', [(13, 11, 1), (9, 8, 25)])
def test_ideal_run_that_stops_inside_an_output_block(cuda_lib, grid, use_float32, to_maxloop):
    """Against a subclass that takes the separate calls: the same steps, history
    and state, for a freeze-out that the run passes between two outputs."""
    from clvisc_b200.ideal import CLIdeal

    class Separate(CLIdeal):
        def stepUpdate(self, step, jet_eloss_src=None):
            CLIdeal.stepUpdate(self, step, jet_eloss_src)

    cfg = make_cfg(*grid, use_float32=use_float32, ntskip=8)
    runs = []
    for cls in (CLIdeal, Separate):
        i = cls(cfg)
        i.load_ini(seeded_ic(cfg, seed=3, edmax=20.0))
        runs.append(i)
    probe = Separate(cfg)
    probe.load_ini(seeded_ic(cfg, seed=3, edmax=20.0))
    probe.evolve(max_loops=14, save_hypersf=False, save_bulk=False, plot_bulk=False)
    efrz = 0.5 * float(probe.history[10][1] + probe.history[11][1])  # passed in the step to 11, outputs at 8 and 16
    for i in runs:
        i.efrz = efrz
        i.params.efrz = efrz
        i.evolve(max_loops=14, save_bulk=False, plot_bulk=False, to_maxloop=to_maxloop)
    a, b = runs
    assert len(a.history) == len(b.history) == (14 if to_maxloop else 12)
    assert a.history == b.history and a.tau == b.tau and a.edmax == b.edmax
    assert_same('ev', a.d_ev[1].cpu().numpy(), b.d_ev[1].cpu().numpy())
    assert a.num_of_sf == b.num_of_sf and (a.num_of_sf > 0) == (grid[2] > 1)  # no cubes in a plane
    np.testing.assert_array_equal(a.hypersf_to_host()[0], b.hypersf_to_host()[0])
