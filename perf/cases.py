"""The workloads this backend is timed on: what a user of the hydro backend has
it do, through its public classes, from one small (2+1)D event to the
385 x 385 x 115 event, with the surface, the spectra and the learned surrogate.

Hydro states are synthetic mid-evolution states made from the seed alone:
seeded hotspots with plateau and Gaussian tails along eta_s, outward flow with
fluctuations, and a shear tensor boosted from a traceless rest-frame tensor of
Navier-Stokes size, so that it is transverse and traceless as in a run. A pass
restores the state from a snapshot, as a restart from a checkpoint does, and
evolves it. exact() restates the same equations in 64 bits with plain torch.
"""
import math
import os
import tempfile

import numpy as np
import torch

DEV = 'cuda' if torch.cuda.is_available() else 'cpu'


# ------------------------------------------------------------------- cases
def _step(name, nx, ny, nz, steps, fp64=False, arithmetic='fast', bulk=False, eos='lattice_pce165', dx=0.16, dt=0.02):
    return {'name': name, 'kind': 'step', 'nx': nx, 'ny': ny, 'nz': nz, 'steps': steps, 'fp64': fp64,
            'arithmetic': arithmetic, 'bulk': bulk, 'eos': eos, 'dx': dx, 'dt': dt}


def _event2d(name, nx, ny, fp64=False, bulk=False, eos='lattice_pce165'):
    return {'name': name, 'kind': 'event', 'nx': nx, 'ny': ny, 'nz': 1, 'steps': 20, 'fp64': fp64,
            'arithmetic': 'fast', 'bulk': bulk, 'eos': eos, 'dx': 0.16, 'dt': 0.02}


def _ideal(name, nx, ny, nz, steps, fp64, eos):
    return {'name': name, 'kind': 'ideal', 'nx': nx, 'ny': ny, 'nz': nz, 'steps': steps, 'fp64': fp64, 'eos': eos,
            'dx': 0.16, 'dt': 0.02}


def _batch(name, events, lo, hi, fp64=False):
    return {'name': name, 'kind': 'batch', 'events': events, 'lo': lo, 'hi': hi, 'steps': 20, 'fp64': fp64,
            'bulk': True, 'eos': 'lattice_pce165', 'dx': 0.16, 'dt': 0.02}


def _surface(name, nx, ny, nz, skip, fp64=False):
    return {'name': name, 'kind': 'surface', 'nx': nx, 'ny': ny, 'nz': nz, 'skip': skip, 'fp64': fp64,
            'eos': 'lattice_pce165', 'dx': 0.16, 'dt': 0.02}


def _spectra(name, n, viscous, fp64=False):
    return {'name': name, 'kind': 'spectra', 'n': n, 'viscous': viscous, 'fp64': fp64, 'pid': 211}


def _unet(name, batch, size, train):
    return {'name': name, 'kind': 'unet', 'batch': batch, 'size': size, 'train': train}


def listed():
    return [
        # one small (2+1)D event between two freeze-out checks: launches and
        # latency count (the smallest grid of the batched workload)
        _event2d('event_121x121_fp32', 121, 121),
        # ideal boost-invariant hydro, conformal EOS, double precision
        _ideal('ideal_101x101_fp64', 101, 101, 1, 20, True, 'ideal_gas'),
        # the single (3+1)D viscous event on the ordinary grid
        _step('step_201x201x105_fp32', 201, 201, 105, 2),
        # the large event of the headline benchmark
        _step('step_385x385x115_fp32', 385, 385, 115, 2, dx=0.08, dt=0.01),
        # double precision, ragged against every tile size
        _step('step_161x145x77_fp64', 161, 145, 77, 2, fp64=True),
        # the reference's arithmetic bit for bit (parity and regression runs)
        _step('step_97x93x65_exact', 97, 93, 65, 2, arithmetic='exact'),
        # shear and bulk viscosity in (3+1)D
        _step('step_129x121x61_bulk', 129, 121, 61, 2, bulk=True),
        # ideal (3+1)D evolution with its default diagnostics
        _ideal('ideal_201x201x61_fp32', 201, 201, 61, 4, False, 'lattice_pce165'),
        # event-by-event (2+1)D runs advanced together, shear and bulk
        _batch('batch_32_events_bulk', 32, 121, 301),
        # the freeze-out surface between two output times
        _surface('surface_201x201x105', 201, 201, 105, 2),
        # Cooper-Frye spectrum of one species with the viscous correction
        _spectra('spectra_40k_viscous', 40000, True),
        # one optimiser step of the surrogate: forward, backward, Adam
        _unet('surrogate_train_32', 32, 128, True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges: grids from 41 to 385 cells across and
    1, or 8 to 115, along eta_s, odd sizes among them, no larger than the
    385 x 385 x 115 event."""
    kind = rng.choice(['step', 'step', 'step', 'event', 'ideal', 'batch', 'surface', 'spectra', 'unet'])
    nx, ny, nz = _log_int(rng, 41, 385), _log_int(rng, 41, 385), _log_int(rng, 8, 115)
    if kind == 'step':
        what = rng.choice(['fast', 'fast', 'fast', 'fp64', 'exact', 'bulk'])
        if what != 'fast':
            nx, ny = min(nx, 201), min(ny, 201)
        c = _step('', nx, ny, nz, rng.choice([1, 2]), fp64=what == 'fp64', bulk=what == 'bulk',
                  arithmetic='exact' if what == 'exact' else 'fast',
                  eos=rng.choice(['lattice_pce165', 'lattice_pce165', 'lattice_pce150', 'ideal_gas']))
    elif kind == 'event':
        c = _event2d('', min(nx, 301), min(ny, 301), fp64=rng.random() < 0.25, bulk=rng.random() < 0.5)
    elif kind == 'ideal':
        flat = rng.random() < 0.4
        c = _ideal('', min(nx, 251), min(ny, 251), 1 if flat else nz, 20 if flat else 4, rng.random() < 0.5,
                   rng.choice(['ideal_gas', 'lattice_pce165']))
    elif kind == 'batch':
        c = _batch('', _log_int(rng, 4, 64), 121, rng.choice([151, 201, 251, 301]))
    elif kind == 'surface':
        c = _surface('', min(nx, 301), min(ny, 301), nz, rng.choice([1, 2]), fp64=rng.random() < 0.25)
    elif kind == 'spectra':
        c = _spectra('', _log_int(rng, 2000, 120000), rng.random() < 0.6, fp64=False)
    else:
        c = _unet('', rng.choice([8, 12, 16, 24, 32]), rng.choice([64, 128]), rng.random() < 0.5)
    del c['name']
    return c


# ------------------------------------------------------------------ inputs
def _cfg(c, nx=None, ny=None, nz=None):
    from clvisc_b200.config import read_config, set_real
    cfg = read_config([])
    cfg.NX, cfg.NY, cfg.NZ = (c['nx'], c['ny'], c['nz']) if nx is None else (nx, ny, nz)
    cfg.DX = cfg.DY = c['dx']
    cfg.DZ = 0.15
    cfg.DT = c['dt']
    cfg.TAU0 = 1.0
    cfg.eos_type = c['eos']
    cfg.use_float32 = not c['fp64']
    cfg.arithmetic = c.get('arithmetic', 'fast')
    etaos = 0.16 if c['kind'] == 'batch' else 0.08
    cfg.ETAOS_XMIN, cfg.ETAOS_YMIN, cfg.ETAOS_LEFT_SLOP, cfg.ETAOS_RIGHT_SLOP = 0.18, etaos, 0.0, 0.0
    if c.get('bulk'):
        cfg.ZETAOS_MAX, cfg.ZETAOS_T0, cfg.ZETAOS_WIDTH, cfg.ZETAOS_SKEW = 0.05, 0.18, 0.02, 0.0
    cfg.TFRZ = 0.137
    cfg.ntskip = 20
    cfg.nxskip = cfg.nyskip = c.get('skip', 2)
    cfg.nzskip = 1
    cfg.fPathOut = os.path.join(tempfile.gettempdir(), 'clv_perf')
    return set_real(cfg)


def _dtype(c):
    return torch.float64 if c['fp64'] else torch.float32


def _gen(seed):
    return torch.Generator(device='cpu').manual_seed(int(seed))


def _uniform(g, lo, hi, *shape):
    return (lo + (hi - lo) * torch.rand(*shape, generator=g, dtype=torch.float64)).to(DEV)


def _state(nx, ny, nz, dx, seed, dt, bulk, dtype, peak=25.0):
    """ev (4, nx, ny, nz), pi (10 or 11, ...), udiff (4, ...) and the energy
    density of the last prediction (nx, ny, nz), at tau = 1 fm."""
    g = _gen(seed)
    ax = lambda n, d: (torch.arange(n, dtype=torch.float64, device=DEV) - n // 2) * d
    x, y, z = ax(nx, dx), ax(ny, dx), ax(nz, 0.15)
    rx, ry, rz = 0.5 * nx * dx, 0.5 * ny * dx, max(0.5 * nz * 0.15, 1.0)
    n = 120
    px, py = (torch.randn(n, generator=g, dtype=torch.float64).to(DEV) * (0.32 * r) for r in (rx, ry))
    w, width = _uniform(g, 0.2, 2.0, n), _uniform(g, 0.5, 0.9, n)
    gx = torch.exp(-(x[:, None] - px) ** 2 / (2 * width ** 2))
    gy = torch.exp(-(y[:, None] - py) ** 2 / (2 * width ** 2))
    exy = (gx * w) @ gy.T
    h = torch.exp(-torch.clamp(z.abs() - 0.45 * rz, min=0.0) ** 2 / (2 * (0.25 * rz) ** 2))
    f = lambda t: t.to(dtype)
    e = f(peak * exy / exy.max())[:, :, None] * f(h)
    ph = _uniform(g, 0.0, 2 * math.pi, 6)
    k = _uniform(g, 1.0, 3.0, 6)
    X, Y, Z = f(x)[:, None, None], f(y)[None, :, None], f(z)[None, None, :]
    r = torch.sqrt(1.0 + (X / (0.45 * rx)) ** 2 + (Y / (0.45 * ry)) ** 2)
    wob = lambda i: 0.04 * torch.sin(k[i].to(dtype) * X + ph[i].to(dtype)) * torch.cos(k[i + 1].to(dtype) * Y + ph[i + 1].to(dtype))
    one = torch.ones_like(e)
    vx = (0.55 * (X / (0.45 * rx)) / r + wob(0)) * one
    vy = (0.55 * (Y / (0.45 * ry)) / r + wob(2)) * one
    vz = (0.08 * torch.tanh(Z / rz) + 0.5 * wob(4)) * one if nz > 1 else torch.zeros_like(e)
    ev = torch.stack([e, vx, vy, vz])
    del one, r
    v2 = vx * vx + vy * vy + vz * vz
    gam = 1.0 / torch.sqrt(1.0 - v2)
    # rest-frame shear: Navier-Stokes of the longitudinal expansion, with a
    # modulated transverse part
    a = 0.03 * e
    mod = wob(1) * 5.0
    S = {(1, 1): a * (1 + mod), (2, 2): a * (1 - mod), (3, 3): -2.0 * a, (1, 2): 0.4 * a * mod, (1, 3): 0.0 * a,
         (2, 3): 0.0 * a}
    s = lambda i, j: S[(min(i, j), max(i, j))]
    v = {1: vx, 2: vy, 3: vz}
    wv = {i: s(i, 1) * vx + s(i, 2) * vy + s(i, 3) * vz for i in (1, 2, 3)}
    q = wv[1] * vx + wv[2] * vy + wv[3] * vz
    gg = gam * gam / (gam + 1.0)
    pi = torch.zeros((11 if bulk else 10,) + tuple(e.shape), dtype=dtype, device=DEV)
    pi[0] = gam * gam * q
    idx = {(1, 1): 4, (1, 2): 5, (1, 3): 6, (2, 2): 7, (2, 3): 8, (3, 3): 9}
    for i in (1, 2, 3):
        pi[i] = gam * (wv[i] + gg * q * v[i])
        for j in range(i, 4):
            pi[idx[(i, j)]] = s(i, j) + gg * (v[i] * wv[j] + wv[i] * v[j]) + gg * gg * q * v[i] * v[j]
    if bulk:
        pi[10] = -0.01 * e
    du = [0.1 * dt * gam * v[i] for i in (1, 2, 3)]
    ud = torch.stack([v[1] * du[0] + v[2] * du[1] + v[3] * du[2]] + du)
    return ev, pi, ud, e * (1.0 - 1.2 * dt)


def _planes(t, like):
    """(w, nx, ny, nz) as the (w, ld) planes of a field, padding zero."""
    out = torch.zeros_like(like)
    out[:t.shape[0], :t[0].numel()] = t.reshape(t.shape[0], -1)
    return out


def _grids(c):
    """The batched events' grids: sizes spread evenly over [lo, hi], odd."""
    n = c['events']
    size = lambda e: 2 * ((c['lo'] + (c['hi'] - c['lo']) * ((7 * e) % n) // max(1, n - 1)) // 2) + 1
    return [(size(e), size(e), 1) for e in range(n)]


def _later(ev, pi, dt):
    """A state 20 steps on: diluted, with the same flow."""
    ev2 = ev.clone()
    ev2[0] *= (1.0 + 20 * dt) ** -1.5
    return ev2, pi * (1.0 + 20 * dt) ** -1.5


def _surface_elements(c, seed):
    g = _gen(seed)
    n, f = c['n'], lambda t: t.to(_dtype(c))
    eta, phi = _uniform(g, -4.0, 4.0, n), _uniform(g, 0.0, 2 * math.pi, n)
    vr = _uniform(g, 0.0, 0.7, n)
    v = torch.stack([vr * torch.cos(phi), vr * torch.sin(phi), _uniform(g, -0.05, 0.05, n)], 1)
    area = _uniform(g, 0.005, 0.02, n)
    ds = torch.stack([area, -0.6 * area * torch.cos(phi), -0.6 * area * torch.sin(phi), 0.05 * area], 1)
    sf = torch.cat([ds, v, eta[:, None]], 1)
    pi = _uniform(g, -0.006, 0.006, n, 10)
    return f(sf), f(pi) if c['viscous'] else None


def _images(c, seed):
    """Training images (N, n, n) and fields (N, n, n, 6) like the solver's."""
    g = _gen(seed)
    N, n = c['batch'], c['size']
    ax = (torch.arange(n, dtype=torch.float64, device=DEV) - n // 2) * 0.16
    cen, w = _uniform(g, -4.0, 4.0, N, 40, 2), _uniform(g, 0.2, 2.0, N, 40)
    gx = torch.exp(-(ax[None, None, :] - cen[:, :, :1]) ** 2 / 0.5)
    gy = torch.exp(-(ax[None, None, :] - cen[:, :, 1:]) ** 2 / 0.5)
    e = torch.einsum('nk,nkx,nky->nxy', w, gx, gy)
    e = 50.0 * e / e.amax((1, 2), keepdim=True)
    sm = torch.nn.functional.avg_pool2d(e[:, None], 9, 1, 4)[:, 0]
    ux, uy = 0.1 * ax[None, :, None] * torch.ones_like(e), 0.1 * ax[None, None, :] * torch.ones_like(e)
    y = torch.stack([0.05 * sm, ux, uy, 0.004 * sm * ux, 0.002 * sm * ux * uy, 0.004 * sm * uy], -1)
    return e.float(), y.float()


# ----------------------------------------------------------------- prepare
def prepare(case, seed):
    c = case
    s = {'case': c}
    if c['kind'] in ('step', 'event', 'surface'):
        from clvisc_b200.visc import CLVisc
        cfg = _cfg(c)
        ev, pi, ud, e2 = _state(c['nx'], c['ny'], c['nz'], c['dx'], seed, c['dt'], c.get('bulk', False), _dtype(c))
        cap = max(1000, ev[0].numel() // 4) if c['kind'] == 'surface' else 1000
        v = CLVisc(cfg, hypersf_capacity=cap)
        s['v'] = v
        if c['kind'] == 'surface':
            ev2, pi2 = _later(ev, pi, c['dt'])
            s['old'] = _planes(ev, v.ideal.d_ev[1]), _planes(pi, v.d_pi[1])
            v.ideal.d_ev[1].copy_(_planes(ev2, v.ideal.d_ev[1]))
            v.d_pi[1].copy_(_planes(pi2, v.d_pi[1]))
        else:
            s['snap'] = (_planes(ev, v.ideal.d_ev[1]), _planes(pi, v.d_pi[1]), _planes(ud, v.d_udiff),
                         _planes(e2[None], v.ideal.d_ev[2])[0].clone())
    elif c['kind'] == 'ideal':
        from clvisc_b200.ideal import CLIdeal
        v = CLIdeal(_cfg(c), hypersf_capacity=1000)
        s['v'] = v
        s['snap'] = _planes(_state(c['nx'], c['ny'], c['nz'], c['dx'], seed, c['dt'], False, _dtype(c))[0], v.d_ev[1])
    elif c['kind'] == 'batch':
        from clvisc_b200.batch import CLViscBatch
        grids = _grids(c)
        # the launch shape autotune() picks for this workload
        tiles = sum(((ny + 59) // 60) * ((nx + 15) // 16) for nx, ny, _ in grids)
        b = CLViscBatch(_cfg(c, *grids[0]), grids, max_loops=c['steps'], stop_at_freezeout=False,
                        launch=('tile', 64, 16, tiles))
        arenas = [torch.zeros_like(t) for t in (b.d_ev[1], b.d_pi[1], b.d_udiff, b.d_ev[2])]
        for e, ((nx, ny, nz), (ld, oe, op, _, _)) in enumerate(zip(grids, b.layout)):
            st = _state(nx, ny, nz, c['dx'], seed * 1000 + e, c['dt'], True, _dtype(c))
            for arena, off, t in zip(arenas, (oe, op, oe, oe), (st[0], st[1], st[2], st[3][None])):
                w = t.shape[0]
                arena[off:off + w * ld].view(w, ld)[:, :nx * ny * nz] = t.reshape(w, -1)
        s['b'], s['snap'] = b, arenas
    elif c['kind'] == 'spectra':
        from clvisc_b200.spectra import SmoothSpec
        sf, pi = _surface_elements(c, seed)
        s['v'] = SmoothSpec(sf, 0.137, pi, 12.0, use_float32=not c['fp64'])
    else:
        from clvisc_b200.surrogate import Surrogate
        s['x'], s['y'] = _images(c, seed)
        s['v'] = Surrogate(c['batch'], c['size'], seed=seed)
        s['v'].fit_scales(s['y'])
    return s


# --------------------------------------------------------------------- run
def run(s):
    c, v = s['case'], s.get('v')
    if c['kind'] in ('step', 'event'):
        ev, pi, ud, e2 = s['snap']
        v.ideal.d_ev[1].copy_(ev)
        v.d_pi[1].copy_(pi)
        v.d_udiff.copy_(ud)
        v.ideal.d_ev[2][0].copy_(e2)
        v.update_time(-1)
        if c['kind'] == 'step':
            for n in range(c['steps']):
                v.step(n)
        else:
            v.evolve(max_loops=c['steps'], save_hypersf=False, force_run_to_maxloop=True)
        return {'ev': v.ideal.d_ev[1], 'pi': v.d_pi[1]}
    if c['kind'] == 'surface':
        v.ideal.d_ev_old.copy_(s['old'][0])
        v.d_pi_old.copy_(s['old'][1])
        v.ideal.d_num_of_sf.zero_()
        v.tau_old = v.cfg.TAU0
        v.update_time(19)
        v.get_hypersf(20, 20, False)
        i = v.ideal
        return {'count': i.d_num_of_sf, 'ds': i.d_hypersf[:, :4], 'veta': i.d_hypersf[:, 4:], 'txyz': i.d_sf_txyz,
                'pi': v.d_pi_sf}
    if c['kind'] == 'ideal':
        v.d_ev[1].copy_(s['snap'])
        v.update_time(-1)
        b = v.bulkinfo
        for rows in vars(b).values():  # the diagnostics of the pass before
            if isinstance(rows, list):
                rows.clear()
        v.evolve(max_loops=c['steps'], save_hypersf=False, save_bulk=False, plot_bulk=True)
        return {'ev': v.d_ev[1], 'ecc': [b.ecc1_vs_rapidity[-1], b.ecc2_vs_rapidity[-1]], 'plane': b.plane_sums[-1],
                'energy': b.energy[-1], 'entropy': b.entropy_total[-1], 'exy': b.exy[-1]}
    if c['kind'] == 'batch':
        b = s['b']
        for dst, src in zip((b.d_ev[1], b.d_pi[1], b.d_udiff, b.d_ev[2]), s['snap']):
            dst.copy_(src)
        b.evolve()
        return {'ev': b.d_ev[1], 'pi': b.d_pi[1]}
    if c['kind'] == 'spectra':
        return v.calc(c['pid'])
    if not c['train']:
        return v.predict(s['x'])
    # one step of Surrogate.train
    net = v.net
    net.buf['x'].copy_(s['x'] * v.in_scale)
    out = net.forward()
    loss = net.loss((s['y'].reshape(-1, 6) / v.out_scale).contiguous(), v.wch)
    net.backward()
    gn = torch.linalg.vector_norm(net.grads)
    net.grads.mul_(torch.clamp(1.0 / (gn + 1e-6), max=1.0))
    net.adam(1e-3)
    return {'out': out, 'loss': loss, 'grads': net.grads, 'params': net.params}


# -------------------------------------------------------------------- work
def _unet_layers():
    return [(32, 32, 0), (32, 64, 1), (64, 64, 1), (64, 128, 2), (128, 128, 2), (128, 256, 3), (256, 256, 3),
            (384, 128, 2), (128, 128, 2), (192, 64, 1), (64, 64, 1), (96, 32, 0), (32, 32, 0)]


def work(case):
    """Bytes: the state read and written once a step (ev, pi, udiff), the
    surface's corner energies, the elements, the images and parameters.
    Operations: about 1500 a cell and Runge-Kutta stage (viscous), 400
    (ideal), 50 an element and momentum point, 2 a multiply-add of the
    convolutions."""
    c = case
    r = 8 if c.get('fp64') else 4
    if c['kind'] in ('step', 'event', 'ideal'):
        cells = c['nx'] * c['ny'] * c['nz']
        planes = 4 if c['kind'] == 'ideal' else 19 if c['bulk'] else 18
        ops = 800.0 if c['kind'] == 'ideal' else 3000.0
        return {'bytes': 2.0 * planes * r * cells * c['steps'], 'flops': ops * cells * c['steps']}
    if c['kind'] == 'batch':
        cells = sum(a * b for a, b, _ in _grids(c))
        return {'bytes': 2.0 * 19 * r * cells * c['steps'], 'flops': 2400.0 * cells * c['steps']}
    if c['kind'] == 'surface':
        cells = c['nx'] * c['ny'] * c['nz']
        # the corner energies of both times, and the copy that keeps the new
        # state for the next output time
        return {'bytes': 2.0 * r * cells / c['skip'] ** 2 + 28.0 * r * cells, 'flops': 40.0 * cells / c['skip'] ** 2}
    if c['kind'] == 'spectra':
        return {'bytes': float(c['n'] * (18 if c['viscous'] else 8) * r), 'flops': 50.0 * c['n'] * 41 * 15 * 48}
    px = c['batch'] * c['size'] ** 2
    mac = sum(9.0 * a * b * px / 4 ** l for a, b, l in _unet_layers()) + px * (9 * 32 + 32 * 6)
    par = 9 * sum(a * b for a, b, _ in _unet_layers())
    return {'bytes': float(28 * px + 4 * par * (7 if c['train'] else 1)), 'flops': 2 * mac * (3 if c['train'] else 1)}


# ------------------------------------------------------------------- exact
class _Eos64(object):
    """Linear interpolation in the EOS table (its rows are input data)."""

    def __init__(self, name):
        from clvisc_b200.eos import Eos, TABLE_SHAPE
        t, m = Eos(name).create_table(*TABLE_SHAPE[name])
        self.t = torch.from_numpy(t.reshape(-1, 4).astype(np.float64)).to(DEV)
        self.e0 = float(np.float32(m['ed_start']))
        self.de = float(np.float32(m['ed_step']))

    def __call__(self, e, col):
        x = (e - self.e0) / self.de
        i = torch.clamp(x.floor(), 0, self.t.shape[0] - 2).long()
        col = self.t[:, col].contiguous()
        lo = col[i]
        return lo + (x - i) * (col[i + 1] - lo)


def _f32(x):
    return float(np.float32(x))


_PI = {(0, 0): 0, (0, 1): 1, (0, 2): 2, (0, 3): 3, (1, 1): 4, (1, 2): 5, (1, 3): 6, (2, 2): 7, (2, 3): 8, (3, 3): 9}


def _pi(i, j):
    return _PI[(min(i, j), max(i, j))]


def _sh(t, axis, d):
    n = t.shape[axis]
    return t.index_select(axis, torch.clamp(torch.arange(n, device=t.device) + d, 0, n - 1))


def _limit(l, m, r):
    a, b = r - m, m - l
    s = torch.minimum(1.1 * torch.minimum(a.abs(), b.abs()), 0.5 * (a + b).abs())
    return torch.where(a * b > 0, torch.copysign(s, a), torch.zeros_like(a))


def _faces(F, axis):
    """Flux difference of face values given on n + 1 faces."""
    n = F.shape[axis] - 1
    return F.narrow(axis, 1, n) - F.narrow(axis, 0, n)


def _sides(t, axis):
    """A cell field on the left and right of the n + 1 faces (edges repeat)."""
    n = t.shape[axis]
    k = torch.arange(n + 1, device=t.device)
    return t.index_select(axis, torch.clamp(k - 1, 0)), t.index_select(axis, torch.clamp(k, max=n - 1))


def _mid(t, axis):
    left, right = _sides(t, axis)
    return 0.5 * (left + right)


def _gamma(v, acu):
    return 1.0 / torch.sqrt(torch.clamp(1.0 - v[0] ** 2 - v[1] ** 2 - v[2] ** 2, min=acu))


def _solve(P, T00, M, bulk=None):
    """e = T00 - M v with (T00 + P(e)) v = M, by bisection."""
    lo, hi = torch.zeros_like(M), torch.ones_like(M)
    for _ in range(54):
        v = 0.5 * (lo + hi)
        pr = P(T00 - M * v, 1)
        if bulk is not None:
            pr = pr + bulk
        up = (T00 + pr) * v - M > 0
        hi, lo = torch.where(up, v, hi), torch.where(up, lo, v)
    return T00 - M * 0.5 * (lo + hi)


def _recover(P, T0m, tau, acu, bulk=None):
    """T^{tau mu} tau -> (e, v), with the floors of the path."""
    T00 = torch.clamp(T0m[0], min=acu) / tau
    T = [torch.where(t.abs() < acu, torch.zeros_like(t), t / tau) for t in T0m[1:]]
    M = torch.sqrt(T[0] ** 2 + T[1] ** 2 + T[2] ** 2)
    big = M > T00
    f = torch.where(big, 0.999 * T00 / torch.where(big, M, torch.ones_like(M)), torch.ones_like(M))
    T = [t * f for t in T]
    M = torch.where(big, 0.999 * T00, M)
    e = torch.clamp(_solve(P, T00, M, bulk), min=0.0)
    pr = P(e, 1) if bulk is None else P(e, 1) + bulk
    den = torch.clamp(T00 + pr, min=acu)
    return e, [torch.where(e < acu, torch.zeros_like(t), t / den) for t in T], T


def _visc_stage(P, k, step, tau, ev, pi, ev1, pi1, ud, e2, src, acu):
    """One stage: the new (ev, pi), the sources; k: the run's constants."""
    dt, D = k['dt'], (k['dx'], k['dx'], k['dz'] * tau)
    bulk = pi[10] if len(pi) > 10 else None
    g = _gamma(ev[1:], acu)
    p0 = P(ev[0], 1)
    pr = p0 if bulk is None else p0 + bulk
    u = [g, g * ev[1], g * ev[2], g * ev[3]]
    h = (ev[0] + pr) * g
    Q = [tau * (h * u[c] - (pr if c == 0 else 0.0) + pi[c]) for c in range(4)]
    S = [torch.zeros_like(g) for _ in range(4 + len(pi))] if src is None else src
    uz = u[3] / tau
    for m, t in ((0, 2 * pi[3]), (1, pi[6]), (2, pi[8]), (3, pi[0] + pi[9]), (6, pi[1]), (8, pi[2]), (9, 2 * pi[3])):
        S[4 + m] = S[4 + m] - uz * t
    S[0] = S[0] - (h * g * ev[3] ** 2 + pr + pi[9])
    S[3] = S[3] - (h * g * ev[3] + pi[3])
    grad = []
    for a in range(3):
        vh, ph = _mid(ev[1 + a], a), _mid(pr, a) * tau
        up = lambda q: _limit(_sh(q, a, -1), q, _sh(q, a, 1))
        for c in range(4 + len(pi)):
            q = Q[c] if c < 4 else g * pi[c - 4]
            (ql, qr), (sl, sr) = _sides(q, a), _sides(up(q), a)
            # the edge's ghost cells are flat
            sl.select(a, 0).zero_()
            sr.select(a, -1).zero_()
            al, ar = ql + 0.5 * sl, qr - 0.5 * sr
            F = 0.5 * (ar + al) * vh - 0.5 * (ar - al)
            if c < 4:
                p0l, p0r = _sides(pi[c], a)
                pal, par = _sides(pi[_pi(a + 1, c)], a)
                F = F + ((ph if c == 0 else 0.0) - 0.5 * tau * (p0l + p0r)) * vh + 0.5 * tau * (pal + par)
                if c == a + 1:
                    F = F + ph
            S[c] = S[c] - _faces(F, a) / D[a]
        d = [_limit(_sh(x, a, -1), x, _sh(x, a, 1)) / D[a] for x in u]
        if a == 2:
            d[0], d[3] = d[0] + u[3] / tau, d[3] + u[0] / tau
        grad.append(d)
    # pi
    g1 = _gamma(ev1[1:], acu)
    uo = [g1, g1 * ev1[1], g1 * ev1[2], g1 * ev1[3]]
    un = [a + b for a, b in zip(uo, ud)] if step == 1 else u
    udt = [x / dt for x in ud] if step == 1 else [(a - b) / dt for a, b in zip(un, uo)]
    us = uo if step == 1 else un
    es, en = (ev1[0], e2) if step == 1 else (ev[0], ev[0])
    da = [[udt[c], grad[0][c], grad[1][c], grad[2][c]] for c in range(4)]
    DU = [sum(us[b] * da[c][b] for b in range(4)) for c in range(4)]
    theta = udt[0] + grad[0][1] + grad[1][2] + grad[2][3]
    T, sd = P(es, 2), P(es, 3)
    eta_s = torch.where(T < k['xmin'], k['left'] * (T - k['xmin']), k['right'] * (T - k['xmin'])) + k['ymin']
    etav = eta_s * sd * 0.19733
    otp = T / (3.0 * torch.clamp(eta_s, min=acu) * 0.19733)
    gm = (1.0, -1.0, -1.0, -1.0)
    W = [sum(gm[l] * pi[_pi(m, l)] * DU[l] for l in range(4)) for m in range(4)]
    new, den = [None] * len(pi), un[0] + dt * otp
    for m in range(4):
        for n in range(m, 4):
            gmn = gm[m] if m == n else 0.0
            sig = gm[m] * da[n][m] + gm[n] * da[m][n] - (us[m] * DU[n] + us[n] * DU[m]) \
                - 2.0 / 3.0 * (gmn - us[m] * us[n]) * theta
            i = _pi(m, n)
            S[4 + i] = S[4 + i] - pi[i] * (theta / 3.0 + us[0] / tau) - (us[m] * W[n] + us[n] * W[m])
            new[i] = (pi1[i] * uo[0] + S[4 + i] * dt / step + dt * otp * etav * sig) / den
    P2 = P(en, 1)
    if bulk is not None:
        w = k['zw']
        zs = k['zmax'] * w * w / (w * w + (T - k['zt0']) ** 2)
        otb = 14.55 * (1.0 / 3.0 - P(es, 0)) ** 2 * T / (torch.clamp(zs, min=acu) * 0.19733)
        S[14] = S[14] + bulk * (theta / 3.0 - us[0] / tau)
        b = (pi1[10] * uo[0] + S[14] * dt / step - dt * otb * zs * sd * 0.19733 * theta) / (un[0] + dt * otb)
        b = torch.where(b < -P2, -P2, torch.where(b > P2, P2, b))
        new[10] = torch.where(T < k['ztmin'], torch.zeros_like(b), b)
    top = torch.stack([x.abs() for x in new[:10]]).amax(0)
    bad = top > (en + P2) * un[0] ** 2 - P2
    new = [torch.where(bad, torch.zeros_like(x), x) for x in new]
    # e, v
    p1 = P(ev1[0], 1)
    if bulk is not None:
        p1 = p1 + pi1[10]
    h1, old = (ev1[0] + p1) * g1, tau - (step - 1) * dt
    T0m = [(h1 * uo[c] - (p1 if c == 0 else 0.0) + pi1[c]) * old + S[c] * dt / step - new[c] * tau for c in range(4)]
    e, v, _ = _recover(P, T0m, tau, acu, new[10] if bulk is not None else None)
    return [e] + v, new, S


def _consts(c, cfg):
    return {'dt': _f32(cfg.DT), 'dx': _f32(cfg.DX), 'dz': _f32(cfg.DZ), 'xmin': _f32(cfg.ETAOS_XMIN),
            'ymin': _f32(cfg.ETAOS_YMIN), 'left': _f32(cfg.ETAOS_LEFT_SLOP), 'right': _f32(cfg.ETAOS_RIGHT_SLOP),
            'zmax': _f32(cfg.ZETAOS_MAX), 'zt0': _f32(cfg.ZETAOS_T0), 'zw': _f32(cfg.ZETAOS_WIDTH),
            'ztmin': _f32(cfg.ZETAOS_TMIN)}


def _tau(c, n):
    t = 1.0 + n * c['dt']
    return t if c['fp64'] else _f32(t)


def _visc_exact(c, P, st):
    k, acu = _consts(c, _cfg(c, 8, 8, 1)), 1e-14 if c['fp64'] else _f32(1e-7)
    ev, pi, ud = ([x.double() for x in t] for t in st[:3])
    e2 = st[3].double()
    for n in range(c['steps']):
        a, b, S = _visc_stage(P, k, 1, _tau(c, n), ev, pi, ev, pi, ud, e2, None, acu)
        new, pi2, _ = _visc_stage(P, k, 2, _tau(c, n + 1), a, b, ev, pi, ud, e2, S, acu)
        go, gn = _gamma(ev[1:], acu), _gamma(new[1:], acu)
        ud = [gn - go] + [gn * new[i] - go * ev[i] for i in (1, 2, 3)]
        ev, pi, e2 = new, pi2, a[0]
    return torch.stack(ev), torch.stack(pi)


def _ideal_exact(c, P, ev):
    dt, dx, dz = _f32(c['dt']), _f32(c['dx']), _f32(0.15)
    acu = 1e-14 if c['fp64'] else _f32(1e-7)
    ev = [x.double() for x in ev]
    for n in range(c['steps']):
        cur, S = ev, None
        for step in (1, 2):
            tau = _tau(c, n + step - 1)
            g, pr = _gamma(cur[1:], acu), P(cur[0], 1)
            h = (cur[0] + pr) * g
            T = [h * g - pr] + [h * g * cur[i] for i in (1, 2, 3)]
            S = [torch.zeros_like(g) for _ in range(4)] if S is None else S
            S[0] = S[0] - (h * g * cur[3] ** 2 + pr)
            S[3] = S[3] - h * g * cur[3]
            for a in range(3):
                vh, ph = _mid(cur[1 + a], a), _mid(pr, a)
                for q in range(4):
                    (ql, qr) = _sides(T[q], a)
                    sl, sr = _sides(_limit(_sh(T[q], a, -1), T[q], _sh(T[q], a, 1)), a)
                    sl.select(a, 0).zero_()
                    sr.select(a, -1).zero_()
                    al, ar = ql + 0.5 * sl, qr - 0.5 * sr
                    F = 0.5 * (ar + al) * vh - 0.5 * (ar - al)
                    if q == 0:
                        F = F + ph * vh
                    if q == a + 1:
                        F = F + ph
                    S[q] = S[q] - _faces(F, a) * (tau / dx if a < 2 else 1.0 / dz)
            g1, p1 = _gamma(ev[1:], acu), P(ev[0], 1)
            h1, old = (ev[0] + p1) * g1, tau - (step - 1) * dt
            T0 = [(h1 * g1 - p1) * old + S[0] * dt / step]
            T0 += [h1 * g1 * ev[i] * old + S[i] * dt / step for i in (1, 2, 3)]
            T00 = torch.clamp(T0[0], min=acu) / tau
            e, v, Tv = _recover(P, T0, tau, acu)
            # the ideal path keeps its velocities in the coldest cells
            den = torch.clamp(T00 + P(e, 1), min=acu)
            cur = [e] + [t / den for t in Tv]
        ev = cur
    return torch.stack(ev)


def _bulkinfo_exact(c, P, ev):
    """The diagnostics of the state ev at tau = 1 fm."""
    e, vx, vy, vz = (x.double() for x in ev)
    nz = e.shape[2]
    ed = torch.clamp(e, min=1e-10)
    pr = P(ed, 1)
    v2 = vx ** 2 + vy ** 2 + vz ** 2
    u2 = 1.0 / (1.0 - torch.where(v2 > 1, torch.full_like(v2, 0.999999), v2))
    s = lambda t: t.sum((0, 1)).cpu().numpy()
    txx, tyy, tx = s((ed + pr) * u2 * vx ** 2 + pr), s((ed + pr) * u2 * vy ** 2 + pr), s((ed + pr) * u2 * vx)
    m = nz // 2
    d, p, x, y = ed[:, :, m], pr[:, :, m], vx[:, :, m], vy[:, :, m]
    w2 = 1.0 / (1.0 - x ** 2 - y ** 2)
    w = torch.sqrt(w2)
    plane = [(d + p) * w2 * x ** 2 + p, (d + p) * w2 * y ** 2 + p, (d + p) * w2 * x, w * d * torch.sqrt(x * x + y * y),
             w * d, w * P(d, 3), 0 * d, 0 * d]
    u0 = _gamma([vx, vy, vz], 1e-14 if c['fp64'] else _f32(1e-7))
    pr0 = P(e, 1)
    z = ((torch.arange(nz, device=DEV) - nz // 2) * _f32(0.15)).double()
    ch, sh = torch.cosh(z), torch.sinh(z)
    vol = c['dx'] * c['dx'] * 0.15
    en = ((e + pr0) * u0 ** 2 * (ch + vz * sh) - pr0 * ch).sum()
    return {'ecc': [tx / (txx + tyy), (txx - tyy) / (txx + tyy)], 'plane': np.array([float(t.sum()) for t in plane]),
            'energy': float(en) * vol, 'entropy': float((u0 * P(e, 3)).sum()) * vol, 'exy': e[:, :, m].cpu().numpy()}


def _surface_exact(c, P, st):
    """Positions, velocities and pi of the elements, in cube order; the area
    elements come out of a convex hull of points moved at random where they
    are coplanar and have no value in 64 bits."""
    from clvisc_b200.eos import Eos
    ev, pi = st[0], st[1]
    ev2, pi2 = _later(ev, pi, c['dt'])
    efrz = _f32(float(Eos(c['eos']).f_ed(0.137)))
    sk = (c['skip'], c['skip'], 1)
    n = [(m - 1) // k for m, k in zip(ev.shape[1:], sk)]
    at = lambda t, q: t[..., (q & 1) * sk[0]:, ((q >> 1) & 1) * sk[1]:, ((q >> 2) & 1) * sk[2]:][
        ..., ::sk[0], ::sk[1], ::sk[2]][..., :n[0], :n[1], :n[2]]
    E = torch.stack([at(ev[0], q) for q in range(8)] + [at(ev2[0], q) for q in range(8)]).double()
    d = E - efrz
    hit = ~torch.stack([d[q] * d[15 - q] > 0 for q in range(8)]).all(0)
    d = d[:, hit]
    pos = torch.zeros((4, d.shape[1]), dtype=torch.float64, device=DEV)
    num = torch.zeros(d.shape[1], dtype=torch.float64, device=DEV)
    for a in range(16):
        for bit, comp in ((1, 1), (2, 2), (4, 3), (8, 0)):
            if a & bit:
                continue
            b = a | bit
            cut = d[a] * d[b] < 0
            f = torch.where(cut, d[a].abs() / torch.where(cut, (d[a] - d[b]).abs(), torch.ones_like(num)), 0 * num)
            p = [float((a >> 3) & 1), float(a & 1), float((a >> 1) & 1), float((a >> 2) & 1)]
            for q in range(4):
                pos[q] += torch.where(cut, f if q == comp else torch.full_like(f, p[q]), 0 * f)
            num += cut
    ok = num > 0
    mc = (pos / num)[:, ok]
    cube = torch.nonzero(hit)[ok].double()
    wt = []
    for q in range(16):
        side = ((q >> 3) & 1, q & 1, (q >> 1) & 1, (q >> 2) & 1)
        f = [mc[i] if side[i] else 1.0 - mc[i] for i in range(4)]
        wt.append(f[0] * f[1] * f[2] * f[3])

    def mean(old, new):
        return sum(wt[q] * at(old if q < 8 else new, q & 7)[hit][ok].double() for q in range(16))
    v = [mean(ev[i], ev2[i]) for i in (1, 2, 3)]
    dx, dz = _f32(c['dx']), _f32(0.15)
    t0 = 1.0
    t1 = _tau(c, 20)
    org = [-(m // 2) for m in ev.shape[1:]]
    tau = t0 + mc[0] * (t1 - t0)
    x = org[0] * dx + (cube[:, 0] + mc[1]) * sk[0] * dx
    y = org[1] * dx + (cube[:, 1] + mc[2]) * sk[1] * dx
    eta = org[2] * dz + (cube[:, 2] + mc[3]) * dz
    cap = max(1000, ev[0].numel() // 4)

    def full(cols):
        out = torch.zeros((cap, len(cols)), dtype=torch.float64, device=DEV)
        t = torch.stack(cols, 1)[:cap]
        out[:t.shape[0]] = t
        return out
    return {'count': None, 'ds': None, 'veta': full(v + [eta]),
            'txyz': full([tau * torch.cosh(eta), x, y, tau * torch.sinh(eta)]),
            'pi': full([mean(pi[i], pi2[i]) for i in range(10)])}


def _spectra_exact(c, seed):
    from numpy.polynomial import laguerre, legendre
    sf, pi = _surface_elements(c, seed)
    sf = sf.double()
    mass, T = 0.13957, 0.137
    yy = torch.linspace(-8.0, 8.0, 41, dtype=torch.float64, device=DEV)
    pt = torch.from_numpy(laguerre.laggauss(15)[0] / 12.0).to(DEV)
    gx = legendre.leggauss(48)[0][24:][::-1]
    phi = np.empty(48)
    for i in range(24):
        phi[47 - i], phi[i] = np.pi * (gx[i] + 1.0), np.pi * (1.0 - gx[i])
    phi = torch.from_numpy(phi).to(DEV)
    if not c['fp64']:
        yy, pt = yy.float().double(), pt.float().double()
    px, py = pt[:, None] * torch.cos(phi), pt[:, None] * torch.sin(phi)
    mt = torch.sqrt(mass * mass + pt * pt)[:, None] * torch.ones_like(px)
    P = torch.stack([mt, px, py]).reshape(3, -1)
    out = torch.zeros((41, P.shape[1]), dtype=torch.float64, device=DEV)
    for lo in range(0, sf.shape[0], 20000):
        S = sf[lo:lo + 20000]
        g = 1.0 / torch.sqrt(1.0 - S[:, 4] ** 2 - S[:, 5] ** 2 - S[:, 6] ** 2)
        p = pi[lo:lo + 20000].double() if pi is not None else None
        for k in range(41):
            ch, sh = torch.cosh(yy[k] - S[:, 7]), torch.sinh(yy[k] - S[:, 7])
            p0, p3 = ch[:, None] * P[0], -sh[:, None] * P[0]
            p1, p2 = -P[1][None], -P[2][None]
            pu = g[:, None] * (p0 + p1 * S[:, 4:5] + p2 * S[:, 5:6] + p3 * S[:, 6:7])
            f = 1.0 / (torch.exp(pu / T) - 1.0)
            if p is not None:
                q = lambda i: p[:, i:i + 1]
                pp = 12.0 * (p0 * p0 * q(0) + p3 * p3 * q(9) + 2 * p0 * (p1 * q(1) + p2 * q(2) + p3 * q(3))
                             + p1 * p1 * q(4) + 2 * p1 * p2 * q(5) + p2 * p2 * q(7) + 2 * p3 * (p1 * q(3) + p2 * q(6)))
                df = f * (1.0 + f) * pp
                f = f + torch.where(df.abs() > f, torch.sign(df) * f * 0.999, df)
            sig = p0 * S[:, 0:1] + p1 * S[:, 1:2] + p2 * S[:, 2:3] + p3 * S[:, 3:4]
            out[k] += (sig * f).sum(0)
    return (out / (2 * math.pi) ** 3).reshape(41, 15, 48).cpu().numpy()


def _unet_exact(c, seed):
    """The network in 64 bits from the same initial parameters."""
    from clvisc_b200.surrogate import Surrogate
    x, y = _images(c, seed)
    sur = Surrogate(c['batch'], c['size'], seed=seed)
    sur.fit_scales(y)
    net, F = sur.net, torch.nn.functional
    flat = net.params.double().requires_grad_(True)
    par = lambda k: flat[net.offsets[k]:net.offsets[k] + int(np.prod(net.shapes[k]))].reshape(net.shapes[k])
    gelu = lambda t: F.gelu(t)

    def conv(t, name):
        w = par(name + '.w')
        w = w.reshape(3, 3, -1, w.shape[-1]).permute(3, 2, 0, 1)
        return gelu(F.conv2d(t, w, par(name + '.b'), padding=1))
    up = lambda t: F.interpolate(t, scale_factor=2, mode='nearest')
    s1 = conv(conv((x * sur.in_scale).double()[:, None], 'first'), 'e1b')
    s2 = conv(conv(F.avg_pool2d(s1, 2), 'e2a'), 'e2b')
    s3 = conv(conv(F.avg_pool2d(s2, 2), 'e3a'), 'e3b')
    t = conv(conv(F.avg_pool2d(s3, 2), 'e4a'), 'e4b')
    t = conv(conv(torch.cat([up(t), s3], 1), 'd3a'), 'd3b')
    t = conv(conv(torch.cat([up(t), s2], 1), 'd2a'), 'd2b')
    t = conv(conv(torch.cat([up(t), s1], 1), 'd1a'), 'd1b')
    out = t.permute(0, 2, 3, 1).reshape(-1, 32) @ par('head.w') + par('head.b')
    if not c['train']:
        return (out * sur.out_scale.double()).detach().reshape(c['batch'], c['size'], c['size'], 6)
    d = out - y.reshape(-1, 6).double() / sur.out_scale.double()
    loss = (sur.wch.double() * d * d).sum() / d.numel()
    (g,) = torch.autograd.grad(loss, flat)
    g = g * torch.clamp(1.0 / (torch.linalg.vector_norm(g) + 1e-6), max=1.0)
    return {'out': out.detach(), 'loss': loss.detach(), 'grads': g, 'params': None}


def exact(case, seed):
    c = case
    if c['kind'] == 'spectra':
        return _spectra_exact(c, seed)
    if c['kind'] == 'unet':
        return _unet_exact(c, seed)
    P = _Eos64(c['eos'])
    if c['kind'] == 'batch':
        grids = _grids(c)
        stride = [((nx * ny + 63) // 64) * 64 for nx, ny, _ in grids]
        ev = torch.zeros(4 * sum(stride), dtype=torch.float64, device=DEV)
        pi = torch.zeros(11 * sum(stride), dtype=torch.float64, device=DEV)
        at = 0
        for e, ((nx, ny, nz), ld) in enumerate(zip(grids, stride)):
            st = _state(nx, ny, nz, c['dx'], seed * 1000 + e, c['dt'], True, _dtype(c))
            for out, w, t in zip((ev, pi), (4, 11), _visc_exact(c, P, st)):
                out[w * at:w * (at + ld)].view(w, ld)[:, :nx * ny] = t.reshape(w, -1)
            at += ld
        return {'ev': ev, 'pi': pi}
    st = _state(c['nx'], c['ny'], c['nz'], c['dx'], seed, c['dt'], c.get('bulk', False), _dtype(c))
    if c['kind'] == 'surface':
        return _surface_exact(c, P, st)
    cells = c['nx'] * c['ny'] * c['nz']
    ld = ((cells + 63) // 64) * 64

    def planes(t):
        out = torch.zeros((t.shape[0], ld), dtype=torch.float64, device=DEV)
        out[:, :cells] = t.reshape(t.shape[0], -1)
        return out
    if c['kind'] == 'ideal':
        return {'ev': planes(_ideal_exact(c, P, st[0])), **_bulkinfo_exact(c, P, st[0])}
    ev, pi = _visc_exact(c, P, st)
    return {'ev': planes(ev), 'pi': planes(pi)}
