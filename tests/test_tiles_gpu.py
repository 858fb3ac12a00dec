"""Tile, patch and chunk edges of the stage kernels, the surface spectra and
the diagnostics: grids one cell below, at and above a tile's sizes, against
the oracle. Exact-build kernels bit for bit; the tolerance build within its
stated tolerance (1e-5 / 1e-11 of each field's largest magnitude)."""
import numpy as np
import pytest

from clvisc_b200.eos import Eos
from parity_util import assert_same, make_cfg, seeded_ic
from test_fast_gpu import TOL, compare_fields, field_errors

pytestmark = pytest.mark.gpu

BULK = dict(ZETAOS_MAX=0.12, ZETAOS_T0=0.2, ZETAOS_WIDTH=0.05, ZETAOS_SKEW=0.3)


@pytest.mark.parametrize('use_float32', [True, False])
@pytest.mark.parametrize('riemann', [False, True])
@pytest.mark.parametrize('grid', [(1, 8, 32), (3, 9, 33), (5, 7, 24), (67, 17, 31)])
def test_ideal_tiled_edges(cuda_lib, oracle_mod, use_float32, riemann, grid):
    """The tiled ideal stage (eta axes of 24 cells and more), both stages."""
    from clvisc_b200.ideal import CLIdeal
    cfg = make_cfg(*grid, use_float32=use_float32, riemann_test=riemann)
    g, o = CLIdeal(cfg), oracle_mod.OracleIdeal(cfg)
    ic = seeded_ic(cfg, seed=3, flow=0.3)
    g.load_ini(ic)
    o.load_ini(ic)
    for n in range(3):
        for step in (1, 2):
            g.stepUpdate(step)
            o.stepUpdate(step)
            assert_same('stage %d src' % step, g.field_to_host(g.d_Src), o.d_Src)
            assert_same('stage %d ev' % step, g.field_to_host(g.d_ev[3 - step]), o.d_ev[3 - step])
            if step == 1:
                g.update_time(n)
                o.update_time(n)


@pytest.mark.parametrize('use_float32', [True, False])
@pytest.mark.parametrize('arithmetic', ['exact', 'fast'])
@pytest.mark.parametrize('extra', [{}, BULK], ids=['shear', 'bulk'])
@pytest.mark.parametrize('grid', [(1, 9, 1), (7, 1, 1), (8, 8, 1), (9, 17, 1), (41, 33, 1), (3, 8, 24), (9, 17, 33),
                                  (37, 7, 25)])
def test_viscous_edges(cuda_lib, oracle_mod, use_float32, arithmetic, extra, grid):
    """(2+1)D patches and (3+1)D tiles with and without the bulk sector."""
    from clvisc_b200.visc import CLVisc
    cfg = make_cfg(*grid, use_float32=use_float32, arithmetic=arithmetic, **extra)
    v, o = CLVisc(cfg), oracle_mod.OracleVisc(cfg)
    ic = seeded_ic(cfg, seed=17, flow=0.2)
    for h in (v, o):
        h.load_ini(ic)
        h.IS_initialize()
    for n in range(6):
        v.step(n, edmax=(n == 5))
        o.step(n)
    if arithmetic == 'fast':
        compare_fields(v, o, use_float32, 'edges %s' % (grid,))
    else:
        assert_same('ev', v.ideal.field_to_host(v.ideal.d_ev[1]), o.ideal.d_ev[1])
        assert_same('pi', v.pi_to_host(1), o.d_pi[1])
        if v.bulk:
            assert_same('Pi', v.bulk_to_host(1), o.d_bulk[1])
    want = o.ideal.max_energy_density()
    assert abs(v.read_edmax_key() - want) <= (TOL[use_float32] if arithmetic == 'fast' else 0.0) * abs(want)


@pytest.mark.parametrize('use_float32', [True, False])
def test_fast_stage_beyond_the_eos_table(cuda_lib, oracle_mod, use_float32):
    """Energy densities from the table's first texel over its last
    (310.998 GeV/fm^3) into the formula beyond it, no flow: the tolerance
    build's lookup takes the reference's way from the last texel on. The
    formula's power and exponential differ between CUDA and the host library
    by 2 ulp, far inside the tolerance."""
    from clvisc_b200.visc import CLVisc
    cfg = make_cfg(9, 8, 40, use_float32=use_float32, arithmetic='fast')
    v, o = CLVisc(cfg), oracle_mod.OracleVisc(cfg)
    n = 9 * 8 * 40
    ic = np.zeros((n, 4), cfg.real)
    ic[:, 0] = np.linspace(0.0, 400.0, n)
    for h in (v, o):
        h.load_ini(ic)
        h.IS_initialize()
        h.step(0)
    errs = field_errors(v.ideal.field_to_host(v.ideal.d_ev[1]), o.ideal.d_ev[1], v.pi_to_host(1), o.d_pi[1],
                        Eos(cfg.eos_type), float(v.ideal.tau))
    assert max(e for k, e in errs.items() if k != 'components') <= TOL[use_float32], errs


@pytest.mark.parametrize('use_float32', [True, False])
@pytest.mark.parametrize('viscous', [False, True])
@pytest.mark.parametrize('n', [1, 127, 128, 129, 1800])
def test_spectra_element_counts(cuda_lib, oracle_mod, use_float32, viscous, n):
    """One element, a tile's edges, and more chunks than one."""
    from clvisc_b200.spectra import SmoothSpec
    rng = np.random.default_rng(n)
    sf = np.zeros((n, 8))
    sf[:, 0] = rng.uniform(0.01, 0.02, n)
    sf[:, 1:4] = rng.uniform(-0.005, 0.005, (n, 3))
    sf[:, 4:6] = rng.uniform(-0.5, 0.5, (n, 2))
    sf[:, 6] = rng.uniform(-0.05, 0.05, n)
    sf[:, 7] = rng.uniform(-4.0, 4.0, n)
    pi = rng.uniform(-0.006, 0.006, (n, 10)) if viscous else None
    s = SmoothSpec(sf, 0.137, pi, 12.0, use_float32=use_float32)
    got = s.calc(211, mu=0.02)
    want = oracle_mod.spectra(sf, pi, 0.13957, 1.0, -1.0, 0.02, 0.137, 12.0 if viscous else 0.0, s.y, s.pt, s.phi,
                              use_float32)
    # the sums' scale: terms of both signs cancel
    tol = 1e-5 if use_float32 else 1e-11
    assert np.abs(got - want).max() <= tol * np.abs(want).max()


@pytest.mark.parametrize('use_float32', [True, False])
@pytest.mark.parametrize('grid', [(9, 7, 1), (17, 15, 7), (16, 33, 8), (13, 11, 9), (3, 70, 25)])
def test_diagnostics_slice_edges(cuda_lib, use_float32, grid):
    """Sums per eta slice with fewer, as many and more slices than a cluster's
    lanes, and every slice buffer, against numpy in double (conformal gas:
    P(e) is linear, so the table's interpolation is exact to its float32
    texels, 6e-8)."""
    from clvisc_b200.visc import CLVisc
    cfg = make_cfg(*grid, use_float32=use_float32, eos_type='ideal_gas')
    v = CLVisc(cfg)
    v.load_ini(seeded_ic(cfg, seed=2, flow=0.4))
    b = v.ideal.bulkinfo
    b.get(v.ideal.tau, v.ideal.d_ev[1], 1.0, v.d_pi[1])
    NX, NY, NZ = grid
    ev = v.ideal.field_to_host(v.ideal.d_ev[1]).reshape(NX, NY, NZ, 4)
    np.testing.assert_array_equal(b.exz[-1], ev[:, NY // 2, :, 0])
    np.testing.assert_array_equal(b.vx_xy[-1], ev[:, :, NZ // 2, 1])
    np.testing.assert_array_equal(b.ez[-1], ev[NX // 2, NY // 2, :, 0])
    np.testing.assert_array_equal(b.ey[-1], ev[NX // 2, :, NZ // 2, 0])
    e = np.maximum(ev[..., 0].astype(np.float64), 1e-10)
    vx, vy, vz = (ev[..., i].astype(np.float64) for i in (1, 2, 3))
    pr, u2 = e / 3.0, 1.0 / (1.0 - vx ** 2 - vy ** 2 - vz ** 2)
    s = lambda t: t.sum((0, 1))
    txx, tyy, tx = s((e + pr) * u2 * vx ** 2 + pr), s((e + pr) * u2 * vy ** 2 + pr), s((e + pr) * u2 * vx)
    scale = (txx + tyy)
    np.testing.assert_allclose(b.ecc2_vs_rapidity[-1], (txx - tyy) / scale, rtol=0, atol=1e-6)
    np.testing.assert_allclose(b.ecc1_vs_rapidity[-1], tx / scale, rtol=0, atol=1e-6)
    w2 = 1.0 / (1.0 - vx ** 2 - vy ** 2)[:, :, NZ // 2]
    got = b.plane_sums[-1]
    np.testing.assert_allclose(got[4], (np.sqrt(w2) * e[:, :, NZ // 2]).sum(), rtol=1e-12)


def _unet_call(lib, name, *args):
    import ctypes
    import torch
    a = [ctypes.c_void_p(t.data_ptr()) if isinstance(t, torch.Tensor) else t for t in args]
    assert getattr(lib, name)(*a, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0, name


@pytest.mark.parametrize('C,cs,co', [(8, 8, 0), (24, 24, 0), (32, 96, 64), (32, 96, 60), (36, 36, 0), (256, 256, 0)])
@pytest.mark.parametrize('H', [2, 6])
def test_unet_small_layers(cuda_lib, C, cs, co, H):
    """Pooling, upsampling, their gradients, the first layer, the head and the
    bias sums at channel counts, strides and offsets on either side of the
    16-byte path, against torch in FP32. BF16 outputs to their rounding (2^-8
    of the value; one of the scale where terms cancel), FP32 sums over P
    pixels of products of unit size to P 2^-23."""
    import ctypes
    import torch
    import torch.nn.functional as F
    lib, N, W, K = cuda_lib, 3, 10, 6
    g = torch.Generator().manual_seed(C + H)
    rnd = lambda *s: torch.randn(*s, generator=g).cuda()
    bf = lambda t: t.to(torch.bfloat16)
    wide = lambda h, w: bf(rnd(N, h, w, cs))
    f = lambda t: t[..., co:co + C].float().permute(0, 3, 1, 2)
    near = lambda got, want: np.testing.assert_allclose(got.float().cpu().numpy(), want.cpu().numpy(), rtol=2.0 ** -8,
                                                        atol=2.0 ** -8 * 0.01)
    nhwc = lambda t: t.permute(0, 2, 3, 1)
    x = wide(H, W)
    out = torch.zeros(N, H // 2, W // 2, C, dtype=torch.bfloat16, device='cuda')
    _unet_call(lib, 'clv_unet_pool', x, cs, co, N, H, W, C, out)
    near(out, nhwc(F.avg_pool2d(f(x), 2)))
    src, dst = bf(rnd(N, H, W, C)), torch.zeros(N, 2 * H, 2 * W, cs, dtype=torch.bfloat16, device='cuda')
    _unet_call(lib, 'clv_unet_up', src, N, H, W, C, dst, cs, co)
    want = torch.zeros_like(dst)
    want[..., co:co + C] = src.repeat_interleave(2, 1).repeat_interleave(2, 2)
    assert torch.equal(dst, want)
    dgelu = lambda z: torch.autograd.functional.jvp(F.gelu, z, torch.ones_like(z))[1]
    z, gp = bf(rnd(N, H, W, C)), bf(rnd(N, H // 2, W // 2, C))
    gz = torch.zeros_like(z)
    _unet_call(lib, 'clv_unet_skip_grad', x, cs, co, gp, z, N, H, W, C, gz)
    up = gp.float().repeat_interleave(2, 1).repeat_interleave(2, 2)
    near(gz, (x[..., co:co + C].float() + 0.25 * up) * dgelu(z.float()))
    big = wide(2 * H, 2 * W)
    _unet_call(lib, 'clv_unet_up_grad', big, cs, co, z, N, H, W, C, gz)
    near(gz, nhwc(4.0 * F.avg_pool2d(f(big), 2)) * dgelu(z.float()))
    # first layer and its weight gradient
    img, w9, b = rnd(N, H, W), rnd(9, C), rnd(C)
    pre, y = torch.zeros_like(z), torch.zeros(N, H, W, cs, dtype=torch.bfloat16, device='cuda')
    _unet_call(lib, 'clv_unet_first_fwd', img, w9, b, N, H, W, C, pre, y, cs, co)
    k = w9.reshape(3, 3, 1, C).permute(3, 2, 0, 1)
    zz = nhwc(F.conv2d(img[:, None].double(), k.double(), b.double(), padding=1)).float()
    near(pre, zz)
    near(y[..., co:co + C], F.gelu(zz))
    P = N * H * W
    tol = dict(rtol=0, atol=16 * P * 2.0 ** -23)
    nb = int(lib.clv_unet_rows_scratch_bytes(max(9 * C, (C + 1) * K)))
    scratch = torch.zeros(nb // 4 + 4, device='cuda')
    dw = torch.zeros(9, C, device='cuda')
    _unet_call(lib, 'clv_unet_first_wgrad', img, z, N, H, W, C, dw, scratch, ctypes.c_size_t(nb))
    cols = F.unfold(img[:, None].double(), 3, padding=1)  # (N, 9, HW)
    want = torch.einsum('ntp,npc->tc', cols, z.double().reshape(N, H * W, C))
    np.testing.assert_allclose(dw.cpu().numpy(), want.cpu().numpy(), **tol)
    # head, its gradients and a bias sum
    go, wh, bh = rnd(P, K), rnd(C, K), rnd(K)
    o = torch.zeros(P, K, device='cuda')
    _unet_call(lib, 'clv_unet_head_fwd', x, cs, co, wh, bh, ctypes.c_longlong(P), C, K, o)
    want = x[..., co:co + C].double().reshape(P, C) @ wh.double() + bh.double()
    np.testing.assert_allclose(o.cpu().numpy(), want.cpu().numpy(), rtol=0, atol=16 * C * 2.0 ** -23)
    dwb = torch.zeros(C + 1, K, device='cuda')
    _unet_call(lib, 'clv_unet_head_bwd', x, cs, co, z, go, wh, P, C, K, gz, dwb, scratch, ctypes.c_size_t(nb))
    near(gz.reshape(P, C), (go.double() @ wh.double().T).float() * dgelu(z.float()).reshape(P, C))
    xs = x[..., co:co + C].double().reshape(P, C)
    np.testing.assert_allclose(dwb[:C].cpu().numpy(), (xs.T @ go.double()).cpu().numpy(), **tol)
    np.testing.assert_allclose(dwb[C].cpu().numpy(), go.double().sum(0).cpu().numpy(), **tol)
    db = torch.zeros(C, device='cuda')
    _unet_call(lib, 'clv_unet_bias_grad', z, C, ctypes.c_longlong(P), C, db, scratch, ctypes.c_size_t(nb))
    np.testing.assert_allclose(db.cpu().numpy(), z.double().reshape(P, C).sum(0).cpu().numpy(), **tol)
