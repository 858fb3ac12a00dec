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
