"""The tolerance build's FP64 EOS lookup at the energy densities where a row or
a column of the table begins, which a lookup that rounds instead of truncating
gets from the texel before. The reference's formula (eos_table.h:39-62) with the
divisions through reciprocals, restated in numpy."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from clvisc_b200.eos import Eos
from parity_util import make_cfg
from test_fast_gpu import TOL, field_errors

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope='module')
def lookup(tmp_path_factory, cuda_lib):
    out = str(tmp_path_factory.mktemp('eos') / 'libeoscheck.so')
    subprocess.check_call(['nvcc', '-gencode', 'arch=compute_100a,code=sm_100a', '-O3', '--fmad=true', '-prec-div=false',
                           '-prec-sqrt=false', '-Xcompiler', '-fPIC', '-shared', '-o', out,
                           os.path.join(HERE, 'cuda', 'eos_check.cu')])
    f = ctypes.CDLL(out).run_f64
    fp, dp, i, r = ctypes.POINTER(ctypes.c_float), ctypes.POINTER(ctypes.c_double), ctypes.c_int, ctypes.c_float
    f.argtypes = [fp, i, i, r, r, i, r, r, dp, i, dp]
    return f


def restated(table, nrow, ncol, start, step, e):
    f = np.float32
    start, step = f(start), f(step)
    epr = np.float64(step * f(ncol))
    row = np.trunc(e * (1.0 / epr))
    x = e - np.float64(start) - row * epr
    col = np.trunc(x * (1.0 / np.float64(step)))
    r = (x - (col.astype(f) * step).astype(np.float64)) * (1.0 / np.float64(step))
    row, col = row.astype(np.int64), col.astype(np.int64)
    wrap = col + 1 == ncol
    row2, col2 = row + wrap, np.where(wrap, 0, col + 1)
    at = lambda a, b: table[np.clip(a, 0, nrow - 1) * ncol + np.clip(b, 0, ncol - 1)].astype(np.float64)
    r = r[:, None]
    return (1.0 - r) * at(row, col) + r * at(row2, col2)


@pytest.mark.parametrize('nrow,ncol,start,step', [
    (100, 1000, 0.0, 0.01), (100, 1555, 0.0, 0.002), (7, 13, 0.0, 0.3), (1, 40, 0.0, 0.25), (5, 1, 0.0, 0.5),
    (9, 10, 0.05, 0.3), (9, 10, 0.7, 0.3), (9, 10, -0.4, 0.3)])
def test_fp64_lookup(lookup, nrow, ncol, start, step):
    """Row and column starts, their neighbours on either side, energies below
    the table's first texel and random ones; inside the table's last texel but
    one and beyond it."""
    f = np.float32
    n = nrow * ncol
    k = np.arange(n, dtype=np.float64)
    table = np.stack([0.1 + k / n, (k + 1) ** 1.2, np.sqrt(k + 1), (k + 1) ** 0.8], 1).astype(f)
    width, top = np.float64(f(step) * f(ncol)), np.float64(f(step)) * n
    rng = np.random.default_rng(n)
    e = np.concatenate([width * np.arange(nrow), np.float64(f(step)) * rng.integers(0, n, 400),
                        rng.uniform(-0.5 * step, top, 400), [0.0, -0.0, -0.3 * step, -1.7 * step, 0.5 * start]])
    e = np.concatenate([e, np.nextafter(e, np.inf), np.nextafter(e, -np.inf)])
    top32 = f(start) + f(n) * f(step)
    inner = min(top32, f(n - 2) * f(step)) if start == 0.0 else f(-1.0)
    out = np.zeros((e.size, 4))
    p = lambda a, t: a.ctypes.data_as(ctypes.POINTER(t))
    rc = lookup(p(table, ctypes.c_float), nrow, ncol, f(start), f(step), n, top32, inner, p(e, ctypes.c_double), e.size,
                p(out, ctypes.c_double))
    assert rc == 0
    want = restated(table, nrow, ncol, start, step, e)
    # the weight to rounding: 2^-52 of e / step, times the texels' difference
    tol = 4 * 2.0 ** -52 * (top / step + 4) * np.abs(np.diff(table.astype(np.float64), axis=0)).max(0, initial=0.0)
    tol = tol + 4 * 2.0 ** -52 * np.abs(want).max(0)
    bad = np.abs(out - want) > tol
    assert not bad.any(), (e[bad.any(1)][:5], out[bad.any(1)][:5], want[bad.any(1)][:5])


@pytest.mark.parametrize('eos', ['ideal_gas', 'lattice_wb', 'pure_gauge'])
def test_fp64_step_at_row_starts(cuda_lib, oracle_mod, eos):
    """One fused step of fluid at rest with uniform e = 10, 20, .., 300 GeV/fm^3,
    the starts of these tables' rows, against the oracle."""
    from clvisc_b200.visc import CLVisc
    cfg = make_cfg(4, 4, 1, use_float32=False, arithmetic='fast', eos_type=eos)
    v, o = CLVisc(cfg), oracle_mod.OracleVisc(cfg)
    for e in range(10, 301, 10):
        ic = np.zeros((16, 4), cfg.real)
        ic[:, 0] = e
        for h in (v, o):
            h.load_ini(ic)
            h.IS_initialize()
            h.update_time(-1)
            h.step(0)
        errs = field_errors(v.ideal.field_to_host(v.ideal.d_ev[1]), o.ideal.d_ev[1], v.pi_to_host(1), o.d_pi[1],
                            Eos(eos), float(v.ideal.tau))
        assert max(x for q, x in errs.items() if q != 'components') <= TOL[False], (e, errs)


@pytest.mark.parametrize('use_float32', [True, False])
def test_table_that_starts_above_zero(cuda_lib, oracle_mod, use_float32):
    """A user's table that starts 25 texels above zero: energy densities below
    its first texel (clamped, and extrapolated in the texel's own width), and in
    its second row and third row, whose first columns lie below the row's start."""
    from clvisc_b200.visc import CLVisc
    eos = Eos('lattice_pce165')
    eos.ed_start = 0.05
    cfg = make_cfg(9, 8, 40, use_float32=use_float32, arithmetic='fast')
    v, o = CLVisc(cfg, handcrafted_eos=eos), oracle_mod.OracleVisc(cfg, handcrafted_eos=eos)
    n = 9 * 8 * 40
    ic = np.zeros((n, 4), cfg.real)
    ic[:, 0] = np.concatenate([np.linspace(0.0007, 0.11, n // 2), np.linspace(0.1107, 8.0, n // 2)])
    for h in (v, o):
        h.load_ini(ic)
        h.IS_initialize()
        h.step(0)
    errs = field_errors(v.ideal.field_to_host(v.ideal.d_ev[1]), o.ideal.d_ev[1], v.pi_to_host(1), o.d_pi[1], eos,
                        float(v.ideal.tau))
    assert max(x for q, x in errs.items() if q != 'components') <= TOL[use_float32], errs
