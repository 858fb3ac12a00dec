"""Axes longer than a tiled launch's grid: the per-cell kernel, or more planes a
block. The state is uniform along the long axis, so every column must give what a
short axis gives."""
import numpy as np
import pytest

from parity_util import make_cfg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('axis,n', [(1, 8 * 65535 + 1), (0, 5 * 65535 + 1)])
def test_ideal_stage_on_a_long_axis(cuda_lib, axis, n):
    from clvisc_b200.ideal import CLIdeal
    prof = np.linspace(4.0, 1.0, 24)
    out = []
    for m in (4, n):
        g = [1, 1, 24]
        g[axis] = m
        i = CLIdeal(make_cfg(*g, eos_type='ideal_gas'), hypersf_capacity=1000)
        ic = np.zeros((m, 24, 4), np.float32)
        ic[:, :, 0] = prof
        ic[:, :, 3] = 0.1
        i.load_ini(ic.reshape(-1, 4))
        for step in (1, 2):
            i.stepUpdate(step)
        out.append(i.field_to_host(i.d_ev[1]).reshape(m, 24, 4))
    np.testing.assert_array_equal(out[1][[0, 1, n // 2, n - 1]], out[0][:1].repeat(4, 0))
    assert (out[1] == out[1][:1]).all()
