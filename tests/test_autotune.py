"""Launch-shape candidates: tuning must be able to end on what an untuned run
takes."""
import pytest

from clvisc_b200.autotune import candidates


@pytest.mark.parametrize('use_float32', [True, False])
@pytest.mark.parametrize('fast', [True, False])
@pytest.mark.parametrize('nz', [1, 12, 65])
def test_automatic_choice_is_a_candidate(nz, use_float32, fast):
    c = candidates(nz, use_float32, fast)
    assert any(x['kernel'] == 0 and x['chunk'] == 0 and x['tile'] == 0 for x in c)
    assert len({tuple(sorted(x.items())) for x in c}) == len(c)
    if nz == 1:
        assert all(x['kernel'] != 2 for x in c)  # the (3+1)D tiles leave 31 of 32 threads idle
    else:
        assert any(x['kernel'] == 2 and 0 < x['chunk'] < 16 for x in c)


@pytest.mark.gpu
@pytest.mark.parametrize('grid', [(41, 37, 1), (33, 31, 26)])
def test_tune_times_the_automatic_choice(cuda_lib, grid):
    from clvisc_b200.autotune import reset, tune_visc
    from clvisc_b200.visc import CLVisc
    from parity_util import make_cfg, seeded_ic
    cfg = make_cfg(*grid, arithmetic='fast')
    v = CLVisc(cfg)
    v.load_ini(seeded_ic(cfg))
    v.IS_initialize()
    try:
        best, table = tune_visc(v, steps=2)
        own = table['kernel0_tile0_chunk0_blocks2']
        key = 'kernel%d_tile%d_chunk%d_blocks%d' % (best['kernel'], best['tile'], best['chunk'], best['blocks'])
        assert table[key] == min(table.values()) <= own
    finally:
        reset(v)
