"""Wavenumber shards on grids long enough for line cells: every tile range equals the full job
bit for bit from only the lines of its window, wherever the window's edge cuts a cell."""

import pytest
import torch

from pylblrtm_b200 import _lib, engine, shard, synthetic

pytestmark = pytest.mark.gpu


# (lines per cm-1, cut-off, shards): cut-offs that put the window's edge inside a cell, sparse to
# ordinary line densities; the last with a gas that is absent from every other level pair, so that
# cells hold inactive lines
@pytest.mark.parametrize("density,cutoff,world,absent", [(67, 10.3, 4, False), (40, 10.3, 8, False),
                                                         (40, 24.9, 8, False), (9, 7.77, 6, False),
                                                         (40, 10.3, 8, True)])
def test_shard_jobs_equal_the_full_job(cuda, density, cutoff, world, absent):
    lo, hi = 1500.0, 1547.3                                 # 24 tiles, the last one partial
    a, b = lo - cutoff - 1.0, hi + cutoff + 1.0
    sd = synthetic.scale_strengths(synthetic.three_gas_lines(int(density * (b - a)), a, b, seed=density), 1e-4)
    prof = synthetic.profile_from_levels(synthetic.logp_levels(7))
    li = engine.layer_input_from_profile(prof)
    if absent:
        vmr = li.levels_vmr.copy()
        vmr[:, 0, 2:5] = 0.0
        li = engine.LayerInput(gases=li.gases, levels_p=li.levels_p, levels_t=li.levels_t, levels_vmr=vmr)
    grid = engine.make_grid(lo, hi, 0.001, 2.0)
    assert _lib.load().lbl_line_cells_floats(1, grid.n_nu, grid.tile_samples, grid.step, cutoff) > 0
    n_tiles = -(-grid.n_nu // grid.tile_samples)
    job = engine.Job(sd, li, grid, cutoff)
    full = job.run("fp32", deterministic=True).od
    for r in range(world):
        sl = shard.tile_span(n_tiles, world, r)
        first, count = sl.start, sl.stop - sl.start
        win = shard.line_window(sd, grid, cutoff, li.p_max_atm(), first, count)
        sj = engine.Job(sd, li, grid, cutoff, line_window=win)
        assert sj.n_bound < job.n_bound
        od = sj.run("fp32", deterministic=True, tiles=(first, count)).od
        i0 = first * grid.tile_samples
        assert torch.equal(od, full[:, :, i0:i0 + od.shape[2]]), (r, first, count)
