"""Where line cells are built: only on grids whose tiles can use them."""

import pytest

from pylblrtm_b200 import _lib


def _sizes(n_nu, tile, step, cutoff):
    lib = _lib.load()
    return (lib.lbl_line_cells_floats(3, n_nu, tile, step, cutoff), lib.lbl_line_cells_jac_floats(3, n_nu, tile, step, cutoff))


# (points per tile, step, cut-off): a tile's window takes at most 512 cells of a quarter chunk
# (chunks of at most 2,048 points; Jacobian 1,024), three on either side included
@pytest.mark.parametrize("tile,step,cutoff,forward,jacobian", [
    (2000, 0.001, 25.0, True, True),           # the default: 104 and 208 cells
    (5000, 0.0004, 25.0, True, False),         # 312 and 526
    (10000, 0.0002, 25.0, False, False),       # 526 and 1,046
    (20000, 0.0001, 25.0, False, False),
    (250, 0.001, 25.0, False, False),          # 817 (smallest cells: 62 points, taken as 64)
    (390, 0.001, 25.0, False, False),          # 525 cells of 97 points
    (400, 0.001, 25.0, True, True),            # 510 of 100
    (250, 0.001, 10.3, True, True)])
def test_cells_only_where_a_tile_takes_them(tile, step, cutoff, forward, jacobian):
    fwd, jac = _sizes(64 * tile + 1, tile, step, cutoff)
    assert (fwd > 0, jac > 0) == (forward, jacobian) and fwd >= 0 and jac >= 0


# Sizes on either side of the limit: where cells are built they are used (fewer node evaluations than
# line by line), the sums agree with float64 either way, and no cell is built that no tile takes.
@pytest.mark.gpu
@pytest.mark.parametrize("tile,step", [(0.4, 0.001), (0.39, 0.001), (2.0, 0.0004), (2.0, 0.0002)])
def test_built_cells_are_used(cuda, tile, step, monkeypatch):
    from pylblrtm_b200 import engine, synthetic
    lo, cutoff = 1500.0, 25.0
    hi = lo + 20.3 * max(tile, 1.0)
    sd = synthetic.scale_strengths(synthetic.three_gas_lines(6000, lo - cutoff, hi + cutoff, seed=3), 1e-4)
    prof = synthetic.profile_from_levels(synthetic.logp_levels(4))
    job = engine.Job(sd, engine.layer_input_from_profile(prof), engine.make_grid(lo, hi, step, tile), cutoff)
    calls, real = [], _lib.call

    def spy(drop):
        def call(name, *args):
            calls.append(name)
            if drop and name == "lbl_tau_tiles_ml_f32":
                args = args[:-2] + (args[-2] & ~_lib.LBL_LINE_CELLS, args[-1])
            return real(name, *args)
        return call

    monkeypatch.setattr(_lib, "call", spy(False))
    res = job.run("fp32", deterministic=True, count_evals=True)
    built = "lbl_line_cells" in calls
    monkeypatch.setattr(_lib, "call", spy(True))
    by_line = job.run("fp32", deterministic=True, count_evals=True)
    assert built == (job.grid.tile_samples in (400, 5000))
    assert res.evals == by_line.evals and (res.work_split[0] < by_line.work_split[0]) == built
    ref = job.run("fp64").od
    err = ((res.od.double() - ref).abs() / ref).max().item()
    assert err <= ((by_line.od.double() - ref).abs() / ref).max().item() + 5e-7
