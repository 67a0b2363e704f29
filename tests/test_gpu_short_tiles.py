"""Short tiles and the short last tile of a grid: the multi-level sums around the smallest chunk
with a far-field level and the CTA sizes (1, 2, 4 and 8 warps), against the float64 engine."""

import pytest
import torch

from pylblrtm_b200 import engine, synthetic

pytestmark = pytest.mark.gpu


# points of the last tile behind 2,000-point tiles: lanes by lines (8 points, Jacobian 4), then
# level 1; and whole grids of short tiles: 1 to 8 warps per CTA of either kernel
@pytest.mark.parametrize("tile_pts,n_pts", [(2000, 4000 + k) for k in (1, 4, 5, 8, 9, 12, 33, 64, 65)] +
                         [(9, 95), (50, 500), (128, 700), (130, 700), (256, 900), (258, 900), (512, 1300), (513, 1300),
                          (700, 1500), (1025, 2100)])
@pytest.mark.parametrize("deterministic", [False, True])
def test_short_tiles_against_float64(cuda, tile_pts, n_pts, deterministic):
    sd = synthetic.scale_strengths(synthetic.three_gas_lines(4000, 1480.0, 1520.0, seed=4), 1e-4)
    li = engine.layer_input_from_profile(synthetic.logp_profile(5))
    job = engine.Job(sd, li, engine.Grid(1500.0, 0.001, n_pts, tile_pts), 25.0)
    ref = job.run("fp64", count_evals=True)
    res = job.run("fp32", deterministic=deterministic, count_evals=True)
    assert res.evals == ref.evals
    err = lambda od: ((od.double() - ref.od).abs() / ref.od).max().item()
    # the engine's float32 accuracy on long tiles (1e-6) with a third as a margin for the worst point
    assert err(res.od) <= 3e-6
    jac = job.jacobian("H2O", deterministic=deterministic)
    assert err(jac[0]) <= 3e-6
    # derivatives: the same points on one long tile whose window admits the same lines (the
    # cut-off holds the whole list)
    wide = lambda ts: engine.Job(sd, li, engine.Grid(1500.0, 0.001, n_pts, ts), 60.0).jacobian("H2O", deterministic=True)
    for x, y in zip(wide(tile_pts)[1:], wide(2500 if n_pts < 2500 else 5000)[1:]):
        assert ((x - y).abs() / y.abs().amax(dim=2, keepdim=True)).max().item() <= 5e-6
