"""Partial sums of the line cells: lines and cells add up in float64 across threads, so a spectrum of
far wings alone is about as close to float64 by cells as line by line."""

import numpy as np
import pytest
import torch

from pylblrtm_b200 import _lib, engine, synthetic

pytestmark = pytest.mark.gpu


# 3,700 lines per cell (more than a thread sums in float at a time), none within the grid. What the
# cells add beyond the interpolation and the rounding that both paths share is one float32 rounding per
# moment and the node's polynomial. Ratio of the norm errors: 1.12 and 1.16 (od of the Jacobian 1.16
# and 1.18); with float32 sums across threads 1.35 and 1.47 (1.38 and 1.45).
@pytest.mark.parametrize("seed", [1, 2])
def test_far_wings_by_cells_are_as_close_as_line_by_line(cuda, seed, monkeypatch):
    left, right = (synthetic.three_gas_lines(100_000, a, a + 13.5, seed=10 * seed + i) for i, a in enumerate((1475.5, 1551.0)))
    left.lines.update({k: np.concatenate([v, right.lines[k]]) for k, v in left.lines.items()})
    sd = synthetic.scale_strengths(left, 1e-6)
    li = engine.layer_input_from_profile(synthetic.logp_profile(5))
    job = engine.Job(sd, li, engine.make_grid(1500.0, 1540.0, 0.001, 2.0), 25.0)
    ref = job.run("fp64").od
    seen = ref > 0.05 * ref.amax(dim=2, keepdim=True)
    real = _lib.call

    def no_cells(name, *args):
        if name in ("lbl_tau_tiles_ml_f32", "lbl_jacobian_ml_f32"):
            assert args[-2] & _lib.LBL_LINE_CELLS
            args = args[:-2] + (args[-2] & ~_lib.LBL_LINE_CELLS, args[-1])
        return real(name, *args)

    def errors():
        for od in (job.run("fp32", deterministic=True).od, job.jacobian("H2O", deterministic=True)[0]):
            yield ((od.double() - ref) / ref)[seen].square().mean().sqrt().item()

    cells = list(errors())
    monkeypatch.setattr(_lib, "call", no_cells)
    for by_cell, by_line in zip(cells, errors()):
        assert by_cell <= 1.25 * by_line
