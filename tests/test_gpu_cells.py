"""Line cells of the multi-level float32 sums: far lines through their cells' moments against
the same sums line by line and against the float64 engine, over chunk lengths, line densities,
widths and window edges where cells must be refused line by line."""

import numpy as np
import pytest
import torch

from pylblrtm_b200 import _lib, engine, synthetic
from pylblrtm_b200.spectral_data import SpectralData

pytestmark = pytest.mark.gpu


def _job(n_lines, step, tile, cutoff, n_pts, layers, shift, width, clustered, seed):
    lo = 1500.0
    hi = lo + (n_pts - 1.5) * step
    sd = synthetic.three_gas_lines(n_lines, lo - cutoff - 1.0, hi + cutoff + 1.0, seed=seed)
    lines = {k: v.copy() for k, v in sd.lines.items()}
    lines["Sref"] *= 1e-4
    lines["shift"] *= shift
    lines["g_air"] *= width
    lines["g_self"] *= width
    if clustered:                              # half of the lines in one band head
        rng = np.random.default_rng(seed)
        i = rng.random(n_lines) < 0.5
        lines["nu0"][i] = lo - 0.4 * cutoff + rng.exponential(0.02 * cutoff, int(i.sum()))
    sd = SpectralData(lines, dict(sd.tips), dict(sd.molar_masses), sd.molecule)
    prof = synthetic.logp_profile(layers + 1)
    return engine.Job(sd, engine.layer_input_from_profile(prof), engine.make_grid(lo, hi, step, tile), cutoff)


# (lines, step, tile, cut-off, points, layers, shift factor, width factor, clustered)
CASES = [(60_000, 0.001, 2.0, 25.0, 40_001, 6, 1.0, 1.0, False),     # the usual geometry
         (60_000, 0.001, 5.0, 25.0, 40_001, 4, 40.0, 1.0, False),    # three chunks per tile, wide shifts
         (9_000, 0.0023, 1.05, 10.3, 12_001, 5, 1.0, 1.0, True),     # ragged tiles, a band head
         (20_000, 0.001, 0.13, 5.0, 4_001, 5, 1.0, 1.0, False),      # 130-point chunks: the smallest cells
         (300, 0.001, 2.0, 25.0, 40_001, 5, 1.0, 1.0, False),        # sparse: few lines per cell
         (20_000, 0.001, 1.0, 25.0, 20_001, 3, 1.0, 8.0, False)]     # lines broader than a cell


@pytest.mark.parametrize("case", CASES)
def test_cells_against_lines_and_float64(cuda, case, monkeypatch):
    job = _job(*case, seed=int(case[0]))
    grid = job.grid
    assert _lib.load().lbl_line_cells_floats(1, grid.n_nu, grid.tile_samples, grid.step, job.cutoff) > 0
    with_cells = job.run("fp32", deterministic=True, count_evals=True)
    again = job.run("fp32", deterministic=True)
    assert torch.equal(with_cells.od, again.od)
    ref = job.run("fp64")
    real = _lib.call

    def no_cells(name, *args):
        if name == "lbl_tau_tiles_ml_f32":
            args = args[:-2] + (args[-2] & ~_lib.LBL_LINE_CELLS, args[-1])
        return real(name, *args)

    monkeypatch.setattr(_lib, "call", no_cells)
    by_line = job.run("fp32", deterministic=True, count_evals=True)
    assert with_cells.evals == by_line.evals and with_cells.work_split[1:] == by_line.work_split[1:]
    if case[0] >= 9_000 and case[7] == 1.0:
        assert with_cells.work_split[0] < 0.8 * by_line.work_split[0]
    err = lambda od: ((od.double() - ref.od).abs() / ref.od).max().item()
    # the cells' truncation is below 1e-8 of their sum; float32 rounding of either path is ~3e-7
    # of the far sum per point and, in a far wing that dominates, a few times that
    assert err(with_cells.od) <= err(by_line.od) + 5e-7
    l2 = lambda od: ((od.double() - ref.od).norm() / ref.od.norm()).item()
    assert l2(with_cells.od) <= 1.2 * l2(by_line.od) + 2e-8


@pytest.mark.parametrize("case", [c for c in CASES if c[0] != 60_000 or c[5] == 6])
def test_jacobian_cells_against_lines(cuda, case, monkeypatch):
    """The three Jacobian sums and the vector-Jacobian product with and without cells."""
    job = _job(*case, seed=int(case[0]) + 1)
    grid = job.grid
    assert _lib.load().lbl_line_cells_jac_floats(1, grid.n_nu, grid.tile_samples, grid.step, job.cutoff) > 0
    g = torch.rand((1, grid.n_nu), generator=torch.Generator().manual_seed(1), dtype=torch.float64).cuda()
    a, va = job.jacobian("H2O", deterministic=True), job.jacobian("H2O", g_tau=g, deterministic=True)
    assert all(torch.equal(x, y) for x, y in zip(a, job.jacobian("H2O", deterministic=True)))
    seen, real = [], _lib.call

    def no_cells(name, *args):
        if name == "lbl_jacobian_ml_f32":
            seen.append(args[-2] & _lib.LBL_LINE_CELLS)
            args = args[:-2] + (args[-2] & ~_lib.LBL_LINE_CELLS, args[-1])
        return real(name, *args)

    monkeypatch.setattr(_lib, "call", no_cells)
    b, vb = job.jacobian("H2O", deterministic=True), job.jacobian("H2O", g_tau=g, deterministic=True)
    assert seen == [_lib.LBL_LINE_CELLS] * 2
    for x, y in zip(a, b):
        # truncation below 1e-8 of the cells' sums, two float32 evaluations a few 1e-7 apart
        # (two leading terms of w' either way), per point against its layer's largest value
        scale = y.abs().amax(dim=2, keepdim=True).clamp_min(1e-300)
        assert ((x - y).abs() / scale).max().item() <= 2e-6
        assert ((x.double() - y.double()).norm() / y.double().norm()).item() <= 2e-7
    for x, y in zip(va, vb):
        assert torch.all((x - y).abs() <= 2e-6 * y.abs().max())


def test_geometries_without_cells(cuda):
    f = _lib.load().lbl_line_cells_floats
    assert f(3, 40_001, 2000, 0.001, 25.0) > 0
    assert f(3, 5_001, 2000, 0.001, 25.0) == 0          # three chunks: too few to share the cells
    assert f(3, 40_001, 100, 0.001, 25.0) == 0          # chunks shorter than two cells
    assert f(3, 40_001, 2000, 0.001, 3.9) == 0          # no line can be four half-widths out
    assert f(0, 40_001, 2000, 0.001, 25.0) == -1
