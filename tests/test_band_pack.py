"""Native scan and pack of the lines inside the band mask against the general scan and NumPy:
short lists (one thread), lists at the edges of the thread parts, skipped groups, edge values,
narrowed bands and more pairs than the first table holds."""

import numpy as np
import pytest

from pylblrtm_b200 import engine
from pylblrtm_b200.spectral_data import SpectralData


def _list(n, seed, n_iso=3):
    rng = np.random.default_rng(seed)
    lines = {k: rng.uniform(0.0, 1.0, n) for k in engine.LINE_KEYS}
    lines["nu0"] = rng.uniform(600.0, 700.0, n)
    lines["shift"] = rng.uniform(-0.5, 0.5, n)
    lines["mol_id"] = rng.choice([1, 2, 3, 99], n).astype(np.int64)
    lines["iso_id"] = rng.integers(1, n_iso + 1, n).astype(np.int32)
    for i, v in zip(rng.integers(0, n, 6), (np.nan, np.inf, -np.inf, 650.0, 640.0 - 5.0, 660.0 + 5.0)):
        lines["nu0"][i] = v
    lines["shift"][rng.integers(0, n)] = np.nan
    pairs = {(m, i) for m in (1, 2, 3) for i in range(1, n_iso + 1)}
    t = np.array([100.0, 300.0]), np.array([1.0, 2.0])
    return SpectralData(lines, {p: t for p in pairs}, {p: 18.0 for p in pairs}, None)


@pytest.mark.filterwarnings("ignore::RuntimeWarning")
@pytest.mark.parametrize("n,n_iso", [(7, 2), (1000, 30), (65535, 3), (65537, 3), (200_003, 2), (300_000, 40)])
def test_band_scan_and_pack(n, n_iso):
    sd = _list(n, n, n_iso)
    gases, lo, hi, cutoff, p_max = ["H2O", "O3"], 640.0, 660.0, 5.0, 0.9      # CO2 is not in the profile
    st = {}
    groups, gid = engine.select_groups(sd, gases, lo, hi, cutoff, p_max, 2, stats=st)
    got, band, count, smax = engine.select_band(sd, gases, lo, hi, cutoff, p_max, 2)
    assert [(g.mol_id, g.iso_id) for g in got] == [(g.mol_id, g.iso_id) for g in groups]
    assert count == st["band_lines"] and smax == st["max_abs_shift"]
    sb = np.abs(sd.lines["shift"]) * p_max
    inside = lambda a, b: (sd.lines["nu0"] >= a - sb) & (sd.lines["nu0"] <= b + sb)
    assert np.array_equal(band.line[:band.n], np.flatnonzero(inside(lo - cutoff, hi + cutoff)))
    job = engine.Job.__new__(engine.Job)                     # its packing alone, no device
    job.p_max = p_max
    for win in (None, (650.0, 651.0)):
        job.narrowed = win is not None
        job.mask_lo, job.mask_hi = engine.band_edges(lo, hi, cutoff, win)
        want = np.flatnonzero(inside(job.mask_lo, job.mask_hi) & (gid >= 0))
        kept = job._pack(band, None, None, 0)
        assert kept == want.size and (win is not None or kept == count)
        cols, g = np.zeros((7, kept + 1)), np.zeros(kept + 1, np.int32)
        assert job._pack(band, cols, g, kept + 1) == kept
        for c, k in zip(cols, engine.LINE_KEYS):
            assert np.array_equal(c[:kept], sd.lines[k][want], equal_nan=True)
        assert np.array_equal(g[:kept], gid[want])
        if kept:
            with pytest.raises(RuntimeError, match="lbl_pack_band"):
                job._pack(band, cols[:, :kept - 1].copy(), g, kept - 1)


def test_short_columns_are_refused():
    sd = _list(50, 1)
    sd.lines["g_air"] = sd.lines["g_air"][:40]
    with pytest.raises(ValueError, match="as many values"):
        engine.select_band(sd, ["H2O"], 640.0, 660.0, 5.0, 1.0, 2)


@pytest.mark.gpu
@pytest.mark.parametrize("window", [None, (998.0, 1003.0)])
def test_packed_and_whole_uploads_agree(window, monkeypatch):
    """The two uploads (band lines packed, whole list) give the same spectrum bit for bit."""
    import torch

    from pylblrtm_b200 import synthetic
    sd = synthetic.three_gas_lines(20_011, 950.0, 1050.0, seed=5)
    li = engine.layer_input_from_profile(synthetic.logp_profile(5))
    grid = engine.make_grid(999.0, 1002.0, 0.001, 2.0)
    ods, sizes = [], []
    for whole in (False, True):
        monkeypatch.setattr(engine.Job, "_mostly_in_band", lambda self, nu0: whole)
        job = engine.Job(sd, li, grid, 10.0, line_window=window)
        ods.append(job.run("fp32", deterministic=True).od)
        sizes.append((job.n_lines, job.n_bound))
    assert torch.equal(*ods) and sizes[0][0] == sizes[0][1] == sizes[1][1] and sizes[1][0] == 20_011
