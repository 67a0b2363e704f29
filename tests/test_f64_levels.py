"""Float64 engine: the Chebyshev levels, the list of near lines and the direct sums at the
edges of their intervals, and the forms of Re w it takes by distance."""

import ctypes

import numpy as np
import pytest

from oracle import restate


@pytest.mark.parametrize("form,terms,lo,hi,tol", [
    # Weideman's approximation is uniform to ~1e-16 of w(0), so of Re w >= y / (sqrt(pi) 49)
    # it keeps 1e-16 * 87 / y ~ 1e-11 at y = 1e-3 and the rounding of 48 terms above
    ("weideman", 48, 0.0, 49.0, 2e-11),
    # first omitted terms 4e-16 and 3e-16 (|z|^2 = 49, 100); wofz itself carries ~1e-13
    ("series", 22, 49.0, 100.0, 2e-13),
    ("series", 13, 100.0, 400.0, 2e-13)])
def test_re_w_forms(form, terms, lo, hi, tol):
    from scipy.special import wofz
    from pylblrtm_b200.csrc import build
    lib = ctypes.CDLL(build.HOST_LIB)
    fn = getattr(lib, f"lbl_host_{form}_re")
    rng = np.random.default_rng(terms)
    for y0 in (1e-3, 1e-2, 0.3, 2.0, 5.0):
        x = np.sqrt(rng.uniform(max(lo - y0 * y0, 0.0), hi - y0 * y0, 4000))
        y, re = np.full_like(x, y0), np.empty_like(x)
        p = lambda a: ctypes.c_void_p(a.ctypes.data)
        assert fn(p(x), p(y), ctypes.c_longlong(x.size), terms, p(re)) == 0
        ref = wofz(x + 1j * y).real
        assert np.max(np.abs(re / ref - 1.0)) <= tol, y0


# Tile sizes in points around the few-point path (16), a segment's node count and size (16, 32),
# a sub-chunk (256) and a chunk (512); 130 points leave every tile's last one ragged.
@pytest.mark.gpu
@pytest.mark.parametrize("tile_pts,n_pts", [(1, 5), (15, 130), (16, 130), (17, 130), (33, 130), (49, 130),
                                            (257, 600), (273, 600), (513, 1030), (1025, 1300), (1300, 1300)])
def test_levels_against_oracle(tile_pts, n_pts):
    import warnings

    from pylblrtm_b200 import engine, synthetic
    sd = synthetic.three_gas_lines(3000, 995.0, 1015.0, seed=11)      # 1,500 in one sub-chunk's list at 0.005
    prof = synthetic.logp_profile(4)
    step, cutoff = 0.005, 3.0
    lo = 1003.0
    hi = lo + (n_pts - 1.5) * step
    tile = (tile_pts + 0.25) * step
    p, t, v, c = restate.build_layers(prof.pressure_hpa, prof.temperature_k, prof.vmr)
    nu = restate.grid(lo, hi, step)
    assert nu.size == n_pts
    ref = restate.optical_depth(nu, sd.lines, sd.tips, sd.molar_masses, p, t, v, c, cutoff, tile)
    n_ev = restate.count_evals(nu, sd.lines, sd.tips, sd.molar_masses, p, t, v, c, cutoff, tile)
    grid = engine.make_grid(lo, hi, step, tile)
    with warnings.catch_warnings():
        warnings.simplefilter("error")
        res = engine.optical_depth(sd, engine.layer_input_from_profile(prof), grid, cutoff, precision="fp64",
                                   count_evals=True)
    od = res.od[0].cpu().numpy()
    assert res.evals == n_ev
    # interpolation and rounding of ~1,000 terms stay at 1e-14; wofz and the near forms at 1e-12
    assert np.max(np.abs(od / ref - 1.0)) <= 1e-11
    again = engine.optical_depth(sd, engine.layer_input_from_profile(prof), grid, cutoff, precision="fp64")
    assert np.array_equal(again.od[0].cpu().numpy(), od)             # fixed summation order
