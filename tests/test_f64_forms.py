"""Float64 engine: Re w next to the real axis and below it (lines of very small, zero or negative
width), where a form that is only accurate relative to w(0) is not accurate enough."""

import ctypes
import warnings

import numpy as np
import pytest

from oracle import restate


def general_voigt(nu, centers, doppler, lorentz):
    """restate.voigt by the general float64 method (Gautschi's) in place of scipy's wofz."""
    from pylblrtm_b200.csrc import build
    lib = ctypes.CDLL(build.HOST_LIB)
    z = restate.SQRT_LN2 * ((nu[:, None] - centers) + 1j * lorentz) / doppler
    x, y = np.ascontiguousarray(z.real), np.ascontiguousarray(z.imag)
    re, im = np.empty_like(x), np.empty_like(x)
    p = lambda a: ctypes.c_void_p(a.ctypes.data)
    lib.lbl_host_faddeeva_f64(p(x), p(y), ctypes.c_longlong(x.size), p(re), p(im))
    return re * (restate.VOIGT_K / doppler)


# |z|^2 around every change of form: Weideman, quadrature (28.41, 33, 36, 42), 22 terms (49), 13 (100), 7 (400)
BANDS = [(0.0, 9.0), (9.0, 28.4), (28.41, 33.0), (33.0, 36.0), (36.0, 42.0), (42.0, 49.0), (49.0, 64.0), (64.0, 100.0),
         (100.0, 400.0), (400.0, 700.0), (700.0, 1e4)]
WIDTHS = [0.0, 1e-160, 1e-30, 1e-12, 1e-8, 1e-6, 1e-5, 9.9e-5, 1e-4, 9e-4, 2e-3, 0.011, 0.11, 1.0, 3.0]


@pytest.mark.parametrize("sign", [1.0, -1.0])
@pytest.mark.parametrize("y0", WIDTHS)
def test_re_w_no_further_off_than_the_general_method(y0, sign):
    from scipy.special import wofz
    from pylblrtm_b200.csrc import build
    lib = ctypes.CDLL(build.HOST_LIB)
    p = lambda a: ctypes.c_void_p(a.ctypes.data)
    rng = np.random.default_rng(7)
    for lo, hi in BANDS:
        if hi <= y0 * y0:
            continue
        x = np.sqrt(rng.uniform(max(lo - y0 * y0, 0.0), hi - y0 * y0, 3000))
        x[::2] *= -1.0
        y, re, old, im = np.full_like(x, sign * y0), np.empty_like(x), np.empty_like(x), np.empty_like(x)
        n = ctypes.c_longlong(x.size)
        lib.lbl_host_re_w_f64(p(x), p(y), n, p(re))
        lib.lbl_host_faddeeva_f64(p(x), p(y), n, p(old), p(im))
        ref = wofz(x + 1j * y)
        # below the axis Re w changes sign near the core: relative to |w| there
        scale = np.abs(ref) if sign < 0 and lo < 28.0 else np.abs(ref.real)
        keep = scale > 1e-290
        err, err_old = (np.max(np.abs(v - ref.real)[keep] / scale[keep]) if keep.any() else 0.0 for v in (re, old))
        # rounding: exp(-x^2) carries x^2 ulp, wofz a few ulp
        assert err <= 1.05 * err_old + 4e-15 + 2e-16 * hi * (y0 < 1e-3 and hi <= 700.0), (lo, hi, err, err_old)


# One line list, widths from the air-broadening column, at the few-point path (8 points a tile) and in
# chunks with three levels; the reference sums wofz at every point.
@pytest.mark.gpu
@pytest.mark.parametrize("tile_pts", [8, 700])
@pytest.mark.parametrize("width", [0.0, 1e-12, 3e-9, 1e-6, -1e-9, -1e-6, -1e-4])
def test_small_and_negative_widths(tile_pts, width, monkeypatch):
    from pylblrtm_b200 import engine, synthetic
    sd = synthetic.co2_band(12, 719.98, 720.02, seed=5)
    for k in ("g_air", "g_self"):
        sd.lines[k] = np.full(sd.lines["nu0"].size, width)
    prof = synthetic.logp_profile(2)
    lo, step, cutoff = 719.95, 1e-4, 0.3
    hi, tile = lo + 999.5 * step, (tile_pts + 0.25) * step
    p, t, v, c = restate.build_layers(prof.pressure_hpa, prof.temperature_k, prof.vmr)
    nu = restate.grid(lo, hi, step)
    ref = restate.optical_depth(nu, sd.lines, sd.tips, sd.molar_masses, p, t, v, c, cutoff, tile)
    with warnings.catch_warnings():
        warnings.simplefilter("error")
        res = engine.optical_depth(sd, engine.layer_input_from_profile(prof), engine.make_grid(lo, hi, step, tile), cutoff,
                                   precision="fp64")
    od = res.od[0].cpu().numpy()
    # |x| > 6 from every line: the quadrature's 6e-13 and Gaussian tails, which turn an ulp of x into
    # 2 x^2 ulp. Nearer, where every form is only accurate relative to the strongest line's w(0): no
    # further off than the general method's sum. Negative widths cancel against the Gaussian, so
    # relative to the sum for the opposite widths.
    ad = np.sqrt(2 * np.log(2) * 8.314462618 * t[0] / 0.04399) / 299792458.0 * 720.0
    s = np.sqrt(np.log(2)) / ad
    x = np.abs(nu[:, None] - sd.lines["nu0"][None, :]) * s
    near = x.min(axis=1)
    assert np.sum(near > 6.0) > 100 and np.sum(near < 3.0) > 100
    if width >= 0:
        scale = np.abs(ref)
    else:
        up = dict(sd.lines, g_air=-sd.lines["g_air"], g_self=-sd.lines["g_self"])
        scale = restate.optical_depth(nu, up, sd.tips, sd.molar_masses, p, t, v, c, cutoff, tile)
    big = scale > 1e-290
    err = np.abs(od - ref) / np.where(big, scale, 1.0)
    assert np.max(err[0, (near > 6.0) & big[0]]) <= 5e-12
    monkeypatch.setattr(restate, "voigt", general_voigt)
    general = restate.optical_depth(nu, sd.lines, sd.tips, sd.molar_masses, p, t, v, c, cutoff, tile)
    at = near < 3.0
    assert np.max(err[0, at]) <= 1e-12 + np.max(np.abs(general - ref)[0, at] / scale[0, at])


# One line, 24 to 700 Doppler units away, summed point by point: one reciprocal and the series per value, in
# the wings of small, ordinary and large y. The reference sums the asymptotic series in long double (wofz
# carries 5e-15 at y = 36). Ratios to the median take the line's strength out; what is left is a dozen
# roundings of 1.1e-16 (an uncorrected estimate of 1/|z|^2 would show 1e-6, one Newton step 1e-12).
@pytest.mark.gpu
@pytest.mark.parametrize("width", [1e-4, 0.02, 1.0])
def test_reciprocal_of_the_wings(width, monkeypatch):
    from pylblrtm_b200 import engine, synthetic

    def series_voigt(nu, centers, doppler, lorentz):
        z = (restate.SQRT_LN2 * ((nu[:, None] - centers) + 1j * lorentz) / doppler).astype(np.clongdouble)
        u, s = 1 / (z * z), np.zeros_like(z)
        for k in range(30, -1, -1):                          # (2k - 1)!! / 2^k z^-2k by Horner
            s = 1 + (k + np.longdouble(0.5)) * u * s
        return (-(s / z).imag / np.sqrt(np.longdouble(np.pi))).astype(np.float64) * (restate.VOIGT_K / doppler)

    monkeypatch.setattr(restate, "voigt", series_voigt)
    sd = synthetic.co2_band(1, 719.9999, 720.0001, seed=3)
    for k in ("g_air", "g_self"):
        sd.lines[k] = np.full(1, width)
    prof = synthetic.logp_profile(2)
    lo, step, cutoff = 720.02, 5e-4, 1.0
    hi, tile = lo + 999.5 * step, 8.25 * step
    p, t, v, c = restate.build_layers(prof.pressure_hpa, prof.temperature_k, prof.vmr)
    ref = restate.optical_depth(restate.grid(lo, hi, step), sd.lines, sd.tips, sd.molar_masses, p, t, v, c, cutoff, tile)
    res = engine.optical_depth(sd, engine.layer_input_from_profile(prof), engine.make_grid(lo, hi, step, tile), cutoff,
                               precision="fp64")
    ratio = (res.od[0].cpu().numpy() / ref)[0]
    assert np.max(np.abs(ratio / np.median(ratio) - 1.0)) <= 3e-15
