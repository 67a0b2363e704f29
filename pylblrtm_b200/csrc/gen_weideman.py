"""Generate weideman_coeffs.h: coefficients of Weideman's rational approximation.

J.A.C. Weideman (1994), "Computation of the complex error function", SIAM J.
Numer. Anal. 31(5):1497-1518: for Im z >= 0,

    w(z) ~ 2 sum_{n=1..N} a_n Z^(n-1) / (L - iz)^2 + 1 / (sqrt(pi) (L - iz)),
    Z = (L + iz) / (L - iz),  L = (N / sqrt(2))^(1/2),

where a_n are the Fourier coefficients of (L^2 + t^2) exp(-t^2) under the map
t = L tan(theta/2), obtained here by an FFT on 4N points. Three sets: N = 36 (|w|
relative error <= 2e-14 for |z| <= 6), N = 48 (the float64 engine inside |z|^2 < 49: Re w
relative error <= 5e-12 for y >= 1e-3, <= 5e-11 for y >= 1e-4, growing as 1/y below) and N = 28 (the near zones of the float32 multi-level engine and its Jacobians: Re w relative error <= 7e-7
for y >= 1e-4 and <= 1e-8 for y >= 0.01 inside |z|^2 < 36, against
scipy.special.wofz; float32 rounding of the sums is ~1e-7). Beside them the positive nodes
(squared) of 16-point Gauss-Hermite quadrature and 2/pi times their weights, which the float64
engine takes next to the real axis. Run:

    python pylblrtm_b200/csrc/gen_weideman.py > pylblrtm_b200/csrc/weideman_coeffs.h
"""

import numpy as np

SETS = (("LBL_WEIDEMAN", 36), ("LBL_WEIDEMAN28", 28), ("LBL_WEIDEMAN48", 48))


def coefficients(n: int):
    m = 2 * n
    k = np.arange(-m + 1, m)
    big_l = np.sqrt(n / np.sqrt(2.0))
    t = big_l * np.tan(k * np.pi / m / 2.0)
    f = np.concatenate([[0.0], np.exp(-t ** 2) * (big_l ** 2 + t ** 2)])
    a = np.real(np.fft.fft(np.fft.fftshift(f))) / (2 * m)
    return big_l, a[1:n + 1]          # a_1 .. a_N


def print_list(name, values):
    print(f"#define {name} \\")
    for i in range(0, len(values), 3):
        tail = ", \\" if i + 3 < len(values) else ""
        print("    " + ", ".join(repr(float(v)) for v in values[i:i + 3]) + tail)


def main():
    print("// Generated by gen_weideman.py: Weideman (1994) rational approximation of w(z).")
    print("#pragma once")
    for name, n in SETS:
        big_l, a = coefficients(n)
        print(f"#define {name}_N {n}")
        print(f"#define {name}_L {float(big_l)!r}")
        print("// a_1 .. a_N (polynomial in Z: sum a_n Z^(n-1)), as an initializer list")
        print_list(f"{name}_COEFFS", a)
    t, w = np.polynomial.hermite.hermgauss(16)
    print("// 16-point Gauss-Hermite quadrature: t_k^2 and (2/pi) w_k for the eight positive nodes")
    print_list("LBL_HERMITE16_T2", t[8:] ** 2)
    print_list("LBL_HERMITE16_W", w[8:] * 2.0 / np.pi)


if __name__ == "__main__":
    main()
