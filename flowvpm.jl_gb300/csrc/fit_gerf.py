"""Generates the coefficients of the Gaussian-erf pair functions in vpm_math.cuh
(gerf_GQ; gerf_S2_f64 and gerf_h_f64 in FP64).  Run by hand (numpy + scipy, mpmath for the FP64
forms); its output is pasted into the header.

The Gaussian-erf kernel's g(rho) = erf(rho/sqrt2) - sqrt(2/pi) rho e^{-rho^2/2}
(src/FLOWVPM_kernel.jl:45-84) enters the pair term through, with s = rho^2,

    G(s) = g/rho^3,        -H(s)/3 = (G - c2 e/3)/s,      c2 = sqrt(2/pi), e = e^{-s/2}.

Two forms cover s >= 0 with one exponential:

* s < 2 -- Kummer's series erf(x) = (2/sqrt pi) e^{-x^2} sum_n 2^n x^{2n+1}/(2n+1)!!
  turns both into series of positive terms (no cancellation at small s):
      G = c2 e (1/3 + s S2(s)),   -H/3 = c2 e S2(s),   S2(s) = sum_m s^m/(2m+5)!!;
  ten terms reach 2e-9 of S2 at s = 2.
* s >= 2 -- g = 1 - e (erfcx(rho/sqrt2) + c2 rho), erfcx(x) = e^{x^2} erfc(x) being
  smooth there; erfcx(rho/sqrt2) (1 + rho/2) is fitted by a degree-7 polynomial in
  w = A t + B, t = 1/(1 + rho/2), over rho in [sqrt2, 10] (relative least squares on
  Chebyshev nodes).  Beyond rho = 10 the caller caps rho, since e < 2e-22 there and
  G equals its singular form s^-1.5.

The printed check is the worst relative error of the fit itself (double precision).
"""
import numpy as np
from scipy.special import erfcx

K = 0.5
DEG = 7
RHO_LO, RHO_HI = np.sqrt(2.0), 10.0


def fit():
    n = 4000
    x = np.cos(np.pi * (np.arange(n) + 0.5) / n)
    tlo, thi = 1 / (1 + K * RHO_HI), 1 / (1 + K * RHO_LO)
    t = tlo + (thi - tlo) * (x + 1) / 2
    rho = (1 / t - 1) / K
    y = erfcx(rho / np.sqrt(2)) * (1 + K * rho)
    tc, th = (thi + tlo) / 2, (thi - tlo) / 2
    V = np.vander((t - tc) / th, DEG + 1, increasing=True)
    c, *_ = np.linalg.lstsq(V / y[:, None], np.ones_like(y), rcond=None)
    return c, 1 / th, -tc / th


def fit_f64():
    """FP64 forms: Chebyshev interpolation in 50 digits.  erfcx(rho/sqrt2) = t P(w), P of degree 16
    over rho in [sqrt2, 9]; S2 on [0, 2], degree 11.  Lowest powers first."""
    import mpmath as mp
    mp.mp.dps = 50

    def interp(f, deg):   # power coefficients in w on [-1, 1]
        nodes = [mp.cos(mp.pi * (k + mp.mpf(1) / 2) / (deg + 1)) for k in range(deg + 1)]
        V = mp.matrix(deg + 1, deg + 1)
        for i, x in enumerate(nodes):
            for j in range(deg + 1):
                V[i, j] = x ** j
        return mp.lu_solve(V, mp.matrix([f(x) for x in nodes]))

    tlo, thi = 1 / (1 + mp.mpf(9) / 2), 1 / (1 + mp.sqrt(2) / 2)
    tc, th = (thi + tlo) / 2, (thi - tlo) / 2

    def ex(w):
        t = tc + th * w
        rho = 2 * (1 / t - 1)
        return mp.exp(rho * rho / 2) * mp.erfc(rho / mp.sqrt(2)) / t

    def s2(s):
        return mp.nsum(lambda m: s ** m / mp.fac2(2 * m + 5), [0, mp.inf])

    c = interp(lambda w: s2(1 + w), 11)
    poly = [mp.mpf(0)] * 12                       # back to powers of s = 1 + w
    for j in range(12):
        for i in range(j + 1):
            poly[i] += c[j] * mp.binomial(j, i) * mp.mpf(-1) ** (j - i)
    return interp(ex, 16), 1 / th, -tc / th, poly


def main():
    c, A, B = fit()
    rho = np.linspace(RHO_LO, RHO_HI, 100001)
    t = 1 / (1 + K * rho)
    err = np.abs(np.polyval(c[::-1], A * t + B) * t / erfcx(rho / np.sqrt(2)) - 1).max()
    print(f"// w = {float(A)!r} t + {float(B)!r}; fit error {err:.2e}")
    for a in c[::-1]:
        print(f"    {float(a)!r}f,")
    d = 15.0
    print("// S2 series: 1/(2m+5)!!")
    for m in range(10):
        print(f"    {1.0 / d!r}f,")
        d *= 2 * m + 7
    c, A, B, p = fit_f64()
    print(f"// FP64: w = {float(A)!r} t + {float(B)!r}")
    for a in list(c)[::-1]:
        print(f"    {float(a)!r},")
    print("// FP64 S2")
    for a in p[::-1]:
        print(f"    {float(a)!r},")


if __name__ == "__main__":
    main()
