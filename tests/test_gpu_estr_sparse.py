"""The FP32-comp Estr of sets whose particles are far apart against their core sizes: the sums are a few
close pairs, whose displacements a warp's wide box of targets must not round."""
import numpy as np
import pytest
import torch

import vpm_gb300 as vpm

pytestmark = pytest.mark.gpu


def sparse(n, seed, outlier=0.0):
    """A random cloud of the unit cube with cores of 0.01 to 0.03, and J and Gamma of its own."""
    rng = np.random.default_rng(seed)
    x, g, sig, J = rng.random((n, 3)), rng.standard_normal((n, 3)), 0.01 + 0.02 * rng.random(n), rng.standard_normal((n, 9))
    if outlier:
        x[n // 3] = outlier
    return [torch.tensor(a, device="cuda") for a in (x, g, sig, J)]


def bound(x, g, sig, J, kernel):
    """By target: a term z (J_t^T g - v) is rounded to 8 ulp of its two parts and its weight by the
    rounding of s = (r/sigma)^2, 8 ulp of s at a displacement rounded to its own size; terms past the
    kernel's reach, whose weight is below 1e-13 of zeta(0), are left out."""
    out = []
    k = {1: 3 / (4 * np.pi), 2: (2 * np.pi) ** -1.5, 3: 7.5 / (4 * np.pi)}[kernel]
    Jn, gn = J.norm(dim=1), g.norm(dim=1)
    for a in range(0, x.shape[0], 2000):
        s = ((x[a:a + 2000, None] - x[None]) ** 2).sum(2) / sig[None] ** 2
        z, dlog = {1: lambda: (torch.exp(-s ** 1.5), 1.5 * s.sqrt()), 2: lambda: (torch.exp(-s / 2), 0.5 + 0 * s),
                   3: lambda: ((1 + s) ** -3.5, 3.5 / (1 + s))}[kernel]()
        z = (s > 0) * k / sig[None] ** 3 * (z * 8 * 2.0 ** -24 * (1 + dlog * s) + 1e-13)
        out.append((z * (Jn[a:a + 2000, None] + Jn[None]) * gn[None]).sum(1))
    return torch.cat(out)


@pytest.mark.parametrize("kernel", [1, 2, 3])
@pytest.mark.parametrize("n", [33, 700, 1630, 4099])
def test_close_pairs(ctx, n, kernel):
    for seed in range(8):
        x, g, sig, J = sparse(n, seed)
        S = [torch.zeros(n, 3, device="cuda", dtype=torch.float64) for _ in range(2)]
        for precision in (0, 1):
            ctx.estr_dev(x, J, x, g, sig, J, S[precision], kernel, precision)
        err = (S[1] - S[0]).norm(dim=1)
        lim = bound(x, g, sig, J, kernel) + 1e-13 * S[0].norm()
        assert (err <= lim).all(), f"seed {seed}: {float((err / lim).max()):.2f}"


@pytest.mark.parametrize("kernel", [2, 3])
@pytest.mark.parametrize("n", [4099, 12_000])
def test_close_pairs_beside_a_far_particle(ctx, n, kernel):
    x, g, sig, J = sparse(n, 1, outlier=1e3)
    S = [torch.zeros(n, 3, device="cuda", dtype=torch.float64) for _ in range(2)]
    for precision in (0, 1):
        ctx.estr_dev(x, J, x, g, sig, J, S[precision], kernel, precision)
    err = (S[1] - S[0]).norm(dim=1)
    lim = bound(x, g, sig, J, kernel) + 1e-13 * S[0].norm()
    assert (err <= lim).all(), f"{float((err / lim).max()):.2f}"


@pytest.mark.parametrize("kernel", [1, 2, 3])
@pytest.mark.parametrize("n", [33, 700, 1630, 4099])
def test_close_pairs_adjoint(ctx, n, kernel):
    """The same for the Estr adjoint.  Bounds by particle: the terms of the gradients, as the sums of
    their parts' magnitudes, each rounded to 8 ulp (16 ulp where the displacement, kappa = d log(zeta)/ds
    and the pair's weight w multiply) and by the rounding of s as above."""
    k = {1: 3 / (4 * np.pi), 2: (2 * np.pi) ** -1.5, 3: 7.5 / (4 * np.pi)}[kernel]
    for seed in range(8):
        x, g, sig, J = sparse(n, seed)
        Sb = torch.tensor(np.random.default_rng(seed + 99).standard_normal((n, 3)), device="cuda")
        out = []
        for precision in (0, 1):
            o = [torch.zeros(n, *c, device="cuda", dtype=torch.float64) for c in ((3,), (3,), (), (9,))]
            ctx.estr_adjoint_dev(x, g, sig, J, Sb, *o, kernel, precision)
            out.append([v.reshape(n, -1) for v in o])
        Jn, gn, bn = J.norm(dim=1), g.norm(dim=1), Sb.norm(dim=1)
        lim = [torch.zeros(n, device="cuda", dtype=torch.float64) for _ in range(4)]
        for a in range(0, n, 2000):
            t = slice(a, min(n, a + 2000))
            s = ((x[t, None] - x[None]) ** 2).sum(2) / sig[None] ** 2
            z, dlog, kap = {1: lambda: (torch.exp(-s ** 1.5), 1.5 * s.sqrt(), 3 * s.sqrt()),
                            2: lambda: (torch.exp(-s / 2), 0.5 + 0 * s, 1 + 0 * s),
                            3: lambda: ((1 + s) ** -3.5, 3.5 / (1 + s), 7 / (1 + s))}[kernel]()
            e = (s > 0) * k / sig[None] ** 3 * (z * 8 * 2.0 ** -24 * (1 + dlog * s) + 1e-13)
            w = 2 * (Jn[t, None] + Jn[None]) * gn[None] * bn[t, None]
            ex, es = e * kap * s.sqrt() / sig[None] * w, e * (kap * s + 3) / sig[None] * w
            lim[0][t] += ex.sum(1)
            lim[0] += ex.sum(0)
            lim[1] += (e * (Jn[t, None] + Jn[None]) * bn[t, None]).sum(0)
            lim[2] += es.sum(0)
            lim[3][t] += bn[t] * (e * gn[None]).sum(1)
            lim[3] += gn * (e * bn[t, None]).sum(0)
        for p, q, m, name in zip(out[1], out[0], lim, ("x", "Gamma", "sigma", "J")):
            err = (p - q).norm(dim=1)
            m = m + 1e-13 * q.norm()
            assert (err <= m).all(), f"{name}, seed {seed}: {float((err / m).max()):.2f}"
