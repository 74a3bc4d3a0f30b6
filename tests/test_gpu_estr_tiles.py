"""The FP32-comp Estr on fields that mix its inner loop's branches: tiles and 8-source blocks in and
out of reach, coincident particles (inside and across tiles), static particles, remainders."""
import numpy as np
import pytest
import torch

import vpm_gb300 as vpm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel", [1, 2, 3])
@pytest.mark.parametrize("n", [1, 31, 41, 257, 3001])
def test_estr_blocks(n, kernel):
    rng = np.random.default_rng(n + kernel)
    # clusters a few core sizes wide, several reaches apart
    x = rng.integers(0, 3, (n, 3)) * 2.0 + 0.2 * rng.standard_normal((n, 3))
    if n > 40:
        x[n // 2:n // 2 + 10] = x[:10]          # coincident, far apart in the caller's order
        x[-9:] = x[-10]
    J = rng.standard_normal((n, 9))
    if n > 40:                                  # a field's J is the same where its particles coincide
        J[n // 2:n // 2 + 10], J[-9:] = J[:10], J[-10]
    T = lambda a: torch.tensor(a, device="cuda", dtype=torch.float64)       # noqa: E731
    x, gam, sig, J = T(x), T(rng.standard_normal((n, 3))), T(0.05 + 0.1 * rng.random(n)), T(J)
    static = torch.tensor(rng.random(n) < 0.1, device="cuda", dtype=torch.uint8)
    out = []
    for precision in (0, 1):
        S = torch.zeros(n, 3, device="cuda", dtype=torch.float64)
        vpm.default_context().estr_dev(x, J, x, gam, sig, J, S, kernel, precision, static_t=static, static_s=static)
        out.append(S)
    # Bound, target by target: a term z (J_t^T g - v) is rounded to 8 ulp of its two parts, and its
    # weight changes with s = (r/sigma)^2, whose distance is a difference of offsets within the
    # field's extent D, each rounded once: |ds| <= 2 sqrt(s)/sigma * sqrt(3) D 2^-23 + 4 s 2^-24.
    s = ((x[:, None] - x[None]) ** 2).sum(2) / sig[None] ** 2
    z, dlog = {1: lambda: (torch.exp(-s ** 1.5), 1.5 * s.sqrt()), 2: lambda: (torch.exp(-s / 2), 0.5 + 0 * s),
               3: lambda: ((1 + s) ** -3.5, 3.5 / (1 + s))}[kernel]()
    k = {1: 3 / (4 * np.pi), 2: (2 * np.pi) ** -1.5, 3: 7.5 / (4 * np.pi)}[kernel]
    z = k * z * (s > 0) * (1.0 - static.double())[None] / sig[None] ** 3
    D = (x.max(0).values - x.min(0).values).max()
    rel = 8 * 2.0 ** -24 + dlog * (2 * s.sqrt() / sig[None] * 3 ** 0.5 * D * 2.0 ** -23 + 4 * s * 2.0 ** -24)
    Jn, g = J.reshape(n, 9).norm(dim=1), gam.norm(dim=1)
    bound = (z * rel * (Jn[:, None] + Jn[None]) * g[None]).sum(1) + 1e-12 * out[0].norm() + 1e-15
    err = (out[1] - out[0]).norm(dim=1)
    assert (err <= bound).all(), float((err / bound).max())
