"""Particles so far away that r^2 overflows FP32 (parked ones, without strength, too): they add nothing, also
beside near sources in a group."""
import numpy as np
import pytest
import torch

from helpers import normwise, random_cloud

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [0, 1, 2])
@pytest.mark.parametrize("n", [300, 13_000])
@pytest.mark.parametrize("strength", [0.0, 1.0])
def test_particles_past_fp32_distances(ctx, k, n, strength):
    X, G, s = random_cloud(n, seed=n)
    X[7::50] = 1e25
    G[7::50] *= strength
    x, g, sg = (torch.tensor(a, device="cuda") for a in (X, G, s))
    out = []
    for prec in (0, 1):
        U, J = (torch.zeros(n, c, dtype=torch.float64, device="cuda") for c in (3, 9))
        ctx.uj_dev(x, x, g, sg, U, J, k, prec)
        out.append((U.cpu().numpy(), J.cpu().numpy()))
    here = np.ones(n, bool)
    here[7::50] = False
    for a, b, name in zip(out[1], out[0], "UJ"):
        e = normwise(a[here], b[here])[0]
        assert np.isfinite(a[here]).all() and e <= 1e-6, f"{name}: {e:.3e}"
