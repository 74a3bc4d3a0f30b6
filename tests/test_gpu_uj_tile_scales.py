"""The tensor pass of the FP32-comp UJ at the limits of its number ranges: length units, core sizes and
strengths against each other, with ragged last tiles.  The sums are scale-free, so the tolerance is that
of test_gpu_uj_tiles.py (1e-6 of the largest value) in any unit."""
import numpy as np
import pytest
import torch

from helpers import normwise, random_cloud

pytestmark = pytest.mark.gpu


def uj(ctx, X, G, s, k, prec, cross=False):
    """U, J; cross: with the sources in arrays of their own, which the pairwise kernel takes."""
    n = X.shape[0]
    x, g, sg = (torch.tensor(a, device="cuda") for a in (X, G, s))
    U, J = (torch.zeros(n, c, dtype=torch.float64, device="cuda") for c in (3, 9))
    ctx.uj_dev(x, x.clone() if cross else x, g, sg, U, J, k, prec)
    return U.cpu().numpy(), J.cpu().numpy()


def check(ctx, X, G, s, k, what):
    for u, v, name in zip(uj(ctx, X, G, s, k, 1), uj(ctx, X, G, s, k, 0), "UJ"):
        assert np.isfinite(u).all(), f"{what}: {name} not finite"
        e = normwise(u, v)[0]
        assert e <= 1e-6, f"{what}: {name} {e:.3e}"


@pytest.mark.parametrize("k", [2, 3])
@pytest.mark.parametrize("n", [13057, 13060, 13064, 13119])     # last tiles of 1, 4, 8 and 63
@pytest.mark.parametrize("S", [1e-4, 1.0, 1e2, 1.3e2, 1e5])
def test_wide_cores_in_any_unit(ctx, k, n, S):
    X, G, s = random_cloud(n, seed=n)
    for wide in (3.0, 6.0, 30.0):
        check(ctx, S * X, S ** 3 * G, wide * S * s, k, f"k={k} n={n} S={S} wide={wide}")


@pytest.mark.parametrize("tiny", [1e-3, 1e-9, 1e-12])
def test_tiny_cores_among_ordinary_ones(ctx, tiny):
    """Particles without strength whose cores are 1e-4 to 1e-13 of their neighbours' (particles that have
    lost theirs): they add nothing to U and J."""
    X, G, s = random_cloud(13000, seed=11)
    X, s = 1e3 * X, 3e3 * s
    G[5::37] = 0.0
    s[5::37] = tiny
    check(ctx, X, G, s, 2, f"tiny={tiny}")


def test_long_sums_of_one_sign(ctx):
    """J of 100,000 particles of two vortex rings, whose near pairs add up coherently.  The FP32 sums of 4
    near tiles are 8 additions, each rounded to 0.29 ulp rms of a sum within a factor of two: about
    sqrt(8) 0.29 2^-23 / 2 = 4.9e-8."""
    from vpm_gb300 import workloads
    X, G, s = workloads.leapfrog_rings(100_000, 10)
    X = X + 2e-3 * np.random.default_rng(0).standard_normal(X.shape)
    (_, a), (_, b) = uj(ctx, X, G, s, 2, 1), uj(ctx, X, G, s, 2, 0)
    e = normwise(a, b)[1]
    assert e <= 5e-8, f"{e:.3e}"


@pytest.mark.parametrize("k", [2, 3])
@pytest.mark.parametrize("small", [1e-3, 1e-5, 1e-7])
def test_small_strength_components(ctx, k, small):
    """Strengths nearly along z: the small velocity across the plane comes from their small components
    alone, and is as accurate as the large ones: within 1e-6 of its own largest value."""
    X, G, s = random_cloud(20_000, seed=31)
    H = G * [small, small, 1.0]
    a, b = uj(ctx, X, H, s, k, 1)[0], uj(ctx, X, H, s, k, 0)[0]
    for c in range(3):
        e = normwise(a[:, c], b[:, c])[0]
        assert e <= 1e-6, f"U{c}: {e:.3e}"
