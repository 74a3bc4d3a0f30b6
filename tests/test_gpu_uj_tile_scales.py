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


@pytest.mark.parametrize("strengths", ["equal", "one in 2", "one in 8", "one in 64", "lognormal"])
def test_coherent_sums_are_not_low(ctx, strengths):
    """Strengths of one direction in a ball, and the velocity they induce at a distance: the tensor cores
    truncate their sums, which without a correction for the tile's own strengths leaves U low by 0.4e-7 to
    2.4e-7 on average.  Bound: 2e-8 for the approximate square root of the weights (what the pairwise kernel
    shows) and a quarter of an FP32 unit, 3e-8, for the expectation."""
    rng = np.random.default_rng(3)

    def ball(n):
        v = rng.standard_normal((n, 3))
        return v / np.linalg.norm(v, axis=1, keepdims=True) * rng.random((n, 1)) ** (1 / 3)

    n = 12_800
    X = np.concatenate([ball(n), ball(n) + [6.0, 1.8, 0.6]])
    w = {"equal": np.ones(n), "lognormal": np.exp(rng.standard_normal(n))}.get(strengths)
    if w is None:
        w = (rng.random(n) < 1 / int(strengths.split()[-1])) * 1.0
    G = np.concatenate([w[:, None] * [0.2, 0.5, 1.0], np.zeros((n, 3))]) * (1 + 4e-4 * rng.standard_normal((2 * n, 1)))
    s = np.full(2 * n, 0.01)
    a, b = uj(ctx, X, G, s, 0, 1)[0][n:], uj(ctx, X, G, s, 0, 0)[0][n:]
    bias = float(((a - b) * b).sum() / (b * b).sum())
    assert abs(bias) <= 5e-8, f"{bias:.2e}"


@pytest.mark.parametrize("k", [2, 3])
@pytest.mark.parametrize("field", ["cloud", "rings", "one sign", "one in 64", "six decades", "planar"])
def test_no_further_off_than_pair_by_pair(ctx, k, field):
    """U and J of the tensor pass against the pairwise kernel's of the same set in Morton order, both
    against FP64: equal errors (a quarter for chance; U to 6e-8 at least, an FP32 unit)."""
    from vpm_gb300 import workloads
    X, G, s = random_cloud(30_000, seed=8)
    rng = np.random.default_rng(8)
    if field == "rings":
        X, G, s = workloads.leapfrog_rings(30_000, 10)
        X = X + 2e-3 * rng.standard_normal(X.shape)
    elif field == "one sign":
        G = np.abs(G) * [0, 0, 1]
    elif field == "one in 64":
        G[np.arange(len(G)) % 64 > 0] = 0
    elif field == "six decades":
        G = G * 10.0 ** rng.uniform(-6, 0, (len(G), 1))
    elif field == "planar":
        G = G * [1e-5, 1e-5, 1]
    q = ((X - X.min(0)) / (X.max(0) - X.min(0)) * 1023).astype(np.int64)
    key = sum(((q[:, a] >> b) & 1) << (3 * b + a) for b in range(10) for a in range(3))
    X, G, s = (v[np.argsort(key)] for v in (X, G, s))
    ref, tile, pair = uj(ctx, X, G, s, k, 0), uj(ctx, X, G, s, k, 1), uj(ctx, X, G, s, k, 1, cross=True)
    for r, a, b, name in zip(ref, tile, pair, "UJ"):
        for c in range(3) if field == "planar" and name == "U" else (slice(None),):
            e, f = normwise(a[:, c], r[:, c])[1], normwise(b[:, c], r[:, c])[1]
            assert e <= max(1.25 * f, 6e-8 if name == "U" else 0.0), f"{name}{c}: {e:.2e} {f:.2e}"
