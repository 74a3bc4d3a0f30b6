"""The tensor-core tile path of the self-induced FP32-comp UJ (uj_tc.cu), against the FP64 form on
the same set: sizes at its threshold and with ragged last tiles and blocks, sets that put tiles in
each class (near, mid, far) and at the classes' limits, and scales at the ends of its ranges.
Tolerance: the FP32-comp bound of test_gpu_uj.py (1e-6 of the largest value)."""
import numpy as np
import pytest
import torch

from helpers import normwise, random_cloud

pytestmark = pytest.mark.gpu


def _uj(ctx, X, G, s, k, prec):
    n = X.shape[0]
    x, g, sg = (torch.tensor(a, device="cuda") for a in (X, G, s))
    U, J = (torch.zeros(n, c, dtype=torch.float64, device="cuda") for c in (3, 9))
    ctx.uj_dev(x, x, g, sg, U, J, k, prec)
    return U.cpu().numpy(), J.cpu().numpy()


def _check(ctx, X, G, s, k, what):
    a, b = _uj(ctx, X, G, s, k, 1), _uj(ctx, X, G, s, k, 0)
    for u, v, name in zip(a, b, "UJ"):
        assert np.isfinite(u).all(), f"{what}: {name} not finite"
        e = normwise(u, v)[0]
        assert e <= 1e-6, f"{what}: {name} {e:.3e}"


@pytest.mark.parametrize("k", [0, 1, 2, 3])
@pytest.mark.parametrize("n", [10239, 10240, 10241, 12351, 16417])
def test_tile_sizes(ctx, k, n):
    X, G, s = random_cloud(n, seed=n)
    _check(ctx, X, G, s, k, f"k={k} n={n}")


def _sets():
    n = 13000
    X, G, s = random_cloud(n, seed=5)
    yield "dense", (0.15 * X, G, s)                                # most tiles within the core's reach
    yield "offset", (X + np.array([3e4, -2e4, 1e4]), G, s)         # double-float differences
    Y = X.copy()
    Y[: n // 2] = 0.02 * Y[: n // 2] + 40.0                        # a far small cluster (distance ratio, one R)
    yield "clusters", (Y, G, s)
    Y = X.copy()
    Y[1::2] = Y[::2]                                               # coincident pairs
    yield "coincident", (Y, G, s)
    Y = X.copy()
    Y[:, 1:] *= 1e-3
    yield "needle", (Y, G, s)
    yield "cores wider than the tiles", (X, G, 30.0 * s)           # Winckelmans' weights go by the core size
    Y = X.copy()
    Y[:, 1:] = 0.25
    yield "line within a core", (0.1 * Y, G, s)
    H = G * 10.0 ** np.random.default_rng(3).uniform(-12, 0, (n, 1))
    yield "strengths over 12 decades", (X, H, s)
    H = G.copy()
    H[: n // 2] = 0.0
    yield "zero strengths", (X, H, s)
    yield "small scale", (1e-5 * X, 1e-12 * G, 1e-5 * s)
    yield "large scale", (1e5 * X, 1e9 * G, 1e5 * s)
    yield "sigma over 2 decades", (X, G, 10.0 ** np.random.default_rng(4).uniform(-3, -1, n))


@pytest.mark.parametrize("k", [2, 3])
@pytest.mark.parametrize("name,args", list(_sets()), ids=[n for n, _ in _sets()])
def test_tile_classes(ctx, k, name, args):
    _check(ctx, *args, k, f"k={k} {name}")


def test_nonfinite_source_reaches_every_target(ctx):
    X, G, s = random_cloud(13000, seed=6)
    G[777, 1] = np.nan
    U, J = _uj(ctx, X, G, s, 2, 1)
    assert not np.isfinite(U).all(axis=1).any() and not np.isfinite(J).all(axis=1).any()
