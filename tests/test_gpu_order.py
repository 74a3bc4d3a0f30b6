"""The curve ordering of the targets and sources at its edges: one and two particles, remainders of
the counted ranks (33, 35, ...), their last size and that of the 32-bit keys and the next ones, and
sets without extent along some or all axes.  The FP32-comp U, J of the ordered set against the FP64 form's (whose sums do not depend
on the order); tolerance: the FP32-comp bound of test_gpu_uj.py.  The Winckelmans kernel: 65,536
random points of a line have neighbours at 1e-7 core sizes, where the literal FP64 form of the
Gaussian-erf kernel, a difference of nearly equal terms, has no digits left to compare with."""
import numpy as np
import pytest
import torch

from helpers import normwise, random_cloud

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", ["cloud", "line", "plane", "point"])
@pytest.mark.parametrize("n", [1, 2, 700, 1024, 1025, 2049, 4097, 6144, 6145, 65536, 65537, 31, 33, 35, 20479, 20480, 20481])
def test_ordered_sums(ctx, n, shape):
    X, G, s = random_cloud(n, seed=n)
    if shape == "line":
        X[:, 1:] = 0.25
    elif shape == "plane":
        X[:, 2] = -3.0
    elif shape == "point":
        X[:] = (0.3, -0.2, 7.0)
    d = [torch.tensor(a, device="cuda") for a in (X, G, s)]
    out = {}
    for prec in (0, 1):
        U, J = (torch.zeros(n, c, dtype=torch.float64, device="cuda") for c in (3, 9))
        ctx.uj_dev(d[0], d[0], d[1], d[2], U, J, 3, prec)
        out[prec] = U.cpu().numpy(), J.cpu().numpy()
    for a, b, name in zip(out[1], out[0], "UJ"):
        e = normwise(a, b)[0]
        assert np.isfinite(a).all() and e <= 1e-6, f"{name}: {e:.3e}"
