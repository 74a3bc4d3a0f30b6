"""Static targets of the near-field Estr are left as they are, also where a group's sums are split over
several warps (few particles) and added afterwards."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", [50, 3001])
def test_static_targets_are_untouched(ctx, n, precision):
    rng = np.random.default_rng(n)
    T = lambda a: torch.tensor(a, device="cuda", dtype=torch.float64)       # noqa: E731
    x, gam, sig = T(rng.random((n, 3))), T(rng.standard_normal((n, 3))), T(0.1 + 0.1 * rng.random(n))
    static = torch.tensor(rng.random(n) < 0.3, device="cuda", dtype=torch.uint8)
    U, J, S = (torch.zeros(n, c, device="cuda", dtype=torch.float64) for c in (3, 9, 3))
    S.fill_(-0.0)
    ctx.p2p_leaflist_dev(x, gam, sig, U, J, S, leaf_size=20, theta=0.5, precision=precision, sfs=True, static=static)
    assert torch.signbit(S[static.bool()]).all() and (S[static.bool()] == 0).all()
    assert (S[~static.bool()] != 0).any()
