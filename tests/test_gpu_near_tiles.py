"""The near-field UJ sums, FP32-comp against FP64 on the same lists, where the groups of four sources
take each of their branches: targets of several leaves in a group (masks), coincident particles,
pairs on both sides of the series' limit, list lengths that are no multiple of four or 32."""
import numpy as np
import pytest
import torch

import vpm_gb300 as vpm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel", [0, 1, 2, 3])
@pytest.mark.parametrize("n,leaf", [(1, 1), (33, 5), (130, 7), (1501, 50), (4099, 20)])
def test_near_uj_blocks(n, leaf, kernel):
    rng = np.random.default_rng(n + kernel)
    x = rng.random((n, 3))
    if n > 40:
        x[5:9], x[n // 2] = x[4], x[20]                     # coincident
    T = lambda a: torch.tensor(a, device="cuda", dtype=torch.float64)       # noqa: E731
    h = n ** (-1 / 3)
    x, gam, sig = T(x), T(rng.standard_normal((n, 3))), T(h * (0.4 + 1.2 * rng.random(n)))
    ctx = vpm.default_context()
    out = []
    for precision in (0, 1):
        U, J = (torch.zeros(n, k, device="cuda", dtype=torch.float64) for k in (3, 9))
        ctx.p2p_leaflist_dev(x, gam, sig, U, J, leaf_size=leaf, theta=0.5, kernel=kernel, precision=precision)
        out.append((U, J))
    # a pair's terms are rounded to ~16 ulp (displacement, weight, products; J's r^-5 and the singular
    # kernel's nearest pairs included), its distance to one ulp of the unit cube's coordinates' low parts
    for a, b in zip(out[1], out[0]):
        assert (a - b).norm() <= 16 * 2.0 ** -24 * b.norm() + 1e-14


@pytest.mark.parametrize("shift", [0.0, 1e5, 1e7])
def test_near_sums_far_from_the_origin(shift):
    """Coordinates of up to 10^8 core sizes, where FP32 does not resolve a core: the box tests that choose
    the pair form and skip sources have to see the low parts too."""
    rng = np.random.default_rng(8)
    n = 2000
    T = lambda a: torch.tensor(a, device="cuda", dtype=torch.float64)       # noqa: E731
    x, gam, sig = T(rng.random((n, 3)) + shift), T(rng.standard_normal((n, 3))), T(0.1 * (0.7 + 0.6 * rng.random(n)))
    out = []
    for precision in (0, 1):
        U, J, S = (torch.zeros(n, k, device="cuda", dtype=torch.float64) for k in (3, 9, 3))
        vpm.default_context().p2p_leaflist_dev(x, gam, sig, U, J, S, leaf_size=20, theta=0.5, precision=precision, sfs=True)
        out.append((U, J))
    # as above, and the coordinates' own rounding to 2^-48 of the shift against distances near 0.03
    for a, b in zip(out[1], out[0]):
        assert (a - b).norm() <= (16 * 2.0 ** -24 + 5 * shift * 2.0 ** -48 / 0.03) * b.norm()


@pytest.mark.parametrize("leaf,theta", [(1, 0.4), (3, 0.9), (64, 0.0)])
@pytest.mark.parametrize("spread", [1e-9, 3e-8, 1e-7, 1e-6])
def test_lists_of_points_closer_than_fp32_centres(spread, leaf, theta):
    """Points far closer than FP32 resolves across the field: the device's FP32 acceptance test has to
    leave these to FP64, and the lists stay the host builder's."""
    rng = np.random.default_rng(3)
    n = 1200
    x = rng.random((40, 3)).repeat(n // 40, 0) + spread * rng.standard_normal((n, 3)) + 5.0
    host = vpm._lib.leaflist_host(x, leaf, theta)
    dev = vpm.default_context().leaflist_dev(torch.tensor(x, device="cuda"), leaf, theta)
    for h, d in zip(host, dev):
        assert np.array_equal(np.asarray(h), np.asarray(d.cpu() if isinstance(d, torch.Tensor) else d))
