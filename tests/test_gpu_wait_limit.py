"""A wait inside a kernel that runs out: the kernel ends in order, the call returns the timeout status and
the context stays usable.  The limit of 0 rounds (one look) makes the waits of the tensor pass run out at
once."""
import numpy as np
import pytest
import torch

import vpm_gb300 as vpm
from helpers import normwise, random_cloud

pytestmark = pytest.mark.gpu
TIMEOUT = -5


@pytest.mark.parametrize("k", [0, 1, 2, 3])
def test_waits_that_run_out_are_reported(ctx, k):
    n = 13_001
    X, G, s = random_cloud(n, seed=2)
    d = [torch.tensor(a, device="cuda") for a in (X, G, s)]

    def call(c, prec, m=n):
        U, J = (torch.zeros(m, w, dtype=torch.float64, device="cuda") for w in (3, 9))
        c.uj_dev(d[0][:m], d[0][:m], d[1][:m], d[2][:m], U, J, k, prec)
        return U.cpu().numpy(), J.cpu().numpy()

    ref = call(ctx, 0)
    mine = vpm.Context(0)
    try:
        for _ in range(2):
            mine.set_wait_rounds(0)
            with pytest.raises(vpm.VPMError) as e:
                call(mine, 1)
            assert e.value.code == TIMEOUT
            call(mine, 1, 4000)                       # a size without such waits
            P = np.zeros((46, n), order="F")
            P[:3], P[3:6], P[6] = X.T, G.T, s
            with pytest.raises(vpm.VPMError) as e:
                mine.uj(P, n, k, 1, 2)
            assert e.value.code == TIMEOUT
            for a, b in zip(call(ctx, 1), ref):       # another context is not concerned
                assert normwise(a, b)[0] <= 1e-6
            mine.set_wait_rounds(1 << 16)
            for a, b in zip(call(mine, 1), ref):
                assert normwise(a, b)[0] <= 1e-6
    finally:
        mine.close()


def test_wait_rounds_out_of_range():
    c = vpm.Context(0)
    for bad in (-1, (1 << 16) + 1):
        with pytest.raises(vpm.VPMError):
            c.set_wait_rounds(bad)
    c.close()
