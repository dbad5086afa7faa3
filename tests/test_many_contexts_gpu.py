"""Contexts that are alive together share pages of mapped host memory for the energies
of flosic_sic_getvlxc_device, 32 to a page: each must get its own, whatever the order
in which contexts come and go.  The same call on the same inputs gives the same bits."""
import numpy as np
import pytest

from publicrelease_2020_b200 import sic as S
from publicrelease_2020_b200 import workloads as W

pytestmark = pytest.mark.gpu


def test_energies_of_many_contexts():
    import torch

    n = 500
    sysm = W.small_synthetic()
    rng = np.random.default_rng(3)
    rho = torch.zeros((10, n), dtype=torch.float64, device="cuda")
    rho[0] = torch.from_numpy(rng.uniform(0.1, 1.0, n)).cuda()
    v = torch.empty(2 * n, dtype=torch.float64, device="cuda")
    weights = [torch.full((n,), 1.0 + i, dtype=torch.float64, device="cuda") for i in range(40)]

    def open_ctx():
        ctx = S.FlosicSIC()
        ctx.set_geometry(sysm)
        return ctx

    def call(ctx, i):
        return ctx.getvlxc_device(n, rho.data_ptr(), n, weights[i].data_ptr(), v.data_ptr())

    want = []
    for i in range(40):  # one context at a time
        ctx = open_ctx()
        want.append(call(ctx, i))
        ctx.close()
    assert len({tuple(e) for e in want}) == 40
    ctxs = [open_ctx() for _ in range(40)]  # more than a page holds
    try:
        for rounds in range(2):
            for i in list(range(40))[::-1]:
                assert np.array_equal(call(ctxs[i], i), want[i]), i
            for i in range(rounds, 40, 3):  # slots in the middle of both pages go and come again
                ctxs[i].close()
            for i in range(rounds, 40, 3):
                ctxs[i] = open_ctx()
        for i in range(32):  # the first page's contexts, then calls of the others
            ctxs[i].close()
        for i in range(32, 40):
            assert np.array_equal(call(ctxs[i], i), want[i]), i
    finally:
        for c in ctxs:
            c.close()
