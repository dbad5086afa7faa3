"""The launch count of flosic_sic_stats against the kernels that CUDA records
(torch's profiler sees every kernel of the process): each entry point adds as many
as it launches, whatever the route of its calls."""
import pytest

from publicrelease_2020_b200 import sic as S
from publicrelease_2020_b200 import workloads as W
from publicrelease_2020_b200.batch import Batch

pytestmark = pytest.mark.gpu


def _kernels(call):
    import torch
    from torch.profiler import ProfilerActivity, profile

    call()  # buffers are allocated, kernels loaded
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        call()
        torch.cuda.synchronize()
    return sum(1 for e in prof.events() if "flosic::" in e.name)


CYCLES = {
    # both spins in one evaluation; in the mixed mode apart (fewer than 16 FOs a spin)
    "water": (lambda: W.water(seed=0, nrad=12), "fp64", "phi2"),
    "water_mixed": (lambda: W.water(seed=0, nrad=12), "mixed", "phi2"),
    # calls of one slot and of several, FO products on the GPU (40 FOs)
    "synthetic_40": (lambda: W.synthetic(natoms=10, nbasis=128, nmsh=3000, nfo=40, box_ang=7.56, seed=1), "fp64",
                     "phi2"),
    "synthetic_40_mixed": (lambda: W.synthetic(natoms=10, nbasis=128, nmsh=3000, nfo=40, box_ang=7.56, seed=1),
                           "mixed", "phi2"),
    "synthetic_pairs": (lambda: W.small_synthetic(), "fp64", "pairs"),
}


@pytest.mark.parametrize("name", list(CYCLES))
def test_cycle(name):
    make, precision, density = CYCLES[name]
    ctx = S.open_system(make())
    try:
        ctx.set_precision(precision)
        ctx.set_density_mode(density)
        assert _kernels(ctx.cycle) == ctx.stats()["launches"]
    finally:
        ctx.close()


def test_coupot1():
    ctx = S.open_system(W.water(seed=0, nrad=12))
    try:
        counts = []

        def call():
            before = ctx.stats()["launches"]
            ctx.coupot1()
            counts.append(ctx.stats()["launches"] - before)

        assert _kernels(call) == counts[-1]
    finally:
        ctx.close()


def test_batch():
    b = Batch(W.alkane_batch(n=3, seed=100, max_carbons=3, nrad=(6, 8)))
    try:
        assert _kernels(b.cycle) == sum(c.stats()["launches"] for c in b.ctxs)
    finally:
        b.close()
