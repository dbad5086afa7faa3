"""Device memory of a Coulomb evaluation.

The scratch of a cycle is bounded by its coefficient rows: per (pair, FO) 52
doubles, the centre-of-gravity partials (4 doubles) and a byte, per (call, FO) the
geometry (64 bytes), 52 moments and a list entry, beside the arrays on the mesh.
The per-FO kernels' operand order needs no second copy of any of them, and the
partial sums of their call list use memory that the XC step takes anyway."""
import pytest

from publicrelease_2020_b200 import sic as S
from publicrelease_2020_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _held_by_a_cycle(sysm):
    import torch

    ctx = S.open_system(sysm)
    try:
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        ctx.cycle()
        st = ctx.stats()
        return free - torch.cuda.mem_get_info()[0], st["npairs"], st["ncalls"]
    finally:
        ctx.close()


def test_cycle_holds_one_copy_of_its_coefficients():
    small = W.alkane(1, seed=1, nrad=3)
    _held_by_a_cycle(small)  # the kernels' code is loaded
    sysm = W.alkane(9, seed=1, nrad=3)
    held, npairs, ncalls = _held_by_a_cycle(sysm)
    nfo, points = sysm.nfrm[0], sysm.nmsh
    assert sysm.nfrm == (37, 37)  # the spins one after the other, in the same scratch
    assert points > 128 * 75  # one part: a call list in parts is for smaller meshes
    pair_fo = npairs * nfo * (8 * 52 + 8 * 4 + 1)
    call_fo = ncalls * nfo * (64 + 8 * 52 + 4)
    # values, Coulomb and SIC potential and its product with the orbital of both spins, one more of one spin
    mesh = 8 * points * nfo * (2 * 4 + 1)
    # a tenth and 64 MB for the allocator's granules and the many small arrays
    assert held <= 1.1 * (pair_fo + call_fo + mesh) + (64 << 20), (held, pair_fo, call_fo, mesh)
    # a second copy of the coefficients would not pass
    assert 0.1 * (pair_fo + call_fo + mesh) + (64 << 20) < npairs * nfo * 8 * 48
