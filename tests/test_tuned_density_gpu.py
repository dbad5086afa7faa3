"""Per-orbital entries after flosic_sic_autotune in the pair-route density.

The pair-route FO density of a spin is formed from the primitive projections and
the per-FO spheres of that spin's own Coulomb evaluation.  Tuning runs, COUPOT1
and the other spin's evaluation fill the same scratch, so a per-orbital entry
that follows them must evaluate its spin again.  Each sequence is compared with a
context that was never tuned: the same operations in the same order, so every
result is equal bit for bit."""
import dataclasses

import numpy as np
import pytest

from publicrelease_2020_b200 import sic as S
from publicrelease_2020_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _apart():
    """C9H20 with 36 + 37 FOs: more than 64 in all, so a cycle evaluates the spins
    apart and the tuner takes the second, which has more."""
    s = W.alkane(9, seed=1, nrad=3)
    n = s.nwfs[0]
    return dataclasses.replace(s, psi=np.delete(s.psi, n - 1, axis=0), nwfs=(n - 1, n),
                               fods=[s.fods[0][:n - 1], s.fods[1]])


SYSTEMS = {
    "one_spin": lambda: W.small_synthetic(seed=5, natoms=3, nbasis=24, nmsh=5000, nfo=4),
    "together": lambda: W.water(seed=0, nrad=12, functional="GGA-PBE*GGA-PBE"),
    "apart": _apart,
}


def _orbitals(sysm):
    """(spin, FO) of a few FOs, the last spin last."""
    return [(s, k) for s in range(1, sysm.nspn + 1) for k in (1, sysm.nfrm[s - 1])]


@pytest.mark.parametrize("name", list(SYSTEMS))
@pytest.mark.parametrize("between", ["nothing", "coupot1"])
def test_pair_density_after_autotune(name, between):
    sysm = SYSTEMS[name]()
    want, got = [], []
    for tuned, out in ((False, want), (True, got)):
        ctx = S.open_system(sysm)
        try:
            ctx.set_density_mode("pairs")
            if tuned:
                ctx.autotune(reps=1)
                if between == "coupot1":
                    ctx.coupot1()
            for s, k in _orbitals(sysm):
                coul, rhog = ctx.coupot_sic(s, k)
                a = ctx.apotnl_sic(s, k)
                out.append((coul, rhog, a["results"], a["pot"]))
        finally:
            ctx.close()
    for sk, w, g in zip(_orbitals(sysm), want, got):
        for what, x, y in zip(("coulomb", "rhog", "results", "pot"), w, g):
            assert np.array_equal(x, y), (name, sk, what)
