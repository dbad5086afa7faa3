"""Per-FO-geometry Coulomb calls (k_perfo_near, k_perfo_far) at the edges of
their tiles: 8 points per warp, 64 per CTA, 128 per mesh tile; 8 FO slots per
m-tile, 32 or 64 FOs per block, 4 per far group.  NSPN=2, so every call has
per-FO spheres.  The Coulomb potentials are held to the oracle's at the
tolerance of the parity tests (1e-9 of the largest value, FP64) and the mixed
path to its gate (1e-5), with near/far work counts equal to the oracle's."""
import numpy as np
import pytest

from oracle import oracle as O
from publicrelease_2020_b200 import sic as S
from publicrelease_2020_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _system(nfo, npts):
    if nfo < 10:
        sysm = W.synthetic(natoms=max(2, nfo // 3), nbasis=max(16, 4 * nfo + 8), nmsh=4000, nfo=nfo,
                           box_ang=4.0 + 0.4 * max(2, nfo // 3), seed=11, functional="LDA-PW91*LDA-PW91", nspn=2)
    else:  # nonane has 37 FOs per spin
        sysm = W.alkane(9, seed=3, nrad=4)
        n0 = sysm.nwfs[0]
        sysm.psi = np.ascontiguousarray(np.concatenate([sysm.psi[:nfo], sysm.psi[n0:n0 + nfo]]))
        sysm.nwfs = (nfo, nfo)
        sysm.fods = [f[:nfo] for f in sysm.fods]
    n = sysm.nmsh
    idx = np.sort(np.random.default_rng(2).choice(n, npts, replace=False))
    sysm.rmsh = np.ascontiguousarray(sysm.rmsh[idx])
    sysm.wmsh = np.ascontiguousarray(sysm.wmsh[idx] * (n / npts))
    return sysm


@pytest.mark.parametrize("nfo,npts", [(1, 9), (4, 64), (8, 65), (9, 129), (31, 40), (32, 72), (33, 200), (37, 65)])
def test_coulomb_potentials_match_oracle(nfo, npts):
    sysm = _system(nfo, npts)
    orc = O.Oracle(sysm)
    ref = orc.sic_cycle(nthreads=8)
    ctx = S.open_system(sysm)
    try:
        for mode, tol in (("fp64", 1e-9), ("mixed", 1e-5)):
            ctx.set_precision(mode)
            got = ctx.cycle()
            for s in range(2):
                lam = ref["sic"][s][:nfo, :nfo]
                assert np.max(np.abs(got["sic"][s][:nfo, :nfo] - lam)) < tol * np.abs(lam).max(), (mode, s)
                vh = ref["results"][s][:nfo, 5]
                assert np.max(np.abs(got["results"][s][:nfo, 5] - vh)) < tol * np.abs(vh).max(), (mode, s)
            again = ctx.cycle()
            assert all(np.array_equal(again[k], got[k]) for k in ("results", "sic", "debdax", "cfrm")), mode
    finally:
        ctx.close()
