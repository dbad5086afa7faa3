"""Coefficient thresholds of the pair-route FO density, entry by entry.

POISSON1 drops a density polynomial entry (RHOC, and separately every derivative
entry RHOD = f RHOC, f = 1..12) by its own magnitude, at 1e-14
(poisson1.f:855-895).  Between 1e-14 / f and 1e-14 a monomial belongs to
derivative channels only.  With orbitals scaled so that the FO densities
themselves are near 1e-14 such entries carry a good part of every channel.
The orbitals' scale changes no other choice, and both sides keep the same entries
(their coefficients agree to rounding, and an entry that close to the threshold
does not occur), so the channels agree as they do unscaled: to 1e-12 of each
channel's maximum."""
import dataclasses

import numpy as np
import pytest

from oracle import oracle as O
from publicrelease_2020_b200 import sic as S
from publicrelease_2020_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("functional,nch", [("GGA-PBE*GGA-PBE", 10), ("MGGA-SCAN*MGGA-SCAN", 4),
                                            ("LDA-PW91*LDA-PW91", 1)])
@pytest.mark.parametrize("scale", [1e-5, 1e-6, 1e-7])
def test_entries_kept_by_their_own_magnitude(functional, nch, scale):
    base = W.small_synthetic(seed=5, natoms=3, nbasis=24, nmsh=2000, nfo=2, functional=functional)
    sysm = dataclasses.replace(base, psi=base.psi * scale)
    orc = O.Oracle(sysm)
    ctx = S.open_system(sysm)
    try:
        ctx.set_density_mode("pairs")
        for k in range(1, sysm.nfrm[0] + 1):
            _, got = ctx.coupot_sic(1, k)
            _, want, _ = orc.coupot_sic(1, k)
            for ch in range(nch):
                top = np.abs(want[ch]).max()
                assert top > 0.0
                assert np.abs(got[ch] - want[ch]).max() <= 1e-12 * top, (k, ch)
    finally:
        ctx.close()
