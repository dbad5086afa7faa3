"""The call set-up of few (call, FO) pairs, whose moments are formed point by point
without the product form before, on both sides of the rule (444 of them), and
evaluations of one FO or one density, which have no per-FO call.  Potentials
against the oracle with the tolerances of the parity tests."""
import numpy as np
import pytest

from oracle import oracle as O
from publicrelease_2020_b200 import sic as S
from publicrelease_2020_b200 import workloads as W

pytestmark = pytest.mark.gpu


# 48 calls of several slots: 96, 384 and 480 (call, FO)s of both spins
@pytest.mark.parametrize("nfo,calls_fos", [(1, 96), (4, 384), (5, 480)])
def test_potentials_of_a_cycle(nfo, calls_fos):
    sysm = W.small_synthetic(seed=5, natoms=3, nbasis=24, nmsh=2500, nfo=nfo, nspn=2, functional="LDA-PW91*LDA-PW91")
    orc = O.Oracle(sysm)
    ctx = S.open_system(sysm)
    try:
        ctx.cycle()
        assert ctx.stats()["ncalls"] * 2 * nfo == calls_fos
        for s in (1, 2):
            for k in range(1, nfo + 1):
                got, _ = ctx.coupot_sic(s, k)
                want, _, _ = orc.coupot_sic(s, k)
                assert np.abs(got - want).max() < 1e-9 * np.abs(want).max(), (s, k)
    finally:
        ctx.close()


# one FO of one spin; mixed: the columns and split products of the shared-geometry
# kernel are single precision, near 1e-6 of the largest potential
@pytest.mark.parametrize("precision,tol", [("fp64", 1e-9), ("mixed", 1e-5)])
def test_one_fo_and_one_density(precision, tol):
    sysm = W.small_synthetic(seed=5, natoms=3, nbasis=24, nmsh=2500, nfo=1, functional="LDA-PW91*LDA-PW91")
    orc = O.Oracle(sysm)
    ctx = S.open_system(sysm)
    try:
        ctx.set_precision(precision)
        got, _ = ctx.coupot_sic(1, 1)
        want, _, _ = orc.coupot_sic(1, 1)
        assert np.abs(got - want).max() < tol * np.abs(want).max()
        got, want = ctx.coupot1(), orc.coupot1()
        assert np.abs(got - want).max() < tol * np.abs(want).max()
    finally:
        ctx.close()
