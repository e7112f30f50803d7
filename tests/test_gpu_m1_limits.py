"""Radiation moments at the ends of the production formulations' ranges:
zones exactly in equilibrium with the gas (the source's root is the guess) and
moments whose squares are near the ends of the exponent range."""
import numpy as np
import pytest

from phoebus_gb300 import abi
from phoebus_gb300.radiation import RadiationContext
from tests.util import face_region, host, random_rad_block

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("max_iter", [2, 3, 100])
def test_source_at_equilibrium(ctx_fast, max_iter):
    """Without absorption the source's residual is rho Cv T - u, exactly 0 at
    the fluid's temperature and often at a neighbouring double (Cv T rounds
    coarser than T: T just below 2, Cv T just above 1).  The iteration then
    ends on its exact root, and the iteration cap decides the same zones as in
    the reference.  J = 2 - u makes the residual's divisor 2, so both builds
    evaluate the same numbers; a zone counts as solved where scattering moved
    its flux."""
    from oracle.oracle import RadOracle

    orc, rf = RadOracle(), RadiationContext(ctx_fast)
    p = abi.default_params(mhd=0, Cv=0.51)
    rp = abi.default_rad_params(kappa_s=0.7, src_rootfind_maxiter=max_iter)
    hb = random_rad_block((21, 17, 13), 3, 5, vmax=0.0, hmax=0.5)
    rng = np.random.default_rng(17)
    P, R = hb["prim"], hb["rprim"]
    P[abi.PRHO], P[abi.PTMP] = 1.0, rng.uniform(1.97, 1.99, hb.shape)
    P[abi.PENG] = 1.0 * (p.Cv * P[abi.PTMP])
    R[abi.RJ] = 2.0 - P[abi.PENG]
    orc.MomentPrim2Con(rp, p, hb, *hb.entire())
    db = hb.to_device()
    before = hb["rcons"].copy()
    orc.MomentFluidSource(rp, p, hb, 0.5)
    rf.MomentFluidSource(rp, p, db, 0.5)
    ctx_fast.check()
    inner = (slice(None),) + hb.isl()
    got, ref, old = host(db["rcons"])[inner], hb["rcons"][inner], before[inner]
    solved = np.any(ref[abi.RF:abi.RF + 3] != old[abi.RF:abi.RF + 3], axis=0)
    assert np.array_equal(np.any(got[abi.RF:abi.RF + 3] != old[abi.RF:abi.RF + 3], axis=0), solved)
    assert np.abs(got - ref).max() <= 1e-12 * np.abs(ref).max()


@pytest.mark.parametrize("exp10", [-153, -152, -140, 152])
def test_extreme_radiation(ctx_fast, exp10):
    """Moments so small or large that H^2 leaves the range of the production
    reciprocal square root (below 7e-304, normal down to 2e-308; above 1e303)
    keep their flux factor.
    E and F are sums of a few terms of size W^2 J: 1e-12 of J W^2.  With
    scattering: without it the asymptotic flux is 1e20 J / dx, whose square
    overflows in the reference."""
    from oracle.oracle import RadOracle

    orc, rf = RadOracle(), RadiationContext(ctx_fast)
    p, rp = abi.default_params(mhd=0), abi.default_rad_params(kappa_s=3.0)
    hb = random_rad_block((11, 9, 5), 3, 7, vmax=0.6, hmax=0.95)
    hb["rprim"][abi.RJ] = 10.0 ** exp10 * (1.0 + hb["rprim"][abi.RJ])
    size = 10.0 ** exp10
    db = hb.to_device()
    orc.MomentPrim2Con(rp, p, hb, *hb.entire())
    rf.MomentPrim2Con(rp, p, db, *db.entire())
    ctx_fast.check()
    assert np.abs(host(db["rcons"]) - hb["rcons"]).max() <= 1e-12 * size * 3.2
    orc.MomentCalculateOpacities(rp, p, hb)
    db = hb.to_device()
    orc.CalculateFluxes(rp, p, hb)
    rf.CalculateFluxes(rp, p, db)
    ctx_fast.check()
    for d in range(3):
        r = face_region(hb, d)
        for m in range(abi.RNCONS):
            n = d * abi.RNCONS + m
            assert np.abs(host(db["rflux"])[n][r] - hb["rflux"][n][r]).max() <= 1e-12 * size * 32, (d, m)
