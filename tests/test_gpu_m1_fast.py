"""The production build's M1 closure solve (FP32 Newton, FP64 residual) and
closed-form face states against the oracle on Minkowski blocks: flux factors
from 0 to 0.99, warm and cold closure guesses, velocities from rest to 0.6
(beyond, with large flux factors, the residual has several roots and both
builds' Newton paths differ from the oracle's by rounding), zero flux, NaN
input.  Bars: both solves end with a residual step below
2.2e-10 whose error is that step times the slope's (1e-5 at most), so values
agree to rounding amplified by W^4 < 3 -- 1e-12 of the zone's |E| + |F|; the
fluxes are sums of a few such terms: 1e-12 of the face cells' magnitudes."""
import numpy as np
import pytest

from phoebus_gb300 import abi
from phoebus_gb300.fluid import FluidContext  # noqa: F401 (the context fixtures' type)
from phoebus_gb300.radiation import RadiationContext
from tests.util import assert_bitwise, face_region, host, random_rad_block

pytestmark = pytest.mark.gpu


def _block(vmax, hmax, seed, nx=(11, 9, 5)):
    hb = random_rad_block(nx, 3, seed, vmax=vmax, hmax=hmax)
    flat = np.arange(hb.N).reshape(hb.shape)
    for d in range(3):
        hb["rprim"][abi.RH + d][flat % 7 == 2] = 0.0
        hb["prim"][abi.PVEL + d][flat % 11 == 5] = 0.0
    return hb


@pytest.mark.parametrize("vmax,hmax", [(0.0, 0.5), (0.4, 0.99), (0.6, 0.6), (0.3, 1e-6)])
@pytest.mark.parametrize("warm", [False, True])
def test_con_to_prim(ctx_fast, vmax, hmax, warm):
    from oracle.oracle import RadOracle

    orc, rf = RadOracle(), RadiationContext(ctx_fast)
    p, rp = abi.default_params(mhd=0), abi.default_rad_params()
    hb = _block(vmax, hmax, 41)
    orc.MomentPrim2Con(rp, p, hb, *hb.entire())
    if warm:
        orc.MomentCon2Prim(rp, p, hb)
        hb["rprim"][abi.RXI] *= 1.0 + 0.01 * np.sin(np.arange(hb.N)).reshape(hb.shape)
    hb["rcons"][abi.RE, 4, 5, 6] = np.nan
    hb["rcons"][abi.RF + 1, 4, 5, 7] = np.nan
    db = hb.to_device()
    orc.MomentCon2Prim(rp, p, hb)
    rf.MomentCon2Prim(rp, p, db)
    ctx_fast.check()
    got, ref = host(db["rprim"]), hb["rprim"]
    assert_bitwise(got[abi.RFAIL], ref[abi.RFAIL], "c2pfail")
    assert np.array_equal(np.isnan(got), np.isnan(ref))
    ok = ~np.isnan(ref).any(axis=0)
    scale = np.abs(hb["rcons"][abi.RE]) + np.abs(hb["rcons"][abi.RF:abi.RF + 3]).sum(axis=0)
    assert np.all(np.abs(got[abi.RJ] - ref[abi.RJ])[ok] <= 1e-12 * scale[ok])
    for v in (abi.RH, abi.RH + 1, abi.RH + 2, abi.RXI):
        assert np.all(np.abs(got[v] - ref[v])[ok] * ref[abi.RJ][ok] <= 1e-12 * scale[ok]), v


@pytest.mark.parametrize("vmax,hmax", [(0.0, 0.5), (0.4, 0.99), (0.9, 0.9)])
@pytest.mark.parametrize("recon", ["linear", "constant"])
def test_fluxes(ctx_fast, vmax, hmax, recon):
    from oracle.oracle import RadOracle

    orc, rf = RadOracle(), RadiationContext(ctx_fast)
    p, rp = abi.default_params(mhd=0), abi.default_rad_params(recon=recon, kappa_s=3.0, kappa_a=0.5)
    hb = _block(vmax, hmax, 42)
    orc.MomentPrim2Con(rp, p, hb, *hb.entire())
    orc.MomentCalculateOpacities(rp, p, hb)
    db = hb.to_device()
    orc.CalculateFluxes(rp, p, hb)
    rf.CalculateFluxes(rp, p, db)
    ctx_fast.check()
    got, ref = host(db["rflux"]), hb["rflux"]
    W = 1.0 / np.sqrt(1.0 - vmax * vmax)
    # E, F and P of a face state from J and |H| <= J of the stencil's cells
    mag = 10.0 * W * W * np.max(hb["rprim"][abi.RJ]) * (1.0 + 1.0 / (0.5 * min(hb.dx)))
    for d in range(3):
        r = face_region(hb, d)
        for m in range(abi.RNCONS):
            n = d * abi.RNCONS + m
            assert np.abs(got[n][r] - ref[n][r]).max() <= 1e-12 * mag, (d, m)
