"""The production build's con2prim root (FP32 search, FP64 correction) against
the oracle's bracketed iteration on the same conserved zones, where its
acceptance rules can go wrong: launch remainders, tolerances and iteration
caps at the ends of the fast rule, floors and ceilings switching at the root,
cold gas at rest (the root at 1), unmagnetised and strongly magnetised zones,
warm guesses, NaN input."""
import numpy as np
import pytest

from phoebus_gb300 import abi, states
from tests.util import assert_bitwise, host

pytestmark = pytest.mark.gpu


def dev(a):
    import torch

    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def zone_prims(n, seed, W=(1.0, 8.0), sigma=(1e-3, 100.0), logT=(-5.0, 1.0)):
    rho, wv, P, B = states.random_zones_prims(n, seed, W=W, sigma=sigma, logT=logT)
    rho, wv, P, B = rho.copy(), [w.copy() for w in wv], P.copy(), B.copy()
    rest = np.arange(n) % 7 == 3  # cold gas at rest: the root sits at 1
    for w in wv:
        w[rest] = 0.0
    P[rest] = 1e-14 * rho[rest]
    B[:, np.arange(n) % 5 == 1] = 0.0
    gm1 = 1.0 / 3.0
    prim = np.zeros((abi.NPRIM, n))
    prim[abi.PRHO], prim[abi.PENG], prim[abi.PPRS] = rho, P / gm1, P
    prim[abi.PVEL:abi.PVEL + 3], prim[abi.PB:abi.PB + 3] = wv, B
    prim[abi.PGM1], prim[abi.PTMP] = gm1 + 1.0, P / gm1 / rho
    return prim


def run(ctx, oracle, p, cons, prim0):
    import torch

    n = cons.shape[1]
    c, pr, fail = dev(cons), dev(prim0), torch.zeros(n, dtype=torch.float64, device="cuda")
    ctx.ConservedToPrimitiveZones(p, c, pr, fail=fail)
    ctx.check()
    rc, rpr, rfail = cons.copy(), prim0.copy(), np.zeros(n)
    assert oracle.ConservedToPrimitiveZones(p, rc, rpr, fail=rfail) == 0
    assert_bitwise(fail, rfail, "fail")
    return host(pr), rpr, host(c), rc


@pytest.mark.parametrize("n", [1, 31, 129, 5000])
@pytest.mark.parametrize("tol,max_iter", [(1e-3, 100), (1e-8, 20), (1e-12, 100), (2e-3, 100)])
def test_root_within_tolerance(ctx_fast, oracle, n, tol, max_iter):
    """Both ends within the tolerance of the same root: |mu - mu_ref| <= 2 tol
    (plus the residual's own rounding, 1e-13 at these magnetisations); a
    tolerance of 2e-3 lies outside the fast rule."""
    p = abi.default_params(gm1=1.0 / 3.0, c2p_tol=tol, c2p_max_iter=max_iter)
    prim = zone_prims(n, 900 + n)
    cons = oracle.PrimitiveToConservedZones(p, prim)
    got, ref, _, _ = run(ctx_fast, oracle, p, cons, prim * 0.0)
    assert np.abs(got[abi.PMU] - ref[abi.PMU]).max() <= 2.0 * tol + 1e-13


@pytest.mark.parametrize("mhd", [0, 1])
@pytest.mark.parametrize("floor_type", ["ConstantRhoSie", "ExpX1RhoU"])
def test_floors_and_ceilings(ctx_fast, oracle, mhd, floor_type):
    """Floors and ceilings active at the root of many zones: mu within 2 tol,
    and the conserved variables rewritten for the same zones."""
    n, tol = 4000, 1e-10
    p = abi.default_params(gm1=1.0 / 3.0, c2p_tol=tol, c2p_max_iter=100, mhd=mhd)
    prim = zone_prims(n, 77)
    if not mhd:
        prim[abi.PB:abi.PB + 3] = 0.0
    cons = oracle.PrimitiveToConservedZones(p, prim)
    cons[abi.CENG] *= np.where(np.arange(n) % 3 == 0, 0.97, 1.0)  # energies below the solution's
    p.enable_floors, p.enable_ceilings = 1, 1
    p.floor_type = abi.FLOOR[floor_type]
    p.rho0_floor, p.sie0_floor, p.gam0_ceiling, p.sie0_ceiling = 1e-3, 1e-3, 4.0, 5.0
    got, ref, c, rc = run(ctx_fast, oracle, p, cons, prim * 0.0)
    assert np.abs(got[abi.PMU] - ref[abi.PMU]).max() <= 2.0 * tol + 1e-13
    assert_bitwise(np.any(c != cons, axis=0).astype(float), np.any(rc != cons, axis=0).astype(float), "rewritten")


def test_warm_guess_and_nan(ctx_fast, oracle):
    """A stored mu anywhere in (0, 1] gives the same root; NaN zones fail and
    keep their primitives."""
    n, tol = 4000, 1e-10
    p = abi.default_params(gm1=1.0 / 3.0, c2p_tol=tol, c2p_max_iter=100)
    prim = zone_prims(n, 78)
    cons = oracle.PrimitiveToConservedZones(p, prim)
    cons[abi.CRHO, 5], cons[abi.CENG, 6], cons[abi.CMOM, 7] = np.nan, np.nan, np.nan
    prim0 = prim * 0.0
    prim0[abi.PMU] = states.uniform(3, 1, n) ** 2 + 1e-9
    prim0[abi.PMU, ::50] = 1.0
    got, ref, _, _ = run(ctx_fast, oracle, p, cons, prim0)
    ok = np.ones(n, bool)
    ok[5:8] = False
    assert np.abs(got[abi.PMU, ok] - ref[abi.PMU, ok]).max() <= 2.0 * tol + 1e-13
    assert_bitwise(got[:, ~ok], prim0[:, ~ok], "NaN zones")
