"""The production build's con2prim root at the ends of the parameter range:
fast and cold zones, whose residual changes slope at the root, and bounds that
switch beside it."""
import numpy as np
import pytest

from phoebus_gb300 import abi
from tests.util import host

pytestmark = pytest.mark.gpu


def dev(a):
    import torch

    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def zone_prims(n, seed, gm1, Wmax, logsie=(-6.0, 1.0)):
    """Log-uniform Lorentz factor in [1, Wmax] and u / rho, half the zones
    magnetised with B^2 / rho log-uniform in [1e-4, 1e2]."""
    rng = np.random.default_rng(seed)

    def iso():
        c, ph = rng.uniform(-1, 1, n), rng.uniform(0, 2 * np.pi, n)
        s = np.sqrt(1 - c * c)
        return np.stack([s * np.cos(ph), s * np.sin(ph), c])

    rho, sie = 10.0 ** rng.uniform(-6, 0, n), 10.0 ** rng.uniform(*logsie, n)
    W = Wmax ** rng.uniform(0, 1, n)
    prim = np.zeros((abi.NPRIM, n))
    prim[abi.PRHO], prim[abi.PENG], prim[abi.PPRS] = rho, rho * sie, gm1 * rho * sie
    prim[abi.PVEL:abi.PVEL + 3] = np.sqrt(W * W - 1.0) * iso()
    prim[abi.PB:abi.PB + 3] = np.sqrt(10.0 ** rng.uniform(-4, 2, n) * rho) * iso() * (np.arange(n) % 2)
    prim[abi.PGM1], prim[abi.PTMP] = gm1 + 1.0, sie
    return prim


def solve(ctx, p, cons, prim0, learned=False):
    """Primitives, fail flags and statistics of one call; an unbracketed root
    raises."""
    import torch

    c, pr = dev(cons), dev(prim0)
    fail = torch.zeros(cons.shape[1], dtype=torch.float64, device="cuda")
    ctx.c2p_stats(reset=True)
    ctx.ConservedToPrimitiveZones(p, c, pr, fail=fail, learned=learned)
    ctx.check()
    return host(pr), host(fail), host(c), ctx.c2p_stats(reset=True)


def reference(oracle, p, cons, prim0):
    c, pr, fail = cons.copy(), prim0.copy(), np.zeros(cons.shape[1])
    assert oracle.ConservedToPrimitiveZones(p, c, pr, fail=fail) == 0
    return pr, fail, c


@pytest.mark.parametrize("gm1,tol,Wmax", [(2 / 3, 1e-9, 50.0), (2 / 3, 1e-10, 50.0), (1 / 3, 1e-10, 100.0),
                                          (2 / 3, 1e-11, 100.0)])
def test_fast_cold_zones_within_tolerance(ctx_fast, oracle, gm1, tol, Wmax):
    """|mu - mu*| <= tol for every zone, mu* from the bracketed iteration at
    tolerance 1e-15: its half width, and the residual's rounding of 1 - v^2
    (2.2e-16 W^2 of 1 / W in mu = 1 / (h W): at most 2e-14 here) stay below
    1e-13.  Half the zones are cold, half start 1% off the root."""
    n = 400_000
    p = abi.default_params(gm1=gm1, c2p_tol=tol, c2p_max_iter=100)
    prim = zone_prims(n, int(1e3 * gm1 + Wmax), gm1, Wmax)
    cons = oracle.PrimitiveToConservedZones(p, prim)
    mu, _, _ = reference(oracle, abi.default_params(gm1=gm1, c2p_tol=1e-15, c2p_max_iter=200), cons, prim * 0.0)
    mu = mu[abi.PMU]
    prim0 = prim * 0.0
    prim0[abi.PMU, ::2] = np.minimum(mu[::2] * (1.0 + 0.01 * np.sin(np.arange(n)[::2])), 1.0)
    got, _, _, stats = solve(ctx_fast, p, cons, prim0)
    over = np.abs(got[abi.PMU] - mu) > tol + 1e-13
    assert not over.any(), (int(over.sum()), np.abs(got[abi.PMU] - mu).max() / tol)
    assert stats["residual_evals"] < 2 * n  # the fast root is the one taken


@pytest.mark.parametrize("tol", [1e-8, 1e-9, 1e-10])
@pytest.mark.parametrize("bound", ["floor", "ceiling"])
def test_bound_switching_beside_the_root(ctx_fast, oracle, tol, bound):
    """Zones whose velocity is bounded (W = 5) and whose energy floor or ceiling
    switches within 1e-9 to 1e-2 of the root, where the residual's slope changes
    by several times.  From the root backwards, unmagnetised: with vt = mu r the
    unbounded speed, mu = (1 - vt^2) / nu, nu = (1 + a)(1 + e) / W,
    q = (1 + e) / W - 1 + vt r.  Bar as above."""
    n, gm1, W = 200_000, 2.0 / 3.0, 5.0
    rng = np.random.default_rng(41)
    p = abi.default_params(gm1=gm1, c2p_tol=tol, c2p_max_iter=100)
    p.enable_floors, p.rho0_floor, p.sie0_floor = 1, 1e-6, 1e-3
    p.enable_ceilings, p.gam0_ceiling, p.sie0_ceiling = 1, W, 2.0
    e = (1e-3 if bound == "floor" else 2.0) * (1.0 + 10.0 ** rng.uniform(-9, -2, n) * rng.choice([-1.0, 1.0], n))
    vt = rng.uniform(np.sqrt(0.961), 0.999, n)
    a = gm1 * e / (1.0 + e)
    mu = (1.0 - vt * vt) / ((1.0 + a) * (1.0 + e) / W)
    r = vt / mu
    cons = np.zeros((abi.NCONS, n))
    cons[abi.CRHO] = 10.0 ** rng.uniform(-3, 0, n)
    cons[abi.CMOM] = r * cons[abi.CRHO]
    cons[abi.CENG] = ((1.0 + e) / W - 1.0 + vt * r) * cons[abi.CRHO]
    prim0 = np.zeros((abi.NPRIM, n))
    pref = p.__class__.from_buffer_copy(p)
    pref.c2p_tol, pref.c2p_max_iter = 1e-15, 200
    ref, _, _ = reference(oracle, pref, cons, prim0)
    prim0[abi.PMU, ::2] = np.minimum(ref[abi.PMU, ::2] * (1.0 + 0.01 * np.sin(np.arange(n)[::2])), 1.0)
    got, _, _, _ = solve(ctx_fast, p, cons, prim0)
    over = np.abs(got[abi.PMU] - ref[abi.PMU]) > tol + 1e-13
    assert not over.any(), (int(over.sum()), np.abs(got[abi.PMU] - ref[abi.PMU]).max() / tol)


@pytest.mark.parametrize("floor", [0.0, 1e-18, 1e-8])
@pytest.mark.parametrize("sign_tau", [1.0, -1.0])
def test_negative_density(ctx_fast, oracle, floor, sign_tau):
    """D < 0 (an update that overshot): the density is the floor, and where
    that is below the reference's bound on h rho the residual no longer is the
    one of the ideal gas.  Same root and same fail flags as the reference; hydro
    (sqrt(D) divides the field)."""
    n, tol = 4000, 1e-10
    p = abi.default_params(gm1=1 / 3, c2p_tol=tol, c2p_max_iter=100, mhd=0)
    prim = zone_prims(n, 31, 1 / 3, 20.0)
    prim[abi.PB:abi.PB + 3] = 0.0
    cons = oracle.PrimitiveToConservedZones(p, prim)
    cons[abi.CRHO] *= -1.0
    cons[abi.CENG] *= sign_tau
    p.enable_floors, p.rho0_floor, p.sie0_floor = int(floor > 0), floor, floor
    ref, rfail, _ = reference(oracle, p, cons, prim * 0.0)
    got, fail, _, _ = solve(ctx_fast, p, cons, prim * 0.0)
    assert np.array_equal(fail, rfail)
    assert np.array_equal(np.isnan(got[abi.PMU]), np.isnan(ref[abi.PMU]))
    assert np.nanmax(np.abs(got[abi.PMU] - ref[abi.PMU])) <= 2.0 * tol + 1e-13


@pytest.mark.parametrize("tol,max_iter", [(2e-3, 100), (1e-16, 100), (1e-10, 4)])
@pytest.mark.parametrize("n", [129, 5000])
def test_learned_start_outside_the_fast_rule(ctx_fast, oracle, tol, max_iter, n):
    """Tolerances and iteration caps outside the fast rule keep the reference's
    iteration, the learned start included: a network whose output is constant
    (mu = e^-1, bracket e^-4 to 1) brackets every root in between."""
    p = abi.default_params(gm1=1 / 3, c2p_tol=tol, c2p_max_iter=max_iter)
    prim = zone_prims(n, 33, 1 / 3, 8.0, (-5.0, 0.0))
    cons = oracle.PrimitiveToConservedZones(p, prim)
    theta = np.zeros(abi.MLP_NPARAM, dtype=np.float32)
    theta[-2:] = [-1.0, 0.0]
    ctx_fast.mlp_set_weights(theta)
    mu, _, _ = reference(oracle, abi.default_params(gm1=1 / 3, c2p_tol=1e-15, c2p_max_iter=200), cons, prim * 0.0)
    mu = mu[abi.PMU]
    inside = (mu > 1.02 * np.exp(-4.0)) & (mu < 0.98)  # the network's output has BF16 weights
    got, _, _, stats = solve(ctx_fast, p, cons, prim * 0.0, learned=True)
    assert inside.sum() > 0.9 * n and inside.sum() <= stats["learned_accepted"] <= n
    assert stats["residual_evals"] >= 3 * n  # no zone by the fast root
    if max_iter == 100:
        assert np.abs(got[abi.PMU] - mu).max() <= tol + 1e-13


@pytest.mark.parametrize("gm1,rho0,sie0", [(1 / 3, 1e-3, 1e-3), (2 / 3, 1e-5, 1e-1), (1 / 3, 1e-6, 1e-6)])
def test_density_dependent_energy_floor(ctx_fast, oracle, gm1, rho0, sie0):
    """ExpX1RhoU's specific energy floor falls with the zone's density; where it
    holds at the root the fast root still finds it: within the tolerance, the
    same zones rewritten, one to three FP64 evaluations per zone."""
    n, tol = 20_000, 1e-10
    p = abi.default_params(gm1=gm1, c2p_tol=tol, c2p_max_iter=100)
    prim = zone_prims(n, 35, gm1, 20.0)
    cons = oracle.PrimitiveToConservedZones(p, prim)
    cons[abi.CENG] *= np.where(np.arange(n) % 3 == 0, 0.97, 1.0)
    p.enable_floors, p.floor_type, p.rho0_floor, p.sie0_floor = 1, abi.FLOOR["ExpX1RhoU"], rho0, sie0
    ref, rfail, rc = reference(oracle, p, cons, prim * 0.0)
    got, fail, c, stats = solve(ctx_fast, p, cons, prim * 0.0)
    assert np.array_equal(fail, rfail)
    assert np.abs(got[abi.PMU] - ref[abi.PMU]).max() <= 2.0 * tol + 1e-13
    assert np.array_equal(np.any(c != cons, axis=0), np.any(rc != cons, axis=0))
    assert n <= stats["residual_evals"] < 3 * n
