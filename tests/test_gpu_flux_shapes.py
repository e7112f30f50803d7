"""Production fluxes over ragged blocks against the oracle: pencil and segment
remainders of the launch rules (1D to 3D), and states that reach the integer
reconstruction's branches -- flat regions, differences around the weights'
1e-100 floor, steps, per-zone random values, zero and tiny fields.  Bar per
face: 1e-12 of the largest magnitude (face_flux_scale) within its stencils,
two faces to either side: second differences round relative to the largest
value in the stencil, and the states hold ranges of 1e14 within one."""
import numpy as np
import pytest

from phoebus_gb300 import abi, states
from phoebus_gb300.block import Block
from tests.util import _shift, face_flux_scale, face_region, flux_view, report_close

pytestmark = pytest.mark.gpu


def ragged_block(nx, ndim, seed, mhd=True):
    b = Block(nx, 4, ndim, (0.0, 0.0, 0.0), tuple(1.0 / n for n in nx)).alloc()
    n = nx[0] * nx[1] * nx[2]
    rho, wv, P, B = states.random_zones_prims(n, seed, W=(1.0, 3.0), sigma=(1e-3, 1.0))
    rho, P, B = rho.copy(), P.copy(), B.copy()
    wv = [w.copy() for w in wv]
    third = np.arange(n) % (3 * nx[0]) // nx[0]  # by pencil: random, stepped, nearly flat
    step, flat = third == 1, third == 2
    # steps from a constant to random values: symmetric stencils around a flat
    # centre would tie beta_0 and beta_2, and the reference's weights then follow
    # the last bit of that difference
    rho[step] = np.where(np.arange(n)[step] % 11 < 5, 1.0, 0.1 * rho[step])
    P[flat] = 1.0
    rho[flat] = 1.0 + 1e-15 * (np.arange(n)[flat] % 3)
    for d in range(3):
        wv[d][flat] = 1e-20 * (np.arange(n)[flat] % 5)
        B[d][flat] = np.array([0.0, 1e-41, 1e-50, 1e-55, 3e-52])[np.arange(n)[flat] % 5]
        B[d][step] = 0.0
    shp = (nx[2], nx[1], nx[0])
    states._set_interior(b, rho.reshape(shp), [w.reshape(shp) for w in wv], P.reshape(shp),
                         [x.reshape(shp) for x in B], 1.0 / 3.0)
    return b


@pytest.mark.parametrize("recon,solver", [("weno5z", "hll"), ("mp5", "hll"), ("linear", "llf"), ("constant", "llf")])
@pytest.mark.parametrize("nx,ndim", [((4, 4, 4), 3), ((33, 5, 4), 3), ((70, 9, 6), 3), ((131, 5, 7), 3),
                                     ((10, 67, 5), 3), ((37, 23, 1), 2), ((300, 1, 1), 1)])
def test_ragged_blocks(oracle, ctx_fast, recon, solver, nx, ndim):
    p = abi.default_params(Gamma=4.0 / 3.0, recon=recon, riemann=solver, c2p_tol=1e-10, c2p_max_iter=100)
    hb = ragged_block(nx, ndim, 500 + nx[0])
    oracle.PrimitiveToConserved(p, hb)
    db = hb.to_device()
    oracle.CalculateFluxes(p, hb)
    ctx_fast.CalculateFluxes(p, db)
    ctx_fast.check()
    for d in range(ndim):
        sl = (slice(None),) + face_region(hb, d)
        near = face_flux_scale(hb, d)
        scale = np.max([_shift(near, d, k) for k in (-2, -1, 0, 1, 2)], axis=0)
        report_close(flux_view(db["flux"], d)[sl], flux_view(hb["flux"], d)[sl], scale[sl], 1e-12, f"flux d={d}")


@pytest.mark.parametrize("recon", ["weno5z", "mp5", "linear"])
def test_nan_and_infinity_stay_local(ctx_fast, recon):
    """A NaN or an infinity in one zone reaches no face whose stencils do not
    hold it, and leaves the others as they are without it."""
    p = abi.default_params(Gamma=4.0 / 3.0, recon=recon, riemann="hll")
    hb = ragged_block((40, 6, 6), 3, 7)
    clean = hb.to_device()
    ctx_fast.CalculateFluxes(p, clean)
    for bad in (np.nan, np.inf):
        hb["prim"][abi.PRHO, 7, 7, 20] = bad
        db = hb.to_device()
        ctx_fast.CalculateFluxes(p, db)
        ctx_fast.check()
        a, c = flux_view(db["flux"], 0).cpu().numpy(), flux_view(clean["flux"], 0).cpu().numpy()
        a[:, 7, 7, 18:24] = c[:, 7, 7, 18:24] = 0.0  # faces whose stencils hold cell 20
        assert np.array_equal(a, c)
