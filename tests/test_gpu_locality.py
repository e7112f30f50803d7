"""What the production kernels leave alone: faces whose stencils do not hold a
NaN or infinite zone, in every direction, and the stage input where the first
stage keeps it."""
import numpy as np
import pytest

from phoebus_gb300 import abi
from phoebus_gb300.block import Block
from tests.test_gpu_flux_shapes import ragged_block
from tests.util import flux_view, host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("recon", ["weno5z", "mp5", "linear"])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_faces_in_every_direction(ctx_fast, recon, bad):
    """Cell c along direction d enters the states of faces c - 2 .. c + 3 at
    most; every other face keeps its bits (the X2 and X3 sweeps pass states
    through slots that change hands from cell to cell)."""
    p = abi.default_params(Gamma=4.0 / 3.0, recon=recon, riemann="hll")
    hb = ragged_block((40, 14, 12), 3, 7)
    clean = hb.to_device()
    ctx_fast.CalculateFluxes(p, clean)
    at = (9, 10, 20)  # k, j, i
    hb["prim"][(abi.PRHO,) + at] = bad
    db = hb.to_device()
    ctx_fast.CalculateFluxes(p, db)
    ctx_fast.check()
    for d in range(3):
        a, c = host(flux_view(db["flux"], d)), host(flux_view(clean["flux"], d))
        hit = list(at)
        hit[2 - d] = slice(at[2 - d] - 2, at[2 - d] + 4)
        assert not np.array_equal(a[(slice(None),) + tuple(hit)], c[(slice(None),) + tuple(hit)]), d
        a[(slice(None),) + tuple(hit)] = c[(slice(None),) + tuple(hit)] = 0.0
        assert np.array_equal(a, c), d


@pytest.mark.parametrize("beta", [1.0, 0.5])
def test_update_keeps_the_stage_input(ctx_fast, beta):
    """cons holds u0 = beta cons + (1 - beta) base after the update: unchanged for
    beta = 1 and a finite base, to the rounding of its two terms otherwise."""
    import torch

    hb = Block((17, 5, 7), 4, 3, (0.0, 0.0, 0.0), (0.1, 0.2, 0.3)).alloc()
    rng = np.random.default_rng(3)
    for name in ("flux", "cons", "src"):
        hb[name][:] = rng.normal(size=hb[name].shape) * 10.0 ** rng.uniform(-6, 6, hb[name].shape)
    base = rng.normal(size=hb["cons"].shape) * 10.0 ** rng.uniform(-6, 6, hb["cons"].shape)
    db = hb.to_device()
    out = torch.zeros_like(db["cons"])
    ctx_fast.UpdateStage(db, torch.from_numpy(base).cuda(), out, beta, 0.02)
    ctx_fast.check()
    inner = (slice(None),) + hb.isl()
    got, old, b = host(db["cons"])[inner], hb["cons"][inner], base[inner]
    lim = 0.0 if beta == 1.0 else 4.0 * 2.0 ** -53 * (np.abs(beta * old) + np.abs((1.0 - beta) * b))
    assert (np.abs(got - (beta * old + (1.0 - beta) * b)) <= lim).all()
