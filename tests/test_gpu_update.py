"""Production stage update, cons_out = u0 + beta dt (sources - div F) with
u0 = beta cons + (1 - beta) base, over ragged blocks in 1D to 3D: the first
stage (beta = 1, where u0 is cons unless base is not finite) and a later one.
Bar: each of a zone's at most 14 terms and the sums over them round a few
times, 16 units of 2^-53 of the sum of their magnitudes."""
import numpy as np
import pytest

from phoebus_gb300.block import Block
from tests.util import flux_view, host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("beta", [1.0, 0.5])
@pytest.mark.parametrize("nx,ndim", [((5, 1, 1), 1), ((33, 6, 1), 2), ((17, 5, 7), 3)])
def test_update(ctx_fast, nx, ndim, beta):
    import torch

    dx = (0.37, 1.9, 0.011)
    hb = Block(nx, 4, ndim, (0.0, 0.0, 0.0), dx).alloc()
    rng = np.random.default_rng(nx[0])
    for name in ("flux", "cons", "src"):
        hb[name][:] = rng.normal(size=hb[name].shape) * 10.0 ** rng.uniform(-3, 3, hb[name].shape)
    base = rng.normal(size=hb["cons"].shape)
    odd = rng.random(base.shape) < 0.1
    base[odd] = rng.choice([np.nan, np.inf, -np.inf], int(odd.sum()))
    db = hb.to_device()
    out = torch.zeros_like(db["cons"])
    dt = 0.02
    ctx_fast.UpdateStage(db, torch.from_numpy(base).cuda(), out, beta, dt)
    ctx_fast.check()
    inner = (slice(None),) + hb.isl()
    with np.errstate(invalid="ignore"):
        u0 = beta * hb["cons"] + (1.0 - beta) * base
    r, mag = np.zeros_like(base), np.zeros_like(base)
    for d in range(ndim):
        f = flux_view(hb["flux"], d)
        up = np.roll(f, -1, axis=3 - d)
        r -= (up - f) / dx[d]
        mag += (np.abs(up) + np.abs(f)) / dx[d]
    r[1:5] += hb["src"]
    mag[1:5] += np.abs(hb["src"])
    ref = (u0 + beta * dt * r)[inner]
    got = host(out)[inner]
    fin = np.isfinite(ref)
    assert np.array_equal(np.isnan(got), np.isnan(ref)) and np.array_equal(got[np.isinf(ref)], ref[np.isinf(ref)])
    with np.errstate(invalid="ignore"):
        lim = 16.0 * 2.0 ** -53 * (np.abs(beta * hb["cons"]) + np.abs((1.0 - beta) * base) + beta * dt * mag)[inner]
    assert (np.abs(got - ref)[fin] <= lim[fin]).all()
    # the stage leaves u0 in cons
    c = host(db["cons"])[inner]
    assert np.array_equal(np.isnan(c), np.isnan(u0[inner]))
    assert np.abs(c - u0[inner])[fin].max() <= 2.0 ** -50 * np.abs(u0[inner])[fin].max()
