"""The batched con2prim kernels' own instantiations against the single-block
ones (production build): the density-dependent energy floor, and settings outside
the fast root's rule with the learned start.  Same formulas on the same zones:
1e-12 of each variable's largest value, as for the other batched stages; the
learned brackets accepted are equal in number."""
import numpy as np
import pytest

from phoebus_gb300 import abi, states
from tests.test_gpu_batched import copy_blocks
from tests.util import assert_close, host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case", ["ExpX1RhoU", "ExpX1RhoU learned", "outside learned"])
def test_batched_equals_single(ctx_fast, case):
    import torch

    p = abi.default_params(Gamma=4.0 / 3.0, recon="linear", riemann="hll", c2p_tol=1e-10, c2p_max_iter=100)
    if case.startswith("ExpX1RhoU"):
        p.enable_floors, p.floor_type, p.rho0_floor, p.sie0_floor = 1, abi.FLOOR["ExpX1RhoU"], 1e-3, 1e-2
    else:
        p.c2p_tol = 2e-3
    learned = case.endswith("learned")
    if learned:  # a constant network: mu = e^-1, bracket [e^-4, 1]
        theta = np.zeros(abi.MLP_NPARAM, dtype=np.float32)
        theta[-2:] = [-1.0, 0.0]
        ctx_fast.mlp_set_weights(theta)
    a = []
    for n in (8, 12, 9):
        a.append(states.random_block(n, 70 + n).to_device("cuda"))
        ctx_fast.Initialize(p, a[-1])
    ctx_fast.check()
    for x in a:
        if learned:  # cold zones
            x["prim"][abi.PMU] = 0.0
    b = copy_blocks(a)
    out = [[torch.zeros_like(x["cons"]) for x in s] for s in (a, b)]
    dt = 0.1 * min(ctx_fast.EstimateTimestepBlock(p, x, False).item() for x in a)
    stats = []
    for run in range(2):
        ctx_fast.c2p_stats(reset=True)
        if run == 0:
            for x, o in zip(a, out[0]):
                ctx_fast.Stage(p, x, x["cons"].clone(), o, 1.0, dt, learned)
        else:
            ctx_fast.StageBatched(p, b, [x["cons"].clone() for x in b], out[1], 1.0, dt, learned)
        ctx_fast.check()
        stats.append(ctx_fast.c2p_stats(reset=True))
    for x, y, o, q in zip(a, b, out[0], out[1]):
        for name, g, r in (("cons", host(q), host(o)), ("prim", host(y["prim"]), host(x["prim"]))):
            assert np.array_equal(np.isnan(g), np.isnan(r)), name  # zones whose inversion failed
            for v in range(g.shape[0]):
                ok = ~np.isnan(r[v])
                assert_close(g[v][ok], r[v][ok], 1e-12, f"{name}[{v}]")
    for k in ("zones", "residual_evals", "learned_accepted", "failures"):
        assert stats[0][k] == stats[1][k], k
    assert (stats[0]["learned_accepted"] > 0) == learned
