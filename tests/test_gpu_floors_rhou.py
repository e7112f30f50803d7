"""ApplyFloors with ExpX1RhoU, whose specific energy floor is s / max(rho, r): the
reference passes an uninitialised density there (fixup.cpp:285-687), taken as 0 as
in its other calls, so the energy floor is that of a zone at the density floor."""
import pytest

from phoebus_gb300 import abi, states
from tests.util import assert_bitwise

pytestmark = pytest.mark.gpu


def test_apply_floors(oracle, ctx_exact):
    p = abi.default_params(Gamma=4.0 / 3.0, c2p_tol=1e-10, c2p_max_iter=100, enable_floors=1, enable_ceilings=1,
                           floor_type="ExpX1RhoU", rho0_floor=5e-3, sie0_floor=1e-3, gam0_ceiling=3.0, sie0_ceiling=0.5)
    hb = states.random_block(10, 63)
    hb.xmin = (-1.0, -1.0, -1.0)
    oracle.PrimitiveToConserved(p, hb)
    oracle.ConservedToPrimitive(p, hb)
    before = hb["prim"].copy()
    db = hb.to_device()
    oracle.ApplyFloors(p, hb)
    ctx_exact.ApplyFloors(p, db)
    ctx_exact.check()
    inner = (slice(None),) + hb.isl()
    floored = (hb["prim"][inner] != before[inner]).any(axis=0)
    assert 0.05 < floored.mean() < 0.95
    assert_bitwise(db["prim"], hb["prim"], "prim")
    assert_bitwise(db["cons"], hb["cons"], "cons")
