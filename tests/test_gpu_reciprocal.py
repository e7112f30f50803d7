"""The integer-pipe 1/x and 1/sqrt(x) of the production build at the edges of
their fixed-point steps: significands of all zeros, all ones and single bits,
every exponent of the fast range and its ends, both signs (rcp).  Bars: one
ulp of the correctly rounded 1/x, two of 1.0 / sqrt(x) (rounded twice)."""
import numpy as np
import pytest

from phoebus_gb300 import abi
from tests.test_gpu_math import _gpu_eval, _ulps

pytestmark = pytest.mark.gpu


def _edge_args():
    man = [0, 1, (1 << 52) - 1, (1 << 52) - 2] + [1 << k for k in range(52)]
    man += [((1 << 52) - 1) ^ (1 << k) for k in range(52)] + [(1 << 29) - 1, (1 << 29), ((1 << 23) - 1) << 29]
    e = np.concatenate([np.arange(1, 40), np.arange(1000, 1046), np.arange(2010, 2047)]).astype(np.uint64)
    bits = (e[:, None] << np.uint64(52)) | np.array(man, dtype=np.uint64)[None, :]
    return bits.ravel().view(np.float64)


@pytest.mark.parametrize("fn", ["rcp", "rsqrt"])
def test_edges(built, fn):
    lib = abi.load(False)
    x = _edge_args()
    got = _gpu_eval(lib, fn, x, None)
    ref = 1.0 / x if fn == "rcp" else 1.0 / np.sqrt(x)
    # reciprocals of the largest arguments are subnormal: compared absolutely there
    nrm = np.abs(ref) >= np.finfo(float).tiny
    assert _ulps(got[nrm], ref[nrm]).max() <= (1 if fn == "rcp" else 2)
    assert np.abs(got[~nrm] - ref[~nrm]).max(initial=0.0) <= 5e-324
    if fn == "rcp":
        neg = _gpu_eval(lib, fn, -x, None)
        assert np.array_equal(neg, -got)
