"""The reciprocals of the pivots in the FP64 band LDL^T are the division's: decoupled pairs of rows [[d, 1], [1, e]]
have L = fl(1 / d), bit for bit, over mantissas and the whole range of exponents."""
import numpy as np
import pytest

from misc_gb300 import model as M
from misc_gb300.astro import AstroGPU

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lo, hi", [(-30, 31), (-1021, 1022), (-1021, -1015), (1015, 1022)])
def test_reciprocal_pivots_are_the_divisions(lo, hi):
    rng = np.random.default_rng(1)
    n = 40000
    r = np.concatenate([[0], np.cumsum(np.tile([1, 2], n // 2))]).astype(np.int32)
    d = np.ldexp(rng.uniform(1.0, 2.0, n // 2), rng.integers(lo, hi, n // 2)) * rng.choice([-1.0, 1.0], n // 2)
    a = np.empty(r[-1])
    a[0::3], a[1::3], a[2::3] = d, 1.0, 1e300
    f = AstroGPU(M.hex_block(2, 1, 1)).getSparseLDLFact(a, r)
    assert np.array_equal(f[0::3], d) and np.array_equal(f[1::3], 1.0 / d)
