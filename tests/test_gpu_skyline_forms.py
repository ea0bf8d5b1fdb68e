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


def _arrow(n, long):
    """Rows of two entries; the last row has `long`."""
    lens = np.minimum(np.arange(n), 2)
    lens[-1] = long
    r = np.concatenate([[0], np.cumsum(lens + 1)]).astype(np.int32)
    a = np.random.default_rng(3).uniform(-1.0, 1.0, r[-1])
    a[r[1:] - 1] = 5.0
    a[-1] = 2.0 * long + 5.0
    return a, r


@pytest.mark.parametrize("n, long", [(1000, 999), (4000, 500), (4000, 3999), (12000, 1500)])
def test_factor_of_a_profile_with_one_long_row(n, long):
    """Its band is many times the profile: in tiles where that is the shorter way, else by the row sweep (20 and
    59 ms for the last two; 218 and 243 ms in tiles)."""
    import time
    from oracle import Oracle
    a, r = _arrow(n, long)
    m = M.hex_block(2, 1, 1)
    g = AstroGPU(m)
    f = g.getSparseLDLFact(a, r)
    t0 = time.perf_counter()
    f = g.getSparseLDLFact(a, r)
    t = time.perf_counter() - t0
    fo = Oracle(m).ldl_fact(a, r)
    assert np.linalg.norm(f - fo) <= 1e-10 * np.linalg.norm(fo)
    assert t < 0.12
    b = np.random.default_rng(4).standard_normal(n)
    assert np.linalg.norm(g.solveSparseLDLFact(b, fo, r) - Oracle.ldl_solve(fo, r, b)) <= 1e-10 * np.linalg.norm(b)
