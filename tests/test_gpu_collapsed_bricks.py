"""Bricks that name a node twice (collapsed hexahedra: wedges, a pyramid): every entry point that adds into shared
entries from one element's own rows, against the oracle."""
import numpy as np
import pytest

from misc_gb300 import model as M
from misc_gb300.astro import AstroGPU, thermal_props, thermal_state
from oracle import Oracle

pytestmark = pytest.mark.gpu


def _collapsed():
    m = M.hex_block(4, 3, 2, jitter=0.1, seed=4)
    el = m.element_list
    el[5, 3], el[5, 7] = el[5, 2], el[5, 6]      # a wedge
    el[9, 0], el[9, 4] = el[9, 1], el[9, 5]
    el[17, 5:8] = el[17, 4]                      # a pyramid
    return m


def test_thermal_matrix_load_and_heat():
    m = _collapsed()
    g, o = AstroGPU(m), Oracle(m)
    rng = np.random.default_rng(2)
    nm = len(m.material_density)
    cond, sh = np.tile([50.0, 40.0, 30.0, 1.0, 2.0, 3.0], (nm, 1)), np.full(nm, 400.0)
    g.thermal_setup(thermal_props(cond, sh))
    t, tp, td = rng.uniform(10.0, 30.0, (3, m.num_nodes))
    load, mat, cols = g.getThermalSolnLoad(1, thermal_state(t, tp, td, 1, 0.5, 0.1), g.thermal_heat_gen(5.0))
    lo, mo, co, _ = o.thermal_soln_load(cond, sh, 1, t, tp, td, 1, 0.5, 0.1, load=o.thermal_heat_gen(5.0))
    # each entry a sum of at most 8 x 64 products, each rounded once in FP64
    assert np.array_equal(cols, co) and np.abs(mat - mo).max() <= 1e-12 * np.abs(mo).max()
    assert np.linalg.norm(load - lo) <= 1e-12 * np.linalg.norm(lo)


@pytest.mark.parametrize("im", [False, True])
def test_complex_step(im):
    m = M.add_design_variables(_collapsed(), 2, M.DCAT_ELASTIC_MODULUS)
    if im:
        m.element_type = np.full(m.num_els, 81, np.int32)
    g, o = AstroGPU(m), Oracle(m)
    rng = np.random.default_rng(3)
    iu = {"internal_disp": 1e-4 * rng.standard_normal(g.int_vec_size)} if im else {}
    st = M.make_state(g.n, disp=1e-3 * rng.standard_normal(g.n), **iu)
    for d in (1, 2):
        dr, idr = g.getdRelasticdD(d, h=1e-30, state=st)
        odr, oidr = o.drdd_complex(d, h=1e-30, state=st)
        assert np.linalg.norm(dr - odr) <= 1e-12 * np.linalg.norm(odr)
        if im:
            assert np.linalg.norm(idr - oidr) <= 1e-12 * np.linalg.norm(oidr)
