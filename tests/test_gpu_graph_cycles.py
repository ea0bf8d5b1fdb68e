"""The solvers' iterations as captured graphs, on models small enough that they run resident by default
(ASTRO_OPT_RESIDENT 0 takes the graphs): conditional against unrolled cycles, a captured graph used by later solves,
constraints scaled anew, the exits for values that are not numbers, the iteration cap; and the two forms against
each other, FP32 with six DOF a node included."""
import numpy as np
import pytest

from misc_gb300 import model as M
from misc_gb300.astro import (OPT_RESIDENT, SOLVER_FGMRES_LEARNED, SOLVER_FGMRES_MIXED, SOLVER_GMRES_JACOBI_FP64, AstroError,
                              AstroGPU, precond_init, thermal_props)

pytestmark = pytest.mark.gpu

METHODS = [SOLVER_GMRES_JACOBI_FP64, SOLVER_FGMRES_MIXED, SOLVER_FGMRES_LEARNED]


def _block(resident=0):
    g = AstroGPU(M.config2(nx=8, ny=4, nz=4, seed=2))
    g.set_option(OPT_RESIDENT, resident)
    g.getElasticSolnLoad(1, export=False)
    g.assemble_fp32()
    g.scaleElasticMPC()
    return g, g.static_rhs()


@pytest.mark.parametrize("method", METHODS)
def test_unrolled_graph_gives_the_bits_of_the_conditional_one(method):
    g, b = _block()
    u1, s1 = g.solve_static(b, method=method, rtol=1e-10)
    g.set_option(2, 1)  # ASTRO_OPT_UNROLLED_CYCLES
    u2, s2 = g.solve_static(b, method=method, rtol=1e-10)
    assert s1.status == s2.status == 0 and s1.conditional_graph == 1 and s2.conditional_graph == 0
    assert s1.iterations == s2.iterations and np.array_equal(u1, u2)


@pytest.mark.parametrize("method", METHODS)
def test_captured_graph_serves_later_solves(method):
    """Other right-hand sides, and another matrix with its constraints scaled anew, through the graph of the first."""
    g, b = _block()
    u1, s1 = g.solve_static(b, method=method, rtol=1e-10)
    u2, _ = g.solve_static(2 * b, method=method, rtol=1e-10)
    g.getElasticSolnLoad(1, state=M.make_state(g.n, disp=np.random.default_rng(3).normal(0, 1e-4, g.n)), export=False)
    g.scaleElasticMPC()
    g.solve_static(b, method=method, rtol=1e-10)
    g.getElasticSolnLoad(1, export=False)
    g.scaleElasticMPC()
    u3, s3 = g.solve_static(b, method=method, rtol=1e-10)
    assert np.array_equal(u1, u3) and s1.iterations == s3.iterations
    assert np.linalg.norm(u2 - 2 * u1) <= 1e-8 * np.linalg.norm(u2)


def test_graph_falls_back_on_values_that_are_not_numbers():
    g, b = _block()
    p = precond_init(8, 100.0, 3)
    p.set_weights(p.weight_array() * 1e37)  # overflow in FP32
    u, st = g.solve_static(b, method=SOLVER_FGMRES_LEARNED, rtol=1e-10, precond=p)
    assert st.status == 0 and st.fallback == 1 and st.rel_residual <= 1e-10
    b[0] = np.nan
    for method in (SOLVER_GMRES_JACOBI_FP64, SOLVER_FGMRES_MIXED):
        with pytest.raises(AstroError) as e:
            g.solve_static(b, method=method, rtol=1e-10)
        assert e.value.code == 5


@pytest.mark.parametrize("method", METHODS)
def test_graph_iteration_cap(method):
    g, b = _block()
    with pytest.raises(AstroError) as e:
        g.solve_static(b, method=method, rtol=1e-13, restart=5, max_iters=5)
    assert e.value.code == 7


@pytest.mark.parametrize("method", METHODS)
def test_resident_cycle_agrees_with_the_graph(method):
    (g0, b), (g1, _) = _block(0), _block(1)
    (u0, s0), (u1, s1) = (g.solve_static(b, method=method, rtol=1e-10) for g in (g0, g1))
    assert s0.status == s1.status == 0 and s0.fallback == s1.fallback == 0
    # two residuals of 1e-10 apart: by the condition (below 1e4 for this block) in the solutions
    assert np.linalg.norm(u0 - u1) <= 1e-6 * np.linalg.norm(u0)


@pytest.mark.parametrize("resident", [0, 1])
@pytest.mark.parametrize("nx, ny", [(3, 2), (9, 7)])
def test_fp32_cycles_of_six_dof(nx, ny, resident):
    """The Jacobi cycles on a plate whose whole space a few cycles span, the learned ones on a larger one too."""
    g = AstroGPU(M.plate_shell(nx=nx, ny=ny, lx=0.1 * nx, ly=0.1 * ny, t=0.05, E=7.0e10, nu=0.33, rho=2700.0, pressure=1.0e3))
    g.set_option(OPT_RESIDENT, resident)
    g.getElasticSolnLoad(1, export=False)
    g.scaleElasticMPC()
    b = g.static_rhs()
    u, st = g.solve_static(b, method=SOLVER_FGMRES_LEARNED, rtol=1e-8, precond=precond_init(16, 1000.0, 6))
    assert st.status == 0 and st.fallback == 0 and st.rel_residual <= 1e-8
    if nx == 3:
        u, st = g.solve_static(b, method=SOLVER_FGMRES_MIXED, rtol=1e-8, restart=64)
        assert st.status == 0 and st.rel_residual <= 1e-8


def test_thermal_graph_agrees_with_the_resident_iterations():
    m = M.hex_block(7, 6, 5, jitter=0.1, seed=4)
    out = []
    for resident in (0, 1):
        g = AstroGPU(m)
        g.set_option(OPT_RESIDENT, resident)
        hot = np.nonzero(m.node_list[:, 0] < 1e-9)[0] + 1
        k = len(hot)
        nm = len(m.material_density)
        g.thermal_setup(thermal_props(np.tile([50.0, 50.0, 50.0, 0.0, 0.0, 0.0], (nm, 1)), np.full(nm, 400.0),
                                      mpc=(np.arange(k + 1), hot, np.ones(k), np.full(k, 3.0))))
        load = np.zeros(m.num_nodes)
        load += g.getThermalSolnLoad(1, export=False)[0]
        g.scaleThermalMPC()
        load = g.getThermalConstraintLoad(None, load)
        load = g.thermal_heat_gen(1.0e4, thermal_load=load)
        x, st = g.thermal_solve(load, rtol=1e-12)
        out.append((x, st.status, st.iterations))
    assert out[0][1] == out[1][1] == 0 and abs(out[0][2] - out[1][2]) <= 16
    assert np.linalg.norm(out[0][0] - out[1][0]) <= 1e-9 * np.linalg.norm(out[0][0])
