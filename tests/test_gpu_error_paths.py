"""What a call leaves behind when it fails, and what the next call on the same context then does: status words,
waits that are given up, allocations that are refused.  Every failure is made on the host side (a state that is not
a number, a limit that runs out, an allocation that is refused); no kernel faults."""
import numpy as np
import pytest

from misc_gb300 import model as M
from misc_gb300.astro import (OPT_CASES_CLUSTER, OPT_FAIL_ALLOC, OPT_POLL_LIMIT, OPT_RESIDENT, SOLVER_FGMRES_LEARNED, SOLVER_FGMRES_MIXED,
                              SOLVER_GMRES_JACOBI_FP64, AstroError, AstroGPU, precond_init, thermal_props)

pytestmark = pytest.mark.gpu


def _plate(n=8):
    return M.plate_shell(nx=n, ny=n, lx=1.0, ly=1.0, t=0.01, E=7e10, nu=0.33, rho=2700.0, pressure=0.0, clamp="ss", y0=0.0)


def _cases(g, n=8, steps=3):
    pattern = np.zeros((1, g.n))
    pattern[0, g.n_dof_index[(n // 2) * (n + 1) + n // 2, 2] - 1] = 1.0
    return pattern, np.full((1, steps), 10.0)


def test_time_stepping_after_a_failed_factorisation():
    """A factorisation that meets a pivot that is not a number leaves its panel in the plan's status word; the
    twisted many-column solve on the same plan reads that word and does not factor the whole band."""
    g, h = AstroGPU(_plate()), AstroGPU(_plate())
    for c in (g, h):
        c.set_option(7, 2)  # ASTRO_OPT_CASES_TWIST: whenever the split is possible
    pattern, amp = _cases(g)
    ref = h.newmark_cases(1e-5, pattern, amp)[0]
    u = np.zeros(g.n)
    u[g.n // 2] = np.nan
    g.getElasticSolnLoad(1, state=M.make_state(g.n, disp=u), export=False)
    g.scaleElasticMPC()
    with pytest.raises(AstroError) as e:
        g.panels_factor(0)
    assert e.value.code == 4
    assert np.array_equal(g.newmark_cases(1e-5, pattern, amp)[0], ref)


def _block(resident=1, polls=0):
    g = AstroGPU(M.hex_block(7, 6, 5, lx=0.7, ly=0.6, lz=0.5, jitter=0.1, seed=4))
    g.set_option(OPT_RESIDENT, resident)
    g.set_option(OPT_POLL_LIMIT, polls)
    g.getElasticSolnLoad(1, export=False)
    g.assemble_fp32()
    g.scaleElasticMPC()
    return g, g.static_rhs()


@pytest.mark.parametrize("method", [SOLVER_GMRES_JACOBI_FP64, SOLVER_FGMRES_MIXED, SOLVER_FGMRES_LEARNED])
def test_solve_goes_on_when_a_wait_is_given_up(method):
    """A limit of one poll runs out in the first exchange of the resident cycle (and of the power iteration before
    it): the solve goes on as graphs, from the same x, so with their bits; with the limit back the next one is
    resident again."""
    graph, b = _block(resident=0)
    ug, sg = graph.solve_static(b, method=method, rtol=1e-10)
    g, _ = _block()
    u, s = g.solve_static(b, method=method, rtol=1e-10)
    few, _ = _block(polls=1)
    uf, sf = few.solve_static(b, method=method, rtol=1e-10)
    assert sf.status == 0 and sf.fallback == 0 and sf.rel_residual <= 1e-10
    assert np.array_equal(uf, ug) and sf.iterations == sg.iterations
    few.set_option(OPT_POLL_LIMIT, 0)
    ua, sa = few.solve_static(b, method=method, rtol=1e-10)
    assert sa.status == 0 and sa.rel_residual <= 1e-10
    if method != SOLVER_FGMRES_LEARNED:  # (which keeps its eigenvalue estimate, here that of the graph's iteration)
        assert np.array_equal(ua, u) and sa.iterations == s.iterations


def test_resident_six_dof_goes_on_when_a_wait_is_given_up():
    g = AstroGPU(M.plate_shell(nx=9, ny=7, lx=0.9, ly=0.7, t=0.05, E=7.0e10, nu=0.33, rho=2700.0, pressure=1.0e3))
    g.getElasticSolnLoad(1, export=False)
    g.scaleElasticMPC()
    b = g.static_rhs()
    p = precond_init(16, 1000.0, 6)
    for polls in (0, 1, 0):
        g.set_option(OPT_POLL_LIMIT, polls)
        u, st = g.solve_static(b, method=SOLVER_FGMRES_LEARNED, rtol=1e-8, precond=p)
        assert st.status == 0 and st.fallback == 0 and st.rel_residual <= 1e-8


def test_three_contexts_solve_at_once():
    """Resident launches of three contexts, each as wide as the GPU, from three threads."""
    import threading
    made = [_block() for _ in range(3)]
    ref = made[0][0].solve_static(made[0][1], rtol=1e-10)[0]
    out = [None] * 3
    gate = threading.Barrier(3)

    def run(i):
        g, b = made[i]
        gate.wait()
        out[i] = [g.solve_static(b, method=m, rtol=1e-10) for _ in range(4) for m in (SOLVER_GMRES_JACOBI_FP64, SOLVER_FGMRES_LEARNED)]
    threads = [threading.Thread(target=run, args=(i,)) for i in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for res in out:
        for u, st in res:
            assert st.status == 0 and st.rel_residual <= 1e-10
            assert np.linalg.norm(u - ref) <= 1e-6 * np.linalg.norm(ref)


def _thermal(resident=1, polls=0):
    m = M.hex_block(7, 6, 5, jitter=0.1, seed=4)
    g = AstroGPU(m)
    g.set_option(OPT_RESIDENT, resident)
    g.set_option(OPT_POLL_LIMIT, polls)
    hot = np.nonzero(m.node_list[:, 0] < 1e-9)[0] + 1
    k, nm = len(hot), len(m.material_density)
    g.thermal_setup(thermal_props(np.tile([50.0, 50.0, 50.0, 0.0, 0.0, 0.0], (nm, 1)), np.full(nm, 400.0),
                                  mpc=(np.arange(k + 1), hot, np.ones(k), np.full(k, 3.0))))
    load = g.getThermalSolnLoad(1, export=False)[0]
    g.scaleThermalMPC()
    return g, g.thermal_heat_gen(1.0e4, thermal_load=g.getThermalConstraintLoad(None, load))


def test_thermal_solve_goes_on_when_a_wait_is_given_up():
    """The resident conjugate gradients give up in their first exchange, before x moves: the batches that follow
    start where the graph's do.  The cap on the iterations and the next solve are as ever."""
    graph, b = _thermal(resident=0)
    xg, sg = graph.thermal_solve(b, rtol=1e-12)
    x, s = _thermal()[0].thermal_solve(b, rtol=1e-12)
    g, _ = _thermal(polls=1)
    xf, sf = g.thermal_solve(b, rtol=1e-12)
    assert sf.status == 0 and np.array_equal(xf, xg) and sf.iterations == sg.iterations
    with pytest.raises(AstroError) as e:
        g.thermal_solve(b, rtol=1e-12, max_iters=21)
    assert e.value.code == 7
    g.set_option(OPT_POLL_LIMIT, 0)
    xa, sa = g.thermal_solve(b, rtol=1e-12)
    assert sa.status == 0 and np.array_equal(xa, x) and sa.iterations == s.iterations


@pytest.mark.parametrize("twist", [0, 2])
@pytest.mark.parametrize("cluster", [2, 4, 8])
def test_time_stepping_reports_a_wait_that_is_given_up(twist, cluster):
    """A limit of one poll runs out in every stage of the many-column solve: each launch ends by itself, the call
    returns the error, and with the limit back the next call on the context is a fresh context's bit for bit."""
    g, h = AstroGPU(_plate()), AstroGPU(_plate())
    for c in (g, h):
        c.set_option(7, twist)
        c.set_option(OPT_CASES_CLUSTER, cluster)
    pattern, amp = _cases(g)
    ref = h.newmark_cases(1e-5, pattern, amp)[0]
    for graph in (True, False):
        g.set_option(OPT_POLL_LIMIT, 1)
        with pytest.raises(AstroError) as e:
            g.newmark_cases(1e-5, pattern, amp, graph=graph)
        assert e.value.code == 2 and "given up" in str(e.value)
        g.set_option(OPT_POLL_LIMIT, 0)
        assert np.array_equal(g.newmark_cases(1e-5, pattern, amp, graph=graph)[0], ref)


def test_thermal_solve_after_a_refused_allocation():
    """Whichever of the first solve's allocations is refused, the next solve builds what is missing (the table of
    columns among it, which only the first call fills)."""
    x, s = _thermal()[0].thermal_solve(_thermal()[1], rtol=1e-12)
    refused = 0
    for k in range(1, 40):
        g, b = _thermal()
        g.set_option(OPT_FAIL_ALLOC, k)
        try:
            g.thermal_solve(b, rtol=1e-12)
        except AstroError as e:
            assert e.code == 9
            refused += 1
        assert np.array_equal(g.thermal_solve(b, rtol=1e-12)[0], x), k
        if refused < k:
            break
    assert refused >= 10


def _bricks(im=False, dims=(8, 7, 6)):
    m = M.hex_block(*dims, jitter=0.1, seed=4)
    if im:
        m.element_type = np.full(m.num_els, 81, np.int32)
    return m


def _soln_load(m, displaced=True):
    def make():
        g = AstroGPU(m)
        st = None
        if displaced:
            iu = {"internal_disp": np.random.default_rng(2).normal(0.0, 1e-3, g.int_vec_size)} if g.int_vec_size else {}
            st = M.make_state(g.n, disp=np.random.default_rng(1).normal(0.0, 1e-3, g.n), **iu)
        return g, lambda: g.getElasticSolnLoad(1, state=st)
    return make


def _design():
    g = AstroGPU(M.add_design_variables(_bricks(), 1, M.DCAT_ELASTIC_MODULUS))
    st = M.make_state(g.n, disp=np.random.default_rng(1).normal(0.0, 1e-3, g.n))
    return g, lambda: g.getdRelasticdD(1, state=st)[:1]


def _heat():
    m = _bricks()
    g = AstroGPU(m)
    nm = len(m.material_density)
    g.thermal_setup(thermal_props(np.tile([50.0, 40.0, 30.0, 1.0, 2.0, 3.0], (nm, 1)), np.full(nm, 400.0)))
    return g, lambda: (*g.getThermalSolnLoad(1)[:2], g.thermal_heat_gen(2.0))


def _skyline(solve):
    g = AstroGPU(M.hex_block(2, 1, 1))
    lens = np.minimum(np.arange(300), 40)
    r = np.concatenate([[0], np.cumsum(lens + 1)]).astype(np.int32)
    a = np.random.default_rng(3).uniform(-1.0, 1.0, r[-1])
    a[r[1:] - 1] = 60.0
    if not solve:
        return g, lambda: (g.getSparseLDLFact(a, r),)
    fac = AstroGPU(M.hex_block(2, 1, 1)).getSparseLDLFact(a, r)
    return g, lambda: (g.solveSparseLDLFact(np.ones(300), fac, r),)


def _solve(method):
    g, b = _block()
    return g, lambda: (g.solve_static(b, method=method, rtol=1e-10)[0],)


# the call, and the relative tolerance of a result by another route: the same sums (0), the row sweep's (rounding of
# 40 products a row), the graph's (two residuals of 1e-10 apart: by the block's condition)
CALLS = {
    "brick8": (_soln_load(_bricks()), 0.0),
    "brick8_undisplaced": (_soln_load(_bricks(), False), 0.0),
    "brickIM": (_soln_load(_bricks(True)), 0.0),
    "brickIM_two_groups": (_soln_load(_bricks(True, (16, 16, 33))), 0.0),
    "shells": (_soln_load(M.plate_shell(nx=20, ny=17, lx=2.0, ly=1.7, t=0.05, E=7.0e10, nu=0.33, rho=2700.0, pressure=1.0e3)), 0.0),
    "design": (_design, 0.0),
    "heat": (_heat, 0.0),
    "skyline_factor": (lambda: _skyline(False), 1e-13),
    "skyline_solve": (lambda: _skyline(True), 1e-13),
    "thermal_solve": (lambda: (lambda g, b: (g, lambda: (g.thermal_solve(b, rtol=1e-12)[0],)))(*_thermal()), 1e-9),
    "fp64": (lambda: _solve(SOLVER_GMRES_JACOBI_FP64), 1e-6),
    "mixed": (lambda: _solve(SOLVER_FGMRES_MIXED), 1e-6),
    "learned": (lambda: _solve(SOLVER_FGMRES_LEARNED), 1e-6),
}


@pytest.mark.parametrize("name", list(CALLS))
def test_calls_with_a_refused_allocation(name):
    """Each allocation of the first call refused in turn: the call fails with ASTRO_ERR_NOMEM, or, where the refused
    one was scratch of a route that another needs less of, gives that one's result; the next call is as ever."""
    make, tol = CALLS[name]

    def near(out, tol):
        return all(x is None or np.linalg.norm(x - y) <= tol * np.linalg.norm(y) for x, y in zip(out, ref))
    ref = make()[1]()
    routes = 0
    for k in range(1, 60):
        g, call = make()
        g.set_option(OPT_FAIL_ALLOC, k)
        try:
            out = call()
            assert near(out, tol), k
            refused = "refused" in g._err(g.h)  # the context's last message
            routes += refused
        except AstroError as e:
            assert e.code == 9
            refused = True
        g.set_option(OPT_FAIL_ALLOC, 0)
        assert near(call(), tol), k
        if not refused:
            break
    assert not refused and routes >= 1, (k, routes)


def test_first_export_after_a_failed_call():
    """A call that fails leaves work queued on buffers that it has given back; the column numbers of the first export
    are formed on another stream, in a buffer that may be one of them."""
    m = _bricks()
    values, cols = AstroGPU(m).getElasticSolnLoad(1)[2:4]
    g = AstroGPU(m)
    u = np.random.default_rng(1).normal(0.0, 1e-3, g.n)
    for _ in range(3):
        with pytest.raises(AstroError) as e:  # no time step
            g.getElasticSolnLoad(1, state=M.make_state(g.n, disp=u, prev_disp=u, prev_vel=u, prev_acc=u, dynamic=1), export=False)
        assert e.value.code == 1
    v, c = g.getElasticSolnLoad(1)[2:4]
    assert np.array_equal(c, cols) and np.array_equal(v, values)
