"""GPU parity of the thermal path against the oracle through the C ABI: conductivity and
capacitance (rank-ordered thermal load, the reference's CSR values and columns) for bricks with
rotated sections and anisotropic conductivity and for warped shells with rotated layers, static
and transient states; thermal constraints (scaling, constraint load); heat generation; the device
conjugate-gradient solve against a direct solve.  1e-12 relative for element quantities, 1e-10 for
solutions."""
import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg as spla

from misc_gb300 import model as M
from misc_gb300.astro import AstroError, AstroGPU, thermal_props, thermal_state
from oracle import Oracle

pytestmark = pytest.mark.gpu


def _close(a, b, tol):
    assert np.linalg.norm(np.asarray(a) - np.asarray(b)) <= tol * np.linalg.norm(b), np.abs(np.asarray(a) - b).max()


def _materials(nm, seed):
    rng = np.random.default_rng(seed)
    k = rng.uniform(10.0, 60.0, (nm, 3))
    off = rng.uniform(-2.0, 2.0, (nm, 3))
    return np.hstack([k, off]), rng.uniform(400.0, 900.0, nm)


def _rotation(a, b, c):
    ca, sa, cb, sb, cc, sc = np.cos(a), np.sin(a), np.cos(b), np.sin(b), np.cos(c), np.sin(c)
    Rz = np.array([[ca, -sa, 0], [sa, ca, 0], [0, 0, 1]])
    Ry = np.array([[cb, 0, sb], [0, 1, 0], [-sb, 0, cb]])
    Rx = np.array([[1, 0, 0], [0, cc, -sc], [0, sc, cc]])
    return Rz @ Ry @ Rx


def _brick():
    m = M.hex_block(5, 4, 3, lx=1.5, ly=1.0, lz=0.75, seed=2)
    m.section_orient = np.broadcast_to(_rotation(0.3, -0.2, 0.5), m.section_orient.shape).copy()
    return m


def _shell():
    m = M.plate_shell(nx=5, ny=4, lx=2.0, ly=1.0, t=0.03)
    rng = np.random.default_rng(5)
    X = m.node_list.copy()
    X[:, :2] += 0.05 * rng.uniform(-1, 1, (len(X), 2))
    X[:, 2] += 0.02 * rng.uniform(-1, 1, len(X))
    m.node_list = X
    m.layup_angle = np.array([0.3])
    return m


@pytest.fixture(scope="module", params=["brick", "shell"])
def case(request):
    m = _brick() if request.param == "brick" else _shell()
    nm = len(m.material_density)
    cond, sh = _materials(nm, 3)
    X = m.node_list
    nodes = np.nonzero(X[:, 0] <= 1e-9 + X[:, 0].min())[0] + 1
    mpc = (np.arange(len(nodes) + 1), nodes, np.ones(len(nodes)), np.full(len(nodes), 25.0))
    g, o = AstroGPU(m), Oracle(m)
    g.thermal_setup(thermal_props(cond, sh, mpc))
    return m, g, o, cond, sh, mpc


def test_thermal_soln_load_static_and_transient(case):
    m, g, o, cond, sh, mpc = case
    N = m.num_nodes
    rng = np.random.default_rng(7)
    T, pT, pTd = rng.uniform(0, 100, N), rng.uniform(0, 100, N), rng.uniform(-5, 5, N)
    for dyn in (0, 1):
        kw = dict(temp=T, prev_temp=pT, prev_tdot=pTd, dynamic=dyn, gamma=0.6, del_t=0.05)
        lg, mg, cg = g.getThermalSolnLoad(1, state=thermal_state(T, pT, pTd, dyn, 0.6, 0.05))
        lo, mo, co, ro = o.thermal_soln_load(cond, sh, 1, **kw)
        assert np.array_equal(cg, co)
        _close(mg, mo, 1e-12)
        _close(lg, lo, 1e-12)
    assert g.therm_mat_size == len(mo)


def test_thermal_constraints_heat_gen_and_solve(case):
    m, g, o, cond, sh, mpc = case
    N = m.num_nodes
    g.getThermalSolnLoad(1, export=False)
    mm, mr = g.scaleThermalMPC()
    A, b, rows = o.thermal_system(cond, sh, mpc)
    _close(mm, np.concatenate([r[1] for r in rows]), 1e-13)
    _close(mr, [r[2] for r in rows], 1e-13)
    T = np.random.default_rng(3).uniform(0, 50, N)
    _close(g.getThermalConstraintLoad(T), o.thermal_constraint_load(rows, T, np.zeros(N)), 1e-12)
    els = np.array([1, 3, 3, m.num_els])
    _close(g.thermal_heat_gen(7.0, elements=els), o.thermal_heat_gen(7.0, elements=els), 1e-12)
    fe = np.array([1, 2, m.num_els], np.int32)
    fn = np.array([4, 2, 1], np.int32) if m.element_type[0] == 8 else np.array([1, 2, 1], np.int32)
    _close(g.thermal_surface_flux(fe, fn, 3.5), o.thermal_surface_flux(fe, fn, 3.5), 1e-12)
    q = g.thermal_heat_gen(7.0)
    _close(q, o.thermal_heat_gen(7.0), 1e-12)
    rhs = g.getThermalConstraintLoad(None, q.copy())
    x, st = g.thermal_solve(rhs, rtol=1e-12)
    assert st.status == 0
    xr = spla.spsolve(A.tocsc(), rhs)
    _close(x, xr, 1e-9)


def test_thermal_errors():
    m = _brick()
    g = AstroGPU(m)
    with pytest.raises(AstroError):
        g.thermal_setup(thermal_props(np.ones((1, 6)), np.ones(1)))  # fewer materials than the mesh uses
    nm = len(m.material_density)
    cond, sh = _materials(nm, 1)
    g.thermal_setup(thermal_props(cond, sh))
    with pytest.raises(AstroError) as e:
        g.thermal_solve(np.ones(m.num_nodes))
    assert e.value.code == 8


@pytest.mark.parametrize("dims", [(1, 1, 1), (5, 5, 5), (16, 4, 2), (43, 3, 1)])
@pytest.mark.parametrize("dynamic", [0, 1])
def test_brick_matrix_load_and_solve_over_sizes(dims, dynamic):
    """The factorised brick kernel, the constraint load and the conjugate gradients where a CTA or a
    tile of rows is not full: one element, a remainder, exactly one CTA, one element over; constraints
    that share nodes; heat generation on a list with repeats."""
    nx, ny, nz = dims
    m = M.hex_block(nx, ny, nz, lx=nx * 0.3, ly=ny * 0.2, lz=nz * 0.25, seed=nx, jitter=0.2)
    rng = np.random.default_rng(nx)
    nm = len(m.material_density)
    k = rng.uniform(20.0, 60.0, nm)
    cond = np.concatenate([k[:, None] * [1.0, 0.8, 1.2], k[:, None] * rng.uniform(-0.2, 0.2, (nm, 3))], axis=1)
    sh = rng.uniform(300.0, 500.0, nm)
    N = m.num_nodes
    mpc = (np.array([0, 1, 3, 5]), np.array([1, 2, 1, N, 2]), np.array([1.0, 1.0, -0.5, 2.0, 1.0]),
           np.array([10.0, 3.0, 20.0]))
    g, o = AstroGPU(m), Oracle(m)
    g.thermal_setup(thermal_props(cond, sh, mpc))
    t, tp, td = rng.uniform(10.0, 30.0, (3, N))
    els = rng.integers(1, m.num_els + 1, 7)
    st = thermal_state(t, tp, td, dynamic, 0.5, 0.1)
    load, mat, cols = g.getThermalSolnLoad(1, st, g.thermal_heat_gen(5.0, els))
    lo, mo, co, row = o.thermal_soln_load(cond, sh, 1, t, tp, td, dynamic, 0.5, 0.1, load=o.thermal_heat_gen(5.0, els))
    assert np.array_equal(cols, co) and np.abs(mat - mo).max() <= 1e-12 * np.abs(mo).max()
    assert np.linalg.norm(load - lo) <= 1e-12 * np.linalg.norm(lo)
    mm, mr = g.scaleThermalMPC()
    rank = g.current_rank - 1
    C = np.zeros((3, N))
    for r in range(3):
        for q in range(mpc[0][r], mpc[0][r + 1]):
            C[r, rank[mpc[1][q] - 1]] += mm[q]
    f = g.getThermalConstraintLoad(t, load.copy())
    fo = load + C.T @ (mr - C @ t)
    assert np.linalg.norm(f - fo) <= 1e-12 * np.linalg.norm(fo)
    # the solve with two fixed nodes (a diagonal penalty): direct solve of the symmetrically scaled system
    mpc = (np.array([0, 1, 2]), np.array([1, N]), np.ones(2), np.zeros(2))
    g.thermal_setup(thermal_props(cond, sh, mpc))
    _, mat, cols = g.getThermalSolnLoad(1, st)
    mm, _ = g.scaleThermalMPC()
    K = np.zeros((N, N))
    for r in range(N):
        for q in range(row[r], row[r + 1]):
            K[r, cols[q] - 1] += mat[q]
    for q in range(2):
        K[rank[mpc[1][q] - 1], rank[mpc[1][q] - 1]] += mm[q] ** 2
    d = 1.0 / np.sqrt(np.diag(K))
    b = rng.standard_normal(N)
    x, stats = g.thermal_solve(b, rtol=1e-13)
    xd = d * np.linalg.solve(d[:, None] * K * d, d * b)
    assert stats.status == 0 and np.linalg.norm(x - xd) <= 1e-9 * np.linalg.norm(xd)


# rows of a CTA of the resident iterations: 16 (a last CTA of 3), one to four threads a row; 100,878 nodes do not fit
# the SMs' shared memory
@pytest.mark.parametrize("dims", [(10, 10, 10), (24, 17, 13), (40, 30, 21), (50, 45, 42)])
def test_solve_over_sizes(dims):
    nx, ny, nz = dims
    m = M.hex_block(nx, ny, nz, lx=nx * 0.1, ly=ny * 0.1, lz=nz * 0.1, seed=nx, jitter=0.2)
    rng = np.random.default_rng(nx)
    nm = len(m.material_density)
    k = rng.uniform(20.0, 60.0, nm)
    cond = np.concatenate([k[:, None] * np.ones((nm, 3)), np.zeros((nm, 3))], axis=1)
    N = m.num_nodes
    # one node fixed, two tied
    mpc = (np.array([0, 1, 3]), np.array([1, N, N // 2]), np.array([1.0, 1.0, -1.0]), np.zeros(2))
    g = AstroGPU(m)
    g.thermal_setup(thermal_props(cond, np.full(nm, 400.0), mpc))
    _, mat, cols = g.getThermalSolnLoad(1)
    mm, _ = g.scaleThermalMPC()
    rank = g.current_rank - 1
    el = rank[np.asarray(m.element_list)[:, :8] - 1]
    # a row's entries: the nodes of its elements
    pairs = np.unique(np.repeat(el, 8, axis=1).ravel() * np.int64(N) + np.tile(el, (1, 8)).ravel())
    rows = np.concatenate([[0], np.cumsum(np.bincount(pairs // N, minlength=N))])
    A = sp.csr_matrix((mat, cols - 1, rows), shape=(N, N))
    C = sp.csr_matrix((mm, (np.array([0, 1, 1]), rank[mpc[1] - 1])), shape=(2, N))
    b = rng.standard_normal(N)
    x, stats = g.thermal_solve(b, rtol=1e-10)
    assert stats.status == 0 and stats.rel_residual <= 1e-10
    r = np.linalg.norm(b - (A @ x + C.T @ (C @ x)))
    # the recurrence's residual drifts from the true one by roundings of A x (the penalty is 100 max|A|)
    noise = 27 * 1.1e-16 * stats.iterations * np.linalg.norm(abs(A) @ abs(x) + abs(C).T @ (abs(C) @ abs(x)))
    assert r <= 1.01e-10 * np.linalg.norm(b) + noise
