"""The splits of the block-ELL solver by model size: rows a CTA in the products, vector rows a CTA in the
Gram-Schmidt passes.  The residual's products (all sizes of its split, remainders included) against a sparse
product on the host; solves at each split converge and their reported residual is that of the host product."""
import numpy as np
import pytest

from misc_gb300 import model as M
from misc_gb300.astro import SOLVER_FGMRES_LEARNED, SOLVER_FGMRES_MIXED, SOLVER_GMRES_JACOBI_FP64, AstroGPU
from oracle import Oracle

pytestmark = pytest.mark.gpu


def _system(m):
    g, o = AstroGPU(m), Oracle(m)
    _, _, mat, cols, _ = g.getElasticSolnLoad(1)
    mm, _ = g.scaleElasticMPC()
    C = o.mpc_scipy(mm)
    return g, (o.csr_scipy(mat, cols) + C.T @ C).tocsr()


# nodes: 60 and 1,331, remainders of 32 rows; 38,874 | 39,204 (32 | 128 rows a CTA)
@pytest.mark.parametrize("dims", [(4, 3, 2), (10, 10, 10), (20, 20, 21), (20, 20, 22), (30, 32, 37), (32, 32, 35)])
def test_products_match_host(dims):
    g, A = _system(M.hex_block(*dims, jitter=0.1, seed=3))
    u = np.random.default_rng(5).standard_normal(g.n)
    y = A @ u
    # at most 81 products a row and the penalty's, each rounded once in FP64: 2-norm 81 x 1.1e-16
    assert np.linalg.norm(g.apply_operator(u, 64) - y) <= 1e-13 * np.linalg.norm(y)


def test_products_match_host_shells():
    g, A = _system(M.config1())
    u = np.random.default_rng(5).standard_normal(g.n)
    y = A @ u
    assert np.linalg.norm(g.apply_operator(u, 64) - y) <= 1e-13 * np.linalg.norm(y)


# vector rows a CTA: 29,106 -> 128, 48,750 -> 256, 89,373 -> 512, 164,616 -> 1,024; small ones first
@pytest.mark.parametrize("dims", [(1, 1, 1), (5, 3, 2), (20, 20, 21), (24, 24, 25), (30, 30, 30), (37, 37, 37)])
@pytest.mark.parametrize("method", [SOLVER_GMRES_JACOBI_FP64, SOLVER_FGMRES_MIXED, SOLVER_FGMRES_LEARNED])
def test_solves_converge_at_each_split(dims, method):
    m = M.hex_block(*dims, lx=0.1 * dims[0], ly=0.1 * dims[1], lz=0.1 * dims[2], jitter=0.1, seed=3)
    g, A = _system(m)
    if method != SOLVER_GMRES_JACOBI_FP64:
        g.assemble_fp32()
        g.scaleElasticMPC()
    b = g.static_rhs()
    u, st = g.solve_static(b, method=method, rtol=1e-8)
    assert st.status == 0 and st.rel_residual <= 1e-8
    # the reported residual is formed in FP64: against the host's within the products' rounding, which
    # the penalty's entries scale up by ||A|| ||u|| / ||b||
    r = np.linalg.norm(b - A @ u) / np.linalg.norm(b)
    noise = 81 * 1.1e-16 * np.linalg.norm(abs(A) @ abs(u)) / np.linalg.norm(b)
    assert abs(r - st.rel_residual) <= 2.0 * noise + 1e-3 * st.rel_residual, (r, st.rel_residual, noise)


# the resident cycle: fewer rows than SMs, a last CTA with fewer rows, several row groups
@pytest.mark.parametrize("dims", [(2, 1, 1), (7, 6, 5), (10, 10, 10), (16, 15, 14)])
@pytest.mark.parametrize("restart", [7, 64])
@pytest.mark.parametrize("method", [SOLVER_GMRES_JACOBI_FP64, SOLVER_FGMRES_MIXED, SOLVER_FGMRES_LEARNED])
def test_resident_cycle_solves(dims, restart, method):
    m = M.hex_block(*dims, lx=0.1 * dims[0], ly=0.1 * dims[1], lz=0.1 * dims[2], jitter=0.1, seed=4)
    g, A = _system(m)
    b = g.static_rhs()
    u, st = g.solve_static(b, method=method, rtol=1e-8, restart=restart)
    assert st.status == 0 and st.rel_residual <= 1e-8
    r = np.linalg.norm(b - A @ u) / np.linalg.norm(b)
    noise = 81 * 1.1e-16 * np.linalg.norm(abs(A) @ abs(u)) / np.linalg.norm(b)
    assert abs(r - st.rel_residual) <= 2.0 * noise + 1e-3 * st.rel_residual, (r, st.rel_residual, noise)


# one FP64 cycle of k steps against the least residual over the host's Krylov space (6 DOF and 3; the
# thin plate's space of 64 steps moves by 1e-6 under roundings of its products alone)
@pytest.mark.parametrize("shells, k", [(True, 1), (True, 2), (True, 33), (False, 1), (False, 2), (False, 33), (False, 64)])
def test_resident_cycle_takes_the_least_residual(shells, k):
    if shells:
        m = M.plate_shell(nx=9, ny=7, lx=0.9, ly=0.7, t=0.05, E=7.0e10, nu=0.33, rho=2700.0, pressure=1.0e3)
    else:
        m = M.hex_block(7, 6, 5, jitter=0.1, seed=4)
    g, A = _system(m)
    b = g.static_rhs()
    _, st = g.solve_static(b, method=SOLVER_GMRES_JACOBI_FP64, rtol=1e-14, restart=k, max_iters=k, allow_maxit=True)
    AD = A.multiply(1.0 / A.diagonal()[None, :]).tocsr()
    Q = np.zeros((len(b), k + 1))
    Q[:, 0] = b / np.linalg.norm(b)
    for j in range(k):
        w = AD @ Q[:, j]
        for _ in range(2):
            w -= Q[:, : j + 1] @ (Q[:, : j + 1].T @ w)
        Q[:, j + 1] = w / np.linalg.norm(w)
    B = AD @ Q[:, :k]
    y = np.linalg.lstsq(B, b, rcond=None)[0]
    least = np.linalg.norm(b - B @ y) / np.linalg.norm(b)
    # rounding moves the space by eps x the condition of its images (6e4 for the plate's 33), and more per step
    assert abs(st.rel_residual - least) <= 1e-6 * max(least, 1e-2), (st.rel_residual, least)
