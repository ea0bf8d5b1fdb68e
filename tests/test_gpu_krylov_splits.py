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
