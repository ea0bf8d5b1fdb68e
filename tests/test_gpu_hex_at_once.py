"""Solid meshes on both sides of the size up to which all colours' elements are evaluated at once: the assembled
matrix and the residual against the sum of the element matrices and residuals."""
import numpy as np
import pytest

from misc_gb300 import model as M
from misc_gb300.astro import AstroGPU

pytestmark = pytest.mark.gpu


# 1 .. 4 colours of one element or more; 819; 4,096 | 4,352 elements (the bound of bricks); 6,144 | 8,448 (two groups of brickIM)
@pytest.mark.parametrize("dims", [(1, 1, 1), (2, 1, 1), (3, 2, 1), (13, 9, 7), (16, 16, 16), (16, 16, 17), (24, 16, 16), (16, 16, 33)])
@pytest.mark.parametrize("displaced", [False, True])
@pytest.mark.parametrize("im", [False, True])
def test_assembly_is_the_sum_of_the_elements(dims, displaced, im):
    m = M.hex_block(*dims, jitter=0.1, seed=6)
    if im:
        m.element_type = np.full(m.num_els, 81, np.int32)
    g = AstroGPU(m)
    rng = np.random.default_rng(1)
    u, x = 1e-4 * rng.standard_normal(g.n), rng.standard_normal(g.n)
    iu = 1e-5 * rng.standard_normal(max(1, g.int_vec_size)) if im else None
    st = M.make_state(g.n, disp=u, **({"internal_disp": iu} if im else {})) if displaced else None
    ke, ru = g.element_matrices(64, state=st, with_residual=True)
    load = g.getElasticSolnLoad(1, state=st, export=False)[0]
    y = g.apply_operator(x, 64)
    # DOF of the element matrices: component-major over the nodes
    nodes = np.asarray(m.element_list)[:, :8] - 1
    dof = np.concatenate([g.n_dof_index[nodes, v] - 1 for v in range(3)], axis=1)
    ys, ls = np.zeros(g.n), np.zeros(g.n)
    np.add.at(ys, dof, np.einsum("eij,ej->ei", ke, x[dof]))
    np.add.at(ls, dof, ru)
    # up to eight elements a node, 24 products each, rounded once: 192 x 1.1e-16
    assert np.linalg.norm(y - ys) <= 1e-13 * np.linalg.norm(ys)
    if displaced:
        assert np.linalg.norm(load + ls) <= 1e-13 * np.linalg.norm(ls)
