"""The many-column band solve over the band widths where its stages differ: no tile, one, two and three or more
below the diagonal, parts of tiles left over for a second round; forward and backward in one
launch and twisted."""
import ctypes

import numpy as np
import pytest

from misc_gb300 import model as M
from misc_gb300.astro import OPT_CASES_TWIST, AstroGPU
from newmark_cases_ref import newmark_cases
from oracle import Oracle
from oracle import oracle as OO

pytestmark = pytest.mark.gpu


# short side 1, 3, 8, 13, 40 elements: bands of about 18, 30, 60, 90 and 250 DOF (1, 1, 2, 3, 8 tiles)
@pytest.mark.parametrize("dims", [(2, 1), (9, 3), (14, 8), (20, 13), (44, 40)])
@pytest.mark.parametrize("twist", [0, 2])
def test_cases_against_direct_solves(dims, twist):
    nx, ny = dims
    L = OO._lib()  # the device's default shell tangent, whatever another module has set
    L.orc_set_quirk.argtypes = [ctypes.c_int, ctypes.c_int]
    L.orc_set_quirk(1, 0)
    m = M.plate_shell(nx=nx, ny=ny, lx=1.0, ly=ny / nx, t=0.02, E=7e10, nu=0.33, rho=2700.0, pressure=0.0)
    o, g = Oracle(m), AstroGPU(m)
    g.set_option(OPT_CASES_TWIST, twist)
    steps, dt = 3, 1e-5
    rng = np.random.default_rng(2)
    P = np.zeros((5, o.n))
    free = o.n_dof_index[(nx + 1):, 2] - 1
    for c in range(5):
        P[c, rng.choice(free, size=min(3, len(free)), replace=False)] = 1.0
    A = rng.uniform(10.0, 100.0, (5, steps))
    u, v, a, H, info = g.newmark_cases(dt, P, A, history=True)
    Ho, *_ = newmark_cases(o, P, A, dt, 0.25, 0.5, steps)
    # the file of the other many-case tests' bound: double-float copies of an FP64 factor
    for k in range(steps):
        for c in range(5):
            assert np.linalg.norm(H[k, c] - Ho[k, c]) <= 1e-9 * np.linalg.norm(Ho[k, c]), (k, c)
    assert info.last_rel_residual < 1e-10
