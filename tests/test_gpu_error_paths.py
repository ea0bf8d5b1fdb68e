"""What a call leaves behind when it fails, and what the next call on the same context then does: status words,
waits that are given up, allocations that are refused.  Every failure is made on the host side (a state that is not
a number, a limit that runs out, an allocation that is refused); no kernel faults."""
import numpy as np
import pytest

from misc_gb300 import model as M
from misc_gb300.astro import AstroError, AstroGPU

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
