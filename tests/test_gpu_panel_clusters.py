"""The CTAs a panel: the untuned rule, the autotuner's choice for each kind of trailing update, and plans that are
kept where the cluster does not change."""
import numpy as np
import pytest

from misc_gb300 import model as M
from misc_gb300.astro import OPT_BAND_FP64_UPDATE, TUNE_CASES_CLUSTER, TUNE_PANEL_CLUSTER, AstroGPU

pytestmark = pytest.mark.gpu


def _ready(m):
    g = AstroGPU(m)
    g.getElasticSolnLoad(1, export=False)
    g.scaleElasticMPC()
    return g


def test_tuner_offers_the_untuned_choice(tmp_path):
    """A plate wide enough for 16 CTAs with FP64 updates, 8 with the others, whose clusters are portable."""
    g = _ready(M.plate_shell(nx=48, ny=40, lx=1.0, ly=1.0, t=0.01, clamp="ss", y0=0.0))
    assert g.panels_factor(0).cluster_size == 16
    times = {cs: min(g.panels_factor(cs).factor_seconds for _ in range(2)) for cs in (2, 4, 8, 0)}
    cache = tmp_path / "t.txt"
    choice = g.autotune(TUNE_PANEL_CLUSTER, cache)[1]
    assert len(cache.read_text().splitlines()) == 2  # FP64 and double-float
    assert choice == 0 and times[0] < min(times[cs] for cs in (2, 4, 8))  # (37 against 20 ms: twice the pipes)
    assert g.panels_factor(0).cluster_size == 16
    for kind in (3, 2, 0):
        g.set_option(OPT_BAND_FP64_UPDATE, kind)
        times = {cs: min(g.panels_factor(cs).factor_seconds for _ in range(2)) for cs in (2, 4, 8)}
        own = g.panels_factor(0)
        assert own.cluster_size in (2, 4, 8) and times[own.cluster_size] <= 1.1 * min(times.values())
    h = _ready(M.plate_shell(nx=48, ny=40, lx=1.0, ly=1.0, t=0.01, clamp="ss", y0=0.0))
    assert h.autotune(TUNE_PANEL_CLUSTER, cache)[1] == choice and len(cache.read_text().splitlines()) == 2


def test_each_kind_of_update_has_its_own_choice(tmp_path):
    """Many narrow panels: the tuned double-float factorisation is the fastest of its own clusters, not of FP64's."""
    g = _ready(M.panel_batch(96, n_range=(8, 40), n_dvars=0))
    g.autotune(TUNE_PANEL_CLUSTER, tmp_path / "t.txt")
    x = g.panels_solve(np.ones(g.n))[0] if g.panels_factor(0) else None  # the FP64 factor is the context's
    g.set_option(OPT_BAND_FP64_UPDATE, 3)
    times = {cs: min(g.panels_factor(cs).factor_seconds for _ in range(3)) for cs in (2, 4, 8)}
    own = min(g.panels_factor(0).factor_seconds for _ in range(3))
    assert own <= 1.05 * min(times.values()), (own, times)
    assert np.linalg.norm(g.panels_solve(np.ones(g.n))[0] - x) <= 1e-8 * np.linalg.norm(x)


def test_plan_is_kept_when_the_rule_picks_its_cluster():
    """An explicit 8, then 0 on a batch whose rule is 8: the same plan, so the same factor bit for bit, and no
    rebuilding (its ordering is host work of many times the factor's)."""
    g = _ready(M.panel_batch(24, n_range=(6, 14), n_dvars=0))
    b = np.random.default_rng(1).standard_normal(g.n)
    assert g.panels_factor(8).cluster_size == 8
    x8 = g.panels_solve(b)[0]
    assert g.panels_factor(0).cluster_size == 8
    assert np.array_equal(g.panels_solve(b)[0], x8)
    assert g.panels_factor(4).cluster_size == 4
    assert np.linalg.norm(g.panels_solve(b)[0] - x8) <= 1e-10 * np.linalg.norm(x8)


def test_choices_cached_for_earlier_kernels_are_not_applied(tmp_path):
    m = M.plate_shell(nx=8, ny=8, lx=1.0, ly=1.0, t=0.01, E=7e10, nu=0.33, rho=2700.0, pressure=0.0, clamp="ss", y0=0.0)
    cache = tmp_path / "t.txt"
    for what, then, now in ((TUNE_PANEL_CLUSTER, "/panel_cluster/", "/panel_cluster_fp64/"),
                            (TUNE_CASES_CLUSTER, "/cases_cluster/", "/cases_cluster_staged/")):
        g = AstroGPU(m)
        g.newmark_cases(1e-5, np.eye(g.n)[[200, 230]], np.ones((2, 2)))
        g.autotune(what, cache)
        line = [x for x in cache.read_text().splitlines() if now in x][0]
        cache.write_text(" ".join([line.split()[0].replace(now, then), "4", "0.0"]) + "\n")
        g.autotune(what, cache)
        assert any(now in x for x in cache.read_text().splitlines())
