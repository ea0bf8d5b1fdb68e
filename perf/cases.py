"""The work that users of this library have it do, as measurable cases.

Every case is one call sequence of a structural analysis, through the methods of AstroGPU (the
host-array boundary that replaces AStrO's Fortran subroutines), on seeded synthetic meshes of
misc_gb300.model:

  skyline    getSparseLDLFact + solveSparseLDLFact on the caller's row-skyline arrays
  assemble   getElasticSolnLoad of a mesh (bricks, brickIM, shells; undeformed or displaced state),
             exported to the reference CSR or kept on the device and applied to a vector
  solve      the static solve of a block by one of the Krylov solvers, after an FP32 assembly where
             the solver works from one
  panels     a batch of independent shell panels: assembly, band factorisation, displacement and
             design-sensitivity solves (panels.solve_batch)
  newmark    many load cases of a plate stepped through one factorisation
  gradient   the static design gradient of a block by the adjoint
  thermal    conductivity assembly, heat load and solve

The sizes are those of the library's configurations (the 40x8 cantilever plate, the 64x32x32
block, the config-4 and config-5 models, the panel batch) or smaller and odd versions of them.
Nodal results are returned by node, (nodes, components), as a user reads them off.
"""
import math

import numpy as np
import torch

from misc_gb300 import model as M
from misc_gb300 import panels
from misc_gb300.astro import (OPT_SHELL_MEAN_ROT_TERM, SOLVER_FGMRES_LEARNED, SOLVER_FGMRES_MIXED,
                              SOLVER_GMRES_JACOBI_FP64, AstroGPU, thermal_props, thermal_state)

METHODS = {"fp64": SOLVER_GMRES_JACOBI_FP64, "mixed": SOLVER_FGMRES_MIXED, "learned": SOLVER_FGMRES_LEARNED}
RTOL = 1e-12     # of the solves: FP64 answers to the conditioning of the models
DVARS = 8        # design variables of the gradient and of the panels' sensitivities


def listed():
    return [
        # the skyline of the 40x8 cantilever plate (2,214 rows, short rows): the smallest direct
        # solve a drop-in caller makes, all latency
        {"name": "skyline_plate", "kind": "skyline", "comps": 6, "long": 41, "width": 9, "depth": 1},
        # the skyline of a solid block: rows of a hundred entries
        {"name": "skyline_block", "kind": "skyline", "comps": 3, "long": 25, "width": 10, "depth": 9},
        # a small odd block exported to the reference CSR: what a Fortran caller gets per call
        {"name": "brick_export_small", "kind": "assemble", "element": "brick", "nx": 13, "ny": 9, "nz": 7,
         "displaced": False, "export": True},
        # a Newton iteration of the largest block: tangent and residual at a displaced state
        {"name": "brick_newton_large", "kind": "assemble", "element": "brick", "nx": 64, "ny": 32, "nz": 32,
         "displaced": True, "export": False},
        # incompatible-modes bricks at a displaced state, an odd block
        {"name": "brickim_newton", "kind": "assemble", "element": "brickIM", "nx": 25, "ny": 15, "nz": 11,
         "displaced": True, "export": False},
        # a shell plate at a displaced state, as a nonlinear step evaluates it
        {"name": "shell_newton", "kind": "assemble", "element": "shell", "nx": 97, "ny": 64, "nz": 1,
         "displaced": True, "export": False},
        # the solver users pick for a block: FP32 assembly, learned FGMRES, FP64 refinement
        {"name": "solve_learned", "kind": "solve", "method": "learned", "nx": 48, "ny": 24, "nz": 24},
        # the plain FP64 solver on a smaller odd block
        {"name": "solve_fp64", "kind": "solve", "method": "fp64", "nx": 27, "ny": 13, "nz": 11},
        # a batch of panels with their thickness sensitivities
        {"name": "panels_batch", "kind": "panels", "count": 32},
        # load cases of the simply supported plate
        {"name": "newmark_cases", "kind": "newmark", "n": 64, "cases": 17, "steps": 100},
        # design gradient over modulus groups
        {"name": "gradient_block", "kind": "gradient", "nx": 32, "ny": 16, "nz": 15},
        # a thermal step of a block
        {"name": "thermal_block", "kind": "thermal", "nx": 64, "ny": 32, "nz": 32, "dynamic": False},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _block_sides(rng, e_lo, e_hi):
    """A block of about e elements, twice as long as wide, with odd and unequal sides among them."""
    w = (math.exp(rng.uniform(math.log(e_lo), math.log(e_hi))) / 2.0) ** (1.0 / 3.0)
    ny = max(2, int(round(w * rng.uniform(0.85, 1.1))))
    nz = max(2, int(round(w * rng.uniform(0.85, 1.1))))
    nx = max(2, int(min(2.0 * w * rng.uniform(0.85, 1.1), e_hi / (ny * nz))))
    return nx, ny, nz


def draw(rng):
    kind = rng.choice(["skyline", "assemble", "assemble", "solve", "panels", "newmark", "gradient", "thermal"])
    if kind == "skyline":
        depth = rng.choice([1, _log_int(rng, 2, 9)])
        return {"kind": kind, "comps": rng.choice([3, 6]) if depth == 1 else 3, "long": _log_int(rng, 8, 25),
                "width": _log_int(rng, 2, 10), "depth": depth}
    if kind == "assemble":
        el = rng.choice(["brick", "brick", "brickIM", "shell"])
        if el == "shell":
            nx, ny, nz = _log_int(rng, 6, 97), _log_int(rng, 3, 64), 1
        else:
            nx, ny, nz = _block_sides(rng, 60, 65536 if el == "brick" else 4125)
        return {"kind": kind, "element": el, "nx": nx, "ny": ny, "nz": nz, "displaced": rng.random() < 0.7,
                "export": nx * ny * nz < 2000 and rng.random() < 0.5}
    if kind == "solve":
        method = rng.choice(["learned", "learned", "fp64", "mixed"])
        nx, ny, nz = _block_sides(rng, 200, {"learned": 27648, "fp64": 3861, "mixed": 2000}[method])
        return {"kind": kind, "method": method, "nx": nx, "ny": ny, "nz": nz}
    if kind == "panels":
        return {"kind": kind, "count": _log_int(rng, 1, 32)}
    if kind == "newmark":
        return {"kind": kind, "n": _log_int(rng, 8, 64), "cases": rng.randint(1, 17), "steps": _log_int(rng, 10, 100)}
    if kind == "gradient":
        nx, ny, nz = _block_sides(rng, 60, 7680)
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz}
    nx, ny, nz = _block_sides(rng, 60, 65536)
    return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "dynamic": rng.random() < 0.5}


# ---- inputs -------------------------------------------------------------------------------------


def _skyline(case, seed):
    """A symmetric positive definite row skyline as an FE stiffness has it: `comps` equal blocks
    (component-major numbering), each the weighted graph Laplacian of a long x width x depth grid of
    nodes numbered level by level along the long side, the first level held by a penalty.
    Returns (aLTri, ARange, right-hand side), and the dense blocks for exact()."""
    rng = np.random.default_rng(seed)
    L, w, d = case["long"], case["width"], case["depth"]
    n = L * w * d
    idx = np.arange(n)
    pos = np.stack([idx // (w * d), (idx // d) % w, idx % d], axis=1)
    pairs = []
    for off in ((a, b, c) for a in (0, 1) for b in (-1, 0, 1) for c in (-1, 0, 1)):
        if off <= (0, 0, 0):
            continue
        q = pos + np.array(off)
        ok = np.all((q >= 0) & (q < np.array([L, w, d])), axis=1)
        pairs.append(np.stack([idx[ok], (q[ok, 0] * w + q[ok, 1]) * d + q[ok, 2]], axis=1))
    lo, hi = np.sort(np.concatenate(pairs), axis=1).T
    first = np.arange(n)
    np.minimum.at(first, hi, lo)
    start = np.concatenate([[0], np.cumsum(np.arange(n) - first + 1)])
    rows, blocks = [], []
    for _ in range(case["comps"]):
        val = rng.uniform(0.5, 1.5, len(lo))
        diag = 0.01 + np.bincount(lo, val, n) + np.bincount(hi, val, n)
        diag[: w * d] += 1.0e4
        a = np.zeros(start[-1])
        a[start[1:] - 1] = diag
        a[start[hi + 1] - 1 - (hi - lo)] = -val
        rows.append(a)
        blocks.append((diag, lo, hi, val))
    rng_all = np.concatenate([[0]] + [start[1:] + k * start[-1] for k in range(case["comps"])]).astype(np.int32)
    return np.concatenate(rows), rng_all, rng.standard_normal(n * case["comps"]), blocks


def _block(case, seed):
    """A heterogeneous block of the config-2 family (64x32x32 on 4x2x2): jittered nodes, log-normal
    modulus, x = 0 clamped."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    return M.hex_block(nx=nx, ny=ny, nz=nz, lx=nx / 16.0, ly=ny / 16.0, lz=nz / 16.0, seed=seed)


def _grouped_block(case, seed):
    return M.add_design_variables(_block(case, seed), DVARS, M.DCAT_ELASTIC_MODULUS)


def _smooth_disp(m, seed, size):
    """A displaced state by node: a bending-like smooth field plus one per cent of noise."""
    rng = np.random.default_rng(seed)
    x = m.node_list / np.ptp(m.node_list[:, 0])
    a = rng.uniform(0.5, 1.5, (3, 3)) * rng.choice([-1.0, 1.0], (3, 3))
    u = size * (x[:, :1] ** 2 * a[0] + x[:, :1] * x[:, 1:2] * a[1] + x[:, :1] * a[2])
    return u + 0.01 * size * rng.standard_normal(u.shape)


def _face_load(case, seed):
    """Nodal loads (nodes, 3) on the far x face: a uniform traction of 1e6 Pa in +x, split evenly over
    the four nodes of each face, and a tenth of it at random in y and z."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    share = np.zeros((nz + 1, ny + 1))
    for k in (0, 1):
        for j in (0, 1):
            share[k:nz + k, j:ny + j] += 0.25e6 / 16.0 ** 2
    f = np.zeros((nz + 1, ny + 1, nx + 1, 3))
    f[:, :, nx, 0] = share
    f[:, :, nx, 1:] = 0.1 * share[..., None] * np.random.default_rng(seed + 7).standard_normal((nz + 1, ny + 1, 2))
    return f.reshape(-1, 3)


def _thermal_inputs(case, m, seed):
    """(conductivity per material, specific heat, constraints that hold the x = 0 face at the
    temperature it has, temperature, previous temperature, previous rate by node): a step within a
    run, as a transient or a nonlinear steady analysis makes it."""
    rng = np.random.default_rng(seed + 3)
    nm = len(m.material_density)
    k = 45.0 * np.exp(0.3 * rng.standard_normal(nm))
    cond = np.concatenate([k[:, None] * np.array([1.0, 0.9, 1.1]), k[:, None] * np.array([0.05, -0.03, 0.02])], axis=1)
    heat = np.full(nm, 460.0)
    t = 20.0 + 5.0 * rng.standard_normal(m.num_nodes)
    face = np.nonzero(m.node_list[:, 0] == 0.0)[0] + 1
    mpc = (np.arange(len(face) + 1), face, np.ones(len(face)), t[face - 1])
    return cond, heat, mpc, t, t - rng.uniform(0.0, 1.0, m.num_nodes), rng.standard_normal(m.num_nodes)


def _scatter(g, by_node):
    """A nodal field (nodes, components) in global DOF numbering."""
    v = np.zeros(g.n)
    v[g.n_dof_index[:, :by_node.shape[1]] - 1] = by_node
    return v


def _by_node(g, v):
    return v[g.n_dof_index[:, :g.dims.dof_per_node] - 1]


def _assemble_mesh(case, seed):
    if case["element"] == "shell":
        rng = np.random.default_rng(seed)
        return M.plate_shell(nx=case["nx"], ny=case["ny"], lx=case["nx"] * 0.25, ly=case["ny"] * 0.25,
                             t=rng.uniform(0.04, 0.06))
    m = _block(case, seed)
    if case["element"] == "brickIM":
        m.element_type = np.full(m.num_els, 81, np.int32)
    return m


def _assemble_state(case, m, seed):
    """(displacement by node or None, internal DOF or None, the vector the matrix is applied to)."""
    rng = np.random.default_rng(seed + 1)
    dpn = m.dof_per_node
    x = rng.standard_normal((m.num_nodes, dpn))
    if not case["displaced"]:
        return None, None, x
    u = _smooth_disp(m, seed + 2, 1e-2)
    if dpn == 6:
        u = np.concatenate([u, 1e-2 * rng.standard_normal((m.num_nodes, 3))], axis=1)
    n_int = {"brick": 0, "brickIM": 9, "shell": 8}[case["element"]] * m.num_els
    return u, 1e-4 * rng.standard_normal(n_int) if n_int else None, x


# ---- the measured calls -------------------------------------------------------------------------


def prepare(case, seed):
    s = dict(case)
    kind = case["kind"]
    if kind == "skyline":
        s["g"] = AstroGPU(M.shell_beam())  # the handle; the skyline is the caller's own
        s["lt"], s["range"], s["rhs"], _ = _skyline(case, seed)
    elif kind == "assemble":
        m = _assemble_mesh(case, seed)
        g = s["g"] = AstroGPU(m)
        u, iu, x = _assemble_state(case, m, seed)
        s["state"] = M.make_state(g.n, disp=None if u is None else _scatter(g, u), internal_disp=iu)
        s["x"] = _scatter(g, x)
    elif kind == "solve":
        g = s["g"] = AstroGPU(_block(case, seed))
        g.getElasticSolnLoad(1, export=False)
        g.scaleElasticMPC()
        s["b"] = _scatter(g, _face_load(case, seed))
    elif kind == "panels":
        m = s["m"] = M.panel_batch(case["count"], n_range=(8, 36), n_dvars=DVARS)
        rng = np.random.default_rng(seed)  # the batch's meshes are fixed, its thicknesses and pressures drawn
        m.layup_thickness = m.panel_thickness = rng.uniform(0.03, 0.1, case["count"])
        m.panel_pressure = rng.uniform(1.0e2, 1.0e4, case["count"])
        s["g"] = AstroGPU(m)
    elif kind == "newmark":
        m = M.plate_shell(nx=case["n"], ny=case["n"], lx=10.0, ly=10.0, clamp="ss")
        g = s["g"] = AstroGPU(m)
        g.set_option(OPT_SHELL_MEAN_ROT_TERM, 1)
        s["patterns"], s["amplitudes"] = M.config5_cases(m, g.n_dof_index, case["steps"], 1e-5,
                                                         num_random=case["cases"] - 1, seed0=seed % 100003)
        rng = np.random.default_rng(seed)  # a smooth initial deflection of every case
        w = np.sin(np.pi * m.node_list[:, 0] / 10.0) * np.sin(np.pi * (m.node_list[:, 1] + 5.0) / 10.0)
        s["disp"] = np.zeros((case["cases"], g.n))
        s["disp"][:, g.n_dof_index[:, 2] - 1] = 1e-6 * rng.uniform(-1.0, 1.0, (case["cases"], 1)) * w
    elif kind == "gradient":
        m = _grouped_block(case, seed)
        g = s["g"] = AstroGPU(m)
        s["state"] = M.make_state(g.n, disp=_scatter(g, _smooth_disp(m, seed + 2, 1e-4)))
        g.getElasticSolnLoad(1, state=s["state"], export=False)
        g.scaleElasticMPC()
        s["dldu"] = _scatter(g, _face_load(case, seed))
    else:
        m = _block(case, seed)
        g = s["g"] = AstroGPU(m)
        cond, heat, mpc, t, tp, td = _thermal_inputs(case, m, seed)
        g.thermal_setup(thermal_props(cond, heat, mpc))
        order = np.argsort(g.current_rank)  # the temperatures in rank order
        s["rank"] = g.current_rank - 1
        s["temp"] = t[order]
        s["state"] = thermal_state(t[order], tp[order], td[order], dynamic=int(case["dynamic"]), gamma=0.5, del_t=5.0)
    return s


def run(s):
    g, kind = s["g"], s["kind"]
    if kind == "skyline":
        fac = g.getSparseLDLFact(s["lt"], s["range"])
        return {"factor": fac, "soln": g.solveSparseLDLFact(s["rhs"], fac, s["range"])}
    if kind == "assemble":
        load, iload, mat, cols, imat = g.getElasticSolnLoad(1, state=s["state"], export=s["export"])
        out = {"load": _by_node(g, load)}
        if g.int_vec_size:
            out["int_load"] = iload[:g.int_vec_size]
        if s["export"]:
            out.update(mat=mat, cols=cols)
            if g.int_vec_size:
                out["int_mat"] = imat
        else:
            out["Kx"] = _by_node(g, g.apply_operator(s["x"]))
        return out
    if kind == "solve":
        if s["method"] != "fp64":
            g.assemble_fp32()
        u, _ = g.solve_static(s["b"], method=METHODS[s["method"]], rtol=RTOL)
        return {"disp": _by_node(g, u)}
    if kind == "panels":
        u, du, _ = panels.solve_batch(g, s["m"], DVARS)
        return {"disp": u, "ddisp_dd": du}
    if kind == "newmark":
        u, v, a, _, _ = g.newmark_cases(1e-5, s["patterns"], s["amplitudes"], disp=s["disp"])
        return {"disp": u, "vel": v, "acc": a}
    if kind == "gradient":
        dldd, lam, _, _ = g.getTotaldLdD(s["dldu"], state=s["state"], method=SOLVER_FGMRES_LEARNED, rtol=RTOL)
        return {"dldd": dldd, "adjoint": _by_node(g, lam)}
    load = g.thermal_heat_gen(2.0e4)
    load, _, _ = g.getThermalSolnLoad(1, s["state"], load, export=False)
    g.scaleThermalMPC()
    load = g.getThermalConstraintLoad(s["temp"], load)
    dt, _ = g.thermal_solve(load, rtol=RTOL)
    return {"load": load[s["rank"]], "dtemp": dt[s["rank"]]}


def work(case):
    kind = case["kind"]
    if kind == "skyline":
        n, wd = case["long"] * case["width"] * case["depth"], case["width"] * case["depth"] + case["depth"] + 1
        lt = case["comps"] * n * (wd + 1.0)
        return {"bytes": 8.0 * (3 * lt + 2 * case["comps"] * n), "flops": case["comps"] * n * (1.0 * wd * wd + 4 * wd)}
    if kind == "panels":
        # panels of 22 x 22 elements on average: band of (22 + 2) nodes, 6 DOF
        n, bw = case["count"] * 23.0 ** 2 * 6, 24.0 * 6
        return {"bytes": 8.0 * n * (2 * bw + 2 * (DVARS + 1)), "flops": n * bw * (bw + 4.0 * (DVARS + 1))}
    if kind == "newmark":
        n, bw = (case["n"] + 1.0) ** 2 * 6, (case["n"] + 2.0) * 6
        return {"bytes": 8.0 * n * (bw + case["steps"] * (bw + 8.0 * case["cases"])),
                "flops": n * bw * (bw + 4.0 * case["steps"] * case["cases"])}
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    e = float(nx * ny * nz)
    if kind == "assemble" and case["element"] == "shell":
        nodes, blocks = (nx + 1.0) * (ny + 1), (3.0 * nx + 1) * (3 * ny + 1)
        return {"bytes": nodes * (24 + 48 * 3) + e * (256 * 8 + 64 + 200) + blocks * 36 * 8,
                "flops": e * 4 * (32 * 9 * 9 * 2 + 32 * 33 * 9 + 32 * 33 * 9)}
    nodes, blocks = (nx + 1.0) * (ny + 1) * (nz + 1), (3.0 * nx + 1) * (3 * ny + 1) * (3 * nz + 1)
    if kind == "assemble":
        im = case["element"] == "brickIM"
        pairs = 66.0 if im else 36.0
        return {"bytes": nodes * (24 + 24 * 3) + e * (104 + (297 * 8 if im else 0)) + blocks * 9 * 8,
                "flops": e * 8 * (2 * pairs * (54 if case["displaced"] else 27) + 400)}
    if kind == "solve":
        # a solver cannot do without reading the matrix once per decade of the tolerance
        return {"bytes": blocks * (72 + 4) * 12 + nodes * 48, "flops": blocks * 18 * 12 + e * 8000}
    if kind == "gradient":
        return {"bytes": blocks * (72 + 4) * 12 + nodes * 48 + e * 104 * 2, "flops": blocks * 18 * 12 + e * 8 * 2000}
    return {"bytes": nodes * 80 + e * 130 + blocks * (12 * 12 + 8), "flops": blocks * 24 + e * 8 * 36 * 6}


# ---- the same results in 64 bits, by torch -------------------------------------------------------


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _t(a):
    return torch.as_tensor(np.ascontiguousarray(a), device=_device())


def _gauss(m):
    """Per Gauss point of every brick: shape functions (8,), gradients (E, 8, 3), w det J (E,)."""
    el = _t(m.element_list.astype(np.int64) - 1)
    X = _t(m.node_list)[el]
    X = X - X[:, :1]
    sgn = torch.tensor([[-1, -1, -1], [1, -1, -1], [1, 1, -1], [-1, 1, -1], [-1, -1, 1], [1, -1, 1], [1, 1, 1],
                        [-1, 1, 1]], dtype=torch.float64, device=X.device)
    for g in range(8):
        s = torch.tensor([1.0 if g >> k & 1 else -1.0 for k in range(3)], dtype=torch.float64, device=X.device) / 3 ** 0.5
        f = 1.0 + sgn * s
        N = 0.125 * f.prod(1)
        dN = 0.125 * torch.stack([sgn[:, 0] * f[:, 1] * f[:, 2], sgn[:, 1] * f[:, 0] * f[:, 2],
                                  sgn[:, 2] * f[:, 0] * f[:, 1]], dim=1)
        J = torch.einsum("eai,aj->eij", X, dN)
        yield N, torch.einsum("aj,eji->eai", dN, torch.linalg.inv(J)), torch.linalg.det(J)


def _lame(m):
    """Isotropic Lame constants per element."""
    mat = m.material_elastic[m.section_mat_id[m.element_section - 1] - 1]
    E, nu = _t(mat[:, 0].copy()), _t(mat[:, 3].copy())
    return E * nu / ((1 + nu) * (1 - 2 * nu)), E / (2 * (1 + nu))


def _sum_nodes(m, fe):
    """Element-node values (E, 8, c) summed at the nodes."""
    el = _t(m.element_list.astype(np.int64) - 1).reshape(-1)
    return torch.zeros((m.num_nodes, fe.shape[2]), dtype=torch.float64, device=fe.device).index_add_(
        0, el, fe.reshape(-1, fe.shape[2]))


def _hyper(m, u, x):
    """The Green-Lagrange residual at u and the tangent there applied to x, by node."""
    el = _t(m.element_list.astype(np.int64) - 1)
    lam, mu = _lame(m)
    eye = torch.eye(3, dtype=torch.float64, device=lam.device)
    ue = torch.zeros((m.num_els, 8, 3), dtype=torch.float64, device=lam.device) if u is None else _t(u)[el]
    xe = _t(x)[el]
    R = K = 0.0

    def stress(e):
        return lam[:, None, None] * torch.einsum("eii->e", e)[:, None, None] * eye + 2 * mu[:, None, None] * e

    for _, G, wd in _gauss(m):
        H, dF = torch.einsum("eai,eaj->eij", ue, G), torch.einsum("eai,eaj->eij", xe, G)
        F = H + eye
        S = stress(0.5 * (H + H.mT + H.mT @ H))
        dE = F.mT @ dF
        P, dP = F @ S, dF @ S + F @ stress(0.5 * (dE + dE.mT))
        R = R + torch.einsum("e,eij,eaj->eai", wd, P, G)
        K = K + torch.einsum("e,eij,eaj->eai", wd, dP, G)
    return _sum_nodes(m, R), _sum_nodes(m, K)


def _sparse(m, ke, comps):
    """Element matrices (E, 8, c, 8, c) as a sparse matrix over the DOF comps * node + component."""
    el = _t(m.element_list.astype(np.int64) - 1)
    dof = (comps * el[:, :, None] + torch.arange(comps, device=el.device)).reshape(m.num_els, -1)
    k = dof.shape[1]
    ix = torch.stack([dof[:, :, None].expand(-1, k, k).reshape(-1), dof[:, None, :].expand(-1, k, k).reshape(-1)])
    n = comps * m.num_nodes
    return torch.sparse_coo_tensor(ix, ke.reshape(-1), (n, n)).coalesce()


def _cg(A, pen, b):
    """(A + diag(pen)) x = b by Jacobi-preconditioned conjugate gradients, restarted on the true
    residual until it no longer falls."""
    ix, val = A.indices(), A.values()
    d = torch.zeros_like(b).index_add_(0, ix[0], torch.where(ix[0] == ix[1], val, torch.zeros_like(val))) + pen
    A = A.to_sparse_csr()
    x, best = torch.zeros_like(b), None
    for _ in range(4):
        r = b - (A @ x + pen * x)
        nrm = float(r.norm())
        if best is not None and nrm > 0.1 * best:
            break
        best = nrm
        z = r / d
        p, dx, rz, tgt = z.clone(), torch.zeros_like(b), r @ z, 1e-14 * nrm
        for it in range(20000):
            q = A @ p + pen * p
            a = rz / (p @ q)
            dx += a * p
            r = r - a * q
            z = r / d
            rz, old = r @ z, rz
            p = z + (rz / old) * p
            if it % 25 == 24 and float(r.norm()) < tgt:
                break
        x = x + dx
    return x


def _exact_solve(case, seed):
    m = _block(case, seed)
    lam, mu = _lame(m)
    ke = torch.zeros((m.num_els, 8, 3, 8, 3), dtype=torch.float64, device=lam.device)
    for _, G, wd in _gauss(m):
        T = torch.einsum("e,eai,ebj->eaibj", wd, G, G)
        ke += lam[:, None, None, None, None] * T + mu[:, None, None, None, None] * T.transpose(2, 4)
        D = torch.einsum("eaibi->eab", T) * mu[:, None, None]
        for i in range(3):
            ke[:, :, i, :, i] += D
    K = _sparse(m, ke, 3)
    pen = torch.zeros(m.num_nodes, 3, dtype=torch.float64, device=lam.device)
    pen[_t(m.node_list[:, 0] == 0.0)] = (100.0 * K.values().abs().max()) ** 2
    return {"disp": _cg(K, pen.reshape(-1), _t(_face_load(case, seed)).reshape(-1)).reshape(-1, 3)}


def _exact_thermal(case, seed):
    m = _block(case, seed)
    cond, heat, mpc, t, tp, td = _thermal_inputs(case, m, seed)
    c = _t(cond)[_t(m.section_mat_id[m.element_section - 1].astype(np.int64) - 1)]
    k = c[:, torch.tensor([[0, 3, 4], [3, 1, 5], [4, 5, 2]], device=c.device)]
    cap = _t((m.material_density * heat)[m.section_mat_id[m.element_section - 1] - 1])
    gamma, dt = 0.5, 5.0
    ke = torch.zeros((m.num_els, 8, 8), dtype=torch.float64, device=c.device)
    me, q = torch.zeros_like(ke), torch.zeros((m.num_els, 8, 1), dtype=torch.float64, device=c.device)
    for N, G, wd in _gauss(m):
        ke += torch.einsum("e,eai,eij,ebj->eab", wd, G, k, G)
        me += torch.einsum("e,a,b->eab", wd * cap, N, N)
        q += 2.0e4 * torch.einsum("e,a->ea", wd, N)[:, :, None]
    el = _t(m.element_list.astype(np.int64) - 1)
    temp = _t(t)
    R = torch.einsum("eab,eb->ea", ke, temp[el])
    if case["dynamic"]:
        rate = ((temp - _t(tp)) / dt - (1 - gamma) * _t(td)) / gamma
        R = R + torch.einsum("eab,eb->ea", me, rate[el])
        ke = ke + me / (gamma * dt)
    load = (_sum_nodes(m, q) - _sum_nodes(m, R[:, :, None]))[:, 0]
    K = _sparse(m, ke, 1)
    face = _t(mpc[1].astype(np.int64) - 1)
    pen = torch.zeros(m.num_nodes, dtype=torch.float64, device=c.device)
    pen[face] = (100.0 * K.values().abs().max()) ** 2
    load[face] += pen[face] * (_t(mpc[3]) - temp[face])
    return {"load": load, "dtemp": _cg(K, pen, load)}


def exact(case, seed):
    kind = case["kind"]
    if kind == "skyline":
        _, rng_all, rhs, blocks = _skyline(case, seed)
        n = len(rhs) // case["comps"]
        row = np.diff(rng_all[: n + 1])
        fac, soln = [], []
        for c, (diag, lo, hi, val) in enumerate(blocks):
            A = np.diag(diag)
            A[lo, hi] = A[hi, lo] = -val
            C = np.linalg.cholesky(A)
            d = np.diag(C)
            L = C / d
            np.fill_diagonal(L, d * d)
            fac += [L[i, i + 1 - row[i]:i + 1] for i in range(n)]
            soln.append(np.linalg.solve(A, rhs[c * n:(c + 1) * n]))
        return {"factor": np.concatenate(fac), "soln": np.concatenate(soln)}
    if kind == "assemble" and case["element"] == "brick":
        m = _assemble_mesh(case, seed)
        u, _, x = _assemble_state(case, m, seed)
        R, Kx = _hyper(m, u, x)
        if u is None:
            R = torch.zeros_like(R)
        return {"load": -R, "Kx": None if case["export"] else Kx}
    if kind == "solve":
        return _exact_solve(case, seed)
    if kind == "thermal":
        return _exact_thermal(case, seed)
    return None  # shells, brickIM, time stepping, gradients: no short plain form
