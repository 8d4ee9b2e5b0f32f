"""The work a user of this package has it do, as cases that can be timed and checked.

A case is a dict of plain values.  ``listed()`` names the usual ones, ``draw(rng)`` gives one
more of the same ranges, ``prepare(case, seed)`` makes what a program holds before the call,
``run(state)`` makes the call through the public entry points, ``work(case)`` counts the bytes
and operations one call cannot do without, and ``exact(case, seed)`` computes the same outputs in
64 bits with plain PyTorch.

Kinds:

* ``action``    one elastic action of a voxel cell (``op.mech_action`` with damage): the operator
                every 3D solve is made of, and what a user with a Krylov method of their own calls;
* ``pcg``       one constrained mechanics solve by Jacobi PCG in FP64 (``solve_constrained``);
* ``gmg``       the same by FP32 multigrid PCG under FP64 refinement (``solve_constrained_form``);
* ``kkt``       one bound-constrained damage solve of a voxel cell (``solve_h8_scalar_box_kkt``);
* ``increment`` one staggered load increment of a voxel cell (``StaggeredSolver.advance``);
* ``batch``     one staggered load increment of several cells at once (``BatchStaggeredSolver``);
* ``explicit``  explicit time steps of a structured 2D mesh, a damage solve in each
                (``StaggeredSolver.step_full``);
* ``static``    one quasi-static equilibrium solve of a structured 2D mesh (``QuasiStaticSolver``);
* ``grad``      one differentiable damage solve of a structured 2D mesh, forward and backward;
* ``t3``        force, driving energy and damage solve of an unstructured triangle mesh.

The solves run to tight tolerances (1e-10 to 1e-13, about those of the parity tests), where the answer
is a property of the system and not of the stopping point.
"""
import math

import numpy as np
import torch

import phast_b200 as pb
from phast_b200 import solid3d as s3
from phast_b200.solid3d import batch as s3b

KAPPA = 1e-6
E_CELL, NU_CELL, GC_CELL, PORE = 3000.0, 0.35, 0.5, 1e-6  # the pore cell of the benchmark
MIXED = dict(precond="gmg", mixed=True, smooth_degree=1, coarse_degree=6, inner_rtol=1e-5)
MECH_RTOL = 1e-12  # Jacobi PCG in FP64
MIXED_RTOL = 1e-13  # FP64 residual of the refined form: a refinement that ends just below 1e-12 is 1e-9 off


def listed():
    return [
        # the smallest call: one action of the smallest cell of the tests' order of size, where launch and host time count
        {"name": "action_16_f64", "kind": "action", "nx": 16, "ny": 16, "nz": 16, "dtype": "f64", "free_z": False},
        # a cell with odd edges and free faces in z, in the precision of the reference
        {"name": "action_odd_f64", "kind": "action", "nx": 97, "ny": 83, "nz": 110, "dtype": "f64", "free_z": True},
        # the roofline cell of the benchmark: the working set is beyond L2
        {"name": "action_192_f32", "kind": "action", "nx": 192, "ny": 192, "nz": 192, "dtype": "f32", "free_z": False},
        # the reference's own solver at the size of the PF-CZM and closure cells
        {"name": "pcg_32", "kind": "pcg", "nx": 32, "ny": 32, "nz": 32},
        # the benchmark cell's mechanics solve in the chosen form
        {"name": "gmg_64", "kind": "gmg", "nx": 64, "ny": 64, "nz": 64},
        # the benchmark cell's damage solve
        {"name": "kkt_64", "kind": "kkt", "nx": 64, "ny": 64, "nz": 64},
        # a whole load increment of the benchmark cell
        {"name": "increment_64", "kind": "increment", "n": 64, "strain": 0.006},
        # a whole load increment of several particle cells at once
        {"name": "batch_4", "kind": "batch", "sizes": "32,40,48,64", "strain": 0.004},
        # explicit crack branching, the mesh of the 2D dynamic configuration
        {"name": "explicit_400x160", "kind": "explicit", "nx": 400, "ny": 160, "steps": 4, "dtype": "f64"},
        # equilibrium of the notched plate, the mesh of the 2D quasi-static configuration
        {"name": "static_200x200", "kind": "static", "nx": 200, "ny": 200},
        # gradient of a damage solve, the mesh of the 2D gradient configuration
        {"name": "grad_256x256", "kind": "grad", "nx": 256, "ny": 256},
        # an unstructured triangle mesh of the size of the reference's Kalthoff-Winkler example
        {"name": "t3_160x110", "kind": "t3", "nx": 160, "ny": 110},
    ]


def _between(rng, lo, hi):
    """A whole number of [lo, hi], spread over its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["action", "action", "action", "pcg", "gmg", "kkt", "increment", "batch", "explicit", "static",
                       "grad", "t3"])
    if kind == "action":
        n = [_between(rng, 9, 190) for _ in range(3)]
        return {"kind": kind, "nx": n[0], "ny": n[1], "nz": n[2], "dtype": rng.choice(["f32", "f64"]),
                "free_z": rng.random() < 0.3}
    if kind == "pcg":
        return {"kind": kind, "nx": _between(rng, 10, 36), "ny": _between(rng, 10, 36), "nz": _between(rng, 10, 36)}
    if kind == "gmg":
        return {"kind": kind, "nx": 4 * rng.randint(6, 16), "ny": 4 * rng.randint(6, 16), "nz": 4 * rng.randint(6, 16)}
    if kind == "kkt":
        return {"kind": kind, "nx": _between(rng, 16, 64), "ny": _between(rng, 16, 64), "nz": _between(rng, 16, 64)}
    if kind == "increment":
        return {"kind": kind, "n": 4 * rng.randint(8, 16), "strain": round(rng.uniform(0.002, 0.006), 5)}
    if kind == "batch":
        sizes = sorted(4 * rng.randint(8, 14) for _ in range(rng.randint(2, 4)))
        return {"kind": kind, "sizes": ",".join(str(v) for v in sizes), "strain": round(rng.uniform(0.002, 0.004), 5)}
    if kind == "explicit":
        return {"kind": kind, "nx": _between(rng, 40, 400), "ny": _between(rng, 30, 160), "steps": rng.randint(1, 4),
                "dtype": "f64"}
    if kind == "static":
        return {"kind": kind, "nx": _between(rng, 30, 200), "ny": _between(rng, 30, 200)}
    if kind == "grad":
        return {"kind": kind, "nx": _between(rng, 30, 256), "ny": _between(rng, 30, 256)}
    return {"kind": kind, "nx": _between(rng, 20, 160), "ny": _between(rng, 20, 110)}


# ----------------------------------------------------------------------------
# inputs
# ----------------------------------------------------------------------------

def _waves(rng, coords, modes=6, kmax=3):
    """A smooth field with values around one: a few random plane waves over the unit box."""
    out = torch.zeros(coords[0].shape if len(coords) == 1 else torch.broadcast_shapes(*[c.shape for c in coords]),
                      dtype=torch.float64, device=coords[0].device)
    for _ in range(modes):
        phase = float(rng.uniform(0, 2 * math.pi))
        arg = phase
        for c in coords:
            arg = arg + (2 * math.pi * int(rng.integers(-kmax, kmax + 1))) * c
        out += torch.cos(arg)
    return out / math.sqrt(modes / 2.0)


def _cell_axes(case, device="cuda"):
    """Node coordinates over the unit box, broadcastable to (rz, ry, rx)."""
    rz = case["nz"] + (1 if case.get("free_z") else 0)
    ax = lambda n, m: torch.arange(m, dtype=torch.float64, device=device) / n  # noqa: E731
    return (ax(case["nx"], case["nx"])[None, None, :], ax(case["ny"], case["ny"])[None, :, None],
            ax(case["nz"], rz)[:, None, None])


def _cell_slots(case):
    """Voxel material slots (nz, ny, nx): matrix 0 and a central spherical pore 1."""
    c = [(np.arange(case[k]) + 0.5) / case[k] - 0.5 for k in ("nx", "ny", "nz")]
    r2 = c[0][None, None, :] ** 2 + c[1][None, :, None] ** 2 + c[2][:, None, None] ** 2
    return (r2 < 0.2 ** 2).astype(np.uint8)


def _cell_operator(case):
    h = 1.0 / case["nz"]
    grid = s3.VoxelGrid((case["nx"], case["ny"], case["nz"]), (h, h, h),
                        periodic=(True, True, not case.get("free_z", False)))
    phases = [s3.PhaseMaterial("mi_matrix", "isotropic", GC_CELL, "spectral", E_CELL, NU_CELL),
              s3.PhaseMaterial("pore", "isotropic", GC_CELL, "spectral", E_CELL * PORE, NU_CELL)]
    load = s3.LoadCase.ramp("zz", 2, 0.02, 50)
    return s3.PeriodicVoxelPhaseFieldOperator.from_slots(grid, _cell_slots(case), phases, 2 * h, KAPPA, load,
                                                         pinned_node=0)


def _cell_damage(case, rng):
    """Nodal damage between 0 and 0.8, as a cell on its way to a crack has it."""
    w = _waves(rng, _cell_axes(case)).reshape(-1)
    return (0.4 + 0.25 * w).clamp(0.0, 0.8)


def _cell_field(case, rng):
    """A mechanics vector [u~, E]: fluctuations of a tenth of the macro strain, rough at the voxel scale too."""
    axes = _cell_axes(case)
    h = 1.0 / case["nz"]
    u = torch.stack([2e-4 * _waves(rng, axes) for _ in range(3)], -1).reshape(-1)
    gen = torch.Generator(device="cuda").manual_seed(int(rng.integers(1 << 31)))
    u += 1e-3 * h * (torch.rand(u.shape, generator=gen, dtype=torch.float64, device="cuda") - 0.5)
    macro = torch.as_tensor(2e-3 * rng.standard_normal(6), device="cuda")
    return torch.cat([u, macro])


def _cell_history(case, rng):
    """Driving-energy history (E, 8) that damages the cell to about one half in places."""
    ax = [(torch.arange(case[k], dtype=torch.float64, device="cuda") + 0.5) / case[k] for k in ("nx", "ny", "nz")]
    w = _waves(rng, (ax[0][None, None, :], ax[1][None, :, None], ax[2][:, None, None])).reshape(-1, 1)
    gen = torch.Generator(device="cuda").manual_seed(int(rng.integers(1 << 31)))
    q = torch.rand(w.shape[0], 8, generator=gen, dtype=torch.float64, device="cuda")
    gc_ell = GC_CELL * case["nz"] / 2.0
    return 0.15 * gc_ell * torch.exp(1.2 * w) * (0.9 + 0.2 * q)


def _plate(case, split, ratio, material):
    sm = pb.structured_q4_mesh(1.0, ratio, case["nx"], case["ny"])
    mesh = pb.FEMMesh.from_tensors(sm.nodes, sm.quads, element_type="Q4", device="cuda")
    return sm, mesh, pb.Material(energy_split=split, **material)


def _plate_axes(case):
    ax = lambda n: torch.arange(n + 1, dtype=torch.float64, device="cuda") / n  # noqa: E731
    return ax(case["nx"])[None, :], ax(case["ny"])[:, None]


def _plate_elem(case, rng):
    ax = lambda n: (torch.arange(n, dtype=torch.float64, device="cuda") + 0.5) / n  # noqa: E731
    return _waves(rng, (ax(case["nx"])[None, :], ax(case["ny"])[:, None])).reshape(-1)


def _plate_damage(case, rng, notch=True):
    x, y = _plate_axes(case)
    d = (0.25 + 0.15 * _waves(rng, (x, y))).clamp(0.0, 0.6)
    if notch:  # a crack from the left edge to the middle with the profile of the phase field
        s = torch.where(x < 0.5, (y - 0.5).abs(), torch.sqrt((x - 0.5) ** 2 + (y - 0.5) ** 2))
        d = torch.maximum(d, torch.exp(-s / 0.02))
    return d.reshape(-1).contiguous()


STATIC_MAT = dict(E=210000.0, nu=0.3, Gc=2.7, l0=0.01, eta_residual=1e-8, rho=7.8e-9)
DYN_MAT = dict(E=32000.0, nu=0.2, Gc=3e-3, l0=0.01, eta_residual=1e-8, rho=2.45e-9)


def _triangles(case, rng):
    """A jittered triangulation of a plate: nodes (N, 2) and triangles (E, 3) on the host."""
    nx, ny = case["nx"], case["ny"]
    x, y = np.meshgrid(np.linspace(0.0, 1.0, nx + 1), np.linspace(0.0, ny / nx, ny + 1))
    h = 1.0 / nx
    inner = np.zeros(x.shape, dtype=bool)
    inner[1:-1, 1:-1] = True
    x = x + np.where(inner, 0.25 * h * (rng.random(x.shape) - 0.5), 0.0)
    y = y + np.where(inner, 0.25 * h * (rng.random(x.shape) - 0.5), 0.0)
    n0 = (np.arange(ny)[:, None] * (nx + 1) + np.arange(nx)[None, :]).reshape(-1)
    n1, n2, n3 = n0 + 1, n0 + nx + 2, n0 + nx + 1
    flip = (np.arange(n0.size) + np.arange(n0.size) // nx) % 2 == 0
    a = np.where(flip[:, None], np.stack([n0, n1, n2], 1), np.stack([n0, n1, n3], 1))
    b = np.where(flip[:, None], np.stack([n0, n2, n3], 1), np.stack([n1, n2, n3], 1))
    return np.stack([x.reshape(-1), y.reshape(-1)], 1), np.stack([a, b], 1).reshape(-1, 3)


def prepare(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng([int(seed), 1])
    if kind == "action":
        op = _cell_operator(case)
        dt = torch.float32 if case["dtype"] == "f32" else torch.float64
        d = _cell_damage(case, rng).to(dt)
        return {"kind": kind, "op": op, "x": _cell_field(case, rng).to(dt), "d": d}
    if kind in ("pcg", "gmg"):
        op = _cell_operator(case)
        d = _cell_damage(case, rng)
        values = op.mech_fixed_values(float(rng.uniform(0.5e-3, 4e-3)))
        import ctypes
        return {"kind": kind, "op": op, "d": d, "mask": op.mech_fixed_mask(), "values": values,
                "diag": op.mech_diagonal(d=d) if kind == "pcg" else None, "lmax": (ctypes.c_double * 3)(),
                "form": s3.MechForm(**MIXED)}
    if kind == "kkt":
        op = _cell_operator(case)
        H = _cell_history(case, rng)
        lower = (0.1 + 0.1 * _waves(rng, _cell_axes(case))).clamp(0.0, 0.5).reshape(-1).contiguous()
        return {"kind": kind, "system": op.damage_system(H), "lower": lower}
    if kind == "increment":
        n = case["n"]
        radius = 0.2 + 0.02 * float(rng.uniform(-1.0, 1.0))
        model = s3.sphere_pore_model((n, n, n), radius, E=E_CELL, nu=NU_CELL, Gc=GC_CELL, ell_voxels=2.0,
                                     pore_stiffness=PORE)
        cfg = s3.SolverConfig(device="cuda", kappa=KAPPA, pcg_rtol_mech=MIXED_RTOL, damage_linear_tol=1e-12)
        op = s3.PeriodicVoxelPhaseFieldOperator(model, s3.LoadCase.ramp("zz", 2, 0.02, 50), cfg, pinned_node=0)
        solver = s3.StaggeredSolver(op, form=s3.MechForm(**MIXED))
        return {"kind": kind, "solver": solver, "state": solver.initial_state(), "target": case["strain"]}
    if kind == "batch":
        load = s3b.batch_load()
        ops = []
        for k, n in enumerate(int(v) for v in case["sizes"].split(",")):
            cell = s3b.particle_cells(seed=int(seed) * 16 + k, n_cells=1, sizes=(n,))[0]
            ops.append(s3b.build_operator(cell, load))
        cfg = s3.SolverConfig(device="cuda", kappa=ops[0].kappa, pcg_rtol_mech=MIXED_RTOL, damage_linear_tol=1e-12)
        solver = s3b.BatchStaggeredSolver(s3b.PackedCellBatch(ops), load, cfg, form=s3.MechForm(**MIXED))
        return {"kind": kind, "solver": solver, "state": solver.initial_state(), "target": case["strain"]}
    if kind == "explicit":
        sm, mesh, mat = _plate(case, "spectral", case["ny"] / case["nx"], DYN_MAT)
        bcs = pb.BoundaryConditions(mesh.n_nodes, device="cuda")
        notch = (torch.arange(case["nx"] // 2 + 1) + (case["ny"] // 2) * (case["nx"] + 1))
        bcs.add_pf_dirichlet(notch, 1.0)
        dt = torch.float32 if case["dtype"] == "f32" else torch.float64
        solver = pb.StaggeredSolver(mesh, mat, bcs, pb.SolverConfig(
            solver_type="explicit", dt_safety=0.5, damage_every=1, damage_tol=1e-10, bounds_method="projected_cg",
            use_multigrid=False, dtype=dt))
        x, y = _plate_axes(case)
        # a wave train on its way through the plate, and the edge traction that drives it
        u = torch.stack([2e-5 * _waves(rng, (x, y), kmax=8) for _ in range(2)], -1).reshape(-1, 2)
        v = torch.stack([500.0 * _waves(rng, (x, y), kmax=8) for _ in range(2)], -1).reshape(-1, 2)
        f = torch.zeros(case["ny"] + 1, case["nx"] + 1, 2, dtype=torch.float64, device="cuda")
        f[0, :, 1], f[-1, :, 1] = -1.0 / case["nx"], 1.0 / case["nx"]
        solver.f_ext = f.reshape(-1, 2).to(dt)
        d = _plate_damage(case, rng, notch=False) * 0.5
        d[notch.to("cuda")] = 1.0
        H = 0.05 * DYN_MAT["Gc"] / DYN_MAT["l0"] * torch.exp(_plate_elem(case, rng))[:, None].expand(-1, 4)
        return {"kind": kind, "solver": solver, "steps": case["steps"], "u": u.to(dt), "v": v.to(dt),
                "a": torch.zeros_like(u, dtype=dt), "d": d, "H": H.to(dt).contiguous()}
    if kind == "static":
        sm, mesh, mat = _plate(case, "isotropic", 1.0, STATIC_MAT)
        fem = pb.FEMOperators(mesh, mat)
        bcs = pb.BoundaryConditions(mesh.n_nodes, device="cuda")
        bcs.fix(sm.node_sets["bottom"], 0)
        bcs.fix(sm.node_sets["bottom"], 1)
        bcs.add(sm.node_sets["top"], 1, 1.0)
        bcs.load_factor = float(rng.uniform(1e-3, 5e-3))
        mask, vals = bcs.get_masks_and_values()
        solver = pb.QuasiStaticSolver(fem, tol=1e-10, cg_tol=1e-10, backend="cg", cg_max_iter=20000)
        f = torch.zeros(mesh.n_nodes, 2, dtype=torch.float64, device="cuda")
        return {"kind": kind, "solver": solver, "d": 0.9 * _plate_damage(case, rng), "f": f, "mask": mask,
                "vals": vals}
    if kind == "grad":
        sm, mesh, mat = _plate(case, "isotropic", 1.0, STATIC_MAT)
        fem = pb.FEMOperators(mesh, mat)
        solver = pb.PhaseFieldDamageSolver(fem, tol=1e-12, max_iter=20000, bounds_method="projected_cg")
        gc_l0 = STATIC_MAT["Gc"] / STATIC_MAT["l0"]
        H = (0.1 * gc_l0 * torch.exp(1.5 * _plate_elem(case, rng)))[:, None].expand(-1, 4).contiguous()
        gc = STATIC_MAT["Gc"] * torch.exp(0.2 * _plate_elem(case, rng))
        d_prev = _plate_damage(case, rng)
        w = _waves(rng, _plate_axes(case)).reshape(-1).contiguous()
        return {"kind": kind, "solver": solver, "H": H.requires_grad_(True), "gc": gc.requires_grad_(True),
                "d_prev": d_prev.requires_grad_(True), "w": w}
    nodes, tris = _triangles(case, rng)
    mesh = pb.FEMMesh.from_tensors(torch.as_tensor(nodes), torch.as_tensor(tris), element_type="T3", device="cuda")
    fem = pb.FEMOperators(mesh, pb.Material(energy_split="amor", **STATIC_MAT))
    solver = pb.PhaseFieldDamageSolver(fem, tol=1e-12, max_iter=20000, bounds_method="projected_cg")
    n = torch.as_tensor(nodes, device="cuda")
    c = n[torch.as_tensor(tris, device="cuda")].mean(1)
    gc_l0 = STATIC_MAT["Gc"] / STATIC_MAT["l0"]
    H = 0.1 * gc_l0 * torch.exp(1.5 * _waves(rng, (c[:, 0], c[:, 1])))
    d_prev = (0.25 + 0.15 * _waves(rng, (n[:, 0], n[:, 1]))).clamp(0.0, 0.6)
    u = torch.stack([1e-3 * _waves(rng, (n[:, 0], n[:, 1])) for _ in range(2)], -1).contiguous()
    return {"kind": kind, "fem": fem, "solver": solver, "H": H, "d_prev": d_prev, "u": u}


def run(state):
    kind = state["kind"]
    if kind == "action":
        return state["op"].mech_action(state["x"], d=state["d"])
    if kind == "pcg":
        op = state["op"]
        return s3.solve_constrained(op.mech_operator(d=state["d"]), diag=state["diag"], fixed_mask=state["mask"],
                                    fixed_values=state["values"], rtol=MECH_RTOL, maxiter=20000)[0]
    if kind == "gmg":
        return s3.solve_constrained_form(state["op"], state["form"], fixed_mask=state["mask"],
                                         fixed_values=state["values"], d=state["d"], rtol=MIXED_RTOL, maxiter=20000,
                                         lmax_cache=state["lmax"])[0]
    if kind == "kkt":
        return s3.solve_h8_scalar_box_kkt(state["system"], lower_bound=state["lower"], upper_bound=1.0,
                                          initial=state["lower"], linear_tolerance=1e-12).solution
    if kind == "increment":
        new, record = state["solver"].advance(state["state"], state["target"], increment=1)
        return {"x": new.x, "d": new.d, "H": new.H, "stress": new.macro_stress, "elastic": record.elastic,
                "fracture": record.fracture}
    if kind == "batch":
        new, records = state["solver"].advance(state["state"], state["target"])
        return {"x": new.x, "d": new.d, "H": new.H, "stress": new.macro_stress}
    if kind == "explicit":
        s = state["solver"]
        s.u, s.v, s.a = state["u"].clone(), state["v"].clone(), state["a"].clone()
        s.d, s.H_elem = state["d"].clone(), state["H"].clone()
        for _ in range(state["steps"]):
            s.step_full()
        return {"u": s.u, "v": s.v, "d": s.d, "H": s.H_elem}
    if kind == "static":
        return state["solver"].solve(state["d"], state["f"], state["mask"], state["vals"])[0]
    if kind == "grad":
        H, gc, d_prev = state["H"], state["gc"], state["d_prev"]
        d = state["solver"].solve(H, d_prev, Gc_field=gc)
        g_h, g_gc, g_prev = torch.autograd.grad(d, (H, gc, d_prev), grad_outputs=state["w"])
        return {"d": d.detach(), "grad_H": g_h, "grad_Gc": g_gc, "grad_d_prev": g_prev}
    force = state["fem"].internal_force(state["u"], state["d_prev"])
    psi = state["fem"].compute_psi_plus(state["u"])
    return {"force": force, "psi": psi, "d": state["solver"].solve(state["H"], state["d_prev"])}


# ----------------------------------------------------------------------------
# the work of one call: inputs read once, outputs written once, and the operations
# ----------------------------------------------------------------------------

# per voxel and elastic action 884 operations (an FMA counted as two), per damage action 300;
# per Q4 node and action 600 (elastic) or 250 (damage); per triangle 120
def work(case):
    kind = case["kind"]
    if kind in ("action", "pcg", "gmg", "kkt"):
        e = case["nx"] * case["ny"] * case["nz"]
        n = case["nx"] * case["ny"] * (case["nz"] + (1 if case.get("free_z") else 0))
        if kind == "action":
            word = 4 if case["dtype"] == "f32" else 8
            return {"bytes": 7 * n * word + e, "flops": 884 * e}
        if kind == "kkt":  # about forty CG steps
            return {"bytes": 8 * (3 * n + 8 * e) + e, "flops": 40 * 300 * e}
        steps = 12 * max(case["nx"], case["ny"], case["nz"]) if kind == "pcg" else 60
        return {"bytes": 8 * 8 * n + e, "flops": steps * 884 * e}
    if kind == "increment":  # a few passes of a mechanics and a damage solve
        n = case["n"] ** 3
        return {"bytes": 8 * 25 * n, "flops": 4 * (60 * 884 + 40 * 300) * n}
    if kind == "batch":
        n = sum(int(v) ** 3 for v in case["sizes"].split(","))
        return {"bytes": 8 * 25 * n, "flops": 4 * (60 * 884 + 40 * 300) * n}
    n = (case["nx"] + 1) * (case["ny"] + 1)
    if kind == "explicit":
        return {"bytes": 8 * (14 * n + 8 * n), "flops": case["steps"] * (600 + 30 * 250) * n}
    if kind == "static":
        return {"bytes": 8 * 8 * n, "flops": 8 * max(case["nx"], case["ny"]) * 600 * n}
    if kind == "grad":
        return {"bytes": 8 * 16 * n, "flops": 80 * 250 * n}
    return {"bytes": 8 * (8 * n + 4 * 2 * n) + 2 * 12 * n, "flops": 40 * 2 * 120 * n}


# ----------------------------------------------------------------------------
# the same answers in 64 bits, by plain gather, contraction and scatter
# ----------------------------------------------------------------------------

class _Grid:
    """Elements of a uniform grid: corner nodes (E, A), shape values N (Q, A), gradients dN (Q, A, dim), weight w."""

    def __init__(self, shape, periodic, h):
        dim = len(shape)
        red = [n if p else n + 1 for n, p in zip(shape, periodic)]
        idx = torch.meshgrid(*[torch.arange(n, device="cuda") for n in reversed(shape)], indexing="ij")
        idx = [i.reshape(-1) for i in reversed(idx)]  # per axis, first axis fastest
        corners = [[(c >> a) & 1 for a in range(dim)] for c in range(2 ** dim)]
        cols = []
        for c in corners:
            node, stride = 0, 1
            for a in range(dim):
                i = idx[a] + c[a]
                node = node + stride * (i % shape[a] if periodic[a] else i)
                stride *= red[a]
            cols.append(node)
        self.conn = torch.stack(cols, 1)
        self.n = math.prod(red)
        g = 1.0 / math.sqrt(3.0)
        N, dN = np.ones((2 ** dim, 2 ** dim)), np.ones((2 ** dim, 2 ** dim, dim))
        for q, cq in enumerate(corners):
            for a, ca in enumerate(corners):
                f = [0.5 * (1 + (2 * ca[k] - 1) * (2 * cq[k] - 1) * g) for k in range(dim)]
                N[q, a] = math.prod(f)
                for k in range(dim):
                    dN[q, a, k] = (2 * ca[k] - 1) / h[k] * math.prod(f[m] for m in range(dim) if m != k)
        self.N = torch.as_tensor(N, device="cuda")
        self.dN = torch.as_tensor(dN, device="cuda")
        self.w = math.prod(h) / 2 ** dim

    def parts(self):
        step = 1 << 19
        return [slice(s, s + step) for s in range(0, self.conn.shape[0], step)]


def _elastic(grid, lam, mu, d, kappa, x, macro=None):
    """(A(d) x, stress resultant): isotropic stress degraded by g at the Gauss points; lam, mu per element."""
    dim = grid.dN.shape[-1]
    u = x.reshape(grid.n, dim)
    f, total = torch.zeros_like(u), torch.zeros(dim, dim, dtype=torch.float64, device="cuda")
    eye = torch.eye(dim, dtype=torch.float64, device="cuda")
    for p in grid.parts():
        c = grid.conn[p]
        grad = torch.einsum("eai,qaj->eqij", u[c], grid.dN)
        eps = 0.5 * (grad + grad.transpose(-1, -2))
        if macro is not None:
            eps = eps + macro
        g = (1.0 - kappa) * (1.0 - d[c] @ grid.N.T) ** 2 + kappa
        tr = eps.diagonal(dim1=-2, dim2=-1).sum(-1)
        s = 2.0 * mu[p].reshape(-1, 1, 1, 1) * eps + (lam[p].reshape(-1, 1) * tr)[..., None, None] * eye
        s = s * (g * grid.w)[..., None, None]
        f.index_add_(0, c.reshape(-1), torch.einsum("eqij,qaj->eai", s, grid.dN).reshape(-1, dim))
        total += s.sum((0, 1))
    return f, total


def _damage_matrix(grid, gc_over_l, gc_l, H, x):
    """(Gc l K + M(Gc / l + 2 H)) x, coefficients per element, H per Gauss point."""
    y = torch.zeros_like(x)
    for p in grid.parts():
        c = grid.conn[p]
        xe = x[c]
        r = (gc_over_l[p].reshape(-1, 1) + 2.0 * H[p]) * (xe @ grid.N.T)
        k = torch.einsum("ea,qaj,qbj->eb", xe, grid.dN, grid.dN) * gc_l[p].reshape(-1, 1)
        y.index_add_(0, c.reshape(-1), ((r @ grid.N + k) * grid.w).reshape(-1))
    return y


def _damage_load(grid, H):
    b = torch.zeros(grid.n, dtype=torch.float64, device="cuda")
    for p in grid.parts():
        b.index_add_(0, grid.conn[p].reshape(-1), ((2.0 * H[p] * grid.w) @ grid.N).reshape(-1))
    return b


def _damage_diag(grid, gc_over_l, gc_l, H):
    y = torch.zeros(grid.n, dtype=torch.float64, device="cuda")
    kk = grid.dN.square().sum((0, 2))
    for p in grid.parts():
        v = (gc_over_l[p].reshape(-1, 1) + 2.0 * H[p]) @ grid.N.square() + gc_l[p].reshape(-1, 1) * kk
        y.index_add_(0, grid.conn[p].reshape(-1), (v * grid.w).reshape(-1))
    return y


def _cg(action, b, diag, free, x, rtol, most=20000):
    """Jacobi CG on the free entries from x (zero elsewhere in the update) until ||r|| <= rtol ||b_free||."""
    inv = torch.where(free, 1.0 / diag, 0.0)
    r = torch.where(free, b - action(x), 0.0)
    stop = rtol * float(torch.linalg.vector_norm(torch.where(free, b, 0.0)).clamp_min(1e-300))
    if float(torch.linalg.vector_norm(r)) <= stop:
        return x
    z = inv * r
    p, rz = z.clone(), torch.dot(r, z)
    for k in range(most):
        ap = torch.where(free, action(p), 0.0)
        a = rz / torch.dot(p, ap)
        x = x + a * p
        r = r - a * ap
        z = inv * r
        new = torch.dot(r, z)
        if k % 20 == 19 and float(torch.linalg.vector_norm(r)) <= stop:
            break
        p = z + (new / rz) * p
        rz = new
    return x


def _bounded(action, b, diag, lower, fixed, x):
    """The solution of A x = b within [lower, 1], entries `fixed` held: an active-set loop of CG solves."""
    x = torch.minimum(torch.maximum(x, lower), torch.ones_like(x))
    at_low, at_up = torch.zeros_like(fixed), torch.zeros_like(fixed)
    for _ in range(60):
        free = ~(at_low | at_up | fixed)
        x = torch.where(at_low & ~fixed, lower, torch.where(at_up & ~fixed, torch.ones_like(x), x))
        shift = torch.where(free, 0.0, x)
        y = _cg(action, b - action(shift), diag, free, torch.where(free, x, 0.0), 1e-13)
        x = torch.where(free, y, x)
        grad = action(x) - b
        low = (free & (x < lower)) | (at_low & (grad > 0.0))
        up = (free & (x > 1.0)) | (at_up & (grad < 0.0))
        if bool((low == at_low).all()) and bool((up == at_up).all()):
            break
        at_low, at_up = low & ~fixed, up & ~fixed
    return torch.minimum(torch.maximum(x, lower), torch.ones_like(x)), at_low, at_up


def _lame(E, nu):
    return E * nu / ((1 + nu) * (1 - 2 * nu)), E / (2 * (1 + nu))


def _exact_cell(case):
    h = 1.0 / case["nz"]
    grid = _Grid((case["nx"], case["ny"], case["nz"]), (True, True, not case.get("free_z", False)), (h, h, h))
    lam, mu = _lame(E_CELL, NU_CELL)
    factor = torch.where(torch.as_tensor(_cell_slots(case).reshape(-1).astype(np.int64), device="cuda") == 1, PORE,
                         1.0).double()
    return grid, lam * factor, mu * factor


def _voigt(t):
    return torch.stack([t[0, 0], t[1, 1], t[2, 2], t[1, 2], t[0, 2], t[0, 1]])


def _macro(E):
    """Symmetric strain of the Voigt vector (engineering shear)."""
    a, b, c, yz, xz, xy = (E[k] for k in range(6))
    return torch.stack([torch.stack([a, 0.5 * xy, 0.5 * xz]), torch.stack([0.5 * xy, b, 0.5 * yz]),
                        torch.stack([0.5 * xz, 0.5 * yz, c])])


def _exact_mech(case, rng, solve):
    grid, lam, mu = _exact_cell(case)
    m = 3 * grid.n
    # the inputs as prepare() rounds them, then in 64 bits
    dt = torch.float32 if case.get("dtype") == "f32" else torch.float64
    d = _cell_damage(case, rng).to(dt).double()

    def action(x):
        f, s = _elastic(grid, lam, mu, d, KAPPA, x[:m], _macro(x[m:]))
        return torch.cat([f.reshape(-1), _voigt(s)])

    if not solve:
        return action(_cell_field(case, rng).to(dt).double())
    strain = float(rng.uniform(0.5e-3, 4e-3))
    free = torch.ones(m + 6, dtype=torch.bool, device="cuda")
    free[:3] = False
    free[m:] = False  # the ramp fixes every macro component
    x = torch.zeros(m + 6, dtype=torch.float64, device="cuda")
    x[m + 2] = strain
    # Jacobi diagonal: every Gauss point adds w g (mu |dN|^2 + (lam + mu) dN_c^2)
    diag = torch.zeros(grid.n, 3, dtype=torch.float64, device="cuda")
    for p in grid.parts():
        g = ((1.0 - KAPPA) * (1.0 - d[grid.conn[p]] @ grid.N.T) ** 2 + KAPPA) * grid.w
        sq = grid.dN.square()
        k = torch.einsum("eq,qac->eac", g, sq) * (lam[p] + mu[p]).reshape(-1, 1, 1) + \
            torch.einsum("eq,qa->ea", g, sq.sum(-1))[..., None] * mu[p].reshape(-1, 1, 1)
        diag.index_add_(0, grid.conn[p].reshape(-1), k.reshape(-1, 3))
    diag = torch.cat([diag.reshape(-1), torch.ones(6, dtype=torch.float64, device="cuda")])
    y = _cg(action, -action(x), diag, free, torch.zeros_like(x), 1e-13)
    return torch.where(free, y, x)


def _split_2d(lam, mu, eps, g):
    """Spectral-split plane-strain stress with degraded tensile part, and its tensile energy."""
    exx, eyy, exy = eps[..., 0, 0], eps[..., 1, 1], eps[..., 0, 1]
    tr, half = exx + eyy, 0.5 * (exx - eyy)
    r = torch.sqrt(half ** 2 + exy ** 2 + 1e-12)
    e1, e2 = 0.5 * tr + r, 0.5 * tr - r
    n = torch.stack([torch.stack([half + r, exy], -1), torch.stack([exy, r - half], -1)], -2) / (2.0 * r)[..., None, None]
    eye = torch.eye(2, dtype=torch.float64, device="cuda")
    # the off-diagonal of the second projector is minus the first's
    pos = e1.clamp_min(0.0)[..., None, None] * n + e2.clamp_min(0.0)[..., None, None] * (eye - n)
    trp = tr.clamp_min(0.0)
    sp = lam * trp[..., None, None] * eye + 2 * mu * pos
    sm = lam * (tr - trp)[..., None, None] * eye + 2 * mu * (eps - pos)
    psi = 0.5 * lam * trp ** 2 + mu * (e1.clamp_min(0.0) ** 2 + e2.clamp_min(0.0) ** 2)
    return g[..., None, None] * sp + sm, psi


#: Corner order of _Grid's 2D elements and Gauss points (x fastest) is the package's own for Gauss points.
def _exact_explicit(case, seed):
    s = prepare(case, seed)
    solver = s["solver"]
    lam, mu = _lame(DYN_MAT["E"], DYN_MAT["nu"])
    eta = DYN_MAT["eta_residual"]
    h = 1.0 / case["nx"]
    grid = _Grid((case["nx"], case["ny"]), (False, False), (h, h))
    mass = torch.zeros(grid.n, dtype=torch.float64, device="cuda")
    mass.index_add_(0, grid.conn.reshape(-1), torch.full((grid.conn.numel(),), h * h / 4, dtype=torch.float64,
                                                         device="cuda"))
    inv = 1.0 / (DYN_MAT["rho"] * mass + 1e-30)
    dt = float(solver.dt)
    u, v, a, d, H = (s[k].double() for k in ("u", "v", "a", "d", "H"))
    fe = solver.f_ext.double()
    fixed = torch.zeros(grid.n, dtype=torch.bool, device="cuda")
    row = (case["ny"] // 2) * (case["nx"] + 1)
    fixed[row:row + case["nx"] // 2 + 1] = True
    ones = torch.ones(grid.conn.shape[0], dtype=torch.float64, device="cuda")
    gco, gcl = ones * (DYN_MAT["Gc"] / DYN_MAT["l0"]), ones * (DYN_MAT["Gc"] * DYN_MAT["l0"])
    for _ in range(case["steps"]):
        un = u + dt * v + 0.5 * dt * dt * a
        grad = torch.einsum("eai,qaj->eqij", un[grid.conn], grid.dN)
        eps = 0.5 * (grad + grad.transpose(-1, -2))
        g = (1 - d[grid.conn] @ grid.N.T) ** 2 * (1 - eta) + eta
        sig, psi = _split_2d(lam, mu, eps, g)
        f = torch.zeros_like(u)
        f.index_add_(0, grid.conn.reshape(-1), (torch.einsum("eqij,qaj->eai", sig, grid.dN) * grid.w).reshape(-1, 2))
        an = (fe - f) * inv[:, None]
        v = v + 0.5 * dt * (a + an)
        u, a, H = un, an, torch.maximum(H, psi)
        b, diag = _damage_load(grid, H), _damage_diag(grid, gco, gcl, H)
        lower = torch.where(fixed, torch.ones_like(d), d)
        d = _bounded(lambda x: _damage_matrix(grid, gco, gcl, H, x), b, diag, lower, fixed, lower)[0]
    return {"u": u, "v": v, "d": d, "H": H}


def _exact_static(case, seed):
    s = prepare(case, seed)
    lam, mu = _lame(STATIC_MAT["E"], STATIC_MAT["nu"])
    grid = _Grid((case["nx"], case["ny"]), (False, False), (1.0 / case["nx"], 1.0 / case["ny"]))
    ones = torch.ones(grid.conn.shape[0], dtype=torch.float64, device="cuda")
    d, eta = s["d"], STATIC_MAT["eta_residual"]
    action = lambda x: _elastic(grid, lam * ones, mu * ones, d, eta, x)[0].reshape(-1)  # noqa: E731
    held = s["mask"].reshape(-1).bool()
    x = torch.where(held, s["vals"].reshape(-1).double(), 0.0)
    diag = torch.zeros(grid.n, 2, dtype=torch.float64, device="cuda")
    g = ((1.0 - eta) * (1.0 - d[grid.conn] @ grid.N.T) ** 2 + eta) * grid.w
    sq = grid.dN.square()
    k = (lam + mu) * torch.einsum("eq,qac->eac", g, sq) + mu * torch.einsum("eq,qa->ea", g, sq.sum(-1))[..., None]
    diag.index_add_(0, grid.conn.reshape(-1), k.reshape(-1, 2))
    y = _cg(action, -action(x), diag.reshape(-1), ~held, torch.zeros_like(x), 1e-13)
    return torch.where(held, x, y).reshape(-1, 2)


def _exact_grad(case, seed):
    s = prepare(case, seed)
    H, gc, d_prev, w = s["H"].detach(), s["gc"].detach(), s["d_prev"].detach(), s["w"]
    l0 = STATIC_MAT["l0"]
    grid = _Grid((case["nx"], case["ny"]), (False, False), (1.0 / case["nx"], 1.0 / case["ny"]))
    gco, gcl = gc / l0, gc * l0
    action = lambda x: _damage_matrix(grid, gco, gcl, H, x)  # noqa: E731
    diag = _damage_diag(grid, gco, gcl, H)
    none = torch.zeros(grid.n, dtype=torch.bool, device="cuda")
    d, low, up = _bounded(action, _damage_load(grid, H), diag, d_prev, none, d_prev)
    # the adjoint on the free nodes, and the sensitivities of K, M and the load; a node whose two
    # bounds meet at one counts as held from above
    up = up | (d >= 1.0 - 1e-12)
    low = low & ~up
    free = ~(low | up)
    lam = torch.where(free, _cg(action, w, diag, free, torch.zeros_like(w), 1e-13), 0.0)
    le, de = lam[grid.conn], d[grid.conn]
    lk = torch.einsum("ea,qaj,qbj,eb->e", le, grid.dN, grid.dN, de) * grid.w
    lq, dq = le @ grid.N.T, de @ grid.N.T
    g_gc = -(l0 * lk + (lq * dq).sum(-1) * grid.w / l0)
    return {"d": d, "grad_H": 2.0 * grid.w * lq * (1.0 - dq), "grad_Gc": g_gc,
            "grad_d_prev": torch.where(low, w - action(lam), 0.0)}


def _exact_t3(case, seed):
    nodes, tris = _triangles(case, np.random.default_rng([int(seed), 1]))
    s = prepare(case, seed)
    p, c = torch.as_tensor(nodes, device="cuda"), torch.as_tensor(tris, device="cuda")
    e1, e2 = p[c[:, 1]] - p[c[:, 0]], p[c[:, 2]] - p[c[:, 0]]
    det = e1[:, 0] * e2[:, 1] - e1[:, 1] * e2[:, 0]
    area = 0.5 * det.abs()
    # gradients of the barycentric coordinates: the rows of the inverse of [e1 e2]
    g1 = torch.stack([e2[:, 1], -e2[:, 0]], -1) / det[:, None]
    g2 = torch.stack([-e1[:, 1], e1[:, 0]], -1) / det[:, None]
    dN = torch.stack([-(g1 + g2), g1, g2], 1)
    u, d0, H = s["u"], s["d_prev"], s["H"]
    lam, mu = _lame(STATIC_MAT["E"], STATIC_MAT["nu"])
    bulk = STATIC_MAT["E"] / (3 * (1 - 2 * STATIC_MAT["nu"]))
    eta, l0, Gc = STATIC_MAT["eta_residual"], STATIC_MAT["l0"], STATIC_MAT["Gc"]
    grad = torch.einsum("eai,eaj->eij", u[c], dN)
    eps = 0.5 * (grad + grad.transpose(-1, -2))
    tr = eps.diagonal(dim1=-2, dim2=-1).sum(-1)
    trp = tr.clamp_min(0.0)
    eye = torch.eye(2, dtype=torch.float64, device="cuda")
    dev = eps - (tr / 3.0)[:, None, None] * eye
    psi = 0.5 * bulk * trp ** 2 + mu * (dev.square().sum((1, 2)) + (tr / 3.0) ** 2)
    g = (1 - d0[c].mean(1)) ** 2 * (1 - eta) + eta
    sig = g[:, None, None] * (bulk * trp[:, None, None] * eye + 2 * mu * dev) + (bulk * (tr - trp))[:, None, None] * eye
    force = torch.zeros_like(u)
    force.index_add_(0, c.reshape(-1), (torch.einsum("eij,eaj->eai", sig, dN) * area[:, None, None]).reshape(-1, 2))
    r = (2.0 * H + Gc / l0) * area / 12.0
    add = lambda v: torch.zeros_like(d0).index_add_(0, c.reshape(-1), v.reshape(-1))  # noqa: E731

    def action(x):
        xe = x[c]
        k = torch.einsum("eaj,ej->ea", dN, torch.einsum("ea,eaj->ej", xe, dN)) * (Gc * l0 * area)[:, None]
        return add(k + r[:, None] * (xe + xe.sum(1, keepdim=True)))

    diag = add(dN.square().sum(-1) * (Gc * l0 * area)[:, None] + 2.0 * r[:, None].expand(-1, 3))
    load = add((2.0 * H * area / 3.0)[:, None].expand(-1, 3).contiguous())
    none = torch.zeros_like(d0, dtype=torch.bool)
    return {"force": force, "psi": psi, "d": _bounded(action, load, diag, d0, none, d0)[0]}


def exact(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng([int(seed), 1])
    if kind == "action":
        return _exact_mech(case, rng, solve=False)
    if kind in ("pcg", "gmg"):
        return _exact_mech(case, rng, solve=True)
    if kind == "kkt":
        H = _cell_history(case, rng)
        lower = (0.1 + 0.1 * _waves(rng, _cell_axes(case))).clamp(0.0, 0.5).reshape(-1)
        grid, lam, _ = _exact_cell(case)
        ones, ell = torch.ones_like(lam), 2.0 / case["nz"]
        # the scalar system with its history weight 2 (1 - kappa) H
        gco, gcl, Hk = ones * (GC_CELL / ell), ones * (GC_CELL * ell), (1.0 - KAPPA) * H
        b, diag = _damage_load(grid, Hk), _damage_diag(grid, gco, gcl, Hk)
        none = torch.zeros(grid.n, dtype=torch.bool, device="cuda")
        return _bounded(lambda x: _damage_matrix(grid, gco, gcl, Hk, x), b, diag, lower, none, lower)[0]
    if kind in ("increment", "batch"):
        return None  # the whole staggered loop with plain CG takes minutes
    if kind == "explicit":
        return _exact_explicit(case, seed)
    if kind == "static":
        return _exact_static(case, seed)
    if kind == "grad":
        return _exact_grad(case, seed)
    return _exact_t3(case, seed)
