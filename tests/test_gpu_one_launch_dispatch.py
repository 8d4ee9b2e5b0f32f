"""Which solves take one launch, and that the others launch nothing beside their own kernels (needs a B200).

Every solve falls back silently when its one-launch form refuses it.  Here each is run with those
forms switched off (PHASTB_PERSISTENT_PCG=0, read once per process) and as they are by default, and
the launches are counted: a few in all where the iterations are one launch, and exactly as many as
without the form where it does not apply (a free macro strain, a split that is not linear, systems
too large for the SMs).
"""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

SCRIPT = """
import numpy as np, torch
import phast_b200 as pb
from phast_b200 import solid3d as s3, _lib
lib = _lib.load()

def count(name, solve):
    lib.phastb_launch_count_reset()
    solve()
    torch.cuda.synchronize()
    print(name, lib.phastb_launch_count())

def q4(nx, ny, split="isotropic"):
    sm = pb.structured_q4_mesh(1.0, ny / nx, nx, ny)
    mesh = pb.FEMMesh.from_tensors(sm.nodes, sm.quads, element_type="Q4", device="cuda")
    return pb.FEMOperators(mesh, pb.Material(E=210000.0, nu=0.3, Gc=2.7, l0=2.5 / nx, eta_residual=1e-8,
                                             energy_split=split)), sm

rng = np.random.default_rng(1)
for name, nx, ny in (("small", 20, 15), ("fits", 300, 200), ("large", 720, 610)):
    fem, _ = q4(nx, ny)
    s = pb.PhaseFieldDamageSolver(fem, tol=1e-10, max_iter=20000, bounds_method="projected_cg")
    H = torch.as_tensor(fem.material.Gc / fem.material.l0 * rng.uniform(0.0, 0.4, (fem.n_elems, 4)), device="cuda")
    v = torch.as_tensor(rng.uniform(0.0, 0.5, fem.n_nodes), device="cuda")
    count("q4_bounded_" + name, lambda: s.solve(H, v))
    count("q4_linear_" + name, lambda: s.linear_solve(H, v, rtol=1e-10))
for name, nx, ny, split in (("small", 20, 15, "isotropic"), ("fits", 200, 200, "isotropic"),
                            ("tangent", 110, 100, "spectral"), ("large", 400, 380, "isotropic")):
    fem, sm = q4(nx, ny, split)
    bcs = pb.BoundaryConditions(fem.n_nodes, device="cuda")
    bcs.fix(sm.node_sets["bottom"], 0)
    bcs.fix(sm.node_sets["bottom"], 1)
    bcs.add(sm.node_sets["top"], 1, 1e-3)
    mask, vals = bcs.get_masks_and_values()
    s = pb.QuasiStaticSolver(fem, tol=1e-6, cg_tol=1e-8, cg_max_iter=20000, max_iter=2)
    d = torch.as_tensor(rng.uniform(0.0, 0.5, fem.n_nodes), device="cuda")
    u = torch.zeros(fem.n_nodes, 2, dtype=torch.float64, device="cuda")
    count("q4_mech_" + name, lambda: s.solve(d, u, mask, vals))
for name, n in (("small", 12), ("fits", 200), ("large", 300)):
    x, y = np.meshgrid(np.linspace(0, 1, n + 1), np.linspace(0, 1, n + 1))
    n0 = (np.arange(n)[:, None] * (n + 1) + np.arange(n)[None, :]).reshape(-1)
    tris = np.concatenate([np.stack([n0, n0 + 1, n0 + n + 2], 1), np.stack([n0, n0 + n + 2, n0 + n + 1], 1)])
    mesh = pb.FEMMesh.from_tensors(torch.as_tensor(np.stack([x.reshape(-1), y.reshape(-1)], 1)), torch.as_tensor(tris),
                                   element_type="T3", device="cuda")
    mat = pb.Material(E=210000.0, nu=0.3, Gc=2.7, l0=2.5 / n, eta_residual=1e-8, energy_split="amor")
    fem = pb.FEMOperators(mesh, mat)
    s = pb.PhaseFieldDamageSolver(fem, tol=1e-10, max_iter=20000, bounds_method="projected_cg")
    H = torch.as_tensor(mat.Gc / mat.l0 * rng.uniform(0.0, 0.4, fem.n_elems), device="cuda")
    v = torch.as_tensor(rng.uniform(0.0, 0.5, fem.n_nodes), device="cuda")
    count("t3_" + name, lambda: s.solve(H, v))
phases = [s3.PhaseMaterial("mi_matrix", "isotropic", 0.5, "spectral", 3000.0, 0.35),
          s3.PhaseMaterial("fibre", "isotropic", 0.2, "spectral", 9000.0, 0.3)]
for name, n, free in (("small", 8, 0), ("fits", 40, 0), ("free", 8, 1), ("large", 60, 0)):
    load = s3.LoadCase("zz", 2, (0.01,), (0, 1), (3, 4, 5)) if free else s3.LoadCase("zz", 2, (0.01,), (), (0, 1, 3, 4, 5))
    op = s3.PeriodicVoxelPhaseFieldOperator.from_slots(s3.VoxelGrid((n, n, n), (1 / n,) * 3), rng.integers(0, 2, n ** 3),
                                                       phases, 2 / n, 1e-6, load, pinned_node=0)
    d = torch.as_tensor(rng.uniform(0.0, 0.6, op.n_red), device="cuda")
    act, diag = op.mech_operator(d=d), op.mech_diagonal(d=d)
    count("mech_" + name, lambda: s3.solve_constrained(act, diag=diag, fixed_mask=op.mech_fixed_mask(),
                                                       fixed_values=op.mech_fixed_values(0.004), rtol=1e-9))
    H = torch.as_tensor(rng.uniform(0.0, 0.3, (op.n_elements, 8)) * n / 4, device="cuda")
    count("kkt_" + name, lambda: s3.solve_h8_scalar_box_kkt(op.damage_system(H), lower_bound=0.5 * d, upper_bound=1.0,
                                                            initial=0.5 * d, linear_tolerance=1e-12))
    if n % 8 == 0:
        form = s3.MechForm("gmg", mixed=True, smooth_degree=1, coarse_degree=6, inner_rtol=1e-5)
        count("gmg_" + name, lambda: s3.solve_constrained_form(op, form, fixed_mask=op.mech_fixed_mask(),
                                                               fixed_values=op.mech_fixed_values(0.004), d=d,
                                                               rtol=1e-9))
"""


def test_dispatch():
    out = []
    for on in ("1", "0"):
        env = dict(os.environ, PHASTB_PERSISTENT_PCG=on, PYTHONPATH=ROOT)
        p = subprocess.run([sys.executable, "-c", SCRIPT], env=env, cwd=ROOT, capture_output=True, text=True, timeout=500)
        assert p.returncode == 0, p.stderr[-2000:]
        out.append({k: int(v) for k, v in (line.split() for line in p.stdout.split("\n") if line)})
    one, separate = out
    assert one.keys() == separate.keys() and len(one) == 24
    wrong = {}
    for k in one:
        family, form = k.rsplit("_", 1)
        if family == "kkt":
            # a solve per active set, each with a launch or two of its own beside the CG's
            good = 5 * one[k] < separate[k]
        elif family == "gmg":
            good = one[k] < separate[k]  # one launch instead of six on the coarsest level
        elif form in ("large", "free"):
            good = one[k] == separate[k]
        else:
            good = one[k] <= 60 and 2 * one[k] < separate[k]
        if not good:
            wrong[k] = (one[k], separate[k])
    assert not wrong, wrong
