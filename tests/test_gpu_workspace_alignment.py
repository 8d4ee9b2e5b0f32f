"""Solver workspaces that start on an 8-byte boundary (needs a B200).

The one-launch solves exchange 16-byte words inside the caller's workspace; a workspace that is
only 8-byte aligned must be served all the same, by the separate launches.  Each solve is run with
both and must end at the same solution, to the accuracy its own stopping test asks for (1e-10 or
1e-12 of the residual: 1e-7 of the solution leaves three digits for the condition of these systems).
"""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def shift(monkeypatch):
    from phast_b200 import _lib
    get = _lib.Workspace.get

    def shifted(self, nbytes):
        p, n = get(self, int(nbytes) + 256)
        return C.c_void_p(p.value + 8), C.c_size_t(n.value - 8)

    monkeypatch.setattr(_lib.Workspace, "get", shifted)


def both(monkeypatch, solve):
    from phast_b200 import _lib
    lib = _lib.load()
    a, counts = [], []
    for k in range(2):
        if k:
            shift(monkeypatch)
        lib.phastb_launch_count_reset()
        a.append(solve())
        counts.append(lib.phastb_launch_count())
    assert float((a[1] - a[0]).norm()) <= 1e-7 * float(a[0].norm())
    return counts


def q4(nx, ny):
    import phast_b200 as pb
    sm = pb.structured_q4_mesh(1.0, ny / nx, nx, ny)
    mesh = pb.FEMMesh.from_tensors(sm.nodes, sm.quads, element_type="Q4", device="cuda")
    fem = pb.FEMOperators(mesh, pb.Material(E=210000.0, nu=0.3, Gc=2.7, l0=2.5 / nx, eta_residual=1e-8,
                                            energy_split="isotropic"))
    return fem, pb.PhaseFieldDamageSolver(fem, tol=1e-10, max_iter=20000, bounds_method="projected_cg")


@pytest.mark.parametrize("kind", ["bounded", "linear"])
def test_q4(monkeypatch, kind):
    rng = np.random.default_rng(1)
    fem, _ = q4(45, 38)
    H = torch.as_tensor(fem.material.Gc / fem.material.l0 * rng.uniform(0.0, 0.4, (fem.n_elems, 4)), device="cuda")
    v = torch.as_tensor(rng.uniform(0.0, 0.5, fem.n_nodes), device="cuda")

    def solve():
        _, s = q4(45, 38)
        if kind == "bounded":
            d = s.solve(H, v)
            assert s.last_converged
            return d
        x = s.linear_solve(H, v, rtol=1e-12)
        assert s.last_linear_info[1] == 0
        return x

    counts = both(monkeypatch, solve)
    assert counts[0] < 10 < counts[1]  # one launch for the iterations, and launches of their own


def test_t3(monkeypatch):
    import phast_b200 as pb
    from test_gpu_t3_persistent import grid
    nodes, tris = grid(40, 30, np.random.default_rng(7))
    mesh = pb.FEMMesh.from_tensors(torch.as_tensor(nodes), torch.as_tensor(tris), element_type="T3", device="cuda")
    mat = pb.Material(E=210000.0, nu=0.3, Gc=2.7, l0=0.05, eta_residual=1e-8, energy_split="amor")
    fem = pb.FEMOperators(mesh, mat)
    rng = np.random.default_rng(2)
    H = torch.as_tensor(mat.Gc / mat.l0 * rng.uniform(0.3, 0.9, fem.n_elems), device="cuda")
    d0 = torch.as_tensor(rng.uniform(0.0, 0.5, fem.n_nodes), device="cuda")

    def solve():
        s = pb.PhaseFieldDamageSolver(fem, tol=1e-10, max_iter=20000, bounds_method="projected_cg")
        d = s.solve(H, d0)
        assert s.last_converged
        return d

    counts = both(monkeypatch, solve)
    assert counts[0] < 10 < counts[1]


@pytest.mark.parametrize("kind", ["jacobi", "gmg", "kkt"])
def test_cell(monkeypatch, kind):
    from phast_b200 import solid3d as s3
    shape, rng = (16, 24, 16), np.random.default_rng(5)
    h = (1.0 / shape[0],) * 3
    phases = [s3.PhaseMaterial("mi_matrix", "isotropic", 0.5, "spectral", 3000.0, 0.35),
              s3.PhaseMaterial("fibre", "isotropic", 0.2, "spectral", 9000.0, 0.3)]
    load = s3.LoadCase("zz", 2, (0.01,), (), (0, 1, 3, 4, 5))
    op = s3.PeriodicVoxelPhaseFieldOperator.from_slots(s3.VoxelGrid(shape, h), rng.integers(0, 2, int(np.prod(shape))),
                                                       phases, 2 * h[0], 1e-6, load, pinned_node=0)
    d = torch.as_tensor(rng.uniform(0.0, 0.6, op.n_red), device="cuda")
    H = torch.as_tensor(rng.uniform(0.0, 0.3, (op.n_elements, 8)) * 0.5 / (2 * h[0]), device="cuda")
    mask, values = op.mech_fixed_mask(), op.mech_fixed_values(0.004)

    def solve():
        if kind == "kkt":
            return s3.solve_h8_scalar_box_kkt(op.damage_system(H), lower_bound=0.5 * d, upper_bound=1.0,
                                              initial=0.5 * d, linear_tolerance=1e-12, kkt_tolerance=1e-8).solution
        if kind == "jacobi":
            x, info = s3.solve_constrained(op.mech_operator(d=d), diag=op.mech_diagonal(d=d), fixed_mask=mask,
                                           fixed_values=values, rtol=1e-12, maxiter=4000)
        else:
            form = s3.MechForm("gmg", mixed=True, smooth_degree=1, coarse_degree=6, inner_rtol=1e-5)
            x, info = s3.solve_constrained_form(op, form, fixed_mask=mask, fixed_values=values, d=d, rtol=1e-12,
                                                maxiter=2000)
        assert info.converged
        return x

    counts = both(monkeypatch, solve)
    if kind == "jacobi":
        assert counts[0] < 20 < counts[1]
