"""The elastic CG that keeps a small cell on the SMs, over the ways it splits a grid (needs a B200).

One block or many, bricks cut off by the grid, free faces, a depth of one layer, both forms of the
moduli and of the degradation, a free macro strain and cells too large for it (both take separate
launches): each must end at the solution of the system that the elastic action defines.  Tolerance:
the solve stops at rtol ||b|| on a recursive residual, which drifts from the true one by rounding
only (1e-15 of the largest residual per step, far below rtol); a factor of two above it.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

CELLS = [((2, 2, 1), (True, True, True)), ((5, 4, 3), (False, True, False)), ((8, 8, 9), (True, True, True)),
         ((15, 8, 11), (True, False, True)), ((9, 31, 7), (True, True, False)), ((33, 17, 21), (False, True, True)),
         ((36, 35, 36), (True, True, True)), ((61, 40, 52), (True, True, True))]
RTOL = 1e-9


@pytest.mark.parametrize("shape,periodic", CELLS)
@pytest.mark.parametrize("variant", ["iso", "aniso", "gauss", "intact", "free_strain"])
def test_mechanics_solve(shape, periodic, variant):
    from phast_b200 import solid3d as s3
    rng = np.random.default_rng(11)
    h = (1.0 / shape[0], 1.1 / shape[0], 0.9 / shape[0])
    slot = rng.integers(0, 2, int(np.prod(shape)))
    fibre = (s3.PhaseMaterial("fibre", "smeared_laminate", 0.2, "spectral", 7000.0, 0.26,
                              layers=((0.6, 9000.0, 0.3), (0.4, 4000.0, 0.2)))
             if variant == "aniso" else s3.PhaseMaterial("fibre", "isotropic", 0.2, "spectral", 9000.0, 0.3))
    phases = [s3.PhaseMaterial("mi_matrix", "isotropic", 0.5, "spectral", 3000.0, 0.35), fibre]
    load = (s3.LoadCase("zz", 2, (0.01,), (0, 1), (3, 4, 5)) if variant == "free_strain"
            else s3.LoadCase("zz", 2, (0.01,), (), (0, 1, 3, 4, 5)))
    op = s3.PeriodicVoxelPhaseFieldOperator.from_slots(s3.VoxelGrid(shape, h, periodic=periodic), slot, phases,
                                                       2 * h[0], 1e-6, load, pinned_node=0)
    d = torch.as_tensor(rng.uniform(0.0, 0.6, op.n_red), device="cuda")
    if variant == "gauss":
        act = op.mech_operator(op.degradation(d))
        diag = op.mech_diagonal(op.degradation(d))
    elif variant == "intact":
        act = op.mech_operator(torch.ones(op.n_elements, 8, dtype=torch.float64, device="cuda"))
        diag = op.mech_diagonal(torch.ones(op.n_elements, 8, dtype=torch.float64, device="cuda"))
    else:
        act, diag = op.mech_operator(d=d), op.mech_diagonal(d=d)
    mask = op.mech_fixed_mask()
    if not all(periodic):  # no rigid rotations of a cell with free faces: hold a random tenth of the nodes
        held = torch.as_tensor(rng.random(op.n_red) < 0.1, device="cuda")
        mask[:3 * op.n_red] |= held.repeat_interleave(3)
    values = torch.where(mask, torch.as_tensor(rng.uniform(-1e-3, 1e-3, op.n_mech), device="cuda"), 0.0)
    x, info = s3.solve_constrained(act, diag=diag, fixed_mask=mask, fixed_values=values, rtol=RTOL, maxiter=4000)
    assert info.converged and bool((x[mask] == values[mask]).all())
    b = act(values)[~mask]
    assert float(act(x)[~mask].norm()) <= 2 * RTOL * float(b.norm())
