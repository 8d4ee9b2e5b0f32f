"""The damage CG that keeps a voxel cell on the SMs, over the ways it splits a grid (needs a B200).

One block or many, bricks cut off by the grid on every side, free faces, a depth of one layer, cells
too large for it (which take the launch that streams its vectors): each must end at the solution of
the bound-constrained system that the damage operators define.  Tolerance: the linear solves stop at
1e-12 max(||r0||, 1) on a recursive residual; a factor of two above it.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

CELLS = [((2, 2, 1), (True, True, True)), ((5, 4, 3), (False, False, False)), ((16, 14, 2), (True, True, True)),
         ((17, 15, 11), (True, False, True)), ((7, 61, 9), (True, True, False)), ((33, 29, 40), (False, True, True)),
         ((64, 48, 50), (True, True, True)), ((100, 90, 70), (True, True, True))]


@pytest.mark.parametrize("shape,periodic", CELLS)
@pytest.mark.parametrize("history", [True, False])
def test_box_solve(shape, periodic, history):
    from phast_b200 import solid3d as s3
    rng = np.random.default_rng(3)
    h = (1.0 / shape[0], 1.1 / shape[0], 0.9 / shape[0])
    slot = rng.integers(0, 2, int(np.prod(shape)))
    phases = [s3.PhaseMaterial("mi_matrix", "isotropic", 0.5, "spectral", 3000.0, 0.35),
              s3.PhaseMaterial("fibre", "isotropic", 0.2, "spectral", 70000.0, 0.3)]
    load = s3.LoadCase("zz", 2, (0.01,), (), (0, 1, 3, 4, 5))
    op = s3.PeriodicVoxelPhaseFieldOperator.from_slots(s3.VoxelGrid(shape, h, periodic=periodic), slot, phases,
                                                       2 * h[0], 1e-6, load, pinned_node=0)
    H = torch.as_tensor(rng.uniform(0.0, 0.3, (op.n_elements, 8)) * 0.5 / (2 * h[0]), device="cuda") if history \
        else None
    lower = torch.as_tensor(rng.uniform(0.0, 0.4, op.n_red), device="cuda")
    res = s3.solve_h8_scalar_box_kkt(op.damage_system(H), lower_bound=lower, upper_bound=1.0, initial=lower,
                                     linear_tolerance=1e-12, kkt_tolerance=1e-8)
    assert res.satisfies_kkt
    d, s = res.solution, op.damage_scale
    rhs = op.damage_rhs(H, scale=s) if history else torch.zeros_like(d)
    g = op.damage_action(d, H, scale=s) - rhs
    r0 = float((op.damage_action(lower, H, scale=s) - rhs).norm())
    free = (d > lower) & (d < 1.0)
    assert float(g[free].norm()) <= 2e-12 * max(r0, 1.0)
    assert bool((d >= lower).all()) and bool((d <= 1.0).all())
    assert float(g[d <= lower].clamp(max=0.0).norm()) <= 1e-8
