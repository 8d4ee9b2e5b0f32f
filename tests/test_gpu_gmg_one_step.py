"""The V-cycle with one smoothing step, whose residual, smoothing and sums are epilogues of the action (needs a B200).

Level grids that do not fill a brick or split into sub-bricks (the coarsest level's one-launch solve), free faces, a free macro strain, two and three levels, FP64 and
mixed precision: each solve must end at the solution of the system that the elastic action defines.
Tolerance: the stopping test is rtol ||b|| on the FP64 residual (mixed) or on a recursive residual that
drifts from it by rounding only; a factor of two above it.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

CELLS = [((8, 8, 8), (True, True, True)), ((20, 12, 8), (False, True, True)), ((36, 28, 16), (True, True, True)),
         ((16, 60, 24), (True, True, False)), ((48, 44, 48), (True, True, True)), ((64, 64, 60), (True, False, True)),
         ((80, 72, 80), (True, True, True))]
RTOL = 1e-8


@pytest.mark.parametrize("shape,periodic", CELLS)
@pytest.mark.parametrize("mixed", [True, False])
@pytest.mark.parametrize("levels,free_strain", [(3, False), (2, True)])
def test_one_step_cycle(shape, periodic, mixed, levels, free_strain):
    from phast_b200 import solid3d as s3
    rng = np.random.default_rng(17)
    h = (1.0 / shape[0], 1.1 / shape[0], 0.9 / shape[0])
    slot = rng.integers(0, 2, int(np.prod(shape)))
    phases = [s3.PhaseMaterial("mi_matrix", "isotropic", 0.5, "spectral", 3000.0, 0.35),
              s3.PhaseMaterial("fibre", "isotropic", 0.2, "spectral", 9000.0, 0.3)]
    load = (s3.LoadCase("zz", 2, (0.01,), (0, 1), (3, 4, 5)) if free_strain
            else s3.LoadCase("zz", 2, (0.01,), (), (0, 1, 3, 4, 5)))
    op = s3.PeriodicVoxelPhaseFieldOperator.from_slots(s3.VoxelGrid(shape, h, periodic=periodic), slot, phases,
                                                       2 * h[0], 1e-6, load, pinned_node=0)
    d = torch.as_tensor(rng.uniform(0.0, 0.6, op.n_red), device="cuda")
    mask = op.mech_fixed_mask()
    if not all(periodic):  # no rigid rotations of a cell with free faces: hold a random tenth of the nodes
        held = torch.as_tensor(rng.random(op.n_red) < 0.1, device="cuda")
        mask[:3 * op.n_red] |= held.repeat_interleave(3)
    values = torch.where(mask, torch.as_tensor(rng.uniform(-1e-3, 1e-3, op.n_mech), device="cuda"), 0.0)
    form = s3.MechForm("gmg", mixed=mixed, levels=levels, smooth_degree=1, coarse_degree=6)
    x, info = s3.solve_constrained_form(op, form, fixed_mask=mask, fixed_values=values, d=d, rtol=RTOL, maxiter=2000)[:2]
    act = op.mech_operator(d=d)
    assert info.converged and bool((x[mask] == values[mask]).all())
    assert float(act(x)[~mask].norm()) <= 2 * RTOL * float(act(values)[~mask].norm())


@pytest.mark.parametrize("sizes,n", [((32,), 1), ((32, 36, 48), 5), ((96,), 3)])
def test_one_step_cycle_batched(sizes, n):
    """One cell, cells of several sizes in one launch, and cells too many for bricks of one layer."""
    from test_gpu_batch_packed import _setup
    from phast_b200 import solid3d as s3
    cells, load, ops, B = _setup(sizes=sizes, n=n, brick=(16, 8, 8))
    rng = np.random.default_rng(23)
    ds = [torch.as_tensor(rng.uniform(0.0, 0.6, op.n_red), device="cuda") for op in ops]
    values = [op.mech_fixed_values(0.004 + 0.001 * c) for c, op in enumerate(ops)]
    form = s3.MechForm("gmg", mixed=True, smooth_degree=1, coarse_degree=6, inner_rtol=1e-5)
    x, status, its, conv, bn, rn = B.mech_solve(B.pack_nodes(ds), B.pack_mech(values), rtol=RTOL, mixed=True,
                                                form=form, reuse_lmax=False)
    assert status == 0 and conv.all()
    for c, op in enumerate(ops):
        act, free, xc = op.mech_operator(d=ds[c]), ~op.mech_fixed_mask(), B.mech_view(x, c)
        assert float(act(xc)[free].norm()) <= 2 * RTOL * float(act(values[c])[free].norm())
