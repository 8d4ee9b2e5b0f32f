"""The elastic march at the edges of its compiled brick shapes (needs a B200).

The action keeps each element column's face data in registers while it marches in z; the shapes
compiled for themselves (16 x 14, 16 x 8, 14 x 7, 8 x 8), one that is not, a grid one node larger
or smaller than a brick, single-layer bricks, a depth that does not divide the grid and free faces
must all give the oracle's action, in both precisions and with the shape the launch picks itself.
Tolerances: those of the other tile-shape tests.
"""
import pytest
import torch

from conftest import rel
from test_gpu_tiles import build

pytestmark = pytest.mark.gpu

GRIDS = [((16, 14, 3), (True, True, True)), ((17, 15, 4), (True, True, False)), ((31, 27, 5), (False, True, True)),
         ((14, 7, 6), (True, False, True)), ((13, 9, 2), (True, True, True))]
SHAPES = [None, (16, 14, 0), (16, 14, 1), (16, 8, 2), (14, 7, 3), (8, 8, 0), (15, 13, 2)]


@pytest.mark.parametrize("grid,periodic", GRIDS)
@pytest.mark.parametrize("shape", SHAPES)
def test_march_matches_oracle(grid, periodic, shape):
    op, ref, x, d = build(grid, periodic, 5)
    want = ref.mech_action(x, ref.degradation(d))
    if shape is not None:
        shape = (min(shape[0], ref_dim(grid, periodic, 0)), min(shape[1], ref_dim(grid, periodic, 1)), shape[2])
    for dt, tol in ((torch.float64, 1e-12), (torch.float32, 3e-5)):
        saved = op.tile_shape(dt)
        try:
            if shape is not None:
                op.tile_shape(dt, shape)
            y = op.mech_action(torch.as_tensor(x, device="cuda").to(dt), d=torch.as_tensor(d, device="cuda").to(dt))
            assert rel(y.double().cpu().numpy(), want) < tol
        finally:
            op.tile_shape(dt, saved)


def ref_dim(grid, periodic, axis):
    return grid[axis] + (0 if periodic[axis] else 1)
