"""Entries put into the boundary lists by hand: any index of an array, a value per node (CPU, and on the device)."""
import numpy as np
import pytest
import torch

from phast_b200 import BoundaryConditions

ENTRIES = [([0, 2], 0, 1.0), (np.array([1, 3]), 1, 2.0), (slice(4, 6), 0, 3.0), (5, 1, 4.0),
           (torch.tensor([False, False, False, True, False, False]), 0, 5.0),
           (torch.tensor([2, 4], dtype=torch.int32), 1, torch.tensor([6.0, 7.0], dtype=torch.float64)),
           (torch.tensor([0, 1]), 1, torch.tensor([8.0, 9.0], dtype=torch.float64))]


@pytest.mark.parametrize("device", ["cpu", pytest.param("cuda", marks=pytest.mark.gpu)])
def test_entries(device):
    b = BoundaryConditions(6, device=device)
    b.bcs.extend(ENTRIES)
    b.load_factor = 2.0
    mask, vals = b.get_masks_and_values()
    assert mask.device.type == device and vals.device.type == device
    assert mask.tolist() == [[True, True], [False, True], [True, True], [True, True], [True, True], [True, True]]
    assert vals.tolist() == [[2.0, 16.0], [0.0, 18.0], [2.0, 12.0], [10.0, 4.0], [6.0, 14.0], [6.0, 8.0]]
    b.pf_dirichlet_bcs.extend([([1], 0.5), (slice(2, 4), torch.tensor([0.25, 0.75], dtype=torch.float64))])
    pm, pv = b.get_pf_dirichlet_mask_values()
    assert pm.tolist() == [False, True, True, True, False, False] and pv[1:4].tolist() == [0.5, 0.25, 0.75]


def test_entries_outside_the_mesh():
    for bad in ([6], np.array([-7]), 6):
        b = BoundaryConditions(6, device="cpu")
        b.bcs.append((bad, 0, 1.0))
        with pytest.raises(IndexError):
            b.get_masks_and_values()
