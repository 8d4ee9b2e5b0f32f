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


# One entry on 6 nodes, and the nodes that a (6, 2) array indexed by [entry, component] has set, None where it refuses.
# A 1D array (the damage lists) takes or refuses the same index in its own way.
ARRAY_INDICES = [((0, 2), [0, 2], None), ([[0, 1], [2, 3]], [0, 1, 2, 3], None), (..., [0, 1, 2, 3, 4, 5], list(range(6))),
                 (np.int64(3), [3], [3]), (torch.tensor([0, 1, 0, 0, 0, 1], dtype=torch.uint8), None, None),
                 (torch.tensor([[0, 1], [4, 5]]), [0, 1, 4, 5], [0, 1, 4, 5]),
                 ([True, False, False, False, False, True], [0, 5], [0, 5]),
                 (torch.tensor([True, False]), None, None), (torch.tensor([1.0]), None, None)]


@pytest.mark.parametrize("index,nodes,damage_nodes", ARRAY_INDICES)
@pytest.mark.parametrize("device", ["cpu", pytest.param("cuda", marks=pytest.mark.gpu)])
def test_an_entry_indexes_as_an_array(device, index, nodes, damage_nodes):
    b = BoundaryConditions(6, device=device)
    b.add([4], 1, 3.0)
    b.bcs.append((index, 0, 2.0))
    b.add_pf_dirichlet([4], 0.5)
    b.pf_dirichlet_bcs.append((index, 0.25))
    for get, want, base in ((b.get_masks_and_values, nodes, 1), (b.get_pf_dirichlet_mask_values, damage_nodes, None)):
        if want is None:
            with pytest.raises((IndexError, RuntimeError)):
                get()
            continue
        mask, vals = get()
        assert mask.device.type == device and vals.device.type == device
        column = mask[:, 0] if base else mask
        assert column.nonzero().flatten().tolist() == sorted(set(want) | (set() if base else {4}))
        if base:
            assert mask[4, 1] and vals[:, 0].nonzero().flatten().tolist() == want


def test_device_lists_mix_with_entries_put_in_by_hand():
    b = BoundaryConditions(6, device="cpu").add([1], 0, 2.0)
    b.bcs.extend([(slice(3, 5), 1, torch.tensor([1.0, 2.0], dtype=torch.float64)), ((5,), 0, 4.0)])
    assert b.get_masks_and_values()[1].tolist() == [[0, 0], [2, 0], [0, 0], [0, 1], [0, 2], [4, 0]]
