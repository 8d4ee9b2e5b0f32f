"""Dirichlet masks and values are filled where they are used, their nodes checked on the host (CPU)."""
import pytest
import torch

from phast_b200 import BoundaryConditions


def test_boundary_conditions_fill_and_check_their_nodes():
    """Masks and values by node and component, later entries over earlier ones; a node outside the mesh raises."""
    b = BoundaryConditions(5, device="cpu")
    b.fix([0, 1], 0).add([1, -1], 1, 2.0).add(torch.tensor([[1], [2]]), 1, 3.0)
    b.load_factor = 0.5
    mask, vals = b.get_masks_and_values()
    assert mask.tolist() == [[True, False], [True, True], [False, True], [False, False], [False, True]]
    assert vals[:, 1].tolist() == [0.0, 1.5, 1.5, 0.0, 1.0]
    b.add_pf_dirichlet([3, 3, 4], 0.25)
    pm, pv = b.get_pf_dirichlet_mask_values()
    assert pm.tolist() == [False, False, False, True, True] and pv[3:].tolist() == [0.25, 0.25]
    for bad in (5, -6):
        with pytest.raises(IndexError):
            BoundaryConditions(5, device="cpu").fix([0, bad], 0).get_masks_and_values()
        with pytest.raises(IndexError):
            BoundaryConditions(5, device="cpu").add_pf_dirichlet([bad]).get_pf_dirichlet_mask_values()
