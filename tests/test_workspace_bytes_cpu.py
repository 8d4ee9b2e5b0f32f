"""Workspaces hold what their own solve uses (CPU)."""
import pytest


@pytest.mark.parametrize("n", [1, 33, 1000, 70001])
def test_t3_linear_solve_asks_for_no_exchange_words(n):
    """Only the Q4 form of the linear solve has a one-launch form, whose words take 16 bytes a node."""
    from phast_b200 import _lib
    lib = _lib.load()
    words = 2 * ((8 * n + 255) // 256 * 256)
    assert lib.phastb_q4_damage_linear_workspace_bytes(n) - lib.phastb_t3_damage_linear_workspace_bytes(n) == words
