"""The persistent T3 damage solve over its splits of a mesh (needs a B200).

One triangle, one block, blocks that read one another's words or go through the first, a mesh too
large for it, and a node where two fans of triangles meet in a point only (twice as many neighbours
as a fan of its size has).  Each must end at the solution of the bound-constrained system the
operators define: the solve stops on the true residual of its own rows, which differ from the
operator's kernel by round-off (1 %).
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def grid(nx, ny, rng):
    x, y = np.meshgrid(np.linspace(0.0, 1.0, nx + 1), np.linspace(0.0, ny / nx, ny + 1))
    move = 0.2 / nx * (rng.random((2,) + x.shape) - 0.5)
    n0 = (np.arange(ny)[:, None] * (nx + 1) + np.arange(nx)[None, :]).reshape(-1)
    tris = np.concatenate([np.stack([n0, n0 + 1, n0 + nx + 2], 1), np.stack([n0, n0 + nx + 2, n0 + nx + 1], 1)])
    nodes = np.stack([(x + move[0]).reshape(-1), (y + move[1]).reshape(-1)], 1)
    order = rng.permutation(len(nodes)) if nx < 30 else np.arange(len(nodes))  # small meshes: scattered numbering
    out = np.empty_like(nodes)
    out[order] = nodes
    return out, order[tris]


def bowtie(rng):
    a = np.linspace(0.3, 1.2, 6)
    pts = [[0.0, 0.0]] + [[np.cos(t), np.sin(t)] for t in a] + [[-np.cos(t), -np.sin(t)] for t in a]
    tris = [[0, k, k + 1] for k in range(1, 6)] + [[0, k, k + 1] for k in range(7, 12)]
    return np.array(pts), np.array(tris)


MESHES = [("one", lambda r: (np.array([[0.0, 0.0], [1.0, 0.1], [0.2, 0.9]]), np.array([[0, 1, 2]]))),
          ("bowtie", bowtie), ("11x7", lambda r: grid(11, 7, r)), ("40x30", lambda r: grid(40, 30, r)),
          ("90x80", lambda r: grid(90, 80, r)), ("230x220", lambda r: grid(230, 220, r)),
          ("330x300", lambda r: grid(330, 300, r))]


@pytest.mark.parametrize("name,make", MESHES, ids=[m[0] for m in MESHES])
@pytest.mark.parametrize("model", ["AT2", "AT1"])
def test_solve(name, make, model):
    import phast_b200 as pb
    rng = np.random.default_rng(7)
    nodes, tris = make(rng)
    mesh = pb.FEMMesh.from_tensors(torch.as_tensor(nodes), torch.as_tensor(tris), element_type="T3", device="cuda")
    mat = pb.Material(E=210000.0, nu=0.3, Gc=2.7, l0=0.05, eta_residual=1e-8, energy_split="amor", pf_model=model)
    fem = pb.FEMOperators(mesh, mat)
    solver = pb.PhaseFieldDamageSolver(fem, tol=1e-10, max_iter=20000, bounds_method="projected_cg")
    gc_l0 = mat.Gc / mat.l0
    H = torch.as_tensor(gc_l0 * rng.uniform(0.3, 0.9, fem.n_elems), device="cuda")
    d_prev = torch.as_tensor(rng.uniform(0.0, 0.5, fem.n_nodes), device="cuda")
    fixed = torch.zeros(fem.n_nodes, dtype=torch.bool, device="cuda")
    fixed[::13] = True
    d = solver.solve(H, d_prev, pf_dirichlet_mask=fixed, pf_dirichlet_values=torch.ones_like(d_prev))
    assert solver.last_converged
    assert bool((d[fixed] == 1.0).all()) and bool((d >= d_prev).all()) and bool((d <= 1.0).all())
    b, _ = solver.prepare(H)
    g = solver._Ax(d, H) - b
    start = torch.where(fixed, torch.ones_like(d_prev), d_prev)
    scale = max(float(b.norm()), float(torch.where(fixed, 0.0, solver._Ax(start, H) - b).norm()))
    free = ~fixed & (d > d_prev) & (d < 1.0)
    assert float(g[free].norm()) <= 1.01e-10 * scale
    low = ~fixed & (d <= d_prev) & (d < 1.0)
    assert float(g[low].clamp(max=0.0).norm()) <= 1.01e-10 * scale
