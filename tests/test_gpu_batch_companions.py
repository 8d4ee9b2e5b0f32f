"""A cell of a packed batch gives the same bits whatever cells share its launches (needs a B200).

One cell is solved alone and beside others: of other sizes, more of them than one launch of the
coarsest multigrid level takes, and enough large ones that this launch takes deeper bricks.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _solve(sizes, kind):
    from phast_b200 import solid3d as s3
    from phast_b200.solid3d import batch
    load = batch.batch_load()
    ops = [batch.build_operator(c, load) for k, n in enumerate(sizes)
           for c in batch.particle_cells(seed=k, n_cells=1, sizes=(n,))]
    B = batch.PackedCellBatch(ops, brick=(16, 8, 8))
    rng = [np.random.default_rng(100 + k) for k in range(len(ops))]
    d = B.pack_nodes([torch.as_tensor(r.uniform(0.0, 0.6, op.n_red), device="cuda") for r, op in zip(rng, ops)])
    if kind == "kkt":
        H = B.pack_elems([torch.as_tensor(r.uniform(0.0, 1.0, (op.n_elements, 8)), device="cuda")
                          for r, op in zip(rng, ops)])
        x, status, info, _ = B.damage_box_kkt(H, 0.5 * d, 0.5 * d)
        return B.node_view(x, 0).clone(), int(info[0][0])
    form = s3.MechForm("gmg", mixed=True, smooth_degree=1, coarse_degree=6, inner_rtol=1e-5)
    kw = {"f64": {}, "mixed": dict(mixed=True), "gmg": dict(mixed=True, form=form)}[kind]
    x, status, its, *_ = B.mech_solve(d, B.pack_mech([op.mech_fixed_values(0.004) for op in ops]), rtol=1e-6, **kw)
    assert status == 0
    return B.mech_view(x, 0).clone(), int(its[0])


@pytest.mark.parametrize("kind,sizes", [(k, (32, 40, 48, 64)) for k in ("f64", "mixed", "gmg", "kkt")] +
                         [(k, (32,) * 70) for k in ("f64", "gmg", "kkt")] + [("gmg", (96,) * 6)])
def test_cell_does_not_depend_on_its_companions(kind, sizes):
    alone, n_alone = _solve(sizes[:1], kind)
    together, n_together = _solve(sizes, kind)
    assert n_alone == n_together and torch.equal(alone, together)
