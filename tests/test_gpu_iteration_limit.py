"""The iteration limit of the multigrid CG (needs a B200).

The host looks at the solve's state every second iteration, in chunks it launches or in one graph
that loops on the device (PHASTB_DEVICE_LOOP=1, read once per process).  Neither may run past the
limit, odd or even: the unfinished iterate has the same bits from both.
"""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

SCRIPT = """
import hashlib, sys
import numpy as np, torch
from phast_b200 import solid3d as s3
rng = np.random.default_rng(3)
phases = [s3.PhaseMaterial("mi_matrix", "isotropic", 0.5, "spectral", 3000.0, 0.35),
          s3.PhaseMaterial("fibre", "isotropic", 0.2, "spectral", 9000.0, 0.3)]
load = s3.LoadCase("zz", 2, (0.01,), (), (0, 1, 3, 4, 5))
op = s3.PeriodicVoxelPhaseFieldOperator.from_slots(s3.VoxelGrid((16, 16, 24), (1 / 16,) * 3),
                                                   rng.integers(0, 2, 16 * 16 * 24), phases, 0.125, 1e-6, load,
                                                   pinned_node=0)
d = torch.as_tensor(rng.uniform(0.0, 0.6, op.n_red), device="cuda")
for mixed in (False, True):
    form = s3.MechForm("gmg", mixed=mixed, smooth_degree=1, coarse_degree=6)
    for limit in (1, 2, 5, 6):
        x, info = s3.solve_constrained_form(op, form, fixed_mask=op.mech_fixed_mask(),
                                            fixed_values=op.mech_fixed_values(0.004), d=d, rtol=1e-13, maxiter=limit)
        print(mixed, limit, info.iterations, info.converged, hashlib.sha1(x.cpu().numpy().tobytes()).hexdigest())
"""


def test_limit_is_kept():
    out = []
    for loop in ("0", "1"):
        env = dict(os.environ, PHASTB_DEVICE_LOOP=loop, PYTHONPATH=ROOT)
        p = subprocess.run([sys.executable, "-c", SCRIPT], env=env, cwd=ROOT, capture_output=True, text=True, timeout=300)
        assert p.returncode == 0, p.stderr[-2000:]
        out.append(p.stdout.split("\n"))
    assert len(out[0]) == 9 and out[0] == out[1]
    lines = [line.split() for line in out[0][:8]]
    assert all(v[2] == v[1] and v[3] == "False" for v in lines) and len({v[4] for v in lines}) == 8
