"""AFP_ENTRIES_PER_LANE, the tuning limit on a lane's share of a row."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PROGRAM = """
import sys
import numpy as np
from afepack_gb300 import workloads as W
from afepack_gb300.amg import AMGSolver
from afepack_gb300.fem import BoundaryConditionAdmin, Context, Space, assemble
ctx = Context(0)
wl = W.poisson2d_p1(40)
K, M = assemble(Space(ctx, wl.space), wl.acc_stiff, wl.acc_mass)
b = M.vmult(wl.f)
bca = BoundaryConditionAdmin(wl.space)
bca.add(1, 0.0)
bca.apply(K, b)
x = np.zeros_like(b)
AMGSolver(K).solve(x, b, step=0)
np.save(sys.argv[1], x)
"""


def test_entries_per_lane_is_honoured(ctx, tmp_path):
    """More lanes a row add its entries up in another order: one V-cycle differs by rounding, and by no more."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    out = []
    for limit in (None, "0.1"):
        env = dict(os.environ, PYTHONPATH=root)
        env.pop("AFP_ENTRIES_PER_LANE", None)
        if limit:
            env["AFP_ENTRIES_PER_LANE"] = limit
        path = str(tmp_path / f"x{limit}.npy")
        subprocess.run([sys.executable, "-c", PROGRAM, path], check=True, env=env, cwd=root, timeout=300)
        out.append(np.load(path))
    assert not np.array_equal(out[0], out[1])
    assert np.linalg.norm(out[0] - out[1]) <= 1e-10 * np.linalg.norm(out[0])
