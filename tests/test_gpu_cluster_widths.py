"""A single body's solve where the device cannot hold the widest clusters."""
import os
import subprocess
import sys

import numpy as np
import pytest
from conftest import ROOT

pytestmark = pytest.mark.gpu

SCRIPT = """
import sys
import numpy as np
from bounce_softbody_gb300 import b3g, meshes
ctx = b3g.Context(0)
out = []
for dims in [(4, 4, 2), (8, 8, 8), (9, 8, 8), (13, 13, 13), (16, 16, 16)]:
    for precision in (b3g.PRECISION_FP32, b3g.PRECISION_FP64):
        body = b3g.Body(ctx, meshes.tet_grid(*dims, seed=sum(dims), E=1e5, nu=0.3, pin="y0"))
        st = body.step(1.0 / 60.0, b3g.solver_config(max_pcg_iterations=500, pcg_tolerance=1e-5, precision=precision))
        assert st["solve_status"] == "converged"
        out += [a.ravel() for a in body.state()]
        body.close()
ctx.close()
np.save(sys.argv[1], np.concatenate(out))
"""


def test_bodies_are_solved_without_the_widest_clusters(tmp_path):
    """Where a device cannot hold a cluster of 16 CTAs, or any: narrower ones or the grid, the same steps."""
    states = []
    for widest in ("16", "8", "0"):
        path = str(tmp_path / f"{widest}.npy")
        subprocess.run([sys.executable, "-c", SCRIPT, path], cwd=ROOT, env={**os.environ, "B3G_SOLVE_CLUSTER": widest},
                       check=True, timeout=300)
        states.append(np.load(path))
    assert np.array_equal(states[0], states[1]) and np.array_equal(states[0], states[2])
