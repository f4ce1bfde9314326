"""Solves of a body whose row vectors do not all fit the CTAs' shared memory: 195,112 vertices are 6098 row
slices, 41 a CTA, of which shared memory holds the vectors of 38 in the FP64 and BF16 modes (5 KB
a slice) and of all in the FP32 mode, the reference here."""
import numpy as np
import pytest

from bounce_softbody_gb300 import b3g, meshes

pytestmark = pytest.mark.gpu

DT = 1.0 / 60.0
# two solves of one system, each to a relative residual of 1e-5 in the preconditioner's norm; condition number
# of the preconditioned system up to 1e4
TOL = 2e-3


@pytest.mark.parametrize("precond", [b3g.PRECOND_JACOBI, b3g.PRECOND_BLOCK_JACOBI])
@pytest.mark.parametrize("mode", [b3g.CONTACT_PENALTY, b3g.CONTACT_FILTER])
def test_vectors_partly_in_global_memory(ctx, precond, mode):
    desc = meshes.block_on_floor(a=58, b=58, c=58, tilt=0.05)
    v = {}
    for precision in (b3g.PRECISION_FP32, b3g.PRECISION_FP64, b3g.PRECISION_BF16):
        body = b3g.Body(ctx, desc)
        # two Newton iterations: the second starts from the first one's solution; a refresh on the way
        stats = body.step(DT, b3g.solver_config(max_pcg_iterations=1000, pcg_tolerance=1e-5, precision=precision,
                                                preconditioner=precond, contact_mode=mode, refresh_period=25,
                                                force_iterations=2))
        assert stats["solve_status"] == "converged"
        x, v[precision] = body.state()
        assert np.isfinite(x).all()
        body.close()
    ref = v.pop(b3g.PRECISION_FP32)
    assert np.linalg.norm(ref) > 0
    for precision, got in v.items():
        assert np.linalg.norm(got - ref) <= TOL * np.linalg.norm(ref), precision
