"""Phase cycles of the solve launches (B3G_PHASE_PROFILE)."""
import pytest

from bounce_softbody_gb300 import b3g, meshes

pytestmark = pytest.mark.gpu


def test_a_second_solve_launch_loses_no_cycles(ctx, monkeypatch):
    """Each of 600 equal bodies is solved by one CTA, in the first launch or in the second: the cycles are those
    without the second launch. They differ by 1 %; 5 % allowed."""
    monkeypatch.setenv("B3G_PHASE_PROFILE", "1")
    cfg = b3g.solver_config(max_pcg_iterations=100, pcg_tolerance=1e-5)
    cycles = []
    for schedule in ("16,1,0,100000", "16,1,0,100000,2"):
        monkeypatch.setenv("B3G_BATCH_SCHEDULE", schedule)
        bodies = [b3g.Body(ctx, meshes.tet_grid(8, 8, 8, seed=3, E=1e5, nu=0.3, pin="y0")) for _ in range(600)]
        b3g.step_batch(ctx, bodies, 1.0 / 60.0, 1, cfg)
        b3g.batch_phase_cycles(ctx)
        b3g.step_batch(ctx, bodies, 1.0 / 60.0, 2, cfg)
        cycles.append(b3g.batch_phase_cycles(ctx))
        for b in bodies:
            b.close()
    for phase in ("spmv", "update"):
        assert abs(cycles[1][phase] - cycles[0][phase]) <= 0.05 * cycles[0][phase], cycles
