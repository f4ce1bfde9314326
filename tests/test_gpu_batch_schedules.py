"""The schedules of a batch: up to 16 Newton iterations a step takes solve launches with one schedule, with more
the whole-step launch with another, each tuned among candidates of its own and kept."""
import numpy as np
import pytest

from bounce_softbody_gb300 import b3g, meshes

pytestmark = pytest.mark.gpu


def raw_schedule(ctx):
    buf = np.zeros(512, np.int32)
    lib = b3g.load_library()
    assert lib.b3g_batch_schedule(ctx.handle, buf.ctypes.data_as(b3g._ip), buf.size) == 0
    return buf[:5], buf[6], [int(c) for c in buf[7:7 + 2 * buf[5]:2]]


def test_many_newton_iterations_have_a_schedule_of_their_own(ctx, monkeypatch):
    monkeypatch.delenv("B3G_BATCH_SCHEDULE", raising=False)
    monkeypatch.delenv("B3G_AUTOTUNE", raising=False)
    bodies = [b3g.Body(ctx, meshes.tet_grid(*s, seed=sum(s), E=1e5, nu=0.3, pin="y0"))
              for s in [(4, 4, 3), (8, 8, 8), (14, 13, 12), (16, 16, 17)]]

    def step(newton):
        b3g.step_batch(ctx, bodies, 1.0 / 60.0, 1, b3g.solver_config(force_iterations=newton, max_pcg_iterations=50,
                                                                     newton_tolerance=1e-2))
        return raw_schedule(ctx)

    few = step(1)
    many = step(17)
    assert few[0][4] and many[0][4]  # tuned
    assert few[2] and all(c < 10 ** 9 for c in few[2])
    # single CTAs for every body, clusters of 2 to 16 from each threshold that some body reaches, in both orders
    want = {10 ** 9 + o * 10 ** 8 + 10 ** 6 + 999999 for o in (0, 1)}
    want |= {10 ** 9 + o * 10 ** 8 + cl * 10 ** 6 + t for cl in (2, 4, 8, 16) for t in (1, 1024, 2048, 4096) for o in (0, 1)}
    assert set(many[2]) == want
    # each is kept: the same candidates with the same choice, not tuned again
    for newton, first in ((16, few), (30, many), (1, few)):
        again = step(newton)
        assert np.array_equal(again[0], first[0]) and again[1] == first[1] and again[2] == first[2]
    for b in bodies:
        b.close()


@pytest.mark.parametrize("newton,cluster", [(1, 8), (17, 1)])
def test_fixed_rules_without_the_autotuner(ctx, newton, cluster, monkeypatch):
    monkeypatch.delenv("B3G_BATCH_SCHEDULE", raising=False)
    monkeypatch.setenv("B3G_AUTOTUNE", "0")
    bodies = [b3g.Body(ctx, meshes.tet_grid(*s, seed=1, E=1e5, nu=0.3, pin="y0")) for s in [(4, 4, 3), (16, 16, 17)]]
    b3g.step_batch(ctx, bodies, 1.0 / 60.0, 1, b3g.solver_config(force_iterations=newton))
    first, _, candidates = raw_schedule(ctx)
    assert first[0] == cluster and not first[4] and not candidates
    for b in bodies:
        b.close()
