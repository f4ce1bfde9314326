"""The candidates of b3g_batch_schedule as b3g.batch_schedule decodes them (codes of include/b3g.h)."""
import numpy as np
import pytest

from bounce_softbody_gb300 import b3g


@pytest.mark.parametrize("code,want", [
    (16 * 10 ** 6 + 64, dict(cluster=16, order="size", slices_per_cta=64, second_launch_cluster=0)),
    (10 ** 8 + 8 * 10 ** 6 + 4 * 1000 + 256, dict(cluster=8, order="lpt", slices_per_cta=256, second_launch_cluster=4)),
    (10 ** 9 + 4 * 10 ** 6 + 1024, dict(cluster=4, order="size", threshold=1024)),
    (10 ** 9 + 10 ** 8 + 10 ** 6 + 999999, dict(cluster=1, order="lpt", threshold=-1)),
])
def test_candidate_codes(monkeypatch, code, want):
    class Lib:
        @staticmethod
        def b3g_batch_schedule(ctx, out, capacity):
            values = [8, 100, 3, 152, 1, 1, 0, code, 1500]
            for k, v in enumerate(values):
                out[k] = v
            return 0

    class Ctx:
        handle = None

    monkeypatch.setattr(b3g, "load_library", lambda: Lib)
    schedule = b3g.batch_schedule(Ctx)
    assert schedule["candidates_ms"] == [dict(want, ms=1.5)]
    assert (schedule["cluster"], schedule["threshold"], schedule["autotuned"]) == (8, 100, True)
    assert np.iinfo(np.int32).max > code
