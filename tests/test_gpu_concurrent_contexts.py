"""Contexts that step at the same time from their own threads: solve launches of one body (which need every SM
at once), of clusters and of batches share the GPU, and each step is what it is alone."""
import threading

import numpy as np
import pytest

from bounce_softbody_gb300 import b3g, meshes

pytestmark = pytest.mark.gpu

DT = 1.0 / 60.0


def block(dims):
    return meshes.tet_grid(*dims, seed=sum(dims), E=1e5, nu=0.3, pin="y0")


def single(dims, steps, ready, go):
    """Steps of one body: the grid above 4096 vertices, a cluster below."""
    c = b3g.Context(0)
    body = b3g.Body(c, block(dims))
    cfg = b3g.solver_config(max_pcg_iterations=100, pcg_tolerance=1e-5)
    ready.wait()
    go.wait()
    status = [body.step(DT, cfg)["solve_status"] for _ in range(steps)]
    state = body.state()
    c.close()
    return [status], [state]


def batch(newton, steps, ready, go, started=None):
    c = b3g.Context(0)
    bodies = [b3g.Body(c, block((8 + k % 9, 9 + k % 7, 10 + k % 5))) for k in range(160)]
    cfg = b3g.solver_config(max_pcg_iterations=200, pcg_tolerance=1e-5, force_iterations=newton, newton_tolerance=1e-14)
    ready.wait()
    if started is not None:
        started.set()
    status = [[s["solve_status"] for s in b3g.step_batch(c, bodies, DT, 1, cfg)] for _ in range(steps)]
    states = [b.state() for b in bodies]
    c.close()
    return status, states


def together(*jobs):
    ready = threading.Barrier(len(jobs))
    out = [None] * len(jobs)

    def run(k):
        out[k] = jobs[k](ready)

    threads = [threading.Thread(target=run, args=(k,)) for k in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join(120)
    assert all(o is not None for o in out)
    return out


def same(a, b):
    assert all(np.array_equal(x, y) for s, t in zip(a, b) for x, y in zip(s, t))


def now():
    e = threading.Event()
    e.set()
    return e


def test_four_contexts_at_once(monkeypatch):
    monkeypatch.setenv("B3G_BATCH_SCHEDULE", "16,1,0,16,2")
    jobs = [lambda r: single((20, 20, 20), 100, r, now()), lambda r: single((40, 40, 40), 100, r, now()),
            lambda r: single((12, 12, 12), 100, r, now()), lambda r: batch(1, 20, r, now())]
    alone = [together(j)[0] for j in jobs]
    for a, b in zip(alone, together(*jobs)):
        assert all(s == "converged" for step in b[0] for s in step)
        same(a[1], b[1])


def test_a_wait_for_the_gpu_is_no_wait_of_a_team(monkeypatch):
    """A launch that fills the GPU for some seconds, longer than a team's wait lasts: a body's solve launched
    meanwhile starts after it, and none of its waits runs out."""
    monkeypatch.setenv("B3G_BATCH_SCHEDULE", "4,1,0,16")
    alone = together(lambda r: single((20, 20, 20), 5, r, now()))[0]
    started = threading.Event()
    long, during = together(lambda r: batch(1200, 1, r, None, started), lambda r: single((20, 20, 20), 5, r, started))
    assert all(s == "converged" for step in long[0] + during[0] for s in step)
    same(alone[1], during[1])
