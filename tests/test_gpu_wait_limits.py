"""Device waits of the solve launches that run out: with a limit of a few polls ordinary waits do. The
calls return, every body whose solve did not complete reports device_timeout, and the next step with
the default limit is an ordinary one."""
import functools
import time

import numpy as np
import pytest

import oracle
from bounce_softbody_gb300 import b3g, b3g_sparse, meshes

pytestmark = pytest.mark.gpu

DT = 1.0 / 60.0
# a solve to a relative residual of 1e-5, condition numbers up to 1e4: velocities to 1e-3 of their norm
TOL = 1e-3


@pytest.fixture()
def own():
    c = b3g.Context(0)
    yield c
    c.close()


def block(dims):
    return meshes.tet_grid(*dims, seed=sum(dims), E=1e5, nu=0.3, pin="y0")


def config(precision="fp32", newton=1):
    return b3g.solver_config(max_pcg_iterations=500, pcg_tolerance=1e-5, force_iterations=newton, refresh_period=25,
                             precision={"fp32": b3g.PRECISION_FP32, "fp64": b3g.PRECISION_FP64,
                                        "bf16": b3g.PRECISION_BF16}[precision])


@functools.lru_cache(None)
def expected(dims, newton):
    return oracle.simulate(block(dims), 1, dt=DT, newton_iters=newton, max_sub=500, sub_tol=1e-5, bits=64)[:2]


def matches_oracle(dims, body, newton):
    d = block(dims)
    x, v = body.state()
    xr, vr = expected(dims, newton)
    return np.linalg.norm(v - vr) <= TOL * np.linalg.norm(vr) and np.linalg.norm(x - xr) <= TOL * np.linalg.norm(xr - d.x)


# teams of 1 to 16 CTAs; with a second launch; every body on one CTA, where nobody waits
@pytest.mark.parametrize("schedule", ["16,1,0,16", "8,1,0,16,2", "16,1,1,4,4", "4,1,0,100000"])
@pytest.mark.parametrize("newton", [1, 2])
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_batched_waits_that_run_out(own, precision, newton, schedule, monkeypatch):
    monkeypatch.setenv("B3G_BATCH_SCHEDULE", schedule)
    sizes = [(2, 2, 2), (8, 8, 8), (9, 8, 8), (16, 16, 16), (16, 16, 17)] * 4
    descs = [block(s) for s in sizes]
    cfg = config(precision, newton)

    def run(limit):
        bodies = [b3g.Body(own, d) for d in descs]
        own.set_poll_limit(limit)
        stats = b3g.step_batch(own, bodies, DT, 1, cfg)
        own.set_poll_limit(0)
        return bodies, stats

    ref, ref_stats = run(0)
    assert all(s["solve_status"] == "converged" for s in ref_stats)
    states = [b.state() for b in ref]
    for limit in (1, 50, 1000):
        bodies, stats = run(limit)
        late = [s["solve_status"] == "device_timeout" for s in stats]
        if schedule.startswith("4,"):
            assert not any(late)
        elif limit == 1:
            assert any(late)
        # a body is reported, or it took exactly this step
        for b, s, out, (x, v) in zip(bodies, stats, late, states):
            if out:
                continue
            assert s["total_steps"] == 1 and s["solve_status"] == "converged"
            xb, vb = b.state()
            assert np.array_equal(x, xb) and np.array_equal(v, vb)
        for b, d in zip(bodies, descs):
            b.set_state(d.x, np.zeros_like(d.x))
        again = b3g.step_batch(own, bodies, DT, 1, cfg)
        for b, dims, s in zip(bodies, sizes, again):
            assert s["solve_status"] == "converged"
            assert matches_oracle(dims, b, newton)
            b.close()
    for b in ref:
        b.close()


# one cluster, the grid
@pytest.mark.parametrize("dims", [(12, 12, 12), (20, 20, 20)])
@pytest.mark.parametrize("newton", [1, 2])
@pytest.mark.parametrize("precision", ["fp32", "fp64", "bf16"])
def test_single_body_waits_that_run_out(own, precision, newton, dims):
    d = block(dims)
    body = b3g.Body(own, d)
    own.set_poll_limit(1)
    assert body.step(DT, config(precision, newton))["solve_status"] == "device_timeout"
    assert body.stats()["solve_status"] == "device_timeout"
    own.set_poll_limit(0)
    body.set_state(d.x, np.zeros_like(d.x))
    assert body.step(DT, config(precision, newton))["solve_status"] == "converged"
    assert matches_oracle(dims, body, newton)
    body.close()


@pytest.mark.parametrize("n", [3000, 9000])  # one cluster, the grid
def test_sparse_waits_that_run_out(own, n):
    rng = np.random.default_rng(n)
    A = b3g_sparse.SparseMat33(own, n)
    # symmetric and diagonally dominant: 4 I on the diagonal, -0.99 I towards four neighbours
    i = np.concatenate([np.arange(n), np.arange(n - 1), np.arange(1, n), np.arange(n - 50), np.arange(50, n)])
    j = np.concatenate([np.arange(n), np.arange(1, n), np.arange(n - 1), np.arange(50, n), np.arange(n - 50)])
    w = np.concatenate([np.full(n, 4.0), np.full(len(i) - n, -0.99)])
    A.add_blocks(i, j, w[:, None, None] * np.eye(3))
    rhs = rng.standard_normal((n, 3))
    b, x = b3g_sparse.DenseVec3(own, n, rhs), b3g_sparse.DenseVec3(own, n, np.zeros((n, 3)))
    own.set_poll_limit(1)
    assert b3g_sparse.solve_cg(A, b, x, 1000, 1e-5)["status"] == "device_timeout"
    own.set_poll_limit(0)
    x.set(np.zeros((n, 3)))
    out = b3g_sparse.solve_cg(A, b, x, 1000, 1e-5)
    assert out["status"] == "converged"
    # condition number below 4 (1 + 0.99) / (4 (1 - 0.99)) = 199: the solution is off by at most 1e-5 sqrt(199)
    y = np.zeros((n, 3))
    xs = x.get().astype(np.float64)
    np.add.at(y, i, w[:, None] * xs[j])
    assert np.linalg.norm(y - rhs) <= 1e-3 * np.linalg.norm(rhs)
    for o in (A, b, x):
        o.close()


def test_served_requests_whose_waits_run_out(own):
    own.set_poll_limit(1)
    server = b3g.Server(own, 1 << 30, 4, DT, config())
    body = server.add_body(block((20, 20, 20)))
    server.submit(body, 2)
    server.start()
    assert [r["status"] for r in server.drain(60)] == ["device_timeout"]
    own.set_poll_limit(0)
    server.submit(body, 1)
    assert [r["status"] for r in server.drain(60)] == ["done"]
    # a request reports its early steps too
    own.set_poll_limit(1)
    server.submit(body, 1000)
    time.sleep(0.02)
    own.set_poll_limit(0)
    assert [r["status"] for r in server.drain(60)] == ["device_timeout"]
    server.close()
