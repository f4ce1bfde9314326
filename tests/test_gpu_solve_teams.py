"""The solve launches at the sizes where a body's team changes, against the FP64 oracle, and ray
picks at the sizes of their launch.

A body has one row slice per 32 vertices. Alone it is solved by one cluster up to 128 slices and by
a grid of CTAs above, and its rows are assembled slot by slot up to 1024 slices; in a batch its team
is a part of a cluster that doubles with its slices.

Tolerance: every solve stops at a relative residual of 1e-5 in the preconditioner's norm, so a
velocity is off by at most 1e-5 sqrt(condition number) of its norm: 1e-3 for a condition number of
1e4, which the preconditioned systems here (E = 1e5, h = 1/60) stay below. From rest the displacement
of one step is h v, so it has the same bound; rounding x to FP32 adds less than 1e-4 of it."""
import numpy as np
import pytest

import edge_bodies
import oracle
from bounce_softbody_gb300 import b3g, meshes

pytestmark = pytest.mark.gpu

DT = 1.0 / 60.0
TOL = 1e-3
PRECISIONS = {"fp32": b3g.PRECISION_FP32, "fp64": b3g.PRECISION_FP64, "bf16": b3g.PRECISION_BF16}
_expected = {}


def block(dims):
    return meshes.tet_grid(*dims, seed=sum(dims), E=1e5, nu=0.3, pin="y0")


def expected(dims):
    """One step of the oracle in FP64."""
    if dims not in _expected:
        x, v, it, _ = oracle.simulate(block(dims), 1, dt=DT, max_sub=500, sub_tol=1e-5, bits=64)
        _expected[dims] = (x, v, int(it[0]))
    return _expected[dims]


def check(dims, x, v, stats, outer):
    xr, vr, it = expected(dims)
    x0 = block(dims).x
    assert stats["solve_status"] == "converged", (dims, stats)
    if not outer:  # a mode whose iterations are the oracle's
        assert abs(stats["pcg_iterations"] - it) <= max(3, 0.1 * it), dims
    assert np.linalg.norm(v - vr) <= TOL * np.linalg.norm(vr), dims
    assert np.linalg.norm(x.astype(np.float64) - xr) <= TOL * np.linalg.norm(xr - x0), dims


# slices: 1 (part of one), 1, 2, 128 (the last cluster), 136 (the first grid), 1024, 1056
@pytest.mark.parametrize("dims", [(2, 2, 2), (4, 4, 2), (4, 4, 3), (16, 16, 16), (16, 16, 17), (32, 32, 32),
                                  (32, 32, 33)])
@pytest.mark.parametrize("precision", ["fp32", "fp64", "bf16"])
def test_single_body_teams_match_oracle(ctx, precision, dims):
    body = b3g.Body(ctx, block(dims))
    st = body.step(DT, b3g.solver_config(max_pcg_iterations=500, pcg_tolerance=1e-5, precision=PRECISIONS[precision],
                                         refresh_period=25))
    x, v = body.state()
    body.close()
    check(dims, x, v, st, precision == "bf16")


# slices 1, 1, 16, 18, 128, 136: teams of 1, 1, 1, 2, 8 and 16 CTAs at 16 slices a CTA in clusters of
# 16 (8 in clusters of 8), half of that at 32; then with a second launch of clusters of 4 and of 2
@pytest.mark.parametrize("schedule", ["16,1,0,16", "8,1,0,16", "4,1,1,32", "16,1,0,16,4", "16,1,1,4,2"])
@pytest.mark.parametrize("precision", ["fp32", "fp64", "bf16"])
def test_batched_teams_match_oracle(ctx, precision, schedule, monkeypatch):
    sizes = [(2, 2, 2), (4, 4, 2), (8, 8, 8), (9, 8, 8), (16, 16, 16), (16, 16, 17)] * 3
    cfg = b3g.solver_config(max_pcg_iterations=500, pcg_tolerance=1e-5, precision=PRECISIONS[precision],
                            refresh_period=25)

    def run(sched):
        monkeypatch.setenv("B3G_BATCH_SCHEDULE", sched)
        bodies = [b3g.Body(ctx, block(s)) for s in sizes]
        stats = b3g.step_batch(ctx, bodies, DT, 1, cfg)
        assert b3g.batch_schedule(ctx)["cluster"] == int(sched.split(",")[0])
        states = [b.state() for b in bodies]
        for b in bodies:
            b.close()
        return states, stats

    states, stats = run(schedule)
    if precision != "bf16":  # a batched BF16 solve is one with the rounded blocks
        for s, (x, v), st in zip(sizes, states, stats):
            check(s, x, v, st, False)
    # a row's order is fixed and sums are integers with at least FP64's bits: on these bodies the result
    # does not depend on the team
    alone, alone_stats = run("4,1,0,100000")
    for s, (x, v), st, (xa, va), sa in zip(sizes, states, stats, alone, alone_stats):
        assert st["pcg_iterations"] == sa["pcg_iterations"], s
        assert np.array_equal(x, xa) and np.array_equal(v, va), s


@pytest.mark.parametrize("dims", [(4, 4, 3), (16, 16, 17)])  # a cluster, a grid
def test_team_reports_a_nonfinite_solve(ctx, dims):
    d = block(dims)
    body = b3g.Body(ctx, d)
    f = np.zeros((d.n, 3), np.float32)
    f[-1, 1] = np.inf
    body.apply_forces(f)
    st = body.step(DT, b3g.solver_config(max_pcg_iterations=50))
    body.close()
    assert st["solve_status"] == "nonfinite"


# one launch takes up to 64 segments, more go in two launches; 450 triangles are a ragged last block
@pytest.mark.parametrize("count", [1, 63, 64, 65, 130])
def test_ray_casts_do_not_depend_on_their_number(ctx, count):
    body = b3g.Body(ctx, meshes.cloth_grid(16))
    rng = np.random.default_rng(count)
    seg = np.empty((count, 6))
    seg[:, [0, 2]] = rng.uniform(-1.2, 1.2, (count, 2))  # some pass beside the cloth
    seg[:, [3, 5]] = seg[:, [0, 2]] + rng.uniform(-0.2, 0.2, (count, 2))
    seg[:, 1], seg[:, 4] = 3.0, -1.0
    for _ in range(2):  # the scratch is left cleared for the next call
        together = body.ray_cast(seg)
        alone = [body.ray_cast(s[None]) for s in seg]
        for j, part in enumerate(together):
            assert np.array_equal(part, np.concatenate([a[j] for a in alone]))
    body.close()
    assert count < 63 or (together[0].any() and not together[0].all())


# the hub's row has spokes + 1 blocks; slot assembly gives 17 warps one slot column each per pass
@pytest.mark.parametrize("spokes", [15, 16, 17, 33, 90])
def test_rows_longer_than_a_pass_match_oracle(ctx, spokes):
    d = edge_bodies.particles(spokes + 1, seed=spokes)
    d.springs = np.stack([np.zeros(spokes), np.arange(1, spokes + 1)], 1).astype(np.uint32)
    # stretched: a spring at its rest length is on the edge between pulling and slack
    d.spring_L0 = 0.9 * np.linalg.norm(d.x[1:] - d.x[0], axis=1)
    d.spring_ks, d.spring_kd = np.full(spokes, 50.0), np.full(spokes, 0.5)
    body = b3g.Body(ctx, d)
    st = body.step(DT, b3g.solver_config(max_pcg_iterations=500, pcg_tolerance=1e-5, refresh_period=25))
    x, v = body.state()
    body.close()
    xr, vr, _, _ = oracle.simulate(d, 1, dt=DT, max_sub=500, sub_tol=1e-5, bits=64)
    assert st["solve_status"] == "converged"
    assert np.linalg.norm(v - vr) <= TOL * np.linalg.norm(vr)
    assert np.linalg.norm(x - xr) <= TOL * np.linalg.norm(xr - d.x)


# up to 16 Newton iterations a batched step takes launches of their own, one whole-step launch above
@pytest.mark.parametrize("newton", [2, 3, 16, 17])
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_batched_newton_iterations_match_oracle(ctx, precision, newton, monkeypatch):
    monkeypatch.setenv("B3G_BATCH_SCHEDULE", "16,1,0,4,4")
    mixes = [[block((2, 2, 2)), block((9, 8, 8)), block((16, 16, 17))]]  # the rows' short form
    if newton <= 3:  # a cloth at rest is on springs' slack edge: FP32 and FP64 oracles part with every iteration
        mixes.append([block((9, 8, 8)), meshes.cloth_grid(16)])
    for descs in mixes:
        bodies = [b3g.Body(ctx, d) for d in descs]
        cfg = b3g.solver_config(force_iterations=newton, max_pcg_iterations=500, pcg_tolerance=1e-5,
                                precision=PRECISIONS[precision])
        b3g.step_batch(ctx, bodies, DT, 1, cfg)
        for d, b in zip(descs, bodies):
            x, v = b.state()
            xr, vr, _, _ = oracle.simulate(d, 1, dt=DT, newton_iters=newton, max_sub=500, sub_tol=1e-5, bits=64)
            assert np.linalg.norm(v - vr) <= TOL * np.linalg.norm(vr)
            assert np.linalg.norm(x - xr) <= TOL * np.linalg.norm(xr - d.x)
            b.close()


def test_batched_newton_loops_end_at_their_own_iteration(ctx, monkeypatch):
    """Bodies whose loops end early, by tolerance, beside one that goes on; 16 and 17 as above."""
    monkeypatch.setenv("B3G_BATCH_SCHEDULE", "8,1,0,4")
    descs = [block((4, 4, 3)), meshes.tet_grid(6, 6, 6, seed=2, E=2e3, nu=0.3, pin="y0"), block((16, 16, 17))]
    runs = []
    for newton in (16, 17):
        bodies = [b3g.Body(ctx, d) for d in descs]
        cfg = b3g.solver_config(force_iterations=newton, max_pcg_iterations=500, pcg_tolerance=1e-5, newton_tolerance=1e-2)
        for _ in range(3):
            stats = b3g.step_batch(ctx, bodies, DT, 1, cfg)
        runs.append([(b.state(), s) for b, s in zip(bodies, stats)])
        for b in bodies:
            b.close()
    for ((xa, va), sa), ((xb, vb), sb) in zip(*runs):
        assert sa["newton_iterations"] == sb["newton_iterations"] < 16
        assert sa["total_steps"] == sb["total_steps"] == 3
        assert np.linalg.norm(va - vb) <= TOL * np.linalg.norm(vb)
