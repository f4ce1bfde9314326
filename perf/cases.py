"""The work that programs do with b3g, as cases that can be timed and compared.

A case is one frame of a program that keeps its bodies on the GPU: it hands over the particles'
state or forces from host memory, steps, and reads the particles back, as a program written against
the reference does with b3Particle and b3Body::Step. The kinds:

* ``ray``: mouse picking, a few segments against a cloth's triangles;
* ``tet`` / ``cloth`` / ``bw``: one body through ``Body.step``;
* ``batch``: many uneven bodies through ``step_batch`` with page-locked host arrays;
* ``cg``: ``b3SparseSolveCG`` on a matrix of the program's own.

``iters`` is about how many PCG iterations the case's solves take (it only enters ``work``).
"""
import functools

import numpy as np
import torch

from bounce_softbody_gb300 import b3g, b3g_sparse, meshes

H60, H30 = 1.0 / 60.0, 1.0 / 30.0


def listed():
    return [
        # a user clicks on a cloth: the smallest call, all latency
        dict(name="ray_pick", kind="ray", m=97, segments=8),
        # a small odd block with several Newton iterations and block Jacobi, as in a game scene that
        # is stepped accurately; launches and host waits are all there is to it
        dict(name="tet_small_newton", kind="tet", a=9, b=7, c=6, E=2e5, nu=0.33, newton=3, precond=1,
             precision=0, tol=1e-6, max_it=200, refresh=50, h60=True, iters=50),
        # the 10 x 10 x 10 block of the first named workload
        dict(name="tet_10", kind="tet", a=10, b=10, c=10, E=1e5, nu=0.3, newton=1, precond=0, precision=0,
             tol=1e-5, max_it=200, refresh=50, h60=True, iters=32),
        # a block in double precision, ragged against the 32-row slices
        dict(name="tet_fp64", kind="tet", a=29, b=23, c=19, E=1e5, nu=0.3, newton=1, precond=0, precision=1,
             tol=1e-5, max_it=200, refresh=50, h60=True, iters=40),
        # bf16 blocks on a stiff, ill-conditioned block (the precision variant's workload, smaller)
        dict(name="tet_bf16", kind="tet", a=47, b=41, c=37, E=1e6, nu=0.45, newton=1, precond=0, precision=2,
             tol=1e-5, max_it=1500, refresh=25, h60=False, iters=15),
        # the 64 x 64 x 64 block of the named workload: the largest single body
        dict(name="tet_64", kind="tet", a=64, b=64, c=64, E=1e6, nu=0.45, newton=1, precond=0, precision=0,
             tol=1e-5, max_it=1000, refresh=50, h60=False, iters=330),
        # the named 128 x 128 cloth (membrane triangles, springs, contact sphere): 200 iterations
        dict(name="cloth_128", kind="cloth", m=128, max_it=200, iters=200),
        # the testbed's cloth: Baraff-Witkin stretch and shear forces
        dict(name="bw_cloth_61", kind="bw", m=61, max_it=200, iters=28),
        # b3SparseSolveCG on a caller's matrix
        dict(name="sparse_cg", kind="cg", a=23, b=19, c=17, stiff=100.0, tol=1e-5, max_it=200, iters=131),
        # a scene of a dozen uneven blocks
        dict(name="batch_12", kind="batch", count=12, mesh_seed=12, mixed=False, iters=38),
        # the headline's batch of uneven blocks (a third of its bodies, so that setting it up is quick)
        dict(name="batch_160", kind="batch", count=160, mesh_seed=3, mixed=False, iters=38),
        # the bodies of the serving stream: blocks and cloths in one batch
        dict(name="batch_mixed_16", kind="batch", count=16, mesh_seed=7, mixed=True, iters=120),
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["ray", "tet", "tet", "tet", "cloth", "bw", "cg", "batch", "batch", "batch"])
    if kind == "ray":
        return dict(kind=kind, m=rng.randint(20, 128), segments=_log_int(rng, 1, 64))
    if kind == "tet":
        base = _log_int(rng, 5, 48)
        a, b, c = (max(4, int(round(base * rng.uniform(0.75, 1.3)))) for _ in range(3))
        stiff = rng.random() < 0.4
        precision = rng.choice([0, 0, 0, 1, 2])
        newton = rng.choice([1, 1, 1, 2, 3]) if precision == 0 else 1
        return dict(kind=kind, a=a, b=b, c=c, E=1e6 if stiff else round(10.0 ** rng.uniform(4.3, 5.5)),
                    nu=0.45 if stiff else round(rng.uniform(0.2, 0.4), 3), newton=newton,
                    precond=rng.choice([0, 0, 1]) if newton > 1 else 0, precision=precision, tol=1e-5,
                    max_it=1000, refresh=rng.choice([25, 50]), h60=not stiff,
                    iters=15 if precision == 2 else int(6 * base if stiff else 20 + base))
    if kind == "cloth":
        return dict(kind=kind, m=rng.randint(32, 160), max_it=200, iters=200)
    if kind == "bw":
        return dict(kind=kind, m=rng.randint(10, 96), max_it=200, iters=28)
    if kind == "cg":
        a, b, c = (rng.randint(5, 30) for _ in range(3))
        return dict(kind=kind, a=a, b=b, c=c, stiff=round(10.0 ** rng.uniform(0.5, 2.5), 2), tol=1e-5, max_it=200,
                    iters=100)
    mixed = rng.random() < 0.35
    return dict(kind=kind, count=_log_int(rng, 2, 20) if mixed else _log_int(rng, 4, 150),
                mesh_seed=rng.randint(20, 10 ** 6), mixed=mixed, iters=120 if mixed else 38)


# ---------------------------------------------------------------- bodies
@functools.lru_cache(maxsize=1)
def _bodies(key):
    """The meshes of a case (a program's assets: they do not depend on the seed)."""
    c = dict(key)
    if c["kind"] == "ray":
        return [meshes.bw_cloth(c["m"], pinned="corners", stretch_ks=5e3)]
    if c["kind"] == "tet":
        return [meshes.tet_grid(c["a"], c["b"], c["c"], seed=1, E=float(c["E"]), nu=c["nu"], pin="y0")]
    if c["kind"] == "cloth":
        return [meshes.cloth_grid(c["m"])]
    if c["kind"] == "bw":
        return [meshes.bw_cloth(c["m"], pinned="corners", stretch_ks=5e3, stretch_kd=2.0, shear_ks=1e3, shear_kd=1.0)]
    if c["mixed"]:
        return meshes.serving_bodies(c["count"], seed=c["mesh_seed"])
    return meshes.batch_bodies(c["count"], seed=c["mesh_seed"])


def bodies_of(case):
    return _bodies(tuple(sorted((k, v) for k, v in case.items() if k != "name")))


def motion(desc, rng):
    """A body in motion: a smooth bend of a few per cent strain with the velocities that go with it,
    and a little noise on top (springs and triangles then sit clearly on one side of their rest
    length)."""
    x = desc.x
    lo, ext = x.min(0), max(float(np.ptp(x, axis=0).max()), 1e-9)
    u = (x - lo) / ext
    k = rng.uniform(1.0, 2.5, (3, 3))
    phase = rng.uniform(0.0, 2.0 * np.pi, 3)
    amp = 0.03 * ext * rng.uniform(0.6, 1.0, 3)
    wave = u @ k.T + phase
    step = 0.5 * ext / max(round(desc.n ** (1.0 / 3.0)), 2)
    dx = amp * np.sin(wave) + 0.004 * step * rng.standard_normal(x.shape)
    if desc.springs.shape[0] or desc.tris.shape[0]:
        dx = dx + 0.01 * (x - x.mean(0))
    v = 6.0 * amp * np.cos(wave) + 0.02 * step * rng.standard_normal(x.shape)
    v[np.asarray(desc.type) == meshes.STATIC] = 0.0
    return (x + dx).astype(np.float32), v.astype(np.float32)


def config(case):
    return b3g.solver_config(force_iterations=case.get("newton", 1), max_pcg_iterations=case.get("max_it", 200),
                             pcg_tolerance=case.get("tol", 1e-5), refresh_period=case.get("refresh", 50),
                             precision=case.get("precision", 0), preconditioner=case.get("precond", 0))


def step_of(case):
    return H60 if case.get("h60", True) else H30


def _rng(case, seed):
    return np.random.default_rng([seed, sum(ord(ch) for ch in case["kind"])])


def _segments(case, rng, desc, x):
    """Segments through random inner points of random triangles, from well above to well below."""
    t = desc.tris[rng.integers(0, desc.tris.shape[0], case["segments"])].astype(np.int64)
    w = 0.2 + 0.4 * rng.dirichlet(np.ones(3), case["segments"])
    p = np.einsum("sk,skc->sc", w, x[t].astype(np.float64))
    d = np.stack([rng.uniform(-0.05, 0.05, case["segments"]), np.ones(case["segments"]),
                  rng.uniform(-0.05, 0.05, case["segments"])], 1)
    return np.concatenate([p + rng.uniform(1.0, 3.0, (len(p), 1)) * d, p - 2.0 * d], 1).astype(np.float32)


def _cg_system(case, rng):
    """A symmetric positive definite block matrix of a caller: a grid of springs with random
    directions and stiffnesses over random masses, and a right-hand side."""
    a, b, c = case["a"], case["b"], case["c"]
    n = a * b * c
    ids = np.arange(n).reshape(c, b, a)
    pairs = [np.stack([ids[:, :, :-1].ravel(), ids[:, :, 1:].ravel()], 1),
             np.stack([ids[:, :-1].ravel(), ids[:, 1:].ravel()], 1),
             np.stack([ids[:-1].ravel(), ids[1:].ravel()], 1),
             np.stack([ids[:-1, :-1, :-1].ravel(), ids[1:, 1:, 1:].ravel()], 1)]
    pairs = np.concatenate(pairs)
    d = rng.standard_normal((len(pairs), 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    k = case["stiff"] * rng.uniform(0.5, 1.5, len(pairs))
    blk = (k[:, None, None] * (d[:, :, None] * d[:, None, :] + 0.1 * np.eye(3))).astype(np.float32)
    mass = rng.uniform(0.5, 2.0, n).astype(np.float32)
    eye = np.zeros((n, 3, 3), np.float32)
    eye[:, [0, 1, 2], [0, 1, 2]] = mass[:, None]
    i, j = pairs[:, 0], pairs[:, 1]
    rows = np.concatenate([np.arange(n), i, j, i, j])
    cols = np.concatenate([np.arange(n), i, j, j, i])
    vals = np.concatenate([eye, blk, blk, -blk, -blk]).astype(np.float32)  # symmetric blocks
    return n, rows, cols, vals, rng.standard_normal((n, 3)).astype(np.float32)


def prepare(case, seed):
    ctx = b3g.Context(0)
    rng = _rng(case, seed)
    s = dict(case=case, ctx=ctx)
    if case["kind"] == "cg":
        n, rows, cols, vals, rhs = _cg_system(case, rng)
        A = b3g_sparse.SparseMat33(ctx, n)
        A.add_blocks(rows, cols, vals)
        s.update(A=A, b=b3g_sparse.DenseVec3(ctx, n), x=b3g_sparse.DenseVec3(ctx, n), rhs=rhs,
                 guess=np.zeros((n, 3), np.float32))
        A.size()  # the matrix is on the device before it is solved with
        return s
    descs = bodies_of(case)
    bodies = [b3g.Body(ctx, d) for d in descs]
    if case["kind"] in ("ray", "tet", "cloth", "bw"):
        x, v = motion(descs[0], rng)
        s.update(body=bodies[0], x=x, v=v, cfg=config(case), h=step_of(case))
        if case["kind"] == "ray":
            bodies[0].set_state(x, v)
            s["segments"] = _segments(case, rng, descs[0], x)
        return s
    # a batch: the first call on a body list also picks its schedule, which a program does once
    # when the scene is loaded; the bodies then start from the moving state
    cfg = config(case)
    b3g.step_batch(ctx, bodies, H60, 1, cfg, stats=False)
    states = [motion(d, rng) for d in descs]
    for b, (x, v) in zip(bodies, states):
        b.set_state(x, v)
    total = sum(d.n for d in descs)
    host = [torch.empty((total, 3), dtype=torch.float32, pin_memory=True) for _ in range(3)]
    wind = rng.uniform(-1.0, 1.0, 3) * 0.5
    mass = np.concatenate([b.masses() for b in bodies])
    host[0].copy_(torch.from_numpy((mass[:, None] * (wind + 0.2 * rng.standard_normal((total, 3)))).astype(np.float32)))
    s.update(bodies=bodies, cfg=cfg, h=H60, f=host[0], x=host[1], v=host[2])
    return s


def run(s):
    kind = s["case"]["kind"]
    if kind == "ray":
        hit, tri, fraction, normal = s["body"].ray_cast(s["segments"])
        return dict(hit=hit, triangle=tri, fraction=fraction, normal=normal)
    if kind == "cg":
        s["b"].set(s["rhs"])
        s["x"].set(s["guess"])
        b3g_sparse.solve_cg(s["A"], s["b"], s["x"], s["case"]["max_it"], s["case"]["tol"])
        return s["x"].get()
    if kind != "batch":
        body = s["body"]
        body.set_state(s["x"], s["v"])
        body.step(s["h"], s["cfg"], stats=False)
        return body.state()
    ctx, bodies = s["ctx"], s["bodies"]
    b3g.batch_apply_forces(ctx, bodies, s["f"].data_ptr())
    b3g.step_batch(ctx, bodies, s["h"], 1, s["cfg"], stats=False)
    b3g.batch_get_state(ctx, bodies, s["x"].data_ptr(), s["v"].data_ptr())
    return s["x"], s["v"]


# ---------------------------------------------------------------- bytes and operations
def _blocks_per_row(desc):
    """Nonzero 3x3 blocks per row of A on these grids."""
    if desc.tets.shape[0]:
        return 14.6
    return 13.0 if desc.springs.shape[0] else 7.0


def work(case):
    """Inputs read once and results written once (state, element data); the flops of the elements,
    of the assembly and of the PCG iterations (18 per block and 27 per vertex each)."""
    if case["kind"] == "ray":
        n, t = case["m"] ** 2, 2 * (case["m"] - 1) ** 2
        return dict(bytes=12.0 * n + 12.0 * t + 48.0 * case["segments"], flops=60.0 * t * case["segments"])
    if case["kind"] == "cg":
        n = case["a"] * case["b"] * case["c"]
        nnzb = 9.0 * n
        return dict(bytes=40.0 * nnzb + 36.0 * n, flops=case["iters"] * (18.0 * nnzb + 27.0 * n))
    bytes_, flops = 0.0, 0.0
    for d in bodies_of(case):
        T, Tr, S, n = d.tets.shape[0], d.tris.shape[0], d.springs.shape[0], d.n
        elem = 100.0 * T + 16.0 * S + 24.0 * Tr + 80.0 * d.stretch_tris.shape[0] + 80.0 * d.shear_tris.shape[0]
        bytes_ += 48.0 * n + 12.0 * n + elem
        per = 18.0 * _blocks_per_row(d) * n + 27.0 * n
        flops += case.get("newton", 1) * (900.0 * T + 300.0 * (Tr + S) + case["iters"] * per)
    return dict(bytes=bytes_, flops=flops)


# ---------------------------------------------------------------- the same in 64 bits
def _t(a, dev):
    return torch.as_tensor(np.asarray(a), device=dev)


def _f64(a, dev):
    """A float array as the body holds it (rounded to 32 bits), in 64 bits."""
    return _t(np.asarray(a, np.float32), dev).double()


def _add(n, ids, val):
    out = torch.zeros((n, 3), dtype=torch.float64, device=val.device)
    return out.index_add_(0, ids.reshape(-1), val.reshape(-1, 3))


def _masses(d, rest, dev):
    """b3Body::ResetMass: fixture masses lumped to their vertices, 1 where there are none."""
    m = torch.zeros(d.n, dtype=torch.float64, device=dev)
    if d.tets.shape[0]:
        t = _t(d.tets.astype(np.int64), dev)
        e = rest[t[:, 1:]] - rest[t[:, :1]]
        vol = torch.linalg.det(e).abs() / 6.0
        m.index_add_(0, t.reshape(-1), (0.25 * vol * _f64(d.tet_density, dev))[:, None].expand(-1, 4).reshape(-1))
    if d.tris.shape[0]:
        t = _t(d.tris.astype(np.int64), dev)
        area = 0.5 * torch.linalg.cross(rest[t[:, 1]] - rest[t[:, 0]], rest[t[:, 2]] - rest[t[:, 0]]).norm(dim=1)
        m.index_add_(0, t.reshape(-1), (area / 3.0 * _f64(d.tri_density, dev))[:, None].expand(-1, 3).reshape(-1))
    return torch.where(m > 0, m, torch.ones_like(m))


def _polar(F):
    """The rotation of F by Newton's iteration R <- (R + R^-T) / 2."""
    R = F
    for _ in range(12):
        R = 0.5 * (R + torch.linalg.inv(R).transpose(1, 2))
    return R


def _outer(a, b):
    return a[..., :, None] * b[..., None, :]


def _tet_terms(d, rest, X, V, W, h, dev):
    t = _t(d.tets.astype(np.int64), dev)
    E, nu = _f64(d.tet_E, dev), _f64(d.tet_nu, dev)
    lam, mu = nu * E / ((1 + nu) * (1 - 2 * nu)), E / (2 * (1 + nu))
    e = (rest[t[:, 1:]] - rest[t[:, :1]]).transpose(1, 2)  # columns e1 e2 e3
    vol = torch.linalg.det(e).abs() / 6.0
    inv = torch.linalg.inv(e)
    g = torch.cat([-inv.sum(1, keepdim=True), inv], 1)  # (T, 4, 3): the shape gradients
    F = torch.einsum("tar,tac->trc", X[t], g)
    G = F + torch.einsum("tar,tac->trc", W[t], g)
    R = _polar(F)
    eye = torch.eye(3, dtype=torch.float64, device=dev)
    U = R.transpose(1, 2) @ G - eye
    S = mu[:, None, None] * (U + U.transpose(1, 2)) + (lam * U.diagonal(dim1=1, dim2=2).sum(1))[:, None, None] * eye
    rhs = -h * vol[:, None, None] * torch.einsum("tac,tbc,tdb->tad", g, S, R)
    rg = torch.einsum("trc,tac->tar", R, g)
    c = h * h * vol
    K = torch.einsum("t,tar,tbs->tarbs", c * lam, rg, rg) + torch.einsum("t,tbr,tas->tarbs", c * mu, rg, rg)
    K = K + torch.einsum("t,tab,rs->tarbs", c * mu, torch.einsum("tac,tbc->tab", rg, rg), eye)
    return t, K.reshape(-1, 12, 12), rhs


def _spring_terms(d, X, V, W, h, dev):
    """Tension-only springs; the stiffness keeps the reference's unnormalised outer product. (The
    cloth's membrane triangles are left out: their stiffness scales with the fourth power of twice
    a triangle's area, 1e-14 of the springs' here.)"""
    t = _t(d.springs.astype(np.int64), dev)
    ks, kd, L0 = _f64(d.spring_ks, dev), _f64(d.spring_kd, dev), _f64(d.spring_L0, dev)
    dx = X[t[:, 0]] - X[t[:, 1]]
    L = dx.norm(dim=1)
    n = dx / L[:, None]
    on = (L > L0).double()
    eye = torch.eye(3, dtype=torch.float64, device=dev)
    q = 1.0 - L0 / L
    Ks = (on * ks)[:, None, None] * (_outer(dx, dx) * (1 - q)[:, None, None] + q[:, None, None] * eye)
    f = -(on * ks * (L - L0))[:, None] * n
    f = f - (kd * (n * (V[t[:, 0]] - V[t[:, 1]])).sum(1))[:, None] * n
    f = f - torch.einsum("erc,ec->er", Ks, W[t[:, 0]] - W[t[:, 1]])
    B = h * h * Ks + h * kd[:, None, None] * _outer(n, n)
    K = torch.cat([torch.cat([B, -B], 2), torch.cat([-B, B], 2)], 1)
    return t, K, torch.stack([h * f, -h * f], 1)


def _bw_terms(d, rest, X, V, W, h, dev):
    """Baraff-Witkin stretch and shear triangles with the rest frame of Initialize."""
    out = []
    for tris, par, shear in ((d.stretch_tris, d.stretch_params, False), (d.shear_tris, d.shear_params, True)):
        if not tris.shape[0]:
            continue
        t = _t(tris.astype(np.int64), dev)
        p = _f64(par, dev)
        ab, ac = rest[t[:, 1]] - rest[t[:, 0]], rest[t[:, 2]] - rest[t[:, 0]]
        du1 = ab.norm(dim=1)
        dv1 = torch.zeros_like(du1)
        du2, dv2 = (ac * ab).sum(1) / du1, torch.linalg.cross(ab, ac).norm(dim=1) / du1
        det = du1 * dv2 - du2 * dv1
        alpha = 0.5 * det.abs()
        gu = torch.stack([dv1 - dv2, dv2, -dv1], 1) / det[:, None]
        gv = torch.stack([du2 - du1, -du2, du1], 1) / det[:, None]
        wu, wv = torch.einsum("ea,eac->ec", gu, X[t]), torch.einsum("ea,eac->ec", gv, X[t])
        f = torch.zeros((t.shape[0], 3, 3), dtype=torch.float64, device=dev)
        K = torch.zeros((t.shape[0], 3, 3, 3, 3), dtype=torch.float64, device=dev)
        eye = torch.eye(3, dtype=torch.float64, device=dev)
        if shear:
            dC = alpha[:, None, None] * (gu[:, :, None] * wv[:, None] + gv[:, :, None] * wu[:, None])
            C = alpha * (wu * wv).sum(1)
            f = f - (p[:, 0] * (C + (dC * W[t]).sum((1, 2))) + p[:, 1] * (dC * V[t]).sum((1, 2)))[:, None, None] * dC
            K = torch.einsum("e,ear,ebs->earbs", h * h * p[:, 0] + h * p[:, 1], dC, dC)
        else:
            for g, w, (ks, kd, b) in ((gu, wu, p[:, 0:3].T), (gv, wv, p[:, 3:6].T)):
                ln = w.norm(dim=1)
                n = w / ln[:, None]
                C = alpha * (ln - b)
                q = torch.where(ln > b, C * alpha / ln, torch.zeros_like(ln))
                Ks = ks[:, None, None] * ((alpha ** 2 - q)[:, None, None] * _outer(n, n) + q[:, None, None] * eye)
                KW = torch.einsum("erc,ec->er", Ks, torch.einsum("ea,eac->ec", g, W[t]))
                dCdt = alpha * (torch.einsum("ea,eac->ec", g, V[t]) * n).sum(1)
                f = f - (g * (ks * C * alpha + kd * dCdt * alpha)[:, None])[:, :, None] * n[:, None] - g[:, :, None] * KW[:, None]
                M = h * h * Ks + (h * kd * alpha ** 2)[:, None, None] * _outer(n, n)
                K = K + torch.einsum("ea,eb,ers->earbs", g, g, M)
        out.append((t, K.reshape(-1, 9, 9), h * f))
    return out


def _pcg(apply, b, x, minv, tol, max_it, warm):
    """b3SparseSolveCG: Jacobi PCG, exit when r.M^-1 r <= tol^2 r0.M^-1 r0."""
    r = b - apply(x) if warm else b.clone()
    s = minv(r)
    d = s.clone()
    delta0 = delta = float((r * s).sum())
    it = 0
    while it < max_it and delta > tol * tol * delta0:
        q = apply(d)
        alpha = delta / float((d * q).sum())
        x = x + alpha * d
        r = r - alpha * q
        s = minv(r)
        new = float((r * s).sum())
        d = s + (new / delta) * d
        delta = new
        it += 1
    return x


def _exact_step(case, d, x, v, fext, dev):
    h = float(np.float32(step_of(case)))
    rest, x0, v0 = _f64(d.x, dev), _f64(x, dev), _f64(v, dev)
    m = _masses(d, rest, dev)
    dyn = _t(np.asarray(d.type) == meshes.DYNAMIC, dev)
    damp = _f64(d.damping, dev)
    mask = dyn.double()[:, None]
    md = (m * (1.0 + h * damp))[:, None]
    grav = _f64(d.gravity, dev)
    fe = fext if fext is not None else torch.zeros_like(x0)
    X, V = x0, v0
    y = torch.zeros_like(x0)
    newton = case.get("newton", 1)
    # bf16 blocks are only a preconditioner: that mode solves the full system its own way
    tol = 1e-9 if case.get("precision", 0) == 2 else case.get("tol", 1e-5)
    max_it = 5000 if case.get("precision", 0) == 2 else case.get("max_it", 200)
    err0 = None
    for k in range(newton):
        W = (x0 - X) + h * V
        terms = []
        if d.tets.shape[0]:
            terms.append(_tet_terms(d, rest, X, V, W, h, dev))
        if d.springs.shape[0]:
            terms.append(_spring_terms(d, X, V, W, h, dev))
        terms += _bw_terms(d, rest, X, V, W, h, dev)
        b = m[:, None] * (v0 - V) + h * (fe + m[:, None] * grav - (damp * m)[:, None] * V)
        D = torch.zeros((d.n, 3, 3), dtype=torch.float64, device=dev)
        for ids, K, rhs in terms:
            b = b + _add(d.n, ids, rhs)
            nv = ids.shape[1]
            diag = K.reshape(-1, nv, 3, nv, 3).diagonal(dim1=1, dim2=3).permute(0, 3, 1, 2)
            D.index_add_(0, ids.reshape(-1), diag.reshape(-1, 3, 3))
        D = D + md[:, :, None] * torch.eye(3, dtype=torch.float64, device=dev)
        D[~dyn] = torch.eye(3, dtype=torch.float64, device=dev)
        b = b * mask

        def apply(p):
            pm = p * mask
            out = md * pm
            for ids, K, _ in terms:
                q = torch.bmm(K, pm[ids].reshape(len(ids), -1, 1))
                out = out + _add(d.n, ids, q)
            return out * mask + p * (1.0 - mask)

        if case.get("precond", 0) == 1:
            Di = torch.linalg.inv(D)
            minv = lambda r: torch.einsum("nrc,nc->nr", Di, r)  # noqa: E731
        else:
            Dd = D.diagonal(dim1=1, dim2=2)
            minv = lambda r: r / Dd  # noqa: E731
        y = _pcg(apply, b, y, minv, tol, max_it, k > 0)
        V = V + y
        X = x0 + h * V
        err = float((y * y).sum())
        eps2 = float(np.float32(1.1920929e-07)) ** 2
        if (err0 is None and err <= eps2) or (err0 is not None and err <= eps2 * err0):
            break
        err0 = err if err0 is None else err0
    return X.cpu().numpy(), V.cpu().numpy()


def _exact_rays(case, seed):
    """Every triangle against every segment (the reference's b3TriangleShape::RayCast)."""
    d = bodies_of(case)[0]
    rng = _rng(case, seed)
    x, _ = motion(d, rng)
    seg = _segments(case, rng, d, x).astype(np.float64)
    t = d.tris.astype(np.int64)
    A, B, C = (x.astype(np.float64)[t[:, k]] for k in range(3))
    N = np.cross(B - A, C - A)
    n = N / np.linalg.norm(N, axis=1, keepdims=True)
    fraction, normal = [], []
    for s in seg:
        p1, dr = s[:3], s[3:] - s[:3]
        num, den = ((A - p1) * n).sum(1), n @ dr
        f = np.where(den != 0, num / np.where(den == 0, 1.0, den), -1.0)
        Q = p1 + f[:, None] * dr
        inside = (f >= 0) & (f <= 1)
        for P, R in ((B, C), (C, A), (A, B)):
            inside &= (np.cross(P - Q, R - Q) * N).sum(1) >= 0
        f = np.where(inside, f, np.inf)
        k = int(np.argmin(f))
        fraction.append(f[k])
        normal.append(-n[k] if num[k] > 0 else n[k])
    return dict(hit=None, triangle=None, fraction=np.array(fraction), normal=np.array(normal))


def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if case["kind"] == "ray":
        return _exact_rays(case, seed)
    rng = _rng(case, seed)
    if case["kind"] == "cg":
        n, rows, cols, vals, rhs = _cg_system(case, rng)
        r, c, B = _t(rows, dev), _t(cols, dev), _t(vals, dev).double()
        apply = lambda p: _add(n, r, torch.einsum("erc,ec->er", B, p[c]))  # noqa: E731
        D = torch.zeros((n, 3), dtype=torch.float64, device=dev)
        D.index_add_(0, r[r == c], B[r == c].diagonal(dim1=1, dim2=2))
        b = _t(rhs, dev).double()
        return _pcg(apply, b, torch.zeros_like(b), lambda q: q / D, case["tol"], case["max_it"], False).cpu().numpy()
    descs = bodies_of(case)
    if case["kind"] != "batch":
        x, v = motion(descs[0], rng)
        return _exact_step(case, descs[0], x, v, None, dev)
    if case["mixed"] or sum(d.n for d in descs) > 400_000:
        return None  # over 20 seconds, or cloths whose solves stop unfinished at the iteration cap
    states = [motion(d, rng) for d in descs]
    wind = rng.uniform(-1.0, 1.0, 3) * 0.5
    mass = [_masses(d, _f64(d.x, dev), dev) * _t(np.asarray(d.type) == meshes.DYNAMIC, dev) for d in descs]
    total = sum(d.n for d in descs)
    mass32 = torch.cat(mass).float().cpu().numpy()
    f = (mass32[:, None] * (wind + 0.2 * rng.standard_normal((total, 3)))).astype(np.float32)
    xs, vs, at = [], [], 0
    for d, (x, v) in zip(descs, states):
        X, V = _exact_step(case, d, x, v, _t(f[at:at + d.n], dev).double(), dev)
        at += d.n
        xs.append(X)
        vs.append(V)
    return np.concatenate(xs), np.concatenate(vs)
