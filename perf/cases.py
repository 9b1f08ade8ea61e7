"""The work whose speed is measured: substeps of single scenes and of a batch in
the forms the framework is used in, and the surrogate network's forward pass
and gradient.

A simulation case is what a program does between two looks at the state: it
puts a particle state into the simulator, recomputes the prescribed levels
where the scene refines, advances a few substeps and reads the particles back.
Starting every pass from the same state keeps the work of a pass the same
however often it is run.  The states are bodies in mid-motion (a smooth
velocity field with its gradient in C, strained F, some plastic volume change
in snow), not the rest states the scenes start from.

`exact` restates the substep over dense torch arrays in 64 bits.  Decisions
that follow from 32-bit positions (base cells) are taken from the 32-bit value.
"""
import ctypes
import math
import os
import random
import sys

import torch
import torch.nn.functional as nnf

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "adaptive-gimp_b200"))

from agimp import AdaptiveGIMP  # noqa: E402
from agimp.batch import SceneBatch  # noqa: E402
from agimp.surrogate import MLP  # noqa: E402

DEV = "cuda:0"

ELASTIC = dict(E=1e4 / 100.0, nu=0.2, gravity=-9.8, boundary="sticky", snow=False, normalize=False)
SNOW2 = dict(E=1.4e5 / 1000.0, nu=0.2, gravity=-9.8, boundary="sticky", snow=True, normalize=True)
SNOW3 = dict(E=1e5 / 400.0, nu=0.25, gravity=-9.8, boundary="sticky", snow=True, normalize=True)
SPHERES = dict(E=1.4e5 / 400.0, nu=0.2, gravity=-9.8, boundary="sticky", snow=True, normalize=True)
DEMO = dict(E=5e3, nu=0.2, gravity=-100.0, boundary="ref_slip", snow=False, normalize=False)


def listed():
    sim = dict(kind="sim", substeps=10, refine=False, static=False)
    return [
        # the 2D demo: 20,000 particles on 4 levels, ten substeps per drawn frame
        dict(sim, name="demo2d", dim=2, level=4, coarsest=16, body="demo", n=20000, scale=1.0, dt=2e-5, **DEMO),
        # the 3D demo: 50,000 particles, one substep per drawn frame (the smallest call)
        dict(sim, name="demo3d", dim=3, level=3, coarsest=16, body="demo", n=50000, scale=1.0, dt=1e-4,
             **DEMO) | dict(substeps=1),
        # a static quadtree: two elastic boxes, 21 thousand particles
        dict(sim, name="static2d", dim=2, level=3, coarsest=64, body="boxes", n=2, scale=1.0, dt=1e-4,
             **ELASTIC) | dict(static=True),
        # dynamic 2D snow on 4 levels, levels recomputed every ten substeps
        dict(sim, name="dynamic2d", dim=2, level=4, coarsest=64, body="boxes", n=3, scale=1.0, dt=5e-5,
             **SNOW2) | dict(refine=True),
        # 256 independent 2D scenes of 2..4 levels stepped by shared launches
        dict(kind="batch", name="batch2d", scenes=256, substeps=10, dt=1e-4, scale=1.0, **ELASTIC),
        # the 3D snow sphere at a third of its size: small dynamic 3D scenes
        dict(sim, name="sphere3d_small", dim=3, level=3, coarsest=64, body="spheres", n=1, scale=0.35, dt=5e-5,
             **SNOW3) | dict(refine=True),
        # a static 3D map on 2 levels, elastic boxes of ragged extents
        dict(sim, name="static3d", dim=3, level=2, coarsest=64, body="boxes", n=2, scale=1.31, dt=1e-4,
             **ELASTIC) | dict(static=True, substeps=4),
        # the 3D snow sphere: 1.9M particles on 3 levels up to 256^3 (the headline scene)
        dict(sim, name="sphere3d", dim=3, level=3, coarsest=64, body="spheres", n=1, scale=1.0, dt=5e-5,
             **SNOW3) | dict(refine=True, substeps=5),
        # two colliding snow spheres: 15.5M particles on 4 levels up to 512^3 (the largest scene)
        dict(sim, name="spheres3d", dim=3, level=4, coarsest=64, body="spheres", n=2, scale=0.8, dt=3e-5,
             **SPHERES) | dict(refine=True, substeps=3),
        # surrogate return map over a large scene's particles, and over the few that yield in a small one
        dict(kind="mlp_forward", name="mlp_forward", rows=2000000),
        dict(kind="mlp_forward", name="mlp_forward_small", rows=20003),
        # one gradient of the surrogate's training loop at its default batch
        dict(kind="mlp_grad", name="mlp_grad", rows=65536),
    ]


def draw(rng):
    def span(lo, hi):
        return math.exp(rng.uniform(math.log(lo), math.log(hi)))

    t = rng.random()
    if t < 0.1:
        return dict(kind="mlp_forward", rows=int(span(1000, 2000000)))
    if t < 0.2:
        return dict(kind="mlp_grad", rows=int(span(1000, 1000000)))
    if t < 0.3:
        return dict(kind="batch", scenes=int(span(3, 256)), substeps=rng.randint(4, 10), dt=1e-4,
                    scale=rng.uniform(0.3, 1.0), **ELASTIC)
    dim = rng.choice((2, 3))
    static = rng.random() < 0.4
    c = dict(kind="sim", dim=dim, static=static, level=rng.randint(2, 4 if dim == 2 else 3), coarsest=64)
    if rng.random() < 0.3:
        c.update(body="demo", n=int(span(3000, 300000)), scale=rng.uniform(0.7, 1.0), dt=2e-5, coarsest=rng.choice((16, 32)),
                 refine=False, static=False, substeps=rng.randint(1, 10), **dict(DEMO, normalize=True))
    else:
        body = rng.choice(("boxes", "spheres"))
        c.update(body=body, n=rng.randint(1, 3) if body == "boxes" else rng.randint(1, 2),
                 scale=span(0.3, 1.2) if dim == 2 else span(0.3, 1.0),
                 dt=5e-5, refine=not static, substeps=rng.randint(2, 10) if dim == 2 else rng.randint(2, 5),
                 **(ELASTIC if static else SNOW2 if dim == 2 else SNOW3))
    return c


# ---------------------------------------------------------------------------
# inputs
def _generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _lattice(dim, finest, inside, lo, hi, gen):
    """Two points per axis and finest cell whose lattice place lies inside the shape, jittered by half a spacing."""
    h = 0.5 / finest
    axes = [torch.arange(math.floor(a / h), math.ceil(b / h), device=DEV, dtype=torch.float64) * h + 0.5 * h
            for a, b in zip(lo, hi)]
    p = torch.stack(torch.meshgrid(*axes, indexing="ij"), -1).reshape(-1, dim)
    p = p[inside(p)]
    u = torch.rand(p.shape, generator=gen, device=DEV, dtype=torch.float64)
    return p + (u - 0.5) * h


def _bodies(case):
    """[(kind, lo or centre, hi or radius)] of a scene."""
    if "boxes" in case:
        return case["boxes"]
    d, s, n = case["dim"], case["scale"], case["n"]
    if case["body"] == "boxes":
        side = [(0.2, 0.2, 0.17), (0.2, 0.2, 0.23), (0.16, 0.21, 0.19)] if not case["refine"] else \
            [(0.17, 0.14), (0.21, 0.24), (0.13, 0.22)]
        mid = [(0.3, 0.45, 0.4), (0.65, 0.7, 0.6), (0.72, 0.3, 0.5)]
        return [("box", [mid[i][k] - 0.5 * s * side[i][k % len(side[i])] for k in range(d)],
                 [mid[i][k] + 0.5 * s * side[i][k % len(side[i])] for k in range(d)]) for i in range(n)]
    if n == 1:
        return [("sphere", [0.5, 0.6, 0.5][:d], 0.15 * s)]
    return [("sphere", [0.35, 0.5, 0.5][:d], 0.15 * s), ("sphere", [0.65, 0.5, 0.5][:d], 0.15 * s)]


def _positions(case, gen):
    """Positions and prescribed levels."""
    d, L = case["dim"], case["level"]
    finest = case["coarsest"] << (L - 1)
    if case["body"] == "demo":
        # two boxes of uniformly drawn particles, coarser levels towards the middle of each
        half, size, xs, gs = case["n"] // 2, 0.4 if d == 2 else 0.3, [], []
        for k, m in enumerate((half, case["n"] - half)):
            u = torch.rand((m, d), generator=gen, device=DEV, dtype=torch.float64)
            lo = [(0.2, 0.1, 0.2), (0.4 if d == 2 else 0.2, 0.55, 0.2)][k][:d]
            xs.append(u * size * case["scale"] + torch.tensor(lo, device=DEV, dtype=torch.float64))
            g = torch.full((m,), L - 1, device=DEV, dtype=torch.int32)
            for l, edge in reversed(list(enumerate(((0.2, 0.1, 0.03) if d == 2 else (0.05, 0.01))[:L - 1]))):
                g[((u >= edge) & (u <= 1 - edge)).all(1)] = l
            gs.append(g)
        return torch.cat(xs), torch.cat(gs)
    xs = []
    for kind, a, b in _bodies(case):
        if kind == "box":
            ta, tb = (torch.tensor(t, device=DEV, dtype=torch.float64) for t in (a, b))
            xs.append(_lattice(d, finest, lambda p: ((p >= ta) & (p < tb)).all(1), a, b, gen))
        else:
            tc = torch.tensor(a, device=DEV, dtype=torch.float64)
            xs.append(_lattice(d, finest, lambda p: ((p - tc) ** 2).sum(1) < b * b, [q - b for q in a],
                               [q + b for q in a], gen))
    x = torch.cat(xs)
    return x, torch.full((len(x),), L - 1, device=DEV, dtype=torch.int32)


def _state(case, seed):
    """A body in mid-motion: float32 particle arrays on the GPU."""
    gen = _generator(seed)
    d, finest = case["dim"], case["coarsest"] << (case["level"] - 1)
    x, g = _positions(case, gen)
    x = x.float().clamp_(0.03, 0.97)
    n = len(x)
    r = torch.rand(64, generator=gen, device=DEV, dtype=torch.float64).tolist()
    fast = 20.0 if case["body"] == "demo" else 2.0
    v, C, F = torch.empty((n, d), device=DEV), torch.zeros((n, d, d), device=DEV), torch.empty((n, d, d), device=DEV)
    kv, kf = 9.0 + 4.0 * r[0], 14.0 + 5.0 * r[1]
    amp, strain = 0.3 * fast, 0.006 if case["snow"] else 0.03
    for i in range(d):
        j = (i + 1) % d
        ph = kv * x[:, j] + 6.28 * r[2 + i]
        v[:, i] = amp * torch.sin(ph) + fast * (r[6 + i] - 0.5)
        C[:, i, j] = amp * kv / finest * torch.cos(ph)
        for k in range(d):
            F[:, i, k] = strain * torch.sin(kf * x[:, (i + k) % d] + 6.28 * r[10 + 3 * i + k]) + float(i == k)
    s = dict(x=x, v=v, F=F, C=C, m=torch.ones(n, device=DEV), g=g,
             Jp=1.0 + 0.01 * torch.sin(kf * x[:, 0] + r[30]) if case["snow"] else torch.ones(n, device=DEV))
    return {k: t.contiguous() for k, t in s.items()}


def _coarse_levels(case, bodies):
    """A static level map constant on each coarsest cell: the finest level within two coarse cells of a body or
    below y = 0.25, the next within four, level 0 elsewhere."""
    d, c, L = case["dim"], case["coarsest"], case["level"]
    cov = torch.zeros((1, 1) + (c,) * d, device=DEV)
    for kind, a, b in bodies:
        lo, hi = (a, b) if kind == "box" else ([q - b for q in a], [q + b for q in a])
        cov[(0, 0) + tuple(slice(math.floor(p * c), math.ceil(q * c)) for p, q in zip(lo, hi))] = 1
    pool = nnf.max_pool2d if d == 2 else nnf.max_pool3d
    near, mid = (pool(cov, 2 * k + 1, 1, k)[0, 0] > 0 for k in (2, 4))
    low = ((torch.arange(c, device=DEV) + 0.5) / c < 0.25).reshape((1, c) + (1,) * (d - 2))
    lv = torch.where(mid, max(L - 2, 0), 0)
    return torch.where(near | low, L - 1, lv).to(torch.int8)


def _simulator(case, s):
    kw = dict(E=case["E"], nu=case["nu"], gravity=(0.0, case["gravity"], 0.0)[:case["dim"]],
              boundary_mode=case["boundary"], plasticity="snow" if case["snow"] else None,
              invalid_nodes="normalize" if case["normalize"] else "raw")
    return AdaptiveGIMP(case["dim"], case["level"], case["coarsest"], len(s["x"]), lambda sim: sim.set_particles(**s),
                        None, **kw)


def _scene_cases(case, seed):
    """The scenes of a batch: 2..4 levels, finest 256 or 512, one to three boxes, 2k..60k particles (lognormal).
    Their shapes are the case's own; the seed moves the particles."""
    rng = random.Random(7 * case["scenes"])
    out = []
    for i in range(case["scenes"]):
        L, fin, nb = rng.randint(2, 4), rng.choice((256, 512)), rng.randint(1, 3)
        n = min(max(rng.lognormvariate(math.log(12000.0), 0.8), 2000.0), 60000.0) * case["scale"]
        w = math.sqrt(n / 4.0 / nb) / fin  # side of each box: 4 particles per finest cell
        q = rng.uniform(0.7, 1.4)
        y = rng.uniform(0.15, 0.6)
        step = 0.8 / nb
        boxes = []
        for k in range(nb):
            wx, wy = min(w * q, 0.9 * step), w / q
            x0 = 0.1 + k * step + rng.uniform(0.0, step - wx)
            boxes.append(("box", [x0, y], [x0 + wx, min(y + wy, 0.95)]))
        out.append(dict(case, kind="sim", dim=2, level=L, coarsest=fin >> (L - 1), body="given", n=nb, boxes=boxes,
                        refine=False, static=True))
    return out


def _mlp_inputs(case, seed):
    """Trial states around the yield surface: features of the sizes the snow scenes hand over."""
    gen = _generator(seed)
    n = case["rows"]
    X = torch.randn((n, 7), generator=gen, device=DEV) * torch.tensor([.6, .5, .6, .3, .2, .0, .0], device=DEV)
    T = torch.stack([-0.8 * X[:, 0].clamp(min=0.15), -0.5 * X[:, 1].clamp(min=0.15), -0.8 * X[:, 2].clamp(max=-0.5),
                     0.7 * X[:, :3].sum(1)], 1).contiguous()
    k = [(7, 64), (64,), (64, 64), (64,), (64, 4), (4,)]
    P = [torch.randn(s, generator=gen, device=DEV) * ((1.0 / s[0]) ** 0.5 if len(s) == 2 else 0.1) for s in k]
    return X, T, torch.cat([p.reshape(-1) for p in P])


# ---------------------------------------------------------------------------
def prepare(case, seed):
    if case["kind"] == "sim":
        s = _state(case, seed)
        sim = _simulator(case, s)
        if case["static"]:
            sim.set_coarse_level_map(_coarse_levels(case, _bodies(case)).cpu().numpy())
        up = {k: s[k] for k in ("x", "v", "F", "C") + (("Jp",) if case["snow"] else ())}
        return dict(case=case, sim=sim, up=up)
    if case["kind"] == "batch":
        scenes = _scene_cases(case, seed)
        states = [_state(sc, int(seed) * 1000 + i) for i, sc in enumerate(scenes)]
        sims = []
        for sc, s in zip(scenes, states):
            sim = _simulator(sc, s)
            sim.set_coarse_level_map(_coarse_levels(sc, _bodies(sc)).cpu().numpy())
            sims.append(sim)
        batch = SceneBatch(sims)
        up = {k: torch.cat([s[k] for s in states]) for k in ("x", "v", "F", "C")}
        out = torch.empty(up["x"].shape, pin_memory=True).numpy()
        return dict(case=case, sims=sims, batch=batch, up=up, out=out)
    X, T, P = _mlp_inputs(case, seed)
    mlp = MLP(params=P.cpu().numpy())
    return dict(case=case, mlp=mlp, X=X, T=T, grad=torch.empty(mlp.nparam, device=DEV),
                loss=torch.empty(1, device=DEV))


def run(state):
    case = state["case"]
    if case["kind"] == "sim":
        sim = state["sim"]
        sim.set_particles(**state["up"])
        if case["refine"]:
            sim.refine_levels(3)
        sim.substep(case["dt"], case["substeps"])
        out = dict(x=sim.x_p.to_torch(), v=sim.v_p.to_torch(), F=sim.F_p.to_torch(), C=sim.C_p.to_torch())
        if case["snow"]:
            out["Jp"] = sim.Jp.to_torch()
        if case["refine"]:
            out["g"] = sim.g_p.to_torch()
        if case["substeps"] == 1:
            out["fl"] = sim.fl_p.to_torch()
        return out
    if case["kind"] == "batch":
        state["batch"].set_particles(**state["up"])
        state["batch"].substep(case["dt"], case["substeps"])
        return state["batch"].positions(state["out"], blocking=False)
    m, X = state["mlp"], state["X"]
    if case["kind"] == "mlp_forward":
        return m.forward(X)
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    m._L.agimp_mlp_grad(m._h, *(ctypes.c_void_p(t.data_ptr()) for t in (X, state["T"])), len(X),
                        *(ctypes.c_void_p(t.data_ptr()) for t in (state["grad"], state["loss"])), st)
    return dict(grad=state["grad"], loss=state["loss"])


def _count(case):
    """Particles of a scene (lattice places inside its shapes)."""
    if case["body"] == "demo":
        return case["n"]
    total, h = 0, 0.5 / (case["coarsest"] << (case["level"] - 1))
    for kind, a, b in _bodies(case):
        if kind == "box":
            total += math.prod((q - p) / h for p, q in zip(a, b))
        else:
            total += (math.pi * b * b if case["dim"] == 2 else 4.0 / 3.0 * math.pi * b ** 3) / h ** case["dim"]
    return int(total)


def work(case):
    """Each substep reads and writes every particle once (P2G x, v, F, C, m; G2P x, F in, x, v, C, F out; Jp with
    snow); the state goes in and comes out once.  Flops: the 3^d stencil both ways, the stress and the F update."""
    if case["kind"].startswith("mlp"):
        per = 7 * 64 + 64 * 64 + 64 * 4
        fwd = case["kind"] == "mlp_forward"
        return dict(bytes=44 * case["rows"], flops=2 * per * case["rows"] * (1 if fwd else 3))
    scenes = _scene_cases(case, 0) if case["kind"] == "batch" else [case]
    total = dict(bytes=0, flops=0)
    for sc in scenes:
        d, n = sc["dim"], _count(sc)
        per = 4 * (2 * d + 2 * d * d + 1) + 4 * (3 * d + 3 * d * d) + (12 if sc["snow"] else 0)
        state = 4 * (2 * d + 2 * d * d)
        total["bytes"] += n * (per * case["substeps"] + 2 * state + (d * 4 + 4 if sc["refine"] else 0))
        total["flops"] += n * case["substeps"] * (3 ** d * (4 * d + 2) * 2 + 40 * d)
    return total


# ---------------------------------------------------------------------------
# the same in 64 bits
def exact(case, seed):
    if case["kind"].startswith("mlp"):
        return _exact_mlp(case, seed)
    if case["kind"] == "batch":
        return None  # hundreds of scenes one after another take far over 20 seconds
    s = _state(case, seed)
    lv = _coarse_levels(case, _bodies(case)) if case["static"] else None
    g = s["g"].long()
    if case["refine"]:
        g = _exact_levels(case, s["x"], 3)
    q = {k: s[k].double() for k in ("x", "v", "F", "C", "Jp")}
    fl = None
    for _ in range(case["substeps"]):
        fl = _exact_substep(case, q, g, lv)
    out = dict(x=q["x"], v=q["v"], F=q["F"], C=q["C"])
    if case["snow"]:
        out["Jp"] = q["Jp"]
    if case["refine"]:
        out["g"] = g
    if case["substeps"] == 1:
        out["fl"] = fl
    return out


def _exact_mlp(case, seed):
    X, T, P = _mlp_inputs(case, seed)
    k, o, W = [(7, 64), (64,), (64, 64), (64,), (64, 4), (4,)], 0, []
    for s in k:
        n = math.prod(s)
        W.append(P[o:o + n].double().reshape(s).requires_grad_(True))
        o += n
    h = nnf.silu(X.double() @ W[0] + W[1])
    y = nnf.silu(h @ W[2] + W[3]) @ W[4] + W[5]
    if case["kind"] == "mlp_forward":
        return y.detach()
    loss = ((y - T.double()) ** 2).sum(1).mean()
    g = torch.autograd.grad(loss, W)
    return dict(grad=torch.cat([t.reshape(-1) for t in g]), loss=loss.detach().reshape(1))


def _exact_levels(case, x, band):
    """Prescribed levels from the Chebyshev depth of a particle's finest cell below the free surface."""
    d, L = case["dim"], case["level"]
    sz = case["coarsest"] << (L - 1)
    cell = (x * sz).long()
    empty = torch.ones((1, 1) + (sz,) * d, device=DEV)
    empty[(0, 0) + tuple(cell.T)] = 0
    g = torch.zeros(len(x), dtype=torch.long, device=DEV)
    pool = nnf.max_pool2d if d == 2 else nnf.max_pool3d
    for k in reversed(range(L - 1)):
        t = band * (2 ** (k + 1) - 1)
        e = nnf.pad(empty, (t, t) * d, value=1.0)
        for a in range(d):
            e = pool(e, tuple(2 * t + 1 if b == a else 1 for b in range(d)), 1)
        g[e[(0, 0) + tuple(cell.T)] > 0] = L - 1 - k
    return g


def _corners(d, n=2):
    return [tuple((a // n ** (d - 1 - k)) % n for k in range(d)) for a in range(n ** d)]


def _polar(F):
    X = F.clone()
    for _ in range(20):
        X = 0.5 * (X + torch.linalg.inv(X).transpose(1, 2))
    return X


def _eigen(E):
    """Eigenvalues and eigenvectors of symmetric matrices [n, d, d] (cyclic Jacobi)."""
    d = E.shape[1]
    E, V = E.clone(), torch.eye(d, device=E.device, dtype=E.dtype).expand_as(E).clone()
    for _ in range(8):
        for i, j in [(a, b) for a in range(d) for b in range(a + 1, d)]:
            th = 0.5 * torch.atan2(2 * E[:, i, j], E[:, j, j] - E[:, i, i])
            R = torch.eye(d, device=E.device, dtype=E.dtype).repeat(len(E), 1, 1)
            R[:, i, i], R[:, j, j], R[:, i, j], R[:, j, i] = th.cos(), th.cos(), th.sin(), -th.sin()
            E, V = R.transpose(1, 2) @ E @ R, V @ R
    return E.diagonal(dim1=1, dim2=2), V


def _exact_substep(case, q, g, lv):
    d, L, c, dt = case["dim"], case["level"], case["coarsest"], case["dt"]
    sz, H = c << (L - 1), 4
    x, x32 = q["x"], q["x"].float()

    def at(t, I):  # an array stored over [-4, size + 8) at indices I [..., d]
        return t[tuple((I + H).unbind(-1))]

    def base(l):  # base cells as 32-bit positions give them
        return (x32 * float(c << l) + 0.5).long() - 1

    size = [c << l for l in range(L)]
    corner = torch.tensor(_corners(d), device=DEV)
    act = [torch.zeros((s + 12,) * d, dtype=torch.bool, device=DEV) for s in size]

    def put(t, I, value=True):
        t[tuple((I + H).unbind(-1))] = value

    # active cells
    if lv is None:
        for l in range(L):
            b = base(l)[g == l]
            for o in corner:
                put(act[l], b + o)
        cul = [torch.zeros_like(a) for a in act]
        for l in range(1, L):
            I = act[l].nonzero() - H
            l0 = torch.full((len(I),), -1, device=DEV)
            for p in range(l):
                l0 = torch.where(at(act[p], I >> (l - p)), p, l0)
            for p in range(l):
                put(cul[p], (I >> (l - p))[(l0 >= 0) & (p >= l0)])
        for l in range(L):
            if l:
                K = cul[l - 1].nonzero() - H
                for o in corner:
                    J = 2 * K + o
                    put(act[l], J[((J >= -H) & (J < size[l] + 8)).all(1)])
            act[l] &= ~cul[l]
    else:
        def look(I):  # level of a finest cell, its cell activated inside the domain
            inr = ((I >= 0) & (I < sz)).all(-1)
            lev = torch.where(inr, lv.long()[tuple((I.clamp(0, sz - 1) >> (L - 1)).unbind(-1))], L - 1)
            for l in range(L):
                put(act[l], (I >> (L - 1 - l))[inr & (lev == l)])
            return lev
        fb = base(L - 1)
        for o in _corners(d, 4):
            look(fb + torch.tensor(o, device=DEV) - 1)
        lev = look(fb)
        for l in range(L):
            b = base(l)[lev == l]
            for o in corner:
                look((b + o) * (1 << (L - 1 - l)))
    # node classes on the finest lattice [0, sz]: 1 activated, 2 ghost, 4 T-junction
    nm = torch.zeros((sz + 1,) * d, dtype=torch.uint8, device=DEV)

    def mark(l, J, bit, only_empty=False):
        P = J * (1 << (L - 1 - l))
        P = P[((P >= 0) & (P <= sz)).all(-1)]
        w = tuple(P.unbind(-1))
        if only_empty:
            e = nm[w] == 0
            w = tuple(t[e] for t in w)
        nm[w] |= bit

    faces, ghosts = [], []
    for l in range(L):
        I = act[l].nonzero() - H
        for o in corner:
            mark(l, I + o, 1)
    for l in range(1, L):
        I = act[l].nonzero() - H
        for f in range(2 * d):
            ax, side = f >> 1, f & 1
            I1 = I.clone()
            I1[:, ax] += -1 if side else 1
            I1 = I1[((I1 >= 0) & (I1 < size[l])).all(1)]
            I1 = I1[~at(act[l], I1)]
            lp = torch.full((len(I1),), -1, device=DEV)
            for p in range(l):
                lp = torch.where(at(act[p], I1 >> (l - p)), p, lp)
            I1, lp = I1[lp >= 0], lp[lp >= 0]
            for o in _corners(d):
                J = I1 + torch.tensor(o, device=DEV)
                if o[ax] == side:
                    faces.append((l, J[((J & ((1 << (l - lp)) - 1)[:, None]) != 0).any(1)]))
                for p in range(1, l + 1):
                    ghosts.append((p, (I1[lp < p] >> (l - p)) + torch.tensor(o, device=DEV)))
    for l, J in faces:
        mark(l, J, 4)
    for l, J in ghosts:
        mark(l, J, 2, only_empty=True)
    # levels of the particles
    fl = torch.full((len(x),), -1, device=DEV)
    for l in range(L):
        b = base(l)
        hit = torch.zeros(len(x), dtype=torch.bool, device=DEV)
        for o in corner:
            hit |= at(act[l], b + o)
        fl = torch.where(hit, l, fl)
    # particles to grid
    mu, la = case["E"] / (2 * (1 + case["nu"])), case["E"] * case["nu"] / ((1 + case["nu"]) * (1 - 2 * case["nu"]))
    hard = torch.exp(10.0 * (1 - q["Jp"])) if case["snow"] else torch.ones_like(q["Jp"])
    J = torch.linalg.det(q["F"])
    S = (2 * mu * hard)[:, None, None] * (q["F"] - _polar(q["F"])) @ q["F"].transpose(1, 2) + \
        (la * hard * J * (J - 1))[:, None, None] * torch.eye(d, device=DEV, dtype=torch.float64)
    grid = [torch.zeros(((s + 12) ** d, d + 1), dtype=torch.float64, device=DEV) for s in size]
    stencil = []
    for l in range(L):
        p = (fl == l).nonzero()[:, 0]
        b = base(l)[p]
        t = x[p] * (c << l) - (b + 1)
        W = [(0.5 - t) ** 2, 1.5 - 2 * t * t, (0.5 + t) ** 2]
        G = [t - 0.5, -2 * t, t + 0.5]
        lin = torch.zeros(len(p), dtype=torch.long, device=DEV)
        for k in range(d):
            lin = lin * (size[l] + 12) + b[:, k] + H
        stencil.append((p, t, W, G, lin))

    def nodes(l):  # every stencil node: flat index, weight, gradient, offset
        p, t, W, G, lin = stencil[l]
        for o in _corners(d, 3):
            w = math.prod([W[o[k]][:, k] for k in range(1, d)], start=W[o[0]][:, 0]) / 2 ** d
            dw = torch.stack([math.prod([(G if k == a else W)[o[k]][:, k] for k in range(1, d)],
                                        start=(G if a == 0 else W)[o[0]][:, 0]) for a in range(d)], 1) / 2 ** (d - 1)
            off = 0
            for k in range(d):
                off = off * (size[l] + 12) + o[k]
            yield lin + off, w, dw, torch.tensor(o, device=DEV, dtype=torch.float64) - (t + 1)

    for l in range(L):
        p = stencil[l][0]
        Sp = -dt * (c << l) * S[p]
        for i, w, dw, dpos in nodes(l):
            mom = w[:, None] * (q["v"][p] + (q["C"][p] @ dpos[:, :, None])[:, :, 0]) + (Sp @ dw[:, :, None])[:, :, 0]
            grid[l].index_add_(0, i, torch.cat([mom, w[:, None]], 1))
    grid = [t.reshape((s + 12,) * d + (d + 1,)) for t, s in zip(grid, size)]
    dom = [t[tuple(slice(H, H + s + 1) for _ in range(d))] for t, s in zip(grid, size)]  # nodes [0, size]
    cls = [nm[tuple(slice(None, None, 1 << (L - 1 - l)) for _ in range(d))] for l in range(L)]
    isact = [(t & 5) == 1 for t in cls]
    tg = [((t & 4) == 4) | ((t & 7) == 2) for t in cls]

    # restriction, fine to coarse
    for l in range(L - 1, 0, -1):
        f = nnf.pad(torch.where(tg[l][..., None], dom[l], 0.0), (0, 0) + (1, 1) * d)
        add = torch.where(isact[l][..., None], dom[l], 0.0)[tuple(slice(None, None, 2) for _ in range(d))].clone()
        for o in _corners(d, 3):
            w = 0.5 ** sum(k != 1 for k in o)
            add += w * f[tuple(slice(k, k + 2 * size[l - 1] + 1, 2) for k in o)]
        dom[l - 1] += torch.where((cls[l - 1] > 0)[..., None], add, 0.0)
    # grid update
    for l in range(L):
        mass = dom[l][..., d:]
        has = mass > 0
        vel = dom[l][..., :d] / torch.where(has, mass, 1.0)
        upd = vel.clone()
        upd[..., 1] += case["gravity"] * dt
        P = torch.arange(size[l] + 1, device=DEV) * (1 << (L - 1 - l))
        band = (P < 4) | (P > sz - 4)
        wall = [band.reshape([-1 if k == a else 1 for k in range(d)]) for a in range(d)]
        for a in range(d):
            w = wall[a] if case["boundary"] == "ref_slip" else math.prod([~t for t in wall[1:]], start=~wall[0]) == 0
            upd[..., a] = torch.where(w, 0.0, upd[..., a])
        rest = vel if case["normalize"] else dom[l][..., :d]
        new = torch.where(isact[l][..., None], upd, rest)
        dom[l][..., :d] = torch.where(has, new, dom[l][..., :d])
    # prolongation, coarse to fine
    for l in range(1, L):
        up = torch.where((cls[l - 1] > 0)[..., None], dom[l - 1][..., :d], 0.0)
        even = torch.ones((), dtype=torch.bool, device=DEV)
        for a in range(d):
            n = up.shape[a]
            mid = 0.5 * (up.narrow(a, 0, n - 1) + up.narrow(a, 1, n - 1))
            both = torch.stack([up.narrow(a, 0, n - 1), mid], a + 1).flatten(a, a + 1)
            up = torch.cat([both, up.narrow(a, n - 1, 1)], a)
            even = even & (torch.arange(size[l] + 1, device=DEV) % 2 == 0).reshape([-1 if k == a else 1 for k in range(d)])
        keep = torch.where(even[..., None], torch.where(isact[l][..., None], up, 0.0), dom[l][..., :d])
        dom[l][..., :d] = torch.where(tg[l][..., None], up, keep)
    # grid to particles
    for l in range(L):
        p = stencil[l][0]
        v, C = torch.zeros_like(q["v"][p]), torch.zeros_like(q["C"][p])
        flat = grid[l].reshape(-1, d + 1)
        for i, w, dw, _ in nodes(l):
            gv = flat[i, :d]
            v += w[:, None] * gv
            C += gv[:, :, None] * dw[:, None, :]
        q["v"][p], q["C"][p] = v, C
        q["x"][p] += dt * v
        q["F"][p] = (torch.eye(d, device=DEV, dtype=torch.float64) + dt * (c << l) * C) @ q["F"][p]
    if case["snow"]:
        lo, hi, F = 1 - 2.5e-2, 1 + 7.5e-3, q["F"]
        E = F.transpose(1, 2) @ F
        out = (E.diagonal(dim1=1, dim2=2) + (E.abs().sum(2) - E.diagonal(dim1=1, dim2=2).abs())).amax(1) > hi * hi
        out |= (E.diagonal(dim1=1, dim2=2) - (E.abs().sum(2) - E.diagonal(dim1=1, dim2=2).abs())).amin(1) < lo * lo
        p = out.nonzero()[:, 0]
        w, V = _eigen(E[p])
        s = w.sqrt()
        cl = s.clamp(lo, hi)
        F[p] = F[p] @ (V * (cl / s)[:, None, :]) @ V.transpose(1, 2)
        q["Jp"][p] *= s.prod(1) / cl.prod(1)
    return fl
