"""The work that is timed: what a program that uses this framework has it do,
through its public entry points (mfgpu.Context, Level, Hier, Server).

Kinds of case:
  patch   one mf_patch_update call: the drop-in for the reference's per-patch
          updateState, at the patch sizes of a block-structured mesh
  level   one step of a level of patches resident on the device: chained
          asynchronous steps (a production time loop) or the synchronous call
          whose dt the program reads (a driver that plans its own steps)
  hier    one step of a coupled three-level hierarchy
  serve   a batch of requests of the serving engine, host state in, host
          state out, with a few steps between

Problems: the Orszag-Tang vortex (single-fluid MHD, periodic) and the
four-fluid heliosphere (plasma, three neutral populations, GLM, charge
exchange, inner wind sphere, far-field sides), each with seeded smooth
disturbances so that no two seeds hold the same state.  exact() evaluates the
RK2 step of both in 64-bit torch.
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "ms-flukss-multifluid_gb300"))

import mfgpu  # noqa: E402
from mfgpu import amr, serving  # noqa: E402

DEVICE = "cuda" if torch.cuda.is_available() else "cpu"
CFL = 0.4
PREC = {"fp64": mfgpu.PREC_FP64, "fast": mfgpu.PREC_FP64_FAST, "mixed": mfgpu.PREC_MIXED,
        "ce32": mfgpu.PREC_MIXED_CE32}
TIME = {"rk2": mfgpu.TA_RK2, "hancock": mfgpu.TA_HANCOCK}


def listed():
    return [
        # a small 2D patch, one call: latency and launches
        {"name": "patch_orszag_32", "kind": "patch", "problem": "orszag", "n": 32,
         "prec": "fp64", "fluxes": False},
        # a 16^3 patch of the multi-fluid model with its fluxes out for the
        # flux registers: the call an AMR driver makes per patch
        {"name": "patch_helio_16", "kind": "patch", "problem": "helio", "n": 16,
         "prec": "fp64", "fluxes": True},
        # the 256^2 vortex as one patch, the parity precision
        {"name": "orszag_256", "kind": "level", "problem": "orszag", "n": 256, "cuts": "256",
         "prec": "fp64", "time": "rk2", "ct": 0, "sync": False},
        # a larger 2D level in uneven patches, mixed precision, dt read back
        {"name": "orszag_500_mixed", "kind": "level", "problem": "orszag", "n": 500,
         "cuts": "128,93,150,129", "prec": "mixed", "time": "rk2", "ct": 0, "sync": True},
        # the 128^3 heliosphere in 512 patches of 16^3: the production run
        {"name": "helio_128", "kind": "level", "problem": "helio", "n": 128, "cuts": "16",
         "prec": "fp64", "time": "rk2", "ct": 0, "sync": False},
        {"name": "helio_128_mixed", "kind": "level", "problem": "helio", "n": 128, "cuts": "16",
         "prec": "mixed", "time": "rk2", "ct": 0, "sync": False},
        # a medium run in the fast FP64 form
        {"name": "helio_64_fast", "kind": "level", "problem": "helio", "n": 64, "cuts": "16",
         "prec": "fast", "time": "rk2", "ct": 0, "sync": False},
        # a small run in uneven, odd patches, the driver reading dt
        {"name": "helio_46_ragged", "kind": "level", "problem": "helio", "n": 46,
         "cuts": "9,21,16", "prec": "fp64", "time": "rk2", "ct": 0, "sync": True},
        # the Hancock predictor-corrector
        {"name": "helio_48_hancock", "kind": "level", "problem": "helio", "n": 48, "cuts": "16",
         "prec": "fp64", "time": "hancock", "ct": 0, "sync": False},
        # constrained transport of the magnetic field
        {"name": "orszag_192_ct", "kind": "level", "problem": "orszag", "n": 192, "cuts": "64",
         "prec": "fp64", "time": "rk2", "ct": 1, "sync": False},
        # three coupled refinement levels, subcycled
        {"name": "hier_32", "kind": "hier", "n": 32, "prec": "fp64"},
        # six requests of the serving engine
        {"name": "serve_2d", "kind": "serve", "problem": "orszag", "sizes": "64,96,160,128,224,64",
         "steps": 6, "prec": "mixed"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _pieces(rng, n, k):
    """n cut into k uneven pieces of at least 8 cells."""
    left, out = n, []
    for i in range(k - 1, 0, -1):
        p = rng.randint(8, max(8, min(left - 8 * i, 2 * left // (i + 1))))
        out.append(p)
        left -= p
    return ",".join(str(p) for p in out + [left])


def draw(rng):
    kind = rng.choice(("patch", "patch", "level", "level", "level", "level", "hier", "serve"))
    if kind == "patch":
        problem = rng.choice(("orszag", "helio"))
        n = _log(rng, 16, 200) if problem == "orszag" else rng.randint(8, 32)
        return {"kind": kind, "problem": problem, "n": n,
                "prec": rng.choice(("fp64", "fp64", "fast", "mixed")),
                "fluxes": rng.random() < 0.5}
    if kind == "hier":
        return {"kind": kind, "n": 16 * rng.randint(1, 4), "prec": rng.choice(("fp64", "mixed"))}
    if kind == "serve":
        sizes = ",".join(str(_log(rng, 64, 256)) for _ in range(rng.randint(2, 8)))
        return {"kind": kind, "problem": "orszag", "sizes": sizes, "steps": rng.randint(2, 8),
                "prec": rng.choice(("fp64", "mixed"))}
    problem = rng.choice(("orszag", "helio", "helio"))
    time = rng.choice(("rk2", "rk2", "rk2", "hancock"))
    ct = 1 if problem == "orszag" and rng.random() < 0.25 else 0
    n = _log(rng, 64, 700) if problem == "orszag" else 2 * _log(rng, 20, 56)
    cuts = _pieces(rng, n, rng.randint(2, 3)) if rng.random() < 0.6 else \
        str(rng.choice([p for p in (8, 10, 12, 14, 16, 20, 22, 32, 64, n) if n % p == 0]))
    prec = rng.choice(("fp64", "fp64", "fast", "mixed", "ce32"))
    return {"kind": kind, "problem": problem, "n": n, "cuts": cuts, "prec": prec, "time": time,
            "ct": ct, "sync": rng.random() < 0.5}


# ---------------------------------------------------------------------------
# parameters, geometry, initial states
# ---------------------------------------------------------------------------
def params(case):
    prec, ta = PREC[case["prec"]], TIME[case.get("time", "rk2")]
    n = case["n"]
    if case.get("kind") == "hier":
        return amr.orszag3d_params(n, ta, prec)
    if case["problem"] == "orszag":
        p = mfgpu.orszag_params(n, ta, prec)
        if case.get("ct"):
            p.divb_cleaning, p.use_8wave = 1, 0
        return p
    # a patch case is one patch of a mesh of 128^3 cells
    return mfgpu.helio_params(128 if case["kind"] == "patch" else n, time_approximation=ta,
                              precision=prec)


def cut_boxes(n, cuts, sd):
    """Valid boxes of the domain cut alike in each direction (x fastest);
    one number: equal pieces of that length."""
    c = [int(x) for x in cuts.split(",")]
    c = c if len(c) > 1 else [c[0]] * (n // c[0])
    e = np.concatenate([[0], np.cumsum(c)]).tolist()
    assert e[-1] == n
    r = range(len(c))
    return [([e[i], e[j], e[k] if sd == 3 else 0],
             [e[i + 1] - 1, e[j + 1] - 1, e[k + 1] - 1 if sd == 3 else 0])
            for k in (r if sd == 3 else range(1)) for j in r for i in r]


def _axes(p, lo, hi):
    """Cell centres x, y, z on the box [lo, hi], broadcast to (nz, ny, nx)."""
    ax = [(torch.arange(lo[d], hi[d] + 1, device=DEVICE, dtype=torch.float64) + 0.5) * p.dx
          - p.sun_center[d] for d in range(3)]
    return ax[0][None, None, :], ax[1][None, :, None], ax[2][:, None, None]


def _cons(p, w):
    """Conserved state (list of component tensors) of primitives w."""
    h = p.gamma - 1.0
    mag = (w[5] ** 2 + w[6] ** 2 + w[7] ** 2) / (4.0 * math.pi)
    u = [w[0], w[0] * w[1], w[0] * w[2], w[0] * w[3],
         w[4] / h + 0.5 * (w[0] * (w[1] ** 2 + w[2] ** 2 + w[3] ** 2) + mag), w[5], w[6], w[7]]
    s = 8
    if len(w) % 5 == 4:
        u.append(w[8])
        s = 9
    for q in range(s, len(w), 5):
        r, a, b, c, e = w[q:q + 5]
        u += [r, r * a, r * b, r * c, e / h + 0.5 * r * (a * a + b * b + c * c)]
    return u


def orszag_fields(p, lo, hi, seed):
    """Orszag-Tang vortex with seeded phases and a weak third component."""
    r = np.random.RandomState(seed % (1 << 31))
    x, y, z = _axes(p, lo, hi)
    tp = 2.0 * math.pi
    a, f = r.uniform(-0.1, 0.1, 6), r.uniform(0.0, tp, 6)
    g = p.gamma
    p0 = g / (4.0 * math.pi)
    zero = torch.zeros_like(x + y + z)
    w = [p0 * g * (1.0 + a[0] * torch.sin(tp * (x + y) + f[0])) + zero,
         -torch.sin(tp * y + f[1]) * (1.0 + a[1]) + zero,
         torch.sin(tp * x + f[2]) * (1.0 + a[2]) + zero,
         0.1 * a[3] * torch.sin(tp * (x - y) + f[3]) + zero,
         p0 * (1.0 + a[4] * torch.cos(tp * (x - y) + f[4])) + zero,
         -torch.sin(tp * y + f[1]) + zero, torch.sin(2.0 * tp * x + f[2]) + zero,
         0.2 * a[5] * torch.sin(tp * (x + y) + f[5]) + zero]
    return torch.stack(_cons(p, w))


def wind(p, u, x, y, z, t):
    """The state inside the inner sphere: radial wind, spiral field whose
    sign changes across the equator (untilted current sheet)."""
    r2 = x * x + y * y + z * z
    r = torch.sqrt(r2)
    rr = r / p.sun_int_bc_radius
    xy = torch.sqrt(x * x + y * y)
    ct, cf, sf = z / r, x / xy, y / xy
    st = torch.sqrt(1.0 - ct * ct)
    rho = p.sun_rho / rr ** 2
    pr = p.sun_p / rr ** (2.0 * p.gamma)
    br = p.dir_br * p.sun_b / rr ** 2
    bp = -p.sun_beta * br * r * st
    s = torch.where(z > 0, 1.0, -1.0)
    b = [br * st * cf - bp * sf, br * st * sf + bp * cf, br * ct + 0.0 * r]
    e = pr / (p.gamma - 1.0) + 0.5 * (rho * p.sun_v ** 2
                                      + (b[0] ** 2 + b[1] ** 2 + b[2] ** 2) / (4.0 * math.pi))
    new = [rho, rho * p.sun_v * st * cf, rho * p.sun_v * st * sf, rho * p.sun_v * ct, e,
           s * b[0], s * b[1], s * b[2]]
    inside = r2 <= p.reinit_r0 ** 2
    for q in range(8):
        u[q] = torch.where(inside, new[q], u[q])


def helio_fields(p, lo, hi, seed):
    """Interstellar inflow with seeded smooth disturbances of every fluid
    around the inner wind sphere."""
    r = np.random.RandomState(seed % (1 << 31))
    x, y, z = _axes(p, lo, hi)
    zero = torch.zeros_like(x + y + z)

    def mode(amp, axes=(1, 1, 1)):
        k = [int(v) * m for v, m in zip(r.randint(1, 4, 3), axes)]
        return amp * r.uniform(0.4, 1.0) * torch.sin(
            math.pi * (k[0] * x + k[1] * y + k[2] * z) + r.uniform(0.0, 2.0 * math.pi)) + zero

    wp, wn = mfgpu.helio_inflow()
    w = [wp[0] * (1.0 + mode(0.1))] + [wp[1 + d] + mode(0.1) for d in range(3)]
    w += [wp[4] * (1.0 + mode(0.1))]
    w += [wp[5 + d] + mode(0.01, [int(e != d) for e in range(3)]) for d in range(3)]
    w += [zero]
    for f in range(3):
        q = wn[5 * f:5 * f + 5]
        w += [q[0] * (1.0 + mode(0.1))] + [q[1 + d] + mode(0.1) for d in range(3)]
        w += [q[4] * (1.0 + mode(0.1))]
    u = _cons(p, w)
    wind(p, u, x, y, z, 0.0)
    return torch.stack(u)


def fields(case, p, lo, hi, seed):
    return (orszag_fields if case["problem"] == "orszag" else helio_fields)(p, lo, hi, seed)


# ---------------------------------------------------------------------------
# device memory of a level as tensors
# ---------------------------------------------------------------------------
class _Window:
    """A level's memory for torch; holds the level, so that a tensor over it
    never outlives it."""

    def __init__(self, level, ptr, n):
        self.level = level
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<f8", "data": (ptr, False),
                                         "version": 3, "strides": None}


def valid_views(level):
    """Tensors over the valid cells of every patch: one (patch, component, z,
    y, x) tensor where all patches have one shape, else one per patch."""
    ng, sd, nc = level.ctx.ng, level.ctx.p.space_dim, level.ctx.nc
    flat = torch.as_tensor(_Window(level, level.patch_fab_ptr(0), level.ndoubles), device="cuda")
    shapes = [tuple(hi[d] - lo[d] + 1 for d in (2, 1, 0)) for lo, hi in level.boxes]
    g = (ng if sd == 3 else 0, ng, ng)

    def window(count, off, shape, step):
        f = [shape[d] + 2 * g[d] for d in range(3)]
        s = (f[1] * f[2], f[2], 1)
        o = off + sum(g[d] * s[d] for d in range(3))
        return torch.as_strided(flat, (count, nc) + shape, (step, f[0] * f[1] * f[2]) + s, o)

    off = level.offsets
    if len(set(shapes)) == 1:
        return [window(len(off), off[0], shapes[0], off[1] - off[0] if len(off) > 1 else 0)]
    return [window(1, o, s, 0)[0] for o, s in zip(off, shapes)]


def fill(views, boxes, U):
    """Copy the domain state U (nc, z, y, x) into a level's valid cells."""
    if len(views) == 1:
        v, n = views[0], len(boxes)
        c = tuple(v.shape[2:])
        nb = [U.shape[1 + d] // c[d] for d in range(3)]
        assert nb[0] * nb[1] * nb[2] == n
        t = U.reshape(U.shape[0], nb[0], c[0], nb[1], c[1], nb[2], c[2])
        v.copy_(t.permute(1, 3, 5, 0, 2, 4, 6).reshape(v.shape))
        return
    for v, (lo, hi) in zip(views, boxes):
        v.copy_(U[:, lo[2]:hi[2] + 1, lo[1]:hi[1] + 1, lo[0]:hi[0] + 1])


def gather(boxes, U):
    """U laid out as valid_views(...)."""
    parts = [U[:, lo[2]:hi[2] + 1, lo[1]:hi[1] + 1, lo[0]:hi[0] + 1] for lo, hi in boxes]
    return [torch.stack(parts)] if len({tuple(t.shape) for t in parts}) == 1 else parts


# ---------------------------------------------------------------------------
# prepare
# ---------------------------------------------------------------------------
def patch_boxes(case, p):
    """Valid box of a patch case (a helio patch crosses the wind sphere's
    edge) and the box of its fab."""
    n, sd, ng = case["n"], p.space_dim, mfgpu.num_ghost(p)
    lo = [0, 0, 0] if sd == 2 else [66, 60, 52]
    hi = [lo[d] + (n - 1 if d < sd else 0) for d in range(3)]
    return (lo, hi), mfgpu.grow(lo, hi, ng, sd)


def inner(U, g, sd):
    return U[..., slice(g, -g) if sd == 3 else slice(None), g:-g, g:-g] if g else U


def hier_boxes(n):
    """Three levels: the domain, its middle half and the middle quarter."""
    def cube(lo, hi, s):
        r = range(lo, hi, s)
        return [((i, j, k), (i + s - 1, j + s - 1, k + s - 1)) for k in r for j in r for i in r]
    return [cube(0, n, n // 3 if n == 48 else n // 2), cube(n // 2, 3 * n // 2, n // 2),
            cube(3 * n // 2, 5 * n // 2, n // 2)]


def prepare(case, seed):
    stream = torch.cuda.current_stream().cuda_stream
    if case["kind"] == "serve":
        p = serving.physics_params(2, PREC[case["prec"]])
        ctx = mfgpu.Context(p)
        server = mfgpu.Server(ctx, 2.0e9, max_runs=16)
        requests = []
        for k, n in enumerate(int(s) for s in case["sizes"].split(",")):
            q = serving.run_physics(p, n)
            U = orszag_fields(q, [0, 0, 0], [n - 1, n - 1, 0], seed + 101 * k).cpu().numpy()
            requests.append((mfgpu.run_spec([n, n], serving.PATCH[2], 1.0 / n, CFL), U))
        return {"kind": "serve", "server": server, "requests": requests, "steps": case["steps"],
                "stream": stream}
    p = params(case)
    if case["kind"] == "hier":
        ps = [p, amr.level_params(p, 2), amr.level_params(p, 4)]
        eps = 0.1 + 0.2 * np.random.RandomState(seed % (1 << 31)).rand()
        h = amr.DeviceHierarchy(mfgpu, ps, hier_boxes(case["n"]), [2, 2],
                                lambda q, lo, hi: amr.orszag3d_state(q, lo, hi, eps))
        views = [v for lev in h.levels for v in valid_views(lev)]
        return {"kind": "hier", "hier": h, "views": views, "dt": CFL * h.compute_dt(),
                "stream": stream}
    ctx = mfgpu.Context(p)
    if case["kind"] == "patch":
        (lo, hi), (flo, fhi) = patch_boxes(case, p)
        sd = p.space_dim
        U0 = fields(case, p, flo, fhi, seed).contiguous()
        U = U0.clone()
        dt = CFL * wave_dt(p, inner(U0, ctx.ng, sd))
        F = None
        if case["fluxes"]:
            F = []
            for d in range(sd):
                fh = [hi[e] + (1 if e == d else 0) for e in range(3)]
                F.append((torch.zeros(mfgpu.fab_shape(lo, fh, ctx.nc), dtype=torch.float64,
                                      device="cuda"), lo, fh))
        torch.cuda.synchronize()
        return {"kind": "patch", "ctx": ctx, "U": U, "U0": U0, "boxes": (flo, fhi, lo, hi),
                "dt": dt, "F": F, "valid": inner(U, ctx.ng, sd), "stream": stream}
    sd, n = p.space_dim, case["n"]
    boxes = cut_boxes(n, case["cuts"], sd)
    level = mfgpu.Level(ctx, boxes)
    views = valid_views(level)
    fill(views, boxes, fields(case, p, [0, 0, 0], [n - 1, n - 1, n - 1 if sd == 3 else 0], seed))
    torch.cuda.synchronize()
    level.autotune(3)
    dt = CFL * level.compute_dt()[0]
    if not case["sync"]:
        level.seed_dt(dt, CFL, stream)
    return {"kind": "level", "level": level, "views": views, "dt": dt, "sync": case["sync"],
            "stream": stream}


# ---------------------------------------------------------------------------
# run
# ---------------------------------------------------------------------------
def run(s):
    if s["kind"] == "patch":
        s["U"].copy_(s["U0"])  # the driver's copy of the patch it is about to update
        F = s["F"] and [(t.data_ptr(), lo, hi) for t, lo, hi in s["F"]]
        _, dt, _ = s["ctx"].patch_update(s["U"].data_ptr(), *s["boxes"], s["dt"], F=F,
                                         stream=s["stream"])
        return {"U": s["valid"], "F": [t for t, _, _ in s["F"]] if F else [], "dt": dt}
    if s["kind"] == "level":
        if not s["sync"]:
            s["level"].step_async(s["stream"])
            return {"U": s["views"]}
        _, dt, _, _ = s["level"].step(s["dt"], s["stream"])
        s["dt"] = CFL * dt
        return {"U": s["views"], "dt": dt}
    if s["kind"] == "hier":
        dt = s["hier"].step(s["dt"], s["stream"])
        s["dt"] = CFL * dt
        return {"U": s["views"], "dt": dt}
    server = s["server"]
    ids = [server.admit(spec, U) for spec, U in s["requests"]]
    for _ in range(s["steps"]):
        server.step(s["stream"])
    server.sync(s["stream"])
    return {"U": [server.retire(i) for i in ids]}


# ---------------------------------------------------------------------------
# work: the conserved state read and written once a step; the operations of
# the scheme (add, multiply, divide and root one each) on each cell and face
# ---------------------------------------------------------------------------
ROE, VAN_LEER, LIMIT = 480, 75, 6          # a face; a face and neutral; a value and direction
PRIM, EXCHANGE, UPDATE = 20, 110, 3        # a fluid; a neutral; a value and direction


def work(case):
    if case["kind"] == "serve":
        cells = [int(n) ** 2 for n in case["sizes"].split(",")]
        sd, nc, nn, steps = 2, 8, 0, case["steps"]
    elif case["kind"] == "hier":
        cells = [sum(math.prod(b - a + 1 for a, b in zip(lo, hi)) for lo, hi in boxes) * 2 ** lv
                 for lv, boxes in enumerate(hier_boxes(case["n"]))]
        sd, nc, nn, steps = 3, 8, 0, 1
    else:
        helio = case["problem"] == "helio"
        sd, nc, nn = (3, 24, 3) if helio else (2, 8, 0)
        cells, steps = [case["n"] ** sd], 1
    flux = ROE + VAN_LEER * nn + 2 * LIMIT * nc + UPDATE * nc
    stage = sd * flux + PRIM * (1 + nn) + EXCHANGE * nn + 60
    stages = 1 if case.get("time") == "hancock" else 2
    out = 8.0 * nc * sum(cells) * sd if case.get("fluxes") else 0.0
    return {"bytes": 16.0 * nc * sum(cells) * steps + out,
            "flops": float(stage) * stages * sum(cells) * steps}


# ---------------------------------------------------------------------------
# exact: the RK2 step in 64 bits, on whole arrays
# ---------------------------------------------------------------------------
I4PI = 1.0 / (4.0 * math.pi)


def _fluids(p):
    return [(9 if p.divb_cleaning == 5 else 8) + 5 * f for f in range(p.n_fluids - 1)]


def prim(p, U):
    """Primitive variables of the conserved state."""
    W = U.clone()
    for s in [0] + _fluids(p):
        rho = U[s] if p.n_fluids == 1 else U[s].clamp(min=p.smallr)
        ke = (U[s + 1] ** 2 + U[s + 2] ** 2 + U[s + 3] ** 2) / rho
        mag = I4PI * (U[5] ** 2 + U[6] ** 2 + U[7] ** 2) if s == 0 else 0.0
        W[s] = rho
        W[s + 1:s + 4] = U[s + 1:s + 4] / rho
        W[s + 4] = ((p.gamma - 1.0) * (U[s + 4] - 0.5 * (ke + mag))).clamp(min=p.smallp)
    return W


def wave_dt(p, U):
    """dx over the largest signal speed."""
    W = prim(p, U)
    b = [I4PI * W[5 + d] ** 2 / W[0] for d in range(3)]
    a2 = p.gamma * W[4] / W[0]
    h = 0.5 * (a2 + b[0] + b[1] + b[2])
    top = torch.stack([W[1 + d].abs() + torch.sqrt(h + torch.sqrt(h * h - a2 * b[d]))
                       for d in range(3)]).max()
    for s in _fluids(p):
        v = W[s + 1:s + 4].abs().amax(0) + torch.sqrt(p.gamma * W[s + 4] / W[s])
        top = torch.maximum(top, v.max())
    return p.dx / float(top)


def padded(p, U):
    """Primitives of a domain state with two ghost layers on each side:
    periodic images, or the far-field state (the second and third neutral
    population continue the nearest cell's)."""
    W, sd = prim(p, U), p.space_dim
    fluids = _fluids(p)
    for d in range(sd):
        ax = 3 - d
        n = W.shape[ax]
        if p.periodic[d]:
            W = torch.cat([W.narrow(ax, n - 2, 2), W, W.narrow(ax, 0, 2)], ax)
            continue
        ends = []
        for at in (0, n - 1):
            g = W.narrow(ax, at, 1).clone()
            for q in range(8):
                g[q] = p.bc_plasma[q]
            g[8] = 0.0
            for q in range(5):
                g[fluids[0] + q] = p.bc_neutral1[q]
            ends.append(torch.cat([g, g], ax))
        W = torch.cat([ends[0], W, ends[1]], ax)
    return W


def roe(p, L, R, d, seven):
    """Roe flux of ideal MHD (eight waves, or seven with the normal field
    held), arithmetic averages."""
    n, s, t = d, (d + 1) % 3, (d + 2) % 3
    g, h = p.gamma, p.gamma - 1.0

    def side(w):
        rho, v, b, pg = w[0], [w[1 + e] for e in (n, s, t)], [w[5 + e] for e in (n, s, t)], w[4]
        rho, pg = rho.clamp(min=p.smallr), pg.clamp(min=p.smallp)
        m = [rho * x for x in v]
        mag = 0.5 * I4PI * (b[0] ** 2 + b[1] ** 2 + b[2] ** 2)
        e = pg / h + 0.5 * (m[0] * v[0] + m[1] * v[1] + m[2] * v[2]) + mag
        pt = pg + mag
        vb = v[0] * b[0] + v[1] * b[1] + v[2] * b[2]
        f = [m[0], v[0] * m[0] - b[0] * b[0] * I4PI + pt, v[0] * m[1] - b[0] * b[1] * I4PI,
             v[0] * m[2] - b[0] * b[2] * I4PI, v[0] * (e + pt) - b[0] * vb * I4PI,
             v[0] * b[1] - b[0] * v[1], v[0] * b[2] - b[0] * v[2]]
        return rho, v, b, pg, m, e, pt, f

    rl, vl, bl, gl, ml, el, ptl, fl = side(L)
    rr, vr, br, gr, mr, er, ptr, fr = side(R)
    rho = 0.5 * (rl + rr)
    v = [0.5 * (a + b) for a, b in zip(vl, vr)]
    b = [0.5 * (x + y) for x, y in zip(bl, br)]
    bt2 = b[1] ** 2 + b[2] ** 2
    mag = 0.5 * I4PI * (b[0] ** 2 + bt2)
    kk = 0.5 * (v[0] ** 2 + v[1] ** 2 + v[2] ** 2)
    cc = g * (0.5 * (ptl + ptr) - mag) / rho
    al, ar = g * gl / rl, g * gr / rr
    cc = torch.minimum(torch.maximum(cc, torch.minimum(al, ar)), torch.maximum(al, ar))
    c, bb = torch.sqrt(cc), I4PI * b[0] ** 2 / rho
    ba = torch.sqrt(bb)
    tiny = bt2 < p.small_b ** 2
    bt = torch.sqrt(torch.where(tiny, 1.0, bt2))
    hy = torch.where(tiny, math.sqrt(0.5), b[1] / bt)
    hz = torch.where(tiny, math.sqrt(0.5), b[2] / bt)
    sz = cc + 2.0 * mag / rho
    root = torch.sqrt((sz * sz - 4.0 * cc * bb).clamp(min=0.0))
    slow = torch.minimum((0.5 * (sz - root)).clamp(min=0.0), cc)
    fast = torch.maximum(0.5 * (sz + root), cc)
    slow = torch.where(tiny, torch.minimum(bb, cc), slow)
    fast = torch.where(tiny, torch.maximum(bb, cc), fast)
    af, a_s = torch.sqrt(fast), torch.sqrt(slow)
    gap = fast - slow
    ok = (gap >= 1e-8) & (cc > slow) & (fast > cc)
    wf = torch.sqrt(torch.where(ok, (cc - slow) / torch.where(ok, gap, 1.0), 1.0))
    ws = torch.sqrt(torch.where(ok, (fast - cc) / torch.where(ok, gap, 1.0), 0.0))
    turned = (gap >= 1e-8) & (cc <= slow)
    wf, ws = torch.where(turned, 0.0, wf), torch.where(turned, 1.0, ws)
    floor = p.entropy_fix * (v[0].abs() + v[1].abs() + v[2].abs() + af)

    def speed(x):
        z = x.abs()
        return torch.where(z >= floor, z, 0.5 * (z * z + floor * floor) / floor)

    sg = torch.where(b[0] >= 0, 1.0, -1.0)
    dr, de = rl - rr, el - er
    dm = [x - y for x, y in zip(ml, mr)]
    db = [x - y for x, y in zip(bl, br)]
    work_b = b[1] * db[1] + b[2] * db[2] + (0.0 if seven else b[0] * db[0])
    dp = -h * (-kk * dr + v[0] * dm[0] + v[1] * dm[1] + v[2] * dm[2] - de + I4PI * work_b)
    dv = [(x - a * dr) / rho for x, a in zip(dm, v)]
    # jumps along and across the transverse field
    dv_b, dv_x = hy * dv[1] + hz * dv[2], hy * dv[2] - hz * dv[1]
    db_b, db_x = hy * db[1] + hz * db[2], hy * db[2] - hz * db[1]
    spr, s2pr = torch.sqrt(math.pi * rho), torch.sqrt(2.0 * math.pi * rho)
    e0 = speed(v[0]) * (dr - dp / cc)
    q2 = math.sqrt(0.5)
    a1 = speed(v[0] + ba) * (q2 * dv_x - 0.5 * sg * db_x / s2pr)
    a2 = speed(v[0] - ba) * (q2 * dv_x + 0.5 * sg * db_x / s2pr)
    pf = 0.5 * wf * dp / (cc * rho) + 0.25 * ws * db_b / (c * spr)
    ps = 0.5 * ws * dp / (cc * rho) - 0.25 * wf * db_b / (c * spr)
    xf = 0.5 * (wf * af * dv[0] - ws * a_s * sg * dv_b) / cc
    xs = 0.5 * (ws * a_s * dv[0] + wf * af * sg * dv_b) / cc
    f1, f2 = speed(v[0] + af) * (xf + pf), speed(v[0] - af) * (pf - xf)
    s1, s2 = speed(v[0] + a_s) * (xs + ps), speed(v[0] - a_s) * (ps - xs)
    sf, df, ss, ds = f1 + f2, f1 - f2, s1 + s2, s1 - s2
    r0 = e0 + rho * (wf * sf + ws * ss)
    rn = wf * af * df + ws * a_s * ds
    rb = sg * (wf * af * ds - ws * a_s * df)
    rx = q2 * (a1 + a2)
    rs, rt = hy * rb - hz * rx, hz * rb + hy * rx
    rp = rho * cc * (wf * sf + ws * ss)
    mb = 2.0 * spr * c * (ws * sf - wf * ss)
    mx = -sg * s2pr * (a1 - a2)
    bs, bz = hy * mb - hz * mx, hz * mb + hy * mx
    bn = 0.0 if seven else speed(v[0]) * db[0]
    re = r0 * kk + rho * (v[0] * rn + v[1] * rs + v[2] * rt) + rp / h \
        + I4PI * (b[1] * bs + b[2] * bz + (0.0 if seven else b[0] * bn))
    add = [r0, v[0] * r0 + rho * rn, v[1] * r0 + rho * rs, v[2] * r0 + rho * rt, re, bs, bz]
    out = [0.5 * (x + y + z) for x, y, z in zip(fl, fr, add)]
    F = [None] * 8
    F[0], F[1 + n], F[1 + s], F[1 + t], F[4], F[5 + s], F[5 + t] = out
    F[5 + n] = torch.zeros_like(rho) if seven else 0.5 * bn
    return F


def van_leer(p, L, R, d):
    """Van Leer flux-vector splitting of one neutral gas."""
    g, h = p.gamma, p.gamma - 1.0

    def half(w, sg):
        rho, pg, v = w[0].clamp(min=p.smallr), w[4].clamp(min=p.smallp), [w[1], w[2], w[3]]
        u = sg * v[d]
        a = torch.sqrt(g * pg / rho)
        e = pg / h + 0.5 * rho * (v[0] ** 2 + v[1] ** 2 + v[2] ** 2)
        m = 0.25 * rho * (u + a) ** 2 / a
        inner_, full = u.abs() < a, u >= a
        mass = torch.where(inner_, m, torch.where(full, rho * u, 0.0))
        mom = torch.where(inner_, m * (u + (2.0 * a - u) / g),
                          torch.where(full, rho * u * u + pg, 0.0))
        f = [sg * mass] + [sg * mass * x for x in v] + [sg * mass * (e + pg) / rho]
        f[1 + d] = mom
        return f

    return [a + b for a, b in zip(half(L, 1.0), half(R, -1.0))]


def stage(p, W, U, origin, dt, ch, cp, t):
    """One stage of the cells U, from the primitives W around them (two cells
    more on each side); returns the new state and the fluxes."""
    sd, dx = p.space_dim, p.dx
    glm = p.divb_cleaning == 5
    fluids = _fluids(p)
    core = inner(W, 2, sd)
    new, divb, fluxes = U.clone(), torch.zeros_like(U[0]), []
    for d in range(sd):
        ax = 3 - d
        V = W
        for e in range(sd):
            if e != d:
                V = V.narrow(3 - e, 2, V.shape[3 - e] - 4)
        m = V.shape[ax]
        df = V.narrow(ax, 1, m - 1) - V.narrow(ax, 0, m - 1)
        a, b = df.narrow(ax, 0, m - 2), df.narrow(ax, 1, m - 2)
        slope = 0.5 * torch.where(a * b > 0, torch.where(a.abs() < b.abs(), a, b), 0.0)
        mid = V.narrow(ax, 1, m - 2)
        L = (mid + slope).narrow(ax, 0, m - 3)
        R = (mid - slope).narrow(ax, 1, m - 3)
        F = torch.zeros_like(L)
        for q, f in enumerate(roe(p, L, R, d, glm)):
            F[q] = f
        if glm:
            bl, br, sl, sr = L[5 + d], R[5 + d], L[8], R[8]
            F[5 + d] = 0.5 * (sl + sr + ch * (bl - br))
            F[8] = 0.5 * ch * (ch * (bl + br) + sl - sr)
        for s in fluids:
            for q, f in enumerate(van_leer(p, L[s:s + 5], R[s:s + 5], d)):
                F[s + q] = f
        k = m - 4
        new = new - dt / dx * (F.narrow(ax, 1, k) - F.narrow(ax, 0, k))
        bn = 0.5 * (L[5 + d] + R[5 + d])
        divb = divb + bn.narrow(ax - 1, 1, k) - bn.narrow(ax - 1, 0, k)
        fluxes.append(F)
    if p.use_8wave:
        x = -divb * dt / dx
        B, v = I4PI * core[5:8], core[1:4]
        new[1:4] += x * B
        new[4] += x * (B * v).sum(0)
        new[5:8] += x * v
    if glm:
        new[8] *= math.exp(-dt * ch * ch / (cp * cp))
    X = None
    if p.charge_exchange or p.reinit_sphere:
        hi = [origin[e] + U.shape[3 - e] - 1 for e in range(3)]
        X = _axes(p, origin, hi)
    if p.charge_exchange:
        exchange(p, core, new, X, dt, fluids)
    if p.reinit_sphere:
        u = list(new[:8])
        wind(p, u, *X, t + dt)
        new[:8] = torch.stack(u)
    floors(p, new, fluids)
    return new, fluxes


def exchange(p, W, U, X, dt, fluids):
    """Charge exchange of the plasma with the neutral populations; new
    neutrals join the population of their region."""
    rho, v, T = W[0], W[1:4], W[4] / W[0]
    r2 = X[0] ** 2 + X[1] ** 2 + X[2] ** 2
    ur = (v[0] * X[0] + v[1] * X[1] + v[2] * X[2]) / torch.sqrt(r2)
    temp = p.region_t_coeff * T
    wind_ = ur.abs() >= 0.6 * p.sun_v
    hot = (temp >= 1.0e6) & (r2 > p.sun_r ** 2)
    reg = torch.where(wind_, torch.where(hot, 2, 3), torch.where(temp >= p.region_tmlim, 2, 1))
    loss = []
    for s in fluids:
        rn, vn, Tn = W[s], W[s + 1:s + 4], 2.0 * W[s + 4] / W[s]
        dv = v - vn
        dv2 = (dv * dv).sum(0)
        pi = math.pi
        ud = torch.sqrt(4.0 * (T + Tn) / pi + dv2)
        upm = torch.sqrt(16.0 * T / pi + 2.25 * pi * Tn + 4.0 * dv2)
        uhm = torch.sqrt(2.25 * pi * T + 16.0 * Tn / pi + 4.0 * dv2)
        upe = torch.sqrt((4.0 * T + 64.0 * Tn / 9.0) / pi + dv2)
        uhe = torch.sqrt((64.0 * T / 9.0 + 4.0 * Tn) / pi + dv2)
        sig = (p.ce_sigma_a - p.ce_sigma_b * torch.log(p.ce_scale_vel * ud)) ** 2
        rate = p.ce_sigma_scale * sig * rn * rho
        # what the plasma loses (as ions) and gains (from this population)
        gain_m = rate * (vn * ud - dv * (Tn / upm))
        loss_m = -rate * (v * ud + dv * (T / uhm))
        gain_e = rate * (0.5 * (vn * vn).sum(0) * ud - (dv * vn).sum(0) * Tn / upm + 0.75 * Tn * upe)
        loss_e = -rate * (0.5 * (v * v).sum(0) * ud + T * ((dv * v).sum(0) / uhm + 0.75 * uhe))
        loss.append((rate * ud, gain_m, gain_e, loss_m, loss_e))
    all_m, all_e = sum(x[3] for x in loss), sum(x[4] for x in loss)
    U[1:4] += dt * (sum(x[1] for x in loss) + all_m)
    U[4] += dt * (sum(x[2] for x in loss) + all_e)
    total = sum(x[0] for x in loss)
    for k, (s, (rate, gm, ge, _, _)) in enumerate(zip(fluids, loss)):
        here = reg == k + 1
        U[s] += dt * torch.where(here, total - rate, -rate)
        U[s + 1:s + 4] -= dt * (gm + torch.where(here, all_m, 0.0))
        U[s + 4] -= dt * (ge + torch.where(here, all_e, 0.0))


def floors(p, U, fluids):
    """Density and pressure floors of every fluid."""
    h = p.gamma - 1.0
    for f, s in enumerate([0] + fluids):
        fd = p.smallr if f < 2 else 1e-6 if f == 2 else 1e-7
        fp = p.smallp if f < 2 else 1e-8 if f == 2 else 1e-9
        rho, v = U[s], U[s + 1:s + 4] / U[s]
        k = 0.5 * (v * v).sum(0)
        mag = 0.5 * I4PI * (U[5:8] ** 2).sum(0) if s == 0 else 0.0
        pr = h * (U[s + 4] - mag - rho * k)
        low = (rho < fd) | (pr < fp)
        r = rho.clamp(min=fd)
        U[s + 4] = torch.where(low, pr.clamp(min=fp) / h + r * k + mag, U[s + 4])
        U[s + 1:s + 4] = torch.where(low, r * v, U[s + 1:s + 4])
        U[s] = r


def step(p, U, dt, ch, cp, t=0.0):
    """One RK2 step of a whole domain; the new state and its dt."""
    U1, _ = stage(p, padded(p, U), U, [0, 0, 0], dt, ch, cp, t)
    U2, _ = stage(p, padded(p, U1), U1, [0, 0, 0], 0.5 * dt, ch, cp, t)
    U2 = U2 + 0.5 * (U - U1)
    ndt = wave_dt(p, U2)
    if p.neutral_sun_bc:  # neutrals pass through the sun
        n = [U.shape[3 - d] - 1 for d in range(3)]
        x, y, z = _axes(p, [0, 0, 0], n)
        m = (x > 0) & (x * x + y * y + z * z <= p.sun_r ** 2)
        s = _fluids(p)[0]
        for q, sg in enumerate((1.0, 1.0, -1.0, -1.0, 1.0)):
            U2[s + q] = torch.where(m, sg * U2[s + q].flip(2), U2[s + q])
    return U2, ndt


def exact(case, seed):
    if case["kind"] == "hier" or case.get("ct") or case.get("time", "rk2") != "rk2":
        return None  # no 64-bit form of these outside the framework's own
    if case["kind"] == "serve":
        base, out = serving.physics_params(2, PREC[case["prec"]]), []
        for k, n in enumerate(int(s) for s in case["sizes"].split(",")):
            p = serving.run_physics(base, n)
            U = orszag_fields(p, [0, 0, 0], [n - 1, n - 1, 0], seed + 101 * k)
            dt = CFL * wave_dt(p, U)
            for _ in range(case["steps"]):
                U, nd = step(p, U, dt, p.dedner_ch, p.dedner_cp)
                dt = min(CFL * nd, dt * p.max_dt_growth)
            out.append(U.cpu().numpy())
        return {"U": out}
    p = params(case)
    if case["kind"] == "patch":
        (lo, hi), (flo, fhi) = patch_boxes(case, p)
        sd = p.space_dim
        U = fields(case, p, flo, fhi, seed)
        dt = CFL * wave_dt(p, inner(U, 4, sd))
        at = [[flo[d] + (g if d < sd else 0) for d in range(3)] for g in (2, 4)]
        ch, cp = p.dedner_ch, p.dedner_cp
        U1, F1 = stage(p, prim(p, U), inner(U, 2, sd), at[0], dt, ch, cp, 0.0)
        U2, F2 = stage(p, prim(p, U1), inner(U1, 2, sd), at[1], 0.5 * dt, ch, cp, 0.0)
        U2 = U2 + 0.5 * (inner(U, 4, sd) - inner(U1, 2, sd))
        F = [0.5 * (inner(a, 2, sd) + b) for a, b in zip(F1, F2)] if case["fluxes"] else []
        return {"U": U2, "F": F, "dt": wave_dt(p, U2)}
    n, sd = case["n"], p.space_dim
    U = fields(case, p, [0, 0, 0], [n - 1, n - 1, n - 1 if sd == 3 else 0], seed)
    U, ndt = step(p, U, CFL * wave_dt(p, U), p.dedner_ch, p.dedner_cp)
    out = {"U": gather(cut_boxes(n, case["cuts"], sd), U)}
    return {**out, "dt": ndt} if case["sync"] else out
