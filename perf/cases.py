"""Workloads of the solver that its speed is measured on.

Every case goes through the package's public entry points (Solve, Batch, Server) as a user's
program does. The sizes are those of the package's own workloads: the production pipe
(512 x 128 x 128, bench.py), the small FP64 pipe (64 x 32 x 32), the mixed-size ensemble and the
served request stream (streamwise 32..256, cross-sections 24..96, workloads.py) and the geometry
of pipe.m (300 core planes, 120 x 120, R = 50). A pass of a stepping case is one `step(n)` call on
fields that stay on the device; its outputs are the device fields in their storage type.
"""
import math
import random

import numpy as np
import torch

import flowcontrast_b200 as fb

DTYPES = {"f64": fb.F64, "f32": fb.F32, "f16": fb.F16}
TYPESTR = {"f64": "<f8", "f32": "<f4", "f16": "<f2"}
ITEM = {"f64": 8, "f32": 4, "f16": 2}
MONITOR = 50             # monitor and gauge period (the reference's)

_ctx = None


def context():
    """The program's one context (a device and a stream)."""
    global _ctx
    if _ctx is None:
        _ctx = fb.Context(0)
    return _ctx


# ---------------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------------
def pipe(name, dtype, L, n, steps, geometry="circle", order=0):
    return {"name": name, "kind": "pipe", "dtype": dtype, "L": L, "n": n, "steps": steps,
            "geometry": geometry, "order": order}


def listed():
    return [
        # one time step at a time on a small pipe: a program that reads the flow after every step
        pipe("tiny_f32_single_step", "f32", 32, 24, 1),
        # the validation pipe (64 x 32 x 32, R = 15, FP64): short runs against an oracle
        pipe("small_f64", "f64", 64, 32, 50),
        # one ordinary pipe of odd sizes on its own: a member of a parameter study
        pipe("medium_f32_odd", "f32", 151, 61, 50),
        # the production pipe in the three storage forms
        pipe("production_f32", "f32", 512, 128, 50),
        pipe("production_f64", "f64", 512, 128, 25),
        pipe("production_f16", "f16", 512, 128, 25),
        # the reference's demo: pipe.m's geometry as a mask, driven by the seam pressure jump
        pipe("pipe_m_f32", "f32", 300, 120, 50, geometry="pipe.m"),
        # a rough pipe: one cross-section per plane
        pipe("rough_f32", "f32", 192, 96, 10, geometry="rough"),
        # the paper's corrector: order 6 blended with 4 at 0.4
        pipe("order6_f32", "f32", 256, 96, 10, order=6),
        # the mixed-size ensemble, 64 pipes advanced together
        {"name": "ensemble_f32", "kind": "ensemble", "count": 64, "sizes": 20261203, "steps": 32},
        # statistics every step: plane statistics and full-volume profiles, read out at the end
        {"name": "statistics_f64", "kind": "stats", "L": 256, "n": 96, "samples": 8},
        # a burst of requests through the server: host fields in, host fields out
        {"name": "served_burst", "kind": "served", "count": 12, "sizes": 20261204},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["pipe", "rough", "order6", "ensemble", "stats", "served"],
                       [10, 1, 1, 2, 1, 1])[0]
    if kind == "ensemble":
        return {"kind": "ensemble", "count": _log_int(rng, 4, 40), "sizes": rng.randrange(1 << 30),
                "steps": rng.choice([16, 24, 32])}
    if kind == "stats":
        return {"kind": "stats", "L": _log_int(rng, 32, 256), "n": _log_int(rng, 24, 96),
                "samples": rng.randint(2, 8)}
    if kind == "served":
        return {"kind": "served", "count": rng.randint(4, 12), "sizes": rng.randrange(1 << 30)}
    if kind in ("rough", "order6"):
        c = pipe("", "f32", _log_int(rng, 32, 192), _log_int(rng, 32, 96), 10,
                 geometry="rough" if kind == "rough" else "circle", order=6 if kind == "order6" else 0)
    else:
        c = pipe("", rng.choice(["f32", "f32", "f64", "f16"]), _log_int(rng, 32, 512),
                 _log_int(rng, 24, 128), 1)
        c["geometry"] = rng.choice(["circle", "circle", "pipe.m"]) if c["n"] >= 40 else "circle"
        if c["geometry"] == "pipe.m" and c["dtype"] == "f16":
            c["geometry"] = "circle"
        c["steps"] = rng.choice([1, 10, 25])
    del c["name"]
    return c


# ---------------------------------------------------------------------------------------
# physics and geometry
# ---------------------------------------------------------------------------------------
def ensemble_sizes(case):
    """L uniform in [32, 256], n uniform in [24, 96], Re log-uniform in [50, 3000]."""
    rng = random.Random(case["sizes"])
    return [(rng.randint(32, 256), rng.randint(24, 96),
             math.exp(rng.uniform(math.log(50.0), math.log(3000.0)))) for _ in range(case["count"])]


def served_requests(case):
    """(L, n, Re, steps): cells log-uniform from 32^3 to 256 x 96 x 96, n log-uniform in [24, 96]."""
    rng = random.Random(case["sizes"])
    out = []
    for _ in range(case["count"]):
        cells = math.exp(rng.uniform(math.log(32.0 ** 3), math.log(256.0 * 96 * 96)))
        n = _log_int(rng, 24, 96)
        L = min(256, max(32, round(cells / (n * n))))
        re = math.exp(rng.uniform(math.log(50.0), math.log(5000.0)))
        out.append((L, n, re, rng.randint(50, 200)))
    return out


def flow(geometry, L, n, order=0, re=None):
    """Radius, peak velocity and solver parameters. Production-like pipes: bulk Re 5300 at
    nu = 0.0111; ensemble members: bulk velocity 0.1 at their Re."""
    R = n / 2.0 - (10.0 if geometry == "pipe.m" else 3.0 if geometry == "rough" else 1.0)
    p = {"tblend": 0.02, "pin": 0.0, "d1": 2, "blend": 0.4 if order == 6 else 1.0, "order": order}
    if re is not None:
        ub, p["nu"] = 0.1, 2 * R * 0.1 / re
    else:
        p["nu"] = 0.0111
        ub = min(0.46, 5300.0 * p["nu"] / (2 * R))
    g = 8 * p["nu"] * ub / R ** 2
    if geometry == "pipe.m":             # the pressure jump that balances the same wall friction
        p["pin"], p["blend"], g = 3 * g * L, 0.0, 0.0
    p["fz"] = -g
    return R, 2 * ub, p


def cross_section(geometry, L, n, R):
    """The mask a program would hand over: None (the analytic circle), a pipe.m cross-section
    (circle of diameter n - 20 inside ten wall cells), or one rough cross-section per plane."""
    c = (n - 1) / 2.0
    if geometry == "circle":
        return None
    if geometry == "pipe.m":
        o = (n - 20) / 2.0
        i = np.arange(n) - 9.0
        inside = (i[None, :] - o) ** 2 + (i[:, None] - o) ** 2 <= o * o
        inside &= ((i >= 1) & (i <= n - 20))[None, :] & ((i >= 1) & (i <= n - 20))[:, None]
        return np.where(inside, 0, 125).astype(np.uint8)
    y, x = np.mgrid[0:n, 0:n] - c
    z = np.arange(L)[:, None, None] * (2 * np.pi / L)
    th, r = np.arctan2(y, x)[None], np.hypot(x, y)[None]
    wall = R + 0.7 * (np.sin(3 * th) * np.cos(z) + np.sin(5 * th + 1.0) * np.cos(2 * z))
    return np.where(r <= wall, 0, 125).astype(np.uint8)


def fluid_of(mask, n, R):
    """Boolean fluid cells, (1 or L, n, n)."""
    if mask is None:
        y, x = np.mgrid[0:n, 0:n] - (n - 1) / 2.0
        return (x ** 2 + y ** 2 <= R ** 2)[None]
    return (mask == 0).reshape(-1, n, n)


def start_fields(L, n, R, umax, fluid, seed, dtype):
    """(4, L, n, n) on the GPU: Poiseuille flow in -w, uniform noise, and four random-phase
    streamwise modes at 5 % of the peak velocity; p = 0."""
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    dev = {"device": "cuda", "dtype": torch.float64}
    c = (n - 1) / 2.0
    x = (torch.arange(n, **dev) - c) / R
    s = torch.clamp(1 - x[None, None, :] ** 2 - x[None, :, None] ** 2, min=0.0)
    th = torch.atan2(x[None, :, None], x[None, None, :])
    z = torch.arange(L, **dev)[:, None, None] * (2 * math.pi / L)
    f = torch.zeros((4, L, n, n), **dev)
    ph = torch.rand((4, 3), generator=gen, **dev) * 2 * math.pi
    for k in range(3):
        f[1 + k] = 1e-3 * umax * (2 * torch.rand((L, n, n), generator=gen, **dev) - 1)
        for m in range(4):
            f[1 + k] += 0.05 * umax * s * torch.sin((m + 1) * z + ph[m, k]) * torch.cos((m + 1) * th)
    f[3] -= umax * s
    f *= torch.from_numpy(fluid).to("cuda")[None]
    return f.to(dtype)


def setup(geometry, L, n, order, re, seed, host_dtype):
    """(domain, parameters, host fields, fluid, radius) of one pipe."""
    R, umax, p = flow(geometry, L, n, order, re)
    mask = cross_section(geometry, L, n, R)
    c = (n - 1) / 2.0
    dom = fb.make_domain(n, n, L, mask=mask, radius=R, cx=c, cy=c)
    prm = fb.Params.make(tblend=p["tblend"], pin=p["pin"], nu=p["nu"], d1=p["d1"], delta=2,
                         blend=p["blend"], monitor_every=MONITOR, force=(0.0, 0.0, p["fz"]),
                         fd_order=p["order"])
    f = start_fields(L, n, R, umax, fluid_of(mask, n, R), seed, host_dtype)
    return dom, prm, f.cpu().numpy()


class _Device:
    """Device memory of a solve, which it keeps alive, for torch.as_tensor."""

    def __init__(self, owner, ptr, shape, strides, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "strides": strides,
                                         "typestr": typestr, "version": 3}


def device_fields(s, dtype, joined=False):
    """The solve's current device fields as tensors (no copy): p, u, v, w, or one (4, L, n, n)."""
    L, ny, nx = s.shape
    es, pitch = ITEM[dtype], s.info()["lx_pitch"]
    row = (es * pitch * ny, es * pitch, es)
    ptrs = s.device_fields()
    if joined:
        return torch.as_tensor(_Device(s, ptrs[0], (4, L, ny, nx), (es * pitch * ny * L,) + row,
                                       TYPESTR[dtype]), device="cuda")
    return [torch.as_tensor(_Device(s, p, (L, ny, nx), row, TYPESTR[dtype]), device="cuda") for p in ptrs]


# ---------------------------------------------------------------------------------------
# prepare, run, work
# ---------------------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind == "pipe":
        dom, prm, f = setup(case["geometry"], case["L"], case["n"], case["order"], None, seed,
                            torch.float64 if case["dtype"] == "f64" else torch.float32)
        s = fb.Solve(context(), dom, prm, DTYPES[case["dtype"]])
        s.set_fields(f)
        s.sync()
        return {"case": case, "solve": s}
    if kind == "stats":
        dom, prm, f = setup("circle", case["L"], case["n"], 0, None, seed, torch.float64)
        s = fb.Solve(context(), dom, prm, fb.F64)
        s.set_fields(f)
        s.sync()
        return {"case": case, "solve": s}
    if kind == "ensemble":
        solves = []
        for i, (L, n, re) in enumerate(ensemble_sizes(case)):
            dom, prm, f = setup("circle", L, n, 0, re, seed * 1000 + i, torch.float32)
            s = fb.Solve(context(), dom, prm, fb.F32)
            s.set_fields(f)
            solves.append(s)
        b = fb.Batch(context(), solves)
        b.sync()
        return {"case": case, "batch": b}
    reqs = [setup("circle", L, n, 0, re, seed * 1000 + i, torch.float32) + (steps,)
            for i, (L, n, re, steps) in enumerate(served_requests(case))]
    return {"case": case, "server": _Closing(fb.Server(0)), "requests": reqs}


class _Closing:
    """A server that is closed with the state that owns it."""

    def __init__(self, server):
        self.server = server

    def __del__(self):
        self.server.close()


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "pipe":
        s = state["solve"]
        s.step(case["steps"])
        return device_fields(s, case["dtype"])
    if kind == "ensemble":
        b = state["batch"]
        b.step(case["steps"])
        return [device_fields(s, "f32", joined=True) for s in b.solves]
    if kind == "stats":
        s = state["solve"]
        for _ in range(case["samples"]):
            s.step(1)
            s.stats_sample()
            s.profile_sample()
        return [s.stats_get()[0], s.profile_get()[0]]
    srv = state["server"].server
    ids = [srv.submit(dom, prm, fb.F32, steps, init=f) for dom, prm, f, steps in state["requests"]]
    srv.drain(60.0)
    return [srv.release(i) for i in ids]


FLOPS_PER_CELL = 220     # predictor (27 equilibrium brackets, factored) and corrector of one cell


def work(case):
    """Per step: the fluid cells' four fields read once and written once in the storage type."""
    kind = case["kind"]
    if kind == "ensemble":
        cells = sum(L * math.pi * (n / 2.0 - 1) ** 2 * case["steps"] for L, n, _ in ensemble_sizes(case))
        return {"bytes": cells * 32, "flops": cells * FLOPS_PER_CELL}
    if kind == "served":
        req = served_requests(case)
        cells = sum(L * math.pi * (n / 2.0 - 1) ** 2 * steps for L, n, _, steps in req)
        host = sum(32 * L * n * n for L, n, _, _ in req)
        return {"bytes": cells * 32 + host, "flops": cells * FLOPS_PER_CELL}
    L, n = case["L"], case["n"]
    if kind == "stats":                  # the step, and one more read of the state per sample
        cells = L * math.pi * (n / 2.0 - 1) ** 2 * case["samples"]
        acc = 2 * 8 * case["samples"] * (22 * n * (L + 20) + 20 * n * n)
        return {"bytes": cells * 96 + acc, "flops": cells * (FLOPS_PER_CELL + 20)}
    R = flow(case["geometry"], L, n)[0]
    cells = L * math.pi * R ** 2 * case["steps"]
    table = 16 if case["geometry"] == "rough" else 0       # wall sums per cell
    return {"bytes": cells * (8 * ITEM[case["dtype"]] + table),
            "flops": cells * (FLOPS_PER_CELL + (25 if case["order"] == 6 else 0))}


# ---------------------------------------------------------------------------------------
# the same in 64 bits, plain torch
# ---------------------------------------------------------------------------------------
def _coefficients(order, b):
    if order == 6:
        return [-7.5 - 0.66666666666 * b, 1.3333333 + 0.16666666666 * b,
                -0.08333333 - 0.0666666666666 * b, 0.01111111 * b]
    return [-6.0 - 1.5 * b, 1.0 + 0.3333333333 * b, -0.0833333333 * b]


def evolve(f, fluid, p, steps, each=None):
    """`steps` time steps of (4, L, n, n) FP64 fields: the D3Q27 equilibrium pull with the wall
    rule (a wall neighbour counts with the centre's p), the coarse-stride corrector, the seam's
    pressure jump and the monitor's gauge."""
    c = _coefficients(p["order"], p["blend"])
    d1, tb, F = p["d1"], p["tblend"], (0.0, 0.0, p["fz"])
    G = d1 * (len(c) - 1)                # widest tap, the padding around the fields
    _, L, n, _ = f.shape
    am = (p["nu"] - 0.16666666) / d1 ** 2
    w1 = {-1: 1 / 6, 0: 2 / 3, 1: 1 / 6}
    cs = [(x, y, z) for z in (-1, 0, 1) for y in (-1, 0, 1) for x in (-1, 0, 1)]
    sl = lambda a, x, y, z: a[..., G + z:G + z + L, G + y:G + y + n, G + x:G + x + n]  # noqa: E731

    def pad(a):                          # periodic in z, zero outside the cross-section
        k = torch.arange(-G, L + G, device=a.device) % L
        return torch.nn.functional.pad(a[..., k, :, :], (G, G, G, G))

    fl = fluid.to(f.dtype).expand(L, n, n)
    flp = pad(fl)
    wall = [sum(w1[x] * w1[y] * w1[z] * k(x, y, z) * (1 - sl(flp, x, y, z)) for x, y, z in cs)
            for k in (lambda x, y, z: 1, lambda x, y, z: x, lambda x, y, z: y, lambda x, y, z: z)]
    gauge = 0.0
    for step in range(1, steps + 1):
        fp = pad(f)
        fp[0, :G] += p["pin"] * flp[:G]
        fp[0, L + G:] -= p["pin"] * flp[L + G:]
        u, v, w = fp[1], fp[2], fp[3]
        q = fp[0] - 1.5 * (u * u + v * v + w * w)
        m = [f[0] * k for k in wall]
        for x, y, z in cs:
            a = sl(u, x, y, z) * x + sl(v, x, y, z) * y + sl(w, x, y, z) * z
            t = (sl(q, x, y, z) + a * (3 + 4.5 * a)) * (w1[x] * w1[y] * w1[z])
            m[0] = m[0] + t
            for k, e in ((1, x), (2, y), (3, z)):
                if e:
                    m[k] = m[k] + t * e
        new = [(m[0] - gauge) * fl]
        for k in (1, 2, 3):
            lap = c[0] * f[k]
            for j in range(1, len(c)):
                o = j * d1
                a = fp[k]
                lap = lap + c[j] * (sl(a, o, 0, 0) + sl(a, -o, 0, 0) + sl(a, 0, o, 0) + sl(a, 0, -o, 0)
                                    + sl(a, 0, 0, o) + sl(a, 0, 0, -o))
            new.append(((m[k] + am * lap + F[k - 1]) * tb + f[k] * (1 - tb)) * fl)
        f = torch.stack(new)
        gauge = float((f[0, 0] - p["pin"]).mul(fl[0]).sum() / fl[0].sum()) if step % MONITOR == 0 else 0.0
        if each:
            each(f)
    return f


def _exact_pipe(geometry, L, n, order, re, seed, dtype, steps, each=None):
    R, umax, p = flow(geometry, L, n, order, re)
    fluid = fluid_of(cross_section(geometry, L, n, R), n, R)
    f0 = start_fields(L, n, R, umax, fluid, seed, dtype).double()
    return f0, evolve(f0, torch.from_numpy(fluid).to("cuda"), p, steps, each)


def exact(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        return [_exact_pipe("circle", L, n, 0, re, seed * 1000 + i, torch.float32, case["steps"])[1]
                for i, (L, n, re) in enumerate(ensemble_sizes(case))]
    if kind == "served":
        return [_exact_pipe("circle", L, n, 0, re, seed * 1000 + i, torch.float32, steps)[1]
                for i, (L, n, re, steps) in enumerate(served_requests(case))]
    L, n = case["L"], case["n"]
    if kind == "stats":
        d2, planes, sums = 10, [], []

        def sample(f):
            z = torch.arange(-d2, L + d2, device="cuda") % L
            planes.append(f[:, z, :, n // 2])
            q, u, v, w = f
            sums.append(torch.stack([a.sum(0) for a in (q, u, v, w, u * u, v * v, w * w, u * v, u * w, v * w)]))

        _exact_pipe("circle", L, n, 0, None, seed, torch.float64, case["samples"], sample)
        mean, dev = torch.zeros_like(planes[0]), torch.zeros((7,) + planes[0].shape[1:], device="cuda",
                                                             dtype=torch.float64)
        for k, s in enumerate(planes):   # the running mean includes the sample
            mean = mean + s
            d = mean / (k + 1) - s
            dev = dev + torch.cat([d.abs(), torch.stack([d[1] * d[2], d[1] * d[3], d[3] * d[2]])])
        N = float(case["samples"])
        return [torch.cat([mean, dev]).reshape(11, -1) / N, torch.stack(sums).sum(0)]
    dtype = torch.float64 if case["dtype"] == "f64" else torch.float32
    f0, f = _exact_pipe(case["geometry"], L, n, case["order"], None, seed, dtype, case["steps"])
    if case["dtype"] == "f16":           # FP16 storage holds w as the deviation from its start's column mean
        f[3] -= f0[3].mean(0).float().double()
    return [f[0], f[1], f[2], f[3]]
