"""Performance cases: forward-modelling solves of le2d's step through the library's entry points.

Every case is one whole user-level call sequence from given inputs to whole outputs:

- ``solve``:   a state held on the GPU goes into a task (``le2d_rows_in``), is advanced by
               ``le2d_step_n`` and comes back into a GPU buffer (``le2d_rows_out``);
- ``loop``:    the same, one ``le_step`` call per time step, as the reference's driver does;
- ``monitor``: the same in chunks of steps with ``le2d_diagnostics`` after each (the
               precision study's energy record);
- ``host``:    page-locked host state, ``le2d_upload``, ``le2d_step_n``, ``le2d_download``;
- ``batch``:   uneven independent solves in one ``le2d_batch``, created, run and read back;
- ``serve``:   requests submitted to a running ``le2d_server`` and their results collected.

Sizes, materials and initial conditions follow ``le2d_b200.workloads``: pressure disks on a
zero field (plus uniform velocity noise in the precision study), c1 in [1, 4], c2/c1 in
[0.3, 0.6], rho in [1, 3], h = 1, Courant number 0.5.
"""
import ctypes
import math
import random

import numpy as np
import torch

from le2d_b200 import capi, workloads

# Arithmetic operations of one node-update in the reference's formulas: per sweep 6 for the
# invariants, 4 x 12 for the limited transport, 12 for the field update.
FLOPS_PER_UPDATE = 2 * (6 + 4 * 12 + 12)
# Fields of each instance beyond this many have no 64-bit value (it would take too long).
EXACT_INSTANCES = 6

_LIBS = {}


def _lib(prec):
    if prec not in _LIBS:
        _LIBS[prec] = capi.Lib(prec)
    return _LIBS[prec]


# ---------------------------------------------------------------- the cases


def listed():
    return [
        # the smallest served grids: launches and latency
        {"name": "tiny_f32", "kind": "solve", "prec": "f", "nx": 100, "ny": 67, "stype": "aos", "steps": 100, "noise": 0.0},
        # the reference driver's own run: 512 x 512, 200 le_step calls
        {"name": "loop_512_f32", "kind": "loop", "prec": "f", "nx": 512, "ny": 512, "stype": "aos", "steps": 200, "noise": 0.0},
        # a mid-sized single solve
        {"name": "solve_1200x900_f32", "kind": "solve", "prec": "f", "nx": 1200, "ny": 900, "stype": "aos", "steps": 150, "noise": 0.0},
        # odd sizes and an odd number of steps
        {"name": "ragged_3001x1777_f32", "kind": "solve", "prec": "f", "nx": 3001, "ny": 1777, "stype": "aos", "steps": 51, "noise": 0.0},
        # the SoA entry point (le_step_soa's far end)
        {"name": "soa_2050x1500_f32", "kind": "solve", "prec": "f", "nx": 2050, "ny": 1500, "stype": "soa", "steps": 64, "noise": 0.0},
        # the precision study: noise on the velocities, diagnostics every 16 steps
        {"name": "monitor_4096_f32", "kind": "monitor", "prec": "f", "nx": 4096, "ny": 4096, "stype": "aos", "steps": 64, "noise": 1e-3, "every": 16},
        # the large single solve
        {"name": "solve_8192_f32", "kind": "solve", "prec": "f", "nx": 8192, "ny": 8192, "stype": "aos", "steps": 100, "noise": 0.0},
        # a solve whose state comes from and goes back to page-locked host memory
        {"name": "host_2048_f32", "kind": "host", "prec": "f", "nx": 2048, "ny": 2048, "stype": "aos", "steps": 200, "noise": 0.0},
        # double precision: the plain grid and the precision study's grid
        {"name": "solve_512_f64", "kind": "solve", "prec": "d", "nx": 512, "ny": 512, "stype": "aos", "steps": 200, "noise": 0.0},
        {"name": "solve_4096_f64", "kind": "solve", "prec": "d", "nx": 4096, "ny": 4096, "stype": "aos", "steps": 32, "noise": 1e-3},
        # the uneven batch: a survey's worth of independent solves
        {"name": "batch_48_f32", "kind": "batch", "prec": "f", "count": 48, "side_lo": 128, "side_hi": 1024, "steps_lo": 200, "steps_hi": 800},
        # a burst of requests at the server
        {"name": "serve_24_f32", "kind": "serve", "prec": "f", "count": 24, "side_lo": 64, "side_hi": 1024, "steps_lo": 100, "steps_hi": 500},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choice(["solve", "solve", "solve", "loop", "monitor", "host", "batch", "serve"])
    prec = rng.choice(["f", "f", "f", "d"])
    if kind in ("batch", "serve"):
        lo = _log_int(rng, 64, 256)
        return {"kind": kind, "prec": prec, "count": rng.randint(4, 32), "side_lo": lo,
                "side_hi": _log_int(rng, lo + 16, 1024), "steps_lo": rng.randint(50, 150),
                "steps_hi": rng.randint(151, 400)}
    side_hi = {"solve": 8192, "loop": 2048, "monitor": 4096, "host": 3000}[kind]
    nx, ny = _log_int(rng, 64, side_hi), _log_int(rng, 64, side_hi)
    most = (5e9 if prec == "f" else 1.2e9) / (nx * ny)  # steps that cost less than the largest listed solve
    steps = max(2, min(_log_int(rng, 20, 400), int(most)))
    case = {"kind": kind, "prec": prec, "nx": nx, "ny": ny, "stype": "aos" if kind == "loop" or rng.random() < 0.75 else "soa",
            "steps": steps, "noise": rng.choice([0.0, 0.0, 1e-3])}
    if kind == "monitor":
        case["every"] = rng.choice([5, 16, 32])
    return case


# ---------------------------------------------------------------- inputs


def _rng(case, seed):
    return np.random.default_rng([int(seed), 20])


def _draw_problem(rng, nx, ny, steps, noise, seed):
    """Material and disks of one solve, drawn as the batched workload draws them."""
    c1 = float(rng.uniform(1.0, 4.0))
    c2 = c1 * float(rng.uniform(0.3, 0.6))
    rho = float(rng.uniform(1.0, 3.0))
    rmax = max(2.0, min(200.0, 0.25 * min(nx, ny)))
    disks = []
    for _ in range(int(rng.integers(2, 9))):
        disks.append((float(rng.uniform(0.1 * (nx - 1), 0.9 * (nx - 1))), float(rng.uniform(0.1 * (ny - 1), 0.9 * (ny - 1))),
                      float(rng.uniform(min(20.0, 0.5 * rmax), rmax)),
                      float(rng.uniform(0.5, 2.0)) * (1.0 if rng.uniform() < 0.5 else -1.0)))
    return workloads.Problem(nx, ny, 1.0, 1.0, c1, c2, rho, 0.5 / c1, steps, disks, noise, int(seed))


def _problem(case, seed):
    return _draw_problem(_rng(case, seed), case["nx"], case["ny"], case["steps"], case["noise"], seed)


def _problems(case, seed):
    """The instances of a batch or the requests at a server: (problem, receiver row or -1).
    Sizes and step counts belong to the case, materials and disks to the seed."""
    sizes, rng, out = random.Random(case["count"] * 4099 + case["side_lo"] * 64 + case["side_hi"]), _rng(case, seed), []
    for k in range(case["count"]):
        nx, ny = (_log_int(sizes, case["side_lo"], case["side_hi"]) for _ in range(2))
        p = _draw_problem(rng, nx, ny, sizes.randint(case["steps_lo"], case["steps_hi"]), 0.0, k)
        out.append((p, ny // 3 if k % 2 else -1))
    return out


RECEIVER_EVERY = 10


def _initial(p, dtype, seed):
    """The state [5][ny][nx] before the first step, on the GPU."""
    f = torch.zeros((5, p.ny, p.nx), dtype=dtype, device="cuda")
    x = torch.arange(p.nx, device="cuda", dtype=dtype)[None, :]
    y = torch.arange(p.ny, device="cuda", dtype=dtype)[:, None]
    for cx, cy, r, s in p.disks:
        real = lambda v: torch.tensor(v, dtype=dtype, device="cuda")  # noqa: E731
        inside = torch.sqrt(((x - real(cx)) ** 2 + (y - real(cy)) ** 2).double()) < real(r).double()
        f[2][inside] = real(s)
        f[4][inside] = real(s)
    if p.noise:
        g = torch.Generator(device="cuda").manual_seed(int(seed) + 7919)
        f[:2] = (torch.rand((2, p.ny, p.nx), generator=g, device="cuda", dtype=torch.float64) * 2 - 1).mul_(p.noise).to(dtype)
    return f


def _layout(f, stype):
    """[5][ny][nx] in the task's own order, flat."""
    return (f.permute(1, 2, 0) if stype == "aos" else f).reshape(-1)


def _pinned(n, dtype):
    """A page-locked numpy array, which lives as long as something refers to it."""
    return torch.zeros(n, dtype=dtype, pin_memory=True).numpy()


# ---------------------------------------------------------------- one pass


class _Single:
    """A task and the buffers of a single solve."""

    def __init__(self, case, seed):
        self.lib = _lib(case["prec"])
        self.case = case
        dtype = torch.float32 if case["prec"] == "f" else torch.float64
        p = _problem(case, seed)
        x = _initial(p, dtype, seed)
        mat = self.lib.le_init_material(p.c1, p.c2, p.rho)
        self.stype = capi.ST_AOS if case["stype"] == "aos" else capi.ST_SOA
        self.task = self.lib.le_init_task(p.dt, (p.hx, p.hy), mat, (p.nx, p.ny), self.stype)
        if case["kind"] == "host":
            self.src, self.dst = (_pinned(5 * p.nx * p.ny, dtype) for _ in range(2))
            self.src[:] = _layout(x, case["stype"]).cpu().numpy()
        else:
            self.x, self.out = x, torch.empty_like(x)

    def __del__(self):
        torch.cuda.synchronize()
        if getattr(self, "task", None) is not None:
            self.lib.le_free_task(self.task)

    def run(self):
        lib, t, c = self.lib, self.task, self.case
        if c["kind"] == "host":
            lib.upload(t, self.src)
            lib.step_n(t, c["steps"])
            lib.download(t, self.dst)
            return {"state": self.dst}
        stream = torch.cuda.current_stream().cuda_stream
        lib.rows_in(t, 0, c["ny"], self.x.data_ptr(), stream)
        record = []
        if c["kind"] == "loop":
            for _ in range(c["steps"]):
                lib.le_step(t)
        elif c["kind"] == "monitor":
            left = c["steps"]
            while left > 0:
                n = min(left, c["every"])
                lib.step_n(t, n)
                _, d = lib.diagnostics(t)
                record.append([d["energy"]] + d["sumsq"] + d["maxabs"])
                left -= n
        else:
            lib.step_n(t, c["steps"])
        lib.rows_out(t, 0, c["ny"], self.out.data_ptr(), stream)
        if record:
            return {"state": self.out, "record": np.array(record, dtype=lib.dtype)}  # no more exact than the state
        return {"state": self.out}


class _Batch:
    """The problems of a batch and the page-locked arrays its results go to."""

    def __init__(self, case, seed):
        self.lib = lib = _lib(case["prec"])
        self.todo, self.bytes = [], 64 << 20
        dtype = torch.float32 if case["prec"] == "f" else torch.float64
        for p, row in _problems(case, seed):
            n = 5 * p.nx * p.ny if row < 0 else p.steps // RECEIVER_EVERY * 2 * p.nx
            out = _pinned(n, dtype)
            prob = lib.le2d_problem(p.nx, p.ny, p.hx, p.hy, p.dt, p.c1, p.c2, p.rho, p.steps, capi.ST_AOS, row, RECEIVER_EVERY)
            self.todo.append((prob, p.disks, row, out))
            self.bytes += lib.task_device_bytes(p.nx, p.ny) + 4096 + (p.steps // RECEIVER_EVERY * 2 * (p.nx + 32) * 8 if row >= 0 else 0)

    def run(self):
        got, n = [], ctypes.c_int(0)
        with capi.Batch(self.lib, self.bytes) as b:
            ids = [b.add(prob, disks=disks) for prob, disks, _, _ in self.todo]
            b.run(256)
            for rid, (_, _, row, out) in zip(ids, self.todo):
                if row < 0:
                    self.lib.lib.le2d_batch_fields(b.h, rid, out.ctypes.data)
                else:
                    self.lib.lib.le2d_batch_receivers(b.h, rid, out.ctypes.data, ctypes.byref(n))
                got.append(out)
        return got


class _Serve:
    """A running server and the requests of one burst."""

    def __init__(self, case, seed):
        self.lib = lib = _lib(case["prec"])
        self.server = capi.Server(lib, 2 << 30, 100, 64)
        self.todo = []
        for p, row in _problems(case, seed):
            prob = lib.le2d_problem(p.nx, p.ny, p.hx, p.hy, p.dt, p.c1, p.c2, p.rho, p.steps, capi.ST_AOS, row, RECEIVER_EVERY)
            self.todo.append((prob, p.disks, capi.LE2D_WANT_FIELDS if row < 0 else capi.LE2D_WANT_RECEIVERS))

    def __del__(self):
        if getattr(self, "server", None) is not None:
            self.server.close()

    def run(self):
        s = self.server
        tickets = [s.submit(prob, disks=disks, want=want) for prob, disks, want in self.todo]
        got = []
        for t in tickets:
            s.wait(t)
            got.append(s.result(t).reshape(-1))
            s.release(t)
        return got


def prepare(case, seed):
    kind = {"batch": _Batch, "serve": _Serve}.get(case["kind"], _Single)
    return kind(case, seed)


def run(state):
    return state.run()


def work(case):
    size = 4 if case["prec"] == "f" else 8
    if case["kind"] in ("batch", "serve"):  # mean of the log-uniform sides and of the steps
        lo, hi = case["side_lo"], case["side_hi"]
        side = (hi - lo) / math.log(hi / lo)
        nodes = case["count"] * side * side
        updates = nodes * 0.5 * (case["steps_lo"] + case["steps_hi"])
        return {"bytes": 5 * size * nodes * 0.5, "flops": FLOPS_PER_UPDATE * updates}
    nodes = case["nx"] * case["ny"]
    return {"bytes": 2 * 5 * size * nodes, "flops": FLOPS_PER_UPDATE * nodes * case["steps"]}


# ---------------------------------------------------------------- the scheme in 64 bits

EPS = 1e-6


def _superbee(r):
    s = torch.maximum(torch.minimum(2 * r, torch.ones_like(r)), torch.clamp(r, max=2.0)).clamp_(min=0.0)
    return torch.where(torch.isnan(r), torch.full_like(r, 2.0), s)


def _transport(w, k, right):
    """The change of an invariant padded by two nodes at each end of its first axis."""
    d = w[1:] - w[:-1]
    kc = 0.5 * (1.0 - k)
    if right:
        p = d + EPS
        f = w[1:-1] + kc * _superbee(p[:-1] / p[1:]) * d[1:]
        return (-k) * (f[1:-1] - f[:-2])
    q = EPS - d
    g = w[1:-1] - kc * _superbee(q[1:] / q[:-1]) * d[:-1]
    return (-k) * (g[1:-1] - g[2:])


def _sweep(vn, vt, sn, sxy, so, m, far):
    """One sweep along the first axis; `far`: the two rows read beyond the last."""
    n = vn.shape[0]
    at = torch.tensor([0, 0] + list(range(n)) + far, device=vn.device)
    a, b = (sn * m["irhoc1"])[at], (sxy * m["irhoc2"])[at]
    v, u = vn[at], vt[at]
    d1, d2 = 0.5 * _transport(v - a, m["k1"], True), 0.5 * _transport(v + a, m["k1"], False)
    d3, d4 = 0.5 * _transport(u - b, m["k2"], True), 0.5 * _transport(u + b, m["k2"], False)
    return (vn + (d1 + d2), vt + (d3 + d4), sn + (d2 - d1) * m["rhoc1"], sxy + m["rhoc2"] * (d4 - d3), so + (d2 - d1) * m["rhoc3"])


def _material(lib, p):
    """The material's products and Courant numbers in 64 bits, from the numbers as the library holds them."""
    c1, c2, rho, dt = (float(lib.dtype(v)) for v in (p.c1, p.c2, p.rho, p.dt))
    mu = rho * c2 * c2
    la = rho * c1 * c1 - 2.0 * mu
    return {"irhoc1": 1.0 / (c1 * rho), "irhoc2": 1.0 / (c2 * rho), "rhoc1": c1 * rho, "rhoc2": c2 * rho,
            "rhoc3": rho * c1 * la / (la + 2.0 * mu), "k1": dt * c1, "k2": dt * c2, "c1": c1, "c2": c2, "rho": rho, "mu": mu, "la": la}


def _advance(f, m, soa):
    vx, vy, sxx, sxy, syy = f
    nx, ny = vx.shape[1], vx.shape[0]
    t = _sweep(vx.T, vy.T, sxx.T, sxy.T, syy.T, m, [nx - 1, nx - 1])
    vx, vy, sxx, sxy, syy = (v.T for v in t)
    far = [max(ny - 5, 0), max(ny - 4, 0)] if soa else [ny - 1, ny - 1]
    vy, vx, syy, sxy, sxx = _sweep(vy, vx, syy, sxy, sxx, m, far)
    return [vx, vy, sxx, sxy, syy]


def _record(f, m):
    vx, vy, sxx, sxy, syy = f
    mu, la = m["mu"], m["la"]
    e = 0.5 * m["rho"] * (vx * vx + vy * vy) + (la + 2 * mu) / (8 * mu * (la + mu)) * (sxx * sxx + syy * syy)
    e = e - 2 * la / (8 * mu * (la + mu)) * sxx * syy + sxy * sxy / (2 * mu)
    return [float(e.sum())] + [float(v.square().sum()) for v in f] + [float(v.abs().max()) for v in f]


def _instance(lib, p, row, prec):
    """What the library returns for one instance: its fields, or the samples of a receiver row."""
    dtype = torch.float32 if prec == "f" else torch.float64
    f, m = list(_initial(p, dtype, 0).double()), _material(lib, p)
    samples = []
    for s in range(p.steps):
        f = _advance(f, m, False)
        if row >= 0 and (s + 1) % RECEIVER_EVERY == 0:
            samples.append(torch.stack([f[0][row], f[1][row]]))
    out = _layout(torch.stack(f), "aos") if row < 0 else torch.stack(samples)
    return out.reshape(-1).cpu().numpy()


def exact(case, seed):
    lib = _lib(case["prec"])
    if case["kind"] in ("batch", "serve"):
        return [_instance(lib, p, row, case["prec"]) if k < EXACT_INSTANCES else None
                for k, (p, row) in enumerate(_problems(case, seed))]
    p = _problem(case, seed)
    dtype = torch.float32 if case["prec"] == "f" else torch.float64
    f, m = list(_initial(p, dtype, seed).double()), _material(lib, p)
    record = []
    for s in range(p.steps):
        f = _advance(f, m, case["stype"] == "soa")
        if case["kind"] == "monitor" and ((s + 1) % case["every"] == 0 or s + 1 == p.steps):
            record.append(_record(f, m))
    f = torch.stack(f)
    if case["kind"] == "host":
        return {"state": _layout(f, case["stype"]).cpu().numpy()}
    return {"state": f, "record": np.array(record)} if record else {"state": f}
