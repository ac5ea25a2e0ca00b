"""The work that programs give this library, as cases that can be timed and compared.

A case is one wind tunnel (or one batch of tunnels) and what a program does with it in a pass:

* a frame: `Fluid.update`, the synchronous step of an interactive loop, with or without the
  headless visuals that such a loop draws after it;
* a run: `Fluid.update_async` over several steps and one wait, as a serving lane or an offline
  job advances a tunnel;
* a batch: `Batch.step`, many uneven tunnels advanced together.

The tunnels are the parity case, the default tunnel and the large grid of `scenarios`, the
800x400 grid of the published CPU table, odd and ragged grids, and batches drawn as the batched
and served scenarios are. Fields start in a developed state (a jet behind the inflow, a wake of
random velocities, a smoke plume) made from the seed. FP32 tunnels leave the blocking depth to
the library; 16-bit tunnels fix it, because with 16-bit storage the depth says how often a value
is rounded, and with it the result.

`exact` is the same step in 64 bits, written with plain torch on the whole grid.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from opensayal_gb300 import Fluid, Source, default_config, native
from opensayal_gb300.batch import Batch
from opensayal_gb300.fluid import visual_defaults

_STORAGE = {"f32": native.STORAGE_F32, "f16": native.STORAGE_F16, "bf16": native.STORAGE_BF16}

# What a tunnel is when the case does not say otherwise: the default tunnel's options.
_TUNNEL = {
    "kind": "tunnel", "width": 1920, "height": 1080, "n": 50, "steps": 1, "frame": True,
    "storage": "f32", "depth": 0, "pressure": False, "viscosity": 0.001, "cell": 1,
    "drain": True, "smoke": True, "decay": False, "drag": 0.0, "g": -5.0, "dt": 0.05, "speed": 2.0,
    "radius": 0.0, "source": False, "visuals": False,
}
_BATCH = {"kind": "batch", "count": 21, "lo": 128, "hi": 1024, "grain": 32, "pick": 4,
          "mixed": False, "depth": 0, "steps": 1}


def _tunnel(name, **more):
    return {"name": name, **_TUNNEL, **more}


def _batch(name, **more):
    return {"name": name, **_BATCH, **more}


def listed():
    return [
        # The smallest grid in use, one synchronous step: launches and latency count.
        _tunnel("frame_256x128", width=256, height=128, g=0.0, drain=False, radius=12.0),
        # An odd small grid of the interactive loop: mouse forcing, drag, smoke decay, pressure.
        _tunnel("frame_333x187_interactive", width=333, height=187, n=30, pressure=True,
                source=True, decay=True, drag=0.1),
        # The grid of the published CPU table: pressure and smoke on, drawn after the step.
        _tunnel("frame_800x400_pressure_drawn", width=800, height=400, pressure=True,
                visuals=True),
        # One served request of the ordinary size on a lane of its own, a chunk of steps.
        _tunnel("run_640x448_n100_x8", width=640, height=448, n=100, steps=8, frame=False),
        # A ragged grid without viscosity and with cells of size 2 (every option off the default).
        _tunnel("frame_1003x771_inviscid_cell2", width=1003, height=771, n=40, viscosity=0.0,
                cell=2),
        # The default tunnel, one synchronous step: the reference's own frame.
        _tunnel("frame_1920x1080"),
        # The same with the pressure on, as the pressure view needs it.
        _tunnel("frame_1920x1080_pressure", pressure=True),
        # The same grid held in 16 bits, a chunk of steps.
        _tunnel("run_1920x1080_bf16_x2", storage="bf16", depth=8, steps=2, frame=False),
        # The largest grid of the benchmark.
        _tunnel("frame_4096x4096_n200", width=4096, height=4096, n=200, dt=0.02),
        _tunnel("frame_4096x4096_n200_f16", width=4096, height=4096, n=200, dt=0.02,
                storage="f16", depth=8),
        # A fixed set of uneven tunnels advanced together, drawn as the batched workload is.
        _batch("batch_21_uneven"),
        # What the server's continuous batch holds at light load: a few tunnels, FP32 and BF16.
        _batch("served_6_mixed", count=6, pick=5, mixed=True, depth=8, steps=2),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


_MOST = 4096 * 4096 * 200  # cells x sweeps x steps of the largest listed case


def draw(rng):
    if rng.random() < 0.25:
        mixed = rng.random() < 0.4
        return {**_BATCH, "count": rng.randint(2, 21), "lo": rng.choice((64, 96, 128)),
                "hi": rng.choice((384, 512, 768, 1024)), "grain": rng.choice((1, 8, 32)),
                "pick": rng.randrange(1 << 20), "mixed": mixed,
                "depth": 8 if mixed else rng.choice((0, 6, 8)), "steps": rng.randint(1, 3)}
    while True:
        c = dict(_TUNNEL)
        c["width"], c["height"] = _log_int(rng, 96, 4096), _log_int(rng, 64, 4096)
        if rng.random() < 0.5:  # usual grids are multiples of 16
            c["width"], c["height"] = (max(64, x // 16 * 16) for x in (c["width"], c["height"]))
        if max(c["width"], c["height"]) > 10 * min(c["width"], c["height"]):
            continue
        c["n"] = rng.choice((20, 30, 40, 50, 50, 75, 100, 200))
        if c["width"] * c["height"] * c["n"] <= _MOST // 16 and rng.random() < 0.3:
            c["frame"], c["steps"] = False, rng.randint(2, 8)
        if c["width"] * c["height"] * c["n"] * c["steps"] <= _MOST:
            break
    c["storage"] = rng.choice(("f32",) * 6 + ("f16", "bf16"))
    if c["storage"] != "f32":
        c["depth"] = rng.choice((4, 8))
    c["pressure"] = rng.random() < 0.25
    c["viscosity"] = rng.choice((0.0, 0.001, 0.001, 0.001, 0.01))
    c["cell"] = rng.choice((1, 1, 1, 1, 2))
    c["drain"] = rng.random() < 0.7
    c["smoke"] = rng.random() < 0.9
    c["decay"] = rng.random() < 0.2
    c["drag"] = rng.choice((0.0, 0.0, 0.0, 0.1))
    c["g"] = rng.choice((0.0, -5.0, -9.8))
    c["dt"] = rng.choice((0.02, 0.05))
    c["speed"] = round(rng.uniform(0.5, 3.0), 2)
    c["source"] = rng.random() < 0.15
    c["visuals"] = c["frame"] and rng.random() < 0.2
    return c


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------


def _config(c):
    k = default_config(c["width"], c["height"])
    k.pipe_height = max(1, c["height"] // 4)
    k.tunnel_speed, k.tunnel_smoke = c["speed"], 1.0
    k.obstacle_center_x, k.obstacle_center_y = c["width"] // 2, c["height"] // 2
    k.obstacle_radius = c["radius"] or min(c["width"], c["height"]) / 30.0
    k.g, k.d_t = c["g"], c["dt"]
    k.projection_n, k.projection_o = c["n"], 1.9
    k.enable_drain, k.enable_pressure = int(c["drain"]), int(c["pressure"])
    k.enable_smoke, k.smoke_enable_decay = int(c["smoke"]), int(c["decay"])
    k.cell_size, k.viscosity, k.drag_coeff = float(c["cell"]), c["viscosity"], c["drag"]
    k.storage, k.projection_block = _STORAGE[c["storage"]], c["depth"]
    return k


def _member_configs(c):
    """The tunnels of a batch, drawn as the batched scenarios are."""
    rng = np.random.default_rng(c["pick"])
    sizes = np.arange(c["lo"], c["hi"] + 1, c["grain"])
    out = []
    for _ in range(c["count"]):
        w, h = int(rng.choice(sizes)), int(rng.choice(sizes))
        k = default_config(w, h)
        k.pipe_height = h // 4
        k.tunnel_speed, k.tunnel_smoke = float(rng.uniform(0.5, 3.0)), 1.0
        k.obstacle_center_x = int(rng.integers(w // 4, 3 * w // 4 + 1))
        k.obstacle_center_y = int(rng.integers(h // 4, 3 * h // 4 + 1))
        k.obstacle_radius = float(rng.uniform(4.0, max(5.0, 0.1 * h)))
        k.g = float(rng.uniform(-10.0, 0.0))
        k.projection_n, k.projection_o = int(rng.choice([50, 100, 200])), 1.9
        k.d_t = 0.05
        if c["mixed"] and rng.random() < 0.5:
            k.storage = native.STORAGE_BF16
        out.append(k)
    return out


def _solid(k, dev):
    """The solid mask, (height, width) with row j of the grid at index j."""
    i = torch.arange(k.width, device=dev)[None, :]
    j = torch.arange(k.height, device=dev)[:, None]
    d2 = (i - k.obstacle_center_x) ** 2 + (j - k.obstacle_center_y) ** 2
    s = d2.double().sqrt() < float(k.obstacle_radius)
    s = s | (i == 0) | (j == 0) | (j == k.height - 1)
    return s if k.enable_drain else s | (i == k.width - 1)


def _state(k, seed, index, dev):
    """u, v and smoke of a developed flow, FP32, (height, width) with row j at index j."""
    g = torch.Generator(device=dev).manual_seed(1_000_003 * int(seed) + index)
    H, W = k.height, k.width

    def noise(a):
        return (torch.rand((H, W), generator=g, device=dev) * 2 - 1) * a

    x = torch.arange(W, device=dev, dtype=torch.float32)[None, :] / W
    y = torch.arange(H, device=dev, dtype=torch.float32)[:, None] - H // 2
    spread = 0.5 * k.pipe_height * (1 + x)
    jet = torch.exp(-((y / spread) ** 4)) * (1 - 0.6 * x)
    open_ = ~_solid(k, dev)
    u = (k.tunnel_speed * jet + noise(0.2)) * open_
    v = (noise(0.2) + 0.1 * jet * torch.sin(12 * math.pi * x)) * open_
    s = (k.tunnel_smoke * jet + noise(0.1)).clamp(0, 1) * open_
    return u, v, s


class _Field:
    """A handle's field as an object that torch takes without a copy. The tensor keeps this
    object, and with it the handle whose memory it is."""

    def __init__(self, owner, ptr, shape, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": typestr,
                                         "data": (int(ptr), False), "version": 3}


def _views(f, owner, pressure):
    """The handle's fields as tensors, (height, width), top row first as they are stored.
    `owner`: what frees them (the Fluid, or the batch that it belongs to)."""
    w = f.fields()
    shape = (w.height, w.width)
    out = {}
    for name in ("vel_x", "vel_y", "smoke"):
        kind = {native.STORAGE_F32: "<f4", native.STORAGE_F16: "<f2"}.get(w.storage, "<i2")
        t = torch.as_tensor(_Field(owner, getattr(w, name), shape, kind), device="cuda")
        out[name] = t.view(torch.bfloat16) if w.storage == native.STORAGE_BF16 else t
    if pressure:
        out["pressure"] = torch.as_tensor(_Field(owner, w.pressure, shape, "<f4"), device="cuda")
    return out


def _fill(f, owner, k, seed, index):
    views = _views(f, owner, bool(k.enable_pressure))
    for name, x in zip(("vel_x", "vel_y", "smoke"), _state(k, seed, index, "cuda")):
        views[name].copy_(x.flip(0))
    return views


def prepare(case, seed):
    if case["kind"] == "batch":
        configs = _member_configs(case)
        if case["mixed"]:  # the server's batch: admitted one by one into its memory budget
            b = Batch.dynamic(block_k=case["depth"], budget_bytes=2 << 30)
            ids = [b.add(k, -1) for k in configs]
        else:
            b = Batch(configs, case["depth"])
            ids = list(range(len(configs)))
        scenarios = [b.scenario(m) for m in ids]
        views = [_fill(f, b, k, seed, q) for q, (f, k) in enumerate(zip(scenarios, configs))]
        torch.cuda.synchronize()
        return {"case": case, "batch": b, "scenarios": scenarios, "views": views}
    k = _config(case)
    f = Fluid(k)
    state = {"case": case, "fluid": f, "views": _fill(f, f, k, seed, 0), "dt": case["dt"],
             "source": Source(True, 0.7, 0.3, _source_at(case)) if case["source"] else None}
    if case["visuals"]:
        v = visual_defaults()
        W, H = case["width"], case["height"]
        aw, ah = W // v.arrow_distance, H // v.arrow_distance
        tw, th = W // v.trace_distance, H // v.trace_distance

        def zeros(*shape):
            return torch.zeros(shape, dtype=torch.int32, device="cuda")

        state["visual"] = v
        state["drawn"] = {"pixels": zeros(H, W), "arrows": zeros(ah, aw, 9),
                          "trace_x": zeros(th, tw, v.trace_length),
                          "trace_y": zeros(th, tw, v.trace_length)}
    torch.cuda.synchronize()
    return state


def _source_at(case):
    return case["width"] // 3, case["height"] // 2


def run(state):
    case = state["case"]
    if case["kind"] == "batch":
        state["batch"].step(case["steps"])
        state["batch"].synchronize()
        return state["views"]
    f = state["fluid"]
    if case["frame"]:
        f.update(state["source"], state["dt"])
    else:
        f.update_async(state["source"], state["dt"], case["steps"])
        f.synchronize()
    if not case["visuals"]:
        return state["views"]
    d = state["drawn"]
    f.render_pixels(d["pixels"].data_ptr())
    f.render_arrows(state["visual"], d["arrows"].data_ptr())
    f.render_traces(state["visual"], state["dt"], d["trace_x"].data_ptr(),
                    d["trace_y"].data_ptr())
    f.synchronize()
    return {**state["views"], **d}


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------


def _tunnel_work(k, steps, visuals=False):
    cells = k.width * k.height
    smoke = bool(k.enable_smoke)
    e = {native.STORAGE_F32: 4}.get(k.storage, 2)
    # u, v and smoke read and written, one byte of mask read, pressure written.
    a_cell = 2 * e * (3 if smoke else 2) + 1 + (4 if k.enable_pressure else 0)
    # A Jacobi update takes 6 operations; a cell's turn in a red/black sweep 9 (and 5 for its
    # pressure); the advections about 40 for each field, the smoke 60 more.
    flops = k.projection_n * (9 + (6 if k.viscosity else 0) + (5 if k.enable_pressure else 0))
    flops += 80 + (100 if smoke else 0)
    total = {"bytes": steps * cells * a_cell, "flops": steps * cells * flops}
    if visuals:
        total["bytes"] += cells * 4
        total["flops"] += cells * 20
    return total


def work(case):
    if case["kind"] == "batch":
        each = [_tunnel_work(k, case["steps"]) for k in _member_configs(case)]
        return {key: sum(w[key] for w in each) for key in ("bytes", "flops")}
    return _tunnel_work(_config(case), case["steps"], case["visuals"])


# ---------------------------------------------------------------------------
# The step in 64 bits
# ---------------------------------------------------------------------------


class _Exact:
    """A tunnel on (height, width) arrays with row j of the grid at index j, FP64."""

    def __init__(self, k, u, v, s):
        self.k, dev = k, u.device
        self.u, self.v, self.s = u.double(), v.double(), s.double()
        self.p = torch.zeros_like(self.u)
        self.i = torch.arange(k.width, device=dev)[None, :]
        self.j = torch.arange(k.height, device=dev)[:, None]
        self.fluid = ~_solid(k, dev)
        ring = torch.zeros((k.height + 2, k.width + 2), dtype=torch.bool, device=dev)
        ring[1:-1, 1:-1] = self.fluid
        self.left, self.right = ring[1:-1, :-2], ring[1:-1, 2:]
        self.below, self.above = ring[:-2, 1:-1], ring[2:, 1:-1]
        inner = torch.zeros_like(self.fluid)
        inner[1:-1, 1:-1] = True
        self.active = self.fluid & inner

    def forces(self, source, dt):
        k, H, i, j = self.k, self.k.height, self.i, self.j
        pipe, half = k.pipe_height // 2, k.smoke_height // 2
        inlet = (i <= k.smoke_length) & (i != 0) & (j >= H // 2 - pipe) & (j <= H // 2 + pipe)
        self.u[inlet.expand_as(self.u)] = k.tunnel_speed
        smoky = inlet & (j >= H // 2 - half) & (j <= H // 2 + half)
        self.s[smoky.expand_as(self.s)] = k.tunnel_smoke
        if k.drag_coeff:
            self.u *= math.exp(-k.drag_coeff * dt)
            self.v *= math.exp(-k.drag_coeff * dt)
        if source is not None:
            smoke, vel, (x, y) = source
            dx, dy = i - x, j - y
            disc = dx * dx + dy * dy < 40 * 40
            self.s[disc] = smoke
            self.u += torch.where(disc, (vel * dx).expand_as(disc).double(), 0.0)
            self.v += torch.where(disc, (vel * dy).expand_as(disc).double(), 0.0)
        self.v += k.g * dt

    def diffuse(self, dt):
        k = self.k
        h = int(k.cell_size)
        a = k.viscosity * dt / (h * h)
        for _ in range(k.projection_n):
            u, new = self.u, self.u.clone()
            around = u[1:-1, :-2] + u[1:-1, 2:] + u[:-2, 1:-1] + u[2:, 1:-1]
            new[1:-1, 1:-1] = (u[1:-1, 1:-1] + a * around) / (1 + 4 * a)
            self.u = new

    def project(self, dt):
        k = self.k
        self.p.zero_()
        count = (self.left.double() + self.right.double() + self.below.double()
                 + self.above.double()).clamp(min=1)
        parity = (self.i + self.j) % 2
        press = k.density * int(k.cell_size) / dt
        gains = []
        for colour in (0, 1):
            gains.append(torch.where(self.active & (parity == colour), k.projection_o / count,
                                     0.0)[1:-1, 1:-1])
        masks = [m[1:-1, 1:-1].double() for m in (self.left, self.right, self.below, self.above)]
        u, v = self.u, self.v
        for sweep in range(2 * k.projection_n):
            uc, ur, vc, vt = u[1:-1, 1:-1], u[1:-1, 2:], v[1:-1, 1:-1], v[2:, 1:-1]
            d = (ur - uc + vt - vc) * gains[sweep & 1]
            if k.enable_pressure:
                self.p[1:-1, 1:-1] += d * press
            uc += d * masks[0]
            ur -= d * masks[1]
            vc += d * masks[2]
            vt -= d * masks[3]

    def extrapolate(self):
        u, v = self.u, self.v
        u[0], v[1], u[-1] = u[1].clone(), 0.0, u[-2].clone()
        v[:, 0] = v[:, 1].clone()
        u[:, 1] = 0.0
        v[:, -1] = v[:, -2].clone()

    def _at(self, f, i, j):
        """f at (i, j) where that is a fluid cell of the grid, else 0; and whether it is."""
        W, H = self.k.width, self.k.height
        on = (i >= 0) & (i < W) & (j >= 0) & (j < H)
        q = j.clamp(0, H - 1) * W + i.clamp(0, W - 1)
        ok = on & self.fluid.reshape(-1)[q]
        return torch.where(ok, f.reshape(-1)[q], 0.0), ok

    def _where(self, x, y):
        h = int(self.k.cell_size)
        i, j = torch.trunc(x / h).long(), torch.trunc(y / h).long()
        return h, i, j, x - i * h, y - j * h

    def sample_u(self, x, y):
        h, i, j, in_x, in_y = self._where(x, y)
        below = in_y <= h / 2.0
        dy = torch.where(below, -1, 1)
        wx = 1 - in_x / h
        wy = 1 - (in_y - h / 2.0).abs() / h
        c, ok = self._at(self.u, i, j)
        got = wy * wx * c + wy * (1 - wx) * self._at(self.u, i + 1, j)[0]
        got += (1 - wy) * wx * self._at(self.u, i, j + dy)[0]
        got += (1 - wy) * (1 - wx) * self._at(self.u, i + 1, j + dy)[0]
        return torch.where(ok, got, 0.0)

    def sample_v(self, x, y):
        h, i, j, in_x, in_y = self._where(x, y)
        dx = torch.where(in_x < h / 2.0, -1, 1)
        wx = 1 - (in_x - h / 2.0).abs() / h
        wy = 1 - in_y / h
        c, ok = self._at(self.v, i, j)
        got = wy * wx * c + wy * (1 - wx) * self._at(self.v, i + dx, j)[0]
        got += (1 - wy) * (1 - wx) * self._at(self.v, i + dx, j + 1)[0]
        got += (1 - wy) * wx * self._at(self.v, i, j + 1)[0]
        return torch.where(ok, got, 0.0)

    def sample_smoke(self, x, y):
        h, i, j, in_x, in_y = self._where(x, y)
        di = torch.where(in_x < h / 2.0, -1, 1)
        dj = torch.where(in_y < h / 2.0, -1, 1)
        got, weights = 0.0, 0.0
        for a, b in ((i, j), (i + di, j), (i, j + dj), (i + di, j + dj)):
            far = torch.hypot(x - (a + 0.5) * h, y - (b + 0.5) * h)
            w = 1 / (far + 1e-6)
            got = got + w * self._at(self.s, a, b)[0]
            weights = weights + w
        return got / weights

    def _mean(self, f, taps):
        total, count = f.clone(), torch.ones_like(f)
        i, j = self.i.expand_as(f), self.j.expand_as(f)
        for dx, dy in taps:
            x, ok = self._at(f, i + dx, j + dy)
            total += x
            count += ok
        return total / count

    def advect(self, dt):
        h = int(self.k.cell_size)
        centre_x, centre_y = (self.i + 0.5) * h, (self.j + 0.5) * h
        edge_x, edge_y = (self.i * h).double(), (self.j * h).double()
        v_at_u = self._mean(self.v, ((-1, 1), (0, 1), (-1, 0)))
        u_at_v = self._mean(self.u, ((1, 0), (0, -1), (1, -1)))
        new_u = self.sample_u(edge_x - self.u * dt, centre_y - v_at_u * dt)
        new_v = self.sample_v(centre_x - u_at_v * dt, edge_y - self.v * dt)
        self.u, self.v = new_u, new_v
        if self.k.enable_smoke and self.k.tunnel_smoke:
            zero = torch.zeros_like(self.u)
            x, y = centre_x + zero, centre_y + zero
            back_x, back_y = x - self.sample_u(x, y) * dt, y - self.sample_v(x, y) * dt
            self.s = self.sample_smoke(back_x, back_y)
            if self.k.smoke_enable_decay:
                self.s = (self.s - self.k.smoke_decay_rate * dt).clamp(min=0)

    def step(self, source, dt):
        self.forces(source, dt)
        if self.k.viscosity:
            self.diffuse(dt)
        self.project(dt)
        self.extrapolate()
        self.advect(dt)


def _exact_fields(k, seed, index, steps, source, dt):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    kind = {native.STORAGE_F16: torch.float16, native.STORAGE_BF16: torch.bfloat16}.get(
        k.storage, torch.float32)
    x = _Exact(k, *(f.to(kind) for f in _state(k, seed, index, dev)))
    dt = float(np.float32(dt))
    for _ in range(steps):
        x.step(source, dt)
    out = {"vel_x": x.u.flip(0), "vel_y": x.v.flip(0), "smoke": x.s.flip(0)}
    if k.enable_pressure:
        out["pressure"] = x.p.flip(0)
    return out


def exact(case, seed):
    if case["kind"] == "batch":
        return [_exact_fields(k, seed, q, case["steps"], None, k.d_t)
                for q, k in enumerate(_member_configs(case))]
    source = None
    if case["source"]:
        source = (float(np.float32(0.7)), float(np.float32(0.3)), _source_at(case))
    out = _exact_fields(_config(case), seed, 0, case["steps"], source, case["dt"])
    if case["visuals"]:  # whole numbers: drawn from the fields above
        out.update(dict.fromkeys(("pixels", "arrows", "trace_x", "trace_y")))
    return out
