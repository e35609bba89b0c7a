"""Workloads that stand for what programs do with this framework, sized from its own benchmark
configurations, its serving stream and its regression decks.

Four kinds:
  solve    one lattice: set the initial state on the device, advance it, read rho and u of every
           node back into pinned host memory (what `bench.py` times end to end);
  monitor  the deck runner's loop: a few steps, then the log statistics, again and again;
  batch    many lattices of uneven size advanced together, then the fields of each;
  serve    one call of the solve server on a short stream of requests.
FP64 fields stay the host arrays that the C-ABI fills; the reduced tiers' fields go on to a torch
program as FP32 tensors on the GPU.
"""
import dataclasses
import ctypes
import math

import numpy as np
import torch

from hippolbm_b200 import capi, deck, serve
from hippolbm_b200.batch import Batch
from hippolbm_b200.deck import Op
from hippolbm_b200.lattice import Lattice

BYTES = {"f64": 8, "f64_strict": 8, "f32": 4, "f16": 2, "bf16": 2}
REST_STARTS = ("cavity", "channel", "sphere", "outlet")  # flows that start from rest; the others sheared


def listed():
    return [
        # the smallest serving solve: launches and latency
        solve("cavity", 24, 30, 27, "f16", "bgk", 400, "cavity_24x30x27_f16"),
        # a regression deck (31^3 nodes, FP64) with the runner's statistics every ten steps
        dict(name="monitor_31_f64", kind="monitor", flow="cavity", nx=31, ny=31, nz=31, tier="f64", collision="bgk",
             steps=200, every=10),
        # the small Couette configuration
        solve("couette", 64, 64, 64, "f64", "bgk", 400, "couette_64_f64"),
        # ordinary ragged serving solves: rows of no round length, every face a boundary
        solve("cavity", 57, 43, 61, "bf16", "bgk", 400, "cavity_57x43x61_bf16"),
        solve("channel", 181, 150, 170, "f16", "bgk", 200, "channel_181x150x170_f16"),
        solve("sphere", 150, 120, 131, "f16", "bgk", 300, "sphere_150x120x131_f16"),
        # a body force (the batch configuration's Poiseuille flow) on a ragged lattice
        solve("poiseuille", 130, 97, 113, "f32", "mrt", 300, "poiseuille_130x97x113_f32_mrt"),
        # the precision study's channel past a sphere at half its scale, outlet included
        solve("outlet", 512, 128, 128, "f64", "mrt", 150, "outlet_512x128x128_f64_mrt"),
        # the batch configuration: uneven Couette, Poiseuille and cavity lattices, both collisions
        dict(name="batch_24_f32", kind="batch", tier="f32", members=24, geometry=20261203, lo=32, hi=128, steps=100),
        # a short serving stream as one call
        dict(name="serve_10_f16", kind="serve", tier="f16", requests=10, geometry=7, lo=24, hi=96, budget=500),
        # large Couette lattices, the headline workload's shape: FP64 (BGK) and FP16 storage (MRT)
        solve("couette", 320, 320, 320, "f64", "bgk", 100, "couette_320_f64"),
        solve("couette", 320, 320, 320, "f16", "mrt", 300, "couette_320_f16_mrt"),
    ]


def solve(flow, nx, ny, nz, tier, collision, steps, name):
    return dict(name=name, kind="solve", flow=flow, nx=nx, ny=ny, nz=nz, tier=tier, collision=collision, steps=steps)


def draw(rng):
    def edge(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["solve"] * 7 + ["monitor", "batch", "serve"])
    if kind == "batch":
        return dict(kind="batch", tier=rng.choice(["f32", "f32", "f16", "f64"]), members=rng.randint(4, 24),
                    geometry=rng.randint(0, 1 << 30), lo=32, hi=rng.choice([64, 96, 128]), steps=2 * rng.randint(20, 40))
    if kind == "serve":
        return dict(kind="serve", tier=rng.choice(["f16", "f16", "bf16", "f32"]), requests=rng.randint(3, 10),
                    geometry=rng.randint(0, 1 << 30), lo=24, hi=rng.randint(48, 96), budget=rng.randint(200, 500))
    if kind == "monitor":
        return dict(kind="monitor", flow=rng.choice(["cavity", "couette", "poiseuille"]), nx=edge(24, 64),
                    ny=edge(24, 64), nz=edge(24, 64), tier=rng.choice(["f64", "f64", "f32"]),
                    collision=rng.choice(["bgk", "mrt"]), steps=100, every=rng.choice([5, 10, 20]))
    flow = rng.choice(["cavity", "channel", "sphere", "outlet", "couette", "couette", "poiseuille"])
    hi = 192 if flow in ("cavity", "channel", "sphere") else 320
    nx, ny, nz = edge(24, hi), edge(24, hi), edge(24, hi)
    if flow == "outlet":  # a long channel: its axis is the largest edge
        nx, ny, nz = 2 * max(nx, ny, nz), min(ny, 160), min(nz, 160)
    # the serving solves (cavity, channel, sphere between velocity planes) collide with BGK
    collision = "bgk" if flow in ("channel", "sphere") else rng.choice(["bgk", "mrt"])
    tier = rng.choice(["f64", "f32", "f16", "f16", "bf16"])
    steps = max(60, min(400, int(1.5e9 / (nx * ny * nz))))
    return dict(kind="solve", flow=flow, nx=nx, ny=ny, nz=nz, tier=tier, collision=collision, steps=steps)


# --------------------------------------------------------------------------------- the flows
def flow_case(flow, nodes, collision, rng):
    """The deck of one flow with its parameters drawn from `rng`."""
    nx, ny, nz = nodes
    tau = float(rng.uniform(0.6, 1.0))
    if flow == "couette":
        c = deck.couette_case(nx, tau, float(rng.uniform(0.01, 0.08)), 0, collision)
        c.cell_dims, c.bmax = (nx - 1, ny - 1, nz - 1), (float(nx - 1), float(ny - 1), float(nz - 1))
        return c
    if flow == "poiseuille":
        return deck.poiseuille_case(nodes, tau, float(rng.uniform(1e-6, 1e-5)), 0, collision)
    if flow == "cavity":
        return deck.lid_cavity_case(nodes, tau, float(rng.uniform(0.02, 0.1)), 0, collision)
    if flow == "outlet":
        r = min(ny, nz) * float(rng.uniform(0.08, 0.12))
        return deck.sphere_channel_case(nodes, (nx / 4.0, ny / 2.0, nz / 2.0), r, 0.56 + 0.2 * (tau - 0.6),
                                        float(rng.uniform(0.02, 0.04)), 0, collision,
                                        deck.MRT_RATES_REST_ONE if collision == "mrt" else None)
    tau = float(rng.uniform(0.8, 1.0))  # velocity planes next to bounce-back edges: stable here
    c = serve.solve_case(flow, nodes, tau, rng)
    u = float(rng.uniform(0.005, 0.015))
    c.boundary_conditions = [Op("neumann", {"U": [u, 0.0, 0.0], "regions": ["plan_yz_0", "plan_yz_l"]})]
    return c


def solve_parts(case, seed):
    """(deck, initial shear velocity or None) of a solve or monitor case."""
    rng = np.random.default_rng(seed)
    c = flow_case(case["flow"], (case["nx"], case["ny"], case["nz"]), case["collision"], rng)
    shear = None if case["flow"] in REST_STARTS else [float(v) for v in rng.uniform(-0.04, 0.04, 2)] + [0.0]
    return c, shear


def batch_decks(case, seed):
    shape, rng = np.random.default_rng(case["geometry"]), np.random.default_rng(seed)
    edges = np.arange(case["lo"], case["hi"] + 1, 8)
    out = []
    for _ in range(case["members"]):
        nodes = tuple(int(v) for v in shape.choice(edges, size=3))
        out.append(flow_case(str(shape.choice(["couette", "poiseuille", "cavity"])), nodes,
                             str(shape.choice(["bgk", "mrt"])), rng))
    return out


def serve_requests(case, seed):
    """Requests that have all arrived: BGK solves with a step budget; half of them also ask for a
    residual that a short solve does not reach, so that the server checks it on the way."""
    shape, rng = np.random.default_rng(case["geometry"]), np.random.default_rng(seed)
    out = []
    for i in range(case["requests"]):
        nodes = tuple(int(round(math.exp(v))) for v in shape.uniform(math.log(case["lo"]), math.log(case["hi"]), 3))
        flow = str(shape.choice(["cavity", "channel", "sphere"]))
        budget = int(shape.integers(case["budget"] // 2, case["budget"] + 1))
        out.append(serve.Request(i, 0.0, flow_case(flow, nodes, "bgk", rng), budget, 1e-30 if i % 2 else None))
    return out


# --------------------------------------------------------------------------- prepare and run
class Fields:
    """The pinned host arrays that a lattice's rho and u are read into."""

    def __init__(self, lat, tier):
        self.lat, self.tier = lat, tier
        nx, ny, nz = lat.n
        self.rho = torch.empty((nz, ny, nx), dtype=torch.float64, pin_memory=True)
        self.u = torch.empty((3, nz, ny, nx), dtype=torch.float64, pin_memory=True)

    def read(self):
        d = ctypes.POINTER(ctypes.c_double)
        capi.check(self.lat.L.hlbm_macro_variables(self.lat.h, ctypes.cast(self.rho.data_ptr(), d),
                                                   ctypes.cast(self.u.data_ptr(), d)))
        if BYTES[self.tier] == 8:
            return [self.rho, self.u]
        return [self.rho.to("cuda").float(), self.u.to("cuda").float()]


def prepare(case, seed):
    if case["kind"] == "serve":
        return dict(case=case, requests=serve_requests(case, seed))
    if case["kind"] == "batch":
        lats = [Lattice.from_case(c, case["tier"]) for c in batch_decks(case, seed)]
        batch = Batch(case["tier"]).tune(10)  # each member's own kernel, the autotuner's pick on this mix
        for lat in lats:
            batch.add(lat)
        return dict(case=case, lats=lats, batch=batch, fields=[Fields(lat, case["tier"]) for lat in lats])
    c, shear = solve_parts(case, seed)
    lat = Lattice.from_case(c, case["tier"])
    return dict(case=case, lat=lat, shear=shear, fields=Fields(lat, case["tier"]))


def initial_state(s):
    lat = s["lat"]
    if s["shear"] is None:
        capi.check(lat.L.hlbm_set_distribution(lat.h, 1.0, None, 0))
    else:
        capi.check(lat.L.hlbm_init_double_couette(lat.h, capi.dvec(s["shear"]), 2))


def run(s):
    case = s["case"]
    if case["kind"] == "serve":
        reqs = [dataclasses.replace(r) for r in s["requests"]]
        serve.serve_batched(reqs, case["tier"], check_every=200, keep_results=True, variant=10)
        return [torch.from_numpy(r.result).float() for r in reqs]
    if case["kind"] == "batch":
        s["batch"].step(case["steps"])
        return [f.read() for f in s["fields"]]
    initial_state(s)
    if case["kind"] == "monitor":
        stats = []
        for _ in range(case["steps"] // case["every"]):
            s["lat"].step(case["every"])
            stats.append(s["lat"].simulation_state())
        stats = np.array(stats) if BYTES[case["tier"]] == 8 else np.array(stats, dtype=np.float32)
        return {"stats": stats, "fields": s["fields"].read()}
    s["lat"].step(case["steps"])
    return s["fields"].read()


def work(case):
    """19 populations read and written and one flag byte per node and step; the fields of each node."""
    if case["kind"] == "serve":
        sizes = [(r.nodes, r.budget, "bgk", 19 * 4) for r in serve_requests(case, 0)]
    elif case["kind"] == "batch":
        sizes = [(int(np.prod(c.nodes)), case["steps"], c.collision, 32) for c in batch_decks(case, 0)]
    else:
        sizes = [(case["nx"] * case["ny"] * case["nz"], case["steps"], case["collision"], 32)]
    es = BYTES[case["tier"]]
    return {"bytes": sum(n * (k * (38 * es + 1) + out) for n, k, _, out in sizes),
            "flops": sum(n * k * (220 if col == "bgk" else 340) for n, k, col, _ in sizes)}


# ------------------------------------------------- the same flows in 64 bits, in plain torch
E = [(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (1, 1, 0), (-1, -1, 0),
     (1, -1, 0), (-1, 1, 0), (1, 0, 1), (-1, 0, -1), (1, 0, -1), (-1, 0, 1), (0, 1, 1), (0, -1, -1), (0, 1, -1),
     (0, -1, 1)]
W = [1 / 3] + [1 / 18] * 6 + [1 / 36] * 12
OPP = [E.index((-x, -y, -z)) for x, y, z in E]
RATES = (1.19, 1.4, 1.2, 1.4, 1.98, 0.0, -475.0 / 63.0, 0.0)


def moment_basis():
    rows = []
    for x, y, z in E:
        c = x * x + y * y + z * z
        a, b, g = 3 * x * x - c, y * y - z * z, 3 * c - 5
        rows.append([1, 19 * c - 30, (21 * c * c - 53 * c + 24) / 2, x, (5 * c - 9) * x, y, (5 * c - 9) * y, z,
                     (5 * c - 9) * z, a, g * a, b, g * b, x * y, y * z, x * z, (y * y - z * z) * x,
                     (z * z - x * x) * y, (x * x - y * y) * z])
    return torch.tensor(rows, dtype=torch.float64).T.contiguous()


def dot(i, a):
    out = 0.0
    for d in range(3):
        if E[i][d]:
            out = out + a[d] if E[i][d] > 0 else out - a[d]
    return out


def equilibrium(i, rho, u, uu):
    eu = dot(i, u)
    return W[i] * rho * (1 + 3 * eu + 4.5 * eu * eu - 1.5 * uu)


class Plain:
    """A deck in lattice units (dx = dt = 1), node arrays as (z, y, x)."""

    def __init__(self, c, shear):
        self.c, self.n = c, c.nodes
        nx, ny, nz = self.n
        g = torch.meshgrid(*[torch.arange(m, dtype=torch.float64, device="cuda") for m in (nz, ny, nx)], indexing="ij")
        self.wall = torch.zeros((nz, ny, nx), dtype=torch.bool, device="cuda")
        for _, _, (center, r) in c.obstacles:
            self.wall |= sum((g[2 - d] - center[d]) ** 2 for d in range(3)) <= r * r
        self.any_wall = bool(self.wall.any())
        self.f = torch.empty((19, nz, ny, nx), dtype=torch.float64, device="cuda")
        zero = torch.zeros((), dtype=torch.float64, device="cuda")
        u = [zero] * 3 if shear is None else [v - v / (0.5 * (nz - 1)) * g[0] for v in shear]
        for i in range(19):
            self.f[i] = equilibrium(i, 1.0, u, sum(v * v for v in u))
        self.M = moment_basis().cuda()
        self.inv = torch.linalg.inv(self.M)
        self.rates = c.mrt_rates or RATES

    def macro(self):
        rho = self.f.sum(0)
        u = torch.stack([sum((self.f[i] if E[i][d] > 0 else -self.f[i]) for i in range(19) if E[i][d]) for d in range(3)])
        u /= rho
        if self.any_wall:
            rho = torch.where(self.wall, 0.0, rho)
            u = torch.where(self.wall, 0.0, u)
        return rho, u

    def collide(self):
        f, om = self.f, 1.0 / self.c.tau
        rho = f.sum(0)
        if self.c.collision == "bgk":
            u = [sum((f[i] if E[i][d] > 0 else -f[i]) for i in range(19) if E[i][d]) / rho for d in range(3)]
            uu = sum(v * v for v in u)
            out = torch.empty_like(f)
            for i in range(19):
                out[i] = f[i] + om * (equilibrium(i, rho, u, uu) - f[i])
        else:
            s_e, s_eps, s_q, s_pi, s_m, w_eps, w_epsj, w_xx = self.rates
            m = (self.M @ f.reshape(19, -1)).reshape(f.shape)
            jx, jy, jz = m[3], m[5], m[7]
            jj, pxx, pww = jx * jx + jy * jy + jz * jz, 2 * jx * jx - jy * jy - jz * jz, jy * jy - jz * jz
            m[1] = s_e * (m[1] + 11 * rho - 19 * jj)
            m[2] = s_eps * (m[2] - w_eps * rho - w_epsj * jj)
            for q, j in ((4, jx), (6, jy), (8, jz)):
                m[q] = s_q * (m[q] + 2 / 3 * j)
            m[9], m[11] = om * (m[9] - pxx), om * (m[11] - pww)
            m[10], m[12] = s_pi * (m[10] - w_xx * pxx), s_pi * (m[12] - w_xx * pww)
            m[13], m[14], m[15] = om * (m[13] - jx * jy), om * (m[14] - jy * jz), om * (m[15] - jx * jz)
            m[16:] *= s_m
            for k in (0, 3, 5, 7):
                m[k] = 0.0
            out = f - (self.inv @ m.reshape(19, -1)).reshape(f.shape)
        if any(self.c.Fext):
            for i in range(1, 19):
                out[i] += 3 * W[i] * sum(e * a for e, a in zip(E[i], self.c.Fext)) * rho
        self.f = torch.where(self.wall, f, out) if self.any_wall else out

    def face(self, region):
        axis, last = {"yz": 0, "xz": 1, "xy": 2}[region[5:7]], region.endswith("_l")
        at = [slice(None)] * 3
        at[2 - axis] = -1 if last else 0
        inside = list(at)
        inside[2 - axis] = -2 if last else 1
        return axis, -1 if last else 1, tuple(at), tuple(inside)

    def stream(self):
        f, new = self.f, torch.empty_like(self.f)
        for i in range(19):
            new[i] = torch.roll(f[i], (E[i][2], E[i][1], E[i][0]), (0, 1, 2))
            if i and self.any_wall:
                new[i] = torch.where(torch.roll(self.wall, (E[i][2], E[i][1], E[i][0]), (0, 1, 2)), f[OPP[i]], new[i])
            for d in range(3):
                if E[i][d] and not self.c.periodic[d]:
                    at = [slice(None)] * 3
                    at[2 - d] = 0 if E[i][d] > 0 else -1
                    new[i][tuple(at)] = f[OPP[i]][tuple(at)]
        for op in self.c.pre_stream_bcs:  # a wall moving in its own plane, on the z face
            if op.name == "cavity_z_l":
                u = [v * (1 + 0.5 / (self.n[2] - 1)) for v in op.slots["U"]]
                for i in range(19):
                    if E[i][2] == -1:
                        new[i][-1] += 6 * W[i] * sum(e * v for e, v in zip(E[i], u))
        outlet = [r for op in self.c.boundary_conditions if op.name == "zero_gradient" for r in op.slots["regions"]]
        for r in outlet:
            axis, sign, at, inside = self.face(r)
            for i in range(19):
                if E[i][axis] == sign:
                    new[i][at] = new[i][inside]
        self.f = new
        for op in self.c.post_stream_bcs + self.c.boundary_conditions:
            if op.name in ("neumann", "lid_driven_cavity"):
                for r in op.slots["regions"]:
                    self.velocity_face(r, op.slots["U"], op.name == "neumann")

    def velocity_face(self, region, U, zou_he):
        axis, sign, at, _ = self.face(region)
        v = [self.f[i][at].clone() for i in range(19)]
        if not zou_he:
            rho, uu = sum(v), sum(a * a for a in U)
            new = {i: equilibrium(i, rho, U, uu) for i in range(19)}
        else:
            flat = [i for i in range(19) if E[i][axis] == 0]
            rho = (sum(v[i] for i in flat) + 2 * sum(v[i] for i in range(19) if E[i][axis] == -sign)) / (1 - sign * U[axis])
            slip = [0.0] * 3
            for t in range(3):
                if t != axis:
                    slip[t] = 0.5 * (sum(v[i] for i in flat if E[i][t] == 1) - sum(v[i] for i in flat if E[i][t] == -1)) - rho * U[t] / 3
            new = {}
            for i in range(19):
                if E[i][axis] == sign:
                    along = [t for t in range(3) if t != axis and E[i][t]]
                    new[i] = v[OPP[i]] + (1 / 6 if along else 1 / 3) * rho * dot(i, U)
                    for t in along:
                        new[i] = new[i] - E[i][t] * slip[t]
        fluid = ~self.wall[at]
        for i, value in new.items():
            self.f[i][at] = torch.where(fluid, value, v[i])

    def step(self, n):
        for _ in range(n):
            self.collide()
            self.stream()
        return self


def exact(case, seed):
    if case["kind"] == "serve":
        return [Plain(r.case, None).step(r.budget).f.cpu() if not r.case.obstacles else None
                for r in serve_requests(case, seed)]
    if case["kind"] == "batch":
        return [[t.cpu() for t in Plain(c, None).step(case["steps"]).macro()] for c in batch_decks(case, seed)]
    p = Plain(*solve_parts(case, seed))
    if case["kind"] == "monitor":
        stats = []
        for _ in range(case["steps"] // case["every"]):
            rho, u = p.step(case["every"]).macro()
            speed = (u * u).sum(0).sqrt()
            stats.append([float(rho.sum()), float(speed.min()), float(speed.max())])
        return {"stats": np.array(stats), "fields": [t.cpu() for t in p.macro()]}
    return [t.cpu() for t in p.step(case["steps"]).macro()]
