"""The work that programs built on this framework have it do, as cases to time and to compare.

Every case is one of the framework's configurations, or that configuration at another size of its range:

  mpm3     ParticleSimulation3: a few steps of a 3D dam break or drop, its grid and positions handed on as device
           buffers (what a renderer on the same GPU takes each frame)
  mpm2     ParticleSimulation: a frame of the 2D dam break, its positions and grid read back
  batch    BatchSimulation: many uneven 2D scenes stepped together, their grids read back
  swe      PatchSimulation: a slice of time of a shallow-water patch
  learned  one interval of the learned coarse shallow-water solver from a kept start state
  train    FluxNet: the loss and the gradients of one training batch

Particles start as the configurations' do (uniform in their cell, jittered from the seed), with a slow swirl for a
velocity, and no closer than JITTER_EDGE to where the sort's cells change, so that the order of the particles in the
first passes is that of their first cells and outputs can be compared slot by slot.
"""
import importlib
import math
import os

import numpy as np
import torch

vf = importlib.import_module("vexelray-sim-fluid_b200")

DEV = "cuda"
JITTER_EDGE = 0.02        # cells
INTERVAL = 3753888        # ticks of the learned solver's interval, as its network was trained
NEVER = 2 ** 31 - 1       # a step budget that does not stop the steps
GRAVITY = 9.8
TAIT_K = 50.0             # m^2/s^2, rho0 = 1


# ------------------------------------------------------------------------------------------------- the cases

def listed():
    return [
        # the 3D configuration: 256^3 nodes, 8.16M particles at 8 a cell, sorted every step, tiled scatter
        {"name": "dam3_256", "kind": "mpm3", "shape": "dam", "nx": 256, "ny": 256, "nz": 256, "fill": 0.3825, "tension": False,
         "schedule": "tile", "graph": False, "steps": 4},
        # the reference's own scale of scene, interactive: a radius-8 drop with surface tension, replayed from graphs
        {"name": "drop3_40_tension", "kind": "mpm3", "shape": "drop", "nx": 40, "ny": 40, "nz": 40, "fill": 0.2, "tension": True,
         "schedule": "auto", "graph": True, "steps": 8},
        # an ordinary scene in an odd box, no tension, the schedule left to the framework (0.3M particles)
        {"name": "dam3_odd_96", "kind": "mpm3", "shape": "dam", "nx": 101, "ny": 87, "nz": 93, "fill": 0.4, "tension": False,
         "schedule": "auto", "graph": True, "steps": 8},
        # a large drop with surface tension on the tiled schedule (1.9M particles in 192^3)
        {"name": "drop3_192_tension", "kind": "mpm3", "shape": "drop", "nx": 192, "ny": 192, "nz": 192, "fill": 0.2,
         "tension": True, "schedule": "tile", "graph": False, "steps": 4},
        # the 2D configuration: 128^2, 4 a cell, Tait pressure, sticky walls, sorted every 10 steps; a frame of 20 steps
        {"name": "dam2_128", "kind": "mpm2", "n": 128, "ny": 128, "count": 8192, "graph": True, "steps": 20},
        # the largest scene of the batch's ranges stepped by itself, launch by launch (the default)
        {"name": "dam2_512", "kind": "mpm2", "n": 512, "ny": 512, "count": 262144, "graph": False, "steps": 20},
        # the batched configuration: 256 scenes, 4k to 262k particles, grids of 64^2 to 512^2
        {"name": "batch_256", "kind": "batch", "scenes": 256, "steps": 64, "low": 4096, "high": 262144, "fields": 1},
        # the shallow-water configuration: 4096^2 cells, bit for bit the reference's arithmetic (the default)
        {"name": "swe_4096", "kind": "swe", "nx": 4096, "ny": 4096, "dx": 1.0, "exact": True, "open": False, "ticks": 1000000},
        # an interactive patch of odd width with an open side, a frame of 1/60 s
        {"name": "swe_201x117_frame", "kind": "swe", "nx": 201, "ny": 117, "dx": 0.05, "exact": True, "open": True,
         "ticks": 16667},
        # the fast arithmetic at the learned configuration's fine size
        {"name": "swe_fast_2048", "kind": "swe", "nx": 2048, "ny": 2048, "dx": 1.0, "exact": False, "open": False,
         "ticks": 1000000},
        # the learned solver's interval at its configuration's size: the network's correction and 16 coarse steps
        {"name": "learned_1024", "kind": "learned", "nx": 1024, "ny": 1024},
        # a training batch of the learned configuration: four 1024^2 samples, forward and backward
        {"name": "train_1024x4", "kind": "train", "nx": 1024, "ny": 1024, "batch": 4},
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(("mpm3", "mpm3", "mpm2", "batch", "swe", "swe", "learned", "train"))
    if kind == "mpm3":
        n = log_int(32, 220)
        return {"kind": kind, "shape": rng.choice(("dam", "drop")), "nx": n, "ny": log_int(max(24, 0.7 * n), n),
                "nz": log_int(max(24, 0.7 * n), n), "fill": round(rng.uniform(0.2, 0.4), 3), "tension": rng.random() < 0.4,
                "schedule": rng.choice(("tile", "auto", "auto")), "graph": rng.random() < 0.5, "steps": 4}
    if kind == "mpm2":
        n = log_int(64, 512)
        return {"kind": kind, "n": n, "ny": log_int(max(48, 0.6 * n), n), "count": log_int(1024, max(2048, n * n)),
                "graph": rng.random() < 0.5, "steps": 20}
    if kind == "batch":
        return {"kind": kind, "scenes": log_int(4, 128), "steps": 32, "low": 4096, "high": log_int(16384, 262144), "fields": 1}
    if kind == "swe":
        nx = log_int(64, 4000)
        return {"kind": kind, "nx": nx, "ny": log_int(max(32, nx // 4), nx), "dx": 1.0, "exact": rng.random() < 0.6,
                "open": rng.random() < 0.3, "ticks": 1000000}
    nx = log_int(128, 1000)
    ny = log_int(max(64, nx // 2), nx)
    return {"kind": "learned", "nx": nx, "ny": ny} if kind == "learned" else \
        {"kind": "train", "nx": nx, "ny": ny, "batch": rng.randint(1, 4)}


# ------------------------------------------------------------------------------------------------- inputs

def jitter(rng, shape):
    """Uniform in a cell, JITTER_EDGE away from its sides and its middle (the two sorts' cell borders)."""
    t = rng.random(shape, dtype=np.float32) * np.float32(2.0)
    half = np.floor(t)
    return half * np.float32(0.5) + np.float32(JITTER_EDGE) + (t - half) * np.float32(0.5 - 2 * JITTER_EDGE)


def mpm3_inputs(case, seed):
    """Positions, velocities, masses, Flip3.params values: a dam in the low corner or a drop in the middle, 8 a cell."""
    rng = np.random.default_rng(seed)
    size = (case["nx"], case["ny"], case["nz"])
    if case["shape"] == "dam":
        ranges = [np.arange(math.ceil(0.05 * n - 0.5), math.ceil((0.05 + f) * n - 0.5), dtype=np.float32)
                  for n, f in zip(size, (0.4, case["fill"], 0.4))]
        cz, cy, cx = np.meshgrid(ranges[2], ranges[1], ranges[0], indexing="ij")
        cells = np.stack([cx.ravel(), cy.ravel(), cz.ravel()], axis=1)
        g = -GRAVITY * size[1]
        bulk = 25 * 2 * -g * len(ranges[1])          # (5 sqrt(2 g H))^2
        dt = min(5e-5 * 256 / max(size), 0.2 / math.sqrt(bulk))
        sigma = 100.0 if case["tension"] else 0.0
    else:
        r = case["fill"] * min(size)
        a = [np.arange(int(n / 2 - r) - 1, int(n / 2 + r) + 2, dtype=np.float32) for n in size]
        cz, cy, cx = np.meshgrid(a[2], a[1], a[0], indexing="ij")
        at = np.stack([cx.ravel(), cy.ravel(), cz.ravel()], axis=1)
        d = at + 0.5 - np.array(size, np.float32) / 2
        cells = at[(d * d).sum(1) <= r * r]
        g, bulk, sigma = 0.0, 200.0 ** 2, 100.0 if case["tension"] else 0.0
        dt = 0.3 / 220
    cells = np.repeat(cells, 8, axis=0)
    pos = (cells + jitter(rng, cells.shape)).astype(np.float32)
    at = [np.ascontiguousarray(pos[:, a]) for a in range(3)]
    amp, k = 0.004 / (case["steps"] * dt), 2 * math.pi / max(size)
    vel = [(amp * np.sin(k * at[(a + 1) % 3])).astype(np.float32) for a in range(3)]
    m = np.full(len(at[0]), 1 / 8, np.float32)
    return at, vel, m, (dt, 0.0, g, 0.0, bulk, 1.0, sigma)


def mpm2_scene(rng, nx, ny, count, ppc=4, lo=4):
    """A dam in the low corner, `ppc` a cell where it fits (more where it cannot); Flip.params values."""
    area = count / ppc
    aspect = math.exp(rng.uniform(math.log(0.5), math.log(2.0)))
    w = int(min(nx - 2 * lo, max(1, round(math.sqrt(area * aspect)))))
    h = int(min(ny - 2 * lo, max(1, math.ceil(area / w))))
    cell = np.arange(count) % (w * h)
    j = jitter(rng, (2, count))
    x = ((lo + cell % w).astype(np.float32) + j[0]).astype(np.float32)
    y = ((lo + cell // w).astype(np.float32) + j[1]).astype(np.float32)
    n = max(nx, ny)
    dt = min(1e-4, 0.4 / (math.sqrt(7 * TAIT_K) * n))
    u = (0.004 * n * np.sin(y * np.float32(2 * math.pi / n))).astype(np.float32)
    v = (0.004 * n * np.sin(x * np.float32(2 * math.pi / n))).astype(np.float32)
    m = np.full(count, w * h / count, np.float32)
    return [x, y], [u, v], m, (dt, 0.0, -GRAVITY * n, TAIT_K * n * n, 1.0)


def batch_inputs(case, seed):
    rng = np.random.default_rng(seed)
    out = []
    shapes = np.random.default_rng(case["scenes"])   # the scenes' sizes go with the case, their particles with the seed
    for _ in range(case["scenes"]):
        n = int(shapes.choice((64, 128, 256, 512)))
        count = int(round(math.exp(shapes.uniform(math.log(case["low"]), math.log(case["high"])))))
        out.append((n, count) + mpm2_scene(rng, n, n, count))
    return out


def bumps(nx, ny, seed, still):
    """h = 1 + 16 seeded Gaussian bumps (the 4096^2 configuration's, scaled with the patch) and its momenta: none, or
    those of a moving sea. float32 tensors on the GPU."""
    rng = np.random.default_rng(seed)
    s = max(max(nx, ny) / 4096, 1 / 16)
    x = torch.arange(nx, dtype=torch.float32, device=DEV)
    y = torch.arange(ny, dtype=torch.float32, device=DEV)[:, None]
    h = torch.ones(ny, nx, device=DEV)
    for _ in range(16):
        amp, sig = rng.uniform(0.1, 0.5), rng.uniform(20, 200) * s
        cx, cy = rng.uniform(0, nx), rng.uniform(0, ny)
        h += amp * torch.exp(-((x - cx) ** 2) / (2 * sig * sig)) * torch.exp(-((y - cy) ** 2) / (2 * sig * sig))
    if still:
        return [h, torch.zeros_like(h), torch.zeros_like(h)]
    k = [2 * math.pi * rng.uniform(1, 4) / max(nx, ny) for _ in range(4)]
    hu = 0.2 * h * torch.sin(k[0] * x + k[1] * y)
    hv = 0.2 * h * torch.cos(k[2] * x - k[3] * y)
    return [h, hu, hv]


def training_samples(case, seed):
    """(S, P, T) per sample: a moving sea; the state an interval later (another sea); the same with a residual of the
    size that the network is trained to take away."""
    nx, ny, out = case["nx"], case["ny"], []
    x = torch.arange(nx, dtype=torch.float32, device=DEV)
    y = torch.arange(ny, dtype=torch.float32, device=DEV)[:, None]
    for b in range(case["batch"]):
        rng = np.random.default_rng((seed, b))
        P = bumps(nx, ny, int(rng.integers(1 << 30)), still=False)
        T = []
        for p in P:
            k = [2 * math.pi * rng.uniform(4, 64) / max(nx, ny) for _ in range(4)]
            T.append(p + 1e-3 * (torch.sin(k[0] * x + k[1] * y) + torch.cos(k[2] * x - k[3] * y)))
        out.append((bumps(nx, ny, int(rng.integers(1 << 30)), still=False), P, T))
    return out


def trained_weights():
    return np.load(os.path.join("vexelray-sim-fluid_b200", "learned_2048_k16.npy"))


def host(planes):
    return [p.cpu().numpy().ravel() for p in planes]


# ------------------------------------------------------------------------------------------------- the program

class DeviceBuffer:
    """A handle's device memory as torch takes it; it keeps the handle alive."""

    def __init__(self, ptr, shape, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f4", "data": (ptr, False), "version": 2}


def view(state, ptr, shape):
    """The tensor over a handle's buffer (a handle alternates between two of each, wrapped once each)."""
    t = state["views"].get(ptr)
    if t is None:
        t = state["views"][ptr] = torch.as_tensor(DeviceBuffer(ptr, shape, state["sim"]), device=DEV)
    return t


EDGES = {False: (vf.EDGE_WALL,) * 4, True: (vf.EDGE_OPEN, vf.EDGE_WALL, vf.EDGE_WALL, vf.EDGE_WALL)}


def prepare(case, seed):
    torch.zeros(1, device=DEV)
    kind, state = case["kind"], {"case": case, "views": {}}
    if kind == "mpm3":
        at, vel, m, p = mpm3_inputs(case, seed)
        sim = vf.ParticleSimulation3(case["nx"], case["ny"], case["nz"], len(m), tension=case["tension"],
                                     schedule={"tile": vf.VF_P2G_TILE, "auto": vf.VF_P2G_AUTO}[case["schedule"]])
        sim.set_graph(case["graph"])
        sim.load(at, vel, m, vf.flip3_params(*p))
    elif kind == "mpm2":
        at, vel, m, p = mpm2_scene(np.random.default_rng(seed), case["n"], case["ny"], case["count"])
        sim = vf.ParticleSimulation(case["n"], case["ny"], case["count"], tait=True, sticky=3)
        sim.set_graph(case["graph"])
        sim.load(*at, *vel, m, vf.flip_params(*p))
    elif kind == "batch":
        scenes = batch_inputs(case, seed)
        sim = vf.BatchSimulation([vf.Scene(n, n, count, vf.flip_params(*p)) for n, count, _, _, _, p in scenes], tait=True,
                                 sticky=3)
        sim.load([s[2][0] for s in scenes], [s[2][1] for s in scenes], [s[3][0] for s in scenes], [s[3][1] for s in scenes],
                 [s[4] for s in scenes])
    elif kind == "swe":
        sim = vf.PatchSimulation(case["nx"], case["ny"], EDGES[case["open"]])
        sim.set_exact(case["exact"])
        sim.load(*host(bumps(case["nx"], case["ny"], seed, still=True)), vf.swe_params(9.81, 0.45, case["dx"], case["dx"], 1e-6))
    elif kind == "learned":
        sim = vf.PatchSimulation(case["nx"], case["ny"])
        start = vf.PatchSimulation(case["nx"], case["ny"])
        for s in (sim, start):
            s.load(*host(bumps(case["nx"], case["ny"], seed, still=False)), vf.swe_params(9.81, 0.45, 2.0, 2.0, 1e-6))
        net = vf.FluxNet(case["nx"], case["ny"], s_flux=1e-3, s_res=1e-3)
        net.params(trained_weights())
        state.update(start=start, net=net)
    else:
        sim = vf.FluxNet(case["nx"], case["ny"], batch=case["batch"], samples=case["batch"], s_flux=1e-3, s_res=1e-3)
        sim.params(trained_weights())
        for slot, sample in enumerate(training_samples(case, seed)):
            for part, planes in enumerate(sample):
                sim.put(slot, part, *host(planes))
    state["sim"] = sim
    return state


def run(state):
    case, sim = state["case"], state["sim"]
    kind = case["kind"]
    if kind == "mpm3":
        sim.advance(case["steps"])
        nodes = case["nx"] * case["ny"] * case["nz"]
        out = {"grid": view(state, sim.device_ptr("gm")[0], (nodes, 4))}
        for a in "xyz":
            out[a] = view(state, sim.device_ptr(a)[0], (sim.particles(),))
        return out
    if kind == "mpm2":
        sim.advance(case["steps"], 10)
        return {"at": sim.positions(), "grid": sim.grid()}
    if kind == "batch":
        sim.advance(case["steps"])
        return {f: np.concatenate([sim.read(s, f) for s in range(case["scenes"])]) for f in ("gm", "gmu", "gmv")[:case["fields"]]}
    if kind == "swe":
        sim.advance(case["ticks"], NEVER)
    elif kind == "learned":
        sim.copy_from(state["start"])
        state["net"].predict(sim)
        sim.advance(INTERVAL, 1024)
        state["net"].apply(sim)
    else:
        gradients, loss = sim.gradients(list(range(case["batch"])))
        return {"gradients": gradients, "loss": loss}
    shape = (case["ny"], case["nx"])
    return {f: view(state, p.value, shape) for f, p in zip(("h", "hu", "hv"), sim.device_state())}


def work(case):
    """A step reads its state and writes it once; nodes with mass are written by the scatter and read by the gather."""
    kind = case["kind"]
    if kind == "mpm3":
        if case["shape"] == "dam":
            cells = 0.4 * case["nx"] * case["fill"] * case["ny"] * 0.4 * case["nz"]
        else:
            cells = 4 / 3 * math.pi * (case["fill"] * min(case["nx"], case["ny"], case["nz"])) ** 3
        return {"bytes": case["steps"] * cells * (8 * 2 * 17 * 4 + 2 * 16), "flops": case["steps"] * cells * 8 * 27 * 30}
    if kind == "mpm2":
        count = case["count"]
        return {"bytes": case["steps"] * (count * 2 * 10 * 4 + count / 4 * 2 * 12), "flops": case["steps"] * count * 9 * 25}
    if kind == "batch":
        lo, hi = case["low"], case["high"]
        count = case["scenes"] * (hi - lo) / math.log(hi / lo)
        return {"bytes": case["steps"] * (count * 2 * 10 * 4 + count / 4 * 2 * 12), "flops": case["steps"] * count * 9 * 25}
    cells = case["nx"] * case["ny"]
    if kind == "swe":
        steps = max(1, math.ceil(case["ticks"] / (0.45 * case["dx"] / 4.2 * 1e6)))
        return {"bytes": steps * cells * 24, "flops": steps * cells * 120}
    conv = 2 * 25 * (3 * 32 + 32 * 32 + 32 * 6)
    if kind == "learned":
        return {"bytes": cells * (16 * 24 + 2 * 24), "flops": cells * (conv + 16 * 120)}
    # the gradients of the weights, and of the two hidden layers, cost what the forward pass does
    return {"bytes": case["batch"] * cells * 36, "flops": case["batch"] * cells * (2 * conv + 2 * 25 * (32 * 32 + 32 * 6))}


# ------------------------------------------------------------------------------------------------- in 64 bits

def held(n, at):
    return at.clamp(1, n - 2)


class Particles64:
    """MLS-MPM with the quadratic spline and APIC in float64, over any number of scenes in two or three dimensions:
    a scene's nodes lie one after another from its base, x fastest."""

    def __init__(self, scenes, tait, sticky, tension):
        one = len(scenes) == 1

        def spread(values, counts):
            v = torch.tensor(values, dtype=torch.float64, device=DEV)
            return v[0] if one else v.repeat_interleave(torch.tensor(counts, device=DEV))

        d = len(scenes[0][0])
        sizes = [s[0] for s in scenes]
        nodes = [math.prod(s) for s in sizes]
        counts = [len(s[3]) for s in scenes]
        base = np.concatenate([[0], np.cumsum(nodes)])
        self.d, self.nodes, self.tait, self.sticky, self.tension = d, int(base[-1]), tait, sticky, tension
        self.x = [torch.from_numpy(np.concatenate([s[1][a] for s in scenes])).to(DEV).double() for a in range(d)]
        self.v = [torch.from_numpy(np.concatenate([s[2][a] for s in scenes])).to(DEV).double() for a in range(d)]
        self.m = torch.from_numpy(np.concatenate([s[3] for s in scenes])).to(DEV).double()
        self.j = torch.ones_like(self.m)
        self.c = [[torch.zeros_like(self.m) for _ in range(d)] for _ in range(d)]
        f32 = [[float(np.float32(v)) for v in s[4]] for s in scenes]    # dt, gravity (d), bulk, rho0[, sigma]
        self.n = [spread([s[a] for s in sizes], counts) for a in range(d)]
        self.base = spread(base[:-1].tolist(), counts)
        self.dt, self.bulk, self.rho0 = (spread([p[k] for p in f32], counts) for k in (0, 1 + d, 2 + d))
        self.node_dt = spread([p[0] for p in f32], nodes)
        self.node_g = [spread([p[1 + a] for p in f32], nodes) for a in range(d)]
        self.node_n = [spread([s[a] for s in sizes], nodes) for a in range(d)]
        self.at = [torch.cat([(torch.arange(k, device=DEV) // math.prod(s[:a])) % s[a] for s, k in zip(sizes, nodes)]).double()
                   for a in range(d)]
        self.size, self.sigma, self.rest = sizes[0], f32[0][-1], f32[0][2 + d]

    def stencil(self):
        cell, off, w = [], [], []
        for a in range(self.d):
            x = torch.minimum(self.x[a].clamp(min=0.5), self.n[a] - 1.5)
            c = torch.minimum(torch.floor(x - 0.5), self.n[a] - 3)
            f = x - c
            cell.append(c)
            off.append(f)
            w.append([0.5 * (1.5 - f) ** 2, 0.75 - (f - 1) ** 2, 0.5 * (f - 0.5) ** 2])
        return cell, off, w

    def nodes_of(self, cell, off, w):
        for k in range(3 ** self.d):
            o = [(k // 3 ** a) % 3 for a in range(self.d)]
            node, stride, weight = self.base, 1.0, 1.0
            for a in range(self.d):
                node = node + (cell[a] + o[a]) * stride
                stride = stride * self.n[a]
                weight = weight * w[a][o[a]]
            yield node.long(), weight, [o[a] - off[a] for a in range(self.d)]

    def step(self):
        d = self.d
        cell, off, w = self.stencil()
        jp = self.bulk * (self.j ** -6 - self.j) if self.tait else self.bulk * (1 - self.j)
        s = 4 * self.dt * self.m / self.rho0 * jp
        self.grid = [torch.zeros(self.nodes, dtype=torch.float64, device=DEV) for _ in range(d + 1)]
        for node, weight, dd in self.nodes_of(cell, off, w):
            wm = weight * self.m
            self.grid[0].index_add_(0, node, wm)
            for a in range(d):
                vel = self.v[a] + sum(self.c[a][e] * dd[e] for e in range(d))
                self.grid[1 + a].index_add_(0, node, wm * vel + weight * s * dd[a])
        mass = self.grid[0]
        full = mass > 1e-9
        safe = torch.where(full, mass, 1.0)
        vel = [torch.where(full, self.grid[1 + a] / safe + self.node_dt * self.node_g[a], 0.0) for a in range(d)]
        if self.tension:
            force = self.tension_force()
            push = torch.where(full, self.node_dt * self.sigma / mass.clamp(min=float(np.float32(0.3)) * self.rest), 0.0)
            vel = [vel[a] + push * force[a].reshape(-1) for a in range(d)]
        for a in range(d):
            if self.sticky:
                for b in range(d):
                    stuck = (self.at[b] < self.sticky) | (self.at[b] > self.node_n[b] - 1 - self.sticky)
                    vel[a] = torch.where(stuck, 0.0, vel[a])
            else:
                vel[a] = torch.where(self.at[a] <= 1, vel[a].clamp(min=0), vel[a])
                vel[a] = torch.where(self.at[a] > self.node_n[a] - 3, vel[a].clamp(max=0), vel[a])
        v = [0.0] * d
        b = [[0.0] * d for _ in range(d)]
        for node, weight, dd in self.nodes_of(cell, off, w):
            for a in range(d):
                part = weight * vel[a][node]
                v[a] = v[a] + part
                for e in range(d):
                    b[a][e] = b[a][e] + part * dd[e]
        self.c = [[4 * b[a][e] for e in range(d)] for a in range(d)]
        self.j = (self.j * (1 + self.dt * sum(self.c[a][a] for a in range(d)))).clamp(0.1, 10)
        for a in range(d):
            x, hi = self.x[a] + self.dt * v[a], self.n[a] - 2
            v[a] = torch.where(x < 1, v[a].clamp(min=0), v[a])
            v[a] = torch.where(x > hi, v[a].clamp(max=0), v[a])
            self.x[a] = torch.minimum(x.clamp(min=1), hi)
        self.v = v

    def tension_force(self):
        """Surface tension's force over sigma on every node: the mass as a colour, blurred six times, its capillary
        stress, and the stress's flux through a node's open faces. Planes are [z][y][x]; axis a is dimension 2 - a."""
        n = self.size
        idx = [held(n[a], torch.arange(-1, n[a] + 1, device=DEV)) for a in range(3)]

        def wide(p):
            return p[idx[2]][:, idx[1]][:, :, idx[0]]

        def cut(p, a, o):
            return p.narrow(2 - a, 1 + o, n[a])

        colour = self.grid[0].reshape(n[2], n[1], n[0])
        full = torch.full_like(colour, self.rest)
        for a in range(3):
            at = torch.arange(n[a], device=DEV)
            half = torch.where(at == 1, 0.5, 1.0) * torch.where(at == n[a] - 2, 0.5, 1.0)
            full = full * half.double().reshape([-1 if 2 - a == k else 1 for k in range(3)])
        colour = (colour / full).clamp(max=1.0)
        for _ in range(6):
            e = wide(colour)
            for a in range(3):
                e = 0.25 * cut(e, a, -1) + 0.5 * cut(e, a, 0) + 0.25 * cut(e, a, 1)
            colour = e
        e = wide(colour)
        inner = [cut(cut(e, (a + 1) % 3, 0), (a + 2) % 3, 0) for a in range(3)]
        g = [0.5 * (cut(inner[a], a, 1) - cut(inner[a], a, -1)) for a in range(3)]
        length = torch.sqrt(g[0] ** 2 + g[1] ** 2 + g[2] ** 2 + 1e-8)
        t = [[(g[(a + 1) % 3] ** 2 + g[(a + 2) % 3] ** 2) / length if a == c else -g[a] * g[c] / length
              for c in range(3)] for a in range(3)]
        cmin = float(np.float32(0.3))
        at = [torch.arange(n[a], device=DEV).reshape([-1 if 2 - a == k else 1 for k in range(3)]) for a in range(3)]
        ring = colour > cmin
        for a in range(3):
            ring = ring & (at[a] >= 1) & (at[a] <= n[a] - 2)
        force = [torch.zeros_like(colour) for _ in range(3)]
        for a in range(3):
            for sign in (-1, 1):
                there = held(n[a], torch.arange(n[a], device=DEV) + sign)
                openf = (ring & (colour.index_select(2 - a, there) > cmin)).double()
                wall = at[a] <= 1 if sign < 0 else at[a] >= n[a] - 2
                for c in range(3):
                    flux = 0.5 * sign * (t[a][c] + t[a][c].index_select(2 - a, there)) * openf
                    force[c] = force[c] + (flux if c == a else torch.where(wall, 0.0, flux))
        return force


def shallow64(planes, dx, edge_open, ticks, courant=0.45, g=9.81, dry=1e-6):
    """The HLL shallow-water step in float64 over `ticks` microseconds, steps in whole ticks."""
    h, hu, hv = (p.double() for p in planes)
    courant, g, dry, dx = (float(np.float32(v)) for v in (courant, g, dry, dx))
    wall = [0.0 if edge_open else 1.0, 1.0, 1.0, 1.0]     # west, east, south, north

    def over(q, depth):
        return torch.where(depth > dry, q / torch.where(depth > dry, depth, 1.0), 0.0)

    def flux(d, qn, qt):
        """Faces along the last axis of states padded by their ghosts."""
        un, ut, c = over(qn, d), over(qt, d), torch.sqrt(g * d)
        L, R = (lambda p: p[:, :-1]), (lambda p: p[:, 1:])
        sl = torch.minimum(L(un) - L(c), R(un) - R(c))
        sr = torch.maximum(L(un) + L(c), R(un) + R(c))
        dry_r, dry_l = R(d) <= dry, L(d) <= dry
        sl = torch.where(dry_r, L(un) - L(c), sl)
        sr = torch.where(dry_r, L(un) + 2 * L(c), sr)
        sl = torch.where(dry_l, R(un) - 2 * R(c), sl)
        sr = torch.where(dry_l, R(un) + R(c), sr)
        lo, hi = sl.clamp(max=0), sr.clamp(min=0)
        span = (hi - lo).clamp(min=1e-30)

        def combine(f, u):
            return (hi * L(f) - lo * R(f) + lo * hi * (R(u) - L(u))) / span

        return combine(qn, d), combine(qn * un + 0.5 * g * d * d, qn), combine(qn * ut, qt)

    def ghosts(p, low, high):
        return torch.cat([low * p[:, :1], p, high * p[:, -1:]], 1)

    left = ticks
    while left > 0:
        speed = float((torch.maximum(over(hu, h).abs(), over(hv, h).abs()) + torch.sqrt(g * h)).max())
        step = min(left, int(min(courant * dx / max(speed, 1e-30), 2000.0) * 1e6))
        left -= step
        r = step * 1e-6 / dx
        f = flux(ghosts(h, 1, 1), ghosts(hu, 1 - 2 * wall[0], 1 - 2 * wall[1]), ghosts(hv, 1, 1))
        q = flux(ghosts(h.T, 1, 1), ghosts(hv.T, 1 - 2 * wall[2], 1 - 2 * wall[3]), ghosts(hu.T, 1, 1))
        new = []
        for p, fx, fy in ((h, f[0], q[0]), (hu, f[1], q[2]), (hv, f[2], q[1])):
            fy = fy.T
            new.append(p - r * (fx[:, 1:] - fx[:, :-1]) - r * (fy[1:] - fy[:-1]))
        h, hu, hv = new[0].clamp(min=0), new[1], new[2]
    return [h, hu, hv]


class Net64:
    def __init__(self):
        p = torch.from_numpy(trained_weights()).to(DEV).double()
        self.p, at = {}, 0
        for name, shape in (("w1", (32, 25, 3)), ("b1", (32,)), ("w2", (32, 25, 32)), ("b2", (32,)), ("w3", (6, 25, 32)),
                            ("b3", (6,))):
            k = math.prod(shape)
            self.p[name] = p[at:at + k].reshape(shape).clone().requires_grad_(True)
            at += k

    @staticmethod
    def conv(x, w, b):
        """x (channels, H, W), as the sum over taps of matrix products."""
        c, hh, ww = x.shape
        pad = torch.nn.functional.pad(x, (2, 2, 2, 2))
        out = b[:, None].expand(-1, hh * ww)
        for t in range(25):
            out = out + w[:, t] @ pad[:, t // 5:t // 5 + hh, t % 5:t % 5 + ww].reshape(c, -1)
        return out.reshape(-1, hh, ww)

    def correction(self, planes):
        """The divergence of the six face fields, the walls' faces zero: (3, H, W)."""
        h, hu, hv = (q.double() for q in planes)
        x = torch.stack([(h - 1) * 4, hu * 4, hv * 4])
        x = torch.relu(self.conv(x, self.p["w1"], self.p["b1"]))
        x = torch.relu(self.conv(x, self.p["w2"], self.p["b2"]))
        y = self.conv(x, self.p["w3"], self.p["b3"])
        pad = torch.nn.functional.pad
        e, n = pad(y[:3, :, :-1], (1, 1)), pad(y[3:, :-1], (0, 0, 1, 1))
        return e[:, :, 1:] - e[:, :, :-1] + n[:, 1:] - n[:, :-1]


def exact(case, seed):
    kind = case["kind"]
    if kind == "mpm3":
        at, vel, m, p = mpm3_inputs(case, seed)
        n = (case["nx"], case["ny"], case["nz"])
        sim = Particles64([(n, at, vel, m, p)], False, 0, case["tension"])
        cell = [np.minimum(np.floor(at[a] - np.float32(0.5)).astype(np.int64), n[a] - 3) for a in range(3)]
        nb = [(n[a] - 2 + 7) // 8 for a in range(3)]
        brick = ((cell[2] >> 3) * nb[1] + (cell[1] >> 3)) * nb[0] + (cell[0] >> 3)
        order = np.argsort(brick * 512 + ((cell[2] & 7) * 8 + (cell[1] & 7)) * 8 + (cell[0] & 7), kind="stable")
        for _ in range(case["steps"]):
            sim.step()
        order = torch.from_numpy(order).to(DEV)
        return {"grid": torch.stack(sim.grid, 1), **{a: sim.x[k][order] for k, a in enumerate("xyz")}}
    if kind == "mpm2":
        at, vel, m, p = mpm2_scene(np.random.default_rng(seed), case["n"], case["ny"], case["count"])
        sim = Particles64([((case["n"], case["ny"]), at, vel, m, p)], True, 3, False)
        cell = [np.minimum(np.floor(at[a]).astype(np.int64), k - 2) for a, k in enumerate((case["n"], case["ny"]))]
        order = torch.from_numpy(np.argsort(cell[1] * (case["n"] - 1) + cell[0], kind="stable")).to(DEV)
        for _ in range(case["steps"]):
            sim.step()
        return {"at": [x[order] for x in sim.x], "grid": sim.grid}
    if kind == "batch":
        sim = Particles64([((n, n), at, vel, m, p) for n, _, at, vel, m, p in batch_inputs(case, seed)], True, 3, False)
        for _ in range(case["steps"]):
            sim.step()
        return dict(zip(("gm", "gmu", "gmv")[:case["fields"]], sim.grid))
    if kind == "swe":
        out = shallow64(bumps(case["nx"], case["ny"], seed, still=True), case["dx"], case["open"], case["ticks"])
        return dict(zip(("h", "hu", "hv"), out))
    if kind == "learned":
        planes = bumps(case["nx"], case["ny"], seed, still=False)
        with torch.no_grad():
            div = Net64().correction(planes)
        out = [q - float(np.float32(1e-3)) * div[k] for k, q in enumerate(shallow64(planes, 2.0, False, INTERVAL))]
        return {"h": out[0].clamp(min=0), "hu": out[1], "hv": out[2]}
    net, total, terms = Net64(), 0.0, case["batch"] * 3 * case["nx"] * case["ny"]
    for S, P, T in training_samples(case, seed):
        r = (torch.stack([q.double() for q in P]) - 1e-3 * net.correction(S) - torch.stack([q.double() for q in T])) / 1e-3
        loss = (r * r).sum() / (2 * terms)
        loss.backward()
        total += float(loss.detach())
        del r, loss
    return {"gradients": torch.cat([q.grad.reshape(-1) for q in net.p.values()]), "loss": total}
