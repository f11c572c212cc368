"""Performance cases of the solver: what a program using this package has it do, from one small
dam break to a 256-scene ensemble, the reverse pass of a step and a rendered frame.

listed() names the cases, draw() makes more of the same ranges, prepare() builds what a program
holds before the call (device state, a Simulator / Ensemble / SSFRenderer), run() is one pass
through the public API, work() the bytes and flops a pass cannot do without, and exact() the same
result in 64 bits from torch alone.

Every pass starts from the same state: a step permutes its inputs in place (Simulator.step), so
run() first loads the state's positions, velocities and iids into the working buffers, as a
program does that loads a checkpoint.  States are those of a running simulation: particles in the
cell order the previous step left, moving.
"""
import importlib.util
import math
import sys
from pathlib import Path

import numpy as np
import torch

SPACING, JITTER, H = 0.05, 0.005, 0.1


def _pbf():
    """The package (its directory name has a hyphen, so it is loaded by path)."""
    name = "pbf_cuda_gb300"
    if name not in sys.modules:
        root = Path.cwd() / "pbf-cuda_gb300"
        spec = importlib.util.spec_from_file_location(name, root / "__init__.py", submodule_search_locations=[str(root)])
        mod = importlib.util.module_from_spec(spec)
        sys.modules[name] = mod
        spec.loader.exec_module(mod)
    return sys.modules[name]


def _step(name, dims, scene="dam", params="reference", niter=4, vorticity=0.0, boundary=0.0, steps=1):
    c = {"kind": "step", "nx": dims[0], "ny": dims[1], "nz": dims[2], "scene": scene, "params": params, "niter": niter,
         "vorticity": vorticity, "boundary": boundary, "steps": steps}
    return dict(c, name=name) if name else c


def _ensemble(name, scenes, lo, hi, params="dam_break", sides=0):
    c = {"kind": "ensemble", "scenes": scenes, "lo": lo, "hi": hi, "sides": sides, "params": params, "niter": 4}
    return dict(c, name=name) if name else c


def _gradient(name, dims, grid):
    c = {"kind": "gradient", "nx": dims[0], "ny": dims[1], "nz": dims[2], "gx": grid[0], "gy": grid[1], "gz": grid[2],
         "params": "reference", "niter": 4}
    return dict(c, name=name) if name else c


def _ssf(name, dims, size, blur=0, smooth=2, shading=0):
    c = {"kind": "ssf", "nx": dims[0], "ny": dims[1], "nz": dims[2], "width": size[0], "height": size[1], "blur": blur,
         "smooth": smooth, "shading": shading}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest scene of the tests and of the ensemble: launches and latency decide
        _step("step_1728", (12, 12, 12)),
        # the single dam break
        _step("step_8000", (20, 20, 20)),
        # the double dam break with the reference application's moving boundary: every step has new limits
        _step("frames_moving_wall_32768", (16, 32, 32), scene="double_dam_moving", steps=6),
        # the optional terms (vorticity confinement, boundary density) on an odd-sized scene, two iterations
        _step("step_options_65231", (37, 41, 43), niter=2, vorticity=0.05, boundary=0.05),
        # the million-particle scene with the reference's parameters: fluid at rest density
        _step("step_1048576", (128, 64, 128)),
        # the same scene with the benchmark's parameters (particles leave their cells within a step)
        _step("step_1048576_dam_break", (128, 64, 128), params="dam_break"),
        # the state long runs of those parameters end in: cells of 131,072 particles at one position
        _step("step_clustered_1048576", (64, 64, 64), scene="clustered", params="dam_break"),
        # 256 uneven scenes in one launch per pass
        _ensemble("ensemble_256", 256, 12, 40),
        # one evaluation of the inverse problem on one step: taped step, density loss, reverse pass
        _gradient("gradient_15625", (25, 25, 25), (32, 16, 16)),
        # the reverse pass where one thread takes a particle
        _gradient("gradient_262144", (64, 64, 64), (32, 32, 32)),
        # a frame of the fluid surface at the reference's window size, its default settings
        _ssf("ssf_1048576_1600x1200", (128, 64, 128), (1600, 1200)),
        # a small preview frame: gaussian filter, three passes
        _ssf("ssf_32768_640x480", (32, 32, 32), (640, 480), blur=1, smooth=3),
    ]


def _draw_dims(rng, lo, hi):
    """Three lattice sides, odd ones among them, of about a log-uniform particle count in [lo, hi]."""
    n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    side = n ** (1.0 / 3.0)
    a = max(4, round(side * rng.uniform(0.75, 1.35)))
    b = max(4, round(side * rng.uniform(0.75, 1.35)))
    return a, b, max(4, int(n / (a * b)))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "step", "ensemble", "gradient", "ssf"])
    if kind == "step":
        scene = rng.choice(["dam", "dam", "double_dam_moving", "clustered"])
        if scene == "clustered":
            return _step(None, _draw_dims(rng, 8000, 262144), scene=scene, params="dam_break")
        if scene == "double_dam_moving":
            return _step(None, _draw_dims(rng, 800, 65536), scene=scene, steps=rng.randint(2, 6))
        params = rng.choice(["reference", "reference", "dam_break"])
        return _step(None, _draw_dims(rng, 700, 1048576), params=params, niter=rng.choice([1, 2, 3, 4, 4, 6]),
                     vorticity=rng.choice([0.0, 0.0, 0.05]), boundary=rng.choice([0.0, 0.0, 0.05]))
    if kind == "ensemble":
        lo = rng.randint(8, 14)
        return _ensemble(None, round(math.exp(rng.uniform(math.log(2), math.log(250)))), lo, rng.randint(lo + 2, 38),
                         params=rng.choice(["dam_break", "reference"]), sides=rng.randint(1, 1 << 20))
    if kind == "gradient":
        return _gradient(None, _draw_dims(rng, 500, 262144), (rng.randint(9, 32), rng.randint(9, 32), rng.randint(9, 32)))
    return _ssf(None, _draw_dims(rng, 2000, 1048576), (rng.randint(160, 800) * 2 + rng.randint(0, 1), rng.randint(120, 600) * 2),
                blur=rng.choice([0, 0, 1]), smooth=rng.randint(1, 3), shading=rng.choice([0, 0, 3, 4, 7]))


# ---- inputs --------------------------------------------------------------------------------


def _params(case):
    """The solver parameters of a case, y up: the reference's defaults, or the dam-break benchmark's."""
    scenes = _pbf().scenes
    if case["params"] == "dam_break":
        p = scenes.scene_params(case["niter"])
    else:
        p = scenes.reference_params()
        p.niter = case["niter"]
        p.up[0], p.up[1], p.up[2] = 0.0, 1.0, 0.0
    p.vorticity_eps = case.get("vorticity", 0.0)
    p.k_boundaryDensity = case.get("boundary", 0.0)
    return p


def _lattice(dims, origin, gen):
    """A jittered lattice, (n, 3) float32."""
    axes = [torch.arange(d, device="cuda", dtype=torch.float64) * SPACING + SPACING / 2 + o for d, o in zip(dims, origin)]
    p = torch.stack(torch.meshgrid(*axes, indexing="ij"), -1).reshape(-1, 3)
    p = p + (torch.rand(p.shape, generator=gen, device="cuda", dtype=torch.float64) * 2 - 1) * JITTER
    return p.float()


def _flow(pos, gen):
    """A smooth flow with a little noise: falling, sheared, swirling (metres per second)."""
    k = 2 * math.pi / 3.2
    x, y, z = pos[:, 0], pos[:, 1], pos[:, 2]
    v = torch.stack([0.4 * torch.sin(k * y) + 0.1, 0.3 * torch.sin(k * x) - 0.3, 0.3 * torch.cos(k * (x + y))], 1)
    return v + 0.03 * torch.randn(v.shape, generator=gen, device="cuda")


def _cells(pos, ulim, llim, h):
    """Cell id of every position ((p - llim) / h in float32, truncated, clamped; x slowest) and the cells per axis."""
    f = np.float32
    dims = [max(1, int(math.ceil(float((f(u) - f(l)) / f(h))))) for u, l in zip(ulim, llim)]
    q = []
    for a in range(3):
        low = torch.tensor(float(f(llim[a])), dtype=torch.float32, device=pos.device)
        hh = torch.tensor(float(f(h)), dtype=torch.float32, device=pos.device)
        q.append(((pos[:, a].float() - low) / hh).long().clamp(0, dims[a] - 1))
    return q, dims


def _cell_order(pos, ulim, llim):
    q, d = _cells(pos, ulim, llim, H)
    return torch.sort((q[0] * d[1] + q[1]) * d[2] + q[2], stable=True).indices


def _four(t):
    return torch.cat([t, torch.zeros(t.shape[0], 1, device=t.device)], 1).contiguous()


def _scene(case, gen):
    """(pos (n, 3), vel (n, 3), ulim) of a step or gradient case, in cell order."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    if case.get("scene") == "double_dam_moving":
        box = (4 * nx * SPACING, ny * SPACING, nz * SPACING)
        pos = torch.cat([_lattice((nx, ny, nz), (0, 0, 0), gen), _lattice((nx, ny, nz), (box[0] - nx * SPACING, 0, 0), gen)])
    else:
        box = (2 * nx * SPACING, 2 * ny * SPACING, nz * SPACING)
        pos = _lattice((nx, ny, nz), (0, 0, 0), gen)
    vel = _flow(pos, gen)
    if case.get("scene") == "clustered":  # three times the lattice's particles collapsed onto six points
        pts = [(box[0] - 1e-3, 1e-3, 1e-3), (box[0] - 1e-3, 1e-3, box[2] - 1e-3), (1e-3, 1e-3, box[2] - 1e-3),
               (box[0] / 2, 1e-3, box[2] / 2), (box[0] - 1e-3, box[1] / 2, box[2] / 2), (box[0] / 8, box[1] / 6, box[2] / 4)]
        k = pos.shape[0] // 2
        speed = 0.1 * torch.randn(6, 3, generator=gen, device="cuda")
        pos = torch.cat([pos] + [torch.tensor(p, dtype=torch.float32, device="cuda").expand(k, 3) for p in pts])
        vel = torch.cat([vel] + [speed[c].expand(k, 3) for c in range(6)])
    order = _cell_order(pos, box, (0, 0, 0))
    return pos[order], vel[order], tuple(float(b) for b in box)


def _wall(case, box, seed):
    """(ulim, llim) of each step of a case whose x-max wall moves: x_w = X (1 - (1 - cos(2 pi t / 4 s)) / 8)."""
    t0 = 0.04 + 0.08 * np.random.default_rng(seed).random()
    ts = [t0 + k * 0.0083 for k in range(case["steps"])]
    return [((box[0] * (1 - (1 - math.cos(2 * math.pi * t / 4)) / 8), box[1], box[2]), (0.0, 0.0, 0.0)) for t in ts]


def _ensemble_scenes(case, gen):
    """(pos, vel, boxes, counts): the scenes' particles one scene after the other, each in its cell order; the
    lattices' sides are uniform in [lo, hi], by the case's own number `sides`."""
    sides = np.random.default_rng(case["sides"]).integers(case["lo"], case["hi"] + 1, size=(case["scenes"], 3)).tolist()
    pos, vel, boxes, counts = [], [], [], []
    for d in sides:
        box = tuple(2 * s * SPACING for s in d)
        p = _lattice(d, (0, 0, 0), gen)
        v = _flow(p, gen)
        order = _cell_order(p, box, (0, 0, 0))
        pos.append(p[order])
        vel.append(v[order])
        boxes.append(box)
        counts.append(p.shape[0])
    return torch.cat(pos), torch.cat(vel), boxes, counts


def _buffers(pos, vel):
    n = pos.shape[0]
    s = {"pos0": _four(pos), "vel0": _four(vel), "iid0": torch.arange(n, dtype=torch.int32, device="cuda")}
    for k in ("a_pos", "b_pos", "a_vel", "b_vel"):
        s[k] = torch.zeros(n, 4, device="cuda")
    s["iid"] = torch.zeros(n, dtype=torch.int32, device="cuda")
    return s


def _camera(case):
    """Camera position and focus: the lattice's centre from in front and above (z up)."""
    ex, ey, ez = case["nx"] * SPACING, case["nz"] * SPACING, case["ny"] * SPACING
    focus = (ex / 2, -ey / 2, ez / 2)
    side = max(ex, ey, ez)
    return (focus[0], focus[1] - 1.6875 * side, focus[2] + 0.6875 * side), focus


def prepare(case, seed):
    pbf = _pbf()
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    kind = case["kind"]
    if kind == "ssf":
        p = _lattice((case["nx"], case["ny"], case["nz"]), (0, 0, 0), gen)
        prm = pbf.ssf_default_params(case["width"], case["height"])
        pbf.ssf.look_at(prm, *_camera(case))
        prm.blur_option, prm.smooth_niter, prm.shading_option = case["blur"], case["smooth"], case["shading"]
        return {"case": dict(case), "renderer": pbf.SSFRenderer(prm), "pos": pbf.ssf.z_up(_four(p)),
                "color": torch.zeros(case["height"], case["width"], 4, device="cuda")}
    params = _params(case)
    if kind == "ensemble":
        pos, vel, boxes, counts = _ensemble_scenes(case, gen)
        s = _buffers(pos, vel)
        s["sim"] = pbf.Ensemble(params, boxes, [(0.0, 0.0, 0.0)] * len(boxes), counts)
    else:
        pos, vel, box = _scene(case, gen)
        s = _buffers(pos, vel)
        s["sim"] = pbf.Simulator(params, box, (0.0, 0.0, 0.0), pos.shape[0])
        s["walls"] = _wall(case, box, seed) if case.get("scene") == "double_dam_moving" else None
        if kind == "gradient":
            s["rollout"] = pbf.adjoint.Rollout(s["sim"], every=1, keep=1)
            s["box"], s["dims"], s["target"] = box, (case["gx"], case["gy"], case["gz"]), _target(case, gen)
    s["case"] = dict(case)
    return s


def _target(case, gen):
    """The density a gradient case fits: fluid in the lower x half, smooth, a little noise."""
    x = torch.linspace(0, 1, case["gx"], device="cuda")[:, None, None]
    t = 8000 * torch.sigmoid((0.45 - x) * 12) * torch.ones(case["gx"], case["gy"], case["gz"], device="cuda")
    return t * (1 + 0.05 * torch.randn(t.shape, generator=gen, device="cuda"))


# ---- the pass ------------------------------------------------------------------------------


def run(state):
    case = state["case"]
    if case["kind"] == "ssf":
        return state["renderer"].render(state["pos"], color=state["color"])
    if case["kind"] == "gradient":
        return _run_gradient(state)
    pos, npos, vel, nvel, iid = (state[k] for k in ("a_pos", "b_pos", "a_vel", "b_vel", "iid"))
    pos.copy_(state["pos0"])
    vel.copy_(state["vel0"])
    iid.copy_(state["iid0"])
    sim = state["sim"]
    if case["kind"] == "ensemble":
        sim.step(pos, npos, vel, nvel, iid)
    else:
        for k in range(case["steps"]):
            if k:
                pos, npos, vel, nvel = npos, pos, nvel, vel
            if state["walls"]:
                sim.setLim(*state["walls"][k])
            sim.step(pos, npos, vel, nvel, iid)
    return {"pos": pos, "npos": npos, "vel": vel, "nvel": nvel, "iid": iid}


def _run_gradient(state):
    """Loss |density(x) - target|^2 + 1/2 |v|^2 of the stepped state, and its gradient in the state before the step."""
    grids = _pbf().adjoint
    lo, hi, dims = (0.0, 0.0, 0.0), state["box"], state["dims"]
    pos, vel, iid = state["rollout"].run(state["pos0"], state["vel0"], state["iid0"], 1)
    density = grids.density_grid(pos, lo, hi, dims, H)
    g_pos = grids.density_grid_backward(pos, lo, hi, dims, H, 2.0 * (density - state["target"]))
    g_pos0, g_vel0, g_lim = state["rollout"].backward(g_pos, vel)
    return {"pos": pos, "vel": vel, "iid": iid, "density": density, "g_pos": g_pos0, "g_vel": g_vel0, "g_lim": g_lim}


def work(case):
    """A step reads pos, vel and iid (36 bytes a particle) and writes pos, vel, npos, nvel and iid (68); a pair of
    neighbours costs about 15 flops in each of the 4 niter + 1 gathers (about 33 neighbours at rest density)."""
    n = case.get("nx", 0) * case.get("ny", 0) * case.get("nz", 0)
    if case["kind"] == "ssf":
        pixels = case["width"] * case["height"]
        return {"bytes": 16.0 * n + 16.0 * pixels, "flops": 30.0 * n + 6.0 * 21 * 21 * case["smooth"] * pixels / 2}
    if case["kind"] == "ensemble":
        side = (case["lo"] + case["hi"]) / 2
        n = case["scenes"] * side ** 3
    elif case.get("scene") == "clustered":
        n = n + 6 * (n // 2)
    elif case.get("scene") == "double_dam_moving":
        n = 2 * n
    if case["kind"] == "gradient":
        cells = case["gx"] * case["gy"] * case["gz"]
        return {"bytes": 136.0 * n + 12.0 * cells, "flops": 33.0 * n * (60 * case["niter"] + 15) * 3}
    steps = case.get("steps", 1)
    lattice = n / 4 if case.get("scene") == "clustered" else n
    return {"bytes": 104.0 * n * steps, "flops": 33.0 * lattice * steps * (60 * case["niter"] + 15)}


# ---- the same in 64 bits ---------------------------------------------------------------------


class _Fluid:
    """The step's formulas in float64: one Jacobi solver iteration is lambda_() then delta_p()."""

    def __init__(self, p, ulim, llim, pos, vel):
        f = np.float32
        self.h, self.dt, self.rho0 = float(f(p.h)), float(f(p.dt)), float(f(p.pho0))
        self.inv_dt = float(f(1) / f(p.dt))
        self.poly6, self.spiky = 315.0 / (64 * math.pi * self.h ** 9), -45.0 / (math.pi * self.h ** 6)
        w = self.poly6 * (self.h ** 2 - float(f(p.delta_q)) ** 2) ** 3
        self.corr, self.n_corr = -float(f(p.k_corr)) / w ** float(f(p.n_corr)), float(f(p.n_corr))
        self.eps, self.keps, self.max_dp = float(f(p.lambda_eps)), float(f(p.kernel_eps)), float(f(p.max_dp))
        self.kb, self.cx, self.vort = float(f(p.k_boundaryDensity)), float(f(p.c_XSPH)), float(f(p.vorticity_eps))
        self.ulim = torch.tensor([float(f(u)) for u in ulim], dtype=torch.float64, device="cuda", requires_grad=True)
        self.llim = torch.tensor([float(f(u)) for u in llim], dtype=torch.float64, device="cuda", requires_grad=True)
        self.box = ([float(f(u)) for u in ulim], [float(f(u)) for u in llim])
        self.lim_eps = 1e-3
        g = torch.tensor([-float(f(p.g)) * float(f(p.up[a])) for a in range(3)], dtype=torch.float64, device="cuda")
        # cells come from the predicted positions in float32 (two fused multiply-adds)
        with torch.no_grad():
            v32 = (vel.double() + self.dt * g).float()
            x32 = (pos.double() + self.dt * v32.double()).float()
            q, self.dims = _cells(x32, *self.box, self.h)
            key = (q[0] * self.dims[1] + q[1]) * self.dims[2] + q[2]
            key, self.perm = torch.sort(key, stable=True)
            count = torch.bincount(key, minlength=self.dims[0] * self.dims[1] * self.dims[2])
            self.start = torch.cat([torch.zeros(1, dtype=torch.long, device="cuda"), count.cumsum(0)])
        self.x0 = pos.double()[self.perm]
        self.X = self.x0 + self.dt * (vel.double()[self.perm] + self.dt * g)

    @torch.no_grad()
    def pairs(self, X):
        """(i, j) of every j (i among them) in the cells around i's current cell with |x_i - x_j| < h."""
        (qx, qy, qz), (dx, dy, dz) = _cells(X, *self.box, self.h)
        zlo, zhi = (qz - 1).clamp(min=0), (qz + 1).clamp(max=dz - 1)
        out_i, out_j = [], []
        for a in (-1, 0, 1):
            for b in (-1, 0, 1):
                x, y = qx + a, qy + b
                ok = (x >= 0) & (x < dx) & (y >= 0) & (y < dy)
                base = torch.where(ok, (x * dy + y) * dz, torch.zeros_like(x))
                s = self.start[base + zlo]
                n = torch.where(ok, self.start[base + zhi + 1] - s, torch.zeros_like(s))
                i = torch.repeat_interleave(torch.arange(X.shape[0], device="cuda"), n)
                j = torch.arange(i.shape[0], device="cuda") - (n.cumsum(0) - n)[i] + s[i]
                keep = (X[i] - X[j]).square().sum(1) < self.h ** 2
                out_i.append(i[keep])
                out_j.append(j[keep])
        return torch.cat(out_i), torch.cat(out_j)

    def sum(self, i, v):
        return torch.zeros((self.x0.shape[0],) + v.shape[1:], dtype=torch.float64, device="cuda").index_add(0, i, v)

    def kernels(self, X, i, j):
        """(r, W, spiky gradient, gradient is not zero) of pairs."""
        r = X[i] - X[j]
        q = r.square().sum(1)
        far = q >= self.keps ** 2
        s = torch.where(far, q, torch.ones_like(q)).sqrt()
        F = torch.where(far, self.spiky * (self.h - s) ** 2 / s, torch.zeros_like(s))[:, None] * r
        return r, self.poly6 * (self.h ** 2 - q) ** 3, F

    def boundary(self, X):
        total = 0
        for d in (self.ulim.detach() - X, X - self.llim.detach()):
            k = 2 * 3.14159265359 / 3
            w = torch.where(d <= 0, torch.full_like(d, k), k * (self.h - d) ** 2 * (self.h + d))
            total = total + torch.where(d > self.h, torch.zeros_like(d), w).sum(1)
        return total

    def iterate(self, niter):
        lo, hi = self.llim + self.lim_eps, self.ulim - self.lim_eps
        for _ in range(niter):
            X = self.X
            i, j = self.pairs(X)
            _, W, F = self.kernels(X, i, j)
            self.rho = self.sum(i, W)
            if self.kb:
                self.rho = self.rho + self.kb * self.boundary(X)
            G = F / self.rho0
            S = self.sum(i, G.square().sum(1)) + self.sum(i, G).square().sum(1)
            lam = -(self.rho / self.rho0 - 1) / (S + self.eps)
            other = (i != j)
            f = (lam[i] + lam[j] + self.corr * W ** self.n_corr) * other
            d = (self.sum(i, f[:, None] * F) / self.rho0).clamp(-self.max_dp, self.max_dp)
            u = X + d
            self.X = torch.where(u > hi, hi.expand_as(u), torch.where(u < lo, lo.expand_as(u), u))

    def finish(self):
        self.vel = (self.X - self.x0) * self.inv_dt
        i, j = self.pairs(self.X)
        _, W, F = self.kernels(self.X, i, j)
        w = (2 * W / (self.rho[i] + self.rho[j]))[:, None]
        self.nvel = self.vel + self.cx * self.sum(i, w * (self.vel[j] - self.vel[i]))
        if self.vort:
            u = self.nvel
            F = F * (i != j)[:, None]
            om = self.sum(i, torch.linalg.cross(u[j] - u[i], F))
            eta = self.sum(i, om.norm(dim=1)[j][:, None] * F)
            size = eta.norm(dim=1, keepdim=True)
            nrm = torch.where(size > 0, eta / size.clamp(min=1e-300), torch.zeros_like(eta))
            self.nvel = u + self.dt * self.vort * torch.linalg.cross(nrm, om)


def _zero_w(t):
    return torch.cat([t, torch.zeros(t.shape[0], 1, dtype=t.dtype, device=t.device)], 1)


def _stepped(case, pos, vel, box):
    with torch.no_grad():
        s = _Fluid(_params(case), box, (0, 0, 0), pos, vel)
        s.iterate(case["niter"])
        s.finish()
    return {"pos": _zero_w(s.x0), "npos": _zero_w(s.X), "vel": _zero_w(s.vel), "nvel": _zero_w(s.nvel)}


def exact(case, seed):
    """run()'s floating outputs in float64.  None with the dam-break benchmark's parameters, whose four iterations
    amplify the rounding of any arithmetic to the size of the step (a cluster's pairs would also be too many), and
    None for several chained steps, whose rows are in an order that the float32 positions decide."""
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    if case["kind"] == "ssf":
        return _exact_ssf(case, gen)
    if case["params"] == "dam_break" or case.get("steps", 1) > 1:
        return None
    if case["kind"] == "ensemble":
        pos, vel, boxes, counts = _ensemble_scenes(case, gen)
        got = [_stepped(case, p, v, b) for p, v, b in zip(pos.split(counts), vel.split(counts), boxes)]
        return dict({k: torch.cat([g[k] for g in got]) for k in got[0]}, iid=None)
    pos, vel, box = _scene(case, gen)
    if case["kind"] == "step":
        return dict(_stepped(case, pos, vel, box), iid=None)
    target = _target(case, gen).double()
    x, v = pos.double().requires_grad_(), vel.double().requires_grad_()
    s = _Fluid(_params(case), box, (0, 0, 0), x, v)
    s.iterate(case["niter"])
    s.finish()
    density = _exact_density(case, s.X, box)
    loss = (density - target).square().sum() + 0.5 * s.nvel.square().sum()
    g = torch.autograd.grad(loss, [x, v, s.ulim, s.llim], allow_unused=True)
    g = [torch.zeros(3, dtype=torch.float64, device="cuda") if t is None else t for t in g]
    return {"pos": _zero_w(s.X.detach()), "vel": _zero_w(s.nvel.detach()), "iid": None, "density": density.detach(),
            "g_pos": _zero_w(g[0]), "g_vel": _zero_w(g[1]), "g_lim": torch.cat(g[2:])[None]}


def _exact_density(case, X, box):
    """Poly6 density at the centres of the lattice's cells (differentiable)."""
    dims, h = (case["gx"], case["gy"], case["gz"]), float(np.float32(H))
    step = [float(np.float32(b)) / d for b, d in zip(box, dims)]
    reach = [int(math.ceil(h / s)) + 1 for s in step]
    near = [torch.floor(X[:, a].detach() / step[a]).long() for a in range(3)]
    out = torch.zeros(dims[0] * dims[1] * dims[2], dtype=torch.float64, device="cuda")
    for a in range(-reach[0], reach[0] + 1):
        for b in range(-reach[1], reach[1] + 1):
            for c in range(-reach[2], reach[2] + 1):
                k = [near[0] + a, near[1] + b, near[2] + c]
                d2 = sum((X[:, t] - (k[t].double() + 0.5) * step[t]) ** 2 for t in range(3))
                ok = d2 < h * h
                for t in range(3):
                    ok = ok & (k[t] >= 0) & (k[t] < dims[t])
                sel = ok.nonzero().squeeze(1)
                w = 315.0 / (64 * math.pi * h ** 9) * (h * h - d2[sel]) ** 3
                out = out.index_add(0, ((k[0] * dims[1] + k[1]) * dims[2] + k[2])[sel], w)
    return out.reshape(dims)


def _exact_ssf(case, gen):
    """The rendered colour image: sphere sprites, smoothing, normals, shading."""
    pbf = _pbf()
    W, Hh = case["width"], case["height"]
    p = _lattice((case["nx"], case["ny"], case["nz"]), (0, 0, 0), gen).double()
    P = torch.stack([p[:, 0], -p[:, 2], p[:, 1], torch.ones_like(p[:, 0])], 1)
    prm = pbf.ssf_default_params(W, Hh)
    pbf.ssf.look_at(prm, *_camera(case))
    mat = lambda m: torch.tensor(list(m), dtype=torch.float64, device="cuda").reshape(4, 4)  # noqa: E731  (row vector times it)
    view, proj = mat(prm.view), mat(prm.proj)
    eye = P @ view
    clip = eye @ proj
    w = clip[:, 3]
    ok = (w > 0) & (clip[:, :3].abs() <= w[:, None]).all(1)
    eye, clip, w = eye[ok], clip[ok], w[ok]
    r, pn, pt, pr = prm.radius, prm.p_n, prm.p_t, prm.p_r
    xw, yw = W / 2 * clip[:, 0] / w + W / 2, Hh / 2 * clip[:, 1] / w + Hh / 2
    size = (r * pn * Hh / (-eye[:, 2] * pt)).clamp(min=1)
    x0, x1 = torch.ceil(xw - size / 2 - 0.5).clamp(min=0).long(), (torch.ceil(xw + size / 2 - 0.5) - 1).clamp(max=W - 1).long()
    y0, y1 = torch.ceil(yw - size / 2 - 0.5).clamp(min=0).long(), (torch.ceil(yw + size / 2 - 0.5) - 1).clamp(max=Hh - 1).long()
    cols, rows = (x1 - x0 + 1).clamp(min=0), (y1 - y0 + 1).clamp(min=0)
    depth = torch.full((Hh * W,), 100.0, dtype=torch.float64, device="cuda")
    thick = torch.zeros(Hh * W, dtype=torch.float64, device="cuda")
    for part in torch.arange(xw.shape[0], device="cuda").split(1 << 16):
        n = (cols * rows)[part]
        i = torch.repeat_interleave(part, n)
        k = torch.arange(i.shape[0], device="cuda") - torch.repeat_interleave(n.cumsum(0) - n, n)
        px, py = x0[i] + k % cols[i], y0[i] + torch.div(k, cols[i], rounding_mode="floor")
        x, y = (px + 0.5 - xw[i]) * 2 / size[i], (yw[i] - py - 0.5) * 2 / size[i]
        q = x * x + y * y
        z = (1 - q).clamp(min=0).sqrt()
        sel = q <= 1
        at = (py * W + px)[sel]
        depth.scatter_reduce_(0, at, -(eye[i, 2] + z * r)[sel], "amin")
        thick.index_add_(0, at, (2 * r * z)[sel])
    depth, thick = depth.reshape(Hh, W), thick.reshape(Hh, W)
    R, br, bz = prm.kernel_r, 1 / prm.sigma_r, 1 / prm.sigma_z
    fluid = depth <= 99
    for _ in range(case["smooth"]):
        pad = torch.nn.functional.pad(depth, (R, R, R, R))
        total, weight = torch.zeros_like(depth), torch.zeros_like(depth)
        for dx in range(-R, R + 1):
            for dy in range(-R, R + 1):
                s = pad[R + dy:R + dy + Hh, R + dx:R + dx + W]
                g = math.exp(-(dx * dx + dy * dy) * br * br)
                if case["blur"] == 0:
                    g = g * torch.exp(-((s - depth) * bz) ** 2)
                total += s * g
                weight += g
        depth = torch.where(fluid, total / weight, depth)
    z = -depth
    fx, bx = torch.roll(z, -1, 1) - z, z - torch.roll(z, 1, 1)
    fy, by = torch.roll(z, -1, 0) - z, z - torch.roll(z, 1, 0)
    dzdx = torch.where(bx.abs() < fx.abs(), bx, fx) if prm.keep_edge == 1 else fx
    dzdy = torch.where(by.abs() < fy.abs(), by, fy) if prm.keep_edge == 1 else fy
    cx, cy = 2 / (W * pn / pr), 2 / (Hh * pn / pt)
    nrm = torch.stack([-cy * dzdx, -cx * dzdy, -cx * cy * z], -1)
    nrm = nrm / nrm.norm(dim=-1, keepdim=True)
    u = ((torch.arange(W, device="cuda", dtype=torch.float64) + 0.5) / W)[None, :].expand(Hh, W)
    v = ((torch.arange(Hh, device="cuda", dtype=torch.float64) + 0.5) / Hh)[:, None].expand(Hh, W)
    pos = torch.stack([(2 * u - 1) * pr * depth / pn, (2 * v - 1) * pt * depth / pn, -depth], -1)
    e = -pos / pos.norm(dim=-1, keepdim=True)
    ne = (nrm * e).sum(-1, keepdim=True)
    r0 = prm.r0
    inv = torch.linalg.inv(view)
    sky = torch.tensor(list(prm.sky), dtype=torch.float64, device="cuda")

    def trace(d):
        """A 10 x 10 checker floor at z = 0, else the sky."""
        wp = torch.cat([pos, torch.ones_like(pos[..., :1])], -1) @ inv
        wd = d @ inv[:3, :3]
        t = -wp[..., 2] / wd[..., 2]
        hit = wp[..., :2] + t[..., None] * wd[..., :2]
        on = (t > 0) & (hit.abs() < 5).all(-1)
        c = ((hit + 5) - torch.floor(hit + 5) > 0.5).sum(-1)
        floor = torch.where(c == 1, 0.6, 0.8).double()
        return torch.where(on[..., None], floor[..., None].expand_as(wd), sky.expand_as(wd))

    if case["shading"] == 3:
        out = nrm
    elif case["shading"] == 4:
        out = (r0 + (1 - r0) * (1 - ne) ** 2).expand_as(nrm)
    else:
        att = torch.exp(-0.5 * thick).clamp(min=0.2)[..., None]
        tint = torch.tensor([6 / 256, 105 / 256, 217 / 256], dtype=torch.float64, device="cuda")
        out = (1 - att) * tint + att * trace(-e - 0.2 * nrm)
        if case["shading"] == 0:
            fres = r0 + (1 - r0) * (1 - ne) ** 3
            out = (1 - fres) * out + fres * trace(-e + 2 * ne * nrm)
    drawn = (depth < prm.p_f)[..., None]
    return torch.where(drawn, torch.cat([out, torch.ones_like(out[..., :1])], -1), torch.zeros(4, dtype=torch.float64, device="cuda"))
