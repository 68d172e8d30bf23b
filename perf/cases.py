"""Timed workloads of the smoke step: what a program that uses this package has it do.

listed() holds the named workloads, draw() more of the same ranges; prepare() makes the inputs and
the handles a program keeps, run() is one pass through the public entry points, work() what a pass
cannot do without, exact() the same pass in 64 bits with plain torch (no code of this package).

Kinds
  step      Simulation.step and a device read of the new density (a renderer on the same GPU)
  simulate  Simulation.simulate: the step with the density copied to the host (the reference's call)
  batch     Batch.step over uneven grids, every member's density read on the device
  serve     a Server that takes a burst of requests and runs them to their last step
  project   smk_project_noalloc on a velocity field that the caller owns
  render    one frame of the headless volume renderer

Fields of a case: nx, ny, nz the grid; scheme 0 the reference's velocity SOR, 1 the pressure form;
sweeps the iterations (scheme 1: their cap); tol the divergence tolerance (0: fixed sweeps), checked
every `check` sweeps; warm 0 pressure from zero each step, 1 from the last step, 2 extrapolated and
with the over-relaxation schedule; storage 0 FP32, 1 BF16, 2 BF16 velocities; solids the share of
random solid cells; obstacle 1 a sphere obstacle; move 1 the source is dragged, so that its position
changes before every step; rest 1 the fluid starts at rest with no smoke; tune 1 the program calls
autotune() once.
"""
import ctypes
import math

import numpy as np
import torch

import smoke_simulation_gb300 as smk
from smoke_simulation_gb300 import scenes, serving


def listed():
    step = dict(kind="step", scheme=0, sweeps=30, tol=0.0, check=6, warm=0, storage=0, solids=0.0, obstacle=0,
                move=0, rest=0, tune=0, dt=0.05, pinned=0)
    case = lambda name, **kw: dict(step, name=name, **kw)  # noqa: E731
    return [
        # the smallest grid of the batched range, stepped alone with the default parameters: a
        # preview or a game effect, where launches are all there is
        case("tiny_step_32", nx=32, ny=32, nz=32, obstacle=1),
        # the reference application: its 80^3 grid, sphere obstacle and smoke source, fluid at rest
        # at the start, simulate() into ordinary host memory as its `new float[]` is
        case("app_simulate_80", kind="simulate", nx=80, ny=80, nz=80, obstacle=1, rest=1),
        # default parameters on a grid of odd sides (no side a multiple of a tile or a vector)
        case("odd_step_97x61x113", nx=97, ny=61, nz=113, solids=0.02),
        # the drop-in call at a production size, the host buffer page-locked
        case("dropin_simulate_256", kind="simulate", nx=256, ny=256, nz=256, solids=0.05, dt=0.02, pinned=1),
        # an interactive scene: pressure form to a tolerance, warm-started, the source dragged
        case("drag_step_64", nx=64, ny=64, nz=64, scheme=1, sweeps=200, tol=1e-4, warm=1, obstacle=1, move=1),
        # fixed sweeps from zero pressure on a ragged grid, no autotuning: the form whose results
        # do not depend on the history
        case("fixed_step_150x117x203", nx=150, ny=117, nz=203, scheme=1, sweeps=40, solids=0.02),
        # the single large grid, as the benchmark solves it: from rest, warm-started
        case("large_step_256", nx=256, ny=256, nz=256, scheme=1, sweeps=200, tol=0.995e-4, warm=2, solids=0.05,
             rest=1, dt=0.02, tune=1),
        # the large mixed-precision grid: BF16 velocities, FP64-checked refinement rounds allowed
        case("mixed_step_512", nx=512, ny=512, nz=512, scheme=1, sweeps=200, tol=1e-4, warm=2, storage=2, solids=0.02,
             rest=1, dt=0.02, tune=1),
        # 64 uneven grids in one grouped step
        dict(kind="batch", name="batch_64", count=64, lo=32, hi=128, sweeps=200, tol=1e-4, check=6, warm=2, storage=0,
             dt=0.05),
        # a burst of requests of mixed sizes on the server's default form
        dict(kind="serve", name="serve_8", count=8, lo=48, hi=192, steps_lo=10, steps_hi=40, storage=2),
        # projection of a caller's own field, fixed memory
        dict(kind="project", name="project_127", nx=127, ny=127, nz=127, sweeps=30, tol=0.0, check=6, solids=0.02),
        # a frame of the reference application's view
        dict(kind="render", name="frame_80", nx=80, ny=80, nz=80, width=1280, height=720, planes=100),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "step", "simulate", "batch", "serve", "project", "render"])
    if kind == "batch":
        lo = _log_int(rng, 24, 64)
        return dict(kind=kind, count=_log_int(rng, 4, 64), lo=lo, hi=_log_int(rng, lo, 128), sweeps=rng.randint(60, 200),
                    tol=rng.choice([1e-4, 1e-3]), check=6, warm=rng.choice([1, 2]), storage=rng.choice([0, 2]), dt=0.05)
    if kind == "serve":
        lo = _log_int(rng, 32, 64)
        steps = rng.randint(5, 20)
        return dict(kind=kind, count=rng.randint(2, 8), lo=lo, hi=_log_int(rng, lo, 192), steps_lo=steps,
                    steps_hi=2 * steps, storage=rng.choice([0, 2]))
    if kind == "project":
        n = [_log_int(rng, 16, 127) for _ in range(3)]
        return dict(kind=kind, nx=n[0], ny=n[1], nz=n[2], sweeps=rng.randint(10, 60), tol=rng.choice([0.0, 1e-3]),
                    check=6, solids=rng.choice([0.0, 0.02]))
    if kind == "render":
        n = [_log_int(rng, 32, 160) for _ in range(3)]
        return dict(kind=kind, nx=n[0], ny=n[1], nz=n[2], width=_log_int(rng, 320, 1920), height=_log_int(rng, 240, 1080),
                    planes=rng.randint(50, 200))
    scheme = 0 if kind == "simulate" else rng.choice([0, 1, 1])
    top = 256 if scheme == 0 else 384
    n = [_log_int(rng, 24, top) for _ in range(3)]
    tol = rng.choice([0.0, 1e-4, 1e-3]) if scheme else 0.0
    return dict(kind=kind, nx=n[0], ny=n[1], nz=n[2], scheme=scheme,
                sweeps=200 if tol else rng.randint(20, 60), tol=tol, check=rng.choice([6, 10]),
                warm=rng.choice([0, 1, 2]) if tol else 0, storage=rng.choice([0, 0, 2, 1]) if scheme else 0,
                solids=rng.choice([0.0, 0.02, 0.05]), obstacle=rng.choice([0, 0, 1]), move=rng.choice([0, 0, 0, 1]),
                rest=rng.choice([0, 0, 1]), tune=rng.choice([0, 0, 1]), dt=rng.choice([0.02, 0.05]),
                pinned=rng.choice([0, 1]))


# ---- inputs ------------------------------------------------------------------------------------

def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _generator(seed):
    return torch.Generator(device=_device()).manual_seed(int(seed) & 0x7FFFFFFF)


def _uniform(gen, shape, lo, hi):
    return torch.rand(shape, generator=gen, device=_device(), dtype=torch.float32) * (hi - lo) + lo


def _axes(nz, ny, nx):
    return (torch.arange(nz, device=_device(), dtype=torch.float32)[:, None, None],
            torch.arange(ny, device=_device(), dtype=torch.float32)[None, :, None],
            torch.arange(nx, device=_device(), dtype=torch.float32)[None, None, :])


def _velocity(gen, shape):
    """One face component: a few large eddies (up to about 3 cells per second) and fine noise."""
    z, y, x = _axes(*shape)
    out = _uniform(gen, shape, -0.1, 0.1)
    for _ in range(2):
        k = (_uniform(gen, (3,), 0.5, 3.0) * (2 * math.pi)).tolist()
        ph = _uniform(gen, (3,), 0.0, 2 * math.pi).tolist()
        a = float(_uniform(gen, (1,), 0.5, 1.5))
        out += a * (torch.cos(x * (k[0] / shape[2]) + ph[0]) * torch.cos(y * (k[1] / shape[1]) + ph[1])
                    * torch.cos(z * (k[2] / shape[0]) + ph[2]))
    return out


def _smoke(gen, shape):
    """A few clouds of density up to 1, nothing elsewhere."""
    z, y, x = _axes(*shape)
    out = torch.zeros(shape, device=_device())
    for _ in range(3):
        c = _uniform(gen, (3,), 0.2, 0.8).tolist()
        r = 0.18 * min(shape)
        d2 = (x - c[0] * shape[2]) ** 2 + (y - c[1] * shape[1]) ** 2 + (z - c[2] * shape[0]) ** 2
        out = torch.maximum(out, torch.exp(-d2 / (r * r)))
    out[out < 0.05] = 0.0
    return out


def _host(t):
    return t.cpu().numpy()


def _scene(case, seed):
    """The scene of a step, simulate or render case (sphere geometry has whole-numbered centres)."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    gen = _generator(seed)
    m = min(nx, ny, nz)
    sc = scenes.Scene("case", nx, ny, nz, dt=case.get("dt", 0.05), steps=1, scheme=case.get("scheme", 0),
                      iterations=case.get("sweeps", 30), tol=case.get("tol", 0.0), check_every=case.get("check", 6))
    warm = case.get("warm", 0)
    sc.warm_start = 1 if warm else 0
    if warm == 2:
        sc.omega_warm, sc.omega_warm_after, sc.warm_extrapolate = 1.75, 2, 0.5
    if case.get("storage", 0) and sc.tol:
        sc.refine, sc.refine_sweeps = 2, 10
    if case.get("solids", 0.0):
        mask = torch.ones((nz, ny, nx), dtype=torch.uint8, device=_device())
        mask[_uniform(gen, (nz, ny, nx), 0.0, 1.0) < case["solids"]] = 0
        mask[:, 0, :] = 0
        sc.mask = _host(mask)
    place = lambda lo, hi: [float(round(float(v) * (n - 1))) for v, n in zip(_uniform(gen, (3,), lo, hi), (nx, ny, nz))]  # noqa: E731
    sources = 1 if case.get("move", 0) else 4
    sc.spheres = [(*place(0.2, 0.8), float(max(2, min(6, m // 16)))) for _ in range(sources)]
    if case.get("obstacle", 0):
        sc.obstacles = [(*place(0.35, 0.65), 0.0, 0.0, 0.0, float(max(2, m // 6)))]
    if not case.get("rest", 0):
        sc.rho0 = _host(_smoke(gen, (nz, ny, nx)))
        sc.u0, sc.v0, sc.w0 = (_host(_velocity(gen, (nz + 1, ny + 1, nx + 1))) for _ in range(3))
    return sc


def _cubes(case, seed):
    """The uneven grids of a batch or a burst: cube sides over the range, a sphere solid and a box
    emitter in each."""
    rng = scenes.SplitMix64(int(seed) & 0x7FFFFFFF, lane=9)
    lo, hi, count = case["lo"], case["hi"], case["count"]
    # log-uniform sides, one in each of `count` equal parts of the range: the grids are the case's,
    # what is in them the seed's
    parts = (np.arange(count) + scenes.SplitMix64(count, lane=8).uniform(count)) / count
    sides = np.round(np.exp(math.log(lo) + parts * (math.log(hi) - math.log(lo)))).astype(int)
    steps = scenes.SplitMix64(count, lane=7).integers(count, case.get("steps_lo", 1), case.get("steps_hi", 1) + 1)
    out = []
    for i, n in enumerate(int(s) for s in sides):
        sc = scenes.Scene("cube%d" % i, n, n, n, dt=0.05, steps=1, scheme=1, iterations=case.get("sweeps", 200),
                          tol=case.get("tol", 1e-4), check_every=6, warm_start=1)
        if case.get("warm", 1) == 2:
            sc.omega_warm, sc.omega_warm_after, sc.warm_extrapolate = 1.75, 2, 0.5
        r = b = max(2, n // 8)
        c = [float(v) for v in rng.integers(3, r + 2, n - r - 2)]
        sc.mask = scenes.sphere_mask(n, n, n, [(*c, float(r))], scenes.reference_initial_mask(n, n, n))
        ex, ez = (int(v) for v in rng.integers(2, b + 1, n - b - 1))
        sc.boxes = [(ex - b // 2, 1, ez - b // 2, ex - b // 2 + b, 1 + max(2, b // 2), ez - b // 2 + b, 1.0, 0.0, 0.0)]
        sc.steps = int(steps[i])
        out.append(sc)
    return out


def _drag(source, passes):
    """Where the dragged source is at its `passes`-th step."""
    x, y, z, _ = source
    return x + float(passes % 5) - 2.0, y, z + float(passes % 3) - 1.0


def _own_field(case, seed):
    gen = _generator(seed)
    shape = (case["nz"] + 1, case["ny"] + 1, case["nx"] + 1)
    vel = [_velocity(gen, shape) for _ in range(3)]
    mask = torch.ones((case["nz"], case["ny"], case["nx"]), dtype=torch.uint8, device=_device())
    if case["solids"]:
        mask[_uniform(gen, mask.shape, 0.0, 1.0) < case["solids"]] = 0
    mask[:, 0, :] = 0
    return vel, mask


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind, "passes": 0}
    if kind == "project":
        s["field"], s["mask"] = _own_field(case, seed)
        s["vel"] = [torch.empty_like(t) for t in s["field"]]
        s["params"] = smk.default_params(projection=smk.PROJECT_PRESSURE, max_sweeps=case["sweeps"], tol=case["tol"],
                                         check_every=case["check"])
        s["n"] = (case["nx"], case["ny"], case["nz"])
        return s
    if kind == "batch":
        s["scenes"] = _cubes(case, seed)
        s["sims"] = [smk.from_scene(sc, storage=case["storage"]) for sc in s["scenes"]]
        s["batch"] = smk.Batch(s["sims"])
        s["batch"].set_blocked(137)
        s["out"] = torch.empty(sum(sc.cells for sc in s["scenes"]), dtype=torch.float32, device="cuda")
        at, s["at"] = s["out"].data_ptr(), []
        for sc in s["scenes"]:
            s["at"].append(at)
            at += 4 * sc.cells
        s["dt"] = case["dt"]
        return s
    if kind == "serve":
        s["scenes"] = _cubes(case, seed)
        s["server"] = serving.Server()
        s["storage"] = case["storage"]
        s["out"] = [torch.empty(sc.cell_shape, dtype=torch.float32, device="cuda") for sc in s["scenes"]]
        return s
    sc = _scene(case, seed)
    if kind == "render":
        s["sim"] = smk.from_scene(sc)
        s["view"] = smk.default_render_params(width=case["width"], height=case["height"], planes=case["planes"])
        s["eye"] = torch.empty((case["height"], case["width"], 4), dtype=torch.float32, device="cuda")
        s["rgb"] = torch.empty((case["height"], case["width"], 3), dtype=torch.float32, device="cuda")
        return s
    s["sim"] = sim = smk.from_scene(sc, storage=case["storage"])
    if case["tune"]:
        sim.autotune()
    s["dt"], s["move"] = sc.dt, case["move"]
    s["source"], s["source_id"] = sc.spheres[0], len(sc.boxes)  # ids count the objects in the order added
    if kind == "simulate":
        s["out"] = torch.empty(sc.cell_shape, dtype=torch.float32, pin_memory=bool(case["pinned"])).numpy()
        s["out"][...] = 0.0  # a program's buffer has been written to
    else:
        s["out"] = torch.empty(sc.cell_shape, dtype=torch.float32, device="cuda")
    return s


def run(s):
    kind = s["kind"]
    if kind == "batch":
        s["batch"].step(s["dt"])
        for sim, ptr in zip(s["sims"], s["at"]):
            sim.read_density_device(ptr)
        return s["out"]
    if kind == "serve":
        for sc, out in zip(s["scenes"], s["out"]):
            s["server"].submit(sc, out_device=out, storage=s["storage"])
        s["server"].run_until_idle()
        return s["out"]
    if kind == "project":
        for t, f in zip(s["vel"], s["field"]):
            t.copy_(f)
        u, v, w = s["vel"]
        smk._check(smk.lib().smk_project_noalloc(u.data_ptr(), v.data_ptr(), w.data_ptr(), s["mask"].data_ptr(), *s["n"],
                                                 ctypes.byref(s["params"]), None, None))
        return s["vel"]
    if kind == "render":
        s["sim"].render_into(s["eye"].data_ptr(), s["rgb"].data_ptr(), s["view"])
        return s["eye"], s["rgb"]
    sim = s["sim"]
    if s["move"]:
        sim.update_object_pos(s["source_id"], *_drag(s["source"], s["passes"]))
        s["passes"] += 1
    if kind == "simulate":
        return sim.simulate(s["out"], s["dt"])
    sim.step(s["dt"])
    sim.read_density_device(s["out"].data_ptr())
    return s["out"]


def work(case):
    """Fields read once and written once; the arithmetic of the passes over the cells."""
    kind = case["kind"]

    def step(cells, scheme, sweeps, storage, warm):
        vel = 2 if storage else 4
        rho = 2 if storage == 1 else 4
        return {"bytes": cells * (2 * (3 * vel + rho) + 1 + 4 + (8 if warm else 0)),
                "flops": cells * (150 + sweeps * (9 if scheme else 20))}
    if kind in ("batch", "serve"):
        lo, hi, count = case["lo"], case["hi"], case["count"]
        parts = [(i + 0.5) / count for i in range(count)]
        cells = sum(math.exp(math.log(lo) + p * (math.log(hi) - math.log(lo))) ** 3 for p in parts)
        one = step(cells, 1, 20, case["storage"], 1)
        n = 0.5 * (case.get("steps_lo", 1) + case.get("steps_hi", 1))
        return {k: v * n for k, v in one.items()}
    cells = case["nx"] * case["ny"] * case["nz"]
    if kind == "project":
        return {"bytes": cells * 25, "flops": cells * (12 + 9 * case["sweeps"])}
    if kind == "render":
        pixels = case["width"] * case["height"]
        return {"bytes": cells * 4 + pixels * 28, "flops": 60 * case["planes"] * (pixels // 4 + 512 * 512)}
    return step(cells, case["scheme"], 20 if case["tol"] else case["sweeps"], case["storage"], case["warm"])


# ---- the same pass in 64 bits ------------------------------------------------------------------

class _Exact:
    """One step of the discretisation in float64 on whole arrays shaped (z, y, x): cells
    (nz, ny, nx), faces one longer on every side."""

    def __init__(self, mask, rho, vel, rho_out):
        self.nz, self.ny, self.nx = mask.shape
        self.s = mask != 0
        self.rho, self.rho_out = rho, rho_out
        self.u, self.v, self.w = vel

    def neighbours(self, a, fill=0):
        p = torch.nn.functional.pad(a, (1, 1, 1, 1, 1, 1), value=fill)
        return (p[1:-1, 1:-1, :-2], p[1:-1, 1:-1, 2:], p[1:-1, :-2, 1:-1], p[1:-1, 2:, 1:-1], p[:-2, 1:-1, 1:-1],
                p[2:, 1:-1, 1:-1])

    def interior(self):
        m = torch.zeros((self.nz, self.ny, self.nx), dtype=torch.bool, device=self.rho.device)
        m[1:self.nz - 1, 1:self.ny - 1, 1:self.nx - 1] = True
        return m

    def corner_distance(self, sphere):
        z, y, x = (t.double() for t in _axes(self.nz, self.ny, self.nx))
        return (x - sphere[0]) ** 2 + (y - sphere[1]) ** 2 + (z - sphere[2]) ** 2

    def objects(self, sc, spheres):
        for b in sc.boxes:
            x0, y0, z0, x1, y1, z1 = (int(v) for v in b[:6])
            box = (slice(max(z0, 0), z1), slice(max(y0, 0), y1), slice(max(x0, 0), x1))
            self.rho[box] = self.rho_out[box] = float(b[6])
        for sp in spheres:
            inside = (self.corner_distance(sp) < sp[3] * sp[3]) & self.interior()
            self.rho[inside] = self.rho_out[inside] = 1.0
        if sc.obstacles:
            o = sc.obstacles[-1]
            solid = self.corner_distance(o) < o[6] * o[6]
            self.s = torch.where(self.interior(), ~solid, self.s)

    def forcing(self, dt, gravity, buoyancy, clamp):
        nz, ny, nx = self.nz, self.ny, self.nx
        both = self.s[:, 1:] & self.s[:, :-1]
        r = self.rho[:, 1:]
        self.v[:nz, 1:ny, :nx] += torch.where(both, r * gravity * dt + buoyancy * r * dt, torch.zeros_like(r))
        c = (slice(1, nz), slice(1, ny), slice(1, nx))
        e = (self.u[c] ** 2 + self.v[c] ** 2 + self.w[c] ** 2) * dt
        scale = torch.where(e > clamp * clamp, clamp * clamp / e.clamp_min(1e-300), torch.ones_like(e))
        for f in (self.u, self.v, self.w):
            f[c] *= scale

    def divergence(self):
        nz, ny, nx = self.nz, self.ny, self.nx
        return (self.u[:nz, :ny, 1:] - self.u[:nz, :ny, :nx] + self.v[:nz, 1:, :nx] - self.v[:nz, :ny, :nx]
                + self.w[1:, :ny, :nx] - self.w[:nz, :ny, :nx])

    def cells(self):
        """Number of fluid neighbours, the cells the projection updates, and the two colours."""
        acc = torch.zeros(self.s.shape, dtype=torch.float64, device=self.rho.device)
        for n in self.neighbours(self.s.double()):
            acc += n
        live = self.interior() & self.s & (acc > 0)
        z, y, x = _axes(self.nz, self.ny, self.nx)
        odd = torch.remainder(x + y + z, 2) != 0
        return acc.clamp_min(1.0), live, (live & ~odd, live & odd)

    def project_velocity(self, iterations, omega):
        nz, ny, nx = self.nz, self.ny, self.nx
        acc, _, colours = self.cells()
        n = [a.double() for a in self.neighbours(self.s.double())]
        for _ in range(iterations):
            for colour in colours:
                p = torch.where(colour, -self.divergence() / acc * omega, torch.zeros_like(acc))
                self.u[:nz, :ny, :nx] -= p * n[0]
                self.u[:nz, :ny, 1:] += p * n[1]
                self.v[:nz, :ny, :nx] -= p * n[2]
                self.v[:nz, 1:, :nx] += p * n[3]
                self.w[:nz, :ny, :nx] -= p * n[4]
                self.w[1:, :ny, :nx] += p * n[5]

    def project_pressure(self, sweeps, omega, tol, check):
        nz, ny, nx = self.nz, self.ny, self.nx
        acc, live, colours = self.cells()
        b = torch.where(live, -self.divergence(), torch.zeros_like(acc))
        p = torch.zeros((nz + 2, ny + 2, nx + 2), dtype=torch.float64, device=b.device)
        c = p[1:-1, 1:-1, 1:-1]
        around = (p[1:-1, 1:-1, :-2], p[1:-1, 1:-1, 2:], p[1:-1, :-2, 1:-1], p[1:-1, 2:, 1:-1], p[:-2, 1:-1, 1:-1],
                  p[2:, 1:-1, 1:-1])

        def residual():
            r = b - acc * c
            for n in around:
                r += n
            return r
        for k in range(sweeps):
            if tol > 0 and k % check == 0 and float((residual().abs() * live).max()) <= tol:
                break
            for colour in colours:
                c += torch.where(colour, residual() * (omega / acc), torch.zeros_like(acc))
        for f, axis in ((self.u, 2), (self.v, 1), (self.w, 0)):
            lo = tuple(slice(1, n if a == axis else n - 1) for a, n in enumerate((nz, ny, nx)))
            before = tuple(slice(s.start - 1, s.stop - 1) if a == axis else s for a, s in enumerate(lo))
            f[lo] -= torch.where(self.s[lo] & self.s[before], c[lo] - c[before], torch.zeros_like(c[lo]))

    def sample(self, f, pos, half):
        """Trilinear value at pos = (x, y, z), clamped to [1, n - 1]; half: cell-centred axes."""
        n = (self.nx, self.ny, self.nz)
        index, weight = [], []
        for a in range(3):
            p = pos[a].clamp(max=n[a] - 1).clamp_min(1.0) - (0.5 if half[a] else 0.0)
            i = p.floor()
            w1 = p - i
            i = i.long()
            index.append((i, i + 1 if half[a] else (i + 1).clamp_max(n[a] - 1)))
            weight.append((1 - w1, w1))
        out = torch.zeros_like(pos[0])
        for c in range(8):
            a, b, d = c & 1, (c >> 1) & 1, c >> 2
            out += weight[0][a] * weight[1][b] * weight[2][d] * f[index[2][d], index[1][b], index[0][a]]
        return out

    def advect(self, dt, at_once=1 << 24):
        """The new density (the velocity of the step only where it needs it), z plane by z plane."""
        nz, ny, nx = self.nz, self.ny, self.nx
        new = [torch.zeros_like(f) for f in (self.u, self.v, self.w)]
        planes = max(1, at_once // (nx * ny))
        u, v, w = self.u, self.v, self.w
        for z0 in range(1, nz, planes):
            z1 = min(nz, z0 + planes)
            c = (slice(z0, z1), slice(1, ny), slice(1, nx))

            def at(f, dz, dy, dx):
                return f[z0 + dz:z1 + dz, 1 + dy:ny + dy, 1 + dx:nx + dx]
            au = sum(at(u, dz, dy, dx) for dz in (-1, 0) for dy in (0, -1) for dx in (0, 1)) / 8
            av = sum(at(v, dz, dy, dx) for dz in (-1, 0) for dy in (0, 1) for dx in (0, -1)) / 8
            aw = sum(at(w, dz, dy, dx) for dz in (0, -1) for dy in (0, -1) for dx in (0, -1)) / 8
            z, y, x = (t.double() for t in _axes(nz, ny, nx))
            z, y, x = z[z0:z1], y[:, 1:], x[:, :, 1:]
            one = torch.ones_like(au)
            inside = [x * one <= nx - 2, y * one <= ny - 2, z * one <= nz - 2]
            s = self.s[c]
            for k, (f, half, before) in enumerate(((u, (0, 1, 1), (0, 0, -1)), (v, (1, 0, 1), (0, -1, 0)),
                                                   (w, (1, 1, 0), (-1, 0, 0)))):
                vel = [au, av, aw]
                vel[k] = f[c]
                pos = [(t + 0.5 if h else t) - dt * q for t, h, q in zip((x, y, z), half, vel)]
                ok = s & at(self.s, *before)
                for a in range(3):
                    if a != k:
                        ok = ok & inside[a]
                new[k][c] = torch.where(ok, self.sample(f, pos, half), new[k][c])
        for z0 in range(1, nz - 1, planes):
            z1 = min(nz - 1, z0 + planes)
            c = (slice(z0, z1), slice(1, ny - 1), slice(1, nx - 1))
            z, y, x = (t.double() for t in _axes(nz, ny, nx))
            mean = [(new[0][c] + new[0][z0:z1, 1:ny - 1, 2:nx]) / 2, (new[1][c] + new[1][z0:z1, 2:ny, 1:nx - 1]) / 2,
                    (new[2][c] + new[2][z0 + 1:z1 + 1, 1:ny - 1, 1:nx - 1]) / 2]
            pos = [t + 0.5 - q * dt for t, q in zip((x[:, :, 1:nx - 1], y[:, 1:ny - 1], z[z0:z1]), mean)]
            self.rho_out[c] = torch.where(self.s[c], self.sample(self.rho, pos, (1, 1, 1)), self.rho_out[c])
        return self.rho_out


def _exact_step(sc, storage, spheres):
    dev = _device()
    # values of BF16 storage are rounded before the first pass; the pass itself is exact
    bf = lambda a, on: (a.bfloat16() if on else a).double()  # noqa: E731
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)  # noqa: E731
    e = _Exact(t(sc.initial_mask()), bf(t(sc.initial_density()), storage == 1),
               [bf(t(sc.initial_velocity(k)), storage != 0) for k in "uvw"],
               torch.zeros(sc.cell_shape, dtype=torch.float64, device=dev))
    dt = float(np.float32(sc.dt))
    e.objects(sc, spheres)
    e.forcing(dt, float(np.float32(sc.gravity)), sc.buoyancy, sc.clamp_const)
    if sc.scheme == 0:
        e.project_velocity(sc.iterations, sc.omega)
    else:
        e.project_pressure(sc.iterations, sc.omega, float(np.float32(sc.tol)), sc.check_every)
    return e.advect(dt)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("serve", "render"):
        return None  # many steps; half-precision buffers by definition
    if kind == "project":
        vel, mask = _own_field(case, seed)
        e = _Exact(mask, torch.zeros(mask.shape, dtype=torch.float64, device=mask.device), [f.double() for f in vel], None)
        e.project_pressure(case["sweeps"], 1.9, float(np.float32(case["tol"])), case["check"])
        return [e.u, e.v, e.w]
    if kind == "batch":
        return torch.cat([_exact_step(sc, case["storage"], sc.spheres).reshape(-1) for sc in _cubes(case, seed)])
    sc = _scene(case, seed)
    spheres = [(*_drag(sc.spheres[0], 0), sc.spheres[0][3])] if case["move"] else sc.spheres
    out = _exact_step(sc, case["storage"], spheres)
    return out.cpu().numpy() if kind == "simulate" else out
