"""Timed cases: the work that a user of the implicit MPM snow solver has it do, through the
C ABI's ctypes binding, from a few thousand particles to the largest workload.

Kinds of case:
  substeps  a scene or a batch of scenes given by the host, k fixed-size substeps, the new
            state back on the host (the state a coupled program or a parameter sweep
            exchanges). Host arrays are pinned, as a program that does this often keeps them.
  frame     the same with the CFL time step of the reference's driver instead of k fixed
            ones: "device" is one mpm_advance_to_time, "host" the reference's driver loop (the
            largest particle speed read back, then one substep).
  transfer  a whole checkpoint (every particle field, FP64 arrays) written and read back.
  sort      the stable pair sort offered to callers that own their device memory.

A pass of the first two kinds starts from the same host arrays every time, so every pass
does the same work. "flight" states are nearly unstrained bodies before contact; "impact"
states are strained up to and beyond the yield limits, partly compacted and hardened, and
lie on the ground or press against each other.
"""
import ctypes as C
import math
import random

import numpy as np
import torch

from non_ficks_diffusion_gb300 import capi

DENSITY, NU, DT = 400.0, 0.2, 1e-4
FLUID_DENSITY, FLUID_BULK, FLUID_GAMMA = 2.0, 1.0, 7.0
PPC = 8


def listed():
    return [
        # a first look at a small scene: substeps of a few tens of microseconds, all launch latency
        {"name": "ball_3k_fp32", "kind": "substeps", "precision": "fp32", "material": "snow", "shape": "ball", "state": "flight",
         "scenes": 1, "particles": 3000, "nx": 32, "ny": 32, "nz": 32, "layout": 0, "substeps": 16},
        # a body in an elongated domain with odd grid sizes, after its impact
        {"name": "box_61k_mixed", "kind": "substeps", "precision": "mixed", "material": "snow", "shape": "box", "state": "impact",
         "scenes": 1, "particles": 61000, "nx": 92, "ny": 60, "nz": 76, "layout": 0, "substeps": 16},
        # the 128^3 snowball in the shipped precision of the reference
        {"name": "snowball_237k_fp32", "kind": "substeps", "precision": "fp32", "material": "snow", "shape": "ball", "state": "flight",
         "scenes": 1, "particles": 237000, "nx": 128, "ny": 128, "nz": 128, "layout": 0, "substeps": 16},
        # the same body in double precision (validation runs)
        {"name": "snowball_237k_fp64", "kind": "substeps", "precision": "fp64", "material": "snow", "shape": "ball", "state": "flight",
         "scenes": 1, "particles": 237000, "nx": 128, "ny": 128, "nz": 128, "layout": 0, "substeps": 4},
        # two snowballs in collision on 256^3, mixed precision
        {"name": "snowballs_2m_mixed", "kind": "substeps", "precision": "mixed", "material": "snow", "shape": "pair", "state": "impact",
         "scenes": 1, "particles": 1940000, "nx": 256, "ny": 256, "nz": 256, "layout": 0, "substeps": 8},
        # the snow slab on 512^3, the largest single scene
        {"name": "slab_21m_fp32", "kind": "substeps", "precision": "fp32", "material": "snow", "shape": "slab", "state": "flight",
         "scenes": 1, "particles": 21500000, "nx": 512, "ny": 512, "nz": 512, "layout": 0, "substeps": 2},
        # the batch of 64 scenes of 10^4 to 10^6 particles, mixed precision
        {"name": "batch64_mixed", "kind": "substeps", "precision": "mixed", "material": "snow", "shape": "mix", "state": "flight",
         "scenes": 64, "particles": 215000, "nx": 0, "ny": 0, "nz": 0, "layout": 104, "substeps": 4},
        # the reference's fluid ball with its equation of state
        {"name": "fluid_20k_fp32", "kind": "substeps", "precision": "fp32", "material": "fluid", "shape": "ball", "state": "flight",
         "scenes": 1, "particles": 20000, "nx": 64, "ny": 64, "nz": 64, "layout": 0, "substeps": 16},
        # part of a frame with the CFL time step chosen on the device
        {"name": "frame_40k_mixed", "kind": "frame", "precision": "mixed", "material": "snow", "shape": "pair", "state": "impact",
         "scenes": 1, "particles": 40000, "nx": 64, "ny": 64, "nz": 64, "layout": 0, "seconds": 0.004, "stepping": "device"},
        # the reference's driver loop: speed read back, one substep, for part of a frame
        {"name": "driver_40k_fp32", "kind": "frame", "precision": "fp32", "material": "snow", "shape": "ball", "state": "flight",
         "scenes": 1, "particles": 40000, "nx": 64, "ny": 64, "nz": 64, "layout": 0, "seconds": 0.004, "stepping": "host"},
        # checkpoint of the two snowballs: every field in FP64, in and out
        {"name": "checkpoint_2m", "kind": "transfer", "precision": "mixed", "material": "snow", "shape": "pair", "state": "impact",
         "scenes": 1, "particles": 1940000, "nx": 256, "ny": 256, "nz": 256, "layout": 0},
        # the pair sort near its largest size, on keys of a large grid
        {"name": "sort_1m_24bit", "kind": "sort", "pairs": 1000003, "bits": 24, "values": True},
    ]


def draw(rng):
    kind = rng.choices(["substeps", "frame", "transfer", "sort"], [7, 1, 1, 1])[0]
    if kind == "sort":
        return {"kind": "sort", "pairs": int(math.exp(rng.uniform(math.log(1000), math.log(1 << 20)))),
                "bits": rng.choice([8, 13, 16, 21, 24, 30]), "values": rng.random() < 0.5}
    precision = rng.choices(["fp32", "mixed", "fp64"], [4, 4, 1])[0]
    scenes = 1 if kind != "substeps" or rng.random() < 0.6 else int(round(math.exp(rng.uniform(math.log(2), math.log(64)))))
    most = 2.4e5 if precision == "fp64" else 5e4 if kind == "frame" else 1.2e7
    total = math.exp(rng.uniform(math.log(max(2000, 1500 * scenes)), math.log(most)))
    particles = int(total / scenes)
    material = "fluid" if kind == "substeps" and scenes == 1 and rng.random() < 0.15 else "snow"
    case = {"kind": kind, "precision": precision, "material": material,
            "shape": "mix" if scenes > 1 else rng.choice(["ball", "box", "pair"]), "state": rng.choice(["flight", "impact"]),
            "scenes": scenes, "particles": particles, "nx": 0, "ny": 0, "nz": 0, "layout": rng.randrange(1, 10 ** 6)}
    if scenes == 1:   # a grid on which the body spans a tenth to half of the domain, its axes up to 30 % apart
        n = _grid_cells(particles, rng.uniform(0.07, 0.22))
        case.update({k: max(16, 4 * round(n * rng.uniform(0.85, 1.15) / 4)) for k in ("nx", "ny", "nz")})
    if kind == "substeps":
        case["substeps"] = rng.choice([1, 2, 3, 5, 8]) if total < 3e6 else rng.choice([1, 2, 3])
    elif kind == "frame":
        case.update({"seconds": rng.choice([0.001, 0.0025, 0.004]), "stepping": rng.choice(["device", "host"])})
    return case


def _dt(case):
    """Fixed substep: the presets' 1e-4 for snow, 1e-3 on 64 cells for the fluid, as its cells."""
    return DT if case["material"] == "snow" else 0.064 / max(case["nx"], case["ny"], case["nz"])


def _grid_cells(particles, radius):
    return (particles / (PPC * 4 / 3 * math.pi * radius ** 3)) ** (1 / 3)


# ---------------------------------------------------------------------------------------
# scenes
# ---------------------------------------------------------------------------------------
def _scenes(case):
    """The scenes of a case: grid, shapes (centre, half extents, is it a ball, velocity, Young's
    modulus) and hardening, from the case alone."""
    r = random.Random(case["layout"])
    out = []
    for _ in range(case["scenes"]):
        if case["shape"] == "mix":   # log-uniform over a factor of 100 around the mean, as the batch preset
            n_p = case["particles"] * 4.65 / 100 * 100 ** r.random()
            n = max(16, 4 * round(_grid_cells(n_p, r.uniform(0.08, 0.2)) / 4))
            grid, kind = (n, n, n), r.choice(["ball", "box"])
            E, hardening = r.uniform(0.8e5, 2e5), r.uniform(5, 10)
            v = [r.uniform(-3, 3), r.uniform(-4, 2), r.uniform(-3, 3)]
        else:
            n_p, grid, kind = case["particles"], (case["nx"], case["ny"], case["nz"]), case["shape"]
            E, hardening, v = 1.4e5, 10.0, [0.0, -3.0, 0.0]
        volume = n_p / PPC / (grid[0] * grid[1] * grid[2])
        lowest = 2.0 / grid[1]        # the ground
        impact = case["state"] == "impact"
        if kind == "slab":
            shapes = [((0.5, 0.44, 0.5), (0.25, 0.04, 0.25), False, (0.0, -4.0, 0.0), E)]
        elif kind == "pair":
            h = (volume / 2 / (4 / 3 * math.pi)) ** (1 / 3)
            gap = h * (0.97 if impact else 1.3)
            shapes = [((0.5 - gap, 0.5, 0.5), (h, h, h), True, (3.0, 0.0, 0.0), E),
                      ((0.5 + gap, 0.5 + h / 6, 0.5), (h, h, h), True, (-3.0, 0.0, 0.0), 1.5 * E)]
        else:
            ball = kind == "ball"
            h = (volume / (4 / 3 * math.pi)) ** (1 / 3) if ball else (volume / 8) ** (1 / 3)
            y = lowest + 0.98 * h if impact else 0.6
            shapes = [((0.5, y, 0.5), (h, h, h), ball, tuple(v), E)]
        out.append({"grid": grid, "shapes": shapes, "hardening": hardening})
    return out


def _scene_desc(case, scene):
    d = capi.default_scene()
    fluid = case["material"] == "fluid"
    for a in range(3):
        d.counts[a] = scene["grid"][a]
    d.gravity[1] = -2.0 if fluid else -9.8
    d.cg_abs_tol, d.cg_rel_tol, d.cg_max_iters = 0.0, 1e-5, 50
    d.plastic, d.hardening = int(not fluid), scene["hardening"]
    d.compression_yield, d.stretching_yield = 1 - 2.5e-2, 1 + 7.5e-3
    if fluid:
        d.material, d.bulk_modulus, d.eos_gamma = capi.MATERIAL_EOS_FLUID, FLUID_BULK, FLUID_GAMMA
    d.n_barriers = 6                  # the ground (sticky under snow) and slip walls, two cells from the faces
    for b, (axis, sign) in enumerate([(1, 1), (0, 1), (0, -1), (1, -1), (2, 1), (2, -1)]):
        w = 2.0 / scene["grid"][axis]
        d.barriers[b].normal[axis] = sign
        d.barriers[b].surface[axis] = w if sign > 0 else 1 - w
        d.barriers[b].sticky = int(b == 0 and not fluid)
    return d


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _fields(x, gen, state):
    """Smooth velocity disturbance, deformation gradient and compaction over positions x."""
    dev = x.device
    flight = state == "flight"

    def waves(count):                 # `count` plane waves of wavelength 0.1 to 0.2 domain lengths
        k = torch.randn(3, count, generator=gen, device=dev)
        k = k / k.norm(dim=0) * (2 * math.pi / (0.1 + 0.1 * torch.rand(count, generator=gen, device=dev)))
        return torch.sin(x @ k + 2 * math.pi * torch.rand(count, generator=gen, device=dev))

    v = waves(3) * (0.005 if flight else 0.4)
    e = waves(6) * (1e-4 if flight else 0.02)
    t = waves(3) * (0.05 if flight else 0.3)
    F = torch.zeros(len(x), 3, 3, device=dev)
    for a in range(3):
        F[:, a, a] = 1 + e[:, a] - (0.0 if flight else 0.01)
    for q, (a, b) in enumerate([(0, 1), (0, 2), (1, 2)]):
        F[:, a, b] = F[:, b, a] = 0.5 * e[:, 3 + q]
    for q, (a, b) in enumerate([(0, 1), (0, 2), (1, 2)]):   # then rotations about the three axes
        c, s = torch.cos(t[:, q]), torch.sin(t[:, q])
        ra, rb = F[:, a].clone(), F[:, b].clone()
        F[:, a], F[:, b] = c[:, None] * ra - s[:, None] * rb, s[:, None] * ra + c[:, None] * rb
    jp = torch.ones(len(x), device=dev) if flight else 0.94 + 0.06 * waves(1)[:, 0]
    return v, F.reshape(-1, 9), jp


def _particles(case, seed):
    """Per scene: X, V, Fe, Jp, mass, lambda0, mu0 as FP32 tensors (jittered samples, PPC per cell)."""
    dev = _device()
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    fluid = case["material"] == "fluid"
    out = []
    for scene in _scenes(case):
        cells = torch.tensor(scene["grid"], device=dev, dtype=torch.float32)
        parts = []
        for s, (c, h, ball, vel, E) in enumerate(scene["shapes"]):
            axes = [torch.arange(max(0, int((c[a] - h[a]) * scene["grid"][a]) - 1),
                                 min(scene["grid"][a], int((c[a] + h[a]) * scene["grid"][a]) + 2), device=dev) for a in range(3)]
            g = torch.stack(torch.meshgrid(*axes, indexing="ij"), -1).reshape(-1, 1, 3).float()
            sub = torch.stack(torch.meshgrid(*[torch.arange(2, device=dev)] * 3, indexing="ij"), -1).reshape(1, 8, 3).float()
            x = ((g + (sub + torch.rand(len(g), 8, 3, generator=gen, device=dev)) / 2) / cells).reshape(-1, 3)
            centre, half = torch.tensor(c, device=dev), torch.tensor(h, device=dev)
            # whole sub-cells, by their centres, so that the count does not hang on the jitter
            mid = ((g + (sub + 0.5) / 2) / cells).reshape(-1, 3)
            d = (mid - centre) / half
            keep = (d.square().sum(1) < 1) if ball else (d.abs() < 1).all(1)
            # one body per place: the second ball of a pair leaves out what the first one fills
            if s:
                c0, h0 = (torch.tensor(t, device=dev) for t in scene["shapes"][0][:2])
                keep &= ((mid - c0) / h0).square().sum(1) >= 1
            x = x[keep]
            v, F, jp = _fields(x, gen, case["state"])
            n = len(x)
            mass = (FLUID_DENSITY if fluid else DENSITY) / (PPC * float(np.prod(scene["grid"])))
            full = lambda value, n=n: torch.full((n,), value, device=dev, dtype=torch.float32)  # noqa: E731
            parts.append({"X": x, "V": v + torch.tensor(vel, device=dev), "Fe": F,
                          "Jp": full(FLUID_DENSITY) * (1 + 0.02 * (jp - 1)) if fluid else jp, "mass": full(mass),
                          "lambda0": full(E * NU / ((1 + NU) * (1 - 2 * NU))), "mu0": full(E / (2 * (1 + NU)))})
        out.append({k: torch.cat([p[k] for p in parts]).contiguous() for k in parts[0]})
    return out


# ---------------------------------------------------------------------------------------
# the program around the calls
# ---------------------------------------------------------------------------------------
class _HostArrays:
    """Pinned host arrays of some particle fields over all scenes, and the per-scene views the
    batched transfer calls take."""

    WIDTH = {"X": 3, "V": 3, "Fe": 9, "Jp": 1, "mass": 1, "lambda0": 1, "mu0": 1, "V0": 1}

    def __init__(self, sizes, fields, dtype, valid):
        n = sum(sizes)
        self.field = {k: torch.empty((n, self.WIDTH[k]) if self.WIDTH[k] > 1 else (n,), dtype=dtype, pin_memory=True) for k in fields}
        if valid:
            self.field["valid"] = torch.empty(n, dtype=torch.int32, pin_memory=True)
        self.views = (capi.ParticleArrays * len(sizes))()
        self.ids = (C.c_int * len(sizes))(*range(len(sizes)))
        at = 0
        for view, size in zip(self.views, sizes):
            view.n, view.dtype = size, capi.F64 if dtype == torch.float64 else capi.F32
            for k, t in self.field.items():
                p = t.data_ptr() + at * t.element_size() * (t.shape[1] if t.dim() > 1 else 1)
                setattr(view, k, C.cast(p, C.POINTER(C.c_int)) if k == "valid" else p)
            at += size


def _checked(ctx, status):
    if status != capi.OK:
        raise capi.MPMError(status, ctx.L.mpm_last_error(ctx.h).decode())


def prepare(case, seed):
    if case["kind"] == "sort":
        gen = torch.Generator(device="cuda")
        gen.manual_seed(seed)
        n = case["pairs"]
        keys = torch.randint(0, 1 << case["bits"], (n,), generator=gen, device="cuda", dtype=torch.int64).to(torch.int32)
        vals = torch.randperm(n, generator=gen, device="cuda").to(torch.int32) if case["values"] else None
        return {"case": case, "keys": keys, "vals": vals, "out": (torch.empty_like(keys), torch.empty_like(keys)), "lib": capi.lib()}
    scenes, parts = _scenes(case), _particles(case, seed)
    sizes = [len(p["X"]) for p in parts]
    ctx = capi.Context(precision=case["precision"], max_particles=sum(sizes), max_scenes=len(sizes))
    for scene, p in zip(scenes, parts):
        host = {k: t.double().cpu().numpy() for k, t in p.items() if k not in ("Fe", "Jp")}
        ctx.add_particles(ctx.add_scene(_scene_desc(case, scene)), **host)
    ctx.initialize()
    transfer = case["kind"] == "transfer"
    dtype = torch.float64 if transfer or case["precision"] == "fp64" else torch.float32
    fields = ["X", "V", "Fe", "Jp"] + (["mass", "lambda0", "mu0", "V0"] if transfer else [])
    given, back = _HostArrays(sizes, fields, dtype, transfer), _HostArrays(sizes, fields, dtype, True)
    for k, t in given.field.items():
        if k == "valid":
            t.fill_(1)
        elif k == "V0":
            t.copy_((torch.cat([p["mass"] for p in parts]) / DENSITY).to(dtype))
        else:
            t.copy_(torch.cat([p[k] for p in parts]).to(dtype))
    return {"case": case, "ctx": ctx, "given": given, "back": back, "dx": 1.0 / scenes[0]["grid"][0]}


def run(state):
    case = state["case"]
    if case["kind"] == "sort":
        keys, vals, (k, v) = state["keys"], state["vals"], state["out"]
        status = state["lib"].mpm_sort_pairs_noalloc(keys.data_ptr(), vals.data_ptr() if vals is not None else None, k.data_ptr(),
                                                     v.data_ptr(), len(keys), 0, case["bits"], torch.cuda.current_stream().cuda_stream)
        if status != capi.OK:
            raise capi.MPMError(status, "mpm_sort_pairs_noalloc")
        return {"keys": k, "values": v}
    ctx, given, back = state["ctx"], state["given"], state["back"]
    _checked(ctx, ctx.L.mpm_set_particles_batch(ctx.h, len(given.ids), given.ids, given.views))
    out = dict(back.field)
    if case["kind"] == "substeps":
        ctx.step(_dt(case), case["substeps"])
    elif case["kind"] == "frame":
        ctx.set_time(0.0)
        if case["stepping"] == "device":
            out["substeps"] = ctx.advance_to_time(case["seconds"])
        else:
            out["substeps"] = _driver_loop(ctx, case["seconds"], state["dx"])
    _checked(ctx, ctx.L.mpm_get_particles_batch(ctx.h, len(back.ids), back.ids, back.views))
    return out


def _time_step(vmax, dx, rest):
    """The reference's CFL rule and end-of-frame split: (substep, is it the last)."""
    dt = min(max(0.1 * dx / max(vmax, 1e-2), 1e-6), 5e-3)
    if rest < dt * 1.001:
        return rest, True
    return (0.5 * rest if rest < 2 * dt else dt), False


def _driver_loop(ctx, seconds, dx):
    t, count, last = 0.0, 0, False
    while not last:
        dt, last = _time_step(ctx.max_velocity(0), dx, seconds - t)
        ctx.step(dt)
        t, count = t + dt, count + 1
    return count


def work(case):
    """Every particle's state crosses memory once in and once out per substep (20 words in, 16
    changed words out) and once each way over the host link per pass. Arithmetic per particle
    and substep: stress, two 27-node scatters and gathers of the explicit part and G2P and
    two products of the implicit operator, the fewest that a solve of one iteration takes."""
    if case["kind"] == "sort":
        return {"bytes": case["pairs"] * (16 if case["values"] else 12), "flops": 0}
    n, word = case["particles"] * case["scenes"], 8 if case["precision"] == "fp64" else 4
    if case["kind"] == "transfer":
        return {"bytes": 2 * n * (20 * (word + 8) + 8), "flops": 0}
    k = case["substeps"] if case["kind"] == "substeps" else math.ceil(case["seconds"] / (0.1 / case["nx"] / 3.0))
    return {"bytes": n * word * (36 * k + 4 * 16), "flops": n * k * 3700}


# ---------------------------------------------------------------------------------------
# the same in 64 bits, on dense arrays
# ---------------------------------------------------------------------------------------
EXACT_PARTICLE_SUBSTEPS = 4e6        # more would take too long


def exact(case, seed):
    if case["kind"] == "sort":
        return None
    if case["kind"] == "transfer":
        p = _particles(case, seed)[0]
        out = {k: p[k].double() for k in ("X", "V", "Fe", "Jp", "mass", "lambda0", "mu0")}
        return dict(out, V0=(p["mass"] / DENSITY).double(), valid=None)
    k = case.get("substeps") or 12
    if case["particles"] * case["scenes"] * k > EXACT_PARTICLE_SUBSTEPS:
        return None
    ends = []
    for scene, p in zip(_scenes(case), _particles(case, seed)):
        s = _Exact(case, scene, p)
        if case["kind"] == "frame":
            t, last = 0.0, False
            while not last:
                step, last = _time_step(float(s.V[s.valid].square().sum(1).max()) ** 0.5, 1.0 / scene["grid"][0], case["seconds"] - t)
                s.substep(step)
                t += step
        else:
            for _ in range(k):
                s.substep(_dt(case))
        ends.append({"X": s.X, "V": s.V, "Fe": s.F.reshape(-1, 9), "Jp": s.Jp})
    out = {f: torch.cat([e[f] for e in ends]) for f in ends[0]}
    return dict(out, valid=None, **({"substeps": None} if case["kind"] == "frame" else {}))


class _Exact:
    """One scene in FP64: quadratic B-spline transfers, fixed-corotated snow with its yield
    limits or the fluid, and the conjugate-gradient solve with the solver's stopping rule."""

    def __init__(self, case, scene, p):
        self.case, self.n = case, torch.tensor(scene["grid"], device=p["X"].device, dtype=torch.float64)
        self.fluid = case["material"] == "fluid"
        self.hardening = scene["hardening"]
        self.X, self.V, self.F, self.Jp = p["X"].double(), p["V"].double(), p["Fe"].double().reshape(-1, 3, 3), p["Jp"].double()
        self.m, self.lam0, self.mu0 = p["mass"].double(), p["lambda0"].double(), p["mu0"].double()
        self.valid = torch.ones(len(self.X), dtype=torch.bool, device=self.X.device)
        self.gravity = torch.tensor([0.0, -2.0 if self.fluid else -9.8, 0.0], device=self.X.device, dtype=torch.float64)
        self._stencil()
        density = self._gather(self._scatter(lambda w, g: (self.m * w)[:, None], 1), lambda w, g, s: s[:, 0] * w)
        self.V0 = self.m / (density * float(self.n.prod()))

    def _stencil(self):
        x = self.X * self.n
        cell = x.floor()
        lo = cell.long().amin(0) - 1
        self.shape = (cell.long().amax(0) + 2 - lo).tolist()
        self.lo, self.base = lo, cell.long() - 1 - lo
        t = x - cell - 0.5                       # offset from the cell's centre, in cells
        self.w = torch.stack([0.5 * (0.5 - t) ** 2, 0.75 - t * t, 0.5 * (0.5 + t) ** 2], 1)
        self.dw = torch.stack([t - 0.5, -2 * t, t + 0.5], 1) * self.n
        self.nodes = self.shape[0] * self.shape[1] * self.shape[2]

    def _offsets(self):
        for i in range(3):
            for j in range(3):
                for k in range(3):
                    node = ((self.base[:, 0] + i) * self.shape[1] + self.base[:, 1] + j) * self.shape[2] + self.base[:, 2] + k
                    wx, wy, wz = self.w[:, i, 0], self.w[:, j, 1], self.w[:, k, 2]
                    g = torch.stack([self.dw[:, i, 0] * wy * wz, wx * self.dw[:, j, 1] * wz, wx * wy * self.dw[:, k, 2]], 1)
                    yield node, wx * wy * wz, g

    def _scatter(self, value, width):
        out = torch.zeros(self.nodes, width, device=self.X.device, dtype=torch.float64)
        for node, w, g in self._offsets():
            v = value(w, g)
            out.index_add_(0, node[self.valid], v[self.valid])
        return out

    def _gather(self, nodal, value):
        total = 0.0
        for node, w, g in self._offsets():
            total = total + value(w, g, nodal[node])
        return total

    def _plasticity(self):
        U, s, Vt = torch.linalg.svd(self.F)
        c = s.clamp(1 - 2.5e-2, 1 + 7.5e-3)
        v = self.valid
        self.Jp = torch.where(v, self.Jp * s.prod(1) / c.prod(1), self.Jp)
        self.F = torch.where(v[:, None, None], U * c[:, None, :] @ Vt, self.F)
        self.R = U @ Vt
        e = torch.exp(self.hardening * (1 - self.Jp))
        self.lam, self.mu = e * self.lam0, e * self.mu0

    @staticmethod
    def _cofactor(F):
        return torch.stack([torch.linalg.cross(F[:, 1], F[:, 2]), torch.linalg.cross(F[:, 2], F[:, 0]), torch.linalg.cross(F[:, 0], F[:, 1])], 1)

    def _product(self, u):
        """The elastic force differential of nodal displacements u."""
        G = self._gather(u, lambda w, g, s: s[:, :, None] * g[:, None, :])
        if self.fluid:
            e = self.lam * G.diagonal(dim1=1, dim2=2).sum(1)
            return self._scatter(lambda w, g: e[:, None] * g, 3)
        dF = G @ self.F
        H, J = self._cofactor(self.F), torch.linalg.det(self.F)
        S, M = self.R.transpose(1, 2) @ self.F, self.R.transpose(1, 2) @ dF
        # R^T dR = [[0, -a, -b], [a, 0, -c], [b, c, 0]] with (S W + W S) = M - M^T
        K = torch.stack([torch.stack([S[:, 0, 0] + S[:, 1, 1], S[:, 2, 1], -S[:, 2, 0]], 1),
                         torch.stack([S[:, 2, 1], S[:, 0, 0] + S[:, 2, 2], S[:, 1, 0]], 1),
                         torch.stack([-S[:, 2, 0], S[:, 1, 0], S[:, 1, 1] + S[:, 2, 2]], 1)], 1)
        L = torch.stack([M[:, 1, 0] - M[:, 0, 1], M[:, 2, 0] - M[:, 0, 2], M[:, 2, 1] - M[:, 1, 2]], 1)
        adj = self._cofactor(K)
        abc = (adj @ L[:, :, None])[:, :, 0] / torch.linalg.det(K)[:, None]
        a, b, c = abc.unbind(1)
        z = torch.zeros_like(a)
        W = torch.stack([torch.stack([z, -a, -b], 1), torch.stack([a, z, -c], 1), torch.stack([b, c, z], 1)], 1)
        cr = torch.linalg.cross
        dH = torch.stack([cr(dF[:, 1], self.F[:, 2]) + cr(self.F[:, 1], dF[:, 2]), cr(dF[:, 2], self.F[:, 0]) + cr(self.F[:, 2], dF[:, 0]),
                          cr(dF[:, 0], self.F[:, 1]) + cr(self.F[:, 0], dF[:, 1])], 1)
        dP = (2 * self.mu[:, None, None] * (dF - self.R @ W) + (self.lam * (H * dF).sum((1, 2)))[:, None, None] * H
              + (self.lam * (J - 1))[:, None, None] * dH)
        A = self.V0[:, None, None] * dP @ self.F.transpose(1, 2)
        return self._scatter(lambda w, g: (A @ g[:, :, None])[:, :, 0], 3)

    def substep(self, dt):
        self._stencil()
        if self.fluid:
            pw = self.Jp ** (FLUID_GAMMA - 1)
            self.lam = self.V0 * FLUID_BULK * FLUID_GAMMA * pw
            stress = (-self.V0 / self.Jp * FLUID_BULK * pw)[:, None, None] * torch.eye(3, device=self.X.device, dtype=torch.float64)
        else:
            self._plasticity()
            J = torch.linalg.det(self.F)
            P = 2 * self.mu[:, None, None] * (self.F - self.R) + (self.lam * (J - 1))[:, None, None] * self._cofactor(self.F)
            stress = self.V0[:, None, None] * P @ self.F.transpose(1, 2)
        grid = self._scatter(lambda w, g: torch.cat([(self.m * w)[:, None], (self.m * w)[:, None] * self.V,
                                                     (self.m * w)[:, None] * self.gravity - (stress @ g[:, :, None])[:, :, 0]], 1), 7)
        m = grid[:, :1]
        there = m > 0
        m = torch.where(there, m, torch.ones_like(m))
        v = grid[:, 1:4] / m
        b, held = self._collide(v + dt * grid[:, 4:] / m)
        b, held = b * there, held | ~there
        x = b.clone()

        def system(u):
            return dt * dt / m * self._product(u) + u

        def norm(u):
            return float(u.square().sum(1).max()) ** 0.5

        tol = 1e-5 * norm(b)
        r = torch.where(held, torch.zeros_like(b), b - system(x))
        s, rho, iters = torch.zeros_like(b), 0.0, 0
        while norm(r) > tol and iters < 50:
            rr = float((m * r * r).sum())
            s = r + (rr / rho if iters else 0.0) * s
            q = torch.where(held, torch.zeros_like(b), system(s) * there)
            alpha = rr / float((m * s * q).sum())
            x, r, rho, iters = x + alpha * s * there, r - alpha * q, rr, iters + 1
        self._to_particles(x, v * there, dt)

    def _collide(self, v):
        axes = [(torch.arange(self.shape[a], device=v.device) + self.lo[a] + 0.5) / self.n[a] for a in range(3)]
        x = torch.stack(torch.meshgrid(*axes, indexing="ij"), -1).reshape(-1, 3)
        held = torch.zeros(len(x), 1, dtype=torch.bool, device=v.device)
        for b, (axis, sign) in enumerate([(1, 1), (0, 1), (0, -1), (1, -1), (2, 1), (2, -1)]):
            w = 2.0 / self.n[axis]
            inside = (x[:, axis] < w) if sign > 0 else (x[:, axis] > 1 - w)
            held |= inside[:, None]
            if b == 0 and not self.fluid:
                v = torch.where(inside[:, None], torch.zeros_like(v), v)
            else:
                into = inside & (sign * v[:, axis] < 0)
                v = v.clone()
                v[into, axis] = 0.0
        return v, held

    def _to_particles(self, x, v, dt):
        new = self._gather(x, lambda w, g, s: s * w[:, None])
        change = self._gather(x - v, lambda w, g, s: s * w[:, None])
        G = self._gather(x, lambda w, g, s: s[:, :, None] * g[:, None, :])
        on = self.valid[:, None]
        if self.fluid:
            self.Jp = torch.where(self.valid, self.Jp / (1 + dt * G.diagonal(dim1=1, dim2=2).sum(1)), self.Jp)
        else:
            self.F = torch.where(on[:, :, None], self.F + dt * G @ self.F, self.F)
        self.V = torch.where(on, 0.9 * (self.V + change) + 0.1 * new, self.V)
        self.X = torch.where(on, self.X + dt * new, self.X)
        edge = 0.5 / self.n
        self.valid = self.valid & ((self.X >= edge) & (self.X <= 1 - edge)).all(1)
