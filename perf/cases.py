"""The performance cases of the library: what its users have it do, over the range they do it in.

Each case is one call of a program that has its fields on the GPU and goes on from there: a film
is drained for some steps, a batch of bubbles for some more, points are coloured, a surrogate is
trained or rolled out, a frame is drawn, rays are traced, a cluster is moved. A simulator's state
is its own between passes, so a further pass goes on where the last one ended, as a simulation
does. Sizes are those of the library's configurations and benchmark (resolution 128 and 2048, the
64 x 128 default grid, foam bubbles of 32 to 512 rows, 81 wavelengths, 256 x 512 training grids,
32,768 rays), with odd grids beside them.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

import soap_bubble_simulation_gb300 as sbs
from soap_bubble_simulation_gb300 import _native as N

DIFFUSION = 1e-9  # m^2/s, of h and of the surfactant (the defaults of both solvers)
RADIUS = 0.025  # m, the default bubble
CRIT_CPU = 10e-9


def stable_dt(nt: int, np_: int, radius: float = RADIUS, most: float = 1e-3) -> float:
    """The configurations' 1 ms, or what keeps the explicit step stable up to the poles."""
    dth, dph = math.pi / (nt - 1), 2.0 * math.pi / np_
    rate = DIFFUSION / radius**2 * (1.0 / dth**2 + 1.0 / (dph * math.sin(dth)) ** 2)
    return float(np.float32(min(most, 0.2 / rate)))


def is_stable(case: dict) -> bool:
    return case["dt"] <= stable_dt(case["nt"], case["np"], case.get("radius", RADIUS), 1e9) * 1.01


# --- cases ---------------------------------------------------------------------------------------
def wgsl(nt, np_, passes, marangoni=False, check=0, dt=None):
    return {"kind": "wgsl", "nt": nt, "np": np_, "passes": passes, "marangoni": marangoni, "check": check,
            "dt": stable_dt(nt, np_) if dt is None else dt}


def cpu(resolution, steps):
    return {"kind": "cpu", "nt": resolution, "np": 2 * resolution, "steps": steps,
            "dt": stable_dt(resolution, 2 * resolution)}


def listed():
    return [
        # one rendered frame of the interactive simulator: the default grid, ten passes a frame;
        # what it costs is latency and launches
        {"name": "frame_64x128", "kind": "frame", "nt": 64, "np": 128, "passes": 10, "frame_dt": 1.0 / 60.0},
        # one simulated second of the default configuration (resolution 128, 1 ms, regeneration
        # fronts on), in the reference's CPU semantics
        {"name": "cpu_128", **cpu(128, 1000)},
        # the same solver on the finest configured bubble
        {"name": "cpu_2048", **cpu(2048, 96)},
        # the headline run: 2048 x 4096, 1 ms, with a volume check every 100 passes. At this dt the
        # rings next to the poles are unstable, in any arithmetic (so there is no exact result).
        {"name": "wgsl_2048", **wgsl(2048, 4096, 400, check=100, dt=1e-3)},
        # a grid that no tile divides, with the Marangoni term
        {"name": "marangoni_517x1037", **wgsl(517, 1037, 200, marangoni=True)},
        # a foam: bubbles of very different sizes advanced together
        {"name": "foam_384", "kind": "foam", "bubbles": 384, "steps": 800, "rmin": 32, "rmax": 512, "step": 32},
        # spectral colours of a film's surface points on the tensor cores
        {"name": "spectral_4m", "kind": "spectral", "n": 4_194_304, "nl": 81, "mode": "tc"},
        # training iterations of the surrogate (gradients and updated weights), its usual batch
        {"name": "train_256", "kind": "train", "nt": 256, "np": 512, "batch": 8, "iters": 8, "act": "gelu"},
        # the surrogate advancing the finest bubble, the plain solver checking one interval in eight
        {"name": "rollout_2048", "kind": "rollout", "nt": 2048, "np": 4096, "passes": 512, "every": 8,
         "act": "gelu", "dt": 1e-3},
        # one headless frame to host memory
        {"name": "shade_1080p", "kind": "shade", "width": 1920, "height": 1080},
        # the light rays of one frame at the default settings
        {"name": "branched_32768", "kind": "branched", "rays": 32768, "steps": 400, "scatterers": 800},
        # a foam cluster's motion: twenty steps, then the bubbles read back
        {"name": "cluster_40000", "kind": "cluster", "n": 40000, "steps": 20, "dt": 1e-3},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "cpu", "cpu", "wgsl", "wgsl", "wgsl", "foam", "spectral", "train", "rollout", "shade",
                       "branched", "cluster"])
    if kind == "frame":
        nt = _log(rng, 16, 256)
        return {"kind": kind, "nt": nt, "np": 2 * nt + rng.choice([0, 0, 1, 2]), "passes": rng.randint(2, 20),
                "frame_dt": 1.0 / 60.0}
    if kind == "cpu":
        r = _log(rng, 33, 2000)
        return cpu(r, min(1000, max(10, int(4e8 * rng.uniform(0.3, 1.0) / (2 * r * r)))))
    if kind == "wgsl":
        nt = _log(rng, 48, 2000)
        np_ = int(nt * rng.uniform(1.0, 2.05))
        return wgsl(nt, np_, min(1000, max(10, int(2e9 * rng.uniform(0.2, 1.0) / (nt * np_)))),
                    marangoni=rng.random() < 0.5, check=rng.choice([0, 50, 100]))
    if kind == "foam":
        return {"kind": kind, "bubbles": _log(rng, 12, 300), "steps": rng.randint(50, 400), "rmin": 32,
                "rmax": rng.choice([128, 256, 512]), "step": rng.choice([2, 2, 32])}
    if kind == "spectral":
        return {"kind": kind, "n": _log(rng, 10_000, 4_000_000), "nl": rng.choice([81, 81, 41, 16, 128]),
                "mode": rng.choice(["tc", "fp32"])}
    if kind == "train":
        nt = rng.choice([64, 96, 128, 250, 256])
        return {"kind": kind, "nt": nt, "np": 2 * nt, "batch": rng.randint(1, 8), "iters": rng.randint(2, 8),
                "act": rng.choice(["gelu", "hswish"])}
    if kind == "rollout":
        nt = _log(rng, 128, 2000) // 2 * 2
        return {"kind": kind, "nt": nt, "np": 2 * nt, "passes": 64 * rng.randint(2, 8), "every": rng.choice([4, 8]),
                "act": rng.choice(["gelu", "hswish"]), "dt": 1e-3}
    if kind == "shade":
        h = _log(rng, 200, 2000)
        return {"kind": kind, "width": int(h * rng.uniform(1.0, 1.8)), "height": h}
    if kind == "branched":
        return {"kind": kind, "rays": _log(rng, 2000, 60000), "steps": rng.randint(50, 400),
                "scatterers": rng.randint(100, 1200)}
    return {"kind": "cluster", "n": _log(rng, 300, 200000), "steps": rng.randint(5, 20), "dt": 1e-3}


# --- inputs --------------------------------------------------------------------------------------
def _modes(nt, np_, seed):
    """A film of 550 nm with 16 smooth modes, clamped to [100, 1000] nm (f64, on the GPU)."""
    g = np.random.default_rng([seed, 1])
    a, m, n = g.normal(0.0, 60e-9, 16), g.integers(1, 9, 16), g.integers(0, 9, 16)
    psi, chi = g.uniform(0.0, 2 * math.pi, 16), g.uniform(0.0, 2 * math.pi, 16)

    def t(x):
        return torch.as_tensor(x, dtype=torch.float64, device="cuda")

    th = torch.arange(nt, dtype=torch.float64, device="cuda") * (math.pi / (nt - 1))
    ph = torch.arange(np_, dtype=torch.float64, device="cuda") * (2 * math.pi / np_)
    u = t(a) * torch.cos(t(m) * th[:, None] + t(psi))
    v = torch.cos(t(n) * ph[:, None] + t(chi))
    return (550e-9 + u @ v.T).clamp(100e-9, 1000e-9).float().contiguous()


def _surfactant(nt, np_, seed):
    g = torch.Generator(device="cuda").manual_seed(seed * 7919 + 2)
    return 0.4 + 0.2 * torch.rand((nt, np_), generator=g, device="cuda")


def _foam_bubbles(case):
    """Diameters log-uniform in 2 - 80 mm (scaled with the largest grid), rows in proportion: a
    case's bubbles are the same for every seed, their films differ."""
    g = np.random.default_rng([case["bubbles"], case["rmax"], 3])
    top = 0.080 * case["rmax"] / 512.0
    d = np.exp(g.uniform(math.log(0.002), math.log(top), case["bubbles"]))
    step = case["step"]
    res = np.clip(step * np.round(512.0 * d / 0.080 / step), case["rmin"], case["rmax"]).astype(np.uint32)
    return res, (d / 2).astype(np.float32)


def _foam_dt(res, rad):
    return min(stable_dt(int(r), 2 * int(r), float(a)) for r, a in zip(res, rad))


def _foam_fields(case, res, seed):
    g = torch.Generator(device="cuda").manual_seed(seed * 7919 + 4)
    cells = int(sum(2 * int(r) * int(r) for r in res))
    base = torch.as_tensor(np.repeat(np.random.default_rng([seed, 5]).uniform(300e-9, 800e-9, len(res)),
                                     2 * res.astype(np.int64) ** 2), device="cuda")
    h = (base * (0.95 + 0.1 * torch.rand(cells, generator=g, device="cuda"))).float()
    c = 0.4 + 0.2 * torch.rand(cells, generator=g, device="cuda")
    return h, c


def _spectral_inputs(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed * 7919 + 6)
    u = torch.rand((3, case["n"]), generator=g, device="cuda")
    t, c, nf = 10.0 + 1490.0 * u[0], u[1].contiguous(), 1.30 + 0.10 * u[2]
    wl = np.linspace(380.0, 780.0, case["nl"]).astype(np.float32)
    lobes = [(600.0, 40.0, 1.0), (440.0, 20.0, 0.35), (550.0, 45.0, 1.0), (450.0, 25.0, 1.7)]
    b = [a * np.exp(-0.5 * ((wl - mu) / s) ** 2) for mu, s, a in lobes]
    cmf = np.ascontiguousarray(np.stack([b[0] + b[1], b[2], b[3]], axis=1), dtype=np.float32)
    return t, c, nf, wl, cmf


def _cluster(case, seed):
    pos, rad = sbs.fcc_foam(case["n"], seed=seed)
    return pos, rad


class _Buffer:
    """A simulator's device field as torch sees it (the rows' padding left out); it keeps the
    simulator, whose memory this is."""

    def __init__(self, sim, f):
        self.sim = sim
        self.__cuda_array_interface__ = {"shape": (f.num_theta, f.num_phi), "typestr": "<f4", "version": 2,
                                         "data": (f.ptr, False), "strides": (f.pitch * 4, 4)}


def _tensor(sim, field):
    return torch.as_tensor(_Buffer(sim, field), device="cuda")


def _fields(sim):
    return [_tensor(sim, sim.current_thickness_buffer()), _tensor(sim, sim.current_concentration_buffer())]


def _dev(t):
    return ctypes.c_void_p(t.data_ptr())


def _gpu_sim(case, seed, marangoni=False):
    nt, np_ = case["nt"], case["np"]
    sim = sbs.GPUDrainageSimulator(None, 500e-9, np_, nt)
    p = sim.params()
    p.dt = case.get("dt", p.dt)
    p.marangoni_enabled = 1 if marangoni else 0
    sim.update_params(p)
    h, c = _modes(nt, np_, seed), _surfactant(nt, np_, seed)
    torch.cuda.synchronize()
    sim.set_thickness_device(h.data_ptr(), h.numel())
    N.call("sbs_drainage_set_concentration", sim.handle, _dev(c), c.numel(), N.MEM_DEVICE)
    return sim


def prepare(case, seed):
    kind = case["kind"]
    if kind == "frame":
        sim = _gpu_sim(case, seed)
        sim.enabled = True
        sim.steps_per_frame = case["passes"]
        return {"case": case, "sim": sim}
    if kind == "wgsl":
        return {"case": case, "sim": _gpu_sim(case, seed, case["marangoni"])}
    if kind == "cpu":
        cfg = sbs.SimulationConfig.default()
        cfg.resolution, cfg.dt = case["nt"], case["dt"]
        sim = sbs.DrainageSimulator(cfg)
        h = _modes(case["nt"], case["np"], seed)
        torch.cuda.synchronize()
        sim.set_thickness_device(h.data_ptr(), h.numel())
        return {"case": case, "sim": sim}
    if kind == "foam":
        res, rad = _foam_bubbles(case)
        p = sbs.DrainageParams.default()
        p.dt = _foam_dt(res, rad)
        foam = sbs.FoamDrainage(res, rad, p)
        h, c = _foam_fields(case, res, seed)
        torch.cuda.synchronize()
        at = np.concatenate([[0], np.cumsum(2 * res.astype(np.int64) ** 2)])
        parts = [(b, int(at[b]), int(at[b + 1] - at[b])) for b in range(len(res))]
        for b, first, n in parts:
            N.call("sbs_foam_set_thickness", foam._h, b, _dev(h[first:]), n, N.MEM_DEVICE)
            N.call("sbs_foam_set_concentration", foam._h, b, _dev(c[first:]), n, N.MEM_DEVICE)
        return {"case": case, "foam": foam, "parts": parts, "h": h, "c": c}
    if kind == "spectral":
        t, c, nf, wl, cmf = _spectral_inputs(case, seed)
        return {"case": case, "t": t, "c": c, "nf": nf, "wl": wl, "cmf": cmf,
                "rgb": torch.empty((case["n"], 3), device="cuda")}
    if kind == "train":
        net = sbs.DrainageSurrogate(seed=seed, activation=case["act"])
        g = np.random.default_rng([seed, 7])
        for k in range(8):
            p = sbs.field_params(case["nt"], case["np"], dt=stable_dt(case["nt"], case["np"]),
                                 viscosity=float(10 ** g.uniform(-4, -2)), bubble_radius=float(g.uniform(0.02, 0.04)))
            net.add_trajectory(_modes(case["nt"], case["np"], seed * 97 + k).cpu().numpy(),
                               _surfactant(case["nt"], case["np"], seed * 97 + k).cpu().numpy(), p, pairs=2)
        return {"case": case, "net": net, "seed": seed}
    if kind == "rollout":
        return {"case": case, "net": sbs.DrainageSurrogate(seed=seed, activation=case["act"]),
                "sim": _gpu_sim(case, seed)}
    if kind == "shade":
        g = np.random.default_rng([seed, 8])
        u = sbs.BubbleUniform.default()
        u.set_time(float(g.uniform(0.0, 60.0)))
        cam = sbs.Camera(case["width"] / case["height"], distance=float(g.uniform(0.07, 0.12)),
                         yaw=float(g.uniform(0.0, 6.0)), pitch=float(g.uniform(-0.5, 0.5)))
        return {"case": case, "uniform": u, "camera": cam,
                "lut": sbs.generate_interference_lut_array(u.refractive_index, 1.0)}
    if kind == "branched":
        p = sbs.BranchedFlowParams.default()
        p.patch_enabled, p.num_rays, p.ray_steps, p.num_scatterers = 0, case["rays"], case["steps"], case["scatterers"]
        flow = sbs.BranchedFlowSimulator(p)
        flow.scatterers = sbs.generate_scatterers(p, time=float(np.random.default_rng([seed, 9]).uniform(0.0, 60.0)))
        return {"case": case, "flow": flow, "film": (_modes(64, 128, seed) * 2e4).cpu().numpy(), "time": 1.5}
    pos, rad = _cluster(case, seed)
    return {"case": case, "sim": sbs.FoamSimulator(pos, rad)}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "frame":
        sim = state["sim"]
        sim.step(case["frame_dt"])
        return _fields(sim)
    if kind == "wgsl":
        sim = state["sim"]
        volumes = None
        if case["check"]:
            volumes = sim.run_checked(case["dt"], case["passes"], case["check"])
        else:
            sim.run(case["passes"])
        return [*_fields(sim), volumes]
    if kind == "cpu":
        sim = state["sim"]
        sim.step_n(case["dt"], case["steps"])
        return [_tensor(sim, sim.thickness_device())]
    if kind == "foam":
        foam, h, c = state["foam"], state["h"], state["c"]
        foam.run(case["steps"])
        for b, first, n in state["parts"]:
            N.call("sbs_foam_get_thickness", foam._h, b, ctypes.c_void_p(h.data_ptr() + 4 * first), n, N.MEM_DEVICE)
            N.call("sbs_foam_get_concentration", foam._h, b, ctypes.c_void_p(c.data_ptr() + 4 * first), n,
                   N.MEM_DEVICE)
        return [h, c]
    if kind == "spectral":
        mode = N.SPECTRAL_TC_BF16 if case["mode"] == "tc" else N.SPECTRAL_FP32
        N.call("sbs_spectral_rgb", _dev(state["t"]), _dev(state["c"]), _dev(state["nf"]), case["n"],
               N.ptr(state["wl"]), case["nl"], N.ptr(state["cmf"]), mode, _dev(state["rgb"]), N.MEM_DEVICE,
               ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        return [state["rgb"]]
    if kind == "train":
        net = state["net"]
        losses = net.train(8, case["iters"], batch=case["batch"], lr=1e-3, seed=state["seed"])
        return [losses, net.params]
    if kind == "rollout":
        sim = state["sim"]
        stats = state["net"].rollout(sim, case["passes"], check_every=case["every"], tol=1.0, mode="fused")
        return [_tensor(sim, sim.current_thickness_buffer()), stats["surrogate"], stats["failed_checks"]]
    if kind == "shade":
        return sbs.render_frame(state["uniform"], state["camera"], case["width"], case["height"], lut=state["lut"])
    if kind == "branched":
        return state["flow"].step(state["film"], state["time"])
    sim = state["sim"]
    sim.step(case["dt"], case["steps"])
    b = sim.bubbles()
    return [b["position"], b["velocity"], b["ids"], sim.connection_count()]


# --- the work a pass cannot do without --------------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind in ("frame", "wgsl"):
        cells = case["nt"] * case["np"]
        # per cell and pass: two five-point operators, the gravity term, two updates (34); the
        # Marangoni term adds the surfactant's gradient and its two couplings (17)
        ops = 34 + (17 if case.get("marangoni") else 0)
        return {"bytes": 16.0 * cells, "flops": float(ops) * cells * case["passes"]}
    if kind == "cpu":
        # the five-point operator over value and remainder, the gravity term, a compensated update
        cells = case["nt"] * case["np"]
        return {"bytes": 16.0 * cells, "flops": 38.0 * cells * case["steps"]}
    if kind == "foam":
        res, _ = _foam_bubbles(case)
        cells = float(sum(2 * int(r) * int(r) for r in res))
        return {"bytes": 16.0 * cells, "flops": 34.0 * cells * case["steps"]}
    if kind == "spectral":
        # per wavelength: a phase, its cosine, the Airy quotient, three multiply-adds
        return {"bytes": 24.0 * case["n"], "flops": 16.0 * case["n"] * case["nl"]}
    if kind == "train":
        cells = case["nt"] * case["np"] * case["batch"]
        return {"bytes": 12.0 * cells * case["iters"], "flops": 131e3 * cells * case["iters"]}
    if kind == "rollout":
        cells = case["nt"] * case["np"]
        intervals = case["passes"] // 64
        checks = -(-intervals // case["every"])
        return {"bytes": 12.0 * cells, "flops": cells * (46656.0 * intervals + 34.0 * 64 * checks)}
    if kind == "shade":
        # five simplex evaluations and the table look-up where the bubble is (about half the frame)
        px = case["width"] * case["height"]
        return {"bytes": 4.0 * px, "flops": 1000.0 * px}
    if kind == "branched":
        # per ray and step: the position, four samples, about 72 nearby scatterers
        return {"bytes": 512 * 256 * 8.0, "flops": 900.0 * case["rays"] * case["steps"]}
    # per bubble and step: about 700 neighbours in range at 20 operations
    return {"bytes": 64.0 * case["n"], "flops": 14000.0 * case["n"] * case["steps"]}


# --- the same in 64 bits ------------------------------------------------------------------------------
def _five_point(x, b, e, f):
    """Rows 1 .. nt-2 of F (phi curvature) + E (theta slope) + b (theta curvature); phi periodic."""
    c = x[1:-1]
    lap = f * (torch.roll(c, -1, 1) + torch.roll(c, 1, 1) - 2 * c)
    return lap + e * (x[2:] - x[:-2]) + b * (x[2:] + x[:-2] - 2 * c)


def _rows(nt, np_, floor):
    th = torch.arange(1, nt - 1, dtype=torch.float64, device="cuda")[:, None] * (math.pi / (nt - 1))
    dth, dph = math.pi / (nt - 1), 2.0 * math.pi / np_
    s = torch.sin(th)
    ss = s.clamp_min(floor)
    return s, 1.0 / dth**2, torch.cos(th) / ss / (2.0 * dth), 1.0 / (ss * dph) ** 2, ss, dth, dph


def _exact_wgsl(h, c, passes, dt, radius, marangoni=False, check=0):
    h, c = h.double(), c.double()
    nt, np_ = h.shape
    s, b, e, f, ss, dth, dph = _rows(nt, np_, 1e-4)
    p = sbs.DrainageParams.default()
    grav = -p.density * p.gravity / (3.0 * p.viscosity) * s
    d, ds = p.diffusion_coeff / radius**2, p.surfactant_diffusion / radius**2
    w = torch.sin(torch.arange(nt, dtype=torch.float64, device="cuda") * dth) * (radius**2 * dth * dph)
    volumes = []
    for k in range(passes):
        hi, ci = h[1:-1], c[1:-1]
        lap = _five_point(h, b, e, f)
        dh, dc = d * lap + grav * hi**3, ds * _five_point(c, b, e, f)
        if marangoni:
            gt = (c[2:] - c[:-2]) / (2.0 * dth * radius)
            gp = (torch.roll(ci, -1, 1) - torch.roll(ci, 1, 1)) / (2.0 * dph * radius * ss)
            dh = dh + p.marangoni_coeff * p.gamma_reduction * torch.sqrt(gt * gt + gp * gp) * hi * hi
            dc = dc + 0.001 * lap * ci
        thin = hi < p.critical_thickness
        h2, c2 = h.clone(), c.clone()
        h2[1:-1] = torch.where(thin, hi, (hi + dt * dh).clamp_min(0.0))
        c2[1:-1] = torch.where(thin, ci, (ci + dt * dc).clamp(0.0, 1.0))
        h, c = h2, c2
        if check and (k + 1) % check == 0:
            volumes.append(float((h.sum(1) * w).sum()))
    return h, c, np.array(volumes)


def _exact_cpu(h, steps, dt):
    h = h.double()
    nt, np_ = h.shape
    s, b, e, f, _, dth, dph = _rows(nt, np_, 1e-10)
    grav, d = -1000.0 * 9.81 / (3.0 * 0.001) * s, DIFFUSION / RADIUS**2
    theta = torch.arange(nt, dtype=torch.float64, device="cuda")[:, None] * dth
    phi = torch.arange(np_, dtype=torch.float64, device="cuda")[None, :] * dph
    fronts, spawn, time = [], 0.5, 0.0
    for _ in range(steps):
        hi = h[1:-1]
        dh = d * _five_point(h, b, e, f) + grav * hi**3
        new = torch.where(hi < CRIT_CPU, hi, (hi + dt * dh).clamp_min(0.0))
        h = torch.cat([new[:1].mean().expand(1, np_), new, new[-1:].mean().expand(1, np_)])
        spawn -= dt
        if spawn <= 0.0:  # a marginal-regeneration front starts at the equator
            fronts.append([abs(math.sin(time * 7.89 + 1.23)) * 2 * math.pi, 0.3 + abs(math.sin(time * 3.21)) * 0.4,
                           0.05 + abs(math.cos(time * 5.67)) * 0.05, 0.0])
            fronts = fronts[-8:]
            spawn = 2.0 * (0.5 + abs(math.sin(time * 12.345)))
        for q in fronts:
            q[3] = min(q[3] + q[2] * dt, math.pi / 2)
        fronts = [q for q in fronts if q[3] < math.pi / 2 * 0.95]
        if fronts:
            inside = torch.zeros((nt, np_), dtype=torch.bool, device="cuda")
            for centre, width, _, extent in fronts:
                gap = (phi - centre).abs()
                gap = torch.where(gap > math.pi, 2 * math.pi - gap, gap)
                inside |= ((theta - math.pi / 2).abs() <= extent) & (gap < width / 2)
            h = torch.where(inside, h * (1.0 - (1.0 - 0.85) * 0.5 * dt), h)
        time += dt
    return h


def _exact_spectral(case, seed):
    t, c, nf, wl, cmf = _spectral_inputs(case, seed)
    m = torch.as_tensor(cmf, device="cuda").double()
    lam = torch.as_tensor(wl, device="cuda").double()
    out = []
    for a in range(0, case["n"], 1 << 18):
        ti, ci, ni = (x[a : a + (1 << 18)].double()[:, None] for x in (t, c, nf))
        ct = torch.sqrt((1.0 - (1.0 - ci * ci).clamp_min(0.0) / (ni * ni)).clamp_min(0.0))
        rs = (ci - ni * ct) / (ci + ni * ct).clamp_min(1e-4)
        rp = (ni * ci - ct) / (ni * ci + ct).clamp_min(1e-4)
        r = (rs * rs + rp * rp) * 0.5
        finesse = 4.0 * r / (1.0 - r).clamp_min(0.001) ** 2
        s2 = torch.cos(2.0 * math.pi * ni * ti * ct / lam) ** 2
        out.append((finesse * s2 / (1.0 + finesse * s2)) @ m)
    return torch.cat(out)


def _exact_cluster(case, seed):
    pos, rad = (torch.as_tensor(x, device="cuda").double() for x in _cluster(case, seed))
    vel = torch.zeros_like(pos)
    p = sbs.FoamPhysics.default()
    g = torch.tensor(list(p.gravity), dtype=torch.float64, device="cuda")
    area = 4.0 * math.pi * rad**2
    mass = area * 500e-9 * p.density
    net = (mass * g.norm() - 4.0 / 3.0 * math.pi * rad**3 * 1.2 * g.norm()).clamp_min(0.0)
    rows = max(1, (1 << 25) // case["n"])
    for _ in range(case["steps"]):
        force = (g / g.norm()) * net[:, None] - vel * (6.0 * math.pi * p.viscosity * rad)[:, None]
        for a in range(0, case["n"], rows):
            delta = pos[None, :] - pos[a : a + rows, None]
            dist = delta.norm(dim=2)
            radii = rad[None, :] + rad[a : a + rows, None]
            apart = dist >= 1e-6
            pull = torch.where((dist < 3 * radii) & (dist > radii),
                               p.van_der_waals_strength * rad[None, :] * rad[a : a + rows, None] / dist**2, 0.0)
            pull = pull - p.repulsion_stiffness * (radii - dist).clamp_min(0.0) ** 1.5
            pull = pull + torch.where((dist < 1.2 * radii) & (dist > 0.95 * radii), 2.0 * (1.2 * radii - dist), 0.0)
            pull = torch.where(apart, pull / dist, 0.0)
            force[a : a + rows] += (delta * pull[:, :, None]).sum(1)
        vel = (vel + force / mass.clamp_min(1e-9)[:, None] * case["dt"]) * p.damping
        speed = vel.norm(dim=1, keepdim=True)
        vel = torch.where(speed > 0.1, vel * (0.1 / speed), vel)
        pos = pos + vel * case["dt"]
    return pos, vel


def exact(case, seed):
    """What run() returns on these inputs, from the definitions in 64 bits. None: bytes and counts
    (the frame, the rays), the BF16 network (its rounded activations are part of its definition), a
    run with an unstable dt, or more than the time there is."""
    kind = case["kind"]
    if kind == "frame":
        dt = sbs.DrainageParams.default().dt  # every pass of a frame is one of the uniform's dt
        if not is_stable({**case, "dt": dt}):
            return None
        h, c, _ = _exact_wgsl(_modes(case["nt"], case["np"], seed), _surfactant(case["nt"], case["np"], seed),
                              case["passes"], dt, RADIUS)
        return [h, c]
    if kind == "wgsl":
        if not is_stable(case):
            return None
        h, c, v = _exact_wgsl(_modes(case["nt"], case["np"], seed), _surfactant(case["nt"], case["np"], seed),
                              case["passes"], case["dt"], RADIUS, case["marangoni"], case["check"])
        return [h, c, v if case["check"] else None]
    if kind == "cpu":
        return [_exact_cpu(_modes(case["nt"], case["np"], seed), case["steps"], case["dt"])]
    if kind == "foam":
        if case["bubbles"] * case["steps"] > 12000:
            return None
        res, rad = _foam_bubbles(case)
        dt = _foam_dt(res, rad)
        h, c = _foam_fields(case, res, seed)
        at, hs, cs = 0, [], []
        for r, a in zip(res, rad):
            n = 2 * int(r) * int(r)
            x, y, _ = _exact_wgsl(h[at : at + n].view(int(r), -1), c[at : at + n].view(int(r), -1), case["steps"], dt,
                                  float(a))
            hs.append(x.reshape(-1))
            cs.append(y.reshape(-1))
            at += n
        return [torch.cat(hs), torch.cat(cs)]
    if kind == "spectral":
        return [_exact_spectral(case, seed)]
    if kind == "cluster":
        if case["n"] ** 2 * case["steps"] > 4e10:
            return None
        pos, vel = _exact_cluster(case, seed)
        return [pos, vel, None, None]
    return None
