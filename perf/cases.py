"""The workloads that this framework's speed is measured on, and the same results in plain 64-bit torch.

Each case is one call (or one forward and backward) that a user's program makes through the public entry
points: `runtime.trace` on a packed grid, `propagator.solve` on host arrays, `runtime.pack_grid`,
`adjoint.detector_image` and its backward, `diagnostics` on a trace's Jones vectors, and a batch of jobs
through `serving.RayServer`. Fields, wavelength, plasma and beams are those of the benchmark
configurations: a 5 mm cube probed at 532 nm, a sinusoidal slab (1e18 cm^-3), a parabolic trough
(5e18 cm^-3) or a turbulent box (1e19 cm^-3, 20 % RMS, Te = 20 eV, Z = 1).

`exact` integrates the same steps (fourth-order Runge-Kutta-Nystrom or classical RK4, steps cut at the grid's
faces, straight lines outside) in FP64 torch from the inputs alone.
"""
import math

import numpy as np
import torch

from sloth_b200 import adjoint, runtime
from sloth_b200.core import physics
from sloth_b200.core.domain import ScalarDomain
from sloth_b200.core.propagator import solve
from sloth_b200.processing import diagnostics
from sloth_b200.serving import RayServer

L = 5e-3              # box (m)
LWL = 532e-9          # probe wavelength (m)
TE, ZION = 20.0, 1.0  # plasma of the inverse-bremsstrahlung cases
C = 299792458.0
DEV = "cuda"


# ---------------------------------------------------------------------------
# Cases
# ---------------------------------------------------------------------------
def _trace(field, nx, ny, nz, rays, *, precision="f32", ib=False, axis=2, saves=1, state=False, plane=True,
           integrator="rkn", beam="gaussian", waist=1.5e-3, jitter=0.0):
    return {"kind": "trace", "field": field, "nx": nx, "ny": ny, "nz": nz, "rays": rays, "precision": precision,
            "ib": ib, "axis": axis, "saves": saves, "state": state, "plane": plane, "integrator": integrator,
            "beam": beam, "waist": waist, "jitter": jitter}


def listed():
    return [
        # the small configuration: 1e4 rays through the 128^3 slab, where launches and latency count
        dict(_trace("sinusoid", 128, 128, 128, 10_000, waist=1e-3), name="trace slab 128 1e4"),
        # the trough: a 1000 x 1000 launch lattice with 1 mrad of jitter, projected to the far face
        dict(_trace("trough", 256, 256, 256, 1_000_000, beam="lattice", jitter=1e-3), name="trace trough 256 1e6"),
        # a request of the serving stream's median size, ragged, with transmission
        dict(_trace("kolmogorov", 192, 192, 192, 217_003, ib=True), name="trace turbulent 192 2e5"),
        # the headline: 1e7 rays through the 512^3 turbulent box, with transmission
        dict(_trace("kolmogorov", 512, 512, 512, 10_000_000, ib=True), name="trace turbulent 512 1e7"),
        # the all-FP64 tracer that FP32 results are validated against
        dict(_trace("kolmogorov", 256, 256, 256, 400_000, ib=True, precision="f64"), name="trace turbulent 256 4e5 f64"),
        # a depth scan along x of a box with three different odd extents: 11 saves with the rays' states
        dict(_trace("kolmogorov", 201, 97, 143, 300_007, ib=True, axis=0, saves=11, state=True, plane=False),
             name="trace depths x 3e5"),
        # the drop-in call on host arrays: upload, pack, trace, results in numpy
        {"kind": "solve", "field": "kolmogorov", "n": 256, "rays": 1_000_000, "ib": True, "name": "solve host 256 1e6"},
        # a new density on the device made ready for tracing, as each frame of a simulation is
        {"kind": "pack", "nx": 512, "ny": 512, "nz": 512, "dtype": "f32", "precision": "f32", "name": "pack 512"},
        # one iteration of fitting a density to a detector image
        {"kind": "image", "n": 128, "rays": 1_000_000, "steps": 400, "ckpt": 20, "npx": 256, "sigma": 2.0,
         "precision": "f32", "name": "image grad 128 1e6"},
        # the same while a fit is set up: a coarse box, few rays, ragged checkpoint segments
        {"kind": "image", "n": 61, "rays": 30_011, "steps": 150, "ckpt": 13, "npx": 97, "sigma": 1.5,
         "precision": "f32", "name": "image grad 61 3e4"},
        # a trace's rays through a shadowgraphy telescope onto the full camera chip
        {"kind": "optics", "rays": 10_000_000, "dtype": "f32", "chain": "shadow", "bin_scale": 1, "weights": False,
         "name": "shadowgram 1e7"},
        # a burst of requests of mixed grids and ray counts through the request server
        {"kind": "serve", "jobs": 8, "median": 200_000, "name": "serve 8 jobs"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    k = rng.random()
    if k < 0.5:
        f64 = rng.random() < 0.2
        field = rng.choice(["sinusoid", "trough", "kolmogorov", "kolmogorov"])
        if rng.random() < 0.6:
            nx = ny = nz = _log_int(rng, 48, 300 if f64 else 512)
        else:
            nx, ny, nz = (_log_int(rng, 40, 300) for _ in range(3))
        axis = 2 if rng.random() < 0.7 else rng.randrange(2)
        saves = 1 if rng.random() < 0.7 else rng.randint(2, 12)
        along = (nx, ny, nz)[axis]
        most = (1.5e9 if f64 else 8e9) / (2.0 * along * max(1.0, max(nx, ny, nz) / along))
        return _trace(field, nx, ny, nz, _log_int(rng, 3_000, min(8e6 / max(1, saves / 3), most)),
                      precision="f64" if f64 else "f32", ib=field == "kolmogorov" and rng.random() < 0.7, axis=axis,
                      saves=saves, state=saves > 1 and rng.random() < 0.5, plane=saves == 1 and rng.random() < 0.6,
                      integrator="rk4" if rng.random() < 0.1 else "rkn",
                      waist=rng.choice([1e-3, 1.5e-3, 3e-3]), jitter=rng.choice([0.0, 0.0, 1e-3, 5e-3]))
    if k < 0.6:
        return {"kind": "solve", "field": rng.choice(["sinusoid", "kolmogorov"]), "n": _log_int(rng, 64, 300),
                "rays": _log_int(rng, 1e4, 2e6), "ib": rng.random() < 0.5}
    if k < 0.7:
        return {"kind": "pack", "nx": _log_int(rng, 40, 450), "ny": _log_int(rng, 40, 450), "nz": _log_int(rng, 40, 450),
                "dtype": rng.choice(["f32", "f32", "f64"]), "precision": rng.choice(["f32", "f32", "f64"])}
    if k < 0.85:
        return {"kind": "image", "n": _log_int(rng, 32, 160), "rays": _log_int(rng, 5e3, 1e6), "steps": rng.randint(80, 400),
                "ckpt": rng.randint(8, 32), "npx": rng.randint(48, 300), "sigma": rng.choice([1.0, 1.5, 2.0, 3.0]),
                "precision": "f64" if rng.random() < 0.15 else "f32"}
    if k < 0.95:
        return {"kind": "optics", "rays": _log_int(rng, 1e4, 1e7), "dtype": rng.choice(["f32", "f32", "f64"]),
                "chain": rng.choice(["shadow", "schlieren", "refracto"]), "bin_scale": rng.choice([1, 2, 5, 10]),
                "weights": rng.random() < 0.4}
    return {"kind": "serve", "jobs": rng.randint(2, 10), "median": _log_int(rng, 5e4, 4e5)}


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _gen(seed, salt):
    return torch.Generator(device=DEV).manual_seed((int(seed) * 1_000_003 + salt) % (1 << 62))


def _field(kind, shape, seed):
    """Density (m^-3, float32, CUDA) of the given shape over the box."""
    g = _gen(seed, 1)
    x = torch.linspace(-L / 2, L / 2, shape[0], dtype=torch.float64, device=DEV)
    shift = float(torch.rand((), generator=g, device=DEV, dtype=torch.float64))
    if kind == "sinusoid":
        prof = 1e24 * (1.0 + 0.1 * torch.sin(2 * math.pi * (x / 0.5e-3 + shift)))
        return prof.float()[:, None, None].expand(shape).contiguous()
    if kind == "trough":
        prof = 5e24 * (1.0 + ((x + 1e-4 * (shift - 0.5)) / 2e-3) ** 2)
        return prof.float()[:, None, None].expand(shape).contiguous()
    white = torch.randn(shape, generator=g, device=DEV)
    spec = torch.fft.rfftn(white)
    del white
    hs = [L / (n - 1) for n in shape]
    k2 = 0
    for a in range(3):
        f = torch.fft.rfftfreq(shape[a], d=hs[a], device=DEV) if a == 2 else torch.fft.fftfreq(shape[a], d=hs[a], device=DEV)
        k2 = k2 + ((2 * math.pi * f) ** 2).reshape([-1 if b == a else 1 for b in range(3)])
    k = k2.sqrt_()
    kmin = 2 * math.pi / L
    amp = torch.where((k >= kmin) & (k <= math.pi / max(hs)), k.clamp_min(kmin) ** (-11.0 / 6.0), 0.0)
    spec *= amp
    del k, k2, amp
    f = torch.fft.irfftn(spec, s=shape)
    del spec
    f -= f.mean()
    f *= 0.2 / f.square().mean().sqrt()
    return (1e25 * (1.0 + f)).clamp_min_(0.0).contiguous()


def _rays(n, axis, seed, beam="gaussian", waist=1.5e-3, jitter=0.0):
    """Collimated rays (6, n), FP64 on the device, entering the box at its near face along `axis`."""
    g = _gen(seed, 2)
    r = torch.zeros((6, n), dtype=torch.float64, device=DEV)
    t = [a for a in range(3) if a != axis]
    if beam == "lattice":
        side = math.isqrt(n - 1) + 1
        i = torch.arange(n, device=DEV)
        step = 0.8 * L / max(1, side - 1)
        r[t[0]] = -0.4 * L + step * (i // side)
        r[t[1]] = -0.4 * L + step * (i % side)
    else:
        for a in t:
            r[a] = torch.randn(n, generator=g, device=DEV, dtype=torch.float64) * (waist / 2)
    r[axis] = -L / 2
    s = [torch.zeros(n, dtype=torch.float64, device=DEV)] * 2
    if jitter:
        s = [torch.sin(torch.randn(n, generator=g, device=DEV, dtype=torch.float64) * jitter) for _ in t]
    r[3 + t[0]], r[3 + t[1]] = C * s[0], C * s[1]
    r[3 + axis] = C * torch.sqrt(1.0 - s[0] ** 2 - s[1] ** 2)
    return r


def _geom(shape):
    return (-L / 2,) * 3, tuple(L / (n - 1) for n in shape)


def _schedule(shape, saves, geom=None):
    return runtime.schedule_times([math.sqrt(8.0) * L] if saves == 1 else np.linspace(0.0, L, saves), (geom or _geom(shape))[1])


def _domain_geom(n):
    """Origin and spacing of a ScalarDomain, whose coordinates are float32."""
    e = float(np.float32(L / 2))
    return (-e,) * 3, (2 * e / (n - 1),) * 3


def _trace_inputs(case, seed):
    shape = (case["nx"], case["ny"], case["nz"])
    dt = torch.float32 if case["precision"] == "f32" else torch.float64
    ne = _field(case["field"], shape, seed)
    rays = _rays(case["rays"], case["axis"], seed, case["beam"], case["waist"], case["jitter"]).to(dt)
    return shape, ne, rays


def _solve_inputs(case, seed):
    shape = (case["n"],) * 3
    return shape, _field(case["field"], shape, seed), _rays(case["rays"], 2, seed).float()


def _pack_inputs(case, seed):
    ne = _field("kolmogorov", (case["nx"], case["ny"], case["nz"]), seed)
    return ne if case["dtype"] == "f32" else ne.double()


def _image_spec(case):
    return adjoint.box_detector(L, n_px=case["npx"], sigma_px=case["sigma"], n_steps=case["steps"], ckpt_every=case["ckpt"])


def _image_inputs(case, seed):
    dt = torch.float32 if case["precision"] == "f32" else torch.float64
    ne = _field("kolmogorov", (case["n"],) * 3, seed).to(dt)
    rays = _rays(case["rays"], 2, seed).to(dt)
    # the image to fit: the undeflected beam with a fringe pattern
    m = case["npx"]
    u = (torch.arange(m, dtype=torch.float64, device=DEV) + 0.5) * (L / m) - L / 2
    s = 0.75e-3
    g = torch.exp(-0.5 * (u / s) ** 2) * (L / m / s / math.sqrt(2 * math.pi))
    fringe = 1.0 + 0.2 * torch.cos(2 * math.pi * (u / 0.4e-3 + seed % 7 / 7))
    return ne, rays, (case["rays"] * (g * fringe)[:, None] * g[None, :]).to(dt)


_CHAINS = {"shadow": (diagnostics.Shadowgraphy, "two_lens_solve"), "schlieren": (diagnostics.Schlieren, "DF_solve"),
           "refracto": (diagnostics.Refractometry, "incoherent_solve")}


def _optics_inputs(case, seed):
    """Jones vectors (4, N) of a deflected beam at the object plane (m, rad), and weights."""
    g = _gen(seed, 3)
    n = case["rays"]
    dt = torch.float32 if case["dtype"] == "f32" else torch.float64
    rf = torch.randn((4, n), generator=g, device=DEV, dtype=torch.float64)
    rf[0::2] *= 2.5e-3
    rf[1::2] *= 6e-3
    w = torch.rand(n, generator=g, device=DEV, dtype=torch.float64).to(dt) if case["weights"] else None
    return rf.to(dt), w


def _serve_inputs(case, seed):
    """(field, n, rays) of each job: sinusoid and turbulent boxes of the stream's sizes, lognormal ray counts."""
    r = np.random.RandomState(case["jobs"] * 1009 + case["median"] % 1009)   # sizes belong to the case, not the seed
    jobs = []
    for j in range(case["jobs"]):
        n = int(r.choice([64, 128, 192, 256]))
        kind = "kolmogorov" if r.rand() < 0.5 else "sinusoid"
        rays = int(np.clip(case["median"] * math.exp(r.randn()), 1e4, 2e6))
        jobs.append((kind, n, rays, _field(kind, (n,) * 3, seed + 17 * j), _rays(rays, 2, seed + 17 * j).float()))
    return jobs


class _Server(RayServer):
    def __del__(self):
        self.close()


def prepare(case, seed):
    k = case["kind"]
    if k == "trace":
        shape, ne, rays = _trace_inputs(case, seed)
        origin, spacing = _geom(shape)
        grid = runtime.pack_grid(ne, origin, spacing, physics.omega_of(LWL), precision=case["precision"])
        kw = dict(axis=case["axis"], project=case["plane"], plane=L / 2, want_state=case["state"],
                  integrator=case["integrator"], inv_brems=case["ib"])
        if case["ib"]:
            kw.update(Te=TE, Z=ZION)
        return {"kind": k, "grid": grid, "rays": rays, "sched": _schedule(shape, case["saves"]), "kw": kw}
    if k == "solve":
        shape, ne, rays = _solve_inputs(case, seed)
        extra = dict(inv_brems=True, Te=TE, Z=ZION) if case["ib"] else {}
        dom = ScalarDomain(L, case["n"], ne=ne.cpu().numpy(), probing_direction="z", **extra)
        return {"kind": k, "domain": dom, "rays": rays.cpu().numpy()}
    if k == "pack":
        ne = _pack_inputs(case, seed)
        return {"kind": k, "ne": ne, "geom": _geom(tuple(ne.shape)), "precision": case["precision"]}
    if k == "image":
        ne, rays, target = _image_inputs(case, seed)
        return {"kind": k, "ne": ne.requires_grad_(True), "rays": rays, "target": target, "spec": _image_spec(case),
                "geom": _geom((case["n"],) * 3), "precision": case["precision"]}
    if k == "optics":
        rf, w = _optics_inputs(case, seed)
        return {"kind": k, "rf": rf, "w": w, "chain": case["chain"], "bin_scale": case["bin_scale"]}
    jobs = _serve_inputs(case, seed)
    need = sum(16 * n ** 3 + 110 * rays + (2 << 20) for _, n, rays, _, _ in jobs)
    return {"kind": k, "server": _Server(need + (64 << 20)), "jobs": jobs}


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------
def run(state):
    k = state["kind"]
    if k == "trace":
        o = runtime.trace(state["grid"], state["rays"], state["sched"], **state["kw"])
        return {key: v for key, v in o.items() if key != "total_steps"}   # the sum of "steps"
    if k == "solve":
        rf, amp, _ = solve(state["rays"], state["domain"], L, lwl=LWL, detector_plane=L / 2, verbose=False)
        return {"rf": rf, "amp": amp}
    if k == "pack":
        g = runtime.pack_grid(state["ne"], *state["geom"], physics.omega_of(LWL), precision=state["precision"])
        return {"grid": g.data, "q_max": g.q_max, "q_min": g.q_min, "ne_max": g.ne_max}
    if k == "image":
        ne = state["ne"]
        ne.grad = None
        img = adjoint.detector_image(ne, state["rays"], state["spec"], origin=state["geom"][0],
                                     spacing=state["geom"][1], lwl=LWL, precision=state["precision"])
        (img - state["target"]).square().sum().backward()
        return {"image": img.detach(), "grad": ne.grad}
    if k == "optics":
        cls, chain = _CHAINS[state["chain"]]
        d = cls(state["rf"], weights=state["w"], verbose=False)
        getattr(d, chain)()
        d.histogram(bin_scale=state["bin_scale"])
        return {"H": d.H}
    server, jobs = state["server"], state["jobs"]
    live = []
    for j, (kind, n, _, ne, rays) in enumerate(jobs):
        ib = kind == "kolmogorov"
        live.append(server.submit(j, ne, *_geom((n,) * 3), (n,) * 3, rays, lwl=LWL, detector_plane=L / 2, inv_brems=ib,
                                  Te=TE, Z=ZION))
    out = server.run_until_done(live)
    res = {}
    for j, job in enumerate(live):
        res[str(j)] = {key: v for key, v in out[job.id].items() if key != "total_steps"}
        server.release(job)
    return res


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------
def _trace_work(shape, axis, rays, *, ib, saves=1, state=False, real=4, rk4=False, waist=1.5e-3, lattice=False):
    steps = rays * 2.0 * (shape[axis] - 1) * max(1.0, (max(shape) - 1) / (shape[axis] - 1))
    # 7 multiply-adds per channel and sample, and about 45 operations a step for the sums
    flops = steps * ((4 if rk4 else 3) * 14 * (5 if ib else 4) + 45)
    # the part of the grid that the beam crosses
    across = 0.64 if lattice else min(1.0, math.pi * (1.25 * waist / L) ** 2)
    grid = across * 4 * real * shape[0] * shape[1] * shape[2]
    per_ray = 6 * real + 5 + saves * (4 * real + 8 + (real if ib else 0) + (6 * real if state else 0))
    return {"bytes": min(grid, rays * shape[axis] * 16.0 * real) + rays * per_ray, "flops": flops}


def work(case):
    k = case["kind"]
    if k == "trace":
        return _trace_work((case["nx"], case["ny"], case["nz"]), case["axis"], case["rays"], ib=case["ib"],
                           saves=case["saves"], state=case["state"], real=4 if case["precision"] == "f32" else 8,
                           rk4=case["integrator"] == "rk4", waist=case["waist"], lattice=case["beam"] == "lattice")
    if k == "solve":
        n = case["n"]
        w = _trace_work((n,) * 3, 2, case["rays"], ib=case["ib"])
        return {"bytes": w["bytes"] + 4.0 * n ** 3, "flops": w["flops"]}
    if k == "pack":
        v = case["nx"] * case["ny"] * case["nz"]
        return {"bytes": v * ((4 if case["dtype"] == "f32" else 8) + (16 if case["precision"] == "f32" else 32)),
                "flops": 15 * v}
    if k == "image":
        n, real = case["n"], 4 if case["precision"] == "f32" else 8
        steps = 0.975 * case["rays"] * case["steps"]
        # the forward's samples and step, the same again for the adjoint's states, and about twice that for their reverse
        return {"bytes": 2.0 * real * n ** 3 + 6.0 * real * case["rays"] + 2.0 * real * case["npx"] ** 2,
                "flops": steps * 4 * (3 * 14 * 3 + 40)}
    if k == "optics":
        real = 4 if case["dtype"] == "f32" else 8
        nx, ny = 3448 // case["bin_scale"], 2574 // case["bin_scale"]
        return {"bytes": case["rays"] * real * (5 if case["weights"] else 4) + 8.0 * nx * ny, "flops": 40.0 * case["rays"]}
    r = np.random.RandomState(case["jobs"] * 1009 + case["median"] % 1009)
    w = {"bytes": 0.0, "flops": 0.0}
    for _ in range(case["jobs"]):
        n = int(r.choice([64, 128, 192, 256]))
        ib = r.rand() < 0.5
        t = _trace_work((n,) * 3, 2, int(np.clip(case["median"] * math.exp(r.randn()), 1e4, 2e6)), ib=ib)
        w = {m: w[m] + t[m] for m in w}
    return w


def tolerance(case):
    k = case["kind"]
    if k in ("trace", "solve", "serve"):
        if case.get("precision") == "f64":
            return {"rel": 1e-11, "max": 1e-6, "differ": 1e-5}
        # 1e-7 over all rays; rays that graze a side face leave it early or late by their rounding, the more of them the
        # wider the beam (against `exact`: 9e-8, 2e-7 and 2e-5 at waists of 1, 1.5 and 3 mm)
        wide = case.get("waist", 1.5e-3)
        return {"rel": 8e-5 if wide > 2e-3 else 1e-6 if wide > 1.2e-3 else 4e-7,
                "max": 8e-2 if wide > 2e-3 else 5e-3 if wide > 1.2e-3 else 1e-3, "differ": 1e-3}
    if k == "pack":
        return {"rel": 1e-7, "max": 1e-6} if case["precision"] == "f32" else {"rel": 1e-14, "max": 1e-12}
    if k == "image":
        return {"rel": 1e-5, "max": 1e-3} if case["precision"] == "f32" else {"rel": 1e-11, "max": 1e-8}
    return {"rel": 1e-12, "max": 1e-11}


# ---------------------------------------------------------------------------
# The same in 64 bits
# ---------------------------------------------------------------------------
NRL = 5.64e4            # omega_pe = NRL sqrt(ne [cm^-3])
ALPHA = 3.14207787e-4   # nc = ALPHA omega^2
E_CHARGE, EPS0 = 1.602176634e-19, 8.8541878188e-12


def _optical_constants():
    omega = 2 * math.pi * (C / LWL)
    nc = ALPHA * omega ** 2
    return omega, nc, NRL ** 2 * nc * 1e-6 / omega ** 2


def _grad3(q):
    """Differences per cell along each axis: central inside, one-sided on the faces."""
    out = []
    for a in range(3):
        n = q.shape[a]
        d = torch.empty_like(q)
        if n > 2:
            d.narrow(a, 1, n - 2).copy_(0.5 * (q.narrow(a, 2, n - 2) - q.narrow(a, 0, n - 2)))
        d.narrow(a, 0, 1).copy_(q.narrow(a, 1, 1) - q.narrow(a, 0, 1))
        d.narrow(a, n - 1, 1).copy_(q.narrow(a, n - 1, 1) - q.narrow(a, n - 2, 1))
        out.append(d)
    return out


def _packed(ne):
    """(n - 1, dq/du, dq/dv, dq/dw) in FP64."""
    _, nc, ope2 = _optical_constants()
    q = ne.double() * (1.0 / nc)
    x = ope2 * q
    return torch.stack([-x / (1.0 + (1.0 - x).clamp_min(0.0).sqrt())] + _grad3(q), dim=-1)


def _kappa():
    omega, nc, ope2 = _optical_constants()
    kq2 = 3.1e-5 * ZION * (nc * 1e-6 / omega) ** 2 * TE ** -1.5
    b_min = ZION * E_CHARGE / (4 * math.pi * EPS0 * TE)
    return kq2, math.log(4.19e5 * math.sqrt(TE) / (omega * b_min)), ope2


class _Tracer:
    """The trace of one ray set, one step of every live ray at a time."""

    def __init__(self, ne, rays, sched, *, axis, plane, ib, rk4=False, geom=None):
        self.shape, self.sched, self.axis, self.plane, self.ib, self.rk4 = tuple(ne.shape), sched, axis, plane, ib, rk4
        self.vol = _packed(ne)
        if ib:
            _, clw, ope2 = _kappa()
            q = ne.double() * (1.0 / _optical_constants()[1])
            x = ope2 * q
            cl = torch.where(x > 1, (clw - 0.5 * torch.log(x.clamp_min(1.0))).clamp_min(2.0), max(2.0, clw))
            self.vol = torch.cat([self.vol, (q * q * cl)[..., None]], dim=-1)
        self.vol = self.vol.reshape(-1, self.vol.shape[-1]).contiguous()
        col = lambda v: torch.tensor(v, dtype=torch.float64, device=DEV)[:, None]  # noqa: E731
        self.o, self.h = (col(v) for v in geom or _geom(self.shape))
        self.lim = col([n - 1.0 for n in self.shape])
        self.S = -0.5 * (sched.dtau / self.h) ** 2
        self.rays = rays.double()

    def sample(self, p, clamp):
        """(gradient accelerations (3, N), n - 1, kappa) at p (3, N); zero outside."""
        p = torch.where(clamp, torch.minimum(p.clamp_min(0.0), self.lim), p)
        inside = ((p >= 0) & (p <= self.lim)).all(0)
        i = torch.minimum(p.clamp_min(0.0).floor(), self.lim - 1)
        i = torch.where(inside, i, 0.0)
        f = torch.where(inside, p - i, 0.0)
        i = i.long()
        b = (i[0] * self.shape[1] + i[1]) * self.shape[2] + i[2]
        v = 0
        for dx in (0, 1):
            wx = f[0] if dx else 1 - f[0]
            for dy in (0, 1):
                wxy = wx * (f[1] if dy else 1 - f[1])
                for dz in (0, 1):
                    w = wxy * (f[2] if dz else 1 - f[2])
                    v = v + w[:, None] * self.vol[b + ((dx * self.shape[1] + dy) * self.shape[2] + dz)]
        v = torch.where(inside[:, None], v, 0.0).T
        return self.S * v[1:4], v[0], (v[4] if self.ib else v[0])

    def step(self, p, w, phi, clamp):
        s = lambda x: self.sample(x, clamp)  # noqa: E731
        a1, g1, k1 = s(p)
        if self.rk4:
            a2, g2, k2 = s(p + 0.5 * phi * w)
            a3, g3, k3 = s(p + 0.5 * phi * (w + 0.5 * phi * a1))
            a4, g4, k4 = s(p + phi * (w + 0.5 * phi * a2))
            dp = phi * w + phi ** 2 * (a1 + a2 + a3) / 6
            return p + dp, w + phi * (a1 + 2 * a2 + 2 * a3 + a4) / 6, phi * (g1 + 2 * g2 + 2 * g3 + g4), phi * (k1 + 2 * k2 + 2 * k3 + k4)
        a2, g2, k2 = s(p + phi * w / 2 + phi ** 2 * a1 / 8)
        a3, g3, k3 = s(p + phi * w + phi ** 2 * a2 / 2)
        return p + phi * w + phi ** 2 * (a1 + 2 * a2) / 6, w + phi * (a1 + 4 * a2 + a3) / 6, phi * (g1 + 4 * g2 + g3), phi * (k1 + 4 * k2 + k3)

    def emit(self, out, j, ids, p, w, ph, tau, drift):
        omega, _, _ = _optical_constants()
        x = self.o + (p + drift * w) * self.h
        v = w * (C * self.h / self.sched.dtau)
        t1, t2 = (a for a in range(3) if a != self.axis)
        back = (x[self.axis] - self.plane) / v[self.axis] if self.plane is not None else 0.0
        for r, a in ((0, t1), (2, t2)):
            out["jones"][j, r, ids] = x[a] - v[a] * back
            out["jones"][j, r + 1, ids] = torch.atan(v[a] / v[self.axis])
        out["state"][j, :3, ids] = x
        out["state"][j, 3:, ids] = v
        out["phase"][j, ids] = ph * (omega / C * self.sched.dtau / 6)
        if self.ib:
            out["amp"][j, ids] = torch.exp(-tau * (_kappa()[0] * self.sched.dtau / 6))

    def run(self):
        sc, n = self.sched, self.rays.shape[1]
        S = sc.n_saves
        nan = lambda *s: torch.full(s, math.nan, dtype=torch.float64, device=DEV)  # noqa: E731
        out = {"jones": nan(S, 4, n), "state": nan(S, 6, n), "phase": nan(S, n)}
        if self.ib:
            out["amp"] = nan(S, n)
        ids = torch.arange(n, device=DEV)
        p = (self.rays[:3] - self.o) / self.h
        w = self.rays[3:] * (sc.dtau / self.h / C)
        ph, tau, lag = (torch.zeros(n, dtype=torch.float64, device=DEV) for _ in range(3))
        exited = torch.zeros(n, dtype=torch.bool, device=DEV)
        check = torch.ones(n, dtype=torch.bool, device=DEV)
        save_j = 0                       # saves come at the same steps for every ray
        for t in range(sc.last_step + 1):
            gone = exited | (check & (((p < 0) & (w <= 0)) | ((p > self.lim) & (w >= 0))).any(0))
            due = save_j < S and t == sc.first_save + save_j * sc.save_every
            if due:
                self.emit(out, save_j, ids, p, w, ph, tau, lag)
                save_j += 1
            if t % 16 == 0 or due or t == sc.last_step:
                # rays that left for good: their later saves lie on straight lines
                for j in range(save_j, S):
                    late = sc.first_save + j * sc.save_every - t
                    self.emit(out, j, ids[gone], p[:, gone], w[:, gone], ph[gone], tau[gone], late + lag[gone])
                live = ~gone
                ids, p, w, ph, tau, lag = ids[live], p[:, live], w[:, live], ph[live], tau[live], lag[live]
                exited = exited[live]
                if not ids.numel() or save_j >= S:
                    break
            inside = ((p >= 0) & (p <= self.lim)).all(0)
            pn = p + w
            hi, lo = (self.lim - p) / w, -p / w
            phi = torch.where(pn > self.lim, hi, 1.0)
            phi = torch.minimum(phi, torch.where(pn < 0, lo, 1.0)).amin(0).clamp(0.0, 1.0)
            phi = torch.where(inside, phi, 1.0)
            cut = (phi < 1.0) & ~exited
            near = ((pn > self.lim - 0.02) | (pn < 0.02)).any(0)
            p1, w1, dg, dk = self.step(p, w, phi, inside & (cut | near))
            p, w = torch.where(exited, p + w, p1), torch.where(exited, w, w1)
            ph, tau = ph + torch.where(exited, 0.0, dg), tau + torch.where(exited, 0.0, dk)
            exited, lag = exited | cut, torch.where(cut, 1.0 - phi, lag)
            check = ~inside | cut | near
        return out


def _exact_trace(ne, rays, sched, *, axis=2, plane=L / 2, ib=False, rk4=False, state=False, geom=None):
    o = _Tracer(ne, rays, sched, axis=axis, plane=plane, ib=ib, rk4=rk4, geom=geom).run()
    if not state:
        o.pop("state")
    return o


class _Image:
    """The detector image and, through autograd, its gradient."""

    def __init__(self, case):
        self.case, self.n = case, case["n"]
        self.spec = _image_spec(case)
        self.h = L / (self.n - 1)
        self.S = -0.5 * (self.spec.dtau / self.h) ** 2

    def accel(self, vol, p):
        n = self.n
        inside = ((p >= 0) & (p <= n - 1)).all(0)
        i = torch.where(inside, p.detach().clamp(0, n - 2).floor(), 0.0)
        f = torch.where(inside, p - i, 0.0)
        i = i.long()
        b = (i[0] * n + i[1]) * n + i[2]
        a = 0
        for c in range(8):
            d = (c >> 2, (c >> 1) & 1, c & 1)
            w = 1.0
            for ax in range(3):
                w = w * (f[ax] if d[ax] else 1 - f[ax])
            a = a + w[:, None] * vol.index_select(0, b + ((d[0] * n + d[1]) * n + d[2]))
        return self.S * torch.where(inside[:, None], a, 0.0).T

    def segment(self, vol, p, w, m):
        for _ in range(m):
            a1 = self.accel(vol, p)
            a2 = self.accel(vol, p + w / 2 + a1 / 8)
            a3 = self.accel(vol, p + w + a2 / 2)
            p, w = p + w + (a1 + 2 * a2) / 6, w + (a1 + 4 * a2 + a3) / 6
        return p, w

    def splat(self, p, w):
        s, m = self.spec.sigma_px, self.case["npx"]
        t = ((self.spec.plane + L / 2) / self.h - p[2]) / w[2]
        pix = L / m
        img = torch.zeros(m * m, dtype=torch.float64, device=DEV)
        taps = 2 * math.ceil(4 * s) + 1
        idx, g = [], []
        for a in (0, 1):
            at = ((p[a] + t * w[a]) * self.h) / pix - 0.5
            i = torch.floor(at.detach() - 4 * s)[:, None] + 1 + torch.arange(taps, device=DEV)
            u = (i - at[:, None]).abs() / s
            x = (u - 3).clamp(0, 1)
            g.append(torch.exp(-0.5 * u * u) * (1 - x ** 3 * (10 + x * (-15 + 6 * x))) * ((i >= 0) & (i < m)))
            idx.append(i.clamp(0, m - 1).long())
        w2 = g[0][:, :, None] * g[1][:, None, :] / (2 * math.pi * s * s)
        return img.index_add(0, (idx[0][:, :, None] * m + idx[1][:, None, :]).reshape(-1), w2.reshape(-1)).reshape(m, m)

    def final(self, vol, rays, keep):
        """Final rays; with `keep`, also the states at the starts of segments of 16 steps."""
        p = (rays[:3] + L / 2) / self.h
        w = rays[3:] * (self.spec.dtau / self.h / C)
        states = []
        for k in range(0, self.spec.n_steps, 16):
            if keep:
                states.append((p, w))
            p, w = self.segment(vol, p, w, min(16, self.spec.n_steps - k))
        return p, w, states

    def run(self, ne, rays, target):
        ne = ne.double().requires_grad_(True)
        grads = _Grad.apply(ne * (1.0 / _optical_constants()[1]))
        vol = grads.detach().reshape(-1, 3).contiguous()
        chunks = rays.double().split(50_000, dim=1)
        img = 0
        with torch.no_grad():
            for r in chunks:
                img = img + self.splat(*self.final(vol, r, False)[:2])
        dimg = 2 * (img - target.double())
        gvol = torch.zeros_like(vol)
        for r in chunks:
            with torch.no_grad():
                p, w, states = self.final(vol, r, True)
            p, w = p.requires_grad_(True), w.requires_grad_(True)
            gp, gw = torch.autograd.grad(self.splat(p, w), (p, w), dimg)
            for k in reversed(range(len(states))):
                p, w = (x.detach().requires_grad_(True) for x in states[k])
                v = vol.detach().requires_grad_(True)
                q = self.segment(v, p, w, min(16, self.spec.n_steps - 16 * k))
                gp, gw, gv = torch.autograd.grad(q, (p, w, v), (gp, gw))
                gvol += gv
        grads.backward(gvol.reshape(grads.shape))
        return {"image": img, "grad": ne.grad}


class _Grad(torch.autograd.Function):
    """_grad3 stacked last, with its transpose."""

    @staticmethod
    def forward(ctx, q):
        return torch.stack(_grad3(q), dim=-1)

    @staticmethod
    def backward(ctx, g):
        out = torch.zeros(g.shape[:3], dtype=g.dtype, device=g.device)
        for a in range(3):
            d, n = g[..., a], g.shape[a]
            if n > 2:
                mid = 0.5 * d.narrow(a, 1, n - 2)
                out.narrow(a, 2, n - 2).add_(mid)
                out.narrow(a, 0, n - 2).sub_(mid)
            for i in (0, n - 1):
                e = d.narrow(a, i, 1)
                out.narrow(a, min(i + 1, n - 1), 1).add_(e)
                out.narrow(a, max(i - 1, 0), 1).sub_(e)
        return out


def _exact_optics(case, seed):
    rf, wt = _optics_inputs(case, seed)
    mm = rf.clone()
    mm[0::2] *= 1e3
    x, t, y, p = mm.double()
    Ld, R, Lx, Ly = 400.0, 25.0, 18.0, 13.5
    alive = torch.ones_like(x, dtype=torch.bool)

    def travel(d):
        nonlocal x, y
        x, y = x + d * t, y + d * p

    def lens(f1, f2):
        nonlocal t, p
        t, p = t - x / f1, p - y / f2

    def stop(bad):
        nonlocal alive
        alive = alive & ~bad

    if case["chain"] == "shadow":
        travel(Ld), stop(x * x + y * y > R * R), lens(Ld / 2, Ld / 2), travel(2 * Ld)
        stop(x * x + y * y > R * R), lens(Ld / 2, Ld / 2), travel(Ld)
    elif case["chain"] == "schlieren":
        travel(Ld), stop(x * x + y * y > R * R), lens(Ld, Ld), travel(Ld), stop(x * x + y * y < 1.0), travel(Ld)
        stop(x * x + y * y > R * R), lens(Ld, Ld), travel(Ld)
    else:
        travel(3 * Ld / 4), stop(x * x + y * y > R * R), lens(Ld / 2, Ld / 2), travel(3 * Ld / 2)
        stop((x * x > 15.0 ** 2) & (y * y > 30.0 ** 2)), stop(x * x + y * y > R * R), lens(Ld / 3, Ld / 2), travel(Ld)
    nx, ny = 3448 // case["bin_scale"], 2574 // case["bin_scale"]
    ok = alive & (x >= -Lx / 2) & (x <= Lx / 2) & (y >= -Ly / 2) & (y <= Ly / 2)
    ix = torch.bucketize(x[ok], torch.linspace(-Lx / 2, Lx / 2, nx + 1, dtype=torch.float64, device=DEV), right=True) - 1
    iy = torch.bucketize(y[ok], torch.linspace(-Ly / 2, Ly / 2, ny + 1, dtype=torch.float64, device=DEV), right=True) - 1
    H = torch.zeros(nx * ny, dtype=torch.float64, device=DEV)
    w = torch.ones(int(ok.sum()), dtype=torch.float64, device=DEV) if wt is None else wt[ok].double()
    return {"H": H.index_add_(0, iy.clamp(0, ny - 1) * nx + ix.clamp(0, nx - 1), w).reshape(ny, nx)}


def exact(case, seed):
    k = case["kind"]
    if k == "trace":
        shape = (case["nx"], case["ny"], case["nz"])
        if 2.0 * max(shape) * max(case["rays"], 100_000) > 2e9:
            return None
        _, ne, rays = _trace_inputs(case, seed)
        return _exact_trace(ne, rays, _schedule(shape, case["saves"]), axis=case["axis"],
                            plane=L / 2 if case["plane"] else None, ib=case["ib"], rk4=case["integrator"] == "rk4",
                            state=case["state"])
    if k == "solve":
        shape, ne, rays = _solve_inputs(case, seed)
        if 2.0 * case["n"] * max(case["rays"], 100_000) > 2e9:
            return None
        geom = _domain_geom(case["n"])
        o = _exact_trace(ne, rays, _schedule(shape, 1, geom), ib=case["ib"], geom=geom)
        return {"rf": o["jones"][0], "amp": o["amp"][0] if case["ib"] else None}
    if k == "pack":
        ne = _pack_inputs(case, seed)
        q = ne.double() * (1.0 / _optical_constants()[1])
        return {"grid": _packed(ne).reshape(-1), "q_max": max(float(q.max()), 0.0) * (1 + 1e-6),
                "q_min": min(float(q.min()), 0.0) * (1 + 1e-6), "ne_max": float(ne.max())}
    if k == "image":
        if case["rays"] * case["steps"] > 6e7:
            return None
        return _Image(case).run(*_image_inputs(case, seed))
    if k == "optics":
        return _exact_optics(case, seed)
    res = {}
    for j, (kind, n, rays, ne, r) in enumerate(_serve_inputs(case, seed)):
        o = _exact_trace(ne, r, _schedule((n,) * 3, 1), ib=kind == "kolmogorov") if n * rays < 1e8 else None
        res[str(j)] = o
    return res
