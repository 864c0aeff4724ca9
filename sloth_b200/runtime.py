"""Device runtime over the C ABI: device-resident grids, trace launches,
workspaces and output buffers, all as torch CUDA tensors.

Every compute call goes through ``libsloth_b200.so``; this module only owns
memory and streams. There is no CPU path: on a machine without an sm_100
device the library returns an error and ``SlothError`` is raised.
"""
from __future__ import annotations

import math
import struct
import threading
import weakref
from collections import OrderedDict
from dataclasses import dataclass
from typing import Optional

import numpy as np
import torch

from . import _capi as capi
from .core import physics

C = physics.C


def _stream_ptr(stream) -> int:
    if stream is None:
        return int(torch.cuda.current_stream().cuda_stream)
    return int(stream.cuda_stream)


def require_device(device=None) -> torch.device:
    """The CUDA device to run on; raises if there is none (no CPU fallback)."""
    if not torch.cuda.is_available():
        raise capi.SlothError(capi.SLOTH_ERR_NO_DEVICE, "sloth_b200 needs a CUDA device (B200, sm_100)")
    capi.load()
    dev = torch.device(device) if device is not None else torch.device("cuda", torch.cuda.current_device())
    return dev


def uniform_axis(coords) -> tuple[float, float, int]:
    """(origin, spacing, n) of a uniformly spaced coordinate array; raises
    NotImplementedError for a non-uniform one (the tracers index a uniform grid)."""
    c = np.asarray(coords, dtype=np.float64).ravel()
    n = c.size
    if n < 2:
        raise ValueError("each grid axis needs at least 2 points")
    h = (c[-1] - c[0]) / (n - 1)
    if not h > 0:
        raise ValueError("grid coordinates must be increasing")
    dev = np.max(np.abs(c - (c[0] + h * np.arange(n))))
    if dev > 1e-3 * h:
        raise NotImplementedError("non-uniform grid coordinates are not supported by the B200 tracers")
    return float(c[0]), float(h), n


@dataclass
class DeviceGrid:
    """A packed (c0, dq/du, dq/dv, dq/dw) grid resident in HBM: c0 = n - 1 in
    the trace layout (what the tracers read), c0 = q in the value layout (the
    K0 sampler's)."""
    data: torch.Tensor
    desc: capi.SlothGridDesc
    precision: str
    omega: float
    n: tuple
    origin: tuple
    spacing: tuple
    q_max: float = 0.0         # max of the q channel (ne/nc) over the grid; 0 = unknown
    q_min: float = float("inf")  # a lower bound of min(q, 0) over the grid; inf = unknown
    ne_max: float = float("nan")  # largest ne (m^-3) packed, from the device reduction
    layout: str = "trace"

    @property
    def nc(self) -> float:
        return physics.critical_density(self.omega)

    @property
    def extent_lo(self):
        return tuple(self.origin)

    @property
    def extent_hi(self):
        return tuple(o + h * (k - 1) for o, h, k in zip(self.origin, self.spacing, self.n))


_STAGE_BYTES = 8 << 20
_STAGE_PIECES = 8


class _Staging:
    """Pinned pieces that pageable memory passes through: at most _STAGE_PIECES of
    _STAGE_BYTES with copies in flight, so that a host that is faster than its streams waits and
    page-locks no more than these. The caching allocator hands a piece out again once
    its copy is done; an event behind every few pieces holds the host back."""

    def __init__(self):
        self._marks = []                   # (event, pieces before it since the last one), oldest first
        self._open, self._stream = 0, None   # pieces behind the last mark, and their stream

    def _mark(self):
        if self._open:
            done = torch.cuda.Event()
            done.record(self._stream)
            self._marks.append((done, self._open))
            self._open = 0

    def take(self, nbytes: int):
        """A piece of nbytes (uint8), or None where the host has no memory to pin."""
        while self._open + sum(k for _, k in self._marks) >= _STAGE_PIECES:
            self._marks.pop(0)[0].synchronize()
        return _pinned(nbytes, torch.uint8)

    def used(self, stream):
        """The copy queued last on `stream` uses the piece taken last."""
        if stream != self._stream:
            self._mark()
            self._stream = stream
        self._open += 1
        if 2 * self._open >= _STAGE_PIECES:
            self._mark()


def upload(src: torch.Tensor, dst: torch.Tensor, *, wait: bool = True,
           staging: Optional[_Staging] = None) -> torch.Tensor:
    """Copy the CPU tensor src into the CUDA tensor dst (same shape and dtype,
    both contiguous) on the current stream. src may be changed or freed once this
    returns, pinned or not (numpy arrays over pinned memory, as solve() returns
    them, too): a pinned source is copied as it is and the call waits for the copy,
    unless ``wait`` is False, where the caller keeps src unchanged until
    it has waited for the stream itself. Pageable memory goes through the pinned pieces of
    ``staging`` (the call's own by default), which the host's threads
    fill while the previous piece is copied (the driver's own staging fills
    them with one thread: 67 MB in 5.6 ms)."""
    src = src.detach()
    if src.is_pinned():
        dst.copy_(src, non_blocking=True)
        if wait:
            torch.cuda.current_stream(dst.device).synchronize()
        return dst
    if src.nbytes <= _STAGE_BYTES // 8:
        return dst.copy_(src, non_blocking=True)
    staging = staging or _Staging()
    s, d = src.reshape(-1), dst.view(-1)
    m = _STAGE_BYTES // src.element_size()
    for a in range(0, s.numel(), m):
        part = s[a:a + m]
        piece = None                       # the last one goes back first
        piece = staging.take(part.nbytes)
        if piece is None:
            d[a:].copy_(s[a:], non_blocking=True)
            break
        piece = piece.view(s.dtype)
        piece.copy_(part)
        d[a:a + m].copy_(piece, non_blocking=True)
        staging.used(torch.cuda.current_stream(dst.device))
    return dst


def _pinned(shape, dtype):
    """A pinned host tensor, or None where the host has no more memory to pin."""
    try:
        return torch.empty(shape, dtype=dtype, pin_memory=True)
    except RuntimeError:
        return None


# Pinned results that callers hold at a time: three full camera images in FP64 (a loop holds
# the last while it makes the next). A block that the pinned allocator has free takes 71 MB
# in 1.34 ms, ordinary memory through pinned pieces 2.9 (cpu() 32.5); but a caller that keeps every result would
# page-lock, and pay for, a new block each time (52 ms), so beyond this results are ordinary memory.
_PINNED_RESULT_BYTES = 256 << 20
_pinned_results = 0
_pinned_lock = threading.RLock()           # reentrant: a result may go while it is held
_pinned_refs: dict = {}                    # the references whose callbacks give the bytes back


class _Held(weakref.ref):
    """Reference to a pinned result that gives its bytes back when it goes (weakref.finalize
    does as much in 10 us more)."""
    __slots__ = ("nbytes",)


def _release(ref):
    global _pinned_results
    with _pinned_lock:
        _pinned_results -= ref.nbytes
        _pinned_refs.pop(id(ref), None)


def _hold(result: np.ndarray, nbytes: int):
    """Count a pinned result for as long as it (or a view of it) lives."""
    global _pinned_results
    ref = _Held(result, _release)
    ref.nbytes = nbytes
    with _pinned_lock:
        _pinned_results += nbytes
        _pinned_refs[id(ref)] = ref


def download(t: torch.Tensor) -> np.ndarray:
    """The CUDA tensor t as a numpy array: in pinned memory when it is large and
    callers hold no more than _PINNED_RESULT_BYTES of such results, otherwise in ordinary memory."""
    nbytes = t.nbytes
    if nbytes <= _STAGE_BYTES // 8:
        return t.cpu().numpy()
    stream = torch.cuda.current_stream(t.device)
    if _pinned_results + nbytes <= _PINNED_RESULT_BYTES:
        h = _pinned(t.shape, t.dtype)
        if h is not None:
            h.copy_(t, non_blocking=True)
            out = h.numpy()
            _hold(out, nbytes)             # while the copy runs
            stream.synchronize()
            return out
    s = t.detach().reshape(-1)
    host = torch.empty(t.shape, dtype=t.dtype)
    d = host.view(-1)
    m = _STAGE_BYTES // t.element_size()
    ahead = []                                                 # (piece, event, start) on their way, three at most

    def land():
        piece, done, a = ahead.pop(0)
        done.synchronize()
        d[a:a + m].copy_(piece[:d[a:a + m].numel()])
        return piece

    for a in range(0, s.numel(), m):
        piece = land() if len(ahead) == 3 else _pinned(min(m, s.numel()), t.dtype)
        if piece is None:                                      # no memory to pin
            if ahead:
                piece = land()
            else:
                d[a:].copy_(s[a:])
                break
        piece[:s[a:a + m].numel()].copy_(s[a:a + m], non_blocking=True)
        done = torch.cuda.Event()
        done.record(stream)
        ahead.append((piece, done, a))
    while ahead:
        land()
    return host.numpy()


def _from_order_key(key: int) -> float:
    """The double of an order key of sloth_grid_pack_range (as int64)."""
    b = key & 0xFFFFFFFFFFFFFFFF
    if b == 0xFFFFFFFFFFFFFFFF:
        return float("nan")
    b = b ^ (1 << 63) if b >> 63 else b ^ 0xFFFFFFFFFFFFFFFF
    return struct.unpack("<d", struct.pack("<Q", b))[0]


def pack_grid(ne, origin, spacing, omega, *, precision="f32", device=None, stream=None,
              out: Optional[torch.Tensor] = None, ne_scale: Optional[float] = None,
              layout: str = "trace", with_range: bool = True) -> DeviceGrid:
    """K1: pack ne (m^-3, (nx, ny, nz) array or tensor) into a device grid.

    ``ne`` may be a numpy array, a CPU tensor (pinned for a fast copy) or a
    CUDA tensor; float32 and float64 are read as they are. q = ne * ne_scale
    with ne_scale = 1/nc(omega) unless given. ``layout`` 'trace' (the
    tracers' grid) stores n - 1 of the plasma refractive index in channel 0,
    'values' stores q there (for the K0 sampler). The density's range, which
    the tracers' fast paths use, is the one thing the call waits for;
    ``with_range=False`` leaves it unknown and does not wait.
    """
    if layout not in ("trace", "values"):
        raise ValueError("layout must be 'trace' or 'values'")
    dev = require_device(device)
    if isinstance(ne, np.ndarray):
        ne = torch.from_numpy(np.ascontiguousarray(ne))
    if ne.dtype not in (torch.float32, torch.float64):
        ne = ne.to(torch.float32)
    if ne.dim() != 3:
        raise ValueError("ne must be a 3-D (nx, ny, nz) array")
    ne = ne.contiguous()
    if ne.device.type != "cuda":
        # with the range, its wait at the end covers this copy
        ne = upload(ne, torch.empty(ne.shape, dtype=ne.dtype, device=dev), wait=not with_range)
    n = tuple(int(k) for k in ne.shape)
    desc = capi.grid_desc(n, origin, spacing)
    rb = 4 if precision == "f32" else 8
    nbytes = capi.load().sloth_grid_bytes(desc, rb)
    if nbytes == 0:
        raise ValueError(f"invalid grid {n}")
    if out is None:
        out = torch.empty(nbytes // rb, dtype=torch.float32 if rb == 4 else torch.float64, device=dev)
    scale = 1.0 / physics.critical_density(omega) if ne_scale is None else float(ne_scale)
    lib = capi.load()
    ope2 = physics.ope_ratio2(omega) if layout == "trace" else 0.0
    geom = (out, desc, precision, float(omega), n, tuple(map(float, origin)), tuple(map(float, spacing)))
    run_on = stream if stream is not None else torch.cuda.current_stream(dev)
    if stream is not None:
        # ne (or its copy made here) and out belong to the current stream: `stream` waits
        # for them, and their memory for `stream`
        run_on.wait_stream(torch.cuda.current_stream(dev))
        ne.record_stream(run_on)
        out.record_stream(run_on)
    if not with_range:
        if layout == "trace":
            fn = lib.sloth_grid_pack_trace_f32 if rb == 4 else lib.sloth_grid_pack_trace_f64
            rc = fn(desc, capi.ptr(ne), int(ne.dtype == torch.float64), scale, ope2, capi.ptr(out), _stream_ptr(run_on))
        else:
            fn = lib.sloth_grid_pack_f32 if rb == 4 else lib.sloth_grid_pack_f64
            rc = fn(desc, capi.ptr(ne), int(ne.dtype == torch.float64), scale, capi.ptr(out), _stream_ptr(run_on))
        capi.check(rc, "sloth_grid_pack")
        return DeviceGrid(*geom, layout=layout)
    with torch.cuda.stream(run_on):
        rng = torch.empty(2, dtype=torch.int64, device=dev)
        capi.check(lib.sloth_grid_pack_range(desc, capi.ptr(ne), int(ne.dtype == torch.float64), int(rb == 8), scale,
                                             ope2, capi.ptr(out), capi.ptr(rng), _stream_ptr(run_on)),
                   "sloth_grid_pack_range")
        ne_max, neg_min = (_from_order_key(k) for k in rng.tolist())   # the one wait of the call
    q_max, q_min = ne_max * scale, -neg_min * scale
    return DeviceGrid(*geom, q_max=max(q_max, 0.0) * (1.0 + 1e-6), q_min=min(q_min, 0.0) * (1.0 + 1e-6), ne_max=ne_max,
                      layout=layout)


def sample(grid: DeviceGrid, points, *, stream=None) -> torch.Tensor:
    """K0: (4, N) interpolated (c0, dq/du, dq/dv, dq/dw) at points (3, N) in
    metres (c0 = q in the value layout)."""
    pts = torch.as_tensor(points, dtype=torch.float64)
    pts = pts.to(grid.data.device).contiguous()
    n = pts.shape[1]
    out = torch.empty((4, n), dtype=grid.data.dtype, device=grid.data.device)
    fn = capi.load().sloth_sample_f32 if grid.precision == "f32" else capi.load().sloth_sample_f64
    if stream is not None and stream != torch.cuda.current_stream(grid.data.device):
        stream.wait_stream(torch.cuda.current_stream(grid.data.device))   # pts and out are made on the current stream
        pts.record_stream(stream)
        out.record_stream(stream)
    capi.check(fn(grid.desc, capi.ptr(grid.data), capi.ptr(pts), n, capi.ptr(out), _stream_ptr(stream)),
               "sloth_sample")
    return out


@dataclass
class Schedule:
    """Fixed-step schedule: every step is dtau (metres of c*t); save j is
    taken after step first_save + j*save_every."""
    dtau: float
    first_save: int
    save_every: int
    n_saves: int

    @property
    def last_step(self) -> int:
        return self.first_save + (self.n_saves - 1) * (self.save_every if self.n_saves > 1 else 0)


def nominal_step(spacing) -> float:
    """Path-length step: half the smallest grid spacing."""
    return 0.5 * min(spacing)


def schedule_times(tau_saves, spacing) -> Schedule:
    """Schedule whose saves land exactly on uniformly spaced c*t values
    tau_saves[j] = tau_saves[0] + j*d (tau_saves[0] is 0 or the only save);
    the step is the largest dtau <= nominal_step that divides d."""
    tau_saves = np.asarray(tau_saves, dtype=np.float64)
    h = nominal_step(spacing)
    if tau_saves.size == 1:
        T = float(tau_saves[0])
        if T <= 0:
            return Schedule(h, 0, 1, 1)
        m = max(1, math.ceil(T / h - 1e-9))
        return Schedule(T / m, m, 1, 1)
    if abs(tau_saves[0]) > 0:
        raise ValueError("multi-save schedules start at t = 0")
    d = float(tau_saves[1] - tau_saves[0])
    m = max(1, math.ceil(d / h - 1e-9))
    return Schedule(d / m, 0, m, int(tau_saves.size))


_ws_cache: OrderedDict = OrderedDict()     # (device, stream, thread) -> workspace, oldest first
_ws_lock = threading.Lock()
_WS_KEPT = 8


def _workspace(n: int, dev, stream) -> torch.Tensor:
    """The scratch memory of a trace of n rays on `stream`: one per stream and thread,
    because a trace's kernels must not meet another's in it (two threads' launches on one stream may
    alternate). The _WS_KEPT used last are kept; they belong to their stream, so one that is
    given back is reused behind the kernels that still use it."""
    need = int(capi.load().sloth_trace_workspace_bytes(n))
    key = (dev.index, int(stream.cuda_stream), threading.get_ident())
    with _ws_lock:
        t = _ws_cache.get(key)
        if t is not None and t.numel() >= need:
            _ws_cache.move_to_end(key)
            return t
    with torch.cuda.stream(stream):
        t = torch.empty(need, dtype=torch.uint8, device=dev)
    with _ws_lock:
        _ws_cache[key] = t
        _ws_cache.move_to_end(key)
        while len(_ws_cache) > _WS_KEPT:
            _ws_cache.popitem(last=False)
    return t


def integrator_code(integrator: str) -> int:
    """SLOTH_INTEGRATOR_* of 'rkn' or 'rk4'."""
    codes = {"rkn": capi.SLOTH_INTEGRATOR_RKN, "rk4": capi.SLOTH_INTEGRATOR_RK4}
    if integrator not in codes:
        raise ValueError(f"integrator must be 'rkn' or 'rk4', not {integrator!r}")
    return codes[integrator]


def trace(grid: DeviceGrid, rays: torch.Tensor, sched: Schedule, *, axis=2, project=False, plane=0.0,
          inv_brems=False, Te=None, Z=None, want_state=False, want_phase=True, want_amp=None,
          want_status=True, want_steps=True, stream=None, workspace: Optional[torch.Tensor] = None,
          outputs: Optional[dict] = None, events=None, integrator: str = "rkn") -> dict:
    """K2/K3: trace rays (6, N) (device tensor of the grid's precision).

    ``integrator`` is 'rkn' (fourth-order Runge-Kutta-Nystrom, three field
    samples per step, the default) or 'rk4' (classical RK4, four samples).

    Returns a dict of device tensors: jones [S,4,N], optional state [S,6,N],
    phase [S,N] (float64), amp [S,N], status [N] (uint8), steps [N] (int32),
    total_steps [1] (int64 view of the kernel's counter). ``events`` is an
    optional pair of recorded torch.cuda.Event(enable_timing=True) that the
    library re-records around the tracer kernel alone.
    """
    if grid.layout != "trace":
        raise ValueError("the tracers read grids packed with layout='trace'")
    dtype = torch.float32 if grid.precision == "f32" else torch.float64
    own = []                               # tensors made here
    if rays.dtype != dtype or rays.device != grid.data.device or not rays.is_contiguous():
        rays = rays.to(device=grid.data.device, dtype=dtype).contiguous()
        own.append(rays)
    if rays.dim() != 2 or rays.shape[0] != 6:
        raise ValueError("rays must have shape (6, N)")
    n = int(rays.shape[1])
    S = sched.n_saves
    dev = grid.data.device
    if want_amp is None:
        want_amp = inv_brems
    o = outputs if outputs is not None else {}

    def buf(key, shape, dt, want=True):
        if not want:
            o.pop(key, None)
            return None
        t = o.get(key)
        if t is None or tuple(t.shape) != tuple(shape) or t.dtype != dt:
            t = torch.empty(shape, dtype=dt, device=dev)
            o[key] = t
            own.append(t)
        return t

    jones = buf("jones", (S, 4, n), dtype)
    state = buf("state", (S, 6, n), dtype, want_state)
    phase = buf("phase", (S, n), torch.float64, want_phase)
    amp = buf("amp", (S, n), dtype, want_amp)
    status = buf("status", (n,), torch.uint8, want_status)
    steps = buf("steps", (n,), torch.int32, want_steps)
    total = buf("total_steps", (1,), torch.int64)
    p = capi.SlothTraceParams()
    p.omega = grid.omega
    p.dtau = sched.dtau
    p.first_save = sched.first_save
    p.save_every = max(1, sched.save_every)
    p.n_saves = S
    p.probing_axis = int(axis)
    p.project_to_plane = int(bool(project))
    p.plane = float(plane)
    p.inv_brems = int(bool(inv_brems))
    if inv_brems:
        kq2, clw, ope2 = physics.kappa_factors(Te, Z, grid.omega)
        p.kappa_q2, p.coulomb_log_w, p.ope_ratio2 = kq2, clw, ope2
    else:
        p.kappa_q2, p.coulomb_log_w, p.ope_ratio2 = 0.0, 2.0, physics.ope_ratio2(grid.omega)
    p.q_max = float(grid.q_max)
    p.q_min = float(grid.q_min)
    p.integrator = integrator_code(integrator)
    out = capi.SlothTraceOutputs()
    out.jones = capi.ptr(jones)
    out.state = capi.ptr(state)
    out.phase = capi.ptr(phase)
    out.amp = capi.ptr(amp)
    out.status = capi.ptr(status)
    out.steps = capi.ptr(steps)
    out.total_steps = capi.ptr(total)
    if events is not None:
        out.trace_event_begin = int(events[0].cuda_event)
        out.trace_event_end = int(events[1].cuda_event)
    run_on = stream if stream is not None else torch.cuda.current_stream(dev)
    if stream is not None and own and stream != torch.cuda.current_stream(dev):
        # made on the current stream, used on `stream`
        stream.wait_stream(torch.cuda.current_stream(dev))
        for t in own:
            t.record_stream(stream)
    ws = workspace if workspace is not None else _workspace(n, dev, run_on)
    fn = capi.load().sloth_trace_f32 if grid.precision == "f32" else capi.load().sloth_trace_f64
    capi.check(fn(grid.desc, capi.ptr(grid.data), p, capi.ptr(rays), n, out, capi.ptr(ws), ws.numel(),
                  _stream_ptr(run_on)), "sloth_trace")
    return o


_lane_cache: dict = {}


def _lanes(dev):
    """Two side streams of the device (created once) for trace_to_host."""
    key = str(dev)
    lanes = _lane_cache.get(key)
    if lanes is None:
        lanes = (torch.cuda.Stream(dev), torch.cuda.Stream(dev))
        _lane_cache[key] = lanes
    return lanes


STREAM_CHUNK_RAYS = 1 << 24
STREAM_END_RAYS = 1 << 19


def _chunk_bounds(n: int, cs: int) -> list:
    """Chunk boundaries of n rays for trace_to_host: at most `cs` rays per
    chunk. Above 8 * STREAM_END_RAYS rays (8 * cs when cs is smaller) the
    first and the last chunk hold only that many, because the first chunk's
    copy in and the last chunk's copy out are the only copies no trace hides;
    below it every chunk is alike. Chunks between the ends differ in size by
    one ray at most.

    Each chunk is one trace launch, and a launch costs more than its rays'
    share (its ramp and the tail of its tile queue: at 512^3 with a 3 mm
    waist beam, 3M rays trace at 114 ms per 1e7 rays against 102 ms in one
    launch of 1e7). So the default takes chunks as large as the end chunks'
    traces can hide the middle chunks' copies behind: 1e7 rays go through as
    0.5M, 9M and 0.5M (118 ms for solve() with that beam against 126 ms as
    0.5M, three of 3M and 0.5M)."""
    if n <= 0:
        return [0, 0]

    def split(lo, hi):
        m = hi - lo
        k = max(1, -(-m // cs))
        q, r = divmod(m, k)
        return [lo + i * q + min(i, r) for i in range(k + 1)]

    end = min(cs, STREAM_END_RAYS)
    if n <= 8 * end:
        return split(0, n)
    return [0] + split(end, n - end) + [n]


def trace_to_host(grid: DeviceGrid, rays, sched: Schedule, *, want: dict, chunk_rays: Optional[int] = None,
                  stream=None, **kw):
    """Trace rays (6, N) and return the requested outputs as numpy arrays,
    streaming the rays through the device in chunks.

    ``rays`` is a host or device tensor or a numpy array. ``want`` maps output
    names ("jones", "state", "phase", "amp", "status", "steps") to "all"
    (every save) or "last" (the last save; per-ray outputs ignore it). The
    other keywords are those of ``trace``.

    Chunk c runs on side stream c % 2: its rays are copied in, traced, and
    its outputs copied into pinned host arrays at the chunk's columns. While
    one chunk traces, the other stream's copies run, so the host<->device
    traffic hides under the tracer except for the first chunk's rays and the
    last chunk's outputs. Each ray's arithmetic does not depend on the other
    rays of its launch, so the results are bitwise those of one trace of all
    N rays.

    Returns (dict of numpy arrays, total ray-steps, seconds from the first
    copy to the last output on the host).
    """
    import time

    dtype = torch.float32 if grid.precision == "f32" else torch.float64
    dev = grid.data.device
    src = torch.from_numpy(np.ascontiguousarray(rays)) if not isinstance(rays, torch.Tensor) else rays
    if src.dim() != 2 or src.shape[0] != 6:
        raise ValueError("rays must have shape (6, N)")
    if src.stride(1) != 1:
        src = src.contiguous()
    n = int(src.shape[1])
    S = sched.n_saves
    bounds = _chunk_bounds(n, int(chunk_rays or STREAM_CHUNK_RAYS))
    n_chunks = len(bounds) - 1
    inv_brems = bool(kw.get("inv_brems", False))
    want = {k: v for k, v in want.items() if k != "amp" or inv_brems}

    def host_shape(k):
        rows = {"jones": (4,), "state": (6,)}.get(k, ())
        if k in ("status", "steps"):
            return (n,)
        return ((S,) if want[k] == "all" else ()) + rows + (n,)

    hdt = {"jones": dtype, "state": dtype, "amp": dtype, "phase": torch.float64, "status": torch.uint8,
           "steps": torch.int32}
    host = {k: torch.empty(host_shape(k), dtype=hdt[k], pin_memory=True) for k in want}
    totals = torch.empty(n_chunks, dtype=torch.int64, pin_memory=True)
    cur = stream if stream is not None else torch.cuda.current_stream(dev)
    ready = torch.cuda.Event()
    ready.record(cur)
    lanes = _lanes(dev)
    for lane in lanes:
        lane.wait_event(ready)
    outs = ({}, {})
    stage = [None, None]
    staging = _Staging()                   # one for the call: the host may run ahead of the lanes
    t0 = time.perf_counter()
    for c in range(n_chunks):
        a, b = bounds[c], bounds[c + 1]
        li = c % 2
        lane = lanes[li]
        with torch.cuda.stream(lane):
            m = b - a
            st = stage[li]
            if st is None or st.shape[1] != m or st.dtype != src.dtype:
                st = torch.empty((6, m), dtype=src.dtype, device=dev)
                stage[li] = st
            for r in range(6):
                if src.device.type == "cuda":
                    st[r].copy_(src[r, a:b], non_blocking=True)
                else:
                    upload(src[r, a:b], st[r], wait=False, staging=staging)   # the lanes are waited for below
            rc = st if src.dtype == dtype else st.to(dtype)
            o = trace(grid, rc, sched, stream=lane, outputs=outs[li],
                      want_state="state" in want, want_phase="phase" in want, want_amp="amp" in want,
                      want_status="status" in want, want_steps="steps" in want, **kw)
            for k, h in host.items():
                d = o[k]
                if k in ("status", "steps"):
                    h[a:b].copy_(d, non_blocking=True)
                    continue
                if want[k] == "last":
                    d = d[-1]
                    if d.dim() == 1:
                        h[a:b].copy_(d, non_blocking=True)
                    else:
                        for r in range(d.shape[0]):
                            h[r, a:b].copy_(d[r], non_blocking=True)
                    continue
                for s_ in range(S):
                    if d.dim() == 2:
                        h[s_, a:b].copy_(d[s_], non_blocking=True)
                    else:
                        for r in range(d.shape[1]):
                            h[s_, r, a:b].copy_(d[s_, r], non_blocking=True)
            totals[c:c + 1].copy_(o["total_steps"], non_blocking=True)
    for lane in lanes:
        lane.synchronize()
        cur.wait_stream(lane)
    dt = time.perf_counter() - t0
    return {k: h.numpy() for k, h in host.items()}, int(totals.sum()), dt
