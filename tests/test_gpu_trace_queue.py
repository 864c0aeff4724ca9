"""The tracer's ray queue, pre-pass and builds at the sizes where they change: part
of a warp, one ray around whole warps, around the rays that a full GPU's warps take
first, around the largest trace of the build that fetches the next cell ahead (with rays
along each axis and some that run backwards), and around the pre-pass's bucket counts
(a scan of one word, of one and of several CTAs). Each ray's result does not depend on the other rays of its
launch, so every size gives bitwise the rays of one larger trace, which the oracle's rays confirm."""
import numpy as np
import pytest
import torch

from helpers import run_oracle
from sloth_b200 import runtime, workloads
from sloth_b200.core import physics

pytestmark = pytest.mark.gpu

L = 5e-3


def _trace(n_rays, rays, grid, sched, **kw):
    o = {k: torch.full(s, v, dtype=d, device="cuda") for k, s, d, v in (
        ("jones", (sched.n_saves, 4, n_rays), rays.dtype, 7e9), ("phase", (sched.n_saves, n_rays), torch.float64, 7e9),
        ("status", (n_rays,), torch.uint8, 99), ("steps", (n_rays,), torch.int32, -5))}
    return runtime.trace(grid, rays[:, :n_rays].contiguous(), sched, outputs=o, **kw)


@pytest.mark.parametrize("precision", ["f32", "f64"])
@pytest.mark.parametrize("shape,axis,ib,integ", [((20, 33, 24), 2, True, "rkn"), ((2, 2, 40), 2, False, "rkn"),
                                                 ((31, 18, 27), 0, True, "rkn"), ((19, 22, 30), 1, False, "rkn"),
                                                 ((20, 33, 24), 2, True, "rk4"),
                                                 ((90, 80, 81), 1, True, "rkn")])      # a grid of more than 6 MB
def test_every_ray_once_and_bitwise_the_same(precision, shape, axis, ib, integ):
    h = tuple(L / (k - 1) for k in shape)
    g = torch.Generator().manual_seed(3)
    ne = (torch.rand(shape, generator=g) * 2e25).float()
    grid = runtime.pack_grid(ne, (-L / 2,) * 3, h, physics.omega_of(532e-9), precision=precision)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    # the largest trace of the build that fetches ahead
    ahead = sms * 32 * (12 if 16 * shape[0] * shape[1] * shape[2] > 6 << 20 else 4)
    most = sms * 16 * 32 + 33            # the warps at 16 per SM, and one more warp's worth
    assert most - 33 > ahead             # so the builds are compared
    rays = workloads.gaussian_beam(most, waist=3e-3, L=L, jitter=5e-2, seed=2, device="cuda", dtype=torch.float64)
    to = {0: [2, 0, 1], 1: [0, 2, 1], 2: [0, 1, 2]}[axis]      # the beam along `axis`
    rays = rays[to + [3 + k for k in to]].contiguous()
    back = torch.arange(most, device="cuda") % 7 == 3           # some rays run backwards from the far face
    rays[axis, back] = L / 2
    rays[3 + axis, back] *= -1.0
    rays = rays.to(torch.float32 if precision == "f32" else torch.float64)
    sched = runtime.schedule_times([0.0, L, 2 * L], h)
    kw = dict(axis=axis, inv_brems=ib, Te=20.0 if ib else None, Z=1.0 if ib else None, integrator=integ)
    keys = ["jones", "phase", "status", "steps"] + (["amp"] if ib else [])
    whole = _trace(most, rays, grid, sched, **kw)
    assert int(whole["total_steps"]) == int(whole["steps"].sum(dtype=torch.int64))
    # around a scheduler's share of rays (8 and 32 per warp on four warps per SM), the small pre-pass (6144 rays), the
    # pre-pass's bucket counts and the two builds
    for n in (1, 2, 8, 9, 31, 32, 33, 64, 255, 257, sms * 4 * 8, sms * 4 * 8 + 1, sms * 4 * 32, sms * 4 * 32 + 1, 6144, 6145,
              32768, 32769, ahead, ahead + 1, 65537, most - 33, most - 1):
        part = _trace(n, rays, grid, sched, **kw)
        for k in keys:
            assert torch.equal(part[k], whole[k][..., :n]), (n, k)
        assert int(part["total_steps"]) == int(part["steps"].sum(dtype=torch.int64))
    assert int(whole["status"].max()) <= 2 and float(whole["jones"].abs().max()) < 1e9
    few = 257
    ref = run_oracle(ne.numpy(), rays[:, :few].double().cpu().numpy(), (-L / 2,) * 3, h, physics.omega_of(532e-9), sched,
                     axis=axis, inv_brems=ib, Te=20.0, Z=1.0, integrator=integ)
    err = np.abs(whole["jones"][..., :few].double().cpu().numpy() - ref["jones"])
    err[:, [0, 2]] /= L
    if precision == "f64":
        assert err.max() < 1e-9
    else:                                # rays that graze a face may leave by their rounding
        assert np.quantile(err, 0.98) < 1e-6
    assert (whole["status"][:few].cpu().numpy() != ref["status"]).mean() < 0.01
