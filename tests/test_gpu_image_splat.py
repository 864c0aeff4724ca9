"""The detector image's splat where its ways of adding a ray change: windows
that fit a block's tiles, windows larger than a tile, rays far apart, on the detector's
edge and off it, blocks with one ray and a ragged last block; and the forward's
checkpoint and warp remainders. Against the torch FP64 model, for each probing axis."""
import math

import pytest
import torch

from oracle import adjoint_torch as at
from sloth_b200 import adjoint, workloads
from sloth_b200.core import physics

pytestmark = pytest.mark.gpu

L = 5e-3
OM = physics.omega_of(532e-9)


@pytest.mark.parametrize("precision", ["f32", "f64"])
@pytest.mark.parametrize("n,n_px,sigma,axis,ckpt,spread", [
    (1, (40, 33), 1.5, 2, 5, 1.0), (33, (200, 180), 0.4, 0, 32, 1.0), (255, (64, 64), 2.0, 1, 1, 0.02),
    (257, (300, 20), 1.0, 2, 7, 1.0), (700, (128, 128), 3.9, 0, 21, 0.3), (520, (90, 120), 8.0, 1, 22, 1.3),
    (1500, (500, 500), 2.0, 2, 20, 1.2)])
def test_image_matches_the_model(precision, n, n_px, sigma, axis, ckpt, spread):
    dt = torch.float32 if precision == "f32" else torch.float64
    steps, m = 45, 14
    h = L / (m - 1)
    ne = workloads.kolmogorov_box(m, L=L, mean=1e26, rms=0.3, seed=n).to(dt)   # leaves of their own below
    g = torch.Generator().manual_seed(n)
    rays = torch.zeros((6, n), dtype=torch.float64)
    t = [a for a in range(3) if a != axis]
    for a in t:
        rays[a] = (torch.rand(n, generator=g, dtype=torch.float64) - 0.5) * L * spread
        rays[3 + a] = physics.C * 0.02 * (torch.rand(n, generator=g, dtype=torch.float64) - 0.5)
    rays[axis] = -L / 2
    rays[3 + axis] = physics.C
    rays = rays.to(dt)
    spec = adjoint.DetectorSpec(window=(-L / 2, L / 2, -L / 2, L / 2), plane=L / 2, dtau=L / (0.975 * steps), n_px=n_px,
                                axis=axis, sigma_px=sigma, n_steps=steps, ckpt_every=ckpt)
    kw = dict(dtau=spec.dtau, n_steps=steps, axis=axis, plane=spec.plane, window=spec.window, n_px=n_px, sigma_px=sigma)
    x = ne.double().clone().requires_grad_(True)
    ref = at.detector_image(x, (-L / 2,) * 3, (h,) * 3, OM, rays.double(), **kw)
    w = torch.rand(n_px, generator=g, dtype=torch.float64)
    (ref * w).sum().backward()
    y = ne.detach().cuda().requires_grad_(True)
    stats = {}
    img = adjoint.detector_image(y, rays.cuda(), spec, origin=(-L / 2,) * 3, spacing=(h,) * 3, omega=OM,
                                 precision=precision, stats=stats)
    (img * w.cuda().to(dt)).sum().backward()
    ref = ref.detach()
    # a sum of at most n terms of relative rounding eps, and detector points off by
    # about 1e-6 (FP32) or 1e-14 of the box in pixels of size L / n_px: the profile's slope is below 1 / sigma
    eps, pos = (6e-8, 1e-6) if precision == "f32" else (1e-16, 1e-14)
    tol = 8 * (eps * math.sqrt(n) * 8 + pos * max(n_px) / sigma)
    assert float((img.detach().double().cpu() - ref).abs().max()) <= tol * float(ref.abs().max())
    err = (y.grad.double().cpu() - x.grad).norm() / x.grad.norm()
    assert float(err) <= (1e-3 if precision == "f32" else 1e-9)
    assert 0 < int(stats["ray_steps"]) <= n * steps
