"""Traces on streams and threads of their own: each has a workspace to itself, and
what a call makes on the current stream is there, and stays there, for the stream that it runs on."""
import threading

import pytest
import torch

from sloth_b200 import runtime, workloads
from sloth_b200.core import physics

pytestmark = pytest.mark.gpu

L = 5e-3


def _case(n_rays, seed):
    m = 40
    h = L / (m - 1)
    grid = runtime.pack_grid(workloads.kolmogorov_box(m, L=L, seed=seed), (-L / 2,) * 3, (h,) * 3,
                             physics.omega_of(532e-9))
    rays = workloads.gaussian_beam(n_rays, waist=2e-3, L=L, seed=seed, device="cuda")
    return grid, rays, runtime.schedule_times([L], (h,) * 3)


def _same(a, b):
    return all(torch.equal(a[k], b[k]) for k in ("jones", "phase", "status", "steps", "total_steps"))


@pytest.mark.parametrize("own_streams", [False, True])
def test_concurrent_traces_have_their_own_workspaces(own_streams):
    cases = [_case(n, i) for i, n in enumerate((30_000, 200_001, 9_000, 77_777))]
    ref = [runtime.trace(*c) for c in cases]
    torch.cuda.synchronize()
    used, got = {}, {}

    def work(i):
        s = torch.cuda.Stream() if own_streams else torch.cuda.default_stream()
        with torch.cuda.stream(s):
            used[i] = runtime._workspace(cases[i][1].shape[1], cases[i][1].device, s).data_ptr()
            got[i] = [runtime.trace(*cases[i]) for _ in range(10)]
        s.synchronize()

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(cases))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert len(set(used.values())) == len(cases)
    assert len(runtime._ws_cache) <= runtime._WS_KEPT
    for i, r in enumerate(ref):
        assert all(_same(o, r) for o in got[i]), i


def test_tensors_made_by_the_call_belong_to_its_stream_too():
    """FP64 rays are cast on the current stream, whose work is late; the trace runs on another
    stream, and the current one allocates anew at once."""
    grid, rays, sched = _case(100_000, 7)
    ref = runtime.trace(grid, rays, sched)
    torch.cuda.synchronize()
    a = torch.rand((4096, 4096), device="cuda")
    b = torch.empty_like(a)
    late = torch.zeros(rays.shape, dtype=torch.float64, device="cuda")
    s = torch.cuda.Stream()
    for _ in range(100):
        torch.mm(a, a, out=b)
    late.copy_(rays)
    with torch.cuda.stream(s):
        for _ in range(100):
            torch.mm(a, a)
    out = runtime.trace(grid, late, sched, stream=s)
    pts = runtime.sample(grid, torch.zeros((3, 4)), stream=s)
    junk = [torch.full(rays.shape, 3.0, device="cuda") for _ in range(4)]
    torch.cuda.synchronize()
    del junk
    assert _same(out, ref)
    assert torch.equal(pts, runtime.sample(grid, torch.zeros((3, 4))))
