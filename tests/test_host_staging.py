"""Staged host copies: around the stage's size, where no memory can be pinned, and
sources that the caller changes or frees as soon as the call returns."""
import gc

import numpy as np
import pytest
import torch

from sloth_b200 import runtime, workloads
from sloth_b200.core import physics
from sloth_b200.processing import diagnostics

STAGE = runtime._STAGE_BYTES // 4          # float32 elements of one piece


@pytest.mark.parametrize("n", [1, STAGE // 8, STAGE // 8 + 1, 2 * STAGE, 2 * STAGE + 3])
def test_upload_without_pinned_memory(monkeypatch, n):
    monkeypatch.setattr(runtime, "_pinned", lambda shape, dtype: None)
    src = torch.rand(n, requires_grad=True)
    assert torch.equal(runtime.upload(src, torch.empty(n)), src.detach())


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, STAGE // 8, STAGE // 8 + 1, STAGE, STAGE + 1, 2 * STAGE + 3])
@pytest.mark.parametrize("fail_at", [None, 0, 1])
def test_staged_copies_round_trip(monkeypatch, n, fail_at):
    made, pinned = [], runtime._pinned

    def some(shape, dtype):
        made.append(shape)
        return None if fail_at is not None and len(made) > fail_at else pinned(shape, dtype)

    monkeypatch.setattr(runtime, "_pinned", some)
    src = torch.rand(n)
    dev = runtime.upload(src, torch.empty(n, device="cuda"))
    assert torch.equal(dev.cpu(), src)
    assert torch.equal(torch.from_numpy(runtime.download(dev)), src)


def _busy(ms=20.0):
    """About `ms` of work on the current stream, so that what follows it is still pending when the host goes on."""
    a = torch.rand((4096, 4096), device="cuda")
    a @ a
    e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
    e[0].record()
    a @ a
    e[1].record()
    torch.cuda.synchronize()
    for _ in range(max(1, int(ms / e[0].elapsed_time(e[1])))):
        a @ a


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1000, 300_000])                  # below and above a pageable copy's stage
@pytest.mark.parametrize("stacked", [False, True])
def test_diagnostic_takes_a_snapshot_of_pinned_rays(n, stacked):
    """solve() and trace_and_save_depths() return numpy arrays over pinned memory: a
    Diagnostic holds their values at its construction."""
    saves = torch.empty((3, 4, n), dtype=torch.float64, pin_memory=True)
    rf = saves.numpy()
    rf[:] = np.random.default_rng(n).normal(size=rf.shape) * 1e-3
    want = rf[-1].copy()
    _busy()
    d = diagnostics.Shadowgraphy(rf if stacked else rf[-1], verbose=False)
    rf[:] = 7.0                                                 # before the queued work can have finished
    torch.cuda.synchronize()
    np.testing.assert_array_equal(d._rf_in.cpu().numpy(), want)


@pytest.mark.gpu
@pytest.mark.parametrize("with_range", [True, False])
def test_pack_grid_takes_a_snapshot_of_pinned_densities(with_range):
    ne = torch.rand((60, 61, 62), generator=torch.Generator().manual_seed(1)).pin_memory()
    kw = dict(precision="f32", layout="values", ne_scale=1.0)
    ref = runtime.pack_grid(ne.cuda(), (0.0,) * 3, (1e-5,) * 3, physics.omega_of(532e-9), **kw).data.clone()
    _busy()
    g = runtime.pack_grid(ne, (0.0,) * 3, (1e-5,) * 3, physics.omega_of(532e-9), with_range=with_range, **kw)
    ne.fill_(7.0)
    torch.cuda.synchronize()
    assert torch.equal(g.data, ref)


@pytest.mark.gpu
def test_a_host_ahead_of_its_stream_pins_no_more_pieces(monkeypatch):
    """While the stream has not come to the first copy, no more than the pieces in flight are taken."""
    make, late = runtime._pinned, []
    src = torch.rand(12 * STAGE + 5)
    dst = torch.empty(src.numel(), device="cuda")
    src[:100].pin_memory()                                      # the allocator is there
    _busy(100.0)
    before = torch.cuda.Event()
    before.record()

    def pinned(shape, dtype):
        late.append(not before.query())
        return make(shape, dtype)
    monkeypatch.setattr(runtime, "_pinned", pinned)
    runtime.upload(src, dst)
    assert torch.equal(dst.cpu(), src)
    assert len(late) == 13 and 1 <= sum(late) <= runtime._STAGE_PIECES


@pytest.mark.gpu
def test_a_chunked_trace_of_pageable_rays_pins_no_more_pieces(monkeypatch):
    """Ten chunks whose uploads stand behind their lanes' traces share one set of pieces."""
    n, L = 1_500_000, 5e-3
    m = 24
    h = L / (m - 1)
    grid = runtime.pack_grid(workloads.kolmogorov_box(m, L=L, seed=1), (-L / 2,) * 3, (h,) * 3, physics.omega_of(532e-9))
    rays = workloads.gaussian_beam(n, waist=2e-3, L=L, seed=2).double().numpy()      # rows of 1.2 MB per chunk
    sched = runtime.schedule_times([L], (h,) * 3)
    made, flying = [], []

    class Staging(runtime._Staging):
        def __init__(self):
            super().__init__()
            made.append(self)

        def used(self, stream):
            super().used(stream)
            flying.append(self._open + sum(k for _, k in self._marks))
    monkeypatch.setattr(runtime, "_Staging", Staging)
    got, steps, _ = runtime.trace_to_host(grid, rays, sched, want={"jones": "all", "steps": "all"}, chunk_rays=150_000)
    assert len(made) == 1 and len(flying) == 60 and max(flying) <= runtime._STAGE_PIECES
    whole = runtime.trace(grid, torch.from_numpy(rays).float().cuda(), sched)
    assert torch.equal(torch.from_numpy(got["jones"]), whole["jones"].cpu()) and steps == int(whole["total_steps"])


@pytest.mark.gpu
@pytest.mark.parametrize("n", [STAGE // 8 + 1, STAGE, STAGE + 1, 4 * STAGE + 3])
@pytest.mark.parametrize("strided", [False, True])
def test_results_in_ordinary_memory(monkeypatch, n, strided):
    monkeypatch.setattr(runtime, "_PINNED_RESULT_BYTES", 0)
    t = torch.rand((n, 2), device="cuda")[:, 0] if strided else torch.rand(n, device="cuda")
    got = runtime.download(t)
    assert not torch.from_numpy(got).is_pinned()
    assert torch.equal(torch.from_numpy(got), t.cpu())


@pytest.mark.gpu
def test_callers_hold_a_bounded_amount_of_pinned_results():
    t = torch.rand(runtime._PINNED_RESULT_BYTES // 4 // 3 + 1, device="cuda")         # two fit, three do not
    want = t.cpu()
    is_pinned = lambda a: torch.from_numpy(a).is_pinned()  # noqa: E731
    gc.collect()
    assert runtime._pinned_results == 0, "results of other tests are gone"
    kept = [runtime.download(t) for _ in range(4)]
    assert [is_pinned(a) for a in kept] == [True, True, False, False]
    assert all(torch.equal(torch.from_numpy(a), want) for a in kept)
    part = kept[0][5:]
    del kept
    assert runtime._pinned_results == t.nbytes           # the view holds its array
    del part
    assert runtime._pinned_results == 0
    assert is_pinned(runtime.download(t))
