"""Staged host copies: around the stage's size, and where no memory can be pinned."""
import pytest
import torch

from sloth_b200 import runtime

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
