"""The grid pack at the edges of its patches (8 x 64 points), of its walks along the
first axis and of the smallest grid, with densities from negative to far above
the critical one, infinite and NaN, against the same formula in torch FP64, and the
density range it returns."""
import math

import pytest
import torch

from sloth_b200 import runtime
from sloth_b200.core import physics

pytestmark = pytest.mark.gpu

OMEGA = physics.omega_of(532e-9)


def _formula(ne, trace):
    q = ne.double() * (1.0 / physics.critical_density(OMEGA))
    x = physics.ope_ratio2(OMEGA) * q
    c0 = -(x / (1.0 + (1.0 - x).clamp_min(0.0).sqrt())) if trace else q
    if trace:
        c0 = torch.where(torch.isnan(q), q, c0)
    out = [c0]
    for a in range(3):
        n = q.shape[a]
        i = torch.arange(n, device=q.device)
        hi, lo = q.index_select(a, (i + 1).clamp_max(n - 1)), q.index_select(a, (i - 1).clamp_min(0))
        w = torch.where((i == 0) | (i == n - 1), 1.0, 0.5).double().reshape([-1 if b == a else 1 for b in range(3)])
        out.append(w * (hi - lo))
    return torch.stack(out, dim=-1)


@pytest.mark.parametrize("shape", [(2, 2, 2), (3, 8, 64), (5, 9, 65), (66, 7, 63), (4, 17, 129), (131, 2, 33)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("special", [False, True])
def test_pack_is_the_formula(shape, dtype, special):
    g = torch.Generator().manual_seed(sum(shape))
    nc = physics.critical_density(OMEGA)
    ne = (torch.rand(shape, generator=g, dtype=torch.float64) * 1.3 * nc).to(dtype)
    ne.view(-1)[: 4] = torch.tensor([-0.2, 0.984, 0.985, 40.0], dtype=torch.float64).to(dtype) * nc
    if special:
        ne.view(-1)[-3:] = torch.tensor([math.inf, -math.inf, 0.0]).to(dtype)
        ne.view(-1)[ne.numel() // 2] = math.nan
    ne = ne.cuda()
    for layout in ("trace", "values"):
        ref = _formula(ne, layout == "trace")
        for precision in ("f64", "f32"):
            p = runtime.pack_grid(ne, (0.0,) * 3, (1e-5,) * 3, OMEGA, precision=precision, layout=layout)
            got = p.data.view(*shape, 4).double()
            assert torch.equal(torch.isnan(got), torch.isnan(ref))
            ok = ~torch.isnan(ref)
            if precision == "f64":
                assert torch.equal(got[ok], ref[ok])
            else:
                # correctly rounded, or next to it where the FP64 value is within its own rounding of a tie
                want = ref.float().double()
                assert bool(((got == want) | ((got - ref).abs() <= 0.5001 * 2.0 ** -23 * ref.abs()))[ok].all())
            if special:
                assert math.isnan(p.ne_max) and math.isnan(p.q_max)
            else:
                assert p.ne_max == float(ne.max())
                assert p.q_min == float(ne.min()) * (1.0 / nc) * (1.0 + 1e-6)


def test_pack_on_a_side_stream():
    ne = (torch.rand((40, 40, 40), device="cuda") * 1e25)
    s = torch.cuda.Stream()
    a = runtime.pack_grid(ne, (0.0,) * 3, (1e-5,) * 3, OMEGA)
    b = runtime.pack_grid(ne, (0.0,) * 3, (1e-5,) * 3, OMEGA, stream=s)
    torch.cuda.synchronize()
    assert torch.equal(a.data, b.data) and a.ne_max == b.ne_max


@pytest.mark.parametrize("source", ["host", "transposed"])
def test_pack_on_a_side_stream_without_the_range(source):
    """The call returns before its pack has run: the device copy of ne that it made
    stays its own although the caller allocates on the current stream at once."""
    ne = torch.rand((40, 40, 40), generator=torch.Generator().manual_seed(2)) * 1e25
    ref = runtime.pack_grid(ne, (0.0,) * 3, (1e-5,) * 3, OMEGA).data
    src = ne if source == "host" else ne.transpose(0, 2).contiguous().cuda().transpose(0, 2)
    out = torch.empty_like(ref)
    a = torch.rand((4096, 4096), device="cuda")
    b = torch.empty_like(a)
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        for _ in range(200):                                     # tens of ms
            torch.mm(a, a, out=b)
    runtime.pack_grid(src, (0.0,) * 3, (1e-5,) * 3, OMEGA, stream=s, with_range=False, out=out)
    junk = [torch.full((40, 40, 40), 7e25, device="cuda") for _ in range(4)]
    assert not s.query()
    torch.cuda.synchronize()
    del junk
    assert torch.equal(out, ref)
