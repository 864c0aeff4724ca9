"""The detector histogram's bins against numpy.histogram2d where rounding decides: values
on and next to every edge, ranges far from zero, whose edges are about a hundred
units in the last place apart, and the smallest and largest bin counts. Counts are whole numbers
and must be equal."""
import numpy as np
import pytest

from sloth_b200.processing import diagnostics

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(1, 1), (7, 3), (3448, 2), (2, 65536)])
@pytest.mark.parametrize("lo,hi", [(-9.0, 9.0), (0.0, 0.3), (1e6, 1e6 + 1e-3), (-1e9, -1e9 + 1.0), (1e-300, 3e-300)])
def test_bins_are_numpys(nx, ny, lo, hi):
    rng = np.random.default_rng(nx + ny)

    def values(n):
        e = np.linspace(lo, hi, n + 1)
        e = e[rng.integers(0, n + 1, 4000)]
        return np.concatenate([e, np.nextafter(e, np.inf), np.nextafter(e, -np.inf), rng.uniform(lo, hi, 4000),
                               [lo, hi, np.nan, np.inf, -np.inf, lo - (hi - lo), hi + (hi - lo)]])
    x, y = values(nx), values(ny)
    rays = np.stack([x, np.zeros_like(x), y, np.zeros_like(y)])
    _, _, H = diagnostics.run_optics(rays, [], hist=(nx, ny, (lo, hi), (lo, hi)))
    ok = np.isfinite(x) & np.isfinite(y)
    ref, _, _ = np.histogram2d(x[ok], y[ok], bins=[np.linspace(lo, hi, nx + 1), np.linspace(lo, hi, ny + 1)])
    np.testing.assert_array_equal(H.cpu().numpy(), ref.T)
