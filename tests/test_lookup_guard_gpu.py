"""Table cells of shallow targets under fine grids at high elevations: the
float32 lookups decide every cell as float64 does, or leave it to float64.
Rough crossings of zero rms height take the float64 lookups and are otherwise
the same sum, so the two float64 forms agree to the float64 form's bound (1e-9
of the peak; one pair in another cell shows at 1e-4 and more)."""

import numpy as np
import pytest

from tests.test_short_paths_gpu import C, K0
from tests.util import field_errors

pytestmark = pytest.mark.gpu


def _tilted(n, d, z0, tilt, rms, seed):
    from radar_sounder_simulator_gb300.scenes import (facets_from_vertices,
                                                      random_field)
    ax = (np.arange(n + 1) - 0.481 * n) * d
    X, Y = np.meshgrid(ax, ax)
    Z = z0 + tilt * (X - 0.6 * Y) + random_field(
        n + 1, d, 6 * d, rms, np.random.default_rng(seed))
    return facets_from_vertices(X, Y, Z)


@pytest.mark.parametrize("refraction", ["joint", "sequential"])
@pytest.mark.parametrize("cell,depth,z0,tilt,alt,ni", [
    (5.0, 10.0, 3100.3, 0.0, 600.0, 1), (5.0, 12.0, 3100.3, 0.05, 4000.0, 1),
    (10.0, 20.0, 3817.7, 0.05, 12000.0, 1), (5.0, 15.0, 2411.9, 0.1, 900.0, 2),
    (25.0, 60.0, 3400.1, 0.02, 9000.0, 2)])
def test_cells_match_float64_lookups(cell, depth, z0, tilt, alt, ni,
                                     refraction):
    from radar_sounder_simulator_gb300.multilayer import refracted_cluttergram
    n, T = 160, 128
    layers = [_tilted(n, cell, z0 - depth * j, tilt, 0.12 * cell, 5 + j)
              for j in range(ni)]
    bed = _tilted(n - 10, cell * 0.993, z0 - depth * ni, tilt, 0.1 * cell, 9)
    rng = np.random.default_rng(17)
    half = 0.3 * n * cell
    s = np.sort(rng.uniform(-half, half, T))
    pos = np.column_stack([s, 0.4 * s + rng.uniform(-1, 1, T),
                           z0 + alt + rng.uniform(-1, 1, T)])
    uct = np.tile([0.0, -1.0, 0.0], (T, 1))
    kw = dict(mode="coherent", t0=2 * (alt - 0.15 * n * cell * tilt - 30) / C,
              dt=4e-9, n_samples=400, c=C, gamma=0.2, k0=K0,
              refraction=refraction, out_dtype=np.complex128)
    args = (pos, uct, bed, layers, [1.0, 1.8, 3.15][:ni + 1],
            [0.0, 5.0, 9.0][:ni + 1])
    got, _ = refracted_cluttergram(*args, **kw, precision="fp64")
    split, _ = refracted_cluttergram(*args, **kw, precision="split")
    if refraction == "joint":
        ref, _ = refracted_cluttergram(*args, **kw, precision="fp64",
                                       crossed_sigma=[0.0] * ni)
        assert np.abs(got - ref).max() <= 1e-9 * np.abs(ref).max()
    e = field_errors(split, got)
    assert e["rel_l2"] <= 1e-4 and e["phase_rad"] <= 1e-3, e
