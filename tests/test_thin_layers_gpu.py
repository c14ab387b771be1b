"""Refracted paths through layers a few metres apart that nearly meet, under a
platform kilometres away: legs ten thousand times shorter than the path, whose
crossings the float64 form still solves to the reference's validity limit.
Float64 form within 1e-9 of the peak, dropped power (single precision) within
1e-6."""

import numpy as np
import pytest

from oracle import refracted as oref
from tests.test_short_paths_gpu import C, K0, _layer, _track

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["coherent", "incoherent"])
@pytest.mark.parametrize("refraction", ["joint", "sequential"])
@pytest.mark.parametrize("ni,alt,d,eps", [
    (1, 20000.0, 50.0, [1.0, 3.15]), (2, 20000.0, 50.0, [2.0, 1.0, 3.0]),
    (2, 8000.0, 30.0, [1.0, 1.7, 2.4]), (3, 8000.0, 50.0, [1.0, 3.15, 5.0, 3.0])])
def test_layers_that_nearly_meet(ni, alt, d, eps, refraction, mode):
    from radar_sounder_simulator_gb300.multilayer import refracted_cluttergram
    layers = [_layer(72, 77, d, -3.0 * j, 0.03 * d, 200 + j)
              for j in range(ni)]
    bed = _layer(70, 75, 0.97 * d, -3.0 * ni - 3.0, 0.04 * d, 290)
    pos, uct = _track(4, alt, step=30.0)
    kw = dict(mode=mode, t0=2 * (alt * np.sqrt(eps[0]) - 60.0) / C, dt=2e-8,
              n_samples=400, c=C, refraction=refraction)
    if mode == "coherent":
        kw.update(gamma=0.2, k0=K0)
    args = (pos, uct, bed, layers, eps, [0.0, 8.0, 12.0, 15.0][:ni + 1])
    ref, drop = oref.refracted_cluttergram(*args, **kw)
    got, gd = refracted_cluttergram(
        *args, **kw, precision="fp64",
        out_dtype=np.complex128 if mode == "coherent" else np.float64)
    assert np.abs(got - ref).max() <= 1e-9 * np.abs(ref).max()
    assert np.abs(gd - drop).max() <= 1e-6 * drop.max()
