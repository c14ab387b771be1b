"""Several prepared batches alive at once: a later batch of another shape or
with other options leaves the earlier ones launchable. Each replays its own
one-call result (float32 sums in another order: 1e-5, as in the batches' other
tests)."""

import numpy as np
import pytest

from tests.test_short_paths_gpu import C, K0, _layer, _track
from tests.util import rel_l2

pytestmark = pytest.mark.gpu


def _same(batch):
    for plan, (field, _) in zip(batch.plans, batch.run()):
        got, one = field.cpu().numpy(), plan.run()[0].cpu().numpy()
        assert rel_l2(got, one) <= 1e-5


@pytest.mark.parametrize("rough", [False, True])
@pytest.mark.parametrize("tuning", [(256, 8, 16, 0), (128, 8, 16, 0)])
def test_surface_batches_of_other_forms(tuning, rough):
    from radar_sounder_simulator_gb300.batch import CoherentBatch
    from radar_sounder_simulator_gb300.coherent import prepare_coherent
    f = _layer(20, 24, 9.0, 0.0, 1.5, 3)
    pos, uct = _track(9, 500.0)
    ph = np.exp(2j * np.pi * np.random.default_rng(1).random(len(f.areas)))
    pv = np.tile([0.0, 0.94, 0.34], (9, 1))

    def batch(n_samples, **opt):
        if rough:
            opt.update(d_phi_area=True, roughness=(
                0.1, 2.0, ph.astype(np.complex64), 12, "exponential"))
        return CoherentBatch([prepare_coherent(
            pos, uct, f.centers, f.normals, f.areas, f.e1, f.e2, k=K0,
            gamma=-0.3, t0=2 * 495.0 / C, dt=5e-9, n_samples=n_samples, c=C,
            precision="split", **opt)], tuning)
    # 48-100 KB of histograms, then forms with a few KB
    first = [batch(1400, taper_s=0.3), batch(30), batch(1300, split_sides=True),
             batch(40, pattern=("dipole", pv, np.float64(0.), np.float64(0.)))]
    for b in first + first[::-1]:
        _same(b)


@pytest.mark.parametrize("refraction", ["sequential", "joint"])
@pytest.mark.parametrize("rough", [False, True])
def test_refracted_batches_of_other_sizes(rough, refraction):
    from radar_sounder_simulator_gb300.batch import RefractedBatch
    from radar_sounder_simulator_gb300.multilayer import prepare_refracted
    top, bed = _layer(20, 24, 9.0, 0.0, 1.0, 3), _layer(18, 20, 9.0, -80.0,
                                                        1.5, 4)
    pos, uct = _track(9, 500.0)
    ph = np.exp(2j * np.pi * np.random.default_rng(1).random(len(bed.areas)))
    opt = {}
    if rough:
        opt.update(d_phi_area=True, roughness=(
            0.1, 2.0, ph.astype(np.complex64), 12, "exponential"))

    def batch(n_samples):
        return RefractedBatch([prepare_refracted(
            pos, uct, bed, [top], [1.0, 3.15], [0.0, 10.0], mode="coherent",
            refraction=refraction, k0=K0, gamma=0.2, t0=2 * 560.0 / C,
            dt=5e-9, n_samples=n_samples, c=C, precision="split", **opt)])
    first = [batch(1400), batch(60)]      # 87 and 4 KB of histograms
    for b in first + first[::-1]:
        _same(b)
