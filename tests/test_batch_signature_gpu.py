"""A tuned decomposition is kept by what was timed: batches whose options take
different kernels have different keys in the tuning cache."""

import pytest

from tests.test_short_paths_gpu import C, K0, _layer, _track

pytestmark = pytest.mark.gpu


def test_signature_tells_kernel_forms_apart():
    import numpy as np

    from radar_sounder_simulator_gb300.batch import CoherentBatch
    from radar_sounder_simulator_gb300.coherent import prepare_coherent
    f = _layer(20, 24, 9.0, 0.0, 1.5, 3)
    pos, uct = _track(9, 500.0)
    pv = np.tile([0.0, 0.94, 0.34], (9, 1))

    def batch(tuning=None, **opt):
        return CoherentBatch([prepare_coherent(
            pos, uct, f.centers, f.normals, f.areas, f.e1, f.e2, k=K0,
            gamma=-0.3, t0=2 * 495.0 / C, dt=5e-9, n_samples=64, c=C,
            precision="split", **opt)], tuning)
    plain = batch().signature()
    beam = batch(pattern=("dipole", pv, np.float64(0.), np.float64(0.)))
    keys = [plain, beam.signature(), batch(taper_s=0.3).signature()]
    assert len(set(map(repr, keys))) == 3
    # the same work has the same key, whatever it is prepared for
    assert batch((128, 4, 4, 0)).signature() == plain
