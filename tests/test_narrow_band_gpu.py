"""Frequency synthesis (split form) of narrow bands and of long paths. The band response's CTA
is as wide as the band, down to two threads, so its shared tables -- four
traces, 32 Faddeeva coefficients -- take several turns to fill; a carrier phase of
millions of radians has a low part that no longer is small. Against the
float64 oracle within the split form's bounds (relative L2 1e-4, phase 1e-3
rad, power 0.01 dB above -60 dB of the peak)."""

import numpy as np
import pytest

from oracle import lpa
from oracle import multifreq as omf
from tests.test_multifreq_gpu import C, _scene, q32, split_ok

pytestmark = pytest.mark.gpu

ROUGH = {"smooth": None, "gaussian": (0.2, 3.0, 40, "gaussian", False),
         "gaussian_area": (0.2, 3.0, 40, "gaussian", True),
         "exponential_area": (0.2, 3.0, 40, "exponential", True)}


@pytest.mark.parametrize("kind", list(ROUGH) + ["full"])
@pytest.mark.parametrize("K", [1, 16, 17, 100, 128, 240, 300])
def test_narrow_band_matches_oracle(K, kind):
    from types import SimpleNamespace
    from radar_sounder_simulator_gb300.multifreq import multifreq_traces
    c, nr, a, e1, e2 = _scene(n=9, seed=K)
    f = SimpleNamespace(centers=c, normals=nr, areas=a, e1=e1, e2=e2)
    T = 9
    pos = np.column_stack([np.linspace(-80, 70, T), np.full(T, -5.0),
                           np.full(T, 800.0)])
    tw = 2 * 795.0 / C + np.arange(24) / 30e6
    kw = dict(f0=60e6, bandwidth=15e6, c=C, twtt=tw, n_freq=K)
    q = q32(f)
    k0 = 2 * np.pi * kw["f0"] / C
    frozen, rough, opt, r = kind != "full", None, {}, ROUGH.get(kind)
    if r:
        ph = np.exp(2j * np.pi * np.random.default_rng(K).random(len(c)))
        rough = (r[0], r[1], ph.astype(np.complex64), r[2], r[3])
        opt = dict(roughness=rough, d_phi_area=r[4])
    y = multifreq_traces(pos, c, nr, a, e1, e2, gamma=-0.3, precision="split",
                         freeze_amplitudes=frozen, check_alias=False, **opt,
                         **kw)
    ref = []
    for p in pos:
        if frozen:
            if rough:
                c0, rng = lpa.rough_lpa_field(
                    p, *q, k0, -0.3, r[0], r[1],
                    rough[2].astype(np.complex128), r[2], area_only=r[4],
                    acf=r[3])
            else:
                c0, rng = lpa.lpa_field(p, *q, k0, -0.3)
            ref.append(omf.synth_frozen(rng, c0 * np.exp(2j * k0 * rng),
                                        **kw))
        else:
            freqs = omf.band_frequencies(kw["f0"], kw["bandwidth"], K)
            w = omf.window_weights(freqs, kw["f0"], kw["bandwidth"], "hann")
            H = np.array([lpa.lpa_field(p, *q, 2 * np.pi * v / C, -0.3)[0]
                          .sum() for v in freqs])
            ref.append((w / w.sum() * H) @ np.exp(
                2j * np.pi * np.outer(freqs - kw["f0"], tw)))
    split_ok(y, np.array(ref))


@pytest.mark.parametrize("frozen", [True, False])
@pytest.mark.parametrize("alt,f0", [(25e3, 450e6), (400e3, 150e6),
                                    (500e3, 1.3e9), (800e3, 5e9)])
def test_long_paths_match_oracle(alt, f0, frozen):
    """Carrier phases of 5e5, 2.5e6, 2.7e7 and 1.7e8 rad."""
    from types import SimpleNamespace
    from radar_sounder_simulator_gb300.multifreq import multifreq_traces
    c, nr, a, e1, e2 = _scene(n=9, d=2.0, seed=4)
    f = SimpleNamespace(centers=c, normals=nr, areas=a, e1=e1, e2=e2)
    pos = np.column_stack([np.linspace(-80, 70, 3), np.full(3, -5.0),
                           np.full(3, alt)])
    tw = 2 * (alt - 8.0) / C + np.arange(24) / 30e6
    kw = dict(gamma=-0.3, f0=f0, bandwidth=15e6, c=C, twtt=tw, n_freq=64,
              freeze_amplitudes=frozen)
    y = multifreq_traces(pos, c, nr, a, e1, e2, precision="split", **kw)
    ref = np.array([omf.multifreq_profile(p, *q32(f), **kw) for p in pos])
    split_ok(y, ref)
