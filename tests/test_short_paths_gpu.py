"""The kernels' shorter paths at the sizes and options where they can go
wrong, against the float64 oracles: single-crossing and lean joint refracted
paths (both precisions), the surface sum's forms, small float64 calls,
frequency synthesis and transforms at ragged lengths, the incoherent bin
chain's constant quotients, the packed focus pairs, and the drop-in call's
packed staging.

Tolerances are the ones the kernels' other tests hold: float64 form within
1e-9 of the peak; split form relative L2 1e-4, phase 1e-3 rad, power 0.01 dB
above -60 dB (each fifty times what float32 rounding of a path leaves);
incoherent 1e-5 with the same occupied bins.
"""

import numpy as np
import pytest

from oracle import incoherent as oi
from oracle import lpa
from oracle import multifreq as omf
from oracle import processing as op
from oracle import refracted as oref
from oracle import waveform as owf
from tests.util import field_errors

pytestmark = pytest.mark.gpu
C = 299792458.0
K0 = 2 * np.pi * 60e6 / C


def _layer(ny, nx, d, z0, rms, seed, flip=False):
    from radar_sounder_simulator_gb300.scenes import (facets_from_vertices,
                                                      random_field)
    n = max(ny, nx) + 1
    Z = z0 + random_field(n, d, 12 * d, rms, np.random.default_rng(seed))
    X, Y = np.meshgrid((np.arange(nx + 1) - 0.47 * nx) * d,
                       (np.arange(ny + 1) - 0.52 * ny) * d)
    f = facets_from_vertices(X, Y, Z[:ny + 1, :nx + 1])
    if flip:
        f.normals = -f.normals
    return f


def _track(T, z, step=9.0):
    s = (np.arange(T) - T / 2.2) * step
    pos = np.column_stack([s, 0.2 * s + 3.0, z + 0.3 * np.sin(s)])
    return pos, np.tile([0.2, -0.98, 0.0], (T, 1))


def _split_ok(got, ref):
    e = field_errors(got, ref)
    assert e["rel_l2"] <= 1e-4 and e["phase_rad"] <= 1e-3, e
    assert e["power_db"] <= 0.01, e


PATHS = [
    # T, crossings, joint, options
    (1, 1, False, {}),
    (9, 1, False, dict(pattern=True, split_sides=True)),
    (3, 1, False, dict(crossed_sigma=[0.05], taper_s=0.2)),
    (5, 1, False, dict(eps=[1.5, 1.0, 2.0])),     # dense above rare
    (5, 1, False, dict(extra=True)),               # a leg below: general path
    (3, 1, False, dict(flip=True)),                # downward normals
    (2, 1, True, {}),
    (3, 2, True, dict(flip=True)),
    (9, 2, True, dict(pattern=True)),
    (3, 3, True, dict(pad_to=4)),
    (5, 4, True, dict(split_sides=True)),
    (5, 2, True, dict(joint_newton=2)),            # budget: general path
    (5, 2, True, dict(joint_newton=3)),            # split lean, FP64 general
    (4, 2, False, {}),                             # chain, float32 lookups
]


@pytest.mark.parametrize("precision", ["split", "fp64"])
@pytest.mark.parametrize("T,ni,joint,opt", PATHS)
def test_refracted_paths_match_oracle(T, ni, joint, opt, precision):
    if precision == "split" and opt.get("joint_newton") == 2:
        pytest.skip("the split form's validity bound is wider than float64's")
    from radar_sounder_simulator_gb300.multilayer import refracted_cluttergram
    opt = dict(opt)
    n, flip = 23, opt.pop("flip", False)
    layers = [_layer(n, n + 4, 13.0, -60.0 * j, 1.0, 40 + j, flip)
              for j in range(ni)]
    bed = _layer(n - 3, n + 6, 11.0, -60.0 * ni - 40.0, 2.0, 60)
    eps = opt.pop("eps", [1.0, 1.7, 2.4, 2.9, 3.15][:ni + 1])[:ni + 1]
    att = [0.0, 8.0, 12.0, 15.0, 20.0][:ni + 1]
    if opt.pop("extra", False):
        layers.append(_layer(n, n, 13.0, -60.0, 1.0, 41))
        eps, att = [1.0, 1.7, 2.4], [0.0, 8.0, 12.0]
    pos, uct = _track(T, 700.0)
    kw = dict(mode="coherent", t0=2 * 690.0 * np.sqrt(eps[0]) / C, dt=1.2e-8, n_samples=150,
              c=C, gamma=0.2, k0=K0,
              refraction="joint" if joint else "sequential")
    if opt.pop("pattern", False):
        pv = np.tile([0.0, 0.94, 0.34], (T, 1))
        kw["pattern"] = ("dipole", pv, np.float64(0.0), np.float64(0.0))
    kw.update(opt)
    ref, drop = oref.refracted_cluttergram(pos, uct, bed, layers, eps, att,
                                           **kw)
    got, gd = refracted_cluttergram(pos, uct, bed, layers, eps, att, **kw,
                                    precision=precision,
                                    out_dtype=np.complex128)
    if precision == "fp64":
        assert np.abs(got - ref).max() <= 1e-9 * np.abs(ref).max()
    else:
        _split_ok(got, ref)


@pytest.mark.parametrize("eps", [[1.0, 3.15, 5.0], [2.0, 1.0, 3.0],
                                 [1.0, 1.05, 1.1]])
@pytest.mark.parametrize("ni,refraction", [(1, "sequential"), (1, "joint"),
                                           (2, "sequential"), (2, "joint")])
@pytest.mark.parametrize("alt", [50.0, 140.0])
def test_flat_rays_match_oracle(alt, ni, refraction, eps):
    """A platform 50 m over a scene a kilometre wide: rays near grazing and
    the critical angle, where the reference's ten lookup iterations end short
    of their root and pick other cells."""
    from radar_sounder_simulator_gb300.multilayer import refracted_cluttergram
    layers = [_layer(24, 29, 40.0, -30.0 * j, 8.0 if j == 0 else 2.4, 70 + j)
              for j in range(ni)]
    bed = _layer(20, 26, 41.0, -30.0 * ni - 30.0, 8.0, 90)
    pos, uct = _track(3, alt, step=50.0)
    args = (pos, uct, bed, layers, eps[:ni + 1], [0.0, 1.0, 1.0][:ni + 1])
    kw = dict(mode="coherent", t0=0.0, dt=4e-8, n_samples=600, c=C,
              gamma=0.2, k0=K0, refraction=refraction)
    ref, _ = oref.refracted_cluttergram(*args, **kw)
    for precision in ("fp64", "split"):
        got, _ = refracted_cluttergram(*args, **kw, precision=precision,
                                       out_dtype=np.complex128)
        if precision == "fp64":
            assert np.abs(got - ref).max() <= 1e-9 * np.abs(ref).max()
        else:
            assert field_errors(got, ref)["rel_l2"] <= 1e-4


SURFACE = [
    dict(), dict(pattern=True), dict(taper_s=0.3, split_sides=True),
    dict(interp_bins=True), dict(pattern=True, interp_bins=True)]


@pytest.mark.parametrize("precision", ["split", "fp64"])
@pytest.mark.parametrize("T,ny,nx", [(1, 9, 7), (7, 31, 18), (10, 64, 65)])
def test_surface_forms_match_oracle_and_batch(T, ny, nx, precision):
    """Every form of the surface sum by itself, and all of them in one batch
    (which then takes the widest)."""
    from radar_sounder_simulator_gb300.batch import CoherentBatch
    from radar_sounder_simulator_gb300.coherent import prepare_coherent
    f = _layer(ny, nx, 9.0, 0.0, 1.5, ny)
    pos, uct = _track(T, 500.0)
    q = [np.asarray(v, np.float32).astype(np.float64)
         for v in (f.centers, f.normals, f.areas, f.e1, f.e2)]
    plans, refs = [], []
    for opt in SURFACE:
        kw = dict(opt)
        if kw.pop("pattern", False):
            pv = np.tile([0.0, 0.94, 0.34], (T, 1))
            kw["pattern"] = ("dipole", pv, np.float64(0.0), np.float64(0.0))
        kw.update(k=K0, gamma=-0.3, t0=2 * 495.0 / C, dt=5e-9, n_samples=90,
                  c=C)
        refs.append(lpa.coherent_cluttergram(pos, uct, *q, **kw)[0])
        plans.append(prepare_coherent(pos, uct, f.centers, f.normals, f.areas,
                                      f.e1, f.e2, precision=precision, **kw))

    def check(out, which=slice(None)):
        for p, (field, drop), ref in zip(plans[which], out, refs[which]):
            got = p.to_numpy(field, drop, np.complex128)[0]
            if precision == "fp64":
                assert np.abs(got - ref).max() <= 1e-9 * np.abs(ref).max()
            else:
                _split_ok(got, ref)
    check([p.run() for p in plans])
    check(CoherentBatch(plans).run())
    check(CoherentBatch(plans[:1]).run(), slice(0, 1))
    check(CoherentBatch(plans[:2]).run(), slice(0, 2))


@pytest.mark.parametrize("B,taps", [(1, 3), (3, 2), (5, 9), (17, 33)])
def test_short_transforms(B, taps):
    """Two to 64-point transforms against the direct sum."""
    from radar_sounder_simulator_gb300.waveform import compress_tensor
    import torch
    rng = np.random.default_rng(B)
    x = (rng.normal(size=(3, B)) + 1j * rng.normal(size=(3, B))).astype(
        np.complex64)
    p = rng.normal(size=taps) + 1j * rng.normal(size=taps)
    y = compress_tensor(torch.as_tensor(x, device="cuda"), p, taps // 2,
                        method="fft", precision="split").cpu().numpy()
    ref = owf.convolve_fast_time(x, p, taps // 2)
    # one float32 rounding of each result, plus the double-float transforms
    assert np.abs(y - ref).max() <= 2.0 ** -23 * np.abs(ref).max()


@pytest.mark.parametrize("K,B", [(17, 33), (255, 1), (1023, 96), (1025, 41)])
def test_band_synthesis_at_ragged_lengths(K, B):
    from radar_sounder_simulator_gb300.multifreq import multifreq_traces
    f = _layer(9, 7, 25.0, 0.0, 1.0, 5)
    pos, _ = _track(3, 900.0)
    cols = (f.centers, f.normals, f.areas, f.e1, f.e2)
    r0 = np.linalg.norm(pos[0] - f.centers, axis=1).min()
    tw = 2 * r0 / C - 2e-7 + np.arange(B) / 30e6
    kw = dict(gamma=-0.3, f0=60e6, bandwidth=15e6, c=C, twtt=tw, n_freq=K,
              freeze_amplitudes=True)
    y = multifreq_traces(pos, *cols, precision="split", check_alias=False,
                         **kw)
    q = [np.asarray(v, np.float32).astype(np.float64) for v in cols]
    ref = np.array([omf.multifreq_profile(p, *q, **kw) for p in pos])
    _split_ok(y, ref)


@pytest.mark.parametrize("c", [C, 16777215.0 * 8, 2.0 ** 28])
@pytest.mark.parametrize("dt", [2e-9, 1.0 / 30e6, 2.0 ** -26])
def test_incoherent_bins_with_any_constants(c, dt):
    """Bins are the reference's float32 chain for wave speeds and bin widths
    of any mantissa: all ones (no fast quotient), a power of two, odd."""
    from radar_sounder_simulator_gb300.incoherent import (
        incoherent_cluttergram)
    rng = np.random.default_rng(7)
    n = 5000
    cen = np.column_stack([rng.uniform(-900, 900, n),
                           rng.uniform(-900, 900, n), np.zeros(n)])
    pos = np.array([[0.0, 0.0, 2000.0], [3.0, 9.0, 2001.0],
                    [-8.0, 1.0, 1999.0]])
    t0 = 2 * 1990.0 / c
    # facets moved onto bin edges of the first trace, where chains differ
    r = np.linalg.norm(pos[0] - cen, axis=1)
    u = np.round((2 * r / c - t0) / dt) + rng.uniform(-3e-4, 3e-4, n)
    rt = np.maximum((u * dt + t0) * c / 2, 1995.0)
    cen[:, 2] = 2000.0 - np.sqrt(np.maximum(
        rt ** 2 - cen[:, 0] ** 2 - cen[:, 1] ** 2, 1.0))
    nrm = np.tile([0.0, 0.0, 1.0], (n, 1))
    area = 10.0 * 1.013 ** (np.arange(n) % 700)   # a moved facet shows
    uct = np.tile([0.0, -1.0, 0.0], (3, 1))
    kw = dict(t0=t0, dt=dt, n_samples=777, c=c)
    got, gd = incoherent_cluttergram(pos, uct, cen, nrm, area, **kw)
    ref, rd = oi.incoherent_cluttergram(pos, uct, cen, nrm, area, **kw)
    np.testing.assert_array_equal(got > 0, ref > 0)
    assert np.abs(got - ref).max() <= 1e-5 * np.abs(ref).max()
    keep = ref > 0
    assert np.all(np.abs(got - ref)[keep] <= 1e-4 * ref[keep])


@pytest.mark.parametrize("T,nb", [(1, 3), (7, 257), (17, 40)])
def test_focus_pairs_and_zero_delay(T, nb):
    """Odd trace counts (half-used pairs), a window that opens at zero delay,
    empty rows, and amplitudes whose squares leave float32's range."""
    from radar_sounder_simulator_gb300 import processing as gp
    rng = np.random.default_rng(T)
    pos = np.column_stack([np.arange(T) * 2.0, np.zeros(T), np.full(T, 50.)])
    twtt = np.arange(nb) * 1e-8
    for scale in (1.0, 1e-25, 1e25):
        F = scale * (rng.standard_normal((T, nb)) +
                     1j * rng.standard_normal((T, nb))).astype(np.complex64)
        F[T // 2] = 0
        F = F.astype(np.complex64)
        out, pw = gp.focus_field(F, twtt, pos, wavelength=3.0,
                                 aperture_m=8.0, precision="split")
        o64, _ = op.focused_sar(F, twtt, pos, 3.0, 8.0, "hann")
        assert np.abs(out - o64).max() <= 1e-4 * np.abs(o64).max()
        m = np.abs(out.astype(np.complex128)).astype(np.float32)
        with np.errstate(over="ignore", under="ignore"):
            np.testing.assert_allclose(pw, m * m, rtol=4e-7)


@pytest.mark.parametrize("opt", [
    {}, dict(split_sides=True), dict(block_size=32), dict(pattern=True),
    dict(n_samples=20), dict(window_cull=False)])
def test_drop_in_call_equals_plan(opt):
    """The drop-in's packed transfers give what the plan's device tensors
    hold, with and without window offsets (a short window culls blocks)."""
    from radar_sounder_simulator_gb300.coherent import (coherent_cluttergram,
                                                        prepare_coherent)
    T = 5
    f = _layer(24, 71, 12.0, 0.0, 1.0, 3)
    pos, uct = _track(T, 100.0, step=60.0)
    kw = dict(k=K0, gamma=-0.3, t0=2 * 95.0 / C, dt=1e-8, n_samples=64, c=C,
              block_size=64)
    opt = dict(opt)
    if opt.pop("pattern", False):
        pv = np.tile([0.0, 0.94, 0.34], (T, 1))
        kw["pattern"] = ("dipole", pv, np.float64(0.0), np.float64(0.0))
    kw.update(opt)
    args = (pos, uct, f.centers, f.normals, f.areas, f.e1, f.e2)
    plan = prepare_coherent(*args, **kw)
    field, drop = plan.run()
    for dtype in (np.complex64, np.complex128):
        got, gd = coherent_cluttergram(*args, **kw, out_dtype=dtype)
        want, wd = plan.to_numpy(field, drop, dtype)
        assert got.shape == want.shape and got.dtype == want.dtype
        # float64 sums in another order, then one rounding
        tol = 1e-12 if dtype == np.complex128 else 1.2e-7
        assert np.abs(got - want).max() <= tol * np.abs(want).max()
        np.testing.assert_allclose(gd, wd, rtol=2e-7)
    q = [np.asarray(v, np.float32).astype(np.float64) for v in args[2:]]
    kw.pop("block_size"), kw.pop("window_cull", None)
    ref = lpa.coherent_cluttergram(pos, uct, *q, **kw)[0]
    assert np.abs(got - ref).max() <= 1e-9 * np.abs(ref).max()
