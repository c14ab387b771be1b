"""The work that users of this framework have it do, as timed cases.

A case is a call, or a short chain of calls, of the public entry points on a
seeded synthetic scene: the drop-in NumPy call, a device-resident plan run
again and again, a batch of jobs, one gradient step of an inversion. Scene
statistics (50 m-rms exponential surfaces, an ice column with two weak
horizons over a bed, firn index, attenuation, bands, pulse, aperture) are
those of the repository's benchmark configurations; sizes run from one small
call to the benchmark's 512^2 facets x 1024 traces.

Single-precision results are handed on as the drop-in calls hand them on
(complex64 fields, float32 powers and dropped power); the float64 form's are
left in float64.

``exact`` restates every case in float64 with plain torch operations: the
facet field, the refracted path as two-point Snell solves and a Newton solve
of the joint stationarity, the roughness series, pulse compression,
backprojection, frequency synthesis, and the gradient of windowed power.
The dropped power of the culled kernels depends on which out-of-window facets
a trace's culling window happens to hold, so it has no value of its own.
"""

import math
from types import SimpleNamespace

import numpy as np
import torch

C = 299792458.0
EPS_LEG = [1.0, 2.6, 3.15, 3.15315]     # air, firn, ice, ice below a horizon
ATT_LEG = [0.0, 10.0, 10.0, 10.0]       # dB/km, two-way
DEPTHS = [0.0, -300.0, -1200.0, -2500.0]
RELIEF = [(20.0, 5000.0), (5.0, 1000.0), (5.0, 1000.0), (300.0, 5000.0)]


# --------------------------------------------------------------------------
# the cases
# --------------------------------------------------------------------------
def listed():
    return [
        # One small drop-in call on NumPy arrays with default options (the
        # float64 form): what a script or notebook does first, and what a
        # unit of a parameter study costs when it is not batched.
        dict(name="call_64sq_fp64", kind="surface", api="call", ny=64, nx=64,
             spacing=25.0, traces=32, step=20.0, bins=512, f0=60e6,
             alt=3000.0, precision="fp64", sides=False, rough=False,
             pattern="none", then="field"),
        # The plain single-surface run (the benchmark's first configuration)
        # from a device-resident plan, with pulse compression of its output:
        # a latency-sized step that sweeps repeat.
        dict(name="plain_128sq_chirp", kind="surface", api="plan", ny=128,
             nx=128, spacing=100.0, traces=256, step=50.0, bins=2048,
             f0=60e6, alt=20000.0, precision="split", sides=False,
             rough=False, pattern="none", then="chirp"),
        # A full-size surface radargram and the two processing steps behind
        # it: facet sum, range compression, focused SAR.
        dict(name="radargram_512sq_sar", kind="surface", api="plan", ny=512,
             nx=512, spacing=50.0, traces=1024, step=25.0, bins=2048,
             f0=60e6, alt=20000.0, precision="split", sides=False,
             rough=False, pattern="none", then="focus"),
        # A ragged design-sweep batch: surfaces of several sizes, bands and
        # tabulated beams through one persistent launch.
        dict(name="sweep_batch_6", kind="batch", jobs=6, ny=301, nx=256,
             spacing=25.0, traces=333, step=25.0, bins=2048, f0=60e6,
             alt=15000.0, rough=False),
        # The float64 form (the default precision) of the surface sum, left
        # and right of the track kept apart, from a plan.
        dict(name="surface_256sq_fp64", kind="surface", api="plan", ny=256,
             nx=256, spacing=50.0, traces=100, step=25.0, bins=1024,
             f0=60e6, alt=20000.0, precision="fp64", sides=True, rough=False,
             pattern="dipole", then="field"),
        # The first horizon of the multilayer scene: one crossing, the
        # sequential solve, at full size.
        dict(name="horizon_512sq_seq", kind="refracted", ny=512, nx=512,
             spacing=50.0, traces=1024, step=25.0, bins=2048, f0=60e6,
             alt=20000.0, crossed=1, joint=False, precision="split",
             rough=False),
        # The bed of the multilayer scene under three crossings, the joint
        # solve: the largest share of the benchmark's step.
        dict(name="bed_512sq_joint3", kind="refracted", ny=512, nx=512,
             spacing=50.0, traces=1024, step=25.0, bins=2048, f0=60e6,
             alt=20000.0, crossed=3, joint=True, precision="split",
             rough=False),
        # A rough bed (per-facet rms height and correlation length, taper)
        # of the multi-band configuration, one band.
        dict(name="rough_bed_400_150mhz", kind="refracted", ny=411, nx=400,
             spacing=25.0, traces=500, step=25.0, bins=1000, f0=150e6,
             alt=20000.0, crossed=1, joint=False, precision="split",
             rough=True),
        # The default precision of the refracted drop-in, the joint solve
        # through two crossings, at the size a float64 check run takes.
        dict(name="horizon2_120x96_fp64", kind="refracted", ny=96, nx=120,
             spacing=50.0, traces=40, step=25.0, bins=1024, f0=60e6,
             alt=20000.0, crossed=2, joint=True, precision="fp64",
             rough=False),
        # One step of an inversion for bed reflectivity, roughness and
        # attenuation: windowed power, dB misfit, its gradient.
        dict(name="inversion_256sq", kind="adjoint", ny=256, nx=256,
             spacing=25.0, traces=512, step=12.5, bins=1024, f0=60e6,
             alt=20000.0),
        # Frequency-sampled synthesis of every trace of a short track.
        dict(name="modef_128x96_k768", kind="modef", ny=96, nx=128,
             spacing=100.0, traces=100, step=50.0, bins=1024, n_freq=768,
             f0=60e6, alt=20000.0),
        # Incoherent (power) radargram at full size.
        dict(name="incoherent_512sq", kind="incoherent", ny=512, nx=512,
             spacing=50.0, traces=1024, step=25.0, bins=2048, f0=60e6,
             alt=20000.0, sides=False),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: a kind, then sizes spread over the listed range, odd
    ones among them."""
    kind = rng.choice(["surface", "surface", "surface", "refracted",
                       "refracted", "refracted", "refracted", "batch",
                       "adjoint", "modef", "incoherent"])
    f0 = rng.choice([30e6, 60e6, 60e6, 150e6, 195e6, 450e6])
    alt = float(rng.randrange(12000, 25001, 500))
    spacing = rng.choice([25.0, 50.0]) if f0 < 100e6 else 25.0
    step = rng.choice([12.5, 25.0])
    bins = _log(rng, 512, 2048)
    ny, nx = _log(rng, 64, 512), _log(rng, 64, 512)
    traces = _log(rng, 32, 1024)
    if kind == "surface":
        fp64 = rng.random() < 0.3
        if fp64:
            ny, nx, traces = (_log(rng, 48, 256), _log(rng, 48, 256),
                              _log(rng, 16, 200))
        rough = rng.random() < 0.4 and not fp64
        return dict(kind=kind, api=rng.choice(["plan", "plan", "call"]),
                    ny=ny, nx=nx, spacing=spacing, traces=traces, step=step,
                    bins=bins, f0=f0, alt=alt,
                    precision="fp64" if fp64 else "split",
                    sides=rng.random() < 0.25, rough=rough,
                    pattern=rng.choice(["none", "none", "dipole", "beam"]),
                    then="field" if fp64 else
                    rng.choice(["field", "chirp"]))
    if kind == "refracted":
        crossed = rng.choice([1, 1, 2, 3])
        fp64 = rng.random() < 0.25
        if fp64:
            ny, nx, traces = (_log(rng, 32, 110), _log(rng, 32, 128),
                              _log(rng, 8, 48))
        rough = crossed == 1 and not fp64 and rng.random() < 0.5
        return dict(kind=kind, ny=ny, nx=nx, spacing=spacing, traces=traces,
                    step=step, bins=bins, f0=f0, alt=alt, crossed=crossed,
                    joint=crossed > 1, precision="fp64" if fp64 else "split",
                    rough=rough)
    if kind == "batch":
        return dict(kind=kind, jobs=rng.randrange(2, 9),
                    ny=_log(rng, 64, 320), nx=_log(rng, 64, 320),
                    spacing=25.0, traces=_log(rng, 32, 512), step=25.0,
                    bins=bins, f0=60e6, alt=alt, rough=rng.random() < 0.4)
    if kind == "adjoint":
        # the line stays over the scene it inverts
        ny, nx = _log(rng, 64, 300), _log(rng, 64, 300)
        return dict(kind=kind, ny=ny, nx=nx, spacing=25.0, traces=traces,
                    step=min(12.5, 25.0 * nx / traces),
                    bins=max(bins, 800), f0=rng.choice([60e6, 150e6]),
                    alt=alt)
    if kind == "modef":
        return dict(kind=kind, ny=_log(rng, 32, 128), nx=_log(rng, 32, 128),
                    spacing=100.0, traces=_log(rng, 16, 128), step=50.0,
                    bins=_log(rng, 256, 1024), n_freq=rng.randrange(200, 1025),
                    f0=60e6, alt=20000.0)
    return dict(kind=kind, ny=ny, nx=nx, spacing=spacing, traces=traces,
                step=step, bins=bins, f0=f0, alt=alt,
                sides=rng.random() < 0.3)


# --------------------------------------------------------------------------
# seeded inputs (host arrays, as a scene builder hands them over)
# --------------------------------------------------------------------------
def _layer(ny, nx, spacing, rms, corr, z0, rng):
    """ny x nx facets of a random surface with exponential correlation:
    mean edges, corner mean, upward normal."""
    my, mx = ny + 1, nx + 1
    ky = 2 * np.pi * np.fft.fftfreq(my, spacing)
    kx = 2 * np.pi * np.fft.rfftfreq(mx, spacing)
    full = 2 * np.pi * np.fft.fftfreq(mx, spacing)
    def spec(k2):
        return (1.0 + k2 * corr ** 2) ** -1.5
    h = np.sqrt(spec(ky[:, None] ** 2 + kx[None] ** 2))
    power = np.mean(spec(ky[:, None] ** 2 + full[None] ** 2))
    w = rng.standard_normal((my, mx))
    z = z0 + rms * np.fft.irfft2(np.fft.rfft2(w) * h, s=(my, mx)) / \
        math.sqrt(power)
    x = (np.arange(mx) - nx / 2.0) * spacing
    y = (np.arange(my) - ny / 2.0) * spacing
    za, zb, zc, zd = z[:-1, :-1], z[:-1, 1:], z[1:, :-1], z[1:, 1:]
    n = ny * nx
    e1 = np.zeros((n, 3))
    e2 = np.zeros((n, 3))
    cen = np.empty((n, 3))
    e1[:, 0] = spacing
    e1[:, 2] = (((zb + zd) - (za + zc)) / 2.0).ravel()
    e2[:, 1] = spacing
    e2[:, 2] = (((zc + zd) - (za + zb)) / 2.0).ravel()
    cen[:, 0] = np.broadcast_to(0.5 * (x[:-1] + x[1:]), (ny, nx)).ravel()
    cen[:, 1] = np.broadcast_to(0.5 * (y[:-1] + y[1:])[:, None],
                                (ny, nx)).ravel()
    cen[:, 2] = ((za + zb + zc + zd) / 4.0).ravel()
    raw = np.stack([-e1[:, 2] * spacing, -e2[:, 2] * spacing,
                    np.full(n, spacing * spacing)], 1)
    area = np.sqrt((raw * raw).sum(1))
    cell = np.stack([np.repeat(np.arange(ny), nx),
                     np.tile(np.arange(nx), ny)], 1)
    return SimpleNamespace(centers=cen, normals=raw / area[:, None],
                           areas=area, e1=e1, e2=e2, cell=cell,
                           grid_shape=(ny, nx), phase_keys=None)


def _track(case, rng):
    """A nearly straight flight line: heading within a few degrees of +x,
    a cross-track offset, a slow wander of a few metres."""
    n = case["traces"]
    s = (np.arange(n) - (n - 1) / 2.0) * case["step"]
    a = math.radians(rng.uniform(-4.0, 4.0))
    ph = rng.uniform(0.0, 2 * np.pi, 2)
    lat = rng.uniform(-300.0, 300.0) + 3.0 * np.sin(2 * np.pi * s / 4000.0 +
                                                    ph[0])
    z = case["alt"] + 2.0 * np.sin(2 * np.pi * s / 3000.0 + ph[1])
    pos = np.column_stack([s * math.cos(a) - lat * math.sin(a),
                           s * math.sin(a) + lat * math.cos(a), z])
    uct = np.tile([math.sin(a), -math.cos(a), 0.0], (n, 1))
    return pos, uct


def _speckle(n, rng):
    return ((rng.standard_normal(n) + 1j * rng.standard_normal(n)) /
            math.sqrt(2.0)).astype(np.complex64)


def _fresnel(e1, e2):
    a, b = math.sqrt(e1), math.sqrt(e2)
    return (a - b) / (a + b)


def _terms(x):
    return int(np.clip(math.ceil(x + 6.0 * math.sqrt(x) + 5.0), 10, 300))


def _window(pos, f, f0, frac=0.25, eps=(), tops=()):
    """Start and sample spacing of a window for a band of ``frac`` x f0: it
    opens 200 m before the target's nearest return, taken along straight
    rays with the excess path of the media (``eps`` below each of ``tops``)
    down to each facet."""
    dt = 1.0 / (2.0 * frac * f0)
    cen = f.centers[::97]
    r = np.linalg.norm(pos[::max(1, len(pos) // 64), None] - cen[None],
                       axis=-1)
    floors = list(tops[1:]) + [-np.inf]
    for e, top, floor in zip(eps, tops, floors):
        r = r + (math.sqrt(e) - 1.0) * np.maximum(
            0.0, top - np.maximum(cen[:, 2], floor))
    return 2.0 * (r.min() - 200.0) / C, dt


def _pattern(kind, n, lean=0.0):
    """The antenna tuple of the calls: a cross-track-tilted dipole or a
    60-degree Gaussian beam tabulated on 64 angles, boresight near nadir."""
    if kind == "dipole":
        return ("dipole", np.tile([0.0, 1.0, 0.0], (n, 1)), 0.0, 0.0)
    if kind == "beam":
        th = np.linspace(0.0, np.pi / 2, 64)
        g = 2.0 ** (-((th / np.radians(30.0 + 10.0 * lean)) ** 2) / 4.0)
        return ("tabulated", np.tile([0.0, 0.0, -1.0], (n, 1)), th, g)
    return None


def _surface_inputs(case, seed, job=0):
    rng = np.random.default_rng([seed, job, 11])
    f = _layer(case["ny"], case["nx"], case["spacing"], 50.0, 1000.0, 0.0,
               rng)
    pos, uct = _track(case, rng)
    t0, dt = _window(pos, f, case["f0"])
    k = 2 * np.pi * case["f0"] / C
    kw = dict(k=k, gamma=_fresnel(1.0, 3.15), t0=t0, dt=dt,
              n_samples=case["bins"], c=C)
    if case.get("sides"):
        kw["split_sides"] = True
    pat = _pattern(case.get("pattern", "none"), len(pos), 0.5 * job)
    if pat is not None:
        kw["pattern"] = pat
    if case.get("rough"):
        n = len(f.centers)
        sig = rng.uniform(0.05, 0.5, n)
        kw.update(roughness=(sig, rng.uniform(5.0, 50.0, n),
                             _speckle(n, rng),
                             _terms((2 * k * sig.max()) ** 2),
                             "exponential"),
                  taper_s=0.05, d_phi_area=True)
    return SimpleNamespace(f=f, pos=pos, uct=uct, kw=kw, f0=case["f0"])


def _batch_inputs(case, seed):
    """Jobs of a design sweep: sizes, tracks, bands and beams differ. The
    sizes and bands belong to the case, the scenes to the seed."""
    rng = np.random.default_rng([case["ny"], case["nx"], case["traces"],
                                 case["jobs"], 12])
    jobs = []
    for j in range(case["jobs"]):
        one = dict(case, ny=max(16, int(case["ny"] * rng.uniform(0.5, 1.0))),
                   nx=max(16, int(case["nx"] * rng.uniform(0.5, 1.0))),
                   traces=max(4, int(case["traces"] * rng.uniform(0.4, 1.0))),
                   alt=case["alt"] * rng.uniform(0.9, 1.1),
                   f0=float(np.exp(rng.uniform(math.log(30e6),
                                               math.log(450e6)))),
                   pattern="none" if case["rough"] else "beam")
        jobs.append(_surface_inputs(one, seed, job=j + 1))
    return jobs


def _stack(case, seed, tag):
    """The ice column down to the target: crossed interfaces, target, leg
    permittivities and attenuation rates, track."""
    rng = np.random.default_rng([seed, tag])
    nc = case.get("crossed", 1)
    if case.get("rough") or case["kind"] == "adjoint":
        # an ice column over a rough bed: the multilayer scene's surface,
        # the roughness configuration's bed
        layers = [_layer(case["ny"], case["nx"], case["spacing"], rms, corr,
                         z, rng) for rms, corr, z in (
                             RELIEF[0] + (0.0,), (50.0, 1000.0, -1000.0))]
        eps, att = [1.0, 3.15], [0.0, 10.0]
    else:
        layers = [_layer(case["ny"], case["nx"], case["spacing"], *RELIEF[j],
                         DEPTHS[j], rng) for j in range(nc + 1)]
        eps, att = EPS_LEG[:nc + 1], ATT_LEG[:nc + 1]
    pos, uct = _track(case, rng)
    t0, dt = _window(pos, layers[-1], case["f0"],
                     0.15 if case.get("rough") else 0.25, eps[1:],
                     DEPTHS[:len(layers) - 1])
    return rng, layers[:-1], layers[-1], eps, att, pos, uct, t0, dt


def _refracted_inputs(case, seed):
    rng, crossed, target, eps, att, pos, uct, t0, dt = _stack(case, seed, 13)
    k0 = 2 * np.pi * case["f0"] / C
    n = len(target.centers)
    kw = dict(mode="coherent", t0=t0, dt=dt, n_samples=case["bins"], c=C,
              k0=k0, refraction="joint" if case["joint"] else "sequential")
    if case["rough"]:
        sig = np.exp(math.log(0.3) + 0.7 * rng.standard_normal(n))
        nt = _terms((2 * k0 * math.sqrt(eps[-1]) *
                     np.quantile(sig, 0.999)) ** 2)
        kw.update(gamma=_fresnel(eps[-1], 9.0), taper_s=0.05,
                  d_phi_area=True,
                  roughness=(sig, rng.uniform(5.0, 50.0, n),
                             _speckle(n, rng), nt, "exponential"))
    elif len(crossed) == 3:
        kw["gamma"] = 10.0 ** (rng.uniform(-30.0, -5.0, n) / 20.0)
    else:
        kw["gamma"] = _fresnel(eps[-1], 3.3)
    return SimpleNamespace(target=target, crossed=crossed, eps=eps, att=att,
                           pos=pos, uct=uct, kw=kw)


def _adjoint_inputs(case, seed):
    rng, crossed, target, eps, att, pos, uct, t0, dt = _stack(case, seed, 14)
    n = len(target.centers)
    k0 = 2 * np.pi * case["f0"] / C
    sig = np.exp(math.log(0.3) + 0.7 * rng.standard_normal(n))
    nt = _terms((2 * k0 * math.sqrt(eps[-1]) *
                 np.quantile(sig, 0.999)) ** 2)
    R = rng.uniform(-30.0, -5.0, n)
    ph = _speckle(n, rng)
    # measured powers: the level of a diffuse bed under 1 km of ice, with a
    # few dB of speckle from trace to trace
    kj = k0 * math.sqrt(eps[-1])
    amp = kj / (2 * np.pi) * 0.2 * target.areas.mean() / case["alt"] ** 2
    level = n * (0.05 * amp) ** 2 * 10.0 ** -2.0
    target_power = level * 10.0 ** (0.5 * rng.standard_normal(len(pos)))
    return SimpleNamespace(
        target=target, crossed=crossed, eps=eps, att=att, pos=pos, uct=uct,
        R=R.astype(np.float32), sig=sig.astype(np.float32), alpha=10.0,
        corr=10.0, phasors=ph, n_terms=nt, k0=k0, t0=t0, dt=dt,
        bins=case["bins"], target_power=target_power)


def _modef_inputs(case, seed):
    rng = np.random.default_rng([seed, 15])
    f = _layer(case["ny"], case["nx"], case["spacing"], 50.0, 1000.0, 0.0,
               rng)
    pos, uct = _track(case, rng)
    t0, dt = _window(pos, f, case["f0"])
    # the band's resolution cell, sampled at twice the bandwidth
    return SimpleNamespace(f=f, pos=pos, t0=t0, dt=dt, bw=0.25 * case["f0"],
                           twtt=t0 + np.arange(case["bins"]) * dt)


# --------------------------------------------------------------------------
# what a user's program has in hand, and one pass
# --------------------------------------------------------------------------
def _surface_args(s):
    f = s.f
    return (s.pos, s.uct, f.centers, f.normals, f.areas, f.e1, f.e2)


def _pulse(s):
    """The windowed chirp's compressed pulse, 10 us long, as taps."""
    from radar_sounder_simulator_gb300.waveform import compressed_pulse
    return compressed_pulse(0.25 * s.f0, 10e-6, s.kw["dt"], "hann", "chirp")


def prepare(case, seed):
    from radar_sounder_simulator_gb300 import coherent, incoherent, multilayer
    kind = case["kind"]
    if kind == "surface":
        s = _surface_inputs(case, seed)
        if case["api"] == "call":
            return SimpleNamespace(kind="call", args=_surface_args(s),
                                   kw=dict(s.kw, precision=case["precision"]),
                                   then=case["then"], s=s)
        plan = coherent.prepare_coherent(*_surface_args(s), **s.kw,
                                         precision=case["precision"])
        st = SimpleNamespace(kind="surface", plan=plan, then=case["then"],
                             fp64=case["precision"] == "fp64")
        if case["then"] in ("chirp", "focus"):
            from radar_sounder_simulator_gb300.waveform import \
                RangeCompressor
            taps, m = _pulse(s)
            st.compress = RangeCompressor(taps, m, case["bins"],
                                          precision="split")
        if case["then"] == "focus":
            from radar_sounder_simulator_gb300.processing import along_track
            dev = plan.device
            st.twtt = torch.from_numpy(
                s.kw["t0"] + np.arange(case["bins"]) * s.kw["dt"]).to(dev)
            st.arc = torch.from_numpy(along_track(s.pos)).to(dev)
            st.wavelength = C / case["f0"]
        return st
    if kind == "batch":
        from radar_sounder_simulator_gb300.batch import CoherentBatch
        plans = [coherent.prepare_coherent(*_surface_args(s), **s.kw,
                                           precision="split")
                 for s in _batch_inputs(case, seed)]
        return SimpleNamespace(kind="batch", batch=CoherentBatch(plans))
    if kind == "refracted":
        s = _refracted_inputs(case, seed)
        plan = multilayer.prepare_refracted(
            s.pos, s.uct, s.target, s.crossed, s.eps, s.att, **s.kw,
            precision=case["precision"])
        return SimpleNamespace(kind="surface", plan=plan, then="field",
                               fp64=case["precision"] == "fp64")
    if kind == "adjoint":
        from radar_sounder_simulator_gb300.adjoint import WindowPowerModel
        s = _adjoint_inputs(case, seed)
        model = WindowPowerModel(
            s.pos, s.uct, s.target, s.crossed, s.eps, s.att, t0=s.t0,
            dt=s.dt, n_samples=s.bins, c=C, k0=s.k0, window=(0, s.bins),
            alpha_legs=(1,), corr_length=s.corr, phasors=s.phasors,
            n_terms=s.n_terms)
        dev = model.device
        return SimpleNamespace(
            kind="adjoint", model=model,
            params=[torch.tensor(v, device=dev, requires_grad=True)
                    for v in (s.R, s.sig, np.float32(s.alpha))],
            target=torch.tensor(s.target_power, device=dev))
    if kind == "modef":
        from radar_sounder_simulator_gb300.multifreq import prepare_multifreq
        s = _modef_inputs(case, seed)
        f = s.f
        plan = prepare_multifreq(
            s.pos, f.centers, f.normals, f.areas, f.e1, f.e2,
            gamma=_fresnel(1.0, 3.15), f0=case["f0"], bandwidth=s.bw, c=C,
            twtt=s.twtt, n_freq=case["n_freq"], freeze_amplitudes=True,
            check_alias=False, precision="split")
        return SimpleNamespace(kind="modef", plan=plan)
    s = _surface_inputs(dict(case, pattern="none", rough=False), seed)
    f = s.f
    plan = incoherent.prepare_incoherent(
        s.pos, s.uct, f.centers, f.normals, f.areas, t0=s.kw["t0"],
        dt=s.kw["dt"], n_samples=case["bins"], c=C,
        split_sides=case["sides"])
    return SimpleNamespace(kind="incoherent", plan=plan)


def _single(field, dropped):
    """A split-form result as single precision, on the device."""
    return (torch.view_as_complex(field.to(torch.float32)),
            dropped.to(torch.float32))


def run(state):
    s = state
    if s.kind == "call":
        from radar_sounder_simulator_gb300 import coherent_cluttergram
        field, dropped = coherent_cluttergram(*s.args, **s.kw)
        if s.then == "chirp":
            from radar_sounder_simulator_gb300.waveform import \
                convolve_fast_time
            taps, m = _pulse(s.s)
            field = convolve_fast_time(
                field, taps, m, precision=s.kw["precision"]).astype(
                    np.complex64)
        return field, dropped
    if s.kind == "surface":
        field, dropped = s.plan.run()
        if s.fp64:
            return field, dropped
        if s.then == "field":
            return _single(field, dropped)
        if s.plan.split:
            field = field.reshape(s.plan.T, s.plan.n_samples, 2, 2)
        compressed = s.compress.run(field)
        if s.then == "chirp":
            return compressed, dropped.to(torch.float32)
        from radar_sounder_simulator_gb300.processing import focus_tensor
        focused, power = focus_tensor(
            compressed, s.twtt, s.arc, wavelength=s.wavelength,
            aperture_m=1900.0, precision="split")
        return compressed, focused, power
    if s.kind == "batch":
        return [_single(f, d) for f, d in s.batch.run()]
    if s.kind == "adjoint":
        from radar_sounder_simulator_gb300.adjoint import db_misfit
        power = s.model.power(*s.params)
        grads = torch.autograd.grad(db_misfit(power, s.target), s.params)
        return (power.detach().to(torch.float32),) + tuple(grads)
    if s.kind == "modef":
        y = s.plan.run()
        return torch.view_as_complex(y.to(torch.float32))
    return s.plan.run()


# --------------------------------------------------------------------------
# the work a pass cannot do without
# --------------------------------------------------------------------------
def _pair_flops(case):
    """FLOP of one (trace, facet) pair (FMA = 2): the facet field 47; a
    Snell crossing two converged two-point solves of about 110 and 30 of
    radiometry; a joint crossing 150 for its share of two block Newton
    steps besides; a roughness series 10 a term, counted where the series
    has weight (about x + 6 sqrt x terms, the mean over facets)."""
    kind = case["kind"]
    fl = 25.0 if kind == "incoherent" else 47.0
    if kind in ("refracted", "adjoint"):
        nc = case.get("crossed", 1)
        fl = 105.0 + 250.0 * nc + (150.0 * nc if case.get("joint") else 0.0)
    if case.get("rough") or kind == "adjoint":
        deep = kind in ("refracted", "adjoint")
        sig = 0.35 if deep else 0.29
        f0 = 120e6 if kind == "batch" else case["f0"]
        x = (4 * math.pi * f0 / C * sig * (1.775 if deep else 1.0)) ** 2
        fl += 10.0 * min(300.0, x + 6.0 * math.sqrt(x) + 5.0)
    if kind == "adjoint":
        fl = 2.0 * fl + 24.0
    return fl


def work(case):
    ny, nx, T, B = case["ny"], case["nx"], case["traces"], case["bins"]
    jobs = case.get("jobs", 1)
    if jobs > 1:    # mean sizes of the sweep's jobs
        ny, nx, T = 0.75 * ny, 0.75 * nx, 0.7 * T
    n = ny * nx
    kind = case["kind"]
    facet = 28.0 if kind == "incoherent" else 52.0
    if case.get("rough") or kind == "adjoint":
        facet += 16.0
    layers = case.get("crossed", 1) if kind in ("refracted",
                                                "adjoint") else 0
    out = 4.0 if kind == "incoherent" else 8.0
    if case.get("precision") == "fp64" and case.get("api") != "call":
        out = 16.0
    out *= 2 if case.get("sides") else 1
    by = jobs * (n * (facet + 24.0 * layers) + T * (24.0 + B * out))
    fl = jobs * n * T * _pair_flops(case)
    if kind == "adjoint":
        by += n * 16.0
    if kind == "modef":
        K = case["n_freq"]
        fl = n * T * (60.0 + 8.0 * K) + 8.0 * T * K * B
    then = case.get("then", "field")
    lanes = 2 if case.get("sides") else 1
    if then in ("chirp", "focus"):
        N = 1 << math.ceil(math.log2(B + 2 * 10e-6 * 0.5 * case["f0"]))
        fl += lanes * T * (10.0 * N * math.log2(N) + 6.0 * N)
        by += lanes * T * B * 8.0
    if then == "focus":
        fl += T * B * 33.0 * min(T, 1900.0 / case["step"])
        by += T * B * 20.0
    return {"bytes": by, "flops": fl}


# --------------------------------------------------------------------------
# the same in float64, in plain torch
# --------------------------------------------------------------------------
def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _t(a):
    return torch.as_tensor(np.asarray(a, np.float64), device=_dev())


def _q32(a):
    """Facet geometry as the kernels hold it: float32 values."""
    return _t(np.asarray(a, np.float32))


def _rows(a):
    return [a[:, j][None] for j in range(3)]


def _dot(a, b):
    return (a[0] * b[0] + a[1] * b[1]) + a[2] * b[2]


def _sub(a, b):
    return [x - y for x, y in zip(a, b)]


def _sinc(x):
    return torch.where(x == 0, torch.ones_like(x),
                       torch.sin(x) / torch.where(x == 0,
                                                  torch.ones_like(x), x))


def _facets(f):
    return SimpleNamespace(c=_rows(_q32(f.centers)), n=_rows(_q32(f.normals)),
                           a=_q32(f.areas)[None], e1=_rows(_q32(f.e1)),
                           e2=_rows(_q32(f.e2)))


def _chunks(T, n, target=1 << 21):
    step = max(1, target // max(n, 1))
    return [(a, min(a + step, T)) for a in range(0, T, step)]


def _scatter(acc, bins, ok, *parts):
    """Add each part to its trace's bin; acc (t, n, len(parts))."""
    t, n = acc.shape[0], acc.shape[1]
    rows = torch.arange(t, device=acc.device)[:, None] * n
    idx = torch.where(ok, rows + bins, torch.zeros_like(bins))
    for j, p in enumerate(parts):
        flat = torch.zeros(t * n, dtype=torch.float64, device=acc.device)
        flat.index_add_(0, idx.reshape(-1),
                        torch.where(ok, p, torch.zeros_like(p)).reshape(-1))
        acc[:, :, j] += flat.reshape(t, n)


def _gain(pattern, d, sl):
    """One-way field gain of departure directions d for traces ``sl``."""
    kind, pv, pa, pb = pattern
    v = _t(pv)[sl]
    ca = _dot(d, [v[:, j][:, None] for j in range(3)])
    if kind == "dipole":
        return torch.cos((np.pi / 2) * ca) / torch.sqrt(
            torch.clamp(1.0 - ca * ca, min=1e-12))
    th = torch.arccos(torch.clamp(ca, -1.0, 1.0))
    xa, ya = _t(pa), _t(pb)
    j = torch.clamp(torch.searchsorted(xa, th.contiguous(), right=True) - 1,
                    0, len(xa) - 2)
    g = ya[j] + (ya[j + 1] - ya[j]) / (xa[j + 1] - xa[j]) * (th - xa[j])
    g = torch.where(th <= xa[0], ya[0], g)
    return torch.where(th >= xa[-1], ya[-1], g)


def _series(sig, lc, kk, kb2, area, n_terms, slope=False):
    """Exponential-correlation area spectrum: sum over m of the Poisson
    weights of x = (sig kk)^2 and 2 pi (l/m)^2 (1 + kb^2 l^2/m^2)^(-3/2)
    times the facet's edge lengths; with ``slope`` also its x-derivative."""
    x = (sig * kk) ** 2
    p = torch.exp(-x)
    acc = torch.zeros_like(x)
    der = torch.zeros_like(x)
    q = kb2 * lc * lc
    for m in range(1, n_terms + 1):
        before = p
        p = p * x / m
        w = 1.0 + q / (m * m)
        w = 1.0 / (w * torch.sqrt(w) * (m * m))
        acc += p * w
        if slope:
            der += (before - p) * w
    c = 2.0 * np.pi * lc * lc * area
    return (acc * c, der * c) if slope else acc * c


def _lobe(F, rh, k, base, cos, taper, rough, slope=False):
    """Complex amplitude (re, im) of a facet seen along rh at wavenumber k,
    ``base`` the factors in front of cos A sinc sinc; with ``slope`` also
    its derivative with respect to the rms height."""
    d1, d2 = _dot(rh, F.e1), _dot(rh, F.e2)
    base = base * (k / (2 * np.pi)) * cos
    amp = base * F.a * _sinc(k * d1) * _sinc(k * d2)
    if taper is not None:
        c2 = torch.clamp(cos, 1e-9, 1.0) ** 2
        amp = amp * torch.exp(-(1.0 - c2) / (c2 * 2.0 * taper * taper))
    if rough is None:
        return amp, torch.zeros_like(amp)
    sig, lc, pr, pi, nt = rough
    l1, l2 = torch.sqrt(_dot(F.e1, F.e1)), torch.sqrt(_dot(F.e2, F.e2))
    kk = 2.0 * k * cos
    kb2 = (2.0 * k * d1 / l1) ** 2 + (2.0 * k * d2 / l2) ** 2
    mean = torch.exp(-0.5 * (sig * kk) ** 2)
    if not slope:
        root = torch.sqrt(_series(sig, lc, kk, kb2, l1 * l2, nt))
        return amp * mean + base * root * pr, base * root * pi
    D, dD = _series(sig, lc, kk, kb2, l1 * l2, nt, slope=True)
    root = torch.sqrt(D)
    dr = torch.where(D > 0, base * dD * sig * kk * kk / root,
                     torch.zeros_like(D))
    return (amp * mean + base * root * pr, base * root * pi,
            -amp * mean * sig * kk * kk + dr * pr, dr * pi)


def _rough(kw):
    if "roughness" not in kw:
        return None
    sig, lc, ph, nt, _ = kw["roughness"]
    ph = np.asarray(ph, np.complex64)
    return (_q32(sig)[None], _q32(lc)[None], _t(ph.real)[None],
            _t(ph.imag)[None], nt)


def _bin(path, kw):
    """floor((2 path / c - t0) / dt) in float64, the reference's order."""
    return torch.floor((2.0 * path / kw["c"] - kw["t0"]) / kw["dt"])


def _bin_field(field, sl, path, re, im, ok, right, kw):
    b = _bin(path, kw)
    n = kw["n_samples"]
    ok = ok & (b >= 0) & (b < n)
    bi = torch.clamp(b, 0, n - 1).to(torch.int64)
    if right is not None:
        bi = bi + right * n
    _scatter(field[sl], bi, ok, re, im)


def _surface_exact(s):
    """(T, n_seg, 2) field of a surface."""
    F, kw = _facets(s.f), s.kw
    pos = _t(s.pos)
    T, n = len(pos), kw["n_samples"]
    sides = kw.get("split_sides", False)
    field = torch.zeros((T, n * (2 if sides else 1), 2), dtype=torch.float64,
                        device=pos.device)
    rough = _rough(kw)
    for lo, hi in _chunks(T, F.a.shape[1]):
        sl = slice(lo, hi)
        d = _sub([pos[sl, j][:, None] for j in range(3)], F.c)
        r = torch.sqrt((d[0] * d[0] + d[1] * d[1]) + d[2] * d[2])
        rh = [v / r for v in d]
        cos = _dot(rh, F.n)
        # the scalar reflection coefficient is held in double precision
        cr, ci = _lobe(F, rh, kw["k"], float(kw["gamma"]) / (r * r), cos,
                       kw.get("taper_s"), rough)
        if "pattern" in kw:
            g = _gain(kw["pattern"], [-v for v in rh], sl) ** 2
            cr, ci = cr * g, ci * g
        ph = 2.0 * kw["k"] * r
        sn, cs = torch.sin(ph), torch.cos(ph)
        right = None
        if sides:
            u = _t(s.uct)[sl]
            right = (_dot([-v for v in d], [u[:, j][:, None]
                                            for j in range(3)]) >
                     0).to(torch.int64)
        _bin_field(field, sl, r, cr * sn - ci * cs, cr * cs + ci * sn,
                   torch.ones_like(r, dtype=torch.bool), right, kw)
    if sides:   # left, right as the last sample axis
        field = field.reshape(T, 2, n, 2).permute(0, 2, 1, 3).reshape(
            T, 2 * n, 2).contiguous()
    return field


def _two_point(P, Q, O, N, n1, n2):
    """Refraction of the ray P -> Q at the plane through O with normal N:
    crossing, upper leg, cosines on both sides, whether P and Q lie on
    opposite sides."""
    h1, h2 = _dot(_sub(P, O), N), _dot(_sub(Q, O), N)
    a, b = torch.abs(h1), torch.abs(h2)
    foot = [p - h1 * v for p, v in zip(P, N)]
    w = [q - h2 * v - f for q, v, f in zip(Q, N, foot)]
    L = torch.sqrt(_dot(w, w))
    flip = n1 > n2
    ratio = min(n1, n2) / max(n1, n2)
    rare, dense = (b, a) if flip else (a, b)
    sig = L / torch.sqrt(L * L + (a + b) ** 2)
    for _ in range(9):
        v = ratio * sig
        c1, c2 = 1.0 - sig * sig, 1.0 - v * v
        r1, r2 = 1.0 / torch.sqrt(c1), 1.0 / torch.sqrt(c2)
        F = rare * sig * r1 + dense * v * r2 - L
        sig = torch.clamp(sig - F / (rare * r1 / c1 + dense * ratio * r2 /
                                     c2), 0.0, 1.0 - 1e-12)
    t = rare * sig / torch.sqrt(1.0 - sig * sig)
    t = L - t if flip else t
    s1, s2 = torch.sqrt(a * a + t * t), torch.sqrt(b * b + (L - t) ** 2)
    f = t / torch.clamp(L, min=1e-30)
    x = [p + f * v for p, v in zip(foot, w)]
    return x, s1, a / s1, b / s2, h1 * h2 < 0


class _Iface:
    """Lookup of a crossed interface: float32 cell table, least-squares
    (x, y) -> (row, col) fit, area-weighted mean plane."""

    def __init__(self, f):
        A = np.column_stack([f.centers[:, :2], np.ones(len(f.centers))])
        self.coef = np.linalg.lstsq(A, np.asarray(f.cell, np.float64),
                                    rcond=None)[0]
        self.ny, self.nx = f.grid_shape
        w = f.areas / f.areas.sum()
        mp, mn = w @ f.centers, w @ f.normals
        mn = mn / np.linalg.norm(mn)
        self.mp = [float(v) for v in mp]
        self.mn = [float(v) for v in mn]
        n = _q32(f.normals)
        self.tab = torch.cat([_q32(f.centers), n / torch.sqrt(
            (n * n).sum(1, keepdim=True))], 1)

    def plane(self, x):
        rc = [x[0] * self.coef[0, j] + x[1] * self.coef[1, j] +
              self.coef[2, j] for j in range(2)]
        row = torch.clamp(torch.round(rc[0]), 0, self.ny - 1)
        col = torch.clamp(torch.round(rc[1]), 0, self.nx - 1)
        g = self.tab[(row * self.nx + col).to(torch.int64)]
        return [g[..., j] for j in range(3)], [g[..., 3 + j]
                                               for j in range(3)]


def _joint(P, Q, O, N, x, nl):
    """Newton solve of the stationary polyline P -> planes -> Q from the
    crossings x: block-tridiagonal 2 x 2 systems in the planes' bases."""
    ni = len(O)
    basis = []
    for n in N:
        u = [n[2], torch.zeros_like(n[0]), -n[0]]
        inv = 1.0 / torch.sqrt(_dot(u, u))
        u = [c * inv for c in u]
        basis.append((u, [n[1] * u[2] - n[2] * u[1],
                          n[2] * u[0] - n[0] * u[2],
                          n[0] * u[1] - n[1] * u[0]]))
    # onto the planes
    x = [[c - _dot(_sub(xi, o), n) * v for c, v in zip(xi, n)]
         for xi, o, n in zip(x, O, N)]
    for _ in range(6):
        pts = [P] + x + [Q]
        seg = [_sub(pts[i + 1], pts[i]) for i in range(ni + 1)]
        ln = [torch.sqrt(_dot(v, v)) for v in seg]
        d = [[c / l for c in v] for v, l in zip(seg, ln)]
        w = [nl[i] / ln[i] for i in range(ni + 1)]
        pin = [[_dot(b, d[i]) for b in basis[i]] for i in range(ni)]
        pout = [[_dot(b, d[i + 1]) for b in basis[i]] for i in range(ni)]
        f = [[nl[i] * pin[i][r] - nl[i + 1] * pout[i][r] for r in range(2)]
             for i in range(ni)]
        A = [[[w[i] * (float(r == c) - pin[i][r] * pin[i][c]) +
               w[i + 1] * (float(r == c) - pout[i][r] * pout[i][c])
               for c in range(2)] for r in range(2)] for i in range(ni)]
        B = [[[-w[i + 1] * (_dot(basis[i][r], basis[i + 1][c]) -
                            pout[i][r] * pin[i + 1][c])
               for c in range(2)] for r in range(2)] for i in range(ni - 1)]
        inv, rhs = [], []
        for i in range(ni):
            M, y = A[i], [-f[i][0], -f[i][1]]
            if i:
                G = [[sum(B[i - 1][m][r] * inv[i - 1][m][c]
                          for m in range(2)) for c in range(2)]
                     for r in range(2)]
                M = [[M[r][c] - sum(G[r][m] * B[i - 1][m][c]
                                    for m in range(2)) for c in range(2)]
                     for r in range(2)]
                y = [y[r] - sum(G[r][m] * rhs[i - 1][m] for m in range(2))
                     for r in range(2)]
            det = M[0][0] * M[1][1] - M[0][1] * M[1][0]
            inv.append([[M[1][1] / det, -M[0][1] / det],
                        [-M[1][0] / det, M[0][0] / det]])
            rhs.append(y)
        step = [None] * ni
        for i in range(ni - 1, -1, -1):
            y = rhs[i]
            if i < ni - 1:
                y = [y[r] - sum(B[i][r][m] * step[i + 1][m]
                                for m in range(2)) for r in range(2)]
            step[i] = [sum(inv[i][r][m] * y[m] for m in range(2))
                       for r in range(2)]
        x = [[x[i][c] + step[i][0] * basis[i][0][c] +
              step[i][1] * basis[i][1][c] for c in range(3)]
             for i in range(ni)]
    return x


def _te(e1, e2, c1):
    a, b = math.sqrt(e1), math.sqrt(e2)
    c2 = torch.sqrt(torch.clamp(1.0 - (e1 / e2) * (1.0 - c1 * c1), min=0.0))
    return (a * c1 - b * c2) / (a * c1 + b * c2)


def _refracted_pair(s, ifaces, P, F, joint):
    """Radiometry of a chunk of traces x all facets: direction facet ->
    last crossing, its cosine, optical path, spreading, attenuation factor,
    one leg's length below the surface, validity."""
    nl = [math.sqrt(e) for e in s.eps]
    ni = len(ifaces)
    Q = F.c
    cur, planes = P, []
    xs, legs, cin, cout = [], [], [], []
    ok = torch.ones(torch.broadcast_shapes(P[0].shape, Q[0].shape),
                    dtype=torch.bool, device=Q[0].device)
    for i, I in enumerate(ifaces):
        x = _two_point(cur, Q, I.mp, I.mn, nl[i], nl[i + 1])[0]
        o, n = I.plane(x)
        if joint:
            planes.append((o, n))
            xs.append(x)
        else:
            x, s1, c1, c2, side = _two_point(cur, Q, o, n, nl[i], nl[i + 1])
            legs.append(s1)
            cin.append(c1)
            cout.append(c2)
            ok = ok & side
        cur = x
    if joint:
        O, N = [p[0] for p in planes], [p[1] for p in planes]
        xs = _joint(P, Q, O, N, xs, nl)
        pts = [P] + xs + [Q]
        for i in range(ni):
            up, dn = _sub(pts[i], pts[i + 1]), _sub(pts[i + 2], pts[i + 1])
            lu, ld = torch.sqrt(_dot(up, up)), torch.sqrt(_dot(dn, dn))
            a, b = _dot(up, N[i]), _dot(dn, N[i])
            legs.append(lu)
            cin.append(torch.abs(a) / lu)
            cout.append(torch.abs(b) / ld)
            ok = ok & (a * b < 0)
        cur = xs[-1]
    d = _sub(cur, Q)
    last = torch.sqrt(_dot(d, d))
    rh = [c / last for c in d]
    opl, loss, perp, par, tau2 = 0.0, 0.0, 0.0, 0.0, 1.0
    for i in range(ni):
        opl = opl + nl[i] * legs[i]
        loss = loss + legs[i] * (s.att[i] / 1000.0)
        perp = perp + legs[i] / nl[i]
        par = par + legs[i] / (nl[i] * cin[i] ** 2)
        tau2 = tau2 * (1.0 - _te(s.eps[i], s.eps[i + 1], cin[i]) ** 2)
    nj = nl[ni]
    opl = opl + nj * last
    loss = loss + last * (s.att[ni] / 1000.0)
    perp = perp + last / nj
    par = par + last / (nj * cout[-1] ** 2)
    spread = tau2 * (nl[0] * cin[0]) / (nj * cout[-1]) / (
        nl[0] * cin[0] ** 2 * par * nl[0] * perp)
    return rh, _dot(rh, F.n), opl, spread * 10.0 ** (-loss / 10.0), last, ok


def _refracted_exact(s, joint):
    F, kw = _facets(s.target), s.kw
    ifaces = [_Iface(f) for f in s.crossed]
    pos = _t(s.pos)
    T, n = len(pos), kw["n_samples"]
    field = torch.zeros((T, n, 2), dtype=torch.float64, device=pos.device)
    gam = kw["gamma"]
    gam = _t(gam)[None] if np.ndim(gam) else float(gam)
    rough, k0 = _rough(kw), kw["k0"]
    kj = k0 * math.sqrt(s.eps[-1])
    for lo, hi in _chunks(T, F.a.shape[1]):
        sl = slice(lo, hi)
        P = [pos[sl, j][:, None] for j in range(3)]
        rh, cos, opl, spread, _, ok = _refracted_pair(s, ifaces, P, F, joint)
        cr, ci = _lobe(F, rh, kj, gam * spread, cos, kw.get("taper_s"),
                       rough)
        sn, cs = torch.sin(2.0 * k0 * opl), torch.cos(2.0 * k0 * opl)
        _bin_field(field, sl, opl, cr * sn - ci * cs, cr * cs + ci * sn,
                   ok, None, kw)
    return field


def _adjoint_exact(s):
    """Power, and the gradients of the dB misfit with respect to dB
    reflectivity, rms height and attenuation rate."""
    F = _facets(s.target)
    ifaces = [_Iface(f) for f in s.crossed]
    pos = _t(s.pos)
    T, n, N = len(pos), s.bins, F.a.shape[1]
    kw = dict(c=C, t0=s.t0, dt=s.dt, n_samples=n)
    gam = 10.0 ** (_t(s.R)[None] / 20.0)
    rough = (_q32(s.sig)[None], _t(np.float32(s.corr)),
             _t(s.phasors.real)[None], _t(s.phasors.imag)[None], s.n_terms)
    kj = s.k0 * math.sqrt(s.eps[-1])

    def pairs(sl):
        P = [pos[sl, j][:, None] for j in range(3)]
        rh, cos, opl, spread, last, ok = _refracted_pair(s, ifaces, P, F,
                                                         False)
        v = _lobe(F, rh, kj, gam * spread, cos, 0.05, rough, slope=True)
        sn, cs = torch.sin(2.0 * s.k0 * opl), torch.cos(2.0 * s.k0 * opl)
        b = _bin(opl, kw)
        ok = ok & (b >= 0) & (b < n)
        turn = [(v[j] * sn - v[j + 1] * cs, v[j] * cs + v[j + 1] * sn)
                for j in (0, 2)]
        return turn, last, ok, torch.clamp(b, 0, n - 1).to(torch.int64)

    field = torch.zeros((T, n, 2), dtype=torch.float64, device=pos.device)
    ch = _chunks(T, N, 1 << 20)
    for lo, hi in ch:
        sl = slice(lo, hi)
        (c, _), _, ok, b = pairs(sl)
        _scatter(field[sl], b, ok, *c)
    power = (field ** 2).sum((1, 2))
    miss = 10.0 * torch.log10(power / _t(s.target_power))
    g = 2.0 * miss * 10.0 / (math.log(10.0) * power)
    gR = torch.zeros(N, dtype=torch.float64, device=pos.device)
    gS = torch.zeros_like(gR)
    gA = 0.0
    for lo, hi in ch:
        sl = slice(lo, hi)
        (c, dc), last, ok, b = pairs(sl)
        w = torch.where(ok, 2.0 * g[sl][:, None], torch.zeros_like(last))
        fr = torch.gather(field[sl, :, 0], 1, b)
        fi = torch.gather(field[sl, :, 1], 1, b)
        dot = w * (fr * c[0] + fi * c[1])
        gR += dot.sum(0) * (math.log(10.0) / 20.0)
        gS += (w * (fr * dc[0] + fi * dc[1])).sum(0)
        gA = gA - float((dot * last).sum()) * math.log(10.0) / 1e4
    return power, gR, gS, gA


def _compress_exact(x, taps, m):
    """'same'-mode convolution along axis 1 of a complex128 (T, B[, L])."""
    B, M = x.shape[1], len(taps)
    N = B + M - 1
    p = torch.as_tensor(np.asarray(taps, np.complex128), device=x.device)
    shape = (1, -1) + (1,) * (x.dim() - 2)
    y = torch.fft.ifft(torch.fft.fft(x, n=N, dim=1) *
                       torch.fft.fft(p, n=N).reshape(shape), dim=1)
    return y[:, m:m + B]


def _focus_exact(x, twtt, arc, wavelength, aperture):
    T, nb = x.shape
    half, k = aperture / 2.0, 2 * np.pi / wavelength
    t0, dt = float(twtt[0]), float(twtt[1] - twtt[0])
    tw, s = _t(twtt), _t(arc)
    r0 = C * tw / 2.0
    out = torch.zeros_like(x)
    reach = int(np.searchsorted(arc, arc[0] + 2 * half, "right")) + 2
    idx = torch.arange(T, device=x.device)
    for o in range(-reach, reach + 1):
        j = idx + o
        inside = (j >= 0) & (j < T)
        j = torch.clamp(j, 0, T - 1)
        d = s[j] - s
        inside = inside & (torch.abs(d) <= half)
        if not bool(inside.any()):
            continue
        w = torch.where(inside, 0.5 * (1.0 + torch.cos(np.pi * d / half)),
                        torch.zeros_like(d))
        dr = torch.sqrt(r0[None] ** 2 + d[:, None] ** 2) - r0[None]
        pos = ((tw[None] + 2.0 * dr / C) - t0) / dt
        i0 = torch.floor(pos)
        fr = pos - i0
        ok = (i0 >= 0) & (i0 < nb - 1)
        i0 = torch.clamp(i0, 0, nb - 2).to(torch.int64)
        row = x[j]
        v = torch.gather(row, 1, i0) * (1.0 - fr) + torch.gather(
            row, 1, i0 + 1) * fr
        out += torch.where(ok, w[:, None] * v * torch.exp(2j * k * dr),
                           torch.zeros_like(v))
    return out


def _modef_exact(case, s):
    F = _facets(s.f)
    pos = _t(s.pos)
    K, f0 = case["n_freq"], case["f0"]
    off = -s.bw / 2.0 + (np.arange(K) + 0.5) * (s.bw / K)
    freq = _t(f0 + off)
    w = 0.5 + 0.5 * np.cos(2.0 * np.pi * off / s.bw)
    w = _t(w / w.sum())
    syn = torch.exp(2j * np.pi * _t(off)[:, None] * _t(s.twtt)[None])
    k = 2 * np.pi * f0 / C
    out = []
    for t in range(len(pos)):
        d = _sub([pos[t:t + 1, j][:, None] for j in range(3)], F.c)
        r = torch.sqrt(_dot(d, d))
        rh = [v / r for v in d]
        amp, _ = _lobe(F, rh, k, _fresnel(1.0, 3.15) / (r * r),
                       _dot(rh, F.n), None, None)
        ph = (4.0 * np.pi / C) * r[0][:, None] * freq[None]
        a = amp[0][None]
        H = torch.complex(a @ torch.sin(ph), a @ torch.cos(ph))
        out.append((H * w[None].to(torch.complex128)) @ syn)
    return torch.cat(out)


def _incoherent_exact(s, sides):
    """Power sums in float64 of the reference's float32 quantities: the
    range chain and its bin are float32 decisions by definition."""
    f, kw = s.f, s.kw
    dev = _dev()

    def f32(a):
        return torch.as_tensor(np.asarray(a, np.float32), device=dev)
    cen, pos, u = f32(f.centers), f32(s.pos), f32(s.uct)
    nrm, area = _rows(_q32(f.normals)), _q32(f.areas)[None]
    t0, dt, c = (f32(v) for v in (kw["t0"], kw["dt"], kw["c"]))
    T, n = len(pos), kw["n_samples"]
    out = torch.zeros((T, n * (2 if sides else 1), 1), dtype=torch.float64,
                      device=dev)
    drop = torch.zeros(T, dtype=torch.float64, device=dev)
    for lo, hi in _chunks(T, len(cen)):
        sl = slice(lo, hi)
        d = [pos[sl, j][:, None] - cen[:, j][None] for j in range(3)]
        S = (d[0] * d[0] + d[1] * d[1]) + d[2] * d[2]
        b = torch.floor(((2.0 * torch.sqrt(S)) / c - t0) / dt)
        ok = (b >= 0) & (b < n)
        bi = torch.clamp(b, 0, n - 1).to(torch.int64)
        if sides:
            sd = ((-d[0] * u[sl, 0][:, None] + -d[1] * u[sl, 1][:, None]) +
                  -d[2] * u[sl, 2][:, None])
            bi = bi + (sd > 0).to(torch.int64) * n
        d = [v.double() for v in d]
        r2 = _dot(d, d)
        pw = (area * _dot(d, nrm)) ** 2 / (r2 * r2 * r2)
        _scatter(out[sl], bi, ok, pw)
        drop[sl] += torch.where(ok, torch.zeros_like(pw), pw).sum(1)
    out = out[:, :, 0]
    if sides:
        out = out.reshape(T, 2, n).permute(0, 2, 1)
    return out.contiguous(), drop


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return [(torch.view_as_complex(_surface_exact(s)), None)
                for s in _batch_inputs(case, seed)]
    if kind == "refracted":
        field = _refracted_exact(_refracted_inputs(case, seed),
                                 case["joint"])
        if case["precision"] == "fp64":
            return field, None
        return torch.view_as_complex(field), None
    if kind == "adjoint":
        power, gR, gS, gA = _adjoint_exact(_adjoint_inputs(case, seed))
        return power, gR, gS, torch.tensor(gA, dtype=torch.float64)
    if kind == "modef":
        return _modef_exact(case, _modef_inputs(case, seed))
    if kind == "incoherent":
        s = _surface_inputs(dict(case, pattern="none", rough=False), seed)
        return _incoherent_exact(s, case["sides"])
    s = _surface_inputs(case, seed)
    field = _surface_exact(s)
    z = torch.view_as_complex(field)
    if case["api"] == "plan":
        if case["precision"] == "fp64":
            return field, None
        if case["then"] == "field":
            return z, None
    T, B = len(s.pos), case["bins"]
    if case["sides"]:
        z = z.reshape(T, B, 2)
    if case["then"] == "field":
        return z, None
    taps, m = _pulse(s)
    z = _compress_exact(z, taps, m)
    if case["then"] == "chirp":
        return z, None
    seg = np.linalg.norm(np.diff(s.pos, axis=0), axis=1)
    arc = np.concatenate([[0.0], np.cumsum(seg)])
    twtt = s.kw["t0"] + np.arange(B) * s.kw["dt"]
    y = _focus_exact(z, twtt, arc, C / case["f0"], 1900.0)
    return z, y, torch.abs(y) ** 2
