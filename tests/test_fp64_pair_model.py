"""NumPy model of the FP64 surface pair's amplitude (ss_coherent.cu): one
reciprocal root ir serves every quotient by the range. CUDA's rsqrt is good to
an ulp; with one Newton step towards 1 / r the amplitude is as close to an
extended-precision value as with a correctly rounded root and quotients
(5.9e-16 against 5.6e-16 here, 6.5e-16 without the step). Bound: a tenth more,
two of the amplitude's nine roundings being those of ir.
"""

import numpy as np
import pytest

PI = np.longdouble("3.14159265358979323846264338")


def sin_rounded(y):
    """sin(pi y) to its rounding, as sinpi gives it."""
    return np.sin(PI * y.astype(np.longdouble)).astype(np.float64)


@pytest.mark.skipif(np.finfo(np.longdouble).eps > 2e-19,
                    reason="needs an extended-precision long double")
@pytest.mark.parametrize("seed", [0, 1])
def test_amplitude_rounding(seed):
    rng = np.random.default_rng(seed)
    n = 200000
    d = np.column_stack([rng.uniform(-6e3, 6e3, n), rng.uniform(-6e3, 6e3, n),
                         rng.uniform(14e3, 16e3, n)])
    nrm = np.array([0.02, -0.03, 1.0])
    nrm /= np.linalg.norm(nrm)
    e1, e2 = np.array([50.0, 0.0, -1.0]), np.array([0.0, 50.0, 1.5])
    k = 2 * np.pi * 60e6 / 299792458.0

    def dot(a, b):
        return (a[:, 0] * b[0] + a[:, 1] * b[1]) + a[:, 2] * b[2]

    def err(v):
        return float(np.linalg.norm(v - true) / np.linalg.norm(true))
    x = d.astype(np.longdouble)
    rl = np.sqrt(dot(x * x, np.ones(3)))
    y1, y2 = k * dot(x, e1) / rl, k * dot(x, e2) / rl
    true = dot(x, nrm) / rl * np.sin(y1) / y1 * np.sin(y2) / y2 / rl ** 2

    r2 = dot(d * d, np.ones(3))
    r, kp = np.sqrt(r2), k / np.pi
    h = d / r[:, None]
    z1, z2 = dot(h, e1) * kp, dot(h, e2) * kp
    quot = (dot(d, nrm) / r * (sin_rounded(z1) / (np.pi * z1)) *
            (sin_rounded(z2) / (np.pi * z2)) / (r * r))

    ir = (1.0 / np.sqrt(r2.astype(np.longdouble))).astype(np.float64)
    ir *= 1.0 + rng.choice([-1, 0, 1], n) * 2.0 ** -53   # rsqrt's ulp
    e = (1.0 - r.astype(np.longdouble) * ir).astype(np.float64)
    ir = (ir + e.astype(np.longdouble) * ir).astype(np.float64)
    z1, z2 = dot(d, e1) * ir * kp, dot(d, e2) * ir * kp
    kern = (dot(d, nrm) * ir * (sin_rounded(z1) * sin_rounded(z2) /
                                ((np.pi * z1) * (np.pi * z2))) * (ir * ir))
    assert err(kern) <= 1.1 * err(quot)
