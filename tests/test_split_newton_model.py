"""Float32 model of the surface split kernel's range difference as a Newton
step (ss_coherent_split.cu): dr is the float32 difference of the two ranges, r
from a hardware reciprocal root (relative error up to 2^-22.9, drawn here at
its limit with either sign), and one step of dr^2 + 2 r_c dr = N whose residual
is formed exactly.

Bound: the first dr errs by d <= 2^-22.9 r + two roundings of r (r <= 32 km:
7.9e-3 m); the step leaves d^2 / (2 r) (1.0e-9 m), the slope's error 2^-22.4 d
(1.5e-9 m) and three roundings 2^-24 d (1.4e-9 m); N's own terms leave up to
2.5e-9 m at 160 m (test_split_range_model.py). 7e-9 m in all on a straight
block, the middle trace (w = 0) included; 1e-7 and 2e-7 m on bent ones, where
q.eps is a float32 product.
"""

import numpy as np
import pytest

from tests.test_split_range_model import (F32, fma, pairs,  # noqa: F401
                                          two_prod, two_sum)


def _newton(pc, w, C, sign):
    q = pc - C
    qh = q.astype(F32)
    ql = (q - qh).astype(F32)
    rc = np.linalg.norm(q, axis=1)
    rch = rc.astype(F32)
    rcl = (rc - rch).astype(F32)
    w2 = float(np.dot(w, w))
    w2h = F32(w2)
    w2l = F32(w2 - float(w2h))
    # track direction x: q.u is q's first component as a double-float
    lam = float(w[0])
    eps = (w - lam * np.array([1.0, 0.0, 0.0])).astype(F32)
    lh = F32(lam)
    ll = F32(lam - float(lh))
    pq, e = two_prod(np.full(len(q), lh, F32), qh[:, 0])
    lo = (e + fma(lh, ql[:, 0], ll * qh[:, 0]) +
          (qh * eps).sum(1, dtype=F32)).astype(F32)
    Nh, g = two_sum((F32(2) * pq).astype(F32), fma(F32(2), lo, w2h))
    Nl = (g + w2l).astype(F32)
    rr = fma(rch, rch, Nh)
    inv = (1.0 / np.sqrt(rr.astype(np.float64)) *
           (1.0 + sign * 2.0 ** -22.9)).astype(F32)
    dr = fma(rr, inv, -rch)
    big = (F32(2) * rch).astype(F32)
    Dh = (big + dr).astype(F32)
    Dl = fma(F32(2), rcl, (dr - (Dh - big)).astype(F32))
    drl = ((fma(-dr, Dh, Nh) + fma(-dr, Dl, Nl)) *
           (F32(0.5) * inv)).astype(F32)
    return rc + dr.astype(np.float64) + drl.astype(np.float64)


@pytest.mark.parametrize("sign", [-1.0, 1.0])
@pytest.mark.parametrize("w,bound", [
    ((0.0, 0.0, 0.0), 7e-9), ((6.25, 0.0, 0.0), 7e-9),
    ((-75.0, 0.0, 0.0), 7e-9), ((160.0, 0.0, 0.0), 7e-9),
    ((-25.0, 0.3, -0.2), 1e-7), ((160.0, 0.7, 0.7), 2e-7)])
def test_newton_step_range(pairs, w, bound, sign):  # noqa: F811
    pc, C, _ = pairs
    assert np.linalg.norm(pc - C, axis=1).max() < 32e3
    err = np.abs(_newton(pc, np.array(w), C, sign) -
                 np.linalg.norm(pc + np.array(w) - C, axis=1))
    print(w, sign, err.max())
    assert err.max() <= bound
