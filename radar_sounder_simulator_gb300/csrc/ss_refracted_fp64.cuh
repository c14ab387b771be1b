// float64 refracted-path solvers shared by the FP64 kernel and the split
// kernel's exact fallbacks (internal).
#pragma once

#include "ss_refracted.cuh"

namespace ss {

constexpr double kTiny = 1e-30;
constexpr double kEps64 = 2.220446049250313e-16;
constexpr double kCMin = 1e-9;
// Template argument of the deep-stack instantiations: the joint solve's
// arrays hold SS_MAX_IFACE interfaces (in local memory) and the count
// crossed is the call's; every smaller argument is a count of its own.
constexpr int kDeepNI = SS_MAX_IFACE;

struct Snell64 {
  double x[3];
  double c1, c2;  // cosines to the normal on the p side and on the q side
  double s1, s2, res;
  bool valid;
};

__device__ __forceinline__ double dot3v(const double *a, const double *b) {
  return (a[0] * b[0] + a[1] * b[1]) + a[2] * b[2];
}

// sqrt(q) and 1/sqrt(q) of q > 0 from one reciprocal square root: the root
// q * i with one Newton correction (rounded as sqrt does, to the last bit
// or so) at a third of the float64 operations of a root and a quotient.
__device__ __forceinline__ void sqrt_inv64(double q, double &r, double &i) {
  i = rsqrt(q);
  r = q * i;
  r = fma(fma(-r, r, q), 0.5 * i, r);
}

// float32 root of the two-point equation: the float64 solve's start. The
// same safeguarded Newton; it stops after a step below 3e-4 of sigma, which
// leaves ~1e-7 (quadratic convergence).
__device__ __forceinline__ float sigma_seed32(float ar, float bd, float Lh,
                                              float ab, float ratio) {
  const float hi0 = 1.0f - 1e-6f;
  float sig = fminf(Lh * rsqrtf(fmaxf(Lh * Lh + ab * ab, 1e-30f)), hi0);
  float lo = 0.0f, hi = hi0;
  for (int it = 0; it < 8; ++it) {
    const float v = ratio * sig;
    const float r1 = rsqrtf(fmaxf((1.0f - sig) * (1.0f + sig), 1e-30f));
    const float r2 = rsqrtf(fmaxf((1.0f - v) * (1.0f + v), 1e-30f));
    const float F = (ar * sig * r1 + bd * v * r2) - Lh;
    if (F <= 0.0f) lo = sig; else hi = sig;
    const float Fp = ar * r1 * r1 * r1 + bd * ratio * r2 * r2 * r2;
    const float sn = sig - __fdividef(F, fmaxf(Fp, 1e-30f));
    const bool ok = (sn >= lo) && (sn <= hi);
    const float nxt = ok ? sn : 0.5f * (lo + hi);
    const bool done = fabsf(nxt - sig) <= 3e-4f * sig;
    sig = nxt;
    if (done) break;
  }
  return sig;
}

// The reference's own iteration: rays flat enough that its budget may end
// short of the root (multilayer.py:196-266).
static __device__ __noinline__ double sigma_budget64(double ar, double bd,
                                                     double Lh, double ab,
                                                     double ratio,
                                                     int n_iter) {
  const double hi0 = 1.0 - 8.0 * kEps64;
  double sig = fmin(Lh / fmax(sqrt(Lh * Lh + ab * ab), kTiny), hi0);
  double lo = 0.0, hi = hi0;
  for (int it = 0; it < n_iter; ++it) {
    const double v = ratio * sig;
    const double c1 = fmax((1.0 - sig) * (1.0 + sig), kTiny);
    const double c2 = fmax((1.0 - v) * (1.0 + v), kTiny);
    const double sc1 = sqrt(c1), sc2 = sqrt(c2);
    const double F = (ar * sig * (1.0 / sc1) + bd * v * (1.0 / sc2)) - Lh;
    if (F <= 0.0) lo = sig; else hi = sig;
    const double Fp = ar / (c1 * sc1) + (bd * ratio) / (c2 * sc2);
    const double sn = sig - F / fmax(Fp, kTiny);
    const bool ok = (sn >= lo) && (sn <= hi) && isfinite(sn);
    sig = ok ? sn : 0.5 * (lo + hi);
  }
  return sig;
}

// Two-point crossing (refraction.py:78-161, multilayer.py:196-266): the
// safeguarded Newton on sigma = sin(theta) of the rare side. The root is the
// reference's; the way there spends the slow float64 pipe (1/64 of the
// float32 rate) on two or three residuals instead of its fixed 10 or 25
// iterations: a float32 solve starts it at ~1e-7, the residual is float64,
// the slope float32 (a relative slope error of 1e-7 leaves 1e-7 of a step),
// and a step below 1e-9 of sigma leaves less than an ulp, so the iteration
// ends there. Flat rays repeat the reference's iteration: ten steps reach the
// root for every sigma below 0.8, twenty-five below 0.999 (a float64 model
// over random heights, offsets and index ratios). `x_only`: the crossing point
// alone (lookup anchors).
static __device__ __noinline__ void snell64(const double *p, const double *q,
                                            const double *o,
                                            const double *nrm, double n1,
                                            double n2, int n_iter, Snell64 &R,
                                            bool x_only = false) {
  double po[3] = {p[0] - o[0], p[1] - o[1], p[2] - o[2]};
  double qo[3] = {q[0] - o[0], q[1] - o[1], q[2] - o[2]};
  const double h1 = dot3v(po, nrm), h2 = dot3v(qo, nrm);
  const double a = fabs(h1), b = fabs(h2);
  double fp[3], w[3];
  for (int j = 0; j < 3; ++j) {
    fp[j] = p[j] - h1 * nrm[j];
    w[j] = (q[j] - h2 * nrm[j]) - fp[j];
  }
  double L, iL;
  sqrt_inv64(fmax(dot3v(w, w), kTiny * kTiny), L, iL);
  const double s = fmax(a + b + L, kTiny);
  const double inv_s = 1.0 / s;
  const double ah = a * inv_s, bh = b * inv_s, Lh = L * inv_s;
  const bool swap = n1 > n2;
  const double ratio = fmin(n1, n2) / fmax(n1, n2);
  const double ar = swap ? bh : ah, bd = swap ? ah : bh;
  const float ratf = (float)ratio, arf = (float)ar, bdf = (float)bd;
  const double hi0 = 1.0 - 8.0 * kEps64;
  double sig = sigma_seed32(arf, bdf, (float)Lh, (float)(ah + bh), ratf);
  double lo = 0.0, hi = hi0;
  const bool flat = !(sig < (n_iter < 25 ? 0.75 : 0.99));
  if (flat) sig = sigma_budget64(ar, bd, Lh, ah + bh, ratio, n_iter);
  for (int it = 0; it < n_iter && !flat; ++it) {
    const double v = ratio * sig;
    const double r1 = rsqrt(fmax((1.0 - sig) * (1.0 + sig), kTiny));
    const double r2 = rsqrt(fmax((1.0 - v) * (1.0 + v), kTiny));
    const double F = (ar * sig * r1 + bd * v * r2) - Lh;
    if (F <= 0.0) lo = sig; else hi = sig;
    const float f1 = (float)r1, f2 = (float)r2;
    const float Fp = arf * f1 * f1 * f1 + bdf * ratf * f2 * f2 * f2;
    const double sn = sig - F * (double)(1.0f / fmaxf(Fp, 1e-30f));
    const bool ok = (sn >= lo) && (sn <= hi) && isfinite(sn);
    const double nxt = ok ? sn : 0.5 * (lo + hi);
    const bool done = fabs(nxt - sig) <= 1e-9 * fmax(sig, 1e-12);
    sig = nxt;
    if (done) break;
  }
  const double tr =
      ar * sig * rsqrt(fmax((1.0 - sig) * (1.0 + sig), kTiny));
  const double t = fmin(fmax(swap ? Lh - tr : tr, 0.0), Lh);
  const double st = s * t * iL;
  for (int j = 0; j < 3; ++j) R.x[j] = fp[j] + st * w[j];
  if (x_only) return;
  const double d2 = Lh - t;
  double r1, i1, r2, i2;
  sqrt_inv64(fmax(ah * ah + t * t, kTiny * kTiny), r1, i1);
  sqrt_inv64(fmax(bh * bh + d2 * d2, kTiny * kTiny), r2, i2);
  R.res = n1 * t * i1 - n2 * d2 * i2;
  R.s1 = s * r1;
  R.s2 = s * r2;
  R.c1 = ah * i1;
  R.c2 = bh * i2;
  R.valid = (h1 * h2 < 0.0) && (fabs(R.res) <= 1e-9);
}

// Affine (x, y) -> nearest cell; round half to even like np.round.
__device__ __forceinline__ void lookup64(const ss_interface &I, const double *x,
                                         double *pt, double *nr) {
  const double rc0 = __dadd_rn(__dadd_rn(__dmul_rn(x[0], I.coef[0]),
                                         __dmul_rn(x[1], I.coef[2])),
                               I.coef[4]);
  const double rc1 = __dadd_rn(__dadd_rn(__dmul_rn(x[0], I.coef[1]),
                                         __dmul_rn(x[1], I.coef[3])),
                               I.coef[5]);
  const int row = (int)fmin(fmax(rint(rc0), 0.0), (double)(I.ny - 1));
  const int col = (int)fmin(fmax(rint(rc1), 0.0), (double)(I.nx - 1));
  const float *g = I.table + ((size_t)row * I.nx + col) * 6;
  for (int j = 0; j < 3; ++j) {
    pt[j] = (double)g[j];
    nr[j] = (double)g[3 + j];
  }
}

// TE reflection between media i and i + 1 (physics.py:33-67); the roots and
// the quotient of the permittivities come from the host (RefArgs).
__device__ __forceinline__ double fresnel_gamma64(const RefArgs &a, int i,
                                                  double c1) {
  const double n1 = a.eps_root[i], n2 = a.eps_root[i + 1];
  const double s2 = a.eps_quot[i] * (1.0 - c1 * c1);
  const double c2 = sqrt(fmax(1.0 - s2, 0.0));
  return (n1 * c1 - n2 * c2) / (n1 * c1 + n2 * c2);
}

// ---------------------------------------------------------------------
// joint N-interface solve (refraction_joint.py:249-322)
// ---------------------------------------------------------------------
// Geometry of the polyline for in-plane offsets ab from the plane points:
// segment lengths and directions, in-plane projections of the incoming
// (pin) and outgoing (pout) directions, and the stationarity residual
// f_i = n_i pin_i - n_(i+1) pout_i. Lengths in units of the path scale.
template <int NI>
struct JointGeom {
  double y[NI][3], s[NI + 1], is[NI + 1], dh[NI + 1][3], pin[NI][2],
      pout[NI][2], f[NI][2], m;
};

template <int NI>
__device__ __forceinline__ void joint_geom(const double (&B)[NI][3][2],
                                           const double (&D)[NI + 1][3],
                                           const double *nm,
                                           const double (&ab)[NI][2],
                                           JointGeom<NI> &G, int ni = NI) {
  for (int i = 0; i < ni; ++i)
    for (int k = 0; k < 3; ++k)
      G.y[i][k] = B[i][k][0] * ab[i][0] + B[i][k][1] * ab[i][1];
  for (int k = 0; k <= ni; ++k) {
    double d[3];
    for (int j = 0; j < 3; ++j)
      d[j] = D[k][j] + ((k < ni ? G.y[k][j] : 0.0) -
                        (k > 0 ? G.y[k - 1][j] : 0.0));
    sqrt_inv64(fmax(dot3v(d, d), kTiny * kTiny), G.s[k], G.is[k]);
    for (int j = 0; j < 3; ++j) G.dh[k][j] = d[j] * G.is[k];
  }
  G.m = 0.0;
  for (int i = 0; i < ni; ++i)
    for (int c = 0; c < 2; ++c) {
      G.pin[i][c] = B[i][0][c] * G.dh[i][0] + B[i][1][c] * G.dh[i][1] +
                    B[i][2][c] * G.dh[i][2];
      G.pout[i][c] = B[i][0][c] * G.dh[i + 1][0] +
                     B[i][1][c] * G.dh[i + 1][1] +
                     B[i][2][c] * G.dh[i + 1][2];
      G.f[i][c] = nm[i] * G.pin[i][c] - nm[i + 1] * G.pout[i][c];
      G.m += G.f[i][c] * G.f[i][c];
    }
}

// Newton step delta at geometry G: the block-tridiagonal system assembled
// and solved (block Thomas, refraction_joint.py:218-246) in F. Only the
// residual needs float64 on the way to a root: a step with a float32 matrix
// leaves ~1e-7 of itself, less than the quadratic remainder of the first
// steps and less than an ulp of the last. With orthonormal in-plane bases the 2x2 blocks
// follow from the projections, B_i^T (n/s)(I - d d^T) B_j = (n/s)(B_i^T B_j
// - (B_i^T d)(B_j^T d)^T). Returns max |delta|.
template <int NI, class F>
__device__ __forceinline__ F joint_step(const JointGeom<NI> &G,
                                        const F (&BB)[NI][2][2],
                                        const double *nm, F (&delta)[NI][2],
                                        int ni) {
  const F mu = (F)1.8189894035458565e-12;  // Levenberg shift, eps^0.75
  F w[NI + 1], Cm[NI][2][2], dinv[NI][2][2], y[NI][2];
  for (int k = 0; k <= ni; ++k) w[k] = (F)(nm[k] * G.is[k]);
  for (int i = 0; i < ni; ++i) {
    const F p[2] = {(F)G.pin[i][0], (F)G.pin[i][1]};
    const F q[2] = {(F)G.pout[i][0], (F)G.pout[i][1]};
    F M[2][2], rhs[2] = {-(F)G.f[i][0], -(F)G.f[i][1]};
    for (int r = 0; r < 2; ++r)
      for (int c = 0; c < 2; ++c) {
        const F e = r == c ? (F)1 : (F)0;
        M[r][c] = w[i] * (e - p[r] * p[c]) + w[i + 1] * (e - q[r] * q[c]) +
                  e * mu;
      }
    if (i > 0) {
      F cpt[2][2];  // C_{i-1}^T dinv_{i-1}
      for (int r = 0; r < 2; ++r)
        for (int c = 0; c < 2; ++c)
          cpt[r][c] = Cm[i - 1][0][r] * dinv[i - 1][0][c] +
                      Cm[i - 1][1][r] * dinv[i - 1][1][c];
      for (int r = 0; r < 2; ++r) {
        for (int c = 0; c < 2; ++c)
          M[r][c] -= cpt[r][0] * Cm[i - 1][0][c] +
                     cpt[r][1] * Cm[i - 1][1][c];
        rhs[r] -= cpt[r][0] * y[i - 1][0] + cpt[r][1] * y[i - 1][1];
      }
    }
    F det = M[0][0] * M[1][1] - M[0][1] * M[1][0];
    if (fabs(det) < (F)1e-30) det = (F)1e-30;
    const F id = (F)1 / det;
    dinv[i][0][0] = M[1][1] * id;
    dinv[i][0][1] = -M[0][1] * id;
    dinv[i][1][0] = -M[1][0] * id;
    dinv[i][1][1] = M[0][0] * id;
    y[i][0] = rhs[0];
    y[i][1] = rhs[1];
    if (i + 1 < ni) {
      const F pn[2] = {(F)G.pin[i + 1][0], (F)G.pin[i + 1][1]};
      for (int r = 0; r < 2; ++r)
        for (int c = 0; c < 2; ++c)
          Cm[i][r][c] = -w[i + 1] * (BB[i][r][c] - q[r] * pn[c]);
    }
  }
  F dmax = (F)0;
  for (int i = ni - 1; i >= 0; --i) {
    F rr[2] = {y[i][0], y[i][1]};
    if (i < ni - 1)
      for (int r = 0; r < 2; ++r)
        rr[r] -= Cm[i][r][0] * delta[i + 1][0] + Cm[i][r][1] * delta[i + 1][1];
    for (int r = 0; r < 2; ++r) {
      delta[i][r] = dinv[i][r][0] * rr[0] + dinv[i][r][1] * rr[1];
      dmax = fmax(dmax, fabs(delta[i][r]));
    }
  }
  return dmax;
}

// One solve with step matrices in F; false when the step budget (or the
// halving) ran out before the steps became rounding.
template <int NI, class F>
static __device__ __noinline__ bool joint_solve64(
    const double *p, const double *q, const double (&O)[NI][3],
    const double (&Nn)[NI][3], const double *nm, int n_newton,
    int n_backtrack, double (&X)[NI][3], double (&cinc)[NI],
    double (&cout_)[NI], double (&S)[NI + 1], bool &valid, int ni) {
  // the path scale as a power of two: scaling rounds nothing
  const float pq[3] = {(float)(p[0] - q[0]), (float)(p[1] - q[1]),
                       (float)(p[2] - q[2])};
  const int ex = ilogbf(fmaxf(
      sqrtf(pq[0] * pq[0] + pq[1] * pq[1] + pq[2] * pq[2]), 1e-30f));
  const double scale = ldexp(1.0, ex), inv = ldexp(1.0, -ex);
  // in-plane bases (refraction_joint.py:196-204), segment bases and the
  // offsets of the chain of two-point solves (refraction.py) that starts
  // the joint solve
  double B[NI][3][2], D[NI + 1][3], ab[NI][2];
  double cur[3] = {p[0], p[1], p[2]};
  for (int i = 0; i < ni; ++i) {
    const double *n = Nn[i];
    const bool use_z = fabs(n[2]) < 0.9;
    const double a0 = use_z ? 0.0 : 1.0, a2 = use_z ? 1.0 : 0.0;
    double u[3] = {-a2 * n[1], a2 * n[0] - a0 * n[2], a0 * n[1]};
    const double un = rsqrt(fmax(dot3v(u, u), kTiny * kTiny));
    for (int j = 0; j < 3; ++j) u[j] *= un;
    const double v[3] = {n[1] * u[2] - n[2] * u[1], n[2] * u[0] - n[0] * u[2],
                         n[0] * u[1] - n[1] * u[0]};
    for (int j = 0; j < 3; ++j) {
      B[i][j][0] = u[j];
      B[i][j][1] = v[j];
      D[i][j] = (O[i][j] - (i == 0 ? p[j] : O[i - 1][j])) * inv;
    }
    Snell64 R;
    snell64(cur, q, O[i], n, nm[i], nm[i + 1], 25, R, true);
    double y[3];
    for (int j = 0; j < 3; ++j) {
      cur[j] = R.x[j];
      y[j] = (cur[j] - O[i][j]) * inv;
    }
    for (int c = 0; c < 2; ++c)
      ab[i][c] = B[i][0][c] * y[0] + B[i][1][c] * y[1] + B[i][2][c] * y[2];
  }
  for (int j = 0; j < 3; ++j) D[ni][j] = (q[j] - O[ni - 1][j]) * inv;
  F BB[NI][2][2];  // B_i^T B_{i+1}
  for (int i = 0; i + 1 < ni; ++i)
    for (int r = 0; r < 2; ++r)
      for (int c = 0; c < 2; ++c)
        BB[i][r][c] = (F)(B[i][0][r] * B[i + 1][0][c] +
                              B[i][1][r] * B[i + 1][1][c] +
                              B[i][2][r] * B[i + 1][2][c]);
  JointGeom<NI> G;
  joint_geom<NI>(B, D, nm, ab, G, ni);
  bool done = false;
  for (int it = 0; it < n_newton && !done; ++it) {
    F delta[NI][2];
    const F dmax = joint_step<NI, F>(G, BB, nm, delta, ni);
    // A step below 1e-9 of the shortest leg is rounding, and leaves 1e-18 of
    // it. (Of the path it would leave a metre-long leg under 20 km with a
    // residual past the validity limit.)
    double shortest = G.s[0];
    for (int i = 1; i <= ni; ++i) shortest = fmin(shortest, G.s[i]);
    const bool last = dmax < (F)1e-9 * (F)fmin(shortest, 1.0);
    // step halving on |F|^2; the accepted candidate's geometry is the next
    // iteration's
    const double m0 = G.m;
    double keep[NI][2];
    for (int i = 0; i < ni; ++i)
      for (int r = 0; r < 2; ++r) keep[i][r] = ab[i][r];
    double lam = 1.0;
    bool moved = false;
    for (int j = 0; j < n_backtrack; ++j, lam *= 0.5) {
      for (int i = 0; i < ni; ++i)
        for (int r = 0; r < 2; ++r)
          ab[i][r] = keep[i][r] + lam * (double)delta[i][r];
      joint_geom<NI>(B, D, nm, ab, G, ni);
      // in a last step the residual is rounding: the step itself is the
      // correction
      if (G.m < m0 || (last && isfinite(G.m))) {
        moved = true;
        break;
      }
    }
    if (!moved) {  // no step halving helps: every later iteration repeats
      for (int i = 0; i < ni; ++i)
        for (int r = 0; r < 2; ++r) ab[i][r] = keep[i][r];
      joint_geom<NI>(B, D, nm, ab, G, ni);
      break;
    }
    done = last;
  }
  // crossings, legs and validity (refraction_joint.py:143-176): with
  // orthonormal bases the in-plane parts are the projections
  double residual = 0.0;
  bool sides = true, evan = false, fin = true;
  for (int k = 0; k <= ni; ++k) {
    S[k] = G.s[k] * scale;
    fin = fin && isfinite(S[k]);
  }
  for (int i = 0; i < ni; ++i) {
    const double *n = Nn[i];
    for (int j = 0; j < 3; ++j) X[i][j] = O[i][j] + scale * G.y[i][j];
    const double ct1 = dot3v(n, G.dh[i]), ct2 = dot3v(n, G.dh[i + 1]);
    const double q1 = G.pin[i][0] * G.pin[i][0] + G.pin[i][1] * G.pin[i][1];
    const double q2 =
        G.pout[i][0] * G.pout[i][0] + G.pout[i][1] * G.pout[i][1];
    cinc[i] = fabs(ct1) * rsqrt(fmax(ct1 * ct1 + q1, kTiny));
    cout_[i] = fabs(ct2) * rsqrt(fmax(ct2 * ct2 + q2, kTiny));
    const double res = G.f[i][0] * G.f[i][0] + G.f[i][1] * G.f[i][1];
    if (res > residual || isnan(res)) residual = res;
    sides = sides && ct1 * ct2 > 0.0;
    const double lim = nm[i + 1] * (1.0 + 64.0 * kEps64);
    evan = evan || nm[i] * nm[i] * q1 > lim * lim;
    fin = fin && isfinite(X[i][0]) && isfinite(X[i][1]) && isfinite(X[i][2]);
  }
  valid = (residual <= 1e-18) && isfinite(residual) && fin && sides && !evan;
  return done;
}

// The joint solve (refraction_joint.py:249-322). A pair that the budget
// leaves short of its root is judged by the residual it stopped at, which a
// float32 matrix would leave elsewhere: those (none, as a rule) repeat the
// reference's float64 steps.
template <int NI>
static __device__ __forceinline__ void joint64(
    const double *p, const double *q, const double (&O)[NI][3],
    const double (&Nn)[NI][3], const double *nm, int n_newton,
    int n_backtrack, double (&X)[NI][3], double (&cinc)[NI],
    double (&cout_)[NI], double (&S)[NI + 1], bool &valid, int ni = NI) {
  if (!joint_solve64<NI, float>(p, q, O, Nn, nm, n_newton, n_backtrack, X,
                                cinc, cout_, S, valid, ni))
    joint_solve64<NI, double>(p, q, O, Nn, nm, n_newton, n_backtrack, X, cinc,
                              cout_, S, valid, ni);
}

// Path result shared by both solvers (multilayer.py `path` returns).
struct Path64 {
  double d[3], xf[3];  // last crossing - q; first crossing
  bool valid;
  double opl, loss_db, sum_par, sum_perp, tau2, c0, c_last;
};

// The plane of each lookup of the sequential chain: anchored by the float64
// mean-plane crossing.
struct Cell64 {
  __device__ __forceinline__ void operator()(const RefArgs &a, int i,
                                             const double *cur,
                                             const double *q, double *pt,
                                             double *nr) const {
    const ss_interface &I = a.ifc[i];
    Snell64 R;
    snell64(cur, q, I.mean_point, I.mean_normal, a.n_leg[i], a.n_leg[i + 1],
            10, R, true);
    lookup64(I, R.x, pt, nr);
  }
};

template <typename Cell>
static __device__ __forceinline__ void path_chain64(const RefArgs &a,
                                                    const double *p,
                                                    const double *q, Path64 &P,
                                                    Cell cell) {
  double cur[3] = {p[0], p[1], p[2]};
  P.valid = true;
  P.opl = P.loss_db = P.sum_par = P.sum_perp = 0.0;
  P.tau2 = 1.0;
  P.c0 = P.c_last = 1.0;
  for (int i = 0; i < a.ni; ++i) {
    const double n1 = a.n_leg[i], n2 = a.n_leg[i + 1];
    double pt[3], nr[3];
    cell(a, i, cur, q, pt, nr);
    const double inn = rsqrt(dot3v(nr, nr));
    for (int j = 0; j < 3; ++j) nr[j] *= inn;
    Snell64 R;
    snell64(cur, q, pt, nr, n1, n2, 25, R);
    P.valid = P.valid && R.valid;
    const double c_inc = fmax(R.c1, kCMin);
    if (i == 0) {
      P.c0 = c_inc;
      for (int j = 0; j < 3; ++j) P.xf[j] = R.x[j];
    }
    const double g = fresnel_gamma64(a, i, c_inc);
    P.tau2 = P.tau2 * (1.0 - g * g);
    if (a.rough_cross) {
      const double kt = a.k0 * (n1 * c_inc - n2 * R.c2);
      const double sk = a.sig_c[i] * kt;
      P.tau2 = P.tau2 * exp(-2.0 * (sk * sk));
    }
    P.opl = P.opl + n1 * R.s1;
    P.loss_db = P.loss_db + R.s1 * a.att_m[i];
    const double sn = R.s1 * a.inv_n[i];
    P.sum_perp = P.sum_perp + sn;
    P.sum_par = P.sum_par + sn / (c_inc * c_inc);
    P.c_last = fmax(R.c2, kCMin);
    for (int j = 0; j < 3; ++j) cur[j] = R.x[j];
  }
  for (int j = 0; j < 3; ++j) P.d[j] = cur[j] - q[j];
}

static __device__ __noinline__ void path_sequential64(const RefArgs &a,
                                                      const double *p,
                                                      const double *q,
                                                      Path64 &P) {
  path_chain64(a, p, q, P, Cell64());
}

template <int NI>
static __device__ __noinline__ void path_joint64(const RefArgs &a, const double *p,
                             const double *q, Path64 &P) {
  // a deep stack (NI == kDeepNI) holds up to NI interfaces in its arrays
  // and crosses a.ni of them; the other instantiations fold ni to NI
  const int ni = NI == kDeepNI ? a.ni : NI;
  // pass 1: mean-plane chain (10 iterations) anchors the lookups
  double pt[NI][3], nr[NI][3];
  {
    double cur[3] = {p[0], p[1], p[2]};
    for (int i = 0; i < ni; ++i) {
      Snell64 R;
      snell64(cur, q, a.ifc[i].mean_point, a.ifc[i].mean_normal, a.n_leg[i],
              a.n_leg[i + 1], 10, R, true);
      for (int j = 0; j < 3; ++j) cur[j] = R.x[j];
      lookup64(a.ifc[i], R.x, pt[i], nr[i]);
      const double nn = rsqrt(dot3v(nr[i], nr[i]));
      for (int j = 0; j < 3; ++j) nr[i][j] = nr[i][j] * nn;
    }
  }
  double X[NI][3], cinc[NI], cout_[NI], S[NI + 1];
  bool valid;
  joint64<NI>(p, q, pt, nr, a.n_leg, a.n_newton, a.n_backtrack, X, cinc,
              cout_, S, valid, ni);
  P.valid = valid;
  const double c_surf = fmax(cinc[a.k_pad], kCMin);
  double tau2 = 1.0, opl = 0.0, loss = 0.0, sperp = 0.0, spar = 0.0;
  for (int i = 0; i < ni; ++i) {
    const double ci = fmax(cinc[i], kCMin);
    const double g = fresnel_gamma64(a, i, ci);
    tau2 *= (1.0 - g * g);
    if (a.rough_cross) {
      const double kt =
          a.k0 * (a.n_leg[i] * cinc[i] - a.n_leg[i + 1] * cout_[i]);
      const double sk = a.sig_c[i] * kt;
      tau2 *= exp(-2.0 * (sk * sk));
    }
    const double cp = i < a.k_pad ? c_surf : ci;
    const double sn = S[i] * a.inv_n[i];
    opl += a.n_leg[i] * S[i];
    loss += S[i] * a.att_m[i];
    sperp += sn;
    spar += sn / (cp * cp);
  }
  P.tau2 = tau2;
  P.opl = opl;
  P.loss_db = loss;
  P.sum_perp = sperp;
  P.sum_par = spar;
  P.c0 = c_surf;
  P.c_last = fmax(cout_[ni - 1], kCMin);
  for (int j = 0; j < 3; ++j) {
    P.d[j] = X[ni - 1][j] - q[j];
    P.xf[j] = X[0][j];
  }
}

// Full float64 optical path length (crossing legs + final leg) and path
// validity for one pair: the exact reference quantity the split kernel falls
// back to when a pair sits within the bin-edge guard band.
template <int NI>
static __device__ __noinline__ double full_opl64(const RefArgs &a, const double *p,
                                    const double *q, bool &valid) {
  Path64 P;
  if (NI == 0)
    path_sequential64(a, p, q, P);
  else
    path_joint64<NI == 0 ? 1 : NI>(a, p, q, P);
  valid = P.valid;
  return P.opl + a.n_leg[a.leg_last] * sqrt(dot3v(P.d, P.d));
}

}  // namespace ss
