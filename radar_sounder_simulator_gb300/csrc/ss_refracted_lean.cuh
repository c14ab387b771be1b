// Split form of the joint refracted pair through one to four interfaces,
// laid out for few instructions (the kernels are bound by the FP32 issue
// rate: 4,300 warp instructions per pair through three interfaces in the
// general form of ss_refracted_split.cuh).
//
//   * As in the single-crossing path (ss_refracted_one.cuh), vectors are
//     relative to the target facet's centroid q, the mean planes' heights
//     over q and the cells of q's feet are formed once per facet, and each
//     two-point solve of the mean-plane chain starts within one Newton step
//     of its root.
//   * A crossing is (x, y) with its height on the looked-up facet plane, z =
//     c + sx x + sy y: the plane's basis (1, 0, sx), (0, 1, sy) needs no
//     construction and a projection on it two multiply-adds. Newton's method
//     does not depend on the basis, so its iterates are those of the
//     reference's orthonormal one (refraction_joint.py:249-322). The optical
//     path is convex in the crossings (a sum of lengths of affine maps), so
//     full steps converge; a pair that has not settled within the call's
//     step budget is left to the fix-up and the general form's step halving.
//   * The residual, the legs' lengths and the heights off the planes are as
//     in the general form; transmission takes both Snell cosines.
//
// 512^2 facets x 1024 traces through three interfaces: 43.8 -> 20.6 ms (2,060
// instructions per pair; issue 77% at 16 warps per SM, FMA pipe 60%).
#pragma once

#include "ss_refracted_one.cuh"

namespace ss {

constexpr int kLeanMax = 4;

// Planes whose normal leans further than this from the vertical (cosine)
// have no usable height-field basis: their pairs are left to the fix-up.
constexpr float kLeanMinNz = 0.1f;

// Per-facet constants of every interface's lookup, one column per thread in
// shared memory (kOnePerIface floats per interface and thread).
constexpr int kOnePerIface = 5;

struct LeanLegs {
  float n[kLeanMax + 1], nl[kLeanMax + 1], inv[kLeanMax + 1],
      x[kLeanMax + 1];
};

template <int NI>
__device__ __forceinline__ void lean_facet(const OnePlane *M, const float *q,
                                           float *col, int stride) {
#pragma unroll
  for (int i = 0; i < NI; ++i) {
    OneFacet f;
    one_facet(M[i], q, f);
    float *c = col + (size_t)i * kOnePerIface * stride;
    c[0] = f.b;
    c[stride] = f.ri[0];
    c[2 * stride] = f.ri[1];
    c[3 * stride] = f.rf[0];
    c[4 * stride] = f.rf[1];
  }
}

// Newton step (tx, ty) of the crossings of a polyline with unit leg
// directions d, weights w = n / length and gradient (f0, f1), which it uses
// up: blocks of the Hessian from p = B^T d_i and r = B^T d_(i+1), block
// elimination and back substitution. Returns the step's size (a NaN stays
// in it).
template <int NI>
__device__ __forceinline__ float lean_step(
    const float (&w)[NI + 1], const float (&d)[NI + 1][3],
    const float (&sx)[NI], const float (&sy)[NI], float (&f0)[NI],
    float (&f1)[NI], float (&tx)[NI], float (&ty)[NI]) {
  float a00[NI], a01[NI], a11[NI], C[NI][4];
#pragma unroll
  for (int i = 0; i < NI; ++i) {
    const float p0 = __fmaf_rn(sx[i], d[i][2], d[i][0]);
    const float p1 = __fmaf_rn(sy[i], d[i][2], d[i][1]);
    const float r0 = __fmaf_rn(sx[i], d[i + 1][2], d[i + 1][0]);
    const float r1 = __fmaf_rn(sy[i], d[i + 1][2], d[i + 1][1]);
    const float ws = w[i] + w[i + 1];
    const float wp0 = w[i] * p0, wp1 = w[i] * p1;
    const float wr0 = w[i + 1] * r0, wr1 = w[i + 1] * r1;
    const float g01 = sx[i] * sy[i];
    a00[i] = __fmaf_rn(-wp0, p0, __fmaf_rn(-wr0, r0,
                 ws * __fmaf_rn(sx[i], sx[i], 1.0f)));
    a01[i] = __fmaf_rn(-wp0, p1, __fmaf_rn(-wr0, r1, ws * g01));
    a11[i] = __fmaf_rn(-wp1, p1, __fmaf_rn(-wr1, r1,
                 ws * __fmaf_rn(sy[i], sy[i], 1.0f)));
    if (i + 1 < NI) {
      // C_i = -w B_i^T (I - d d^T) B_(i+1) of the shared leg
      const float m0 = __fmaf_rn(sx[i + 1], d[i + 1][2], d[i + 1][0]);
      const float m1 = __fmaf_rn(sy[i + 1], d[i + 1][2], d[i + 1][1]);
      const float ww = w[i + 1];
      C[i][0] = __fmaf_rn(wr0, m0, -ww * __fmaf_rn(sx[i], sx[i + 1], 1.0f));
      C[i][1] = __fmaf_rn(wr0, m1, -ww * (sx[i] * sy[i + 1]));
      C[i][2] = __fmaf_rn(wr1, m0, -ww * (sy[i] * sx[i + 1]));
      C[i][3] = __fmaf_rn(wr1, m1, -ww * __fmaf_rn(sy[i], sy[i + 1], 1.0f));
    }
    if (i > 0) {
      // minus C^T A^-1 of the interface above (a: its inverse)
      const float u00 = C[i - 1][0] * a00[i - 1] + C[i - 1][2] * a01[i - 1];
      const float u01 = C[i - 1][0] * a01[i - 1] + C[i - 1][2] * a11[i - 1];
      const float u10 = C[i - 1][1] * a00[i - 1] + C[i - 1][3] * a01[i - 1];
      const float u11 = C[i - 1][1] * a01[i - 1] + C[i - 1][3] * a11[i - 1];
      a00[i] -= u00 * C[i - 1][0] + u01 * C[i - 1][2];
      a01[i] -= u00 * C[i - 1][1] + u01 * C[i - 1][3];
      a11[i] -= u10 * C[i - 1][1] + u11 * C[i - 1][3];
      f0[i] -= u00 * f0[i - 1] + u01 * f1[i - 1];
      f1[i] -= u10 * f0[i - 1] + u11 * f1[i - 1];
    }
    const float id = rcp_n(a00[i] * a11[i] - a01[i] * a01[i]);
    const float b00 = a11[i] * id, b11 = a00[i] * id;
    a01[i] = -a01[i] * id;
    a00[i] = b00;
    a11[i] = b11;
  }
  float big = 0.0f;
#pragma unroll
  for (int i = NI - 1; i >= 0; --i) {
    float g0 = f0[i], g1 = f1[i];
    if (i + 1 < NI) {
      const float t0 = tx[i + 1 < NI ? i + 1 : i];
      const float t1 = ty[i + 1 < NI ? i + 1 : i];
      g0 -= C[i][0] * t0 + C[i][1] * t1;
      g1 -= C[i][2] * t0 + C[i][3] * t1;
    }
    tx[i] = a00[i] * g0 + a01[i] * g1;
    ty[i] = a01[i] * g0 + a11[i] * g1;
    big += fabsf(tx[i]) + fabsf(ty[i]);
  }
  return big;
}

// Table cells of a pair, the looked-up planes' slopes over q and the
// crossings (X, Y, Z) from q; P = p - q. False when the pair needs the
// fix-up (a cell decision near a boundary, a steep plane, an unsettled
// solve).
template <int NI, int SOLVE = kLookup>
__device__ __forceinline__ bool lean_solve(
    const OnePlane *M, const LeanLegs &k, const ss_interface *ifc,
    int n_newton, const float *col, int stride, const float *q,
    const float (&P)[3], int (&cell)[NI], float (&sx)[NI], float (&sy)[NI],
    float (&X)[NI], float (&Y)[NI], float (&Z)[NI]) {
  float c[NI];
  // mean-plane chain: cells and the crossings that start the solve
  {
    float v[3] = {P[0], P[1], P[2]};
    bool safe = true;
#pragma unroll
    for (int i = 0; i < NI; ++i) {
      const float *fc = col + (size_t)i * kOnePerIface * stride;
      OneFacet f;
      f.b = fc[0];
      f.ri[0] = fc[stride];
      f.ri[1] = fc[2 * stride];
      f.rf[0] = fc[3 * stride];
      f.rf[1] = fc[4 * stride];
      safe = one_cell<SOLVE>(M[i], f, v, ifc[i].ny, ifc[i].nx, 1.0f + 0.5f * i,
                             cell[i], v) && safe;
      // the looked-up plane as a height field over q, and the crossing moved
      // vertically onto it
      float o[3], t[3];
      load_plane(M[i].vec, ifc[i].table, cell[i], o, t);
      safe = safe && fabsf(t[2]) > kLeanMinNz;
      const float iz = rcp_n(t[2]);
      sx[i] = -t[0] * iz;
      sy[i] = -t[1] * iz;
      c[i] = (o[2] - q[2]) -
             __fmaf_rn(sx[i], o[0] - q[0], sy[i] * (o[1] - q[1]));
      X[i] = v[0];
      Y[i] = v[1];
    }
    if (!safe) return false;
  }
  auto heights = [&]() {
#pragma unroll
    for (int i = 0; i < NI; ++i)
      Z[i] = __fmaf_rn(sx[i], X[i], __fmaf_rn(sy[i], Y[i], c[i]));
  };
  // Newton on the stationarity of the optical path
  heights();
  bool settled = false;
#pragma unroll 1
  for (int it = 0; it < n_newton && !settled; ++it) {
    float w[NI + 1], d[NI + 1][3], reach = 0.0f;
#pragma unroll
    for (int s = 0; s <= NI; ++s) {
      const float ux = s == 0 ? P[0] : X[s == 0 ? 0 : s - 1];
      const float uy = s == 0 ? P[1] : Y[s == 0 ? 0 : s - 1];
      const float uz = s == 0 ? P[2] : Z[s == 0 ? 0 : s - 1];
      const float dx = s == NI ? ux : ux - X[s == NI ? 0 : s];
      const float dy = s == NI ? uy : uy - Y[s == NI ? 0 : s];
      const float dz = s == NI ? uz : uz - Z[s == NI ? 0 : s];
      const float l2 = fmaxf(dot3f(dx, dy, dz, dx, dy, dz), 1e-20f);
      const float il = rsq_n(l2);
      if (s == 0) reach = l2 * il;
      w[s] = k.n[s] * il;
      d[s][0] = dx * il;
      d[s][1] = dy * il;
      d[s][2] = dz * il;
    }
    // gradient F_i = B_i^T (n_(i+1) d_(i+1) - n_i d_i)
    float f0[NI], f1[NI], tx[NI], ty[NI];
#pragma unroll
    for (int i = 0; i < NI; ++i) {
      const float p0 = __fmaf_rn(sx[i], d[i][2], d[i][0]);
      const float p1 = __fmaf_rn(sy[i], d[i][2], d[i][1]);
      const float r0 = __fmaf_rn(sx[i], d[i + 1][2], d[i + 1][0]);
      const float r1 = __fmaf_rn(sy[i], d[i + 1][2], d[i + 1][1]);
      f0[i] = __fmaf_rn(k.n[i + 1], r0, -k.n[i] * p0);
      f1[i] = __fmaf_rn(k.n[i + 1], r1, -k.n[i] * p1);
    }
    const float big = lean_step<NI>(w, d, sx, sy, f0, f1, tx, ty);
#pragma unroll
    for (int i = 0; i < NI; ++i) {
      X[i] -= tx[i];
      Y[i] -= ty[i];
    }
    heights();
    // a step of 1e-5 of the path leaves ~1e-10 of it in the crossing, whose
    // effect on the optical path is second order
    settled = big < 1e-5f * reach;
  }
  return settled;
}

// One pair; false when it needs the fix-up.
template <int NI>
__device__ __forceinline__ bool lean_path(
    const OnePlane *M, const LeanLegs &k, const ss_interface *ifc, int k_pad,
    int n_newton, const float *col, int stride, const float *q, float4 A,
    float2 Bp, float tol, PairGeo &G) {
  const float P[3] = {A.x - q[0], A.y - q[1], A.z - q[2]};
  int cell[NI];
  float X[NI], Y[NI], Z[NI], sx[NI], sy[NI];
  if (!lean_solve<NI>(M, k, ifc, n_newton, col, stride, q, P, cell, sx, sy, X,
                      Y, Z))
    return false;
  // legs as double-floats, cosines, residual, heights off the planes
  float uh[3], ul[3], is = 0.0f;
  float opl_h = 0.0f, opl_l = 0.0f, dopl = 0.0f, expo = 0.0f, perp = 0.0f;
  float num = 1.0f, den = 1.0f;   // tau^2 as a quotient
  float res = 0.0f, cin[NI], cout = 1.0f, len[NI + 1];
  float dprev[3] = {0.0f, 0.0f, 0.0f};
  bool ok = true;
#pragma unroll
  for (int s = 0; s <= NI; ++s) {
    df S;
    float dir[3];
    if (s == NI) {
      S = norm3_exact(X[NI - 1], Y[NI - 1], Z[NI - 1], is);
      dir[0] = X[NI - 1];
      dir[1] = Y[NI - 1];
      dir[2] = Z[NI - 1];
    } else {
      const float xs[3] = {X[s == NI ? 0 : s], Y[s == NI ? 0 : s],
                           Z[s == NI ? 0 : s]};
      if (s == 0) {
        float Ph[3], Pl[3];
        one_offset(A, Bp, q, Ph, Pl);
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          float e;
          two_sum(Ph[j], -xs[j], uh[j], e);
          ul[j] = e + Pl[j];
          G.d0[j] = -uh[j];
        }
      } else {
        const float xa[3] = {X[s == 0 ? 0 : s - 1], Y[s == 0 ? 0 : s - 1],
                             Z[s == 0 ? 0 : s - 1]};
#pragma unroll
        for (int j = 0; j < 3; ++j) two_sum(xa[j], -xs[j], uh[j], ul[j]);
      }
      S = norm3_df(uh, ul, is);
#pragma unroll
      for (int j = 0; j < 3; ++j) dir[j] = uh[j];
    }
#pragma unroll
    for (int j = 0; j < 3; ++j) dir[j] *= is;
    len[s] = S.hi;
    // optical path
    float p, e, t, z;
    two_prod(k.n[s], S.hi, p, e);
    e = __fmaf_rn(k.n[s], S.lo, __fmaf_rn(k.nl[s], S.hi, e));
    two_sum(opl_h, p, t, z);
    opl_h = t;
    opl_l += z + e;
    expo = __fmaf_rn(S.hi, k.x[s], expo);
    perp = __fmaf_rn(S.hi, k.inv[s], perp);
    if (s > 0) {
      // interface s - 1, between legs s - 1 (dprev) and s (dir)
      const int i = s - 1;
      float o[3], tn[3];
      load_plane(M[i].vec, ifc[i].table, cell[i], o, tn);
      const float g2 = __fmaf_rn(sy[i], sy[i], __fmaf_rn(sx[i], sx[i], 1.0f));
      const float in = rsq_n(g2);  // 1 / sqrt(1 + sx^2 + sy^2)
      // cosines to the unit normal (-sx, -sy, 1) in
      const float u1 = __fmaf_rn(-sx[i], dprev[0],
                                 __fmaf_rn(-sy[i], dprev[1], dprev[2])) * in;
      const float u2 = __fmaf_rn(-sx[i], dir[0],
                                 __fmaf_rn(-sy[i], dir[1], dir[2])) * in;
      ok = ok && u1 * u2 > 0.0f;
      const float c1 = fabsf(u1);
      cout = fabsf(u2);
      cin[i] = c1;
      const float p0 = __fmaf_rn(sx[i], dprev[2], dprev[0]);
      const float p1 = __fmaf_rn(sy[i], dprev[2], dprev[1]);
      const float r0 = __fmaf_rn(sx[i], dir[2], dir[0]);
      const float r1 = __fmaf_rn(sy[i], dir[2], dir[1]);
      const float h0 = __fmaf_rn(k.n[i + 1], r0, -k.n[i] * p0);
      const float h1 = __fmaf_rn(k.n[i + 1], r1, -k.n[i] * p1);
      // in-plane residual: F^T (B^T B)^-1 F = |F|^2 - (F.s)^2 / (1 + |s|^2)
      const float fs = __fmaf_rn(h0, sx[i], h1 * sy[i]) * in;
      res = fmaxf(res, __fmaf_rn(-fs, fs, __fmaf_rn(h0, h0, h1 * h1)));
      // beyond the critical angle (refraction_joint.py:172)
      const float n1s = k.n[i] * k.n[i], n2s = k.n[i + 1] * k.n[i + 1];
      ok = ok && !(n1s * __fmaf_rn(-c1, c1, 1.0f) > n2s * 1.000016f);
      const float a = k.n[i] * c1, b = k.n[i + 1] * cout;
      num *= 4.0f * a * b;
      den *= (a + b) * (a + b);
      // height over the plane of the stored normal, towards the upper point
      const float yv[3] = {X[i], Y[i], Z[i]};
      float hp = plane_offset(yv, o, q, tn);
      hp = (u1 >= 0.0f) == (tn[2] >= 0.0f) ? hp : -hp;
      dopl = __fmaf_rn(hp, a - b, dopl);
    }
#pragma unroll
    for (int j = 0; j < 3; ++j) dprev[j] = dir[j];
  }
  G.opl = df_make(opl_h, opl_l + dopl);
  G.valid = ok && res <= tol * tol;
  G.att = exp2_n(expo);
  // spreading: l_perp = n0 sum(s/n), l_par = n0 c0^2 sum(s / (n c^2)), flux
  // = n0 c0 / (nj c_last)
  const float cl = fmaxf(cout, 1e-9f);
  float c0 = 1.0f;
#pragma unroll
  for (int i = 0; i < NI; ++i)
    if (i == k_pad) c0 = fmaxf(cin[i], 1e-9f);
  float par = len[NI] * k.inv[NI] * rcp_n(cl * cl);
#pragma unroll
  for (int i = 0; i < NI; ++i) {
    const float ci = i < k_pad ? c0 : fmaxf(cin[i], 1e-9f);
    par = __fmaf_rn(len[i] * k.inv[i], rcp_n(ci * ci), par);
  }
  G.spread = num * rcp_n(den * (k.n[NI] * cl * k.n[0] * c0) * (par * perp));
#pragma unroll
  for (int j = 0; j < 3; ++j) G.rh[j] = dprev[j];
  return true;
}

}  // namespace ss
