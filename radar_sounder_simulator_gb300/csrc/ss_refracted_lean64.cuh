// float64 refracted paths with their float32 part where float32 decides or
// only starts an iteration (FP64 kernel, one to four interfaces).
//
// The float64 pipe runs at 1/64 of the float32 rate, so a pair's cost is its
// count of float64 operations. Two parts of the path need none:
//   * the mean-plane chain only picks table cells. The float32 chain of the
//     split form (ss_refracted_one.cuh) picks the same ones except within a
//     guard band of a cell boundary and for flat rays (beyond 49 degrees on
//     the rarer side), where the float64 chain decides;
//   * Newton's method for the joint crossings forgets its start. The float32
//     solve of ss_refracted_lean.cuh ends ~1e-7 from the root; from there
//     each step with a float64 residual and a float32 matrix gains ~6 digits,
//     so one is enough, as a rule, where a float64 solve from the chain of
//     two-point crossings takes three or four residuals and that chain.
// A joint pair the float32 solve leaves unsettled takes the float64 form.
// Crossings are height fields over the facet's centroid (basis (1, 0, sx),
// (0, 1, sy)): a projection takes one multiply-add, the orthonormal basis
// six operations and its construction thirty.
//
// 120x96 facets x 40 traces through two interfaces: 2.02 -> 0.64 ms (FP64 pipe
// 74%).
#pragma once

#include "ss_refracted_fp64.cuh"
#include "ss_refracted_lean.cuh"

namespace ss {

struct Lean64Consts {
  OnePlane pl[kLeanMax];
  LeanLegs legs;
};

// 1 / x for |x| within float32's normal range: a float32 seed and two Newton
// steps (error 2e-14, then rounding), free of the float64 quotient's range
// handling.
__device__ __forceinline__ double rcp64(double x) {
  double y = (double)rcp_n((float)x);
  y = fma(y, fma(-x, y, 1.0), y);
  return fma(y, fma(-x, y, 1.0), y);
}

// Residual below which the crossings count as converged, squared: 1e-12,
// near the rounding of the leg directions and a thousandth of the validity
// limit.
constexpr float kLeanRes64 = 1e-24f;

template <int NI>
static __device__ __forceinline__ bool lean_path64(
    const RefArgs &a, const Lean64Consts &k, const float *col, const float *qf,
    const double *p, const double *q, Path64 &P) {
  int cell[NI];
  float sf[NI], tf[NI];  // slopes
  double pq[3], x[NI], y[NI], z[NI], sx[NI], sy[NI], c[NI];
  for (int j = 0; j < 3; ++j) pq[j] = p[j] - q[j];
  {
    const float Pf[3] = {(float)pq[0], (float)pq[1], (float)pq[2]};
    float X[NI], Y[NI], Z[NI];
    // two steps fewer than the float64 form has: a pair that settles (a last
    // step of 1e-5) is then one that form converges too
    if (!lean_solve<NI, kLookup64>(k.pl, k.legs, a.ifc, a.n_newton - 2, col, 1, qf, Pf,
                        cell, sf, tf, X, Y, Z))
      return false;
#pragma unroll
    for (int i = 0; i < NI; ++i) {
      x[i] = X[i];
      y[i] = Y[i];
      float o[3], t[3];
      load_plane(k.pl[i].vec, a.ifc[i].table, cell[i], o, t);
      const double iz = rcp64((double)t[2]);
      sx[i] = -(double)t[0] * iz;
      sy[i] = -(double)t[1] * iz;
      c[i] = ((double)o[2] - q[2]) - sx[i] * ((double)o[0] - q[0]) -
             sy[i] * ((double)o[1] - q[1]);
    }
  }
  double d[NI + 1][3], l2[NI + 1], il[NI + 1];
  for (int it = 0;; ++it) {
#pragma unroll
    for (int i = 0; i < NI; ++i) z[i] = c[i] + sx[i] * x[i] + sy[i] * y[i];
#pragma unroll
    for (int s = 0; s <= NI; ++s) {
      const int u = s == 0 ? 0 : s - 1, v = s == NI ? 0 : s;
      const double dx = (s == 0 ? pq[0] : x[u]) - (s == NI ? 0.0 : x[v]);
      const double dy = (s == 0 ? pq[1] : y[u]) - (s == NI ? 0.0 : y[v]);
      const double dz = (s == 0 ? pq[2] : z[u]) - (s == NI ? 0.0 : z[v]);
      l2[s] = fmax(dx * dx + dy * dy + dz * dz, kTiny * kTiny);
      il[s] = rsqrt(l2[s]);
      d[s][0] = dx * il[s];
      d[s][1] = dy * il[s];
      d[s][2] = dz * il[s];
    }
    // gradient of the optical path, and its part in the planes squared
    float f0[NI], f1[NI], res = 0.0f;
#pragma unroll
    for (int i = 0; i < NI; ++i) {
      const double g0 = a.n_leg[i + 1] * (d[i + 1][0] + sx[i] * d[i + 1][2]) -
                        a.n_leg[i] * (d[i][0] + sx[i] * d[i][2]);
      const double g1 = a.n_leg[i + 1] * (d[i + 1][1] + sy[i] * d[i + 1][2]) -
                        a.n_leg[i] * (d[i][1] + sy[i] * d[i][2]);
      f0[i] = (float)g0;
      f1[i] = (float)g1;
      const float fs = __fmaf_rn(f0[i], sf[i], f1[i] * tf[i]);
      const float g2 = __fmaf_rn(tf[i], tf[i], __fmaf_rn(sf[i], sf[i], 1.0f));
      const float r = __fmaf_rn(f0[i], f0[i], f1[i] * f1[i]) -
                      fs * fs * rcp_n(g2);
      // (no maximum of a NaN)
      res = res > r ? res : r;
    }
    if (res <= kLeanRes64) break;
    if (it == 3 || !(res < 1.0f)) return false;
    float w[NI + 1], df_[NI + 1][3], tx[NI], ty[NI];
#pragma unroll
    for (int s = 0; s <= NI; ++s) {
      w[s] = k.legs.n[s] * (float)il[s];
      for (int j = 0; j < 3; ++j) df_[s][j] = (float)d[s][j];
    }
    lean_step<NI>(w, df_, sf, tf, f0, f1, tx, ty);
#pragma unroll
    for (int i = 0; i < NI; ++i) {
      x[i] -= (double)tx[i];
      y[i] -= (double)ty[i];
    }
  }
  double S[NI + 1], cinc[NI], cout_[NI];
#pragma unroll
  for (int s = 0; s <= NI; ++s) {
    S[s] = l2[s] * il[s];
    S[s] = fma(fma(-S[s], S[s], l2[s]), 0.5 * il[s], S[s]);
    if (!isfinite(S[s])) return false;
  }
#pragma unroll
  for (int i = 0; i < NI; ++i) {
    const double in = rsqrt(1.0 + sx[i] * sx[i] + sy[i] * sy[i]);
    const double u1 = (d[i][2] - sx[i] * d[i][0] - sy[i] * d[i][1]) * in;
    const double u2 =
        (d[i + 1][2] - sx[i] * d[i + 1][0] - sy[i] * d[i + 1][1]) * in;
    // wrong sides or beyond the critical angle: left to the float64 form
    if (!(u1 * u2 > 0.0)) return false;
    cinc[i] = fabs(u1);
    cout_[i] = fabs(u2);
    // near grazing the reference's start may be short of its root
    if (fmin(cinc[i], cout_[i]) < 0.15) return false;
    if (a.n_leg[i] * a.n_leg[i] * (1.0 - u1 * u1) >
        a.n_leg[i + 1] * a.n_leg[i + 1])
      return false;
  }
  P.valid = true;
  const double c_surf = fmax(cinc[a.k_pad], kCMin);
  const double i_surf = rcp64(c_surf * c_surf);
  double num = 1.0, den = 1.0, opl = 0.0, loss = 0.0, sperp = 0.0, spar = 0.0;
#pragma unroll
  for (int i = 0; i < NI; ++i) {
    const double ci = fmax(cinc[i], kCMin);
    // 1 - gamma^2 = 4 a b / (a + b)^2 of the index-weighted cosines, the
    // outgoing one from Snell's law as solved
    const double n1c = a.n_leg[i] * ci, n2c = a.n_leg[i + 1] * cout_[i];
    const double sum = n1c + n2c;
    num *= 4.0 * n1c * n2c;
    den *= sum * sum;
    const double ic = i < a.k_pad ? i_surf : rcp64(ci * ci);
    const double sn = S[i] * a.inv_n[i];
    opl += a.n_leg[i] * S[i];
    loss += S[i] * a.att_m[i];
    sperp += sn;
    spar += sn * ic;
  }
  P.tau2 = num * rcp64(den);
  P.opl = opl;
  P.loss_db = loss;
  P.sum_perp = sperp;
  P.sum_par = spar;
  P.c0 = c_surf;
  P.c_last = fmax(cout_[NI - 1], kCMin);
  P.d[0] = x[NI - 1];
  P.d[1] = y[NI - 1];
  P.d[2] = z[NI - 1];
  P.xf[0] = q[0] + x[0];
  P.xf[1] = q[1] + y[0];
  P.xf[2] = q[2] + z[0];
  return true;
}

// Cell and plane of interface i for the ray from `cur` to q, by the float32
// mean-plane crossing; false within the guard band.
__device__ __forceinline__ bool lean_cell64(const RefArgs &a,
                                            const Lean64Consts &k, int i,
                                            const float *col,
                                            const double *cur, const double *q,
                                            double *pt, double *nr) {
  OneFacet f;
  const float *c = col + i * kOnePerIface;
  f.b = c[0];
  f.ri[0] = c[1];
  f.ri[1] = c[2];
  f.rf[0] = c[3];
  f.rf[1] = c[4];
  const float V[3] = {(float)(cur[0] - q[0]), (float)(cur[1] - q[1]),
                      (float)(cur[2] - q[2])};
  int cell;
  float v[3], o[3], t[3];
  if (!one_cell<kLookup64>(k.pl[i], f, V, a.ifc[i].ny, a.ifc[i].nx, 1.0f + 0.5f * i,
                cell, v))
    return false;
  load_plane(k.pl[i].vec, a.ifc[i].table, cell, o, t);
  for (int j = 0; j < 3; ++j) {
    pt[j] = (double)o[j];
    nr[j] = (double)t[j];
  }
  return true;
}

static __device__ __noinline__ void path_lean_chain64(
    const RefArgs &a, const Lean64Consts &k, const float *col, const double *p,
    const double *q, Path64 &P) {
  path_chain64(a, p, q, P,
               [&](const RefArgs &a, int i, const double *cur, const double *q,
                   double *pt, double *nr) {
                 if (!lean_cell64(a, k, i, col, cur, q, pt, nr))
                   Cell64()(a, i, cur, q, pt, nr);
               });
}

}  // namespace ss
