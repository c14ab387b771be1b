// Split form of the refracted pair under one crossed interface (sequential
// solve): the path of every first-horizon and single-surface bed target.
//
// The kernel is bound by the FP32 issue rate, so this path is laid out for
// few instructions per pair:
//   * every vector is relative to the target facet's centroid q, where the
//     crossing is near: the crossing is a short float vector y, the lower
//     leg |y| needs no low parts, and p - q (a double-float) is formed once
//     for both solves;
//   * per facet and once for all traces of the block: the mean plane's
//     height over q and the affine cell of q's foot on it, as an integer and
//     a fraction. A pair's cell is that plus the crossing's offset, a
//     fraction g of the foot-to-foot vector, so its float32 error is ~1e-7
//     of the offset (1e-5 cells at a hundred cells), not of the distance to
//     the table's centre;
//   * the two-point root is the ray parameter sigma = sin(theta) of the
//     rare side. It starts from the paraxial form L / sqrt(L^2 + (a + r b)^2)
//     (r the index ratio) with the dense side's b corrected for its flatter
//     angle to fourth order, within 2e-4 up to 35 degrees (a float32 model
//     over 12-25 km altitude, 0.2-3 km depth), and one Newton step leaves
//     ~1e-7; steeper rays take a second. The iteration needs no bracket; one
//     that has not settled (grazing rays) falls back to the bracketed form;
//   * Fresnel transmission from the two cosines Snell's law already gives:
//     1 - gamma^2 = 4 n1 c1 n2 c2 / (n1 c1 + n2 c2)^2, and the spreading and
//     flux factors folded into one quotient.
//
// 512^2 facets x 1024 traces under one interface: 12.4 -> 5.3 ms (1,542 ->
// 640 instructions per pair; issue 88%, FMA pipe 60%).
#pragma once

#include "ss_df.cuh"
#include "ss_f32.cuh"

namespace ss {

// Root sigma of ar tan(theta) + bd tan(theta') = L, sin(theta') = r
// sin(theta), by bracketed Newton (refraction.py:120-144): the rays the
// short iteration below leaves unsettled.
static __device__ __noinline__ float sigma_bracketed(float ar, float bd,
                                                     float L, float r) {
  const float hi0 = 1.0f - 1e-6f;
  float lo = 0.0f, hi = hi0;
  float sig = fminf(L * rsqrtf(fmaxf(L * L + (ar + bd) * (ar + bd), 1e-30f)),
                    hi0);
  for (int it = 0; it < 25; ++it) {
    const float v = r * sig;
    const float r1 = rsqrtf(fmaxf((1.0f - sig) * (1.0f + sig), 1e-30f));
    const float r2 = rsqrtf(fmaxf((1.0f - v) * (1.0f + v), 1e-30f));
    const float F = (ar * sig * r1 + bd * v * r2) - L;
    if (F <= 0.0f) lo = sig; else hi = sig;
    const float Fp = ar * r1 * r1 * r1 + bd * r * r2 * r2 * r2;
    const float sn = sig - __fdividef(F, fmaxf(Fp, 1e-30f));
    const bool ok = (sn >= lo) && (sn <= hi);
    const float nxt = ok ? sn : 0.5f * (lo + hi);
    const bool done = fabsf(nxt - sig) <= 2.4e-7f * fmaxf(sig, 1e-6f);
    sig = nxt;
    if (done) break;
  }
  return sig;
}

// The reference's lookup solve stops after ten iterations (multilayer.py:
// 352-406), which reach the root for every sigma below 0.8 but leave some
// flat rays short of it (0.04% of those at 0.8-0.9, 1% at 0.98; a float64
// model over random heights, offsets and index ratios) and so pick other
// cells. The float64 form's lookups (kLookup64) leave every ray past kFlatRay
// to its float64 solve, which repeats those iterations; the split form takes
// the root (platforms 30-240 m over a kilometre of rough facets: 1e-6 to
// 2e-5 of the oracle, where the ten float32 iterations were no closer).
constexpr float kFlatRay = 0.75f;
enum { kOnFacet = 0, kLookup = 1, kLookup64 = 2 };

// Fraction of the way from q's foot to p's foot at which the refracted ray
// meets the plane: heights a of p and b of q over it, feet L apart (iL =
// 1/L), r = n_rare / n_dense, `up` when p is on the rare side. kLookup64: NaN
// for a flat ray.
template <int SOLVE>
__device__ __forceinline__ float cross_frac(float a, float b, float L,
                                            float L2, float iL, float r,
                                            float k2, float k4, bool up) {
  const float ar = up ? a : b, bd = up ? b : a;
  const float bdr = bd * r, m0 = ar + bdr;
  const float s0 = L * rsq_n(__fmaf_rn(m0, m0, L2)), x = s0 * s0;
  // tan(theta') / (r tan(theta)) = sqrt((1 - s^2) / (1 - r^2 s^2))
  const float kap = __fmaf_rn(x, __fmaf_rn(x, k4, k2), 1.0f);
  const float m = __fmaf_rn(bdr, kap, ar);
  float sig = L * rsq_n(__fmaf_rn(m, m, L2));
  float off = 0.0f;
  bool settled = false;
#pragma unroll 1
  for (int it = 0; it < 5; ++it) {
    const float v = r * sig;
    const float r1 = rsq_n(__fmaf_rn(-sig, sig, 1.0f));
    const float r2 = rsq_n(__fmaf_rn(-v, v, 1.0f));
    const float t1 = ar * r1, t2 = bdr * r2;
    const float F = __fmaf_rn(sig, t1 + t2, -L);
    const float q1 = r1 * r1, q2 = r2 * r2;
    const float d = F * rcp_n(__fmaf_rn(t1, q1, t2 * q2));
    // q's side offset at sigma - d, to second order in d
    off = up ? t2 * __fmaf_rn(-q2, d, sig) : t1 * __fmaf_rn(-q1, d, sig);
    sig -= d;
    // remaining error ~1.5 tan^2-weighted d^2: below 1.5e-7 of sigma
    settled = d * d * q1 <= 1e-7f * sig * sig;
    // q1 = 1 / (1 - sigma^2)
    if (SOLVE == kLookup64)
      settled = settled && q1 < 1.0f / (1.0f - kFlatRay * kFlatRay);
    if (settled) break;
  }
  if (SOLVE == kLookup64)
    return (settled ? off : __int_as_float(0x7fc00000)) * iL;
  if (!settled) {
    const float s = sigma_bracketed(ar, bd, L, r), v = r * s;
    off = up ? bd * v * rsqrtf(fmaxf((1.0f - v) * (1.0f + v), 1e-30f))
             : ar * s * rsqrtf(fmaxf((1.0f - s) * (1.0f + s), 1e-30f));
  }
  return fminf(fmaxf(off * iL, 0.0f), 1.0f);
}

// Mean plane and affine cell fit of a crossed interface for this path.
struct OnePlane {
  float mp[3], mn[3];      // mean point, unit mean normal
  float mpl[3], mnl[3];    // their low parts (the height over a facet)
  float c[4], cl[4];       // cell fit, row = c0 x + c2 y + c4 (double-float)
  float c4[2], c4l[2];
  float cn[2];             // d cell / d height along the normal
  float r, k2, k4;         // n_rare / n_dense, its paraxial corrections
  int up;                  // the upper medium is the rarer one
  int vec;                 // table rows can be read as float2
};

// Per facet: the mean plane's height over q, and the affine cell of q's
// foot as integer and fraction per axis.
struct OneFacet {
  float b, ri[2], rf[2];
};

__device__ __forceinline__ void one_facet(const OnePlane &M, const float *q,
                                          OneFacet &f) {
  // The height in double-float: from a float32 mean point it was off by up
  // to 1e-4 m at 3 km elevation, under shallow targets and fine grids more
  // than the guard band below (2.3 times it at 5 m cells and 1 m depth).
  {
    float d[3], l[3], p[3], e[3], s0, s1, t0, t1;
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      two_sum(q[j], -M.mp[j], d[j], l[j]);
      l[j] -= M.mpl[j];
      two_prod(d[j], M.mn[j], p[j], e[j]);
    }
    two_sum(p[0], p[1], s0, t0);
    two_sum(s0, p[2], s1, t1);
    f.b = -(s1 + (((t0 + t1) + (e[0] + e[1] + e[2])) +
                  (dot3f(d[0], d[1], d[2], M.mnl[0], M.mnl[1], M.mnl[2]) +
                   dot3f(l[0], l[1], l[2], M.mn[0], M.mn[1], M.mn[2]))));
  }
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    float p0, e0, p1, e1, s0, es, s1, es1;
    two_prod(q[0], M.c[c], p0, e0);
    two_prod(q[1], M.c[2 + c], p1, e1);
    two_sum(p0, p1, s0, es);
    two_sum(M.c4[c], s0, s1, es1);
    const float lo = ((es1 + es) + (e0 + e1)) + M.c4l[c] +
                     __fmaf_rn(q[0], M.cl[c], q[1] * M.cl[2 + c]);
    f.ri[c] = rintf(s1);
    f.rf[c] = ((s1 - f.ri[c]) + lo) + f.b * M.cn[c];
  }
}

// Guard band of the cell decision: kCellAbs + kCellRel x the crossing's
// offset from q's foot, in cells. A float32 model of these lines against
// float64 (twelve scenes of 1-2500 m depth, 50 m to 400 km altitude, 2-50 m
// cells, tilts to 0.1, elevations to 4.2 km, facets to 20 km out, index
// ratios either way, 300,000 pairs each) errs by at most 0.61 of the band
// (2.5 km under 50 m cells from a denser medium; 0.36 from a rarer one, 0.28
// below 300 m of depth).
// Down a chain of interfaces the error grows slowly (1.0e-6 at the third):
// `scale` widens the band there.
constexpr float kCellAbs = 5e-6f, kCellRel = 3e-6f;

// Cell of the mean-plane crossing of the ray from q + P to q, and that
// crossing from q (v, which may be P); false when a coordinate is within the
// guard band of a rounding boundary or the ray is one for float64 (a NaN
// crossing compares false).
template <int SOLVE = kLookup>
__device__ __forceinline__ bool one_cell(const OnePlane &M, const OneFacet &f,
                                         const float *P, int ny, int nx,
                                         float scale, int &cell, float *v) {
  const float vn = dot3f(P[0], P[1], P[2], M.mn[0], M.mn[1], M.mn[2]);
  const float wx = __fmaf_rn(-vn, M.mn[0], P[0]);
  const float wy = __fmaf_rn(-vn, M.mn[1], P[1]);
  const float wz = __fmaf_rn(-vn, M.mn[2], P[2]);
  const float L2 = fmaxf(dot3f(wx, wy, wz, wx, wy, wz), 1e-20f);
  const float iL = rsq_n(L2);
  const float a = fabsf(vn - f.b), b = fabsf(f.b);
  const float g =
      cross_frac<SOLVE>(a, b, L2 * iL, L2, iL, M.r, M.k2, M.k4, M.up);
  const float fr = __fmaf_rn(g, __fmaf_rn(M.c[0], wx, M.c[2] * wy), f.rf[0]);
  const float fc = __fmaf_rn(g, __fmaf_rn(M.c[1], wx, M.c[3] * wy), f.rf[1]);
  const float kr = rintf(fr), kc = rintf(fc);
  // clamped in float32, where the integers are exact
  const float row = fminf(fmaxf(f.ri[0] + kr, 0.0f), (float)(ny - 1));
  const float col = fminf(fmaxf(f.ri[1] + kc, 0.0f), (float)(nx - 1));
  cell = (int)row * nx + (int)col;
  v[0] = __fmaf_rn(g, wx, f.b * M.mn[0]);
  v[1] = __fmaf_rn(g, wy, f.b * M.mn[1]);
  v[2] = __fmaf_rn(g, wz, f.b * M.mn[2]);
  const float rel = kCellRel * scale;
  return fmaxf(__fmaf_rn(rel, fabsf(fr), fabsf(fr - kr)),
               __fmaf_rn(rel, fabsf(fc), fabsf(fc - kc))) <
         0.5f - kCellAbs * scale;
}

// |v| of a vector of floats taken as exact, as a double-float; `inv` its
// float32 reciprocal.
__device__ __forceinline__ df norm3_exact(float x, float y, float z,
                                          float &inv) {
  float qx, ex, qy, ey, qz, ez, s1, e1, sh, e2;
  two_prod(x, x, qx, ex);
  two_prod(y, y, qy, ey);
  two_prod(z, z, qz, ez);
  two_sum(qx, qy, s1, e1);
  two_sum(s1, qz, sh, e2);
  const float sl = (e1 + e2) + (ex + ey + ez);
  inv = rsq_n(fmaxf(sh, 1e-30f));
  const float r0 = sh * inv;
  const float res = __fmaf_rn(-r0, r0, sh) + sl;
  return df_make(r0, res * (0.5f * inv));
}

// The same of a double-float vector (low parts up to a few ulp).
__device__ __forceinline__ df norm3_df(const float *h, const float *l,
                                       float &inv) {
  float qx, ex, qy, ey, qz, ez, s1, e1, sh, e2;
  two_prod(h[0], h[0], qx, ex);
  two_prod(h[1], h[1], qy, ey);
  two_prod(h[2], h[2], qz, ez);
  two_sum(qx, qy, s1, e1);
  two_sum(s1, qz, sh, e2);
  const float sl = (e1 + e2) + (ex + ey + ez) +
                   2.0f * dot3f(h[0], h[1], h[2], l[0], l[1], l[2]);
  inv = rsq_n(fmaxf(sh, 1e-30f));
  const float r0 = sh * inv;
  const float res = __fmaf_rn(-r0, r0, sh) + sl;
  return df_make(r0, res * (0.5f * inv));
}

// Geometry of one pair, shared by every path: optical path, direction facet
// -> last crossing, spreading (transmission and flux included), attenuation
// exponent and the first leg's direction.
struct PairGeo {
  df opl;
  float rh[3], d0[3];  // d0: platform -> first crossing (any length)
  float spread;        // tau^2 flux / (l_par l_perp)
  float att;           // 10^(-loss/10)
  float dloss;         // d loss_db / d alpha (adjoint only)
  bool valid;
};

// Plane point o and stored normal t of a table cell.
__device__ __forceinline__ void load_plane(int vec,
                                           const float *__restrict__ table,
                                           int cell, float *o, float *t) {
  const float *g = table + (size_t)cell * 6;
  if (vec) {
    const float2 u0 = __ldg(reinterpret_cast<const float2 *>(g)),
                 u1 = __ldg(reinterpret_cast<const float2 *>(g) + 1),
                 u2 = __ldg(reinterpret_cast<const float2 *>(g) + 2);
    o[0] = u0.x; o[1] = u0.y; o[2] = u1.x;
    t[0] = u1.y; t[1] = u2.x; t[2] = u2.y;
  } else {
    for (int j = 0; j < 3; ++j) {
      o[j] = __ldg(g + j);
      t[j] = __ldg(g + 3 + j);
    }
  }
}

// t . (y - (o - q)) from exact differences and products: the height of the
// crossing q + y over the plane of normal t through o, to float32 precision
// of the height itself.
__device__ __forceinline__ float plane_offset(const float *y, const float *o,
                                              const float *q,
                                              const float *t) {
  float d[3], dl[3], p0, e0, p1, e1, p2, e2, sh, f1, f2;
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    float oh, ol;
    two_sum(o[j], -q[j], oh, ol);
    two_sum(y[j], -oh, d[j], dl[j]);
    dl[j] -= ol;
  }
  two_prod(d[0], t[0], p0, e0);
  two_prod(d[1], t[1], p1, e1);
  two_prod(d[2], t[2], p2, e2);
  two_sum(p0, p1, sh, f1);
  two_sum(sh, p2, sh, f2);
  return sh + ((f1 + f2) + (e0 + e1 + e2) +
               dot3f(dl[0], dl[1], dl[2], t[0], t[1], t[2]));
}

// Scalars of the one-crossing pair.
struct OneLegs {
  float n1, n1l, n2, n2l, i1, i2;  // indices (double-float), reciprocals
  float x1, x2;                    // -0.332 att / 1000: exp2 exponent per m
};

// p - q of a facet centroid and a double-float platform position.
__device__ __forceinline__ void one_offset(float4 A, float2 B, const float *q,
                                           float *Ph, float *Pl) {
  float e;
  two_sum(A.x, -q[0], Ph[0], e);
  Pl[0] = e + A.w;
  two_sum(A.y, -q[1], Ph[1], e);
  Pl[1] = e + B.x;
  two_sum(A.z, -q[2], Ph[2], e);
  Pl[2] = e + B.y;
}

// Path of one pair through the tangent plane of table cell `cell`.
__device__ __forceinline__ void one_path(const OnePlane &M, const OneLegs &k,
                                         const float *__restrict__ table,
                                         int cell, const float *q,
                                         const float *Ph, const float *Pl,
                                         float tol, PairGeo &G) {
  float o[3], t[3];
  load_plane(M.vec, table, cell, o, t);
  // unit normal to float32 rounding (one Newton step on the seed)
  const float nn = dot3f(t[0], t[1], t[2], t[0], t[1], t[2]);
  float in = rsq_n(nn);
  in = in * __fmaf_rn(-0.5f * nn * in, in, 1.5f);
  const float n[3] = {t[0] * in, t[1] * in, t[2] * in};
  const float b = dot3f(o[0] - q[0], o[1] - q[1], o[2] - q[2], n[0], n[1],
                        n[2]);
  const float vn = dot3f(Ph[0], Ph[1], Ph[2], n[0], n[1], n[2]);
  const float a = vn - b;
  float w[3];
#pragma unroll
  for (int j = 0; j < 3; ++j) w[j] = __fmaf_rn(-vn, n[j], Ph[j]);
  const float L2 =
      fmaxf(dot3f(w[0], w[1], w[2], w[0], w[1], w[2]), 1e-20f);
  const float iL = rsq_n(L2), L = L2 * iL;
  const float aa = fabsf(a), ab = fabsf(b);
  const float fg =
      cross_frac<kOnFacet>(aa, ab, L, L2, iL, M.r, M.k2, M.k4, M.up);
  // crossing from q; legs in double-float
  float y[3], uh[3], ul[3], is1, is2;
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    y[j] = __fmaf_rn(fg, w[j], b * n[j]);
    float e;
    two_sum(Ph[j], -y[j], uh[j], e);
    ul[j] = e + Pl[j];
  }
  const df s2 = norm3_exact(y[0], y[1], y[2], is2);
  const df s1 = norm3_df(uh, ul, is1);
  const float c1 = fmaxf(aa * is1, 1e-9f), c2 = fmaxf(ab * is2, 1e-9f);
  // The float32 crossing is off the plane of the stored normal by its
  // rounding (up to ~1e-4 m), which the optical path takes at first order;
  // its height over that plane towards the upper point, from exact
  // products, times the legs' index-weighted cosines puts it back.
  float hp = plane_offset(y, o, q, t);
  hp = a >= 0.0f ? hp : -hp;
  const float nc1 = k.n1 * c1, nc2 = k.n2 * c2;
  // optical path n1 s1 + n2 s2 + hp (n1 c1 - n2 c2)
  float q1, z1, q2, z2, qs, zs;
  two_prod(k.n1, s1.hi, q1, z1);
  two_prod(k.n2, s2.hi, q2, z2);
  two_sum(q1, q2, qs, zs);
  zs += (z1 + __fmaf_rn(k.n1, s1.lo, k.n1l * s1.hi)) +
        (z2 + __fmaf_rn(k.n2, s2.lo, k.n2l * s2.hi));
  G.opl = df_make(qs, __fmaf_rn(hp, nc1 - nc2, zs));
  // Snell residual (closure form, refraction.py:155) and side test
  const float tq = fg * L, tp = L - tq;
  const float res = k.n1 * tp * is1 - k.n2 * tq * is2;
  G.valid = a * b > 0.0f && fabsf(res) <= tol;
  // tau^2 flux / (l_par l_perp) with 1 - gamma^2 = 4 nc1 nc2 / D^2, D = nc1
  // + nc2; l_perp = n1 (s1/n1 + s2/n2), l_par = n1 c1^2 (s1/(n1 c1^2) +
  // s2/(n2 c2^2)), flux = nc1 / nc2
  const float D = nc1 + nc2;
  const float l1 = s1.hi * k.i1, l2 = s2.hi * k.i2;
  const float cc1 = c1 * c1, cc2 = c2 * c2;
  G.spread = 4.0f * cc1 * cc2 *
             rcp_n(D * D * ((l1 + l2) * __fmaf_rn(l1, cc2, l2 * cc1)));
  G.att = exp2_n(__fmaf_rn(s1.hi, k.x1, s2.hi * k.x2));
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    G.rh[j] = y[j] * is2;
    G.d0[j] = -uh[j];
  }
}

}  // namespace ss
