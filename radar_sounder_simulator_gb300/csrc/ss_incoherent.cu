// Incoherent (power-summing) facet kernel on GB300.
//
// Replaces the jitted program of soundersim kernels/incoherent.py:32-61:
// per facet and trace the power (A cos)^2 / r^4 (weighted g^4 by the antenna
// pattern), binned at floor((2r/c - t0)/dt), out-of-window power dropped into
// a per-trace scalar, optionally split into left/right halves by the sign of
// (c - p) . u_ct. Every facet is summed for every trace (the reference has no
// culling here).
//
// Everything is float32 like the reference. The bin is an integer decision
// that must match the reference's float32 chain
//   r = sqrt((dx^2 + dy^2) + dz^2), tw = (2 r) / c, u = (tw - t0) / dt
// bit for bit, with each operation rounded to nearest. The root is a MUFU
// reciprocal root's with one Newton step, which is the rounded one unless
// the exact root lies within 2^-14 ulp of a midpoint between two floats: the
// exact remainder S - r^2 tells, and those pairs (one in 16,000) take
// __fsqrt_rn. A quotient by a call constant b is x RN(1/b) with the
// reciprocal's low part (Brisebarre and Muller, "Correctly rounded
// multiplication by arbitrary precision constants"), right to an ulp, and one
// remainder step with RN(1/b), which rounds it correctly (Markstein,
// "Computation of elementary functions on the IBM RISC System/6000
// processor"; b's mantissa not all ones). So the chain is the reference's
// with no branch but the rare one, where a bounded estimate sent one pair in
// sixty -- 40% of the warps -- through the full root and quotients.
//
// The arithmetic runs on two traces at a time (packed float32: one issue
// slot for two results, rounded alike).
//
// Work decomposition: the grid is (facet chunks) x (trace blocks of TB
// traces). Each thread takes one facet at a time and evaluates it against
// the TB traces of its block, lane l starting at trace (l + s) mod TB on step
// s, so the 32 lanes of a warp -- 32 neighbouring facets, often in the same
// bin -- spread their shared-memory atomics over TB histograms instead of
// piling onto one address. Dropped power stays in registers (each step s
// maps a thread to one fixed trace). Per-CTA histograms go to scratch and a
// second kernel sums the chunks in a fixed order in float64.
//
// Bound by instruction issue (63 per pair, 68% of the slots at 32 warps per
// SM, a third of them the histogram's compare-and-swap loops): 512^2 facets x
// 1024 traces 855 -> 652 us.
#include <algorithm>
#include <cstdint>
#include <cstring>

#include "ss_chunksum.cuh"
#include "ss_f32.cuh"
#include "ss_f32x2.cuh"
#include "ss_internal.cuh"

namespace ss {

struct IncArgs {
  const float *cx, *cy, *cz, *nx, *ny, *nz, *area;
  const double *pos, *uct, *pv;
  int pv_len, T, N, n_samples, n_seg, stride, split;
  float t0, dt, c;  // window scalars rounded to float32
  // quotients by c / 2 and dt: the divisors negated, reciprocals, low parts
  float nhc, ndt, zc, zcl, zd, zdl;
  float mid;  // bound of the midpoint test, in r ulp(r); negative: exact chain
  int pat_kind, pat_n;
  const double *pa, *pb;
  int n_chunks;
  float *part;        // (n_chunks, T, n_seg) partial histograms
  double *part_drop;  // (n_chunks, T) partial dropped power
};

// Exactly rounded float32 bin coordinate of the reference (geometry.py:6-24).
static __device__ __noinline__ float bin_exact(float S, float c, float t0,
                                               float dt) {
  const float r = __fsqrt_rn(S);
  const float tw = __fdiv_rn(__fmul_rn(2.0f, r), c);
  return __fdiv_rn(__fsub_rn(tw, t0), dt);
}

// RN(x / b): z = RN(1/b), zl its low part, nb = -b.
__device__ __forceinline__ float2 div_const2(float2 x, float z, float zl,
                                             float nb) {
  const float2 q = fma2(x, pk1(z), mul2(x, pk1(zl)));
  return fma2(fma2(q, pk1(nb), x), pk1(z), q);
}

// Two 512-thread CTAs (64 registers) hold 32 warps per SM, with or without an
// antenna pattern: a pattern's 136 registers in 256-thread CTAs left eight
// (512^2 facets x 1024 traces with a dipole 2.49 -> 1.16 ms, with a table
// 4.16 -> 1.88 ms; three or four 256-thread CTAs per SM 1.25 and 1.31, 1.98
// and 2.14).
constexpr int kIncThreads = 512;

template <int TB, bool PAT>
__global__ void __launch_bounds__(kIncThreads, 2)
incoherent_kernel(IncArgs a) {
  extern __shared__ __align__(16) float hist[];  // (TB, stride)
  __shared__ float4 s_p[TB], s_u[TB];
  __shared__ float s_pv[TB][6];
  __shared__ float s_pat[SS_PAT_MAX];
  __shared__ float s_drop[TB];

  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int t_base = blockIdx.y * TB;
  const int nt = min(TB, a.T - t_base);
  int pa_len = 0, pb_len = 0;
  if (PAT) pattern_lengths(a.pat_kind, a.pat_n, pa_len, pb_len);

  if (tid < TB) {
    // missing traces of a short last block get NaN positions: their pairs
    // fail every comparison, bin nowhere and their dropped sums are unused
    float4 p = make_float4(__int_as_float(0x7fc00000), 0.f, 0.f, 0.f);
    float4 u = make_float4(0.f, 0.f, 0.f, 0.f);
    if (tid < nt) {
      const int t = t_base + tid;
      // positions and u_ct rounded to float32 (incoherent.py:86-87)
      p = make_float4((float)a.pos[3 * t], (float)a.pos[3 * t + 1],
                      (float)a.pos[3 * t + 2], 0.f);
      if (a.uct)
        u = make_float4((float)a.uct[3 * t], (float)a.uct[3 * t + 1],
                        (float)a.uct[3 * t + 2], 0.f);
      for (int j = 0; j < 6; ++j)
        s_pv[tid][j] =
            (PAT && a.pv && j < a.pv_len) ? (float)a.pv[a.pv_len * t + j]
                                          : 0.f;
    }
    s_p[tid] = p;
    s_u[tid] = u;
    s_drop[tid] = 0.f;
  }
  if (PAT) {
    for (int j = tid; j < pa_len; j += blockDim.x) s_pat[j] = (float)a.pa[j];
    for (int j = tid; j < pb_len; j += blockDim.x)
      s_pat[pa_len + j] = (float)a.pb[j];
  }
  for (int j = tid; j < TB * a.stride; j += blockDim.x) hist[j] = 0.f;
  __syncthreads();

  // step s always pairs this thread with trace (lane + s) mod TB: its
  // position, histogram row and dropped sum live in registers, two steps to a
  // packed pair (TB = 1: the second half repeats the first and is not used)
  constexpr int H = (TB + 1) / 2;
  float2 px[H], py[H], pz[H];
  float drop[TB];
  int hoff[TB];
#pragma unroll
  for (int s = 0; s < TB; ++s) {
    const int tt = (lane + s) & (TB - 1);
    const float4 P = s_p[tt];
    if (s & 1) {
      px[s / 2].y = P.x;
      py[s / 2].y = P.y;
      pz[s / 2].y = P.z;
    } else {
      px[s / 2] = pk1(P.x);
      py[s / 2] = pk1(P.y);
      pz[s / 2] = pk1(P.z);
    }
    hoff[s] = tt * a.stride - 0x4B000000;
    drop[s] = 0.f;
  }

  const long len = a.N;
  const int i0 = (int)(len * blockIdx.x / a.n_chunks);
  const int i1 = (int)(len * (blockIdx.x + 1) / a.n_chunks);
  const float nsf = (float)a.n_samples;

  for (int i = i0 + tid; i < i1; i += blockDim.x) {
    const float2 cx = pk1(a.cx[i]), cy = pk1(a.cy[i]), cz = pk1(a.cz[i]);
    const float2 nx = pk1(a.nx[i]), ny = pk1(a.ny[i]), nz = pk1(a.nz[i]);
    const float2 ar = pk1(a.area[i]);
#pragma unroll
    for (int h = 0; h < H; ++h) {
      const float2 dx = sub2(px[h], cx);
      const float2 dy = sub2(py[h], cy);
      const float2 dz = sub2(pz[h], cz);
      // (scalar sums: the compiler fuses a packed sum of packed products)
      const float2 x2 = mul2(dx, dx), yy = mul2(dy, dy), z2 = mul2(dz, dz);
      const float2 S = pk(__fadd_rn(__fadd_rn(x2.x, yy.x), z2.x),
                          __fadd_rn(__fadd_rn(x2.y, yy.y), z2.y));
      const float2 y = pk(rsq_n(S.x), rsq_n(S.y));  // 1/r
      // the reference's bin coordinate
      const float2 g = mul2(S, y), hy = mul2(y, pk1(0.5f));
      const float2 r = fma2(pk(__fmaf_rn(-g.x, g.x, S.x),
                               __fmaf_rn(-g.y, g.y, S.y)), hy, g);
      // power (A cos)^2 / r^4 = (A (d . n))^2 / r^6, 1/r to its rounding
      const float2 q =
          mul2(ar, fma2(dz, nz, fma2(dy, ny, mul2(dx, nx))));
      const float2 yr = fma2(fma2(pk(-r.x, -r.y), y, pk1(1.0f)), y, y);
      const float2 y2 = mul2(yr, yr);
      float2 pw = mul2(mul2(q, q), mul2(mul2(y2, y2), y2));
      const float ex = __fmaf_rn(-r.x, r.x, S.x),
                  ey = __fmaf_rn(-r.y, r.y, S.y);
      // 2^k of the binade just below r: a power of two's lower neighbour is
      // half an ulp away
      const float2 rb = mul2(r, pk1(0.99999994f));
      const float2 k2 = pk(__int_as_float(__float_as_int(rb.x) & 0x7f800000),
                           __int_as_float(__float_as_int(rb.y) & 0x7f800000));
      const float2 lim = mul2(mul2(r, k2), pk1(a.mid));
      const float2 tw = div_const2(r, a.zc, a.zcl, a.nhc);
      float2 u = div_const2(sub2(tw, pk1(a.t0)), a.zd, a.zdl, a.ndt);
      if (fabsf(ex) > lim.x || fabsf(ey) > lim.y) {
        u.x = bin_exact(S.x, a.c, a.t0, a.dt);
        u.y = bin_exact(S.y, a.c, a.t0, a.dt);
      }
#pragma unroll
      for (int j = 0; j < 2 && 2 * h + j < TB; ++j) {
        const int s = 2 * h + j;
        const float us = j ? u.y : u.x;
        float p = j ? pw.y : pw.x;
        const float dxs = j ? dx.y : dx.x, dys = j ? dy.y : dy.x,
                    dzs = j ? dz.y : dz.x, ys = j ? y.y : y.x;
        if (PAT) {
          // departure direction antenna -> facet (incoherent.py:45)
          const int tt = (lane + s) & (TB - 1);
          const float gn = gain32(a.pat_kind, a.pat_n, pa_len, s_pat, s_pv[tt],
                                  -dxs * ys, -dys * ys, -dzs * ys);
          const float g2 = gn * gn;
          p *= g2 * g2;
        }
        if (us >= 0.0f && us < nsf) {
          // floor: 2^23 + u rounded down has it in the low mantissa bits
          int seg = __float_as_int(__fadd_rd(us, 8388608.0f));
          if (a.split) {
            const float4 U = s_u[(lane + s) & (TB - 1)];
            // (c - p) . u_ct, rounded like the reference's sum
            const float sd = __fadd_rn(__fadd_rn(__fmul_rn(-dxs, U.x),
                                                 __fmul_rn(-dys, U.y)),
                                       __fmul_rn(-dzs, U.z));
            if (sd > 0.0f) seg += a.n_samples;
          }
          atomicAdd(&hist[hoff[s] + seg], p);
        } else {
          drop[s] += p;
        }
      }
    }
  }
#pragma unroll
  for (int s = 0; s < TB; ++s) {
    const int tt = (lane + s) & (TB - 1);
    if (tt < nt) atomicAdd(&s_drop[tt], drop[s]);
  }
  __syncthreads();
  for (int tt = 0; tt < nt; ++tt) {
    float *dst = a.part + ((size_t)blockIdx.x * a.T + t_base + tt) * a.n_seg;
    for (int j = tid; j < a.n_seg; j += blockDim.x)
      dst[j] = hist[tt * a.stride + j];
  }
  if (tid < nt)
    a.part_drop[(size_t)blockIdx.x * a.T + t_base + tid] = (double)s_drop[tid];
}

// Chunk sums (compensated float32, ~2^-48 relative), in chunk order, into
// the (T, n[, 2]) float32 layout.
__global__ void incoherent_reduce_kernel(const float *part,
                                         const double *part_drop, int T,
                                         int n_seg, int n_samples, int split,
                                         int n_chunks,
                                         ss_incoherent_output out) {
  const long total = (long)T * n_seg;
  for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < total;
       e += (long)gridDim.x * blockDim.x) {
    const int t = (int)(e / n_seg);
    const int b = (int)(e % n_seg);
    ChunkSum<float> cs;
    for (int c = 0; c < n_chunks; ++c)
      cs.add(part[((size_t)c * T + t) * n_seg + b]);
    const double s = cs.value();
    long o = e;
    if (split) {  // (T, 2, n) -> (T, n, 2) [left, right]
      const int side = b / n_samples, bl = b % n_samples;
      o = ((long)t * n_samples + bl) * 2 + side;
    }
    out.power[o] = (float)s;
    if (b == 0) {
      double d = 0.0;
      for (int c = 0; c < n_chunks; ++c) d += part_drop[(size_t)c * T + t];
      out.dropped[t] = (float)d;
    }
  }
}

namespace {

struct IncPlan {
  int tb, n_groups, n_chunks, stride;
  size_t smem;
};

constexpr size_t kIncSmemBudget = 100 * 1024;  // two CTAs per SM
constexpr size_t kIncSmemMax = 200 * 1024;

int inc_plan(const ss_incoherent_opts *o, int T, int N, IncPlan *p) {
  if (!o || T <= 0 || N <= 0 || o->n_samples <= 0) return SS_ERR_ARG;
  const int n_seg = o->n_samples * (o->split_sides ? 2 : 1);
  p->stride = n_seg | 1;  // odd: traces' equal bins fall in distinct banks
  const size_t row = (size_t)p->stride * sizeof(float);
  int tb = 8;
  while (tb > 1 && tb * row > kIncSmemBudget) tb >>= 1;
  if (tb * row > kIncSmemMax) return SS_ERR_UNSUPPORTED;
  p->tb = tb;
  p->smem = tb * row;
  p->n_groups = (T + tb - 1) / tb;
  // two to four waves of two CTAs per SM, the count that fills its last wave
  // best (a wave half full costs a full one); each chunk at least 2048 facets
  // and enough pairs to amortise zeroing and writing its histograms
  const long slots = 2L * sm_count();
  const long most = std::max(1L, std::min((long)N / 2048,
                                          (long)N * tb / (4L * n_seg)));
  long nc = 1;
  double best = 0.0;
  for (long w = 2; w <= 4; ++w) {
    const long k = std::max(1L, std::min(most, w * slots / p->n_groups));
    const long items = k * p->n_groups;
    const double fill =
        (double)items / (double)((items + slots - 1) / slots * slots);
    if (fill > best + 1e-9) {
      best = fill;
      nc = k;
    }
  }
  p->n_chunks = (int)std::max(1L, nc);
  return SS_OK;
}

template <int TB, bool PAT>
int inc_launch_t(const IncArgs &a, const IncPlan &p, cudaStream_t st) {
  cudaError_t e = cudaFuncSetAttribute(
      incoherent_kernel<TB, PAT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
      (int)p.smem);
  if (e != cudaSuccess) return cuda_status(e, "incoherent smem");
  dim3 grid(p.n_chunks, p.n_groups);
  incoherent_kernel<TB, PAT><<<grid, kIncThreads, p.smem, st>>>(a);
  return cuda_status(cudaGetLastError(), "incoherent launch");
}

template <bool PAT>
int inc_launch_p(const IncArgs &a, const IncPlan &p, cudaStream_t st) {
  switch (p.tb) {
    case 8: return inc_launch_t<8, PAT>(a, p, st);
    case 4: return inc_launch_t<4, PAT>(a, p, st);
    case 2: return inc_launch_t<2, PAT>(a, p, st);
    default: return inc_launch_t<1, PAT>(a, p, st);
  }
}

}  // namespace
}  // namespace ss

using namespace ss;

extern "C" size_t ss_incoherent_scratch_bytes(const ss_incoherent_opts *opts,
                                              int32_t n_traces,
                                              int32_t n_facets) {
  IncPlan p;
  if (inc_plan(opts, n_traces, n_facets, &p) != SS_OK) return 0;
  const size_t n_seg = (size_t)opts->n_samples * (opts->split_sides ? 2 : 1);
  const size_t part = (size_t)p.n_chunks * n_traces * n_seg * sizeof(float);
  const size_t drop = (size_t)p.n_chunks * n_traces * sizeof(double);
  return ((part + 255) & ~(size_t)255) + drop;
}

extern "C" int ss_incoherent_fwd(const ss_incoherent_opts *opts,
                                 const ss_facets *facets,
                                 const ss_traces *traces,
                                 const ss_pattern *pattern,
                                 const ss_incoherent_output *out,
                                 void *scratch, size_t scratch_bytes,
                                 void *stream) {
  if (!opts || !facets || !traces || !out || !out->power || !out->dropped) {
    set_error("ss_incoherent_fwd: null argument");
    return SS_ERR_ARG;
  }
  const int T = traces->n_traces, N = facets->n_facets;
  if (!traces->pos || !facets->cx || !facets->cy || !facets->cz ||
      !facets->nx || !facets->ny || !facets->nz || !facets->area ||
      (opts->split_sides && !traces->uct) || !(opts->dt > 0.0) ||
      !(opts->c > 0.0)) {
    set_error("ss_incoherent_fwd: missing input array or bad window");
    return SS_ERR_ARG;
  }
  IncPlan p;
  int st = inc_plan(opts, T, N, &p);
  if (st != SS_OK) {
    set_error(st == SS_ERR_UNSUPPORTED
                  ? "ss_incoherent_fwd: n_samples beyond shared memory"
                  : "ss_incoherent_fwd: bad sizes");
    return st;
  }
  const size_t need = ss_incoherent_scratch_bytes(opts, T, N);
  if (!scratch || scratch_bytes < need) {
    set_error("ss_incoherent_fwd: scratch too small");
    return SS_ERR_SCRATCH;
  }
  const int kind = pattern ? pattern->kind : SS_PAT_ISOTROPIC;
  if (kind != SS_PAT_ISOTROPIC) {
    int pa_len, pb_len;
    pattern_lengths(kind, pattern->n, pa_len, pb_len);
    if (pa_len + pb_len > SS_PAT_MAX) {
      set_error("ss_incoherent_fwd: antenna table too large");
      return SS_ERR_UNSUPPORTED;
    }
    if (!traces->pv || ((pa_len && !pattern->pa) || (pb_len && !pattern->pb))) {
      set_error("ss_incoherent_fwd: pattern arrays missing");
      return SS_ERR_ARG;
    }
  }
  IncArgs a{};
  a.cx = facets->cx; a.cy = facets->cy; a.cz = facets->cz;
  a.nx = facets->nx; a.ny = facets->ny; a.nz = facets->nz;
  a.area = facets->area;
  a.pos = traces->pos;
  a.uct = traces->uct;
  a.pv = traces->pv;
  a.pv_len = traces->pv_len;
  a.T = T;
  a.N = N;
  a.n_samples = opts->n_samples;
  a.n_seg = opts->n_samples * (opts->split_sides ? 2 : 1);
  a.stride = p.stride;
  a.split = opts->split_sides ? 1 : 0;
  // window scalars rounded to float32 (incoherent.py:101-102)
  a.t0 = (float)opts->t0;
  a.dt = (float)opts->dt;
  a.c = (float)opts->c;
  const float hc = 0.5f * a.c;
  a.nhc = -hc;
  a.ndt = -a.dt;
  const double ic = 1.0 / (double)hc, id = 1.0 / (double)a.dt;
  a.zc = (float)ic;
  a.zcl = (float)(ic - (double)a.zc);
  a.zd = (float)id;
  a.zdl = (float)(id - (double)a.zd);
  // The fast chain's quotients want divisors whose mantissa is not all ones
  // and whose products stay clear of float32's range ends; any other call
  // takes the exact chain throughout.
  const auto plain = [](float b) {
    uint32_t bits;
    std::memcpy(&bits, &b, 4);
    return b > 1e-15f && b < 1e15f && (bits & 0x7fffffu) != 0x7fffffu;
  };
  a.mid = plain(hc) && plain(a.dt)
              ? (float)((1.0 - 1.0 / 16384) / 8388608.0)
              : -1.0f;
  a.pat_kind = kind;
  a.pat_n = pattern ? pattern->n : 0;
  a.pa = pattern ? pattern->pa : nullptr;
  a.pb = pattern ? pattern->pb : nullptr;
  a.n_chunks = p.n_chunks;
  const size_t n_seg = (size_t)a.n_seg;
  const size_t part_bytes = (size_t)p.n_chunks * T * n_seg * sizeof(float);
  a.part = reinterpret_cast<float *>(scratch);
  a.part_drop = reinterpret_cast<double *>(
      reinterpret_cast<char *>(scratch) + ((part_bytes + 255) & ~(size_t)255));
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  st = kind != SS_PAT_ISOTROPIC ? inc_launch_p<true>(a, p, s)
                                : inc_launch_p<false>(a, p, s);
  if (st != SS_OK) return st;
  incoherent_reduce_kernel<<<4 * sm_count(), 256, 0, s>>>(
      a.part, a.part_drop, T, a.n_seg, a.n_samples, a.split, p.n_chunks,
      *out);
  return cuda_status(cudaGetLastError(), "incoherent reduce launch");
}
