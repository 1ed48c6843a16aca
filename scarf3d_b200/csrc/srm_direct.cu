// FP32 direct-sum SRM kernels (the "plain" form): for every point,
//   field = scaling * sum_h [ a_h sin(arg_h) + b_h cos(arg_h) ],
//   arg_h = v1*P1 + v2*P2 + v3*P3,  P = M x + bar,
// evaluated in the reference's operation order without FMA contraction
// (scarflib_srm.f90:794-809 structured, :397-406 points, :843-851 scaling).
// The rotated coordinates P are loop invariant in the reference, so they are
// computed once per point. Every point adds its harmonics in table order, two
// additions each, so that fields follow the reference's FP32 sum closely
// (a reordered FP32 sum of 10 000 harmonics differs by ~2e-6).
#include <cuda_runtime.h>

#include "common.cuh"
#include "srm_kernels.h"

namespace scarf {
namespace {

constexpr int kTile = 128;           // harmonics per shared-memory tile
constexpr int kRow = 5;              // floats per table row {v1,v2,v3,a,b}
constexpr int kThreads = 128;
constexpr int kPts = 2;              // points per thread
// Ordered-terms form: points per block (one per lane), warps that evaluate
// terms, harmonics per batch.
constexpr int kOrdWarps = 8;
constexpr int kOrdHarm = 64;

struct DirectArgs {
  float m[9];
  float bar[3];
  float scaling;
  float negative_zero;  // see mul2
  int nh;
  const float* table;  // device, nh x 5
  float* field;
  long long npts;
  // structured
  int n0, n1;
  float ds;
  int off0, off1, off2;  // fs - 2 (so x = (i1 + off) * ds with 1-based i1)
  // points
  const float* x;
  const float* y;
  const float* z;
  // optional: one statistics record per block (count, mean, M2 of its stored values)
  Moments* stats;
};

__device__ __forceinline__ void rotate(const DirectArgs& A, float x, float y, float z, float& p1, float& p2,
                                       float& p3) {
  // ((m1 x + m2 y) + m3 z) + bar, each operation rounded (no contraction).
  p1 = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(A.m[0], x), __fmul_rn(A.m[1], y)), __fmul_rn(A.m[2], z)), A.bar[0]);
  p2 = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(A.m[3], x), __fmul_rn(A.m[4], y)), __fmul_rn(A.m[5], z)), A.bar[1]);
  p3 = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(A.m[6], x), __fmul_rn(A.m[7], y)), __fmul_rn(A.m[8], z)), A.bar[2]);
}

// sin and cos of an FP32 phase, two ways.
// Accurate (kFast = false): CUDA's sincosf, correctly rounded to ~1 ulp with
// full range reduction. Fast (default): the phase reduced to [-pi, pi] by
// Cody-Waite's method (Cody & Waite, "Software Manual for the Elementary
// Functions", 1980) with 2 pi split into two floats C1 + C2 (the residual,
// 6.9e-15, times |j| < 2^22 stays below 3e-8), each product applied by one
// FMA, then the SFU's __sinf/__cosf, whose absolute error on [-pi, pi] is
// about 2^-21.4. C1 has 24 significant bits, so arg - j C1 is exact (a
// multiple of 2^-21 below 2^2 in magnitude, or Sterbenz's case for |j| = 1);
// only the C2 step rounds. For the
// phases here (|arg| < 1e4 rad) the reduced argument is within ~2.5e-7 of
// exact, so each term is within ~6e-7 absolute, and fields agree with the
// FP32 restatement (glibc sinf/cosf) to ~4e-7 of their standard deviation.
// (Phases up to 2^22 * 2 pi = 2.6e7 rad; the FP32 phase itself carries an
// error of several radians long before that.)
constexpr float kInv2Pi = 0x1.45f306p-3f;
constexpr float kTwoPi1 = 0x1.921fb6p+2f;
constexpr float kTwoPi2 = -0x1.777a5cp-23f;

// Nearest integer of arg / (2 pi) for |arg / (2 pi)| < 2^22 on the FMA pipe:
// one FMA adds 1.5 * 2^23 to the exact product (rounding it to an integer,
// nearest even) and a subtraction removes it. rintf itself would issue on
// the SFU's pipe, which __sinf and __cosf already saturate here. Near a
// half-integer either neighbour may be chosen; both leave |r| <= pi + 3e-7.
constexpr float kRoundMagic = 0x1.8p23f;

template <bool kFast>
__device__ __forceinline__ void phase_sincos(float arg, float* sn, float* cs) {
  if constexpr (kFast) {
    const float j = __fsub_rn(__fmaf_rn(arg, kInv2Pi, kRoundMagic), kRoundMagic);
    float r = fmaf(-j, kTwoPi1, arg);
    r = fmaf(-j, kTwoPi2, r);
    *sn = __sinf(r);
    *cs = __cosf(r);
  } else {
    sincosf(arg, sn, cs);
  }
}

// A pair of FP32 values in one 64-bit register, and the packed operations of
// sm_100 on it: each half is rounded as the scalar operation would be, at
// half the issue slots.
using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

// Rounded products. ptxas contracts mul.rn.f32x2 and a following
// add.rn.f32x2 into one fused operation (measured: a quarter of the sums of
// two products came out with the contraction's rounding), so products are
// written as fused operations that add -0.0, which leaves every product as it
// rounds; the -0.0 comes from the kernel's arguments, out of the compiler's
// sight.
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b, f32x2 negative_zero) { return fma2(a, b, negative_zero); }

// phase_sincos of two phases.
template <bool kFast>
__device__ __forceinline__ void phase_sincos2(f32x2 arg, f32x2* sn, f32x2* cs) {
  float s0, s1, c0, c1, r0, r1;
  if constexpr (kFast) {
    const f32x2 q = fma2(arg, pack2(kInv2Pi, kInv2Pi), pack2(kRoundMagic, kRoundMagic));
    const f32x2 j = add2(q, pack2(-kRoundMagic, -kRoundMagic));
    f32x2 r = fma2(j, pack2(-kTwoPi1, -kTwoPi1), arg);
    r = fma2(j, pack2(-kTwoPi2, -kTwoPi2), r);
    unpack2(r, r0, r1);
    s0 = __sinf(r0);
    c0 = __cosf(r0);
    s1 = __sinf(r1);
    c1 = __cosf(r1);
  } else {
    unpack2(arg, r0, r1);
    sincosf(r0, &s0, &c0);
    sincosf(r1, &s1, &c1);
  }
  *sn = pack2(s0, s1);
  *cs = pack2(c0, c1);
}

// Coordinates of point p (clamped to the set), rotated.
template <bool kStructured>
__device__ __forceinline__ void point_coords(const DirectArgs& A, long long p, float& p1, float& p2, float& p3) {
  if (p >= A.npts) p = A.npts - 1;
  float x, y, z;
  if constexpr (kStructured) {
    const long long plane = static_cast<long long>(A.n0) * A.n1;
    const int k = static_cast<int>(p / plane);
    const long long rem = p - static_cast<long long>(k) * plane;
    const int j = static_cast<int>(rem / A.n0);
    const int i = static_cast<int>(rem - static_cast<long long>(j) * A.n0);
    // x = (i + fs(1) - 2) * ds with the 1-based index i+1.
    x = __fmul_rn(static_cast<float>(i + 1 + A.off0), A.ds);
    y = __fmul_rn(static_cast<float>(j + 1 + A.off1), A.ds);
    z = __fmul_rn(static_cast<float>(k + 1 + A.off2), A.ds);
  } else {
    x = __ldg(A.x + p);
    y = __ldg(A.y + p);
    z = __ldg(A.z + p);
  }
  rotate(A, x, y, z, p1, p2, p3);
}

// Two points per thread, in the halves of packed registers. The harmonic rows
// are double-buffered in shared memory with every value stored twice, so that
// a 16-byte load yields packed operands without moves; the next tile's rows
// are loaded into registers while the current tile is summed.
// Bound: the XU pipe, two MUFU operations per point and harmonic (8 pairs per
// clock and SM, 2.33e12/s at 1.965 GHz). Scalar operations (17 issue slots per
// pair and warp against 16 XU cycles) at eight points per thread reached
// 1.61e12 at 2e6 points x 4 000 harmonics and 0.72e12 at 150 001 points, where
// one 4-warp block sat on each SM. Packed, the pair takes 10 slots, and two
// points per thread give four times the warps: 2.09e12 and 1.61e12; four
// points per thread 2.06e12 and 1.46e12.
// Each point adds its harmonics one after another in table order: a field
// does not depend on how its points are spread over threads.
template <bool kStructured, bool kFast>
__global__ void __launch_bounds__(kThreads) srm_direct_kernel(const DirectArgs A) {
  __shared__ __align__(16) f32x2 s_tab[2][kTile * kRow];
  const int tid = threadIdx.x;
  const long long p0 = (static_cast<long long>(blockIdx.x) * kThreads + tid) * kPts;

  float c0[3], c1[3];
  point_coords<kStructured>(A, p0, c0[0], c0[1], c0[2]);
  point_coords<kStructured>(A, p0 + 1, c1[0], c1[1], c1[2]);
  const f32x2 P1 = pack2(c0[0], c1[0]), P2 = pack2(c0[1], c1[1]), P3 = pack2(c0[2], c1[2]);
  f32x2 acc = pack2(0.0f, 0.0f);

  const f32x2 nz = pack2(A.negative_zero, A.negative_zero);
  const int ntiles = (A.nh + kTile - 1) / kTile;
  static_assert(kTile == kThreads, "one table row per thread and tile");
  float row[kRow];  // this thread's row of the tile being fetched
  auto fetch = [&](int t) {
    const int h = t * kTile + tid;
    if (h < A.nh) {
#pragma unroll
      for (int e = 0; e < kRow; ++e) row[e] = __ldg(A.table + static_cast<size_t>(h) * kRow + e);
    }
  };
  auto put = [&](int buf) {
#pragma unroll
    for (int e = 0; e < kRow; ++e) s_tab[buf][tid * kRow + e] = pack2(row[e], row[e]);
  };
  auto harmonic = [&](f32x2 v1, f32x2 v2, f32x2 v3, f32x2 a, f32x2 b) {
    const f32x2 arg = add2(add2(mul2(v1, P1, nz), mul2(v2, P2, nz)), mul2(v3, P3, nz));
    f32x2 sn, cs;
    phase_sincos2<kFast>(arg, &sn, &cs);
    acc = add2(add2(acc, mul2(a, sn, nz)), mul2(b, cs, nz));
  };
  fetch(0);
  put(0);
  __syncthreads();
  for (int t = 0; t < ntiles; ++t) {
    if (t + 1 < ntiles) fetch(t + 1);
    const f32x2* tb = s_tab[t & 1];
    const int rows = min(kTile, A.nh - t * kTile);
    // Two rows (ten packed values, 80 bytes) per step.
    int h = 0;
    for (; h + 2 <= rows; h += 2) {
      const ulonglong2* g = reinterpret_cast<const ulonglong2*>(tb + h * kRow);
      const ulonglong2 q0 = g[0], q1 = g[1], q2 = g[2], q3 = g[3], q4 = g[4];
      harmonic(q0.x, q0.y, q1.x, q1.y, q2.x);
      harmonic(q2.y, q3.x, q3.y, q4.x, q4.y);
    }
    if (h < rows) harmonic(tb[h * kRow], tb[h * kRow + 1], tb[h * kRow + 2], tb[h * kRow + 3], tb[h * kRow + 4]);
    // Tile t + 1 goes into the buffer that tile t - 1 left: every thread is
    // past tile t - 1 since the barrier that opened tile t.
    if (t + 1 < ntiles) put((t + 1) & 1);
    __syncthreads();
  }

  // Normalise (field * scaling) and store.
  float out[kPts];
  unpack2(acc, out[0], out[1]);
  out[0] = __fmul_rn(out[0], A.scaling);
  out[1] = __fmul_rn(out[1], A.scaling);
  float* dst = A.field + p0;
  if (p0 + 1 < A.npts && (reinterpret_cast<uintptr_t>(dst) & 7u) == 0)
    *reinterpret_cast<float2*>(dst) = make_float2(out[0], out[1]);
  else
    for (int q = 0; q < kPts; ++q)
      if (p0 + q < A.npts) dst[q] = out[q];
  if (A.stats) {
    // Statistics of the stored values (FP64): thread, warp (fixed tree), then
    // the block's warps in order; one record per block.
    __shared__ Moments s_warp[kThreads / 32];
    double s1 = 0.0, s2 = 0.0, cnt = 0.0;
    const double shift = p0 < A.npts ? static_cast<double>(out[0]) : 0.0;
#pragma unroll
    for (int q = 0; q < kPts; ++q) {
      if (p0 + q < A.npts) {
        const double d = static_cast<double>(out[q]) - shift;
        s1 += d;
        s2 = fma(d, d, s2);
        cnt += 1.0;
      }
    }
    Moments m = warp_moments(moments_from_shifted(cnt, shift, s1, s2));
    if ((tid & 31) == 0) s_warp[tid >> 5] = m;
    __syncthreads();
    if (tid == 0) {
      Moments b = s_warp[0];
      for (int w = 1; w < kThreads / 32; ++w) b = moments_merge(b, s_warp[w]);
      A.stats[blockIdx.x] = b;
    }
  }
}

// Few points: 32 per block (one per lane). kOrdWarps warps evaluate the terms
// a sin(arg), b cos(arg) of a batch of harmonics into shared memory while one
// more warp adds the previous batch's terms in table order, two dependent
// additions per harmonic, which is all that has to be serial: the field is
// that of srm_direct_kernel bit for bit, with nine warps per 32 points.
// Bound: those additions and a barrier per 64 harmonics. 5 003 points x 4 000
// harmonics: 74 us (with eight points per thread, five blocks of four warps:
// 826 us).
template <bool kStructured, bool kFast>
__global__ void __launch_bounds__(32 * (kOrdWarps + 1)) srm_direct_ordered_kernel(const DirectArgs A) {
  __shared__ float2 s_term[2][kOrdHarm][32];
  __shared__ float s_row[2][kOrdHarm * kRow];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long p = static_cast<long long>(blockIdx.x) * 32 + lane;
  float P1, P2, P3;
  point_coords<kStructured>(A, p, P1, P2, P3);
  float acc = 0.0f;
  const int nbatch = (A.nh + kOrdHarm - 1) / kOrdHarm;
  constexpr int kEach = kOrdHarm / kOrdWarps;
  // The rows of batch b, two table values per evaluating thread (zeros past
  // the table: their terms are never added).
  constexpr int kEval = 32 * kOrdWarps;
  static_assert(kOrdHarm * kRow <= 2 * kEval, "two table values per thread");
  const long long total = static_cast<long long>(A.nh) * kRow;
  auto value = [&](int b, int e) {
    const long long at = static_cast<long long>(b) * kOrdHarm * kRow + e;
    return e < kOrdHarm * kRow && at < total ? __ldg(A.table + at) : 0.0f;
  };
  const int e0 = threadIdx.x, e1 = threadIdx.x + kEval;
  if (warp < kOrdWarps) {
    s_row[0][e0] = value(0, e0);
    if (e1 < kOrdHarm * kRow) s_row[0][e1] = value(0, e1);
  }
  __syncthreads();
  for (int b = 0; b <= nbatch; ++b) {
    if (warp < kOrdWarps) {
      if (b < nbatch) {
        const float n0 = value(b + 1, e0), n1 = value(b + 1, e1);
        const float* rows = &s_row[b & 1][warp * kEach * kRow];
        float2(*dst)[32] = &s_term[b & 1][warp * kEach];
#pragma unroll
        for (int u = 0; u < kEach; ++u) {
          const float* r = rows + u * kRow;
          const float arg = __fadd_rn(__fadd_rn(__fmul_rn(r[0], P1), __fmul_rn(r[1], P2)), __fmul_rn(r[2], P3));
          float sn, cs;
          phase_sincos<kFast>(arg, &sn, &cs);
          dst[u][lane] = make_float2(__fmul_rn(r[3], sn), __fmul_rn(r[4], cs));
        }
        s_row[(b + 1) & 1][e0] = n0;
        if (e1 < kOrdHarm * kRow) s_row[(b + 1) & 1][e1] = n1;
      }
    } else if (b > 0) {
      const int n = min(kOrdHarm, A.nh - (b - 1) * kOrdHarm);
      const float2(*src)[32] = s_term[(b - 1) & 1];
      if (n == kOrdHarm) {
        // Eight terms ahead of the additions.
        float2 t[2][8];
#pragma unroll
        for (int u = 0; u < 8; ++u) t[0][u] = src[u][lane];
#pragma unroll
        for (int c = 0; c < kOrdHarm / 8; ++c) {
          if (c + 1 < kOrdHarm / 8) {
#pragma unroll
            for (int u = 0; u < 8; ++u) t[(c + 1) & 1][u] = src[8 * (c + 1) + u][lane];
          }
#pragma unroll
          for (int u = 0; u < 8; ++u) acc = __fadd_rn(__fadd_rn(acc, t[c & 1][u].x), t[c & 1][u].y);
        }
      } else {
        for (int h = 0; h < n; ++h) acc = __fadd_rn(__fadd_rn(acc, src[h][lane].x), src[h][lane].y);
      }
    }
    __syncthreads();
  }
  if (warp == kOrdWarps) {
    const float out = __fmul_rn(acc, A.scaling);
    const bool in = p < A.npts;
    if (in) A.field[p] = out;
    if (A.stats) {
      const Moments m = warp_moments(Moments{in ? 1.0 : 0.0, in ? static_cast<double>(out) : 0.0, 0.0});
      if (lane == 0) A.stats[blockIdx.x] = m;
    }
  }
}

// The ordered-terms form up to this many points. Measured with 4 000
// harmonics, ordered against two points per thread: SFU sin/cos 74 vs 181 us
// at 5 003 points, 191 vs 225 at 40 000, 327 vs 303 at 80 000; CUDA's sincosf
// 109 vs 455 us, 315 vs 554 and 549 vs 658 there, 991 vs 807 at 150 001.
constexpr long long kOrderedMaxFast = 60000, kOrderedMaxAccurate = 100000;

bool use_ordered(long long npts, bool fast) { return npts <= (fast ? kOrderedMaxFast : kOrderedMaxAccurate); }
// Blocks of a launch; also its statistics records.
long long direct_blocks(long long npts, bool fast) {
  const long long per_block = use_ordered(npts, fast) ? 32 : kThreads * kPts;
  return (npts + per_block - 1) / per_block;
}

template <bool kStructured>
cudaError_t launch_direct(const DirectArgs& A, bool fast, cudaStream_t stream) {
  const long long nb = direct_blocks(A.npts, fast);
  if (nb <= 0) return cudaSuccess;
  const unsigned blocks = static_cast<unsigned>(nb);
  if (use_ordered(A.npts, fast)) {
    if (fast)
      srm_direct_ordered_kernel<kStructured, true><<<blocks, 32 * (kOrdWarps + 1), 0, stream>>>(A);
    else
      srm_direct_ordered_kernel<kStructured, false><<<blocks, 32 * (kOrdWarps + 1), 0, stream>>>(A);
  } else if (fast) {
    srm_direct_kernel<kStructured, true><<<blocks, kThreads, 0, stream>>>(A);
  } else {
    srm_direct_kernel<kStructured, false><<<blocks, kThreads, 0, stream>>>(A);
  }
  return cudaGetLastError();
}

}  // namespace

int g_direct_fast = 1;

void direct_set_sincos(int fast) { g_direct_fast = fast ? 1 : 0; }
int direct_get_sincos() { return g_direct_fast; }

long long direct_stat_records(long long npts) { return direct_blocks(npts, g_direct_fast != 0); }

cudaError_t launch_direct_structured(const scarf_srm_setup& s, const int fs[3], const int n[3], float ds,
                                     const float* d_table, int nh, float* d_field,
                                     cudaStream_t stream, StatRecord* d_stats) {
  DirectArgs A{};
  for (int i = 0; i < 9; ++i) A.m[i] = s.m[i];
  for (int i = 0; i < 3; ++i) A.bar[i] = s.bar[i];
  A.scaling = s.scaling;
  A.negative_zero = -0.0f;
  A.nh = nh;
  A.table = d_table;
  A.field = d_field;
  A.npts = static_cast<long long>(n[0]) * n[1] * n[2];
  A.n0 = n[0];
  A.n1 = n[1];
  A.ds = ds;
  A.off0 = fs[0] - 2;
  A.off1 = fs[1] - 2;
  A.off2 = fs[2] - 2;
  A.stats = d_stats;
  return launch_direct<true>(A, g_direct_fast != 0, stream);
}

cudaError_t launch_direct_points(const scarf_srm_setup& s, const float* d_x, const float* d_y, const float* d_z,
                                 long long npts, const float* d_table, int nh, float* d_field,
                                 cudaStream_t stream, StatRecord* d_stats) {
  DirectArgs A{};
  for (int i = 0; i < 9; ++i) A.m[i] = s.m[i];
  for (int i = 0; i < 3; ++i) A.bar[i] = s.bar[i];
  A.scaling = s.scaling;
  A.negative_zero = -0.0f;
  A.nh = nh;
  A.table = d_table;
  A.field = d_field;
  A.npts = npts;
  A.x = d_x;
  A.y = d_y;
  A.z = d_z;
  A.stats = d_stats;
  return launch_direct<false>(A, g_direct_fast != 0, stream);
}

}  // namespace scarf
