// Inverse transform of the FIM's half spectrum (scarflib_fim.f90:1705-2315): c2c
// along z and y (FFTW_BACKWARD, unnormalised), then c2r along x, each axis in
// one pass over memory.
//
// The grid rule gives axis lengths such as 514 = 2 x 257, for which a general
// transform takes Bluestein's form: with c_n = e^{pi i n^2 / N},
//   X_k = c_k sum_n (x_n c_n) conj(c_{k - n}),
// a cyclic convolution of length M >= 2 N - 1 (Bluestein 1970), here with M
// having no prime factor above 5. A tile of eight transforms sits in shared
// memory (fft_tile.cuh): decimation in frequency forwards, whose output order
// the product with the transformed chirp and the decimation in time backwards
// take as it is; the last stage forwards, the product and the first stage
// backwards are one step in registers. Lengths without larger prime factors take
// a plain transform.
//
// Bound: shared-memory traffic of the stages (1 080 points take eight passes
// over a 69 KB tile). 514^3: cuFFT's transforms took 4.2 ms (z 1.51, y 1.42, x
// 1.26 with its preprocessing) and the statistics 0.11 more; these take 3.2.
//
// The c2r step stores the scaled field (1 / sqrt(n1 n2 n3 dh^n), :1019) and
// records its statistics (:1027-1036), one record per block, as it goes.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "common.cuh"
#include "fft_tile.cuh"
#include "srm_kernels.h"

namespace scarf {
namespace {

using namespace fft;

constexpr int kPairs = 4;               // transform pairs of a tile
constexpr int kTile = 2 * kPairs;       // transforms of a tile
// Blocks of at most 256 threads at 80 registers: three per SM at ~1 100 points.
// With 112 registers (two) the transforms of the 514^3 grid took 3.9 ms, with 64
// (spilling) 3.6, so 3.2.
constexpr int kMaxThreads = 256, kSmThreads = 3 * kMaxThreads;
constexpr size_t kSmemMax = 224 * 1024;

// Device tables of one axis: twiddles of its plan, then (Bluestein) the chirp
// and the transformed chirp in the forward transform's output order, or
// (plain) the output order of the last stage's butterflies; for the real axis
// the roots of its packing.
struct AxisTables {
  const float4* tw;     // {cos, cos, sin, sin}
  const float4* chirp;  // n entries, the same form
  const float4* hat;    // f.n entries
  const int* rev;       // at e - t of the last stage
  const float4* pack;   // e^{2 pi i k / n1}, k <= n1 / 4 (real axis)
};

struct TableArgs {
  FimAxis ax[3];
  float4* tw[3];
  float4* chirp[3];
  float4* hat[3];
  int* rev[3];
  float4* pack;
  int n1;
};

__device__ __forceinline__ float4 dup_root(double turns) {
  double s, c;
  sincospi(2.0 * (turns - rint(turns)), &s, &c);
  return make_float4(static_cast<float>(c), static_cast<float>(c), static_cast<float>(s), static_cast<float>(s));
}
// n^2 / (2 N) modulo 1, exactly reduced
__device__ __forceinline__ double chirp_turns(int n, int N) {
  const long long q = static_cast<long long>(n) * n % (2ll * N);
  return static_cast<double>(q) / (2.0 * N);
}

// blockIdx.y: axis; one warp per table index.
__global__ void __launch_bounds__(128) fim_tables_kernel(const TableArgs A) {
  const int a = blockIdx.y, lane = threadIdx.x & 31;
  const int i = blockIdx.x * 4 + (threadIdx.x >> 5);
  const FimAxis& X = A.ax[a];
  if (X.n == 0) return;  // axis not transformed
  const FftPlan& f = X.f;
  if (lane == 0) {
    if (i < f.n) A.tw[a][i] = dup_root(twiddle_entry(f, i));
    if (X.blue && i < X.n) A.chirp[a][i] = dup_root(chirp_turns(i, X.n));
    const int r = f.r[f.nst - 1];
    if (!X.blue && i < f.n / r) A.rev[a][i * r] = output_order(f, i);
    if (a == 0 && i <= X.n / 2) A.pack[i] = dup_root(static_cast<double>(i) / A.n1);
  }
  if (!X.blue || i >= f.n) return;
  // hat[pos] = (1 / M) sum_m conj(c_m) e^{2 pi i m freq / M}, m = -(N-1) .. N-1
  const int r = f.r[f.nst - 1], g = i / r, t = i - g * r;
  const int freq = output_order(f, g) + t * (f.n / r);
  double re = 0.0, im = 0.0;
  for (int m = lane; m < X.n; m += 32) {
    double cs, cc, ws, wc;
    const double ct = chirp_turns(m, X.n);
    sincospi(2.0 * ct, &cs, &cc);
    const long long q = static_cast<long long>(m) * freq % f.n;
    sincospi(2.0 * static_cast<double>(q) / f.n, &ws, &wc);
    // b_m (w^m + w^-m) = 2 cos(.) conj(c_m); m = 0 once
    const double k = m == 0 ? 1.0 : 2.0 * wc;
    re += k * cc;
    im -= k * cs;
  }
  for (int o = 16; o > 0; o >>= 1) {
    re += __shfl_down_sync(0xffffffffu, re, o);
    im += __shfl_down_sync(0xffffffffu, im, o);
  }
  if (lane == 0) {
    const float x = static_cast<float>(re / f.n), y = static_cast<float>(im / f.n);
    A.hat[a][i] = make_float4(x, x, y, y);
  }
}

__device__ __forceinline__ C2 load2(const float4* t) {
  const ulonglong2 v = __ldg(reinterpret_cast<const ulonglong2*>(t));
  return C2{v.x, v.y};
}
__device__ __forceinline__ C2 times(C2 a, const float4* t) {
  const C2 w = load2(t);
  return cmul(a, w.re, w.im);
}

// The tile's transforms. in(e, p) gives input e < X.n of pair p, out(e, p, v)
// takes output e < X.n.
template <class In, class Out>
__device__ __forceinline__ void transform_tile(const FimAxis& X, const AxisTables& T, ulonglong2* sh, In in, Out out) {
  const FftPlan& f = X.f;
  auto sin = [&](int e, int p) {
    const ulonglong2 v = sh[e * kPairs + p];
    return C2{v.x, v.y};
  };
  auto sout = [&](int e, int p, int, C2 v) { sh[e * kPairs + p] = make_ulonglong2(v.re, v.im); };
  const int last = f.nst - 1, rl = f.r[last], hop = f.n / rl;
  if (!X.blue) {
    stage_any<kPairs>(f, 0, T.tw, in, sout);
    for (int s = 1; s < last; ++s) {
      __syncthreads();
      stage_any<kPairs>(f, s, T.tw, sin, sout);
    }
    __syncthreads();
    stage_any<kPairs>(f, last, T.tw, sin,
                      [&](int e, int p, int t, C2 v) { out(__ldg(T.rev + e - t) + t * hop, p, v); });
    return;
  }
  auto bin = [&](int e, int p) {
    if (e >= X.n) return C2{0ull, 0ull};
    return times(in(e, p), T.chirp + e);
  };
  stage_any<kPairs>(f, 0, T.tw, bin, sout);
  for (int s = 1; s < last; ++s) {
    __syncthreads();
    stage_any<kPairs>(f, s, T.tw, sin, sout);
  }
  __syncthreads();
  product_any<kPairs>(f, T.hat, sin, sout);
  for (int s = last - 1; s > 0; --s) {
    __syncthreads();
    back_any<kPairs>(f, s, T.tw, sin, sout);
  }
  __syncthreads();
  back_any<kPairs>(f, 0, T.tw, sin, [&](int e, int p, int, C2 v) {
    if (e < X.n) out(e, p, times(v, T.chirp + e));
  });
}

// c2c along z or y, in place: blockIdx.x selects eight neighbouring x bins,
// blockIdx.y the row or plane.
__global__ void __launch_bounds__(kMaxThreads, kSmThreads / kMaxThreads) fim_columns_kernel(const FimAxis X, const AxisTables T, float2* spec, int n1h,
                                                                  long long step, long long outer) {
  extern __shared__ __align__(128) unsigned char smem[];
  const int i0 = blockIdx.x * kTile, left = n1h - i0;
  float2* base = spec + blockIdx.y * outer + i0;
  const bool wide = (reinterpret_cast<uintptr_t>(base) & 15u) == 0 && (step & 1) == 0;
  transform_tile(
      X, T, reinterpret_cast<ulonglong2*>(smem),
      [&](int e, int p) {
        const float2* s = base + e * step + 2 * p;
        float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (wide && 2 * p + 1 < left) {
          v = *reinterpret_cast<const float4*>(s);
        } else {
          if (2 * p < left) v.x = s[0].x, v.y = s[0].y;
          if (2 * p + 1 < left) v.z = s[1].x, v.w = s[1].y;
        }
        return C2{pack(v.x, v.z), pack(v.y, v.w)};
      },
      [&](int e, int p, C2 v) {
        float2* d = base + e * step + 2 * p;
        if (wide && 2 * p + 1 < left) {
          *reinterpret_cast<float4*>(d) = make_float4(lo(v.re), lo(v.im), hi(v.re), hi(v.im));
        } else {
          if (2 * p < left) d[0] = make_float2(lo(v.re), lo(v.im));
          if (2 * p + 1 < left) d[1] = make_float2(hi(v.re), hi(v.im));
        }
      });
}

// c2r along x: eight rows per tile, the n1 / 2 + 1 bins of each packed into a
// complex transform of length n1 / 2 (only real parts of bins 0 and n1 / 2).
__global__ void __launch_bounds__(kMaxThreads, kSmThreads / kMaxThreads) fim_rows_kernel(const FimAxis X, const AxisTables T, const float2* spec,
                                                               float* real, long long rows, float scaling, Moments* rec) {
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ Moments s_warp[kMaxThreads / 32];
  const int n = X.n, half = n / 2;
  const long long r0 = static_cast<long long>(blockIdx.x) * kTile;
  const int left = static_cast<int>(rows - r0 < kTile ? rows - r0 : kTile);
  const float2* src = spec + r0 * (n + 1);
  float* dst = real + r0 * (2 * n);
  ulonglong2* sh = reinterpret_cast<ulonglong2*>(smem);
  auto bin = [&](int k, int p) {
    float2 a = make_float2(0.0f, 0.0f), b = a;
    if (2 * p < left) a = __ldg(src + static_cast<long long>(2 * p) * (n + 1) + k);
    if (2 * p + 1 < left) b = __ldg(src + static_cast<long long>(2 * p + 1) * (n + 1) + k);
    return C2{pack(a.x, b.x), pack(a.y, b.y)};
  };
  for (int it = threadIdx.x; it < (half + 1) * kPairs; it += blockDim.x) {
    const int p = it & (kPairs - 1), k = it / kPairs;
    const C2 a = bin(k, p), b = bin(n - k, p);
    if (k == 0) {
      sh[p] = make_ulonglong2(add(a.re, b.re), sub(a.re, b.re));
    } else {
      // Bins 0 < k < n count twice (Hermitian): (A_k + conj A_{n-k}) +
      // i e^{2 pi i k / n1} (A_k - conj A_{n-k}).
      const C2 s = C2{add(a.re, b.re), sub(a.im, b.im)};
      const C2 u = times(C2{sub(a.re, b.re), add(a.im, b.im)}, T.pack + k);
      const C2 z = add_i(s, u);
      sh[k * kPairs + p] = make_ulonglong2(z.re, z.im);
      if (2 * k != n) sh[(n - k) * kPairs + p] = make_ulonglong2(add(s.re, u.im), sub(u.re, s.im));
    }
  }
  __syncthreads();
  double s1[2] = {0.0, 0.0}, s2[2] = {0.0, 0.0}, shift = 0.0;
  int count = 0;
  auto put = [&](int row, int e, float x, float y) {
    x = __fmul_rn(x, scaling);
    y = __fmul_rn(y, scaling);
    *reinterpret_cast<float2*>(dst + static_cast<long long>(row) * (2 * n) + 2 * e) = make_float2(x, y);
    if (count == 0) shift = x;
    const double d = static_cast<double>(x) - shift, g = static_cast<double>(y) - shift;
    s1[0] += d;
    s2[0] = ::fma(d, d, s2[0]);
    s1[1] += g;
    s2[1] = ::fma(g, g, s2[1]);
    count += 2;
  };
  transform_tile(
      X, T, sh,
      [&](int e, int p) {
        const ulonglong2 v = sh[e * kPairs + p];
        return C2{v.x, v.y};
      },
      [&](int e, int p, C2 v) {
        if (2 * p < left) put(2 * p, e, lo(v.re), lo(v.im));
        if (2 * p + 1 < left) put(2 * p + 1, e, hi(v.re), hi(v.im));
      });
  const Moments m = warp_moments(moments_from_shifted(count, shift, s1[0] + s1[1], s2[0] + s2[1]));
  if ((threadIdx.x & 31) == 0) s_warp[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    Moments b = s_warp[0];
    for (int w = 1; w < static_cast<int>(blockDim.x >> 5); ++w) b = moments_merge(b, s_warp[w]);
    rec[blockIdx.x] = b;
  }
}

// ------------------------------------------------------------------- plans --
bool make_axis(int n, FimAxis* X) {
  X->n = n;
  X->blue = 0;
  if (fft_plan(n, &X->f)) return sizeof(float2) * kTile * static_cast<size_t>(n) <= kSmemMax;
  X->blue = 1;
  const int lo = std::max(4, 2 * n - 1);
  double best = 0.0;
  int found = 0;
  for (int m = lo; m <= lo + lo / 4 + 16; ++m) {
    FftPlan f;
    if (!fft_plan(m, &f)) continue;
    const double cost = static_cast<double>(m) * (f.nst + 2);
    if (!found || cost < best) {
      found = m;
      best = cost;
      X->f = f;
    }
  }
  return found && sizeof(float2) * kTile * static_cast<size_t>(found) <= kSmemMax;
}

size_t axis_smem(const FimAxis& X) { return sizeof(float2) * kTile * static_cast<size_t>(X.f.n); }

// The block size that fills an SM (kSmThreads) with the least idle threads.
int axis_threads(const FimAxis& X) {
  int best = 128;
  double best_cost = 1e30;
  for (int t = 64; t <= kMaxThreads; t += 32) {
    const int blocks = static_cast<int>(std::min<size_t>(std::min<size_t>(kSmemMax / axis_smem(X), kSmThreads / t), 16));
    if (blocks < 1) continue;
    double work = 0.0;
    for (int s = 0; s < X.f.nst; ++s) {
      const int items = X.f.n / X.f.r[s] * kPairs;
      work += static_cast<double>((items + t - 1) / t) * t / items;
    }
    const double cost = work / (blocks * t);
    if (cost < best_cost) best_cost = cost, best = t;
  }
  return best;
}

size_t table_bytes(const FimAxis& X) {
  return sizeof(float4) * (2 * static_cast<size_t>(X.f.n) + 2 * static_cast<size_t>(X.n) + 2) + sizeof(int) * static_cast<size_t>(X.f.n);
}

cudaError_t ensure_attributes() {
  static bool done[64] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev >= 0 && dev < 64 && done[dev]) return cudaSuccess;
  const int most = static_cast<int>(kSmemMax);
  e = cudaFuncSetAttribute(fim_columns_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(fim_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
  if (e == cudaSuccess && dev >= 0 && dev < 64) done[dev] = true;
  return e;
}

}  // namespace

bool fim_fft_plan(const int npts[3], bool three, FimFft* P) {
  *P = FimFft{};
  if (npts[0] < 2 || npts[0] % 2 != 0) return false;
  for (int d = 0; d < 3; ++d) P->n[d] = npts[d];
  if (!make_axis(npts[0] / 2, &P->ax[0])) return false;
  if (npts[1] > 1 && !make_axis(npts[1], &P->ax[1])) return false;
  if (three && npts[2] > 1 && !make_axis(npts[2], &P->ax[2])) return false;
  for (int d = 1; d < 3; ++d)
    if (npts[d] > 65535) return false;
  P->tables = 0;
  for (int d = 0; d < 3; ++d)
    if (P->ax[d].n) P->tables += (table_bytes(P->ax[d]) + 255) / 256 * 256;
  return true;
}

long long fim_fft_records(const FimFft& P) {
  return (static_cast<long long>(P.n[1]) * P.n[2] + kTile - 1) / kTile;
}

cudaError_t launch_fim_fft(const FimFft& P, float2* spec, float* real, void* d_tables, float scaling, StatRecord* rec,
                           cudaStream_t stream) {
  cudaError_t e = ensure_attributes();
  if (e != cudaSuccess) return e;
  TableArgs A{};
  AxisTables T[3] = {};
  uint8_t* w = static_cast<uint8_t*>(d_tables);
  int most = 0;
  for (int d = 0; d < 3; ++d) {
    A.ax[d] = P.ax[d];
    const FimAxis& X = P.ax[d];
    if (!X.n) continue;
    float4* q = reinterpret_cast<float4*>(w);
    A.tw[d] = q;
    A.hat[d] = q + X.f.n;
    A.chirp[d] = A.hat[d] + X.f.n;
    float4* pk = A.chirp[d] + X.n;
    if (d == 0) A.pack = pk;
    A.rev[d] = reinterpret_cast<int*>(pk + X.n + 2);
    T[d] = AxisTables{A.tw[d], A.chirp[d], A.hat[d], A.rev[d], d == 0 ? A.pack : nullptr};
    w += (table_bytes(X) + 255) / 256 * 256;
    most = std::max(most, std::max(X.f.n, X.n + 1));
  }
  A.n1 = P.n[0];
  fim_tables_kernel<<<dim3((most + 3) / 4, 3), 128, 0, stream>>>(A);
  const int n1h = P.n[0] / 2 + 1;
  const unsigned tiles = static_cast<unsigned>((n1h + kTile - 1) / kTile);
  const long long row = n1h, plane = row * P.n[1];
  if (P.ax[2].n)
    fim_columns_kernel<<<dim3(tiles, P.n[1]), axis_threads(P.ax[2]), axis_smem(P.ax[2]), stream>>>(P.ax[2], T[2], spec, n1h,
                                                                                                   plane, row);
  if (P.ax[1].n)
    fim_columns_kernel<<<dim3(tiles, P.n[2]), axis_threads(P.ax[1]), axis_smem(P.ax[1]), stream>>>(P.ax[1], T[1], spec, n1h,
                                                                                                   row, plane);
  const long long rows = static_cast<long long>(P.n[1]) * P.n[2];
  fim_rows_kernel<<<static_cast<unsigned>(fim_fft_records(P)), axis_threads(P.ax[0]), axis_smem(P.ax[0]), stream>>>(
      P.ax[0], T[0], spec, real, rows, scaling, rec);
  return cudaGetLastError();
}

}  // namespace scarf
