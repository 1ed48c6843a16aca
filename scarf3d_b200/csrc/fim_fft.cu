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
// backwards are one step in registers. Lengths without prime factors above 7 take
// a plain transform.
//
// N = q p with p prime and p - 1 without prime factors above 7 (514 = 2 x 257)
// takes a shorter way. Indices n = p b + q m and k = (k mod q, k mod p) split the
// transform into q-point ones over b and p-point ones over m without twiddles
// (Good 1958, Thomas 1963), and the p-point ones are, with a primitive root g,
// cyclic convolutions over the non-zero residues (Rader 1968):
//   Y[g^-v] = y[0] + sum_u y[g^u] c_{v - u},  c_d = e^{2 pi i g^-d / p},
// p - 1 points where Bluestein's form takes at least 2 p - 1. The tile's q (p - 1)
// values run through one plan: the q-point stages, then the convolution in each
// of q blocks; the q values of residue 0 are transformed apart, added to the
// convolution through its constant term, and with that term's input they are the
// outputs of residue 0.
//
// Bound: shared-memory traffic of the stages. 514^3: cuFFT's transforms took
// 4.2 ms (z 1.51, y 1.42, x 1.26 with its preprocessing) and the statistics 0.11
// more; Bluestein's form over 1 080 points (69 KB tiles) 3.2, Rader's over 512
// (33 KB) 1.8, 1.7 with inputs copied asynchronously into their slots (all in
// flight at once) and rows stored in order, 1.4 with tables of plain entries and
// 1 024 threads per SM. Radix 7 puts 258 = 6 x 43 (43 - 1 = 6 x 7) there too:
// 258^3 341 -> 208 us. A q beyond 64 would make the serial q-point sums long: Bluestein.
//
// The c2r step stores the scaled field (1 / sqrt(n1 n2 n3 dh^n), :1019) and
// records its statistics (:1027-1036), one record per block, as it goes.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdint>

#include "common.cuh"
#include "fft_tile.cuh"
#include "srm_kernels.h"

namespace scarf {
namespace {

using namespace fft;

constexpr int kPairs = 4;               // transform pairs of a tile
constexpr int kTile = 2 * kPairs;       // transforms of a tile
// Threads of an SM and most of a block, by form: the stages wait for memory and
// barriers, so threads count for more than spills (64 registers: 170 to 310 bytes
// a thread). Transform of 514^3 points
// (Rader's form) 1 675 us with 640 threads of 96 registers, 1 595 with 768 of 80,
// 1 565 with 896 of 72 and 1 398 with 1 024 of 64; 256^3 (plain) 164, 161, 156,
// 153; but 402 x 402 x 202 (Bluestein's along x and y, whose radices are larger)
// 543, 518, 525, 541.
constexpr int sm_threads(int form) { return form == kFimBluestein ? 768 : 1024; }
// A block takes 256 threads, more (up to an SM's) only where the tiles are too
// few, or too large, for blocks of 256 to fill the SMs: 78 x 1407 points, six
// tiles of Bluestein's form, 132 us a call with 256 and 126 with more.
constexpr int most_threads(int form) { return sm_threads(form); }
constexpr int kUsualThreads = 256;
constexpr size_t kSmemMax = 224 * 1024;

// Device tables of one axis: twiddles of its plan, then (Bluestein) the chirp
// and the transformed chirp in the forward transform's output order, or
// (plain) the output order of the last stage's butterflies; for the real axis
// the roots of its packing.
struct AxisTables {
  const float2* tw;     // {cos, sin}
  const float2* chirp;  // n entries, the same form
  const float2* hat;    // f.n entries
  const int* rev;       // at e - t of the last stage (plain)
  // Rader's form: output of each position, position of each input (the q of
  // residue 0 at f.n .. ), outputs of residue 0, roots of the q-point transform.
  const int* dst;
  const int* place;
  const int* zero;
  const float2* roots;
  const int* from;      // slot of each output (real axis, plain and Rader's form)
  const float2* pack;   // e^{2 pi i k / n1}, k <= n1 / 4 (real axis)
};

struct TableArgs {
  FimAxis ax[3];
  float2* tw[3];
  float2* chirp[3];
  float2* hat[3];
  int* rev[3];
  int* dst[3];
  int* place[3];
  int* zero[3];
  float2* roots[3];
  int* from;
  float2* pack;
  int n1;
};

__device__ __forceinline__ float2 table_root(double turns) {
  double s, c;
  sincospi(2.0 * (turns - rint(turns)), &s, &c);
  return make_float2(static_cast<float>(c), static_cast<float>(s));
}
// n^2 / (2 N) modulo 1, exactly reduced
__device__ __forceinline__ double chirp_turns(int n, int N) {
  const long long q = static_cast<long long>(n) * n % (2ll * N);
  return static_cast<double>(q) / (2.0 * N);
}

// b^e modulo p
__device__ __forceinline__ int power_mod(int b, int e, int p) {
  long long r = 1, x = b;
  for (; e > 0; e >>= 1) {
    if (e & 1) r = r * x % p;
    x = x * x % p;
  }
  return static_cast<int>(r);
}
// Frequency at position pos of stages s0 .. s1 - 1, which transform `span` points.
__device__ __forceinline__ int stage_frequency(const FftPlan& f, int s0, int s1, int span, int pos) {
  int k = 0, w = 1;
  for (int s = s0; s < s1; ++s) {
    span /= f.r[s];
    const int d = pos / span;
    pos -= d * span;
    k += d * w;
    w *= f.r[s];
  }
  return k;
}
// Rader's form: the q-point stages see the q blocks only.
__device__ double rader_twiddle(const FimAxis& X, int i) {
  const FftPlan& f = X.f;
  int at = i, len = f.n;
  for (int s = 0; s < X.sq; ++s) {
    const int count = len - f.m[s];
    if (at < count) {
      const int t = at / f.m[s], b = (at - t * f.m[s]) / (X.p - 1);
      return static_cast<double>(b * (t + 1)) / (len / (X.p - 1));
    }
    at -= count;
    len = f.m[s];
  }
  return twiddle_entry(f, i);
}
__device__ void rader_tables(const TableArgs& A, int a, int i, int lane) {
  const FimAxis& X = A.ax[a];
  const FftPlan& f = X.f;
  const int len = X.p - 1;
  if (lane == 0) {
    if (i < f.n) {
      const int j = i / len, u = i - j * len;
      const int from = static_cast<int>((static_cast<long long>(X.p) * j + static_cast<long long>(X.q) * power_mod(X.root, u, X.p)) % X.n);
      A.tw[a][i] = table_root(rader_twiddle(X, i));
      A.place[a][from] = i;
      const int to = static_cast<int>((static_cast<long long>(stage_frequency(f, 0, X.sq, X.q, j)) * X.cq +
                                       static_cast<long long>(power_mod(X.root, len - u, X.p)) * X.cp) % X.n);
      A.dst[a][i] = to;
      if (a == 0) A.from[to] = i;
    }
    if (i < X.q) {
      A.place[a][static_cast<long long>(X.p) * i % X.n] = f.n + i;
      const int to = static_cast<int>(static_cast<long long>(stage_frequency(f, 0, X.sq, X.q, i)) * X.cq % X.n);
      A.zero[a][i] = to;
      if (a == 0) A.from[to] = f.n + i;
    }
    if (i < X.q * X.q) {
      const int j = i / X.q, b = i - j * X.q;
      A.roots[a][i] = table_root(static_cast<double>(b * stage_frequency(f, 0, X.sq, X.q, j) % X.q) / X.q);
    }
  }
  if (i >= f.n) return;
  // hat = (1 / (p - 1)) sum_d c_d e^{2 pi i d freq / (p - 1)}
  const int freq = stage_frequency(f, X.sq, f.nst, len, i % len);
  const int hop = power_mod(X.root, len - 32 % len, X.p);  // g^-32
  long long gd = power_mod(X.root, (len - lane % len) % len, X.p);
  double re = 0.0, im = 0.0;
  for (int d = lane; d < len; d += 32) {
    double s, c;
    const double turns = static_cast<double>(gd) / X.p + static_cast<double>(static_cast<long long>(d) * freq % len) / len;
    sincospi(2.0 * (turns - rint(turns)), &s, &c);
    re += c;
    im += s;
    gd = gd * hop % X.p;
  }
  for (int o = 16; o > 0; o >>= 1) {
    re += __shfl_down_sync(0xffffffffu, re, o);
    im += __shfl_down_sync(0xffffffffu, im, o);
  }
  if (lane == 0) {
    A.hat[a][i] = make_float2(static_cast<float>(re / len), static_cast<float>(im / len));
  }
}

// blockIdx.y: axis; one warp per table index.
__global__ void __launch_bounds__(128) fim_tables_kernel(const TableArgs A) {
  const int a = blockIdx.y, lane = threadIdx.x & 31;
  const int i = blockIdx.x * 4 + (threadIdx.x >> 5);
  const FimAxis& X = A.ax[a];
  if (X.n == 0) return;  // axis not transformed
  const FftPlan& f = X.f;
  if (lane == 0 && a == 0 && i <= X.n / 2) A.pack[i] = table_root(static_cast<double>(i) / A.n1);
  if (X.form == kFimRader) {
    rader_tables(A, a, i, lane);
    return;
  }
  const bool blue = X.form == kFimBluestein;
  if (lane == 0) {
    if (i < f.n) A.tw[a][i] = table_root(twiddle_entry(f, i));
    if (blue && i < X.n) A.chirp[a][i] = table_root(chirp_turns(i, X.n));
    const int r = f.r[f.nst - 1];
    if (!blue && i < f.n / r) {
      const int k = output_order(f, i);
      A.rev[a][i * r] = k;
      if (a == 0)
        for (int t = 0; t < r; ++t) A.from[k + t * (f.n / r)] = i * r + t;
    }
  }
  if (!blue || i >= f.n) return;
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
    A.hat[a][i] = make_float2(static_cast<float>(re / f.n), static_cast<float>(im / f.n));
  }
}

__device__ __forceinline__ C2 times(C2 a, const float2* t) {
  const C2 w = root(t);
  return cmul(a, w.re, w.im);
}

// Slot of input e < X.n in a tile.
template <int kForm>
__device__ __forceinline__ int input_slot(const AxisTables& T, int e) {
  if constexpr (kForm == kFimRader) return __ldg(T.place + e);
  return e;
}

// The tile's transforms, its inputs in the tile's slots. Columns: inputs as
// {re0, im0, re1, im1}, out(e, p, v) takes output e < X.n. Rows (kRows): outputs
// stay in the slots that `from` gives, except for Bluestein's, whose last stage
// has them in order. (Leaving from the last stage of the other forms, eight bytes
// at a time in their order, the rows wrote six times their sectors.)
template <int kForm, bool kRows, class Out>
__device__ __forceinline__ void transform_tile(const FimAxis& X, const AxisTables& T, ulonglong2* sh, Out out) {
  const FftPlan& f = X.f;
  auto sin = [&](int e, int p) {
    const ulonglong2 v = sh[e * kPairs + p];
    return C2{v.x, v.y};
  };
  auto sout = [&](int e, int p, int, C2 v) { sh[e * kPairs + p] = make_ulonglong2(v.re, v.im); };
  auto input = [&](int e, int p) {
    if constexpr (kRows) return sin(e, p);
    const float4 v = *reinterpret_cast<const float4*>(sh + e * kPairs + p);
    return C2{pack(v.x, v.z), pack(v.y, v.w)};
  };
  const int last = f.nst - 1, rl = f.r[last], hop = f.n / rl;
  if constexpr (kForm == kFimPlain) {
    stage_any<kPairs>(f, 0, T.tw, input, sout);
    for (int s = 1; s < last; ++s) {
      __syncthreads();
      stage_any<kPairs>(f, s, T.tw, sin, sout);
    }
    __syncthreads();
    if constexpr (kRows)
      stage_any<kPairs>(f, last, T.tw, sin, sout);
    else
      stage_any<kPairs>(f, last, T.tw, sin,
                        [&](int e, int p, int t, C2 v) { out(__ldg(T.rev + e - t) + t * hop, p, v); });
  } else if constexpr (kForm == kFimRader) {
    const int q = X.q;
    // Residue 0: q-point transforms into slots f.n + q .. (the last threads,
    // which have the fewest butterflies).
    for (int it = blockDim.x - 1 - threadIdx.x; it < q * kPairs; it += blockDim.x) {
      const int p = it & (kPairs - 1), j = it / kPairs;
      C2 v = input(f.n, p);
      for (int b = 1; b < q; ++b) v = v + times(input(f.n + b, p), T.roots + j * q + b);
      sout(f.n + q + j, p, 0, v);
    }
    stage_any<kPairs>(f, 0, T.tw, input, sout);
    for (int s = 1; s < last; ++s) {
      __syncthreads();
      stage_any<kPairs>(f, s, T.tw, sin, sout);
    }
    __syncthreads();
    // A block's constant term: with residue 0's value it is the output of
    // residue 0 (slots f.n ..), and that value joins its product.
    auto constant = [&](int base, int p, C2 v, C2& y) {
      const int j = static_cast<int>((static_cast<float>(base) + 0.5f) * X.inv_len);
      if (j * (X.p - 1) != base) return;
      const C2 z = sin(f.n + q + j, p);
      sout(f.n + j, p, 0, z + v);
      y = y + z;
    };
    auto put = [&](int e, int p, int t, C2 v) {
      if constexpr (kRows)
        sout(e, p, t, v);
      else
        out(__ldg(T.dst + e), p, v);
    };
    if (last == X.sq) {
      product_any<kPairs>(f, T.hat, sin, put, constant);
      __syncthreads();
    } else {
      product_any<kPairs>(f, T.hat, sin, sout, constant);
      for (int s = last - 1; s > X.sq; --s) {
        __syncthreads();
        back_any<kPairs>(f, s, T.tw, sin, sout);
      }
      __syncthreads();
      back_any<kPairs>(f, X.sq, T.tw, sin, put);
    }
    if constexpr (kRows) return;
    for (int it = blockDim.x - 1 - threadIdx.x; it < q * kPairs; it += blockDim.x) {
      const int p = it & (kPairs - 1), j = it / kPairs;
      out(__ldg(T.zero + j), p, sin(f.n + j, p));
    }
  } else {
    auto bin = [&](int e, int p) {
      if (e >= X.n) return C2{0ull, 0ull};
      return times(input(e, p), T.chirp + e);
    };
    stage_any<kPairs>(f, 0, T.tw, bin, sout);
    for (int s = 1; s < last; ++s) {
      __syncthreads();
      stage_any<kPairs>(f, s, T.tw, sin, sout);
    }
    __syncthreads();
    product_any<kPairs>(f, T.hat, sin, sout, [](int, int, C2, C2&) {});
    for (int s = last - 1; s > 0; --s) {
      __syncthreads();
      back_any<kPairs>(f, s, T.tw, sin, sout);
    }
    __syncthreads();
    back_any<kPairs>(f, 0, T.tw, sin, [&](int e, int p, int, C2 v) {
      if (e < X.n) out(e, p, times(v, T.chirp + e));
    });
  }
}

// c2c along z or y, in place: blockIdx.x selects eight neighbouring x bins,
// blockIdx.y the row or plane.
template <int kForm>
__global__ void __launch_bounds__(most_threads(kForm), 1)
    fim_columns_kernel(const FimAxis X, const AxisTables T, float2* spec, int n1h, long long step, long long outer) {
  extern __shared__ __align__(128) unsigned char smem[];
  const int i0 = blockIdx.x * kTile, left = n1h - i0;
  float2* base = spec + blockIdx.y * outer + i0;
  const bool wide = (reinterpret_cast<uintptr_t>(base) & 15u) == 0 && (step & 1) == 0;
  ulonglong2* sh = reinterpret_cast<ulonglong2*>(smem);
  for (int it = threadIdx.x; it < X.n * kPairs; it += blockDim.x) {
    const int p = it & (kPairs - 1), e = it / kPairs;
    const float2* s = base + e * step + 2 * p;
    float2* d = reinterpret_cast<float2*>(sh + input_slot<kForm>(T, e) * kPairs + p);
    if (wide && 2 * p + 1 < left) {
      cp_async16(d, s);
    } else {
      if (2 * p < left) cp_async8(d, s);
      else d[0] = make_float2(0.0f, 0.0f);
      if (2 * p + 1 < left) cp_async8(d + 1, s + 1);
      else d[1] = make_float2(0.0f, 0.0f);
    }
  }
  cp_async_wait();
  __syncthreads();
  transform_tile<kForm, false>(X, T, sh, [&](int e, int p, C2 v) {
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
template <int kForm>
__global__ void __launch_bounds__(most_threads(kForm), 1)
    fim_rows_kernel(const FimAxis X, const AxisTables T, const float2* spec, float* real, long long rows, float scaling,
                    Moments* rec) {
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ Moments s_warp[most_threads(kForm) / 32];
  const int n = X.n, half = n / 2;
  const long long r0 = static_cast<long long>(blockIdx.x) * kTile;
  const int left = static_cast<int>(rows - r0 < kTile ? rows - r0 : kTile);
  const float2* src = spec + r0 * (n + 1);
  float* dst = real + r0 * (2 * n);
  ulonglong2* sh = reinterpret_cast<ulonglong2*>(smem);
  // Bin n waits in the slot behind the others (Bluestein's form: an empty one).
  const int spare = kForm == kFimRader ? X.f.n + 2 * X.q : n;
  auto slot = [&](int k, int p) { return sh + (k == n ? spare : input_slot<kForm>(T, k)) * kPairs + p; };
  for (int it = threadIdx.x; it < (n + 1) * kPairs; it += blockDim.x) {
    const int p = it & (kPairs - 1), k = it / kPairs;
    float2* d = reinterpret_cast<float2*>(slot(k, p));
    const float2* s = src + static_cast<long long>(2 * p) * (n + 1) + k;
    if (2 * p < left) cp_async8(d, s);
    else d[0] = make_float2(0.0f, 0.0f);
    if (2 * p + 1 < left) cp_async8(d + 1, s + n + 1);
    else d[1] = make_float2(0.0f, 0.0f);
  }
  cp_async_wait();
  __syncthreads();
  for (int it = threadIdx.x; it < (half + 1) * kPairs; it += blockDim.x) {
    const int p = it & (kPairs - 1), k = it / kPairs;
    ulonglong2 *pa = slot(k, p), *pb = slot(n - k, p);
    const float4 x = *reinterpret_cast<const float4*>(pa), y = *reinterpret_cast<const float4*>(pb);
    const C2 a = C2{pack(x.x, x.z), pack(x.y, x.w)}, b = C2{pack(y.x, y.z), pack(y.y, y.w)};
    if (k == 0) {
      *pa = make_ulonglong2(add(a.re, b.re), sub(a.re, b.re));
    } else {
      // Bins 0 < k < n count twice (Hermitian): (A_k + conj A_{n-k}) +
      // i e^{2 pi i k / n1} (A_k - conj A_{n-k}).
      const C2 s = C2{add(a.re, b.re), sub(a.im, b.im)};
      const C2 u = times(C2{sub(a.re, b.re), add(a.im, b.im)}, T.pack + k);
      const C2 z = add_i(s, u);
      *pa = make_ulonglong2(z.re, z.im);
      if (2 * k != n) *pb = make_ulonglong2(add(s.re, u.im), sub(u.re, s.im));
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
  auto store = [&](int e, int p, C2 v) {
    if (2 * p < left) put(2 * p, e, lo(v.re), lo(v.im));
    if (2 * p + 1 < left) put(2 * p + 1, e, hi(v.re), hi(v.im));
  };
  transform_tile<kForm, true>(X, T, sh, store);
  if constexpr (kForm != kFimBluestein) {
    __syncthreads();
    for (int it = threadIdx.x; it < n * kPairs; it += blockDim.x) {
      const int p = it & (kPairs - 1), e = it / kPairs;
      const ulonglong2 v = sh[__ldg(T.from + e) * kPairs + p];
      store(e, p, C2{v.x, v.y});
    }
  }
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
size_t axis_smem(const FimAxis& X) {
  return sizeof(float2) * kTile * (static_cast<size_t>(X.f.n) + (X.form == kFimRader ? 2 * X.q : 0) + 1);
}

// Appends the radices of an n-point transform; false when there are none.
bool append_radices(int n, FftPlan* f) {
  if (n == 1) return true;
  FftPlan g{};
  const bool one = n <= 12 && n != 11;  // a single butterfly
  if (one) {
    g.nst = 1;
    g.r[0] = n;
  } else if (!fft_plan(n, &g, 7)) {
    return false;
  }
  if (f->nst + g.nst > FftPlan::kMaxStages) return false;
  for (int s = 0; s < g.nst; ++s) f->r[f->nst++] = g.r[s];
  return true;
}

constexpr int kMostBlocks = 64;  // q of Rader's form: q^2 roots, and serial q-point sums

// n = q p with one prime p above 7, p - 1 without prime factors above 7.
bool rader_axis(int n, FimAxis* X) {
  int q = 1, p = n;
  for (int k : {2, 3, 5, 7})
    while (p % k == 0) p /= k, q *= k;
  if (p < 11 || q > kMostBlocks) return false;
  for (int k = 11; k * k <= p; k += 2)
    if (p % k == 0) return false;
  FftPlan f{};
  if (!append_radices(q, &f)) return false;
  const int sq = f.nst;
  // At least two stages: a barrier then separates a tile's reads from its writes.
  if (!append_radices(p - 1, &f) || f.nst < 2) return false;
  f.n = q * (p - 1);
  int len = f.n;
  for (int s = 0; s < f.nst; ++s) {
    len /= f.r[s];
    f.m[s] = len;
    f.inv_m[s] = 1.0f / static_cast<float>(len);
  }
  X->f = f;
  X->form = kFimRader;
  X->q = q;
  X->p = p;
  X->sq = sq;
  X->inv_len = 1.0f / static_cast<float>(p - 1);
  auto power = [&](long long b, int e) {
    long long r = 1;
    for (b %= p; e > 0; e >>= 1, b = b * b % p)
      if (e & 1) r = r * b % p;
    return r;
  };
  // g is a primitive root when no g^((p - 1) / prime) is 1.
  for (X->root = 2;; ++X->root) {
    bool ok = true;
    for (int k : {2, 3, 5, 7})
      if ((p - 1) % k == 0 && power(X->root, (p - 1) / k) == 1) ok = false;
    if (ok) break;
  }
  X->cp = X->cq = 0;
  for (int v = 0; v < n; v += q)
    if (v % p == 1) X->cp = v;
  for (int v = 0; v < n; v += p)
    if (v % q == 1 % q) {
      X->cq = v;
      break;
    }
  return true;
}

bool make_axis(int n, FimAxis* X) {
  *X = FimAxis{};
  X->n = n;
  X->form = kFimPlain;
  X->q = X->p = 1;
  if (fft_plan(n, &X->f, 7) || rader_axis(n, X)) return axis_smem(*X) <= kSmemMax;
  X->form = kFimBluestein;
  const int lo = std::max(4, 2 * n - 1);
  double best = 0.0;
  int found = 0;
  for (int m = lo; m <= lo + lo / 4 + 16; ++m) {
    FftPlan f;
    if (found && static_cast<double>(m) * (fft_least_stages(m) + 2) >= best) break;
    if (!fft_plan(m, &f)) continue;
    const double cost = static_cast<double>(m) * (f.nst + 2);
    if (!found || cost < best) {
      found = m;
      best = cost;
      X->f = f;
    }
  }
  return found && axis_smem(*X) <= kSmemMax;
}

// The block size that fills an SM (sm_threads) with the least idle threads;
// beyond kUsualThreads only where such blocks leave half of it empty.
int axis_threads(const FimAxis& X, long long tiles) {
  int best = 128;
  double best_cost = 1e30;
  const int fit = static_cast<int>(std::min<size_t>(kSmemMax / axis_smem(X), 16));  // blocks of an SM
  const int share = static_cast<int>(std::min<long long>((tiles + 147) / 148, 16));  // tiles of an SM
  for (int t = 64; t <= most_threads(X.form); t += 32) {
    if (t > kUsualThreads && 2 * best * std::min(share, fit) > sm_threads(X.form)) break;
    const int blocks = std::min(fit, sm_threads(X.form) / t);
    if (blocks < 1) continue;
    double work = 0.0;
    for (int s = 0; s < X.f.nst; ++s) {
      const int items = X.f.n / X.f.r[s] * kPairs;
      work += static_cast<double>((items + t - 1) / t) * t / items;
    }
    const double cost = work / (std::min(blocks, share) * t);
    if (cost < best_cost) best_cost = cost, best = t;
  }
  return best;
}

// Lays the tables of an axis out from w; returns their bytes.
size_t axis_tables(const FimAxis& X, int d, uint8_t* w, TableArgs* A) {
  size_t at = 0;
  auto take = [&](size_t count, size_t size) {
    uint8_t* p = w + at;
    at += (count * size + 15) / 16 * 16;
    return p;
  };
  const size_t m = X.f.n, n = X.n, q = X.q;
  A->tw[d] = reinterpret_cast<float2*>(take(m, sizeof(float2)));
  if (X.form != kFimPlain) A->hat[d] = reinterpret_cast<float2*>(take(m, sizeof(float2)));
  if (X.form == kFimPlain) A->rev[d] = reinterpret_cast<int*>(take(m, sizeof(int)));
  if (X.form == kFimBluestein) A->chirp[d] = reinterpret_cast<float2*>(take(n, sizeof(float2)));
  if (X.form == kFimRader) {
    A->roots[d] = reinterpret_cast<float2*>(take(q * q, sizeof(float2)));
    A->dst[d] = reinterpret_cast<int*>(take(m, sizeof(int)));
    A->place[d] = reinterpret_cast<int*>(take(n, sizeof(int)));
    A->zero[d] = reinterpret_cast<int*>(take(q, sizeof(int)));
  }
  if (d == 0 && X.form != kFimBluestein) A->from = reinterpret_cast<int*>(take(n, sizeof(int)));
  if (d == 0) A->pack = reinterpret_cast<float2*>(take(n / 2 + 1, sizeof(float2)));
  return (at + 255) / 256 * 256;
}

// Raises a kernel's limit of dynamic shared memory, once per device context.
// Only of the kernels that a call launches: raising the limits of all forms
// loads all of them, ~2 ms of a process's first call.
template <class F>
cudaError_t most_smem(F* kernel, std::atomic<unsigned long long> (&done)[64]) {  // done: context ids
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const unsigned long long ctx = current_context_id();
  if (dev >= 0 && dev < 64 && ctx != 0 && done[dev] == ctx) return cudaSuccess;
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kSmemMax));
  if (e == cudaSuccess && dev >= 0 && dev < 64) done[dev] = ctx;
  return e;
}

template <int kForm, class... Args>
cudaError_t launch_columns(dim3 grid, const FimAxis& X, cudaStream_t stream, Args... args) {
  static std::atomic<unsigned long long> done[64];
  const cudaError_t e = most_smem(fim_columns_kernel<kForm>, done);
  const int threads = axis_threads(X, static_cast<long long>(grid.x) * grid.y);
  if (e == cudaSuccess) fim_columns_kernel<kForm><<<grid, threads, axis_smem(X), stream>>>(X, args...);
  return e;
}

template <int kForm, class... Args>
cudaError_t launch_rows(unsigned blocks, const FimAxis& X, cudaStream_t stream, Args... args) {
  static std::atomic<unsigned long long> done[64];
  const cudaError_t e = most_smem(fim_rows_kernel<kForm>, done);
  if (e == cudaSuccess) fim_rows_kernel<kForm><<<blocks, axis_threads(X, blocks), axis_smem(X), stream>>>(X, args...);
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
  TableArgs A{};
  for (int d = 0; d < 3; ++d)
    if (P->ax[d].n) P->tables += axis_tables(P->ax[d], d, nullptr, &A);
  return true;
}

long long fim_fft_records(const FimFft& P) {
  return (static_cast<long long>(P.n[1]) * P.n[2] + kTile - 1) / kTile;
}

cudaError_t launch_fim_fft(const FimFft& P, float2* spec, float* real, void* d_tables, bool tables_ready, float scaling,
                           StatRecord* rec, cudaStream_t stream) {
  TableArgs A{};
  AxisTables T[3] = {};
  uint8_t* w = static_cast<uint8_t*>(d_tables);
  int most = 0;
  for (int d = 0; d < 3; ++d) {
    A.ax[d] = P.ax[d];
    const FimAxis& X = P.ax[d];
    if (!X.n) continue;
    w += axis_tables(X, d, w, &A);
    T[d] = AxisTables{A.tw[d], A.chirp[d], A.hat[d], A.rev[d], A.dst[d], A.place[d], A.zero[d], A.roots[d],
                      d == 0 ? A.from : nullptr, d == 0 ? A.pack : nullptr};
    most = std::max(most, std::max(X.f.n, std::max(X.n + 1, X.q * X.q)));
  }
  A.n1 = P.n[0];
  if (!tables_ready) fim_tables_kernel<<<dim3((most + 3) / 4, 3), 128, 0, stream>>>(A);
  const int n1h = P.n[0] / 2 + 1;
  const unsigned tiles = static_cast<unsigned>((n1h + kTile - 1) / kTile);
  const long long row = n1h, plane = row * P.n[1];
  auto columns = [&](const FimAxis& X, const AxisTables& t, int outer, long long step, long long hop) {
    const dim3 grid(tiles, outer);
    if (X.form == kFimPlain) return launch_columns<kFimPlain>(grid, X, stream, t, spec, n1h, step, hop);
    if (X.form == kFimRader) return launch_columns<kFimRader>(grid, X, stream, t, spec, n1h, step, hop);
    return launch_columns<kFimBluestein>(grid, X, stream, t, spec, n1h, step, hop);
  };
  cudaError_t e = cudaSuccess;
  if (P.ax[2].n && (e = columns(P.ax[2], T[2], P.n[1], plane, row)) != cudaSuccess) return e;
  if (P.ax[1].n && (e = columns(P.ax[1], T[1], P.n[2], row, plane)) != cudaSuccess) return e;
  const long long rows = static_cast<long long>(P.n[1]) * P.n[2];
  const unsigned blocks = static_cast<unsigned>(fim_fft_records(P));
  const FimAxis& X = P.ax[0];
  if (X.form == kFimPlain)
    e = launch_rows<kFimPlain>(blocks, X, stream, T[0], spec, real, rows, scaling, rec);
  else if (X.form == kFimRader)
    e = launch_rows<kFimRader>(blocks, X, stream, T[0], spec, real, rows, scaling, rec);
  else
    e = launch_rows<kFimBluestein>(blocks, X, stream, T[0], spec, real, rows, scaling, rec);
  return e != cudaSuccess ? e : cudaGetLastError();
}

}  // namespace scarf
