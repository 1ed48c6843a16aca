// Structured SRM sums through a non-uniform Fourier transform.
//
// On a regular grid the sum over harmonics (scarflib_srm.f90:794-809) is a
// Fourier sum at arbitrary wavenumbers: with i', j' the indices about the
// grid's middle,
//   field(i, j, k) = scaling Re sum_h E_h(k) e^{2 pi i (wx_h i' + wy_h j')},
//   E_h(k) = (b - i a) e^{i (kx x_mid + ky y_mid + kz z_k + v . bar)},
// and e^{2 pi i w n} for |n| <= N/2 is, to ~2e-7, a weighted sum of the nine
// nearest waves of period M >= 1.5 N (Dutt & Rokhlin 1993; Kaiser-Bessel
// weights, whose Fourier transform is known in closed form). So
//   1. every harmonic adds E_h(k) to 9 x 9 cells (cx, cy) of a wavenumber
//      grid, for every k (the z dependence stays exact): T1[cx][cy][k];
//   2. an inverse FFT of length My along cy gives T2[cx][j][k];
//   3. an inverse real FFT of length Mx along cx gives the field.
// Wavenumbers with wx < 0 are taken as their conjugates (the field is a real
// part), so only cx in [0, Mx/2] is kept; the parts of a harmonic's cells
// outside that range fold back as the cells of a mirror entry (-w, conj E).
// The work is ~1.5 x 2.25 cells per point through two FFT passes plus 81
// multiply-adds per harmonic and plane (144 with the bins' margins), where the factorised contraction
// (srm_tc.cu) takes 12 tensor operations per point and harmonic.
//
// Precision: phases in FP64, E, weights and FFTs in FP32; 2.4e-7 to 1.1e-6 of
// the field's standard deviation (rms) against FP64, where the split-BF16
// contraction has ~5e-6. Summation order is fixed (sorted entries, fixed partial sums),
// so a field is reproducible bit for bit.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdint>

#include "common.cuh"
#include "fft_tile.cuh"
#include "srm_kernels.h"

namespace scarf {
namespace {

constexpr int kW = 9;             // cells per harmonic and gridded axis
constexpr int kB = 4;             // cells per bin
constexpr int kSpan = 3;          // bins that a harmonic's cells can touch
constexpr int kMinM = 24;         // shortest transform (a harmonic's cells never wrap onto themselves)
constexpr double kOversample = 1.5;
constexpr int kSparse = 32;       // entries of a bin that one warp sums
constexpr int kPart = 256;        // entries that one block sums (32 per warp)
constexpr int kScanThreads = 1024;
constexpr int kDense = 2048;      // entries of a start bin ranked by a block, where blocks rank
constexpr int kRankThreads = 1024;
constexpr int kRankWords = 8192;  // bitmap words of a ranking block: 262 144 entry numbers at a time
constexpr int kZT = 8;            // planes of a transform tile
constexpr int kPairs = kZT / 2;
constexpr int kFftMaxThreads = 512;
static_assert((kSpan - 1) * kB + 1 == kW, "a cell bin is reached from exactly kSpan start bins");

struct GridArgs {
  FftPlan fx, fy;      // lengths mx / 2 and my
  int mx, my, hx;      // transform lengths, hx = mx / 2
  int nx, ny, nz;      // logical extents: x, gridded second axis (1: none), z
  int sx, sy;          // index of the grid's middle: i' = i - sx, j' = j - sy
  int ax;              // columns cx < ax that harmonics reach (T1 and T2 hold these)
  int ylo, yhi, ya;    // cells cy < ylo and the last yhi of my that they reach, ya in all (T1's rows)
  int nbx, nby, nkeys; // cell bins along x and y; start-bin keys
  int nent;            // entries: a harmonic and possibly its mirror
  int nh;
  int ranked;          // bins of more than kDense entries are ranked by blocks
  long long ez;        // z pitch of E
  double beta_x, beta_y, inv_i0_x, inv_i0_y;
  double m[9], bar[3], ds;
  int fs[3];           // first index (1-based) of the axes x, y, z of the caller
  int ax_y, ax_z;      // physical axes of the logical second and third axes
  float scaling;
  long long plane;     // elements between consecutive z of the field
  const float* table;
  uint2* keys;         // per entry: start-bin key, order of arrival in its bin
  int* members;        // entries by bin, in order of arrival
  int* place;          // per entry: its place in bin and entry order
  int* counts;         // entries per key
  double4* par;        // per harmonic: phase (turns), wz (turns per index), a, b
  double2* w;          // per harmonic: wx, wy (cells)
  int* bin_start;
  float* weights;      // per sorted entry: x weights of 3 bins, y weights of 3 bins
  // Complex grids, planes in pairs: {re, re', im, im'} of planes 2 q, 2 q + 1.
  // The sums of step 1 have real weights, so its lanes take 8 bytes each,
  // whichever parts these are.
  float2* e;           // [nent][ez]
  // A transform's tile (kZT planes) is one contiguous piece.
  float2* t1;          // [zc / kZT][ax][ya][kZT]
  float2* t2;          // [zc / kZT][ny][ax][kZT]
  float2* partial;     // [slot][kB * kB][zc]
  int* ntasks;         // four counters: tasks, slots, bins with several parts, dense start bins
  int* dense;          // keys of the start bins that blocks rank
  int4* tasks;         // {bin, part, parts, slot} of the bins that blocks sum
  int4* multi;         // {bin, parts, slot, -} of those with several parts
  // Twiddles {cos, sin}: of the plans fx and fy, and
  // e^{2 pi i k / mx} for k <= hx / 2.
  float2* twx;
  float2* twy;
  float2* twr;
  int* revx;
  int* revy;
  int* status;         // error word of the bounded waits
  float* dcx;          // 1 / window transform, times the field's scaling
  float* dcy;
};

__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }

// ------------------------------------------------------------- preparation --
// I0(2 sqrt(z)) = sum_k z^k / (k!)^2 for 0 <= z < 200 (beta <= 28): every term is
// positive, so Horner's rule keeps full relative precision; the first term left
// out is below 1e-13 of the sum. A branch-free third of CUDA's cyl_bessel_i0 and
// the square root of its argument.
constexpr int kBesselTerms = 38;
struct BesselSeries {
  double c[kBesselTerms];
  constexpr BesselSeries() : c() {
    double v = 1.0;
    for (int k = 0; k < kBesselTerms; ++k) {
      c[k] = v;
      v /= static_cast<double>(k + 1) * (k + 1);
    }
  }
};
__device__ __forceinline__ double bessel_i0_of(double z) {
  constexpr BesselSeries s{};
  double v = s.c[kBesselTerms - 1];
#pragma unroll
  for (int k = kBesselTerms - 2; k >= 0; --k) v = fma(v, z, s.c[k]);
  return v;
}

// Kaiser-Bessel weight at distance d (cells) from a harmonic's wavenumber.
__device__ __forceinline__ float kb_weight(double d, double beta, double inv_i0) {
  const double x = d * (2.0 / kW);
  const double t = 1.0 - x * x;
  return t <= 0.0 ? 0.0f : static_cast<float>(bessel_i0_of(0.25 * beta * beta * t) * inv_i0);
}

// One thread per item: every harmonic's wavenumber in cells, its phase at
// the grid's middle and its entries' sort keys; then the twiddles, output
// orders and window transforms of both axes.
__device__ __forceinline__ int first_cell(double c) { return static_cast<int>(ceil(c - 0.5 * kW)); }
__device__ __forceinline__ int floor_bin(int c) { return (c >= 0 ? c : c - (kB - 1)) / kB; }

__device__ float window_inverse(int n, int m, double beta, double inv_i0) {
  const double pi = 3.14159265358979323846;
  const double u = pi * kW * n / m;
  const double r = sqrt(beta * beta - u * u);
  return static_cast<float>(r / (inv_i0 * kW * sinh(r)));
}

__global__ void __launch_bounds__(128) grid_prep_kernel(const GridArgs A) {
  long long t = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  const double two_pi = 6.28318530717958647692;
  if (t < A.nh) {
    const float* r = A.table + 5 * t;
    const double v1 = r[0], v2 = r[1], v3 = r[2];
    double k[3];
    for (int c = 0; c < 3; ++c) k[c] = (v1 * A.m[c] + v2 * A.m[3 + c] + v3 * A.m[6 + c]) * A.ds / two_pi;
    const double c = (v1 * A.bar[0] + v2 * A.bar[1] + v3 * A.bar[2]) / two_pi;
    // Phase at the middle of x and y and at the first z; axes of one point
    // other than these add their constant.
    double ph = c;
    int mid[3] = {A.sx, 0, 0};
    if (A.ny > 1) mid[A.ax_y] = A.sy;
    for (int ax = 0; ax < 3; ++ax) ph += k[ax] * static_cast<double>(A.fs[ax] - 1 + mid[ax]);
    double wx = k[0] - rint(k[0]), wy = A.ny > 1 ? k[A.ax_y] - rint(k[A.ax_y]) : 0.0, wz = k[A.ax_z];
    double a = r[3], b = r[4];
    if (wx < 0.0) {  // the conjugate: (b - i a) e^{i p} -> (b + i a) e^{-i p}
      wx = -wx;
      wy = -wy;
      wz = -wz;
      ph = -ph;
      a = -a;
    }
    if (wy < 0.0) wy += 1.0;
    // A rotation or a caller's draws may not be finite. No cell index comes
    // from such a wavenumber or phase: the harmonic stands at zero wavenumber
    // with a phase that is no number, so that every value of the field is none.
    if (!(isfinite(k[0]) && isfinite(k[1]) && isfinite(k[2]) && isfinite(ph))) {
      wx = wy = wz = 0.0;
      ph = __longlong_as_double(0x7ff8000000000000ll);
    }
    const double cx = wx * A.mx, cy = wy * A.my;
    A.par[t] = make_double4(ph - rint(ph), wz, a, b);
    A.w[t] = make_double2(cx, cy);
    auto key = [&](double x, double y) {
      const int bx = floor_bin(first_cell(x)) + kSpan;  // -kSpan .. nbx - 1, shifted
      if (A.ny == 1) return static_cast<uint32_t>(bx);
      int s = first_cell(y);
      s += s < 0 ? A.my : 0;
      s -= s >= A.my ? A.my : 0;
      return static_cast<uint32_t>(bx * A.nby + s / kB);
    };
    // One atomic per bin and warp: thousands of entries share the bins near
    // zero wavenumber (20 000 harmonics: 11 us with one each, 6 so).
    auto arrive = [&](uint32_t k) {
      if (k >= static_cast<uint32_t>(A.nkeys)) return make_uint2(k, 0u);
      const unsigned same = __match_any_sync(__activemask(), k);
      const int lane = threadIdx.x & 31, leader = __ffs(same) - 1;
      int at = 0;
      if (lane == leader) at = atomicAdd(A.counts + k, __popc(same));
      at = __shfl_sync(same, at, leader);
      return make_uint2(k, static_cast<uint32_t>(at + __popc(same & ((1u << lane) - 1u))));
    };
    A.keys[t] = arrive(key(cx, cy));
    // Mirror entry: cells below 0 or above hx, folded back.
    uint32_t mk = static_cast<uint32_t>(A.nkeys);  // none
    const int s0 = first_cell(cx);
    const double my_y = cy > 0.0 ? A.my - cy : 0.0;
    if (s0 < 0)
      mk = key(-cx, my_y);
    else if (s0 + kW - 1 > A.hx)
      mk = key(A.mx - cx, my_y);
    A.keys[A.nh + t] = arrive(mk);
    return;
  }
  t -= A.nh;
  auto root = [&](double turns) {
    double s, c;
    sincospi(2.0 * turns, &s, &c);
    return make_float2(static_cast<float>(c), static_cast<float>(s));
  };
  if (t < A.hx) {
    A.twx[t] = root(fft::twiddle_entry(A.fx, static_cast<int>(t)));
    return;
  }
  t -= A.hx;
  if (t <= A.hx / 2) {
    A.twr[t] = root(static_cast<double>(t) / A.mx);
    return;
  }
  t -= A.hx / 2 + 1;
  if (t < A.my) {
    if (A.ny > 1) A.twy[t] = root(fft::twiddle_entry(A.fy, static_cast<int>(t)));
    return;
  }
  t -= A.my;
  if (t < A.nx) {
    A.dcx[t] = window_inverse(static_cast<int>(t) - A.sx, A.mx, A.beta_x, A.inv_i0_x) * A.scaling;
    return;
  }
  t -= A.nx;
  if (t < A.ny) {
    A.dcy[t] = A.ny > 1 ? window_inverse(static_cast<int>(t) - A.sy, A.my, A.beta_y, A.inv_i0_y) : 1.0f;
    return;
  }
  t -= A.ny;
  const int gx = A.fx.n / A.fx.r[A.fx.nst - 1];
  if (t < gx) {
    A.revx[t * A.fx.r[A.fx.nst - 1]] = fft::output_order(A.fx, static_cast<int>(t));
    return;
  }
  t -= gx;
  if (A.ny > 1 && t < A.fy.n / A.fy.r[A.fy.nst - 1]) A.revy[t * A.fy.r[A.fy.nst - 1]] = fft::output_order(A.fy, static_cast<int>(t));
}

// Exclusive scan of the entry counts per key (one block).
__global__ void __launch_bounds__(kScanThreads) grid_scan_kernel(const GridArgs A) {
  __shared__ int s_warp[kScanThreads / 32];
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  int carry = 0;
  for (int base = 0; base <= A.nkeys; base += 4 * kScanThreads) {
    int v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int k = base + 4 * t + u;
      v[u] = k < A.nkeys ? A.counts[k] : 0;
    }
    const int mine = v[0] + v[1] + v[2] + v[3];
    int x = mine;
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    int w = s_warp[lane];
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    const int before_warp = warp ? __shfl_sync(0xffffffffu, w, warp - 1) : 0;
    const int all = __shfl_sync(0xffffffffu, w, 31);
    int at = carry + before_warp + x - mine;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int k = base + 4 * t + u;
      if (k <= A.nkeys) A.bin_start[k] = at;
      if (A.ranked && v[u] > kDense) A.dense[atomicAdd(A.ntasks + 3, 1)] = k;
      at += v[u];
    }
    carry += all;
    __syncthreads();
  }
}

// The kSpan x kSpan start bins whose entries reach cell bin (bx, by): lane
// l < 9 holds bin l's entry range.
__device__ __forceinline__ void bin_ranges(const GridArgs& A, int bin, int lane, int* lo, int* hi) {
  const int bx = bin / A.nby, by = bin - bx * A.nby;
  *lo = *hi = 0;
  const int dx = lane / kSpan, dy = lane - dx * kSpan;
  if (lane < kSpan * kSpan && (A.ny > 1 || dy == 0)) {
    int sy = by - dy;
    sy += sy < 0 ? A.nby : 0;
    const int key = (bx - dx + kSpan) * A.nby + sy;
    *lo = A.bin_start[key];
    *hi = A.bin_start[key + 1];
  }
}

// Entries into their bins, in order of arrival; the blocks after them list
// the tasks of bins with more than kSparse entries (one warp per bin): one
// block per kPart entries, whose partial sum gets a slot when the bin has
// several. Task and slot numbers depend on the order of arrival, sums do not.
__global__ void __launch_bounds__(256) grid_bins_kernel(const GridArgs A, int scatter_blocks) {
  if (static_cast<int>(blockIdx.x) < scatter_blocks) {
    const int e = blockIdx.x * 256 + threadIdx.x;
    if (e >= A.nent) return;
    const uint2 k = A.keys[e];
    if (k.x < static_cast<uint32_t>(A.nkeys)) A.members[A.bin_start[k.x] + k.y] = e;
    return;
  }
  const int bin = (blockIdx.x - scatter_blocks) * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (bin >= A.nbx * A.nby) return;
  int lo, hi;
  bin_ranges(A, bin, lane, &lo, &hi);
  const int total = __reduce_add_sync(0xffffffffu, hi - lo);
  if (total <= kSparse) return;
  const int parts = (total + kPart - 1) / kPart;
  int task = 0, slot = 0;
  if (lane == 0) {
    task = atomicAdd(A.ntasks, parts);
    if (parts > 1) {
      slot = atomicAdd(A.ntasks + 1, parts);
      A.multi[atomicAdd(A.ntasks + 2, 1)] = make_int4(bin, parts, slot, 0);
    }
  }
  task = __shfl_sync(0xffffffffu, task, 0);
  slot = __shfl_sync(0xffffffffu, slot, 0);
  for (int p = lane; p < parts; p += 32) A.tasks[task + p] = make_int4(bin, p, parts, slot);
}

// Places of the entries of dense start bins, one block per bin at a time: a
// bitmap of the bin's entry numbers, whose set bits below an entry's are its
// rank. Linear in the bin, where counting every member for each entry
// (grid_entry_kernel) is quadratic. Bound: two passes over the members, one
// block per bin.
__global__ void __launch_bounds__(kRankThreads) grid_rank_kernel(const GridArgs A) {
  __shared__ uint32_t s_bits[kRankWords];
  __shared__ int s_before[kRankThreads], s_warp[kRankThreads / 32];
  constexpr int kEach = kRankWords / kRankThreads;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int n = A.ntasks[3];
  for (int d = blockIdx.x; d < n; d += gridDim.x) {
    const int key = A.dense[d], lo = A.bin_start[key], hi = A.bin_start[key + 1];
    int base = lo;
    for (int e0 = 0; e0 < A.nent; e0 += 32 * kRankWords) {
      for (int w = t; w < kRankWords; w += kRankThreads) s_bits[w] = 0u;
      __syncthreads();
      for (int i = lo + t; i < hi; i += kRankThreads) {
        const uint32_t b = static_cast<uint32_t>(A.members[i] - e0);
        if (b < 32u * kRankWords) atomicOr(s_bits + (b >> 5), 1u << (b & 31u));
      }
      __syncthreads();
      // Set bits before each run of kEach words.
      int mine = 0;
#pragma unroll
      for (int w = 0; w < kEach; ++w) mine += __popc(s_bits[t * kEach + w]);
      int x = mine;
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
      }
      if (lane == 31) s_warp[warp] = x;
      __syncthreads();
      int before = x - mine, all = 0;
      for (int w = 0; w < kRankThreads / 32; ++w) {
        before += w < warp ? s_warp[w] : 0;
        all += s_warp[w];
      }
      s_before[t] = before;
      __syncthreads();
      for (int i = lo + t; i < hi; i += kRankThreads) {
        const int e = A.members[i];
        const uint32_t b = static_cast<uint32_t>(e - e0);
        if (b >= 32u * kRankWords) continue;
        const int word = static_cast<int>(b >> 5);
        int rank = s_before[word / kEach] + __popc(s_bits[word] & ((1u << (b & 31u)) - 1u));
        for (int w = word / kEach * kEach; w < word; ++w) rank += __popc(s_bits[w]);
        A.place[e] = base + rank;
      }
      base += all;
      __syncthreads();  // the bitmap is read
    }
  }
}

// One warp per entry: its place among its bin's entries (ordered by entry
// number: a fixed order makes every sum over a bin reproducible), its weights
// aligned to bins, and E along z: FP64 phases, stepped by 32 planes with one
// complex product.
__global__ void __launch_bounds__(128) grid_entry_kernel(const GridArgs A, int z0, int nzc, int first) {
  const int e = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (e >= A.nent) return;
  const uint32_t key = A.keys[e].x;
  if (key >= static_cast<uint32_t>(A.nkeys)) return;  // no mirror
  int i;
  const int lo = A.bin_start[key], hi = A.bin_start[key + 1];
  if (first && !(A.ranked && hi - lo > kDense)) {
    int before = 0;
    // Four members per load: bins near zero wavenumber hold thousands of
    // entries, each counting all of them.
    const int head = min((lo + 3) & ~3, hi), tail = head + ((hi - head) & ~3);
    if (lo + lane < head) before += A.members[lo + lane] < e ? 1 : 0;
    if (tail + lane < hi) before += A.members[tail + lane] < e ? 1 : 0;
#pragma unroll 4
    for (int k = head + 4 * lane; k < tail; k += 128) {
      const int4 m = *reinterpret_cast<const int4*>(A.members + k);
      before += (m.x < e ? 1 : 0) + (m.y < e ? 1 : 0) + (m.z < e ? 1 : 0) + (m.w < e ? 1 : 0);
    }
    i = lo + __reduce_add_sync(0xffffffffu, before);
    if (lane == 0) A.place[e] = i;
  } else {
    i = A.place[e];
  }
  const bool mirror = e >= A.nh;
  const int h = mirror ? e - A.nh : e;
  double4 p = A.par[h];
  if (mirror) {
    p.x = -p.x;
    p.y = -p.y;
    p.z = -p.z;
  }
  if (first && lane < 2 * kSpan * kB) {
    const double2 c = A.w[h];
    float v;
    if (lane < kSpan * kB) {
      const bool low = first_cell(c.x) < 0;
      const double x = !mirror ? c.x : (low ? -c.x : A.mx - c.x);
      const int cell = floor_bin(first_cell(x)) * kB + lane;
      v = kb_weight(cell - x, A.beta_x, A.inv_i0_x);
      // A cell belongs to the primary entry inside [0, hx], and outside it,
      // folded, to the mirror.
      if (!mirror ? (cell < 0 || cell > A.hx) : (low ? cell < 1 : cell > A.hx - 1)) v = 0.0f;
    } else if (A.ny > 1) {
      const double y = !mirror ? c.y : (c.y > 0.0 ? A.my - c.y : 0.0);
      const int cell = floor_bin(first_cell(y)) * kB + (lane - kSpan * kB);
      v = kb_weight(cell - y, A.beta_y, A.inv_i0_y);
    } else {
      v = lane == kSpan * kB ? 1.0f : 0.0f;
    }
    A.weights[static_cast<size_t>(i) * (2 * kSpan * kB) + lane] = v;
  }
  // E(z) = (b - i a) e^{2 pi i (phase + wz z)} for z = z0 + lane, + 32, ...
  double s, c, ds, dc;
  const double turns = p.x + p.y * static_cast<double>(z0 + lane), step = p.y * 32.0;
  sincospi(2.0 * (turns - rint(turns)), &s, &c);
  sincospi(2.0 * (step - rint(step)), &ds, &dc);
  float2* out = A.e + static_cast<size_t>(i) * A.ez;
  for (int z = lane; z < nzc; z += 32) {
    const float re = static_cast<float>(p.w * c + p.z * s), im = static_cast<float>(p.w * s - p.z * c);
    // Even lanes store both real parts of a pair of planes, odd lanes both
    // imaginary parts.
    const bool odd = lane & 1;
    const float other = __shfl_xor_sync(0xffffffffu, odd ? re : im, 1);
    out[z] = odd ? make_float2(other, im) : make_float2(re, other);
    const double n = c * dc - s * ds;
    s = c * ds + s * dc;
    c = n;
  }
}

// Step 1. A warp sums up to 32 entries of one 4 x 4-cell bin over 32 planes:
// lanes are planes, the 16 cells are registers. The entries' E rows (256
// bytes each) and weights come into shared memory by asynchronous copies, all
// at once: with four entries in flight from registers the load latency of a
// group was most of its time (512^3 x 20 000: 40 us a pass, 16 warps per SM).
// Bins of up to kSparse entries are one warp's; the first blocks take the
// listed tasks, 8 warps each whose sums are added in order through shared
// memory. Bound: FP32 issue (40 multiply-adds per entry and warp).
struct SpreadWarp {
  float2 e[32][32];         // [entry][lane]
  float w[32][2 * kB];      // x and y weights of the bin's cells
};
constexpr int kSpreadWarps = 8;
static_assert(sizeof(SpreadWarp) >= sizeof(float2) * kB * kB * 32, "the partial sums take the entries' place");

template <int KY>  // cells along y: kB, or 1 when only x is gridded
struct BinSum {
  float2 acc[kB][KY];
};
// Entries [beg, end) (at most 32) of the nine ranges lo, hi of lanes 0 .. 8.
template <int KY>
__device__ __forceinline__ void sum_entries(const GridArgs& A, SpreadWarp& W, int lane, int lo, int hi, int beg, int end,
                                            const float2* ez, BinSum<KY>& S) {
#pragma unroll
  for (int i = 0; i < kB; ++i)
#pragma unroll
    for (int j = 0; j < KY; ++j) S.acc[i][j] = make_float2(0.0f, 0.0f);
  const int n = end - beg;
  if (n <= 0) return;
  // Inclusive prefix of the range lengths; lane l resolves visit beg + l to an
  // entry and its bin offset.
  int pre = hi - lo;
#pragma unroll
  for (int o = 1; o < 16; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, pre, o);
    if (lane >= o) pre += y;
  }
  int r = 0;
#pragma unroll
  for (int q = 0; q < kSpan * kSpan; ++q) r += __shfl_sync(0xffffffffu, pre, q) <= beg + lane ? 1 : 0;
  const int rc = min(r, kSpan * kSpan - 1);
  const int ent = __shfl_sync(0xffffffffu, hi, rc) - (__shfl_sync(0xffffffffu, pre, rc) - (beg + lane));
  if (lane < n) {
    const float* w = A.weights + static_cast<size_t>(ent) * (2 * kSpan * kB);
    fft::cp_async16(&W.w[lane][0], w + rc / kSpan * kB);
    fft::cp_async16(&W.w[lane][kB], w + (kSpan + rc % kSpan) * kB);
  }
  for (int u = 0; u < n; ++u) {
    const int en = __shfl_sync(0xffffffffu, ent, u);
    fft::cp_async8(&W.e[u][lane], ez + static_cast<size_t>(en) * A.ez);
  }
  fft::cp_async_wait();
  __syncwarp();
#pragma unroll 2
  for (int u = 0; u < n; ++u) {
    const float4 wx = *reinterpret_cast<const float4*>(&W.w[u][0]), wy = *reinterpret_cast<const float4*>(&W.w[u][kB]);
    const float2 e = W.e[u][lane];
    const float x[4] = {wx.x, wx.y, wx.z, wx.w}, y[4] = {wy.x, wy.y, wy.z, wy.w};
#pragma unroll
    for (int i = 0; i < kB; ++i) {
      const float2 t = make_float2(x[i] * e.x, x[i] * e.y);
#pragma unroll
      for (int j = 0; j < KY; ++j) {
        S.acc[i][j].x = fmaf(y[j], t.x, S.acc[i][j].x);
        S.acc[i][j].y = fmaf(y[j], t.y, S.acc[i][j].y);
      }
    }
  }
}

// T1 cell (cx, cy), plane z of the pass; shift: row_shift of the cell's bin.
__device__ __forceinline__ size_t t1_index(const GridArgs& A, int cx, int cy, int shift, int z) {
  const int g = z / kZT;
  // A single gridded axis goes straight to step 3, as [zc / kZT][ny = 1][ax][kZT].
  return ((static_cast<size_t>(g) * A.ax + cx) * A.ya + (cy - shift)) * kZT + z % kZT;
}
// Cells minus rows of T1 in a row of bins (a bin is in one of the two pieces).
__device__ __forceinline__ int row_shift(const GridArgs& A, int by) { return by * kB >= A.ylo ? A.my - A.ya : 0; }

template <int KY>
__global__ void __launch_bounds__(32 * kSpreadWarps) grid_spread_kernel(const GridArgs A, int task_blocks, int zoff, int zc) {
  extern __shared__ __align__(128) unsigned char smem[];
  SpreadWarp* warps = reinterpret_cast<SpreadWarp*>(smem);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int z = blockIdx.y * 32 + lane;
  const float2* ez = A.e + zoff + z;
  BinSum<KY> S;
  int lo, hi;
  if (static_cast<int>(blockIdx.x) < task_blocks) {
    const int n = A.ntasks[0];
    for (int task = blockIdx.x; task < n; task += task_blocks) {
      const int4 T = A.tasks[task];
      bin_ranges(A, T.x, lane, &lo, &hi);
      const int total = __reduce_add_sync(0xffffffffu, hi - lo);
      const int beg = min(total, T.y * kPart + warp * 32);
      sum_entries(A, warps[warp], lane, lo, hi, beg, min(total, beg + 32), ez, S);
      __syncwarp();  // the warp's entries are read
      float2(*mine)[32] = reinterpret_cast<float2(*)[32]>(&warps[warp]);
#pragma unroll
      for (int c = 0; c < kB * KY; ++c) mine[c][lane] = S.acc[c / KY][c % KY];
      __syncthreads();
      const int bx = T.x / A.nby, by = T.x - bx * A.nby;
#pragma unroll
      for (int q = 0; q < (kB * KY + kSpreadWarps - 1) / kSpreadWarps; ++q) {
        const int c = warp + kSpreadWarps * q;
        if (c >= kB * KY) break;
        float2 v = make_float2(0.0f, 0.0f);
#pragma unroll
        for (int w = 0; w < kSpreadWarps; ++w) v = cadd(v, reinterpret_cast<const float2(*)[32]>(&warps[w])[c][lane]);
        const int cx = bx * kB + c / KY, cy = by * kB + c % KY;
        if (T.z > 1)
          A.partial[(static_cast<size_t>(T.w + T.y) * (kB * KY) + c) * zc + z] = v;
        else if (cx < A.ax && cy < A.my)
          A.t1[t1_index(A, cx, cy, row_shift(A, by), z)] = v;
      }
      __syncthreads();
    }
    return;
  }
  const int bin = (blockIdx.x - task_blocks) * kSpreadWarps + warp;
  if (bin >= A.nbx * A.nby) return;
  const int bx = bin / A.nby, by = bin - bx * A.nby;
  if (by * kB >= A.ylo && by * kB < A.my - A.yhi) return;  // out of reach
  bin_ranges(A, bin, lane, &lo, &hi);
  const int total = __reduce_add_sync(0xffffffffu, hi - lo);
  if (total > kSparse) return;
  sum_entries(A, warps[warp], lane, lo, hi, 0, total, ez, S);
  const int shift = row_shift(A, by);
#pragma unroll
  for (int i = 0; i < kB; ++i) {
    const int cx = bx * kB + i;
    if (cx >= A.ax) break;
#pragma unroll
    for (int j = 0; j < KY; ++j) {
      const int cy = by * kB + j;
      if (cy < A.my) A.t1[t1_index(A, cx, cy, shift, z)] = S.acc[i][j];
    }
  }
}

// The parts of each bin with several, added in order: one block per bin and
// 32 planes at a time.
template <int KY>
__global__ void __launch_bounds__(32 * kB * KY) grid_parts_kernel(const GridArgs A, int zc) {
  const int n = A.ntasks[2], cell = threadIdx.x >> 5, z = blockIdx.y * 32 + (threadIdx.x & 31);
  for (int m = blockIdx.x; m < n; m += gridDim.x) {
    const int4 T = A.multi[m];
    const int bx = T.x / A.nby, by = T.x - bx * A.nby;
    const size_t hop = static_cast<size_t>(kB * KY) * zc;
    const float2* p = A.partial + (static_cast<size_t>(T.z) * (kB * KY) + cell) * zc + z;
    float2 v = make_float2(0.0f, 0.0f);
    int q = 0;
    for (; q + 8 <= T.y; q += 8) {
      float2 x[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) x[u] = p[(q + u) * hop];
#pragma unroll
      for (int u = 0; u < 8; ++u) v = cadd(v, x[u]);
    }
    for (; q < T.y; ++q) v = cadd(v, p[q * hop]);
    const int cx = bx * kB + cell / KY, cy = by * kB + cell % KY;
    if (cx < A.ax && cy < A.my) A.t1[t1_index(A, cx, cy, row_shift(A, by), z)] = v;
  }
}

// The transforms' blocks are persistent: a block takes tiles blockIdx.x,
// blockIdx.x + gridDim.x, ... each by one bulk copy (loaded by the threads
// themselves, a tile's latency was 40 % of its time) into one buffer: the
// copies are covered by the SM's other blocks. A second buffer per block, for
// the next tile, halves the blocks that fit, and the stages' barriers then
// stand open (sums of 512^3 points x 20 000 harmonics 1 771 us with two
// buffers, 1 661 with one; 1024 x 1024 x 100 x 10 000 1 549 and 1 305).
__device__ __forceinline__ void tile_issue(unsigned char* buf, uint64_t* bar, const void* src, uint32_t bytes) {
  mbar_arrive_expect_tx(bar, bytes);
  bulk_g2s(buf, src, bytes, bar);
}

// Step 2: inverse FFT along cy of the planes of a tile (one cx), the ny
// outputs kept.
__global__ void __launch_bounds__(kFftMaxThreads) grid_fft_y_kernel(const GridArgs A, int tiles) {
  using namespace fft;
  constexpr int NP = kPairs;
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ __align__(8) uint64_t s_full;
  const FftPlan& f = A.fy;
  // Rows of the cells in reach, in two pieces; the gap between them is zero.
  const uint32_t low = static_cast<uint32_t>(A.ylo) * NP * 16, bytes = static_cast<uint32_t>(A.ya) * NP * 16;
  const unsigned char* base = reinterpret_cast<const unsigned char*>(A.t1);
  auto issue = [&](int t) {
    const unsigned char* src = base + static_cast<size_t>(t) * bytes;
    mbar_arrive_expect_tx(&s_full, bytes);
    bulk_g2s(smem, src, low, &s_full);
    if (A.yhi) bulk_g2s(smem + static_cast<size_t>(A.my - A.yhi) * NP * 16, src + low, bytes - low, &s_full);
  };
  if (threadIdx.x == 0) {
    mbar_init(&s_full, 1);
    fence_mbar_init();
    if (static_cast<int>(blockIdx.x) < tiles) issue(blockIdx.x);
  }
  __syncthreads();
  ulonglong2* sh = reinterpret_cast<ulonglong2*>(smem);
  auto clear_gap = [&] {
    for (int it = threadIdx.x; it < (A.my - A.ya) * NP; it += blockDim.x) sh[A.ylo * NP + it] = make_ulonglong2(0, 0);
  };
  clear_gap();
  const int rl = f.r[f.nst - 1], hop = f.n / rl, row = A.ax * NP;
  int n = 0;
  for (int t = blockIdx.x; t < tiles; t += gridDim.x, ++n) {
    const bool ok = mbar_wait_bounded(&s_full, n & 1, A.status);
    if (!__syncthreads_and(ok)) {
      // Unwind: the copy in flight lands before the block exits.
      if (threadIdx.x == 0) mbar_wait_drain(&s_full, n & 1);
      return;
    }
    const int g = t / A.ax, cx = t - g * A.ax;
    ulonglong2* dst = reinterpret_cast<ulonglong2*>(A.t2) + static_cast<size_t>(g) * A.ny * row + cx * NP;
    auto in = [&](int e, int p) {
      const ulonglong2 v = sh[e * NP + p];
      return C2{v.x, v.y};
    };
    auto out = [&](int e, int p, int, C2 v) { sh[e * NP + p] = make_ulonglong2(v.re, v.im); };
    auto gout = [&](int e, int p, int u, C2 v) {
      // element e = g R + u; output index rev[g] + u hop, about the middle
      int j = __ldg(A.revy + e - u) + u * hop + A.sy;
      j -= j >= A.my ? A.my : 0;
      if (j < A.ny) dst[static_cast<uint32_t>(j * row + p)] = make_ulonglong2(v.re, v.im);
    };
    for (int s = 0; s + 1 < f.nst; ++s) {
      stage_any<NP>(f, s, A.twy, in, out);
      __syncthreads();
    }
    stage_any<NP>(f, f.nst - 1, A.twy, in, gout);
    __syncthreads();
    clear_gap();
    const long long next = t + static_cast<long long>(gridDim.x);
    if (threadIdx.x == 0 && next < tiles) {
      fence_proxy_async_smem();
      issue(static_cast<int>(next));
    }
  }
}

// Step 3: inverse real FFT along cx of the planes of a tile (one j): the
// hx + 1 inputs (real parts only at 0 and hx; zero from ax on) as one complex transform of
// length hx whose output m is (x[2 m], x[2 m + 1]); x rows leave through
// shared memory, divided by both axes' window transforms.
__global__ void __launch_bounds__(kFftMaxThreads) grid_fft_x_kernel(const GridArgs A, float* field, int zbeg, int nzc,
                                                                    int tiles, Moments* stats) {
  using namespace fft;
  constexpr int NP = kPairs;
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ __align__(8) uint64_t s_full;
  __shared__ Moments s_warp[kFftMaxThreads / 32];
  const FftPlan& f = A.fx;
  const uint32_t bytes = static_cast<uint32_t>(A.ax) * NP * 16;
  const unsigned char* base = reinterpret_cast<const unsigned char*>(A.t2);
  if (threadIdx.x == 0) {
    mbar_init(&s_full, 1);
    fence_mbar_init();
    if (static_cast<int>(blockIdx.x) < tiles) tile_issue(smem, &s_full, base + static_cast<size_t>(blockIdx.x) * bytes, bytes);
  }
  __syncthreads();
  int pitch = (A.nx + 2) / 2 * 2;  // even for the paired stores; half of it odd: no bank conflicts
  if (pitch / 2 % 2 == 0) pitch += 2;
  float* rows = reinterpret_cast<float*>(smem + static_cast<size_t>(A.hx + 1) * NP * 16);
  ulonglong2* sh = reinterpret_cast<ulonglong2*>(smem);
  const int half = f.n / 2;
  const int rl = f.r[f.nst - 1], hop = f.n / rl;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  const bool paired = (A.nx & 1) == 0 && (reinterpret_cast<uintptr_t>(field) & 7u) == 0;
  double s1[2] = {0.0, 0.0}, s2[2] = {0.0, 0.0}, shift = 0.0;
  int count = 0, n = 0;
  for (int t = blockIdx.x; t < tiles; t += gridDim.x, ++n) {
    const bool ok = mbar_wait_bounded(&s_full, n & 1, A.status);
    if (!__syncthreads_and(ok)) {
      if (threadIdx.x == 0) mbar_wait_drain(&s_full, n & 1);
      return;
    }
    const int g = t / A.ny, j = t - g * A.ny, z0 = g * kZT;
    for (int it = threadIdx.x; it < (half + 1) * NP; it += blockDim.x) {
      const int p = it & (NP - 1), k = it / NP;
      const ulonglong2 none = make_ulonglong2(0, 0);
      const ulonglong2 a = k < A.ax ? sh[k * NP + p] : none, b = f.n - k < A.ax ? sh[(f.n - k) * NP + p] : none;
      if (k == 0) {
        sh[p] = make_ulonglong2(add(a.x, b.x), sub(a.x, b.x));
      } else {
        // P = A_k / 2, Q = conj(A_{n-k}) / 2: (P + Q) + i e^{2 pi i k / mx} (P - Q)
        const C2 w = fft::root(A.twr + k);
        const C2 s = scale(C2{add(a.x, b.x), sub(a.y, b.y)}, dup(0.5f));
        const C2 u = cmul(scale(C2{sub(a.x, b.x), add(a.y, b.y)}, dup(0.5f)), w.re, w.im);
        const C2 z = add_i(s, u);
        sh[k * NP + p] = make_ulonglong2(z.re, z.im);
        // index n - k: the conjugate of s - i u
        if (2 * k != f.n) sh[(f.n - k) * NP + p] = make_ulonglong2(add(s.re, u.im), sub(u.re, s.im));
      }
    }
    auto in = [&](int e, int p) {
      const ulonglong2 v = sh[e * NP + p];
      return C2{v.x, v.y};
    };
    auto out = [&](int e, int p, int, C2 v) { sh[e * NP + p] = make_ulonglong2(v.re, v.im); };
    auto rout = [&](int e, int p, int u, C2 v) {
      int i = 2 * (__ldg(A.revx + e - u) + u * hop) + A.sx;
      i -= i >= A.mx ? A.mx : 0;
      if (i < A.nx) {
        *reinterpret_cast<float2*>(rows + 2 * p * pitch + i) = make_float2(lo(v.re), lo(v.im));
        *reinterpret_cast<float2*>(rows + (2 * p + 1) * pitch + i) = make_float2(hi(v.re), hi(v.im));
      }
    };
    for (int s = 0; s + 1 < f.nst; ++s) {
      __syncthreads();
      stage_any<NP>(f, s, A.twx, in, out);
    }
    __syncthreads();
    stage_any<NP>(f, f.nst - 1, A.twx, in, rout);
    __syncthreads();
    const long long next = t + static_cast<long long>(gridDim.x);
    if (threadIdx.x == 0 && next < tiles) {
      fence_proxy_async_smem();
      tile_issue(smem, &s_full, base + static_cast<size_t>(next) * bytes, bytes);
    }
    // Rows of x: one warp per plane at a time, two values per lane where the
    // field's rows are 8-byte aligned. The next tile's rows are written after
    // at least one more barrier.
    const float dy = __ldg(A.dcy + j);
    if (n == 0) shift = rows[0] * (__ldg(A.dcx) * dy);  // any value of the field's size
    auto take = [&](float v, int c) {
      const double d = static_cast<double>(v) - shift;
      s1[c] += d;
      s2[c] = ::fma(d, d, s2[c]);
    };
    for (int z = warp; z < kZT && z0 + z < nzc; z += warps) {
      float* dst = field + static_cast<size_t>(zbeg + z0 + z) * A.plane + static_cast<size_t>(j) * A.nx;
      const float* row = rows + z * pitch;
      if (paired) {
#pragma unroll 4
        for (int i = 2 * lane; i < A.nx; i += 64) {
          float2 v = *reinterpret_cast<const float2*>(row + i);
          const float2 d = __ldg(reinterpret_cast<const float2*>(A.dcx + i));
          v.x *= d.x * dy;
          v.y *= d.y * dy;
          *reinterpret_cast<float2*>(dst + i) = v;
          take(v.x, 0);
          take(v.y, 1);
          count += 2;
        }
      } else {
#pragma unroll 4
        for (int i = lane; i < A.nx; i += 32) {
          const float v = row[i] * (__ldg(A.dcx + i) * dy);
          dst[i] = v;
          take(v, 0);
          ++count;
        }
      }
    }
  }
  if (stats) {
    const Moments m = warp_moments(moments_from_shifted(count, shift, s1[0] + s1[1], s2[0] + s2[1]));
    if (lane == 0) s_warp[warp] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
      Moments b = s_warp[0];
      for (int w = 1; w < warps; ++w) b = moments_merge(b, s_warp[w]);
      stats[blockIdx.x] = b;
    }
  }
}

// ------------------------------------------------------------------- plans --
// Stages of an FFT of length n (primes up to 7): the fewest, with the
// smallest largest radix (registers) among those; descending radices.
// Branches that cannot be better are left out (all of them took up to 50 us for
// a length, on every call).
int least_stages(int n, int most) {
  int stages = 0;
  for (long long p = 1; p < n; p *= most) ++stages;
  return stages;
}
bool factor(int rest, int most, int depth, int* r, int* best, int* nbest) {
  if (rest == 1) {
    if (depth >= 2 && (!*nbest || depth < *nbest || (depth == *nbest && r[0] < best[0]))) {
      std::copy(r, r + depth, best);
      *nbest = depth;
    }
    return true;
  }
  if (depth == FftPlan::kMaxStages) return false;
  for (int k : {12, 10, 9, 8, 7, 6, 5, 4, 3, 2})
    if (k <= most && rest % k == 0) {
      r[depth] = k;
      if (*nbest && depth + 1 + least_stages(rest / k, k) + (r[0] < best[0] ? 0 : 1) > *nbest) continue;
      factor(rest / k, k, depth + 1, r, best, nbest);
    }
  return *nbest > 0;
}
}  // namespace

bool fft_plan(int n, FftPlan* f, int most_prime) {
  if (n < 4) return false;
  int rest = n;
  for (int k : {2, 3, 5, 7})
    while (k <= most_prime && rest % k == 0) rest /= k;
  if (rest != 1) return false;
  int r[FftPlan::kMaxStages], nst = 0;
  f->n = n;
  if (!factor(n, n, 0, r, f->r, &nst)) return false;
  f->nst = nst;
  int len = n;
  for (int s = 0; s < f->nst; ++s) {
    len /= f->r[s];
    f->m[s] = len;
    f->inv_m[s] = 1.0f / static_cast<float>(len);
  }
  return true;
}

int fft_least_stages(int n) { return std::max(2, least_stages(n, 12)); }

constexpr size_t kSmemMax = 224 * 1024;  // dynamic; the kernels keep a little static shared memory

namespace {

// Launch shape of a transform kernel: the block size that fills an SM's
// registers (kFftMaxThreads threads) with the least idle threads in the
// stages' rounds.
struct FftShape {
  int threads, blocks;
  size_t smem;
};
FftShape fft_shape(const FftPlan& f, size_t tile, size_t extra, long long tiles) {
  FftShape best{};
  best.smem = tile + extra;
  double best_cost = 1e30;
  for (int t = 64; t <= kFftMaxThreads; t += 32) {
    const int per_sm = static_cast<int>(std::min<size_t>(std::min<size_t>(kSmemMax / best.smem, kFftMaxThreads / t), 8));
    if (per_sm < 1) continue;
    double work = 0.0;
    for (int s = 0; s < f.nst; ++s) {
      const int items = f.n / f.r[s] * kPairs;
      work += static_cast<double>((items + t - 1) / t) * t / items;
    }
    const double cost = work / (per_sm * t);
    if (cost < best_cost) {
      best_cost = cost;
      best.threads = t;
      best.blocks = static_cast<int>(std::min<long long>(tiles, 148ll * per_sm));
    }
  }
  return best;
}

// Transform length for n outputs: at least 1.5 n, a multiple of 4, with the
// least length x (stages + 2) among lengths up to 15 % longer. `half`: the
// complex transform has half the length (the real axis).
int fft_length(int n, bool half, FftPlan* f) {
  const int lo = std::max(kMinM, static_cast<int>(std::ceil(kOversample * n)));
  int best = 0;
  double best_cost = 0.0;
  for (int m = (lo + 3) / 4 * 4; m <= std::max(lo * 23 / 20, lo + 16); m += 4) {
    FftPlan g;
    const int points = half ? m / 2 : m;
    if (best && static_cast<double>(m) * (fft_least_stages(points) + 2) >= best_cost) break;
    if (!fft_plan(points, &g)) continue;
    const double cost = static_cast<double>(m) * (g.nst + 2);
    if (!best || cost < best_cost) {
      best = m;
      best_cost = cost;
      *f = g;
    }
  }
  return best;
}

size_t align256(size_t v) { return (v + 255) / 256 * 256; }

size_t tile_y(const GridPlan& p) { return sizeof(float2) * kZT * static_cast<size_t>(p.my); }
size_t tile_x(const GridPlan& p) { return sizeof(float2) * kZT * static_cast<size_t>(p.mx / 2 + 1); }
size_t rows_x(const GridPlan& p) { return sizeof(float) * kZT * static_cast<size_t>(p.nx + 4); }

double window_beta(int n, int m) {
  // Shape parameter of the Kaiser-Bessel window for this oversampling
  // (Beatty, Nishimura & Pauly 2005), 2 % below: the least error measured
  // with FP32 weights at 1.5.
  const double sigma = static_cast<double>(m) / n;
  return 0.98 * 3.14159265358979323846 * kW * (1.0 - 0.5 / sigma);
}

}  // namespace

void grid_reach(const scarf_srm_params& p, const scarf_srm_setup& s, double reach[3]) {
  for (int c = 0; c < 3; ++c) {
    double q = 0.0;
    for (int r = 0; r < s.ndim; ++r) q += std::pow(s.m[3 * r + c] / static_cast<double>(p.cl[r]), 2);
    reach[c] = s.kc * std::sqrt(q) * p.ds / 6.28318530717958647692;
  }
}

bool grid_make_plan(const int n[3], int nh, size_t pass_bytes, const double reach[3], GridPlan* P) {
  GridPlan p{};
  if (nh <= 0 || nh > kGridMaxHarmonics || n[0] <= 0 || n[1] <= 0 || n[2] <= 0) return false;
  p.nh = nh;
  p.nx = n[0];
  // The second axis is transformed, the third summed exactly; a single plane
  // leaves (x, y) as x and the third.
  if (n[2] == 1) {
    p.ny = 1, p.nz = n[1], p.ax_y = 2, p.ax_z = 1;
  } else {
    p.ny = n[1], p.nz = n[2], p.ax_y = 1, p.ax_z = 2;
  }
  p.mx = fft_length(p.nx, true, &p.fx);
  if (!p.mx) return false;
  p.my = 1;
  if (p.ny > 1 && !(p.my = fft_length(p.ny, false, &p.fy))) return false;
  if ((p.ny > 1 && tile_y(p) > kSmemMax) || tile_x(p) + rows_x(p) > kSmemMax) return false;
  // Cells that the harmonics' windows reach, with a cell to spare for FP32
  // wavenumbers; all of them where the reach passes the half period.
  p.ax = p.mx / 2 + 1;
  p.ylo = p.my, p.yhi = 0;
  if (reach) {
    auto cells = [&](double turns, int m) { return turns < 0.5 ? static_cast<int>(turns * m + 0.5 * kW) + 3 : m; };
    p.ax = std::min(p.ax, cells(reach[0], p.mx));
    const int low = (cells(reach[p.ax_y], p.my) + kB - 1) / kB * kB;  // whole bins
    if (p.ny > 1 && 2 * low < p.my) p.ylo = p.yhi = low;
  }
  p.ya = p.ylo + p.yhi;
  p.nbx = (p.ax + kB - 1) / kB;
  p.nby = p.ny > 1 ? p.my / kB : 1;
  p.nkeys = (p.nbx + kSpan) * p.nby;
  p.nent = 2 * nh;
  const int nzp = (p.nz + 31) / 32 * 32;
  // Planes per pass: about pass_bytes of T1 and T2 and at most kGridEBytes of E,
  // in as few passes as that takes, of equal multiples of 32 planes (the last
  // may be shorter: 200 planes in two passes are 128 and 72).
  const size_t per_z = sizeof(float2) * static_cast<size_t>(p.ax) * (p.ya + (p.ny > 1 ? p.ny : 0));
  const long long cells_most = static_cast<long long>(1.3 * static_cast<double>(pass_bytes) / per_z);
  const long long e_most = static_cast<long long>(kGridEBytes / (sizeof(float2) * static_cast<size_t>(p.nent)));
  const long long most = std::max<long long>(32, std::min(cells_most, e_most));
  const long long want = (p.nz + most - 1) / most;
  p.zc = static_cast<int>(std::min<long long>((p.nz + 32 * want - 1) / (32 * want) * 32, nzp));
  // E for as many passes as fit its buffer.
  const size_t e_pass = sizeof(float2) * static_cast<size_t>(p.nent) * p.zc;
  const int passes = static_cast<int>(std::max<size_t>(1, kGridEBytes / e_pass));
  p.ez = static_cast<int>(std::min<long long>(static_cast<long long>(passes) * p.zc, (nzp + p.zc - 1) / p.zc * p.zc));
  // At most 9 visits of bins by a primary and 6 by a mirror entry.
  const long long visits = 15ll * nh;
  p.maxtasks = static_cast<int>(visits / kSparse + visits / kPart) + 1;
  p.maxslots = static_cast<int>(2 * (visits / kPart)) + 2;
  size_t off = 0;
  auto take = [&](size_t bytes) {
    const size_t at = off;
    off = align256(off + bytes);
    return at;
  };
  p.off_counts = take(sizeof(int) * (p.nkeys + 4));
  p.off_keys = take(sizeof(uint2) * p.nent);
  p.off_members = take(2 * sizeof(int) * p.nent + sizeof(int) * (p.nent / kDense + 1));
  p.off_par = take(sizeof(double4) * nh);
  p.off_w = take(sizeof(double2) * nh);
  p.off_bins = take(sizeof(int) * (p.nkeys + 2));
  p.off_weights = take(sizeof(float) * 2 * kSpan * kB * static_cast<size_t>(p.nent));
  p.off_e = take(sizeof(float2) * static_cast<size_t>(p.nent) * p.ez);
  p.off_t1 = take(sizeof(float2) * static_cast<size_t>(p.ax) * p.ya * p.zc);
  // T2 takes the place of the partial sums, which are in T1 by then; a single
  // gridded axis has no T2.
  const size_t partial = sizeof(float2) * static_cast<size_t>(p.maxslots) * kB * (p.ny > 1 ? kB : 1) * p.zc;
  const size_t t2 = p.ny > 1 ? sizeof(float2) * static_cast<size_t>(p.ax) * p.ny * p.zc : 0;
  p.off_partial = take(std::max(partial, t2));
  p.off_t2 = p.ny > 1 ? p.off_partial : p.off_t1;
  p.off_tasks = take(sizeof(int4) * (p.maxtasks + p.maxslots));
  p.off_dc = take(sizeof(float) * (p.nx + 2 + p.ny));
  p.off_tables = take(sizeof(float2) * (p.mx + p.my) + sizeof(int) * (p.mx + p.my));
  p.bytes = off;
  *P = p;
  return true;
}

bool grid_pays(const GridPlan& p, const TcPlan& tc) {
  const double cells = static_cast<double>(p.mx / 2) * p.my * p.nz, nh = p.nh;
  const double grid = 93.0 + 1.0e-5 * cells + nh * (0.0045 + (p.ny > 1 ? 3.5e-5 : 0.8e-5) * p.nz);
  const double waves = std::ceil(static_cast<double>(tc.bix) * tc.bjx * tc.bn / 148.0);
  const double flat = p.ny > 1 ? 0.0 : 3.0e-5 * static_cast<double>(p.nx) * p.nz;
  return grid < 50.0 + flat + waves * (19.0 + 0.042 * nh) + 6.0e-6 * nh * (tc.n1 + tc.n2 + tc.n3);
}

int grid_passes(const GridPlan& p) { return (p.nz + p.zc - 1) / p.zc; }
void grid_pass_planes(const GridPlan& p, int pass, int* z0, int* z1) {
  *z0 = pass * p.zc;
  *z1 = std::min(p.nz, *z0 + p.zc);
}
namespace {
// Step 3 of a pass: tiles past the last plane have nothing to store.
int x_tiles(const GridPlan& p, int planes) { return (planes + kZT - 1) / kZT * p.ny; }
FftShape x_shape(const GridPlan& p, int planes) { return fft_shape(p.fx, tile_x(p), rows_x(p), x_tiles(p, planes)); }
}  // namespace

long long grid_stat_records(const GridPlan& p) {  // one per block of every pass's step 3
  long long n = 0;
  for (int pass = 0; pass < grid_passes(p); ++pass) {
    int z0, z1;
    grid_pass_planes(p, pass, &z0, &z1);
    n += x_shape(p, z1 - z0).blocks;
  }
  return n;
}

namespace {
// Dynamic shared-memory limits, raised once per device context.
cudaError_t ensure_grid_attributes() {
  static std::atomic<unsigned long long> done[64];
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const unsigned long long ctx = current_context_id();
  if (dev >= 0 && dev < 64 && ctx != 0 && done[dev] == ctx) return cudaSuccess;
  const int most = static_cast<int>(kSmemMax);
  const int spread = static_cast<int>(sizeof(SpreadWarp) * kSpreadWarps);
  e = cudaFuncSetAttribute(grid_spread_kernel<kB>, cudaFuncAttributeMaxDynamicSharedMemorySize, spread);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(grid_spread_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, spread);
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(grid_fft_y_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(grid_fft_x_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
  if (e == cudaSuccess && dev >= 0 && dev < 64) done[dev] = ctx;
  return e;
}
}  // namespace

cudaError_t launch_grid_structured(const scarf_srm_setup& s, const int fs[3], float ds, const float* d_table,
                                   float* d_field, void* d_work, const GridPlan& p, int* d_status, cudaStream_t stream,
                                   StatRecord* d_stats, const std::function<cudaError_t(int)>& pass_done) {
  cudaError_t e = ensure_grid_attributes();
  if (e != cudaSuccess) return e;
  uint8_t* w = static_cast<uint8_t*>(d_work);
  GridArgs A{};
  A.fx = p.fx, A.fy = p.fy;
  A.mx = p.mx, A.my = p.my, A.hx = p.mx / 2;
  A.nx = p.nx, A.ny = p.ny, A.nz = p.nz;
  A.sx = p.nx / 4 * 2;  // even: outputs come in pairs
  A.sy = p.ny / 2;
  A.ax = p.ax, A.ylo = p.ylo, A.yhi = p.yhi, A.ya = p.ya;
  A.nbx = p.nbx, A.nby = p.nby, A.nkeys = p.nkeys;
  A.nent = p.nent, A.nh = p.nh;
  A.ez = p.ez;
  A.beta_x = window_beta(p.nx, p.mx);
  A.beta_y = window_beta(p.ny, p.my);
  A.inv_i0_x = 1.0 / std::cyl_bessel_i(0.0, A.beta_x);
  A.inv_i0_y = 1.0 / std::cyl_bessel_i(0.0, A.beta_y);
  for (int i = 0; i < 9; ++i) A.m[i] = s.m[i];
  for (int i = 0; i < 3; ++i) A.bar[i] = s.bar[i], A.fs[i] = fs[i];
  A.ds = ds;
  A.ax_y = p.ax_y, A.ax_z = p.ax_z;
  A.scaling = s.scaling;
  A.plane = static_cast<long long>(p.nx) * p.ny;
  A.table = d_table;
  A.status = d_status;
  A.counts = reinterpret_cast<int*>(w + p.off_counts);
  A.ntasks = A.counts + p.nkeys;
  A.keys = reinterpret_cast<uint2*>(w + p.off_keys);
  A.members = reinterpret_cast<int*>(w + p.off_members);
  A.place = A.members + p.nent;
  A.dense = A.place + p.nent;
  A.ranked = p.nh > kGridCountedHarmonics ? 1 : 0;
  A.par = reinterpret_cast<double4*>(w + p.off_par);
  A.w = reinterpret_cast<double2*>(w + p.off_w);
  A.bin_start = reinterpret_cast<int*>(w + p.off_bins);
  A.weights = reinterpret_cast<float*>(w + p.off_weights);
  A.e = reinterpret_cast<float2*>(w + p.off_e);
  A.t1 = reinterpret_cast<float2*>(w + p.off_t1);
  A.t2 = reinterpret_cast<float2*>(w + p.off_t2);
  A.partial = reinterpret_cast<float2*>(w + p.off_partial);
  A.tasks = reinterpret_cast<int4*>(w + p.off_tasks);
  A.multi = A.tasks + p.maxtasks;
  A.twx = reinterpret_cast<float2*>(w + p.off_tables);
  A.twr = A.twx + p.mx / 2;
  A.twy = A.twr + p.mx / 2;
  A.revx = reinterpret_cast<int*>(A.twy + p.my);
  A.revy = A.revx + p.mx;
  A.dcx = reinterpret_cast<float*>(w + p.off_dc);
  A.dcy = A.dcx + p.nx + 1;

  const long long items = static_cast<long long>(p.nh) + 2 * (p.mx + p.my) + p.nx + p.ny;
  // Entry counts and the task counters behind them.
  if ((e = cudaMemsetAsync(A.counts, 0, sizeof(int) * (p.nkeys + 4), stream)) != cudaSuccess) return e;
  grid_prep_kernel<<<static_cast<unsigned>((items + 127) / 128), 128, 0, stream>>>(A);
  grid_scan_kernel<<<1, kScanThreads, 0, stream>>>(A);
  const int nbins = p.nbx * p.nby;
  const int scatter = (p.nent + 255) / 256;
  grid_bins_kernel<<<scatter + (nbins + 7) / 8, 256, 0, stream>>>(A, scatter);
  if (A.ranked) grid_rank_kernel<<<148, kRankThreads, 0, stream>>>(A);
  const int task_blocks = std::min(p.maxtasks, 148 * 4);
  for (int pass = 0; pass < grid_passes(p); ++pass) {
    int z0, z1;
    grid_pass_planes(p, pass, &z0, &z1);
    const int zoff = z0 % p.ez;
    if (zoff == 0) {
      const int nze = (std::min(p.nz - z0, p.ez) + 31) / 32 * 32;
      grid_entry_kernel<<<(p.nent + 3) / 4, 128, 0, stream>>>(A, z0, nze, pass == 0);
    }
    const int planes = (z1 - z0 + 31) / 32 * 32;
    const dim3 gs(task_blocks + (nbins + kSpreadWarps - 1) / kSpreadWarps, planes / 32);
    const dim3 gp(std::min(p.maxslots, 148), planes / 32);
    if (p.ny > 1) {
      grid_spread_kernel<kB><<<gs, 32 * kSpreadWarps, sizeof(SpreadWarp) * kSpreadWarps, stream>>>(A, task_blocks, zoff, p.zc);
      grid_parts_kernel<kB><<<gp, 32 * kB * kB, 0, stream>>>(A, p.zc);
    } else {
      grid_spread_kernel<1><<<gs, 32 * kSpreadWarps, sizeof(SpreadWarp) * kSpreadWarps, stream>>>(A, task_blocks, zoff, p.zc);
      grid_parts_kernel<1><<<gp, 32 * kB, 0, stream>>>(A, p.zc);
    }
    const long long groups = (z1 - z0 + kZT - 1) / kZT;
    if (p.ny > 1) {
      const FftShape y = fft_shape(p.fy, tile_y(p), 0, groups * p.ax);
      grid_fft_y_kernel<<<y.blocks, y.threads, y.smem, stream>>>(A, static_cast<int>(groups * p.ax));
    }
    const FftShape x = x_shape(p, z1 - z0);
    grid_fft_x_kernel<<<x.blocks, x.threads, x.smem, stream>>>(A, d_field, z0, z1 - z0, x_tiles(p, z1 - z0),
                                                               d_stats);
    if (d_stats) d_stats += x.blocks;
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    if (pass_done && (e = pass_done(pass)) != cudaSuccess) return e;
  }
  return cudaGetLastError();
}

}  // namespace scarf
