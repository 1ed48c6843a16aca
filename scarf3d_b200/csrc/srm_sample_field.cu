// Harmonic sampling of one field (scarflib_srm.f90:731-778): the rejection
// tests on the GPU, the stream-order walk and the table rows on the host, as
// the batched sampler (srm_sampler.cu) does, arranged for the latency of a
// single call.
//
// Every thread tests four pairs at a time: its generator is jumped to its
// first draw by four small matrix tables (one matrix-vector product per byte
// of the position), so a field of 1e5 pairs occupies 128 blocks where chains of 256 pairs
// per thread left it on four (107 us of a 397-us call at 500 harmonics). Blocks
// keep the generator's state at each accepted or undecided pair, in stream
// order, and then draw those pairs and the three that follow them with all
// threads (candidate by candidate through fresh jumps took 40-160 us); a second
// kernel packs the blocks' candidates into page-locked host memory. Bound:
// the integer pipe (two generator steps of ~25 operations per pair) for
// large fields, launch and synchronisation latency for small ones.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <vector>

#include "srm_host.h"
#include "srm_kernels.h"
#include "yarn2.cuh"

namespace scarf {
namespace {

using namespace yarn2;

constexpr int kThreads = 256;
constexpr int kEach = 4;                       // pairs per thread and chunk
constexpr int kChunkPairs = kThreads * kEach;  // pairs per block and chunk
constexpr int kDigits = 4;                     // bytes of a thread's position (in units of kEach pairs)

struct Mat32 {
  uint32_t a, b, c, d;  // [[a, b], [c, d]] acting on (r0, r1)
};

// A candidate pair in stream order: the word that the host walk reads (pair
// index, kUndecided when the host has to decide it, kAboveCut when its u
// exceeds the cut-off and the harmonic is dropped), and the draws of the pairs
// q .. q + 3.
constexpr uint32_t kUndecided = 1u << 31, kAboveCut = 1u << 30;
constexpr double kMaxPairs = 1.0e9;                 // below 2^30
constexpr size_t kMaxStaging = size_t(64) << 20;  // page-locked bytes kept between calls
struct Candidate {
  uint32_t word, pad;
  float r[8];
};
struct Draws8 {
  float r[8];
};
struct Header {
  int total, overflow;
};

__device__ uint32_t g_field_pow[kPowWords];
__device__ Mat32 g_field_jump[kDigits][256];  // A^(2 kEach i 256^digit)
__device__ Mat32 g_field_chunk;               // A^(2 kChunkPairs)

struct ScanArgs {
  uint32_t r0, r1;  // generator state after seeding
  float kmin, kmax, kc, cnst, nu, margin;
  int ndim, acf;
  long long pairs;
  int chunks;  // per block
  int cap;     // candidates per block
  int* counts;
  int* overflow;
  Candidate* out;
  const uint32_t* reject;  // certain-reject thresholds (null: none)
};

__device__ __forceinline__ void apply(const Mat32& m, uint32_t& r0, uint32_t& r1) {
  const uint32_t x = sub_m(mulmod32(m.a, r0) + mulmod32(m.b, r1));
  r1 = sub_m(mulmod32(m.c, r0) + mulmod32(m.d, r1));
  r0 = x;
}

// 0 = certain reject, 1 = certain accept, 2 = undecided (as the batched
// scan decides: the host's operations, with a band for the spectrum's ulps).
__device__ __forceinline__ int classify(const ScanArgs& A, float r1, float r2) {
  const float u = __fadd_rn(__fmul_rn(r1, __fsub_rn(A.kmax, A.kmin)), A.kmin);
  const float fv = A.acf == 0 ? __fdiv_rn(1.0f, powf(__fadd_rn(1.0f, __fmul_rn(u, u)), A.nu))
                              : expf(__fmul_rn(-0.25f, __fmul_rn(u, u)));
  double srm = static_cast<double>(u) * static_cast<double>(fv);
  if (A.ndim == 3) srm = srm * static_cast<double>(u);
  const float d = static_cast<float>(srm * static_cast<double>(A.cnst));
  if (r2 < d * (1.0f - A.margin)) return 1;
  if (r2 >= d * (1.0f + A.margin)) return 0;
  return 2;
}

__global__ void __launch_bounds__(kThreads) field_scan_kernel(const ScanArgs A) {
  __shared__ uint32_t sp[kPowWords];
  __shared__ uint32_t s_thr[kRejectBins];
  __shared__ uint32_t s_r0[kChunkPairs], s_r1[kChunkPairs], s_q[kChunkPairs];  // s_q: pair in block << 2 | flag
  __shared__ int s_sum[kThreads / 32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int i = tid; i < kPowWords; i += kThreads) sp[i] = g_field_pow[i];
  if (A.reject)
    for (int i = tid; i < kRejectBins; i += kThreads) s_thr[i] = A.reject[i];
  const long long first = static_cast<long long>(blockIdx.x) * A.chunks * kChunkPairs;
  uint32_t r0 = A.r0, r1 = A.r1;
  const uint32_t at = static_cast<uint32_t>(first / kEach) + tid;
#pragma unroll
  for (int d = 0; d < kDigits; ++d) {
    const uint32_t i = (at >> (8 * d)) & 255u;
    if (i) apply(g_field_jump[d][i], r0, r1);
  }
  const Mat32 hop = g_field_chunk;
  Candidate* out = A.out + static_cast<size_t>(blockIdx.x) * A.cap;
  int base = 0;
  __syncthreads();
  for (int c = 0; c < A.chunks; ++c) {
    const long long q0 = first + static_cast<long long>(c) * kChunkPairs + tid * kEach;
    Gen g{r0, r1, sp};
    uint32_t st0[kEach], st1[kEach];
    int flag[kEach], mine = 0;
#pragma unroll
    for (int i = 0; i < kEach; ++i) {
      st0[i] = static_cast<uint32_t>(g.r0);
      st1[i] = static_cast<uint32_t>(g.r1);
      const uint32_t y1 = g.next(), y2 = g.next();
      flag[i] = 0;
      if (q0 + i < A.pairs && !(A.reject && y2 >= s_thr[y1 >> kRejectShift])) flag[i] = classify(A, to_u01(y1), to_u01(y2));
      mine += flag[i] ? 1 : 0;
    }
    int x = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) s_sum[warp] = x;
    __syncthreads();
    int before = x - mine, total = 0;
#pragma unroll
    for (int w = 0; w < kThreads / 32; ++w) {
      const int v = s_sum[w];
      before += w < warp ? v : 0;
      total += v;
    }
#pragma unroll
    for (int i = 0; i < kEach; ++i)
      if (flag[i]) {
        s_r0[before] = st0[i];
        s_r1[before] = st1[i];
        s_q[before] = static_cast<uint32_t>((c * kChunkPairs + tid * kEach + i) << 2 | flag[i]);
        ++before;
      }
    __syncthreads();
    for (int k = tid; k < total; k += kThreads) {
      if (base + k >= A.cap) break;
      Gen look{s_r0[k], s_r1[k], sp};
      Candidate e;
#pragma unroll
      for (int i = 0; i < 8; ++i) e.r[i] = to_u01(look.next());
      const float u = __fadd_rn(__fmul_rn(e.r[0], __fsub_rn(A.kmax, A.kmin)), A.kmin);
      e.word = static_cast<uint32_t>(first + (s_q[k] >> 2)) | ((s_q[k] & 3u) == 2u ? kUndecided : 0u) |
               (u > A.kc ? kAboveCut : 0u);
      e.pad = 0;
      out[base + k] = e;
    }
    base += total;
    apply(hop, r0, r1);
    // The next chunk writes s_sum and the candidates after its own barriers;
    // s_sum is rewritten before the first of them.
    __syncthreads();
  }
  if (tid == 0) {
    A.counts[blockIdx.x] = base;
    if (base > A.cap) *A.overflow = 1;
  }
}

// The blocks' candidates one after another in page-locked host memory (words
// and draws apart, so that the walk reads four bytes a candidate), and their
// number.
__global__ void __launch_bounds__(128) field_pack_kernel(const int* __restrict__ counts, int cap,
                                                         const Candidate* __restrict__ src, uint32_t* words,
                                                         Draws8* draws, int room, const int* overflow, Header* head) {
  __shared__ int s_sum[4];
  const int b = blockIdx.x, lane = threadIdx.x & 31;
  int before = 0;
  for (int i = threadIdx.x; i < b; i += 128) before += min(counts[i], cap);
  before = __reduce_add_sync(0xffffffffu, before);
  if (lane == 0) s_sum[threadIdx.x >> 5] = before;
  __syncthreads();
  before = s_sum[0] + s_sum[1] + s_sum[2] + s_sum[3];
  const int n = min(counts[b], cap), fit = max(0, min(n, room - before));
  src += static_cast<size_t>(b) * cap;
  for (int i = threadIdx.x; i < fit; i += 128) words[before + i] = src[i].word;
  float2* d = reinterpret_cast<float2*>(draws + before);
  for (int i = threadIdx.x; i < 4 * fit; i += 128) d[i] = *reinterpret_cast<const float2*>(&src[i >> 2].r[2 * (i & 3)]);
  if (b == static_cast<int>(gridDim.x) - 1 && threadIdx.x == 0) {
    head->total = before + n;
    head->overflow = (*overflow != 0 || before + n > room) ? 1 : 0;
  }
}

// ------------------------------------------------------------------- host --
struct Buf {
  void* p = nullptr;
  size_t bytes = 0;
  bool ensure(size_t need) {
    if (need <= bytes) return true;
    release();
    if (static_cast<cudaError_t>(device_alloc(&p, need)) != cudaSuccess) return false;
    bytes = need;
    return true;
  }
  void release() {
    device_free(p, bytes);
    p = nullptr;
    bytes = 0;
  }
};

// One per process, for the current device; guarded by `mu`.
struct FieldSampler {
  std::mutex mu;
  int device = -1;
  unsigned long long ctx = 0;
  Buf work;
  char* host = nullptr;  // page-locked: header, words, draws
  size_t host_bytes = 0;
  std::vector<uint32_t> kept;  // candidates that became harmonics
};
FieldSampler g_field;

Mat32 mat_mul(const Mat32& x, const Mat32& y) {
  auto mm = [](uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    return static_cast<uint32_t>((Yarn2::mulmod(a, b) + Yarn2::mulmod(c, d)) % Yarn2::kMod);
  };
  return Mat32{mm(x.a, y.a, x.b, y.c), mm(x.a, y.b, x.b, y.d), mm(x.c, y.a, x.d, y.c), mm(x.c, y.b, x.d, y.d)};
}

// The generator's tables in this module's device memory, once per device
// context (on every call when the context's id cannot be read).
bool ensure_tables(FieldSampler& S) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return false;
  const unsigned long long ctx = current_context_id();
  if (dev == S.device && ctx != 0 && ctx == S.ctx) return true;
  if (dev != S.device) S.work.release();
  static const std::vector<uint32_t> pw = device_pow_tables();
  static const std::vector<Mat32> jump = [] {
    std::vector<Mat32> t(kDigits * 256 + 1);
    const Mat32 one{static_cast<uint32_t>(Yarn2::kA1), static_cast<uint32_t>(Yarn2::kA2), 1u, 0u};
    Mat32 unit = one;  // A^(2 kEach), kEach = 4: three squarings
    for (int k = 0; k < 3; ++k) unit = mat_mul(unit, unit);
    for (int d = 0; d < kDigits; ++d) {
      Mat32 m{1u, 0u, 0u, 1u};
      for (int i = 0; i < 256; ++i) {
        t[d * 256 + i] = m;
        m = mat_mul(m, unit);
      }
      unit = m;  // A^(2 kEach 256^(d + 1))
    }
    t[kDigits * 256] = t[256 + 1];  // one chunk: 256 units
    return t;
  }();
  static_assert(2 * kEach == 8 && kThreads == 256, "the jump tables' unit and chunk");
  if (cudaMemcpyToSymbol(g_field_pow, pw.data(), sizeof(uint32_t) * pw.size()) != cudaSuccess ||
      cudaMemcpyToSymbol(g_field_jump, jump.data(), sizeof(Mat32) * kDigits * 256) != cudaSuccess ||
      cudaMemcpyToSymbol(g_field_chunk, &jump[kDigits * 256], sizeof(Mat32)) != cudaSuccess)
    return false;
  S.device = dev;
  S.ctx = ctx;
  return true;
}

}  // namespace

void release_field_sampler_memory() {
  std::lock_guard<std::mutex> lk(g_field.mu);
  g_field.work.release();
  if (g_field.host) cudaFreeHost(g_field.host);
  g_field.host = nullptr;
  g_field.host_bytes = 0;
}

namespace {
// One scan of `want` pairs and its walk; kMorePairs when they ran out.
constexpr int kMorePairs = -3;
int sample_pairs(const scarf_srm_params& p, const scarf_srm_setup& s, float* table, long long* pairs_used,
                 void* stream_handle, long long* uncertain, double acc, double want) {
  auto batched = [&] { return srm_sample_device(p, s, table, pairs_used, stream_handle, uncertain); };
  const cudaStream_t stream = static_cast<cudaStream_t>(stream_handle);
  if (want > kMaxPairs || device_sampler_pass_cap() > 0) return batched();
  const long long pairs = static_cast<long long>(want);
  std::unique_lock<std::mutex> lk(g_field.mu);
  FieldSampler& S = g_field;
  if (!ensure_tables(S)) return -2;
  const long long all_chunks = (pairs + kChunkPairs - 1) / kChunkPairs;
  const int chunks = static_cast<int>(std::max(1LL, (all_chunks + 148 * 6 - 1) / (148 * 6)));
  const int blocks = static_cast<int>((all_chunks + chunks - 1) / chunks);
  const double lambda = static_cast<double>(chunks) * kChunkPairs * std::min(1.0, acc);
  const int cap = static_cast<int>(std::ceil(1.25 * lambda + 6.0 * std::sqrt(lambda) + 8.0));
  const double expect = static_cast<double>(pairs) * std::min(1.0, acc);
  const int room = static_cast<int>(1.25 * expect + 8.0 * std::sqrt(expect) + 64.0);
  // Beyond a few million pairs the certain-reject thresholds (20 us of host
  // work) save more than they cost.
  const bool use_reject = pairs > (4ll << 20);
  const size_t off_reject = sizeof(int) * (static_cast<size_t>(blocks) + 4) / 16 * 16 + 16;
  const size_t off_out = off_reject + sizeof(uint32_t) * kRejectBins;
  const size_t off_draws = 64 + sizeof(uint32_t) * static_cast<size_t>((room + 15) / 16 * 16);
  const size_t host_need = off_draws + sizeof(Draws8) * static_cast<size_t>(room);
  if (host_need > kMaxStaging) {
    lk.unlock();
    return batched();
  }
  if (!S.work.ensure(off_out + sizeof(Candidate) * static_cast<size_t>(blocks) * cap)) return -2;
  if (S.host_bytes < host_need) {
    if (S.host) cudaFreeHost(S.host);
    S.host = nullptr;
    S.host_bytes = 0;
    void* h = nullptr;
    const size_t bytes = (host_need + (size_t(1) << 20) - 1) >> 20 << 20;  // whole megabytes: few reallocations
    if (cudaHostAlloc(&h, bytes, cudaHostAllocPortable | cudaHostAllocMapped) != cudaSuccess) return -2;
    S.host = static_cast<char*>(h);
    S.host_bytes = bytes;
  }
  void* dev_host = nullptr;
  if (cudaHostGetDevicePointer(&dev_host, S.host, 0) != cudaSuccess) return -2;
  char* w = static_cast<char*>(S.work.p);
  Yarn2 g;
  g.seed(p.seed);
  ScanArgs A{};
  A.r0 = static_cast<uint32_t>(g.r0);
  A.r1 = static_cast<uint32_t>(g.r1);
  A.kmin = s.kmin;
  A.kmax = s.kmax;
  A.kc = s.kc;
  A.cnst = s.cnst;
  A.nu = s.nu;
  A.margin = kSamplerMargin;
  A.ndim = s.ndim;
  A.acf = p.acf;
  A.pairs = pairs;
  A.chunks = chunks;
  A.cap = cap;
  A.overflow = reinterpret_cast<int*>(w);
  A.counts = A.overflow + 4;
  A.out = reinterpret_cast<Candidate*>(w + off_out);
  uint32_t reject[kRejectBins];
  if (use_reject) {
    sampler_reject_thresholds(s, p.acf, A.margin, reject);
    if (cudaMemcpyAsync(w + off_reject, reject, sizeof(reject), cudaMemcpyHostToDevice, stream) != cudaSuccess)
      return -2;
    A.reject = reinterpret_cast<const uint32_t*>(w + off_reject);
  }
  if (cudaMemsetAsync(A.overflow, 0, sizeof(int), stream) != cudaSuccess) return -2;
  field_scan_kernel<<<blocks, kThreads, 0, stream>>>(A);
  char* dh = static_cast<char*>(dev_host);
  field_pack_kernel<<<blocks, 128, 0, stream>>>(A.counts, cap, A.out, reinterpret_cast<uint32_t*>(dh + 64),
                                                reinterpret_cast<Draws8*>(dh + off_draws), room, A.overflow,
                                                reinterpret_cast<Header*>(dh));
  if (cudaGetLastError() != cudaSuccess || cudaStreamSynchronize(stream) != cudaSuccess) return -2;
  const Header head = *reinterpret_cast<const Header*>(S.host);
  if (head.overflow) {
    lk.unlock();
    return batched();
  }
  const uint32_t* words = reinterpret_cast<const uint32_t*>(S.host + 64);
  const Draws8* draws = reinterpret_cast<const Draws8*>(S.host + off_draws);
  if (S.kept.size() < static_cast<size_t>(p.nharm)) S.kept.resize(p.nharm);
  uint32_t* kept_at = S.kept.data();
  // The walk, in stream order exactly as the serial loop consumes pairs:
  // reject until an accepted pair, then one pair of angles, then (for a kept
  // harmonic) two pairs for a and b. Bound: mispredicted branches. 10 000
  // harmonics of one pair in 20 take 48 us in one loop without a branch on the
  // cut, 67 in a loop over candidates inside one over harmonics with one.
  long long open = 0;
  uint32_t pos = 0;
  int kept = 0, l = 0;
  const int total = head.total, nharm = p.nharm;
  for (int ei = 0; ei < total && l < nharm; ++ei) {
    const uint32_t w = words[ei], q = w & (kAboveCut - 1);
    if (q < pos) continue;
    if (w & kUndecided) {
      ++open;
      if (!sampler_host_accept(s, p.acf, draws[ei].r[0], draws[ei].r[1])) continue;
    }
    const uint32_t keep = w & kAboveCut ? 0u : 1u;
    kept_at[kept] = static_cast<uint32_t>(ei);
    kept += static_cast<int>(keep);
    pos = q + 2 + 2 * keep;
    ++l;
  }
  if (l < nharm) return kMorePairs;
  // Table rows (host libm, ~85 ns each) on the worker pool. Rows started while
  // the walk runs, by workers waiting for it, measured slower: the waiting
  // threads take the processor time of the others.
  constexpr int kRowBlock = 128;
  parallel_tasks((kept + kRowBlock - 1) / kRowBlock, host_threads(), [&](int b) {
    const int r1 = std::min(kept, (b + 1) * kRowBlock);
    for (int r = b * kRowBlock; r < r1; ++r) {
      const float* d = draws[kept_at[r]].r;
      sampler_row(d[0] * (s.kmax - s.kmin) + s.kmin, d + 2, s.ndim, p.cl, table + 5 * static_cast<size_t>(r));
    }
  });
  if (pairs_used) *pairs_used = pos;
  if (uncertain) *uncertain = open;
  return kept;
}

}  // namespace

int srm_sample_field(const scarf_srm_params& p, const scarf_srm_setup& s, float* table, long long* pairs_used,
                     void* stream_handle, long long* uncertain) {
  const double acc = acceptance_rate(s);
  if (acc < kMinAcceptance) return -1;
  // Enough pairs for every harmonic at the expected acceptance, with the
  // batched sampler's margin. Few harmonics of a rare acceptance now and then
  // need more: then twice as many are scanned, from the first (the batched
  // sampler's passes after a scan in vain took longer than they alone: 100
  // harmonics of one pair in 1 100 318 -> 360 us, 67 so). Fields of very many
  // pairs, or that a test caps, take the batched sampler's chained passes.
  double want = p.nharm * (1.0 / acc + 3.0) * 1.1 + 4096.0;
  for (;; want *= 2.0) {
    const int rc = sample_pairs(p, s, table, pairs_used, stream_handle, uncertain, acc, want);
    if (rc != kMorePairs) return rc;
  }
}

}  // namespace scarf
