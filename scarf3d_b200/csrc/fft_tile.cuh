// Inverse FFTs of a tile of transforms in shared memory: two neighbouring
// transforms travel in the halves of packed FP32 registers, so that index
// arithmetic, twiddle loads and instruction issue are shared by both.
//
// A tile holds NP pairs of complex transforms, element e of pair p at
// [e * NP + p] as {re0, re1, im0, im1} (16 bytes). Stages are decimation in
// frequency, in place, with the radices of an FftPlan; outputs come in
// digit-reversed order (fft_output_order).
#pragma once

#include <cstdint>

#include <cuda_runtime.h>

#include "common.cuh"
#include "srm_kernels.h"

namespace scarf {

namespace fft {

// Asynchronous copies of a thread's own elements into shared memory.
__device__ __forceinline__ void cp_async8(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// A pair of FP32 values in one 64-bit register and sm_100's packed operations.
using f2 = unsigned long long;
__device__ __forceinline__ f2 pack(float lo, float hi) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ f2 dup(float v) { return pack(v, v); }
__device__ __forceinline__ float lo(f2 v) { return __uint_as_float(static_cast<uint32_t>(v)); }
__device__ __forceinline__ float hi(f2 v) { return __uint_as_float(static_cast<uint32_t>(v >> 32)); }
__device__ __forceinline__ f2 add(f2 a, f2 b) {
  f2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 sub(f2 a, f2 b) {
  f2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 mul(f2 a, f2 b) {
  f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 fma(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

// Two complex values (one of each transform of a pair).
struct C2 {
  f2 re, im;
};
__device__ __forceinline__ C2 operator+(C2 a, C2 b) { return C2{add(a.re, b.re), add(a.im, b.im)}; }
__device__ __forceinline__ C2 operator-(C2 a, C2 b) { return C2{sub(a.re, b.re), sub(a.im, b.im)}; }
// a + i b, a - i b
__device__ __forceinline__ C2 add_i(C2 a, C2 b) { return C2{sub(a.re, b.im), add(a.im, b.re)}; }
__device__ __forceinline__ C2 sub_i(C2 a, C2 b) { return C2{add(a.re, b.im), sub(a.im, b.re)}; }
// (wr + i wi) a, each of wr, wi in both halves
__device__ __forceinline__ C2 cmul(C2 a, f2 wr, f2 wi) {
  return C2{sub(mul(a.re, wr), mul(a.im, wi)), add(mul(a.re, wi), mul(a.im, wr))};
}
__device__ __forceinline__ C2 scale(C2 a, f2 s) { return C2{mul(a.re, s), mul(a.im, s)}; }

// A complex table entry in both halves.
__device__ __forceinline__ C2 root(const float2* t) {
  const float2 w = __ldg(t);
  return C2{dup(w.x), dup(w.y)};
}

// Twiddles of the composite radices, evaluated by the compiler.
constexpr double cos_series(double x) {
  double t = 1.0, s = 1.0;
  for (int k = 1; k < 16; ++k) {
    t *= -x * x / ((2 * k - 1) * (2 * k));
    s += t;
  }
  return s;
}
constexpr double sin_series(double x) {
  double t = x, s = x;
  for (int k = 1; k < 16; ++k) {
    t *= -x * x / ((2 * k) * (2 * k + 1));
    s += t;
  }
  return s;
}
template <int R>
struct Roots {  // e^{2 pi i k / R}
  float c[R], s[R];
  constexpr Roots() : c(), s() {
    for (int k = 0; k < R; ++k) {
      // angle in [-pi, pi]
      const double x = 6.28318530717958647692 * (2 * k <= R ? k : k - R) / R;
      c[k] = static_cast<float>(cos_series(x));
      s[k] = static_cast<float>(sin_series(x));
    }
  }
};

// Inverse (e^{+i}) DFT of R values in registers, natural order.
template <int R>
struct Dft;
template <>
struct Dft<2> {
  static __device__ __forceinline__ void run(C2* v) {
    const C2 t = v[0];
    v[0] = t + v[1];
    v[1] = t - v[1];
  }
};
template <>
struct Dft<3> {
  static __device__ __forceinline__ void run(C2* v) {
    constexpr float k = 0.86602540378443864676f;
    const C2 t = v[1] + v[2], d = scale(v[1] - v[2], dup(k));
    const C2 m = C2{fma(t.re, dup(-0.5f), v[0].re), fma(t.im, dup(-0.5f), v[0].im)};
    v[0] = v[0] + t;
    v[1] = add_i(m, d);
    v[2] = sub_i(m, d);
  }
};
template <>
struct Dft<4> {
  static __device__ __forceinline__ void run(C2* v) {
    const C2 a = v[0] + v[2], b = v[0] - v[2], c = v[1] + v[3], d = v[1] - v[3];
    v[0] = a + c;
    v[1] = add_i(b, d);
    v[2] = a - c;
    v[3] = sub_i(b, d);
  }
};
template <>
struct Dft<5> {
  static __device__ __forceinline__ void run(C2* v) {
    constexpr float c1 = 0.30901699437494742410f, c2 = -0.80901699437494742410f;  // cos(2 pi / 5), cos(4 pi / 5)
    constexpr float s1 = 0.95105651629515357212f, s2 = 0.58778525229247312917f;   // sin
    const C2 a = v[1] + v[4], b = v[2] + v[3], c = v[1] - v[4], d = v[2] - v[3];
    const C2 m1 = C2{fma(b.re, dup(c2), fma(a.re, dup(c1), v[0].re)), fma(b.im, dup(c2), fma(a.im, dup(c1), v[0].im))};
    const C2 m2 = C2{fma(b.re, dup(c1), fma(a.re, dup(c2), v[0].re)), fma(b.im, dup(c1), fma(a.im, dup(c2), v[0].im))};
    const C2 n1 = C2{fma(d.re, dup(s2), mul(c.re, dup(s1))), fma(d.im, dup(s2), mul(c.im, dup(s1)))};
    const C2 n2 = C2{fma(d.re, dup(-s1), mul(c.re, dup(s2))), fma(d.im, dup(-s1), mul(c.im, dup(s2)))};
    v[0] = v[0] + (a + b);
    v[1] = add_i(m1, n1);
    v[2] = add_i(m2, n2);
    v[3] = sub_i(m2, n2);
    v[4] = sub_i(m1, n1);
  }
};
template <>
struct Dft<7> {
  static __device__ __forceinline__ void run(C2* v) {
    // cos and sin of 2 pi k / 7, k = 1, 2, 3
    constexpr float c[3] = {0.62348980185873353053f, -0.22252093395631440429f, -0.90096886790241912624f};
    constexpr float s[3] = {0.78183148246802980871f, 0.97492791218182360702f, 0.43388373911755812048f};
    const C2 p[3] = {v[1] + v[6], v[2] + v[5], v[3] + v[4]}, d[3] = {v[1] - v[6], v[2] - v[5], v[3] - v[4]};
    const C2 x0 = v[0];
    v[0] = v[0] + (p[0] + (p[1] + p[2]));
#pragma unroll
    for (int k = 1; k <= 3; ++k) {
      C2 m = x0, n = C2{0ull, 0ull};
#pragma unroll
      for (int t = 1; t <= 3; ++t) {
        const int e = k * t % 7, at = (e <= 3 ? e : 7 - e) - 1;
        const f2 cc = dup(c[at]), ss = dup(e <= 3 ? s[at] : -s[at]);
        m = C2{fma(p[t - 1].re, cc, m.re), fma(p[t - 1].im, cc, m.im)};
        n = t == 1 ? scale(d[0], ss) : C2{fma(d[t - 1].re, ss, n.re), fma(d[t - 1].im, ss, n.im)};
      }
      v[k] = add_i(m, n);
      v[7 - k] = sub_i(m, n);
    }
  }
};
template <>
struct Dft<8> {
  static __device__ __forceinline__ void run(C2* v) {
    constexpr float r = 0.70710678118654752440f;
    C2 e[4] = {v[0], v[2], v[4], v[6]}, o[4] = {v[1], v[3], v[5], v[7]};
    Dft<4>::run(e);
    Dft<4>::run(o);
    // o[1] e^{i pi/4}; for o[3] e^{3 i pi/4}: (-p, q)
    const C2 w1 = C2{mul(sub(o[1].re, o[1].im), dup(r)), mul(add(o[1].re, o[1].im), dup(r))};
    const f2 p = mul(add(o[3].re, o[3].im), dup(r)), q = mul(sub(o[3].re, o[3].im), dup(r));
    v[0] = e[0] + o[0];
    v[4] = e[0] - o[0];
    v[1] = e[1] + w1;
    v[5] = e[1] - w1;
    v[2] = add_i(e[2], o[2]);
    v[6] = sub_i(e[2], o[2]);
    v[3] = C2{sub(e[3].re, p), add(e[3].im, q)};
    v[7] = C2{add(e[3].re, p), sub(e[3].im, q)};
  }
};
// R = A B: A-point DFTs over every B-th value, twiddles, B-point DFTs.
template <int A, int B>
struct DftComposite {
  static __device__ __forceinline__ void run(C2* v) {
    constexpr int R = A * B;
    constexpr Roots<R> w{};
    C2 y[B][A];
#pragma unroll
    for (int b = 0; b < B; ++b) {
#pragma unroll
      for (int a = 0; a < A; ++a) y[b][a] = v[B * a + b];
      Dft<A>::run(y[b]);
      if (b > 0) {
#pragma unroll
        for (int k = 1; k < A; ++k) y[b][k] = cmul(y[b][k], dup(w.c[b * k % R]), dup(w.s[b * k % R]));
      }
    }
#pragma unroll
    for (int k = 0; k < A; ++k) {
      C2 t[B];
#pragma unroll
      for (int b = 0; b < B; ++b) t[b] = y[b][k];
      Dft<B>::run(t);
#pragma unroll
      for (int b = 0; b < B; ++b) v[k + A * b] = t[b];
    }
  }
};
template <>
struct Dft<6> : DftComposite<2, 3> {};
template <>
struct Dft<9> : DftComposite<3, 3> {};
template <>
struct Dft<10> : DftComposite<2, 5> {};
template <>
struct Dft<12> : DftComposite<4, 3> {};

// One stage of radix R by the whole block: reads through in(e, p), writes
// through out(e, p, t, v) where t is the butterfly's output number. In place
// when both address the tile: a butterfly writes where it read. tw: the
// plan's twiddles (twiddle_entry); neighbouring
// butterflies read neighbouring entries (one table of e^{2 pi i k / n} read
// with a stride took up to eight cache lines per load, and the load unit was
// what bounded the stages).
template <int R, int NP, class In, class Out>
__device__ __forceinline__ void stage(const FftPlan& f, int s, const float2* __restrict__ tw, In in, Out out) {
  const int m = f.m[s];
  const int len = m * R;
  const float inv_m = f.inv_m[s];
  for (int it = threadIdx.x; it < f.n / R * NP; it += blockDim.x) {
    const int p = it & (NP - 1), g = it / NP;
    const int blk = static_cast<int>((static_cast<float>(g) + 0.5f) * inv_m);
    const int q = g - blk * m;
    const int base = blk * len + q;
    C2 v[R];
#pragma unroll
    for (int t = 0; t < R; ++t) v[t] = in(base + t * m, p);
    Dft<R>::run(v);
    if (m > 1) {
      // The stages before this one have n - len entries in all.
      const float2* w = tw + (f.n - len) + q;
#pragma unroll
      for (int t = 1; t < R; ++t, w += m) {
        const C2 x = root(w);
        v[t] = cmul(v[t], x.re, x.im);
      }
    }
#pragma unroll
    for (int t = 0; t < R; ++t) out(base + t * m, p, t, v[t]);
  }
}
// The last stage forwards, a product with hat[position] and the first stage
// backwards (e^{-i}) in registers: a butterfly of the last stage holds what its
// inverse needs. first(base, p, v, y) sees the butterfly's first value before
// the product and may change it after.
template <int R, int NP, class In, class Out, class First>
__device__ __forceinline__ void product(const FftPlan& f, const float2* __restrict__ hat, In in, Out out, First first) {
  for (int it = threadIdx.x; it < f.n / R * NP; it += blockDim.x) {
    const int p = it & (NP - 1), base = it / NP * R;
    C2 v[R];
#pragma unroll
    for (int t = 0; t < R; ++t) v[t] = in(base + t, p);
    Dft<R>::run(v);
#pragma unroll
    for (int t = 0; t < R; ++t) {
      const C2 x = root(hat + base + t);
      C2 y = cmul(v[t], x.re, x.im);
      if (t == 0) first(base, p, v[0], y);
      v[t] = C2{y.im, y.re};  // the e^{-i} transform is the e^{+i} one with the parts exchanged
    }
    Dft<R>::run(v);
#pragma unroll
    for (int t = 0; t < R; ++t) out(base + t, p, t, C2{v[t].im, v[t].re});
  }
}
// A stage of the e^{-i} transform by decimation in time: stage s undone.
template <int R, int NP, class In, class Out>
__device__ __forceinline__ void back(const FftPlan& f, int s, const float2* __restrict__ tw, In in, Out out) {
  const int m = f.m[s], len = m * R;
  const float inv_m = f.inv_m[s];
  for (int it = threadIdx.x; it < f.n / R * NP; it += blockDim.x) {
    const int p = it & (NP - 1), g = it / NP;
    const int blk = static_cast<int>((static_cast<float>(g) + 0.5f) * inv_m);
    const int q = g - blk * m, base = blk * len + q;
    C2 v[R];
#pragma unroll
    for (int t = 0; t < R; ++t) {
      const C2 x = in(base + t * m, p);
      v[t] = C2{x.im, x.re};
    }
    const float2* w = tw + (f.n - len) + q;
#pragma unroll
    for (int t = 1; t < R; ++t, w += m) {
      // conj(w) x with the parts exchanged is w times the exchanged x
      const C2 x = root(w);
      v[t] = cmul(v[t], x.re, x.im);
    }
    Dft<R>::run(v);
#pragma unroll
    for (int t = 0; t < R; ++t) out(base + t * m, p, t, C2{v[t].im, v[t].re});
  }
}
#define SCARF_FFT_RADICES(CALL, r) \
  switch (r) {                     \
    case 12: CALL(12); break;      \
    case 10: CALL(10); break;      \
    case 9: CALL(9); break;        \
    case 8: CALL(8); break;        \
    case 7: CALL(7); break;        \
    case 6: CALL(6); break;        \
    case 5: CALL(5); break;        \
    case 4: CALL(4); break;        \
    case 3: CALL(3); break;        \
    default: CALL(2); break;       \
  }
template <int NP, class In, class Out>
__device__ __forceinline__ void stage_any(const FftPlan& f, int s, const float2* tw, In in, Out out) {
#define SCARF_FFT_CALL(R) stage<R, NP>(f, s, tw, in, out)
  SCARF_FFT_RADICES(SCARF_FFT_CALL, f.r[s])
#undef SCARF_FFT_CALL
}
template <int NP, class In, class Out, class First>
__device__ __forceinline__ void product_any(const FftPlan& f, const float2* hat, In in, Out out, First first) {
#define SCARF_FFT_CALL(R) product<R, NP>(f, hat, in, out, first)
  SCARF_FFT_RADICES(SCARF_FFT_CALL, f.r[f.nst - 1])
#undef SCARF_FFT_CALL
}
template <int NP, class In, class Out>
__device__ __forceinline__ void back_any(const FftPlan& f, int s, const float2* tw, In in, Out out) {
#define SCARF_FFT_CALL(R) back<R, NP>(f, s, tw, in, out)
  SCARF_FFT_RADICES(SCARF_FFT_CALL, f.r[s])
#undef SCARF_FFT_CALL
}

// Twiddle i < n of a plan: for each stage, [t - 1][q] for t = 1 .. r - 1 and
// q < m, e^{2 pi i q t / (r m)}; returns q t / (r m) (turns).
__device__ __forceinline__ double twiddle_entry(const FftPlan& f, int i) {
  int len = f.n;
  for (int s = 0; s < f.nst; ++s) {
    const int count = len - f.m[s];
    if (i < count) {
      const int t = i / f.m[s], q = i - t * f.m[s];
      return static_cast<double>(q * (t + 1)) / len;
    }
    i -= count;
    len = f.m[s];
  }
  return 0.0;
}

// Butterfly g of the last stage holds elements g R .. g R + R - 1; the index
// of its first output (the others follow at n / R).
__device__ __forceinline__ int output_order(const FftPlan& f, int g) {
  int k = 0, w = 1, pos = g * f.r[f.nst - 1], span = f.n;
  for (int s = 0; s + 1 < f.nst; ++s) {
    span /= f.r[s];
    const int d = pos / span;
    pos -= d * span;
    k += d * w;
    w *= f.r[s];
  }
  return k;
}

}  // namespace fft
}  // namespace scarf
