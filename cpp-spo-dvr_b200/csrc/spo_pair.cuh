// Two FP32 lines at once: packed arithmetic (add, mul, fma .f32x2: one instruction for two independent FP32
// operations, each rounded as the scalar one) and the register DFT of spo_regfft.cuh on pairs of lines. The FP32
// pipe of the B200 takes a packed instruction in two cycles, so it does no more operations per cycle than with
// scalar ones (126 against 118 per SM and cycle measured, of 128), but a kernel bound by its instruction issue
// needs half as many.
#pragma once

#include "spo_regfft.cuh"

namespace spo {

#ifdef __CUDACC__

struct F2 {  // two FP32 values (lane 0 in the low word)
  unsigned long long v;
};
__device__ __forceinline__ F2 f2(float a, float b) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ F2 f2(float a) { return f2(a, a); }
__device__ __forceinline__ void f2_split(F2 a, float& x, float& y) { asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a.v)); }
__device__ __forceinline__ F2 operator+(F2 a, F2 b) {
  F2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 operator*(F2 a, F2 b) {
  F2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}
// Negated as floats: an operand modifier of the next instruction where it has one, else two operations; a 64-bit exclusive
// or is two of the integer pipe's always (configuration 3: Z 1.54 -> 1.49 ms, r 1.51 -> 1.48, xy 1.75 -> 1.71).
__device__ __forceinline__ F2 operator-(F2 a) {
  float x, y;
  f2_split(a, x, y);
  return f2(-x, -y);
}
// a - b as a + (-1) b: one rounding, the same result
__device__ __forceinline__ F2 operator-(F2 a, F2 b) { return fma2(b, f2(-1.0f), a); }

struct C2 {  // two complex values
  F2 x, y;
};
__device__ __forceinline__ C2 c2(F2 x, F2 y) { return C2{x, y}; }
__device__ __forceinline__ C2 c2(float2 a, float2 b) { return C2{f2(a.x, b.x), f2(a.y, b.y)}; }
__device__ __forceinline__ void c2_split(C2 v, float2& a, float2& b) {
  f2_split(v.x, a.x, b.x);
  f2_split(v.y, a.y, b.y);
}
__device__ __forceinline__ C2 cadd(C2 a, C2 b) { return c2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ C2 csub(C2 a, C2 b) { return c2(a.x - b.x, a.y - b.y); }
// a + S i b and a - S i b
template <int S>
__device__ __forceinline__ C2 cadd_i(C2 a, C2 b) {
  return S > 0 ? c2(a.x - b.y, a.y + b.x) : c2(a.x + b.y, a.y - b.x);
}

// The operations of cmul2 and cmul_comp on both lines; the constants w + wl may differ between them.
__device__ __forceinline__ C2 cmul2(C2 a, C2 w, C2 wl) {
  const F2 n = -a.y;
  const F2 cr = fma2(a.x, wl.x, n * wl.y);
  const F2 ci = fma2(a.x, wl.y, a.y * wl.x);
  return c2(fma2(a.x, w.x, fma2(n, w.y, cr)), fma2(a.x, w.y, fma2(a.y, w.x, ci)));
}
// a times the conjugate of w + wl: the same operations on (w.x, -w.y), one value negated instead of three.
__device__ __forceinline__ C2 cmul2_conj(C2 a, C2 w, C2 wl) {
  const F2 n = -a.x;
  const F2 cr = fma2(a.x, wl.x, a.y * wl.y);
  const F2 ci = fma2(n, wl.y, a.y * wl.x);
  return c2(fma2(a.x, w.x, fma2(a.y, w.y, cr)), fma2(n, w.y, fma2(a.y, w.x, ci)));
}
// The same for one constant of both lines (the negated ones come with it, so that no value is negated).
__device__ __forceinline__ C2 cmul2k(C2 a, float wx, float wy, float lx, float ly) {
  const F2 cr = fma2(a.x, f2(lx), a.y * f2(-ly));
  const F2 ci = fma2(a.x, f2(ly), a.y * f2(lx));
  return c2(fma2(a.x, f2(wx), fma2(a.y, f2(-wy), cr)), fma2(a.x, f2(wy), fma2(a.y, f2(wx), ci)));
}
__device__ __forceinline__ F2 dot2_comp(F2 a, F2 b, F2 c, F2 d, F2 tl) {
  const F2 p1 = a * b, e1 = fma2(a, b, -p1);
  const F2 p2 = c * d, e2 = fma2(c, d, -p2);
  const F2 s = p1 + p2, bb = s - p1;
  const F2 es = (p1 - (s - bb)) + (p2 - bb);
  return s + ((es + e1) + (e2 + tl));
}
__device__ __forceinline__ C2 cmul_comp(C2 a, C2 w, C2 wl) {
  const F2 n = -a.y;
  return c2(dot2_comp(a.x, w.x, n, w.y, fma2(a.x, wl.x, n * wl.y)), dot2_comp(a.x, w.y, a.y, w.x, fma2(a.x, wl.y, a.y * wl.x)));
}
// fmul_parts on both lines, one factor s (1 + g) for both: scale and low parts as there.
__device__ __forceinline__ C2 fmul_parts(C2 x, float2 g, float2 gl, float2 sc) {
  const C2 z = cadd(x, cmul2k(x, g.x, g.y, gl.x, gl.y));
  return c2(fma2(z.x, f2(sc.x), z.x * f2(sc.y)), fma2(z.y, f2(sc.x), z.y * f2(sc.y)));
}

template <long K, long N, int S>
__device__ __forceinline__ C2 twiddle_mul2(C2 a) {
  constexpr long k = ((K % N) + N) % N;
  if constexpr (k == 0) {
    return a;
  } else if constexpr (4 * k == N) {
    return S > 0 ? c2(-a.y, a.x) : c2(a.y, -a.x);
  } else if constexpr (2 * k == N) {
    return c2(-a.x, -a.y);
  } else if constexpr (4 * k == 3 * N) {
    return S > 0 ? c2(a.y, -a.x) : c2(-a.y, a.x);
  } else {
    constexpr float c = static_cast<float>(Root<k, N, S>::re), s = static_cast<float>(Root<k, N, S>::im);
    constexpr float cl = static_cast<float>(Root<k, N, S>::re - static_cast<double>(c));
    constexpr float sl = static_cast<float>(Root<k, N, S>::im - static_cast<double>(s));
    if constexpr ((N & (N - 1)) != 0) return cmul_comp(a, c2(f2(c), f2(s)), c2(f2(cl), f2(sl)));
    else return cmul2k(a, c, s, cl, sl);
  }
}

// rdft of spo_regfft.cuh on two lines: the same operations in the same order on each. Radices 5, 7 and 11, which sum in
// FP64, run line by line.
template <int N, int S>
__device__ __forceinline__ void rdft(C2 (&x)[N]) {
  if constexpr (N == 1) {
  } else if constexpr (N == 2) {
    const C2 a = x[0], b = x[1];
    x[0] = cadd(a, b);
    x[1] = csub(a, b);
  } else if constexpr (N == 4) {
    const C2 s02 = cadd(x[0], x[2]), d02 = csub(x[0], x[2]);
    const C2 s13 = cadd(x[1], x[3]), d13 = csub(x[1], x[3]);
    x[0] = cadd(s02, s13);
    x[1] = cadd_i<S>(d02, d13);
    x[2] = csub(s02, s13);
    x[3] = cadd_i<-S>(d02, d13);
  } else if constexpr (N == 3) {  // the root's sine and cosine as two values each
    constexpr float c = static_cast<float>(Root<1, 3, S>::re), sn = static_cast<float>(Root<1, 3, S>::im);
    constexpr float cl = static_cast<float>(Root<1, 3, S>::re - static_cast<double>(c));
    constexpr float sl = static_cast<float>(Root<1, 3, S>::im - static_cast<double>(sn));
    const C2 s = cadd(x[1], x[2]), d = csub(x[1], x[2]);
    const C2 re = c2(fma2(f2(c), s.x, fma2(f2(cl), s.x, x[0].x)), fma2(f2(c), s.y, fma2(f2(cl), s.y, x[0].y)));
    const C2 im = c2(fma2(f2(sn), d.x, f2(sl) * d.x), fma2(f2(sn), d.y, f2(sl) * d.y));
    x[0] = cadd(x[0], s);
    x[1] = cadd_i<+1>(re, im);
    x[2] = cadd_i<-1>(re, im);
  } else if constexpr (N == 5 || N == 7 || N == 11) {
    float2 a[N], b[N];
    static_for<0, N>([&](auto t) { c2_split(x[t], a[t], b[t]); });
    rdft<N, S>(a);
    rdft<N, S>(b);
    static_for<0, N>([&](auto t) { x[t] = c2(a[t], b[t]); });
  } else {
    constexpr int P = first_factor(N);
    constexpr int Q = N / P;
    C2 y[N];
    static_for<0, P>([&](auto p) {
      C2 sub[Q];
      static_for<0, Q>([&](auto q) { sub[q] = x[p + P * q]; });
      rdft<Q, S>(sub);
      static_for<0, Q>([&](auto k1) {
        y[p * Q + k1] = twiddle_mul2<static_cast<long>(SPO_CV(p)) * SPO_CV(k1), N, S>(sub[k1]);
      });
    });
    static_for<0, Q>([&](auto k1) {
      C2 t[P];
      static_for<0, P>([&](auto p) { t[p] = y[p * Q + k1]; });
      rdft<P, S>(t);
      static_for<0, P>([&](auto k2) { x[k1 + Q * k2] = t[k2]; });
    });
  }
}

#endif  // __CUDACC__

}  // namespace spo
