// The kinetic passes of the scattering wave (src/propagation/kinetic_operators.cpp:77-172) as one kernel: a two-level
// transform of N = N1 N2 points along an axis, times the kinetic factor, and back, for tiles of adjacent lanes. Three
// maps between the points and the two levels:
//   kTwiddle  n = n2 + N2 n1, k = k1 + N1 k2, twiddles w_N^(n2 k1) between the levels (T_Z, T_r)
//   kPrime    n = (N2 n1 + N1 n2) mod N for coprime N1, N2: no twiddles, the factors permuted (axis2pfa_kernel)
//   kXy       n = n1 + N1 n2: the two levels are y (N1) and x (N2) of the (x, y) grid, no twiddles (T_xy), with the
//             momentum shift before and after and, as the last factor, the gas-phase step or the scaling of the
//             interaction region's potential step.
//
// The mixed form takes two adjacent lanes per thread as packed FP32 pairs (spo_pair.cuh): 16-byte accesses and half
// the instructions; the next tile's points are copied to shared memory (cp.async, each thread its own) while a tile is
// transformed. Issue bound it before (65 to 75 % of the slots at 4 TB/s: every constant is exact to ~2^-48, which
// costs two to three times the instructions of plain FP32 products); one lane per thread took 1.64, 1.59 and 1.84 ms
// on configuration 3 (Z 128, r 48, 16 x 16), pairs 1.54, 1.51 and 1.75. A grid of resident blocks loops over the tiles, so that the tables are
// staged in shared memory once per block, not once per tile. kinetic factors s e^{i phi} are applied as p (x + x g)
// with p the power of two in s, folded into g and exact, and a product with the rest s / p only where it is not 1.
//
// N1, N2 > 0: compile-time sizes. N1 = N2 = 0: any two sizes up to 16 that rdft has (a switch per level), for the
// lengths without an instantiation and for rectangular (x, y) grids, as FP64 and Wide; the shared-memory Stockham kernels
// they ran on before are 3 to 10 times slower (T_Z of 90 points, r 36, x = y = 10: 1.12 ms).
//
// FP64 and Wide take one lane per thread. FP64 passes run at 4.3 to 5.6 TB/s (other register kernels: 3.9 to 5.0), Wide
// at 2.0 to 2.9, where the FP64 pipe is the limit.
#pragma once

#include "spo_pot5.cuh"

namespace spo {

enum KinMap : int { kTwiddle = 0, kPrime = 1, kXy = 2, kXyShift = 3 };  // kXy: without the momentum shift
constexpr bool kin_is_xy(int map) { return map == kXy || map == kXyShift; }

// The forms of the kernel: float (complex64, pairs of lanes as packed FP32), double (complex128), and Wide: complex64 in
// memory, FP64 in between, one lane per thread, the constants as they are and one rounding per pass.
struct Wide {};
template <typename T> struct KinStored { using type = T; };
template <> struct KinStored<Wide> { using type = float; };
template <typename T> using KinVec = Vec<typename KinStored<T>::type>;

template <typename T>
struct KinArgs {
  Vec<T>* data;
  int n1, n2;
  long long stride, outer_stride;  // between a line's points, between the line sets of consecutive outer indices
  // lanes: groups of `window` adjacent lanes, group_stride apart, the first at lane_offset
  long long group_stride, lane_offset, window;
  unsigned groups, blocks_per_group, n_tiles;
  int log_lines;          // lines per tile = 1 << log_lines (mixed form: pairs of lanes)
  int aligned;            // mixed form: every pair of lanes starts on a 16-byte boundary
  const double2* table;   // N factors (see KinTable), then N twiddles (kTwiddle), as stored in shared memory
  T scale;                // p
  int unit;               // s = p: no remaining scale
  XyArgs<T> xy;           // kXy: shift, gas-phase and scaling tables
};

// Table entries: mixed form: N pairs (p g.x, p g.x, p g.y, p g.y) and (their low parts), for kTwiddle N twiddles
// (w.x, w.x, w.y, w.y) and (their low parts), and where some s is not p N scales (s/p, s/p, low, low); FP64 and Wide: N
// factors, then N twiddles.
template <typename T> struct KinLine;
template <> struct KinLine<float> {
  using type = C2;
  static constexpr int lanes = 2;
  static constexpr int factor_words = 2, twiddle_words = 2, scale_words = 1;  // 16-byte words per entry
};
template <> struct KinLine<double> {
  using type = double2;
  static constexpr int lanes = 1;
  static constexpr int factor_words = 1, twiddle_words = 1, scale_words = 0;
};
template <> struct KinLine<Wide> : KinLine<double> {};
// 16-byte words of a table in shared memory.
template <typename T>
constexpr int kin_words(int map, int n, bool unit) {
  return n * (KinLine<T>::factor_words + (map == kTwiddle ? KinLine<T>::twiddle_words : 0) + (unit ? 0 : KinLine<T>::scale_words));
}

#ifdef __CUDACC__


// factor k on x
__device__ __forceinline__ C2 kin_factor(C2 x, const C2* f, const C2* scale, int k, F2 p, bool unit) {
  const C2 m = cmul2(x, f[2 * k], f[2 * k + 1]);
  C2 z = c2(fma2(x.x, p, m.x), fma2(x.y, p, m.y));
  if (!unit) {
    const C2 s = scale[k];  // (s/p twice, its low part twice)
    z = c2(fma2(z.x, s.x, z.x * s.y), fma2(z.y, s.x, z.y * s.y));
  }
  return z;
}
__device__ __forceinline__ double2 kin_factor(double2 x, const double2* f, const double2*, int k, double, bool) { return cmul(f[k], x); }
// twiddle j on x, conjugated for S > 0
template <bool ODD, int S>
__device__ __forceinline__ C2 kin_twiddle(C2 x, const C2* tw, int j) {
  C2 w = tw[2 * j], l = tw[2 * j + 1];
  if constexpr (ODD) {
    if constexpr (S > 0) {
      w.y = -w.y;
      l.y = -l.y;
    }
    return cmul_comp(x, w, l);
  } else {
    return S > 0 ? cmul2_conj(x, w, l) : cmul2(x, w, l);
  }
}
template <bool ODD, int S>
__device__ __forceinline__ double2 kin_twiddle(double2 x, const double2* tw, int j) {
  return S > 0 ? cmul(x, cconj(tw[j])) : cmul(x, tw[j]);
}
template <typename T, typename P>
__device__ __forceinline__ auto kin_scale(P p) {
  if constexpr (std::is_same_v<T, float>) return f2(p);
  else return static_cast<double>(p);
}

// The lane(s) of a line: `ok` counts those that exist.
__device__ __forceinline__ C2 kin_load(const float2* p, int ok, bool aligned) {
  float2 a = make_float2(0.0f, 0.0f), b = a;
  if (aligned && ok == 2) {
    const float4 v = *reinterpret_cast<const float4*>(p);
    a = make_float2(v.x, v.y);
    b = make_float2(v.z, v.w);
  } else {
    if (ok > 0) a = p[0];
    if (ok > 1) b = p[1];
  }
  return c2(a, b);
}
__device__ __forceinline__ void kin_store(float2* p, C2 v, int ok, bool aligned) {
  float2 a, b;
  c2_split(v, a, b);
  if (aligned && ok == 2) {
    *reinterpret_cast<float4*>(p) = make_float4(a.x, a.y, b.x, b.y);
  } else {
    if (ok > 0) p[0] = a;
    if (ok > 1) p[1] = b;
  }
}
__device__ __forceinline__ double2 kin_load(const double2* p, int ok, bool) { return ok ? *p : make_double2(0.0, 0.0); }
// A point of a thread's line(s) as it lies in memory (mixed form: re, im, re', im') in a word of shared memory, and back.
__device__ __forceinline__ C2 kin_unpack(const float4* w) {
  const float4 v = *w;
  return c2(make_float2(v.x, v.y), make_float2(v.z, v.w));
}
__device__ __forceinline__ float4 kin_pack(C2 v) {
  float2 a, b;
  c2_split(v, a, b);
  return make_float4(a.x, a.y, b.x, b.y);
}
struct alignas(16) KinWideWord {
  float2 v;
};
__device__ __forceinline__ double2 kin_unpack(const KinWideWord* w) { return make_double2(w->v.x, w->v.y); }
__device__ __forceinline__ void kin_store(float2* p, double2 v, int ok, bool) {
  if (ok) *p = make_float2(static_cast<float>(v.x), static_cast<float>(v.y));
}
__device__ __forceinline__ double2 kin_unpack(const double2* w) { return *w; }
__device__ __forceinline__ double2 kin_pack(double2 v) { return v; }
__device__ __forceinline__ void kin_store(double2* p, double2 v, int ok, bool) {
  if (ok) *p = v;
}

// The factor of the potential step that follows T_xy at a point, for the lane(s) of a line.
struct KinPostPair {
  C2 g, gl, s;
  F2 oz;
  bool unit;
};
struct KinPostF64 {
  double2 g;
  double oz;
};
__device__ __forceinline__ KinPostPair kin_post(const float2* t, long long n, long long k, int ok, float oz) {
  const long long j = ok > 1 ? k + 1 : k;
  const float2 s = t[2 * n + k];  // the scale depends on the r point only
  return KinPostPair{c2(t[k], t[j]), c2(t[n + k], t[n + j]), c2(f2(s.x), f2(s.y)), f2(oz), s.x == 1.0f && s.y == 0.0f && oz == 1.0f};
}
__device__ __forceinline__ C2 kin_apply(C2 x, const KinPostPair& w) {
  C2 z = cadd(x, cmul2(x, w.g, w.gl));
  if (!w.unit) {
    z = c2(fma2(z.x, w.s.x, z.x * w.s.y), fma2(z.y, w.s.x, z.y * w.s.y));
    z = c2(z.x * w.oz, z.y * w.oz);
  }
  return z;
}
__device__ __forceinline__ KinPostF64 kin_post(const double2* t, long long, long long k, int ok, double oz) {
  return KinPostF64{ok ? t[k] : make_double2(0.0, 0.0), oz};
}
// entry k of a mixed form's factor table (g, its low part, the scale's two parts)
__device__ __forceinline__ double2 kin_entry(const float2* t, long long n, long long k) {
  const float2 g = t[k], l = t[n + k], s = t[2 * n + k];
  const double sc = static_cast<double>(s.x) + s.y;
  return make_double2(sc * (1.0 + (static_cast<double>(g.x) + l.x)), sc * (static_cast<double>(g.y) + l.y));
}
// the form's kin_post
template <typename T, typename V, typename R>
__device__ __forceinline__ auto kin_post_of(const V* t, long long n, long long k, int ok, R oz) {
  if constexpr (std::is_same_v<T, Wide>) return KinPostF64{ok ? kin_entry(t, n, k) : make_double2(0.0, 0.0), oz};
  else return kin_post(t, n, k, ok, oz);
}
__device__ __forceinline__ double2 kin_apply(double2 x, const KinPostF64& w) { return cscale(cmul(w.g, x), w.oz); }
// x times entry k of a factor table in global memory (the momentum shift), the same for every lane
__device__ __forceinline__ double2 kin_shift(double2 x, const double2* t, int, int k) { return cmul(t[k], x); }
__device__ __forceinline__ double2 kin_shift(double2 x, const float2* t, int n, int k) { return cmul(kin_entry(t, n, k), x); }

// A thread's share of a tile.
template <typename T>
struct KinTile {
  using L = typename KinLine<T>::type;
  using W = std::conditional_t<std::is_same_v<T, float>, float4, std::conditional_t<std::is_same_v<T, Wide>, KinWideWord, double2>>;
  KinVec<T>* base;   // the line's first point
  long long stride;
  int ok;         // existing lanes of the line
  bool aligned;
  int b, s, nt, log_lines;  // line of the tile, thread of the line, threads per line
  L* Y;           // the tile: [n2][n1][line] as loaded, then [n2][k1][line]
};

template <int MAP>
__device__ __forceinline__ int kin_point(int n1, int n2, int N1, int N2) {
  if constexpr (MAP == kTwiddle) return n2 + N2 * n1;
  else if constexpr (kin_is_xy(MAP)) return n1 + N1 * n2;
  else {
    const int n = N2 * n1 + N1 * n2;
    return n >= N1 * N2 ? n - N1 * N2 : n;
  }
}

// The thread's points of a tile into its own words of `buffer` (asynchronous copies; the ragged edge by plain loads).
template <typename T, int MAP>
__device__ __forceinline__ void kin_request(const KinTile<T>& t, typename KinTile<T>::L* buffer, const KinVec<T>* base, int ok, int N1, int N2) {
  for (int n2 = t.s; n2 < N2; n2 += t.nt) {
    auto* const to = reinterpret_cast<typename KinTile<T>::W*>(buffer) + ((n2 * N1) << t.log_lines) + t.b;
    if constexpr (std::is_same_v<T, Wide>) {
      if (ok) {
#pragma unroll 4
        for (int n1 = 0; n1 < N1; ++n1) pot5::copy8(to + (n1 << t.log_lines), base + kin_point<MAP>(n1, n2, N1, N2) * t.stride);
      } else {
        for (int n1 = 0; n1 < N1; ++n1) to[n1 << t.log_lines].v = make_float2(0.0f, 0.0f);
      }
    } else if (ok == KinLine<T>::lanes && t.aligned) {
#pragma unroll 4
      for (int n1 = 0; n1 < N1; ++n1) pot5::copy16(to + (n1 << t.log_lines), base + kin_point<MAP>(n1, n2, N1, N2) * t.stride);
    } else {
      for (int n1 = 0; n1 < N1; ++n1)
        to[n1 << t.log_lines] = kin_pack(kin_load(base + kin_point<MAP>(n1, n2, N1, N2) * t.stride, ok, t.aligned));
    }
  }
  pot5::copy_commit();
}
// Level 1: DFT over n1 for the thread's n2.
template <typename T, int MAP, int N1, bool ODD>
__device__ __forceinline__ void kin_forward(const KinTile<T>& t, const KinArgs<typename KinStored<T>::type>& a, int N2, const typename KinLine<T>::type* tw) {
  using L = typename KinLine<T>::type;
#pragma unroll 1
  for (int n2 = t.s; n2 < N2; n2 += t.nt) {
    L x[N1];
    static_for<0, N1>([&](auto n1) {
      x[n1] = kin_unpack(reinterpret_cast<const typename KinTile<T>::W*>(t.Y) + ((n2 * N1 + SPO_CV(n1)) << t.log_lines) + t.b);
      if constexpr (MAP == kXyShift) x[n1] = kin_shift(x[n1], a.xy.shift_f, N1 * N2, kin_point<MAP>(SPO_CV(n1), n2, N1, N2));
    });
    rdft<N1, -1>(x);
    static_for<0, N1>([&](auto k1) {
      if constexpr (MAP == kTwiddle && SPO_CV(k1) > 0) x[k1] = kin_twiddle<ODD, -1>(x[k1], tw, n2 * SPO_CV(k1));
      t.Y[((n2 * N1 + SPO_CV(k1)) << t.log_lines) + t.b] = x[k1];
    });
  }
}
// Level 2: DFT over n2 for the thread's k1, the factor, and back.
template <typename T, int MAP, int N2, bool ODD>
__device__ __forceinline__ void kin_middle(const KinTile<T>& t, const KinArgs<typename KinStored<T>::type>& a, int N1, const typename KinLine<T>::type* f,
                                           const typename KinLine<T>::type* tw) {
  using L = typename KinLine<T>::type;
  const auto p = kin_scale<T>(a.scale);
  const bool unit = a.unit != 0;
  const L* const scale = f + (KinLine<T>::factor_words + (MAP == kTwiddle ? KinLine<T>::twiddle_words : 0)) * N1 * N2;
#pragma unroll 1
  for (int k1 = t.s; k1 < N1; k1 += t.nt) {
    L y[N2];
    L* const row = t.Y + (k1 << t.log_lines) + t.b;
    static_for<0, N2>([&](auto n2) { y[n2] = row[(SPO_CV(n2) * N1) << t.log_lines]; });
    rdft<N2, -1>(y);
    static_for<0, N2>([&](auto k2) { y[k2] = kin_factor(y[k2], f, scale, k1 + N1 * SPO_CV(k2), p, unit); });
    rdft<N2, +1>(y);
    static_for<0, N2>([&](auto n2) {
      if constexpr (MAP == kTwiddle && SPO_CV(n2) > 0) y[n2] = kin_twiddle<ODD, +1>(y[n2], tw, SPO_CV(n2) * k1);
      row[(SPO_CV(n2) * N1) << t.log_lines] = y[n2];
    });
  }
}
template <typename T, int MAP, int N1, typename P>
__device__ __forceinline__ void kin_back(const KinTile<T>& t, const KinArgs<typename KinStored<T>::type>& a, int N2, bool post, const P& w) {
  using L = typename KinLine<T>::type;
  if (t.ok == 0) return;
#pragma unroll 1
  for (int n2 = t.s; n2 < N2; n2 += t.nt) {
    L x[N1];
    static_for<0, N1>([&](auto k1) { x[k1] = t.Y[((n2 * N1 + SPO_CV(k1)) << t.log_lines) + t.b]; });
    rdft<N1, +1>(x);
    static_for<0, N1>([&](auto n1) {
      const int n = kin_point<MAP>(SPO_CV(n1), n2, N1, N2);
      if constexpr (MAP == kXyShift) x[n1] = kin_shift(x[n1], a.xy.shift_b, N1 * N2, n);
      if constexpr (kin_is_xy(MAP))
        if (post) x[n1] = kin_apply(x[n1], w);
      kin_store(t.base + n * t.stride, x[n1], t.ok, t.aligned);
    });
  }
}

// f(size) for a runtime size among those of rdft up to 16.
template <typename F>
__device__ __forceinline__ void kin_switch(int n, F&& f) {
  switch (n) {
    case 1: f(std::integral_constant<int, 1>{}); break;
    case 2: f(std::integral_constant<int, 2>{}); break;
    case 3: f(std::integral_constant<int, 3>{}); break;
    case 4: f(std::integral_constant<int, 4>{}); break;
    case 5: f(std::integral_constant<int, 5>{}); break;
    case 6: f(std::integral_constant<int, 6>{}); break;
    case 7: f(std::integral_constant<int, 7>{}); break;
    case 8: f(std::integral_constant<int, 8>{}); break;
    case 9: f(std::integral_constant<int, 9>{}); break;
    case 10: f(std::integral_constant<int, 10>{}); break;
    case 11: f(std::integral_constant<int, 11>{}); break;
    case 12: f(std::integral_constant<int, 12>{}); break;
    case 14: f(std::integral_constant<int, 14>{}); break;
    case 15: f(std::integral_constant<int, 15>{}); break;
    default: f(std::integral_constant<int, 16>{}); break;
  }
}

// Registers: the lines of the larger level (4 per point and pair of lanes) and its temporaries.
constexpr int kin_max_threads(int n) { return n > 16 ? 128 : 256; }
constexpr int kin_min_blocks(int n) { return n > 16 ? 3 : n > 8 || n == 0 ? 2 : 3; }

template <typename T, int MAP, int N1C, int N2C>
__global__ void __launch_bounds__(kin_max_threads(N1C > N2C ? N1C : N2C), kin_min_blocks(N1C > N2C ? N1C : N2C))
    kin_kernel(const __grid_constant__ KinArgs<typename KinStored<T>::type> a) {
  using L = typename KinLine<T>::type;
  constexpr bool ANY = N1C == 0;
  const int N1 = ANY ? a.n1 : N1C, N2 = ANY ? a.n2 : N2C, N = N1 * N2;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  L* const f = reinterpret_cast<L*>(smem_raw);
  L* const tw = f + KinLine<T>::factor_words * N;
  KinTile<T> t;
  const int words = kin_words<T>(MAP, N, a.unit != 0);
  L* const tiles = f + words;  // two tiles
  {
    const L* src = reinterpret_cast<const L*>(a.table);
    for (int k = threadIdx.x; k < words; k += blockDim.x) f[k] = src[k];
  }
  t.log_lines = a.log_lines;
  t.b = threadIdx.x & ((1 << a.log_lines) - 1);
  t.s = threadIdx.x >> a.log_lines;
  t.nt = blockDim.x >> a.log_lines;
  t.stride = a.stride;
  t.aligned = a.aligned != 0;
  // twiddle products of lengths with an odd factor are nearly correctly rounded (cmul_comp)
  constexpr bool ODD = ANY || ((N1C * N2C) & (N1C * N2C - 1)) != 0;
  auto locate = [&](unsigned tile, KinVec<T>*& base, int& ok, unsigned& outer, long long& lane) {
    const unsigned rest = tile / a.blocks_per_group, blk = tile - rest * a.blocks_per_group;
    outer = rest / a.groups;
    const unsigned grp = rest - outer * a.groups;
    lane = (static_cast<long long>(blk) << a.log_lines) * KinLine<T>::lanes + t.b * KinLine<T>::lanes;
    ok = lane >= a.window ? 0 : static_cast<int>(min(static_cast<long long>(KinLine<T>::lanes), a.window - lane));
    base = a.data + outer * a.outer_stride + grp * a.group_stride + a.lane_offset + lane;
  };
  unsigned tile = blockIdx.x, outer = 0;
  long long lane = 0;
  if (tile < a.n_tiles) {
    locate(tile, t.base, t.ok, outer, lane);
    kin_request<T, MAP>(t, tiles, t.base, t.ok, N1, N2);
  }
  __syncthreads();
  // Levels 1 and 3 touch the thread's own words of a tile only, so that the next tile but one may overwrite them without
  // a barrier; level 2 lies between two.
  int side = 0;
  for (; tile < a.n_tiles; tile += gridDim.x, side ^= 1) {
    // the next tile's points, on their way during this one
    KinVec<T>* next_base = nullptr;
    int next_ok = 0;
    unsigned next_outer = 0;
    long long next_lane = 0;
    if (tile + gridDim.x < a.n_tiles) {
      locate(tile + gridDim.x, next_base, next_ok, next_outer, next_lane);
      kin_request<T, MAP>(t, tiles + (side ^ 1) * (N << t.log_lines), next_base, next_ok, N1, N2);
    } else {
      pot5::copy_commit();
    }
    t.Y = tiles + side * (N << t.log_lines);
    pot5::copy_wait<1>();  // this tile's points
    if constexpr (ANY) kin_switch(N1, [&](auto n) { kin_forward<T, MAP, SPO_CV(n), ODD>(t, a, N2, tw); });
    else kin_forward<T, MAP, N1C, ODD>(t, a, N2C, tw);
    __syncthreads();
    if constexpr (ANY) kin_switch(N2, [&](auto n) { kin_middle<T, MAP, SPO_CV(n), ODD>(t, a, N1, f, tw); });
    else kin_middle<T, MAP, N2C, ODD>(t, a, N1C, f, tw);
    __syncthreads();
    if constexpr (kin_is_xy(MAP)) {
      const long long izr = a.xy.izr_offset + outer;
      const long long half = static_cast<long long>(a.xy.nr) * a.xy.n_rot;
      const KinVec<T>* const table = xy_post(a.xy, izr) ? a.xy.post_step + (izr >= a.xy.izr_gas_first ? 0 : half) : nullptr;
      decltype(kin_post_of<T>(table, 0ll, 0ll, 0, a.scale)) w{};
      if (table && t.ok)
        w = kin_post_of<T>(table, 2 * half, (izr % a.xy.nr) * a.xy.n_rot + lane, t.ok, a.xy.opt_z[izr / a.xy.nr]);
      if constexpr (ANY) kin_switch(N1, [&](auto n) { kin_back<T, MAP, SPO_CV(n)>(t, a, N2, table != nullptr, w); });
      else kin_back<T, MAP, N1C>(t, a, N2C, table != nullptr, w);
    } else {
      if constexpr (ANY) kin_switch(N1, [&](auto n) { kin_back<T, MAP, SPO_CV(n)>(t, a, N2, false, 0); });
      else kin_back<T, MAP, N1C>(t, a, N2C, false, 0);
    }
    t.base = next_base;
    t.ok = next_ok;
    outer = next_outer;
    lane = next_lane;
  }
}

#endif  // __CUDACC__

}  // namespace spo
