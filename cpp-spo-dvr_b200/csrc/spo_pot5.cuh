// Potential step of the interaction region, mixed form (src/propagation/potential_operator.cpp:84-135,
// angular_transform.cpp:54-114): both theta contractions on the FP64 tensor cores (mma.m8n8k4.f64), the phi
// transforms in registers between them.
//
// A team of H warps (H = 1 for ntheta <= 8, 2 for ntheta <= 16) owns 8 (x, y) columns at a time, warp h the
// theta 8h .. 8h + 7 of every one of them:
//   - forward: X_m[c, theta] = sum_J F[c, J] M_m[theta, J] for every mJ block m, columns as the rows of the
//     product. Lane (c = lane / 4, t = lane % 4) then holds theta 8h + 2t and 8h + 2t + 1 of column c for
//     every phi slot, real and imaginary parts (two products share each matrix fragment): two complete phi lines
//     per lane, so the phi transforms, exp(i A) and the inverse transforms need no exchange at all;
//   - back: out[c, J] = sum_theta X[c, theta] M_m[theta, J]. The accumulator layout of the forward product is the
//     A operand layout of this one when the summed theta are taken in the order 8h + 2 (lane % 4) + i, i = 0, 1:
//     the values go from registers into the tensor core. With H = 2 each warp takes every other phi slot and gets
//     the other warp's eight theta of it through shared memory (FP32).
// Products and sums are FP64 (the matrix exactly as given), rounded once to FP32 per contraction: the FP32 state
// of the mixed form is kept, its contractions lose nothing.
//
// What bounds it: on configuration 3 (2.6e8 values of psi per launch) the tensor core needs 84 multiply-adds per
// value with its padding (1.2 ms), the FP32 pipe about 100 operations per value for the phi transforms and
// exp(i A) (0.8 ms), HBM 9.5 GB (1.5 ms). The FP32 form of the contractions (a 12-bit high part and the rest of
// each matrix entry, two FMAs per term, operands through shared memory) spent 128 FMA-pipe operations and as many
// bytes of shared memory per value and took 5.62 ms.
//
// Data movement: the 8 columns of a team's next item (n_rot contiguous values each) are copied into its F buffer
// by cp.async.bulk as soon as F is free (H = 2: after the exchange, which uses the same memory) (completion counted in bytes on the team's
// mbarrier; odd n_rot, whose columns are not 16-byte multiples, by plain loads). The exp(i A) entries are stored
// in the order in which the lanes read them: per (Z, r) point and representative [phi][pair of theta] as
// (re, re', im, im') with the modulus corrections of G phi together, so the four lanes of a column read 64
// contiguous bytes; the next item's are requested into L2 one item ahead, except by the ring form (ring_of), whose own
// copies run ahead.
//
// psi comes scaled by the absorbers and rot(dt/2): the xy pass before this kernel multiplies every value anyway.
//
// Every wait on an mbarrier is bounded. A team whose wait gives up sets *error_flag, waits (bounded) for the
// copies it has in flight and leaves; the host reads the flag after the step.
#pragma once

#include <cstdint>

#include "spo_pair.cuh"
#include "spo_pot4.cuh"

namespace spo {

namespace pot5 {

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_init_fence() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// Arrives on the barrier, announcing `bytes` more bytes of asynchronous copies for the current phase.
__device__ __forceinline__ void mbar_arrive_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile(
      "{\n\t.reg .b64 state;\n\t"
      "mbarrier.arrive.expect_tx.shared::cta.b64 state, [%0], %1;\n\t}" ::"r"(smem_addr(bar)),
      "r"(bytes)
      : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile(
      "{\n\t.reg .b64 state;\n\t"
      "mbarrier.arrive.shared::cta.b64 state, [%0];\n\t}" ::"r"(smem_addr(bar))
      : "memory");
}

// Waits for the phase with the given parity to complete; false after `limit` polls (kWaitLimit by default).
constexpr int kWaitLimit = 1 << 22;
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, int limit = kWaitLimit) {
  const uint32_t addr = smem_addr(bar);
  for (int i = 0; i < limit; ++i) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(addr), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

// Orders this thread's earlier shared-memory accesses before later asynchronous-proxy writes to them.
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// Asks for `bytes` (a multiple of 16, 16-byte aligned) of global memory to be brought into L2.
__device__ __forceinline__ void prefetch_l2(const void* src, uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(src), "r"(bytes) : "memory");
}

// Bulk copy of `bytes` (a multiple of 16, both addresses 16-byte aligned) from global to this CTA's
// shared memory, completing `bytes` on the barrier.
__device__ __forceinline__ void bulk_copy(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smem_addr(dst)),
      "l"(src), "r"(bytes), "r"(smem_addr(bar))
      : "memory");
}

// Vote of a team (64 threads on named barrier `id`, or one warp): true when any thread's `fail` is set; also a
// barrier of the team.
template <int H>
__device__ __forceinline__ bool team_any(int id, bool fail) {
  if constexpr (H == 1) {
    __syncwarp();
    return __any_sync(0xffffffffu, fail);
  } else {
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 q, %1, 0;\n\t"
        "barrier.cta.red.or.pred p, %2, 64, q;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(r)
        : "r"(fail ? 1u : 0u), "r"(id)
        : "memory");
    return r != 0;
  }
}
template <int H>
__device__ __forceinline__ void team_sync(int id) {
  if constexpr (H == 1) __syncwarp();
  else asm volatile("barrier.cta.sync %0, 64;" ::"r"(id) : "memory");
}

// D += A B, 8 x 8 x 4 in FP64: lane l holds A[l / 4][l % 4], B[l % 4][l / 4], D[l / 4][2 (l % 4) + {0, 1}].
__device__ __forceinline__ void dmma(double& d0, double& d1, double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(d0), "+d"(d1)
      : "d"(a), "d"(b));
}

// Loads of values that are read once, past L1 (whose 28 KB beside the shared memory hold the rotation factors).
__device__ __forceinline__ float4 ld_stream4(const float4* p) {
  float4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ uint2 ld_stream2(const void* p) {
  uint2 v;
  asm volatile("ld.global.nc.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
  return v;
}

// This thread's own asynchronous copies (global -> shared, past L1), in groups.
__device__ __forceinline__ void copy16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copy8(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int PENDING>
__device__ __forceinline__ void copy_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(PENDING) : "memory");
}

// phi whose modulus corrections are stored together (16 or 8 bytes per pair of theta).
constexpr int group_of(int nphi) { return nphi % 4 == 0 ? 4 : 2; }
constexpr int kCols = 8;       // columns per item
// F column stride (values): n_rot and at least 4 zeros behind it, 4 or 12 mod 16 so that the 4 x 8 values of a
// fragment fall on distinct banks.
constexpr int f_stride(int n_rot) {
  int s = (n_rot + 4 + 3) / 4 * 4;
  while (s % 16 != 4 && s % 16 != 12) s += 4;
  return s;
}
// Threads per block: the phi lines of a lane take 4 nphi registers.
constexpr int threads_of(int nphi) { return nphi > 16 ? 384 : nphi > 8 ? 512 : 640; }
// With two warps per team and 28 or 32 phi, the lines (112 or 128 registers) leave no registers for exp(i A) entries in
// flight: each lane copies its entries into the team's buffer instead, kBatches batches of 4 phi (and their corrections)
// ahead, and the row of rot(dt/2) comes with the columns. Configuration 3: 4.08 ms against 4.92 with loads two batches of
// two phi ahead in registers and rot(dt/2) through L1 (3.83 since the ring requests nothing into L2); phi 24 with symmetry maps 1.35 against 1.25 ms, phi 18 0.547
// against 0.525, one warp per team 0.78 against 0.55: there the loads in registers stay.
constexpr bool ring_of(int nphi, int h) { return h == 2 && nphi >= 28 && nphi % 4 == 0; }
constexpr int kBatches = 3, kBatchBytes = 5 * 512;
// Bytes of a team's buffer, used in turn for the columns of its item, (ring) its warps' exp(i A) entries and (H = 2) the
// values that the warps exchange; with (ring) the row of rot(dt/2).
constexpr std::size_t buffer_bytes(int n_rot, int nphi, int h) {
  std::size_t f = sizeof(float2) * kCols * static_cast<std::size_t>(f_stride(n_rot));
  const std::size_t x = h == 2 ? static_cast<std::size_t>(nphi) * 32 * sizeof(float4) : 0;
  const std::size_t r = ring_of(nphi, h) ? 2 * kBatches * kBatchBytes : 0;
  f = f > x ? f : x;
  return f > r ? f : r;
}
constexpr std::size_t team_bytes(int n_rot, int nphi, int h) {
  return buffer_bytes(n_rot, nphi, h) + (ring_of(nphi, h) ? sizeof(double2) * static_cast<std::size_t>(n_rot) : 0);
}

}  // namespace pot5

struct Pot5Args {
  PotArgs<float> p;
  const float4* table;   // exp(i A) - 1: [(Z, r) point][representative][phi][pair of theta] (re, re', im, im')
  const __half2* mods;   // modulus corrections: [point][representative][phi / G][pair of theta][phi % G]
  const double* frags;   // matrix fragments of 32 values: the forward ones, then the transposed ones
  int n_fwd, n_back;     // their numbers
  const int4* slots;     // per phi slot: first irot, J count + 65536 forward steps, first forward and transposed fragment
  const double2* rot;    // (ir, irot): rot(dt/2)
  const uint8_t* phi_map;  // n_xy * nphi, or null (no symmetry)
  int pairs;             // pairs of theta in the table
  int n_cols, n_items;   // columns of the interaction region, items of kCols columns
  int bulk;              // columns are 16-byte multiples: bulk copies
  int poll_limit;        // polls before a wait on an mbarrier gives up
  unsigned extra_tx;     // bytes announced beyond those copied (0; a failure-detection test sets it so that a
                         // barrier phase cannot complete and the wait gives up)
};

template <int NPHI, int H>
__global__ void __launch_bounds__(pot5::threads_of(NPHI), 1) potential5_kernel(Pot5Args g, int* error_flag) {
  using namespace pot5;
  constexpr int G = group_of(NPHI);
  constexpr bool RING = ring_of(NPHI, H);
  const PotArgs<float>& a = g.p;
  const int n_rot = a.n_rot, n_xy = a.n_xy, nr = a.nr;
  const int fcs = f_stride(n_rot);
  extern __shared__ __align__(128) unsigned char smem_raw[];
  double* const mats = reinterpret_cast<double*>(smem_raw);
  int4* const slots = reinterpret_cast<int4*>(mats + 32 * (g.n_fwd + g.n_back));
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32, teams = blockDim.x / (32 * H);
  const int team = warp / H, h = warp % H, bar_id = 1 + team;
  uint64_t* const bars = reinterpret_cast<uint64_t*>(slots + NPHI);
  uint64_t* const bar = bars + team;
  unsigned char* const own = reinterpret_cast<unsigned char*>(bars + ((teams + 1) & ~1)) + team * team_bytes(n_rot, NPHI, H);
  float2* const F = reinterpret_cast<float2*>(own);               // [c][irot], columns of fcs values
  float4* const EX = reinterpret_cast<float4*>(own);              // [reading warp][slot pair][lane], after F is consumed
  double2* const rot_row = reinterpret_cast<double2*>(own + buffer_bytes(n_rot, NPHI, H));  // RING: rot(dt/2) at the item's r point
  if (lane == 0 && h == 0) mbar_init(bar, 1);
  mbar_init_fence();
  for (int k = threadIdx.x; k < 32 * (g.n_fwd + g.n_back); k += blockDim.x) mats[k] = g.frags[k];
  for (int k = threadIdx.x; k < NPHI; k += blockDim.x) slots[k] = g.slots[k];
  for (int k = h * 32 + lane; k < kCols * fcs; k += 32 * H) F[k] = make_float2(0.0f, 0.0f);
  __syncthreads();
  const double* const mf = mats + lane;
  const double* const mb = mats + 32 * g.n_fwd + lane;

  const int c = lane >> 2, t = lane & 3;
  const int i0 = a.initial_channel;
  const uint32_t col_bytes = static_cast<uint32_t>(n_rot * sizeof(float2));
  const int step = gridDim.x * teams;

  // The columns of an item into F: one warp's lanes issue a bulk copy each (H = 2: warp 0), or every lane loads.
  auto issue = [&](int item) {
    const int col0 = item * kCols;
    const int ncol = min(kCols, g.n_cols - col0);
    if (g.bulk) {
      if (h == 0) {
        fence_proxy_async();
        const int izr = col0 / n_xy;
        const bool row = RING && (col0 + ncol - 1) / n_xy == izr;  // one r point
        if (lane == 0) mbar_arrive_tx(bar, col_bytes * ncol + (row ? 2 * col_bytes : 0u) + g.extra_tx);
        __syncwarp();
        if (row && lane == kCols) bulk_copy(rot_row, g.rot + (izr % nr) * n_rot, 2 * col_bytes, bar);
        if (lane < ncol) bulk_copy(F + lane * fcs, a.psi + static_cast<long long>(col0 + lane) * n_rot, col_bytes, bar);
      }
    } else {
      for (int k = h * 32 + lane; k < ncol * n_rot; k += 32 * H) {
        const int cc = k / n_rot;
        F[cc * fcs + k - cc * n_rot] = a.psi[static_cast<long long>(col0) * n_rot + k];
      }
    }
  };
  // The columns, exp(i A) rows and corrections of an item into L2 (column c by one lane). Not in the ring form, whose copies run
  // 12 phi ahead by themselves: 888 teams had 29 MB of rows ahead besides those in use, and about as much as the table was
  // read again from DRAM (1.49 times the algorithmic bytes; configuration 3: 4.12 ms with the rows and psi requested, 4.11 with
  // the request after the phi phase, 3.90 with psi alone, 3.83 without). Nor does it pay for phi 28, symmetry maps or odd n_rot
  // (64 x 48 x 12 x 12, without/with: J 13 1.30/1.34, with maps 1.33/1.35; J 12, n_rot 169, 1.26/1.29, with maps 1.33/1.33; J 15 with
  // maps 1.14/1.22).
  auto prefetch = [&](int item) {
    const int col = item * kCols + lane;
    if (h == 0 && lane < kCols && col < g.n_cols) {
      const int izr = col / n_xy, ixy = col - izr * n_xy;
      const long long e = (static_cast<long long>(izr) * a.n_rep + (g.phi_map ? __ldg(a.rep_of + ixy) : ixy)) * NPHI * g.pairs;
      prefetch_l2(g.table + e, static_cast<uint32_t>(NPHI * g.pairs * sizeof(float4)));
      const uint32_t mod_bytes = static_cast<uint32_t>(NPHI * g.pairs * sizeof(__half2));
      if (mod_bytes % 16 == 0) prefetch_l2(g.mods + e, mod_bytes);
      if (H == 2 && g.bulk) prefetch_l2(a.psi + static_cast<long long>(col) * n_rot, col_bytes);
    }
  };

  int item = blockIdx.x * teams + team;
  uint32_t parity = 0;
  if (item < g.n_items) {
    issue(item);
    if constexpr (!RING) prefetch(item);
  }
  for (; item < g.n_items; item += step) {
    const bool ok = !g.bulk || mbar_wait(bar, parity, g.poll_limit);
    if (team_any<H>(bar_id, !ok)) {
      if (lane == 0 && h == 0) {
        *static_cast<volatile int*>(error_flag) = 1;  // host memory: a plain store, no atomic
        mbar_wait(bar, parity, g.poll_limit);  // bounded: no copy lands after the team has left
      }
      return;
    }
    parity ^= 1u;

    // ---- the item's columns: the specular wave into the initial channel (the absorbers and rot(dt/2) are in psi)
    const int col = item * kCols + c;
    const bool col_ok = col < g.n_cols;
    const int izr = min(col, g.n_cols - 1) / n_xy, ixy = min(col, g.n_cols - 1) - izr * n_xy;
    const int ir = izr % nr;
    if (!col_ok) {
      for (int j = h * 4 + t; j < n_rot; j += 4 * H) F[c * fcs + j] = make_float2(0.0f, 0.0f);
    } else if (h == 0 && t == 0) {
      const float2 chi = a.chi[izr], s = a.sp2sc[ixy], sl = a.sp2sc[n_xy + ixy];
      const double2 r0 = g.rot[ir * n_rot + i0];
      const double sx = static_cast<double>(s.x) + sl.x, sy = static_cast<double>(s.y) + sl.y;
      const double ux = sx * chi.x - sy * chi.y, uy = sx * chi.y + sy * chi.x;
      float2* const v = F + c * fcs + i0;
      *v = make_float2(static_cast<float>(v->x + (ux * r0.x - uy * r0.y)), static_cast<float>(v->y + (ux * r0.y + uy * r0.x)));
    }
    team_sync<H>(bar_id);

    // ---- forward contraction, two slots at a time (p and nphi - p, usually of equal J count)
    C2 x[NPHI];  // the lane's two phi lines: theta 8 h + 2 t and 8 h + 2 t + 1
    const float2* const fl = F + c * fcs + t;
    static_for<0, NPHI / 2>([&](auto q) {
      constexpr int PA = SPO_CV(q) == 0 ? 0 : SPO_CV(q);
      constexpr int PB = SPO_CV(q) == 0 ? NPHI / 2 : NPHI - SPO_CV(q);
      const int4 sa = slots[PA], sb = slots[PB];
      const int nk = sa.y >> 16;  // the same for both (the shorter block's fragments end in zeros)
      double ar0 = 0, ar1 = 0, ai0 = 0, ai1 = 0, br0 = 0, br1 = 0, bi0 = 0, bi1 = 0;
      const float2 *fa = fl + sa.x, *fb = fl + sb.x;
      const double *ma = mf + 32 * (sa.z + h * nk), *mc = mf + 32 * (sb.z + h * nk);
#pragma unroll 1
      for (int k = 0; k < nk; ++k) {
        const float2 u = fa[4 * k];
        const double m = ma[32 * k];
        dmma(ar0, ar1, u.x, m);
        dmma(ai0, ai1, u.y, m);
        if constexpr (SPO_CV(q) != 0) {
          const float2 v = fb[4 * k];
          const double n = mc[32 * k];
          dmma(br0, br1, v.x, n);
          dmma(bi0, bi1, v.y, n);
        }
      }
      x[PA] = c2(f2(static_cast<float>(ar0), static_cast<float>(ar1)), f2(static_cast<float>(ai0), static_cast<float>(ai1)));
      x[PB] = c2(f2(static_cast<float>(br0), static_cast<float>(br1)), f2(static_cast<float>(bi0), static_cast<float>(bi1)));
    });
    team_sync<H>(bar_id);
    const int next = item + step;
    if (next < g.n_items) {
      if (H == 1 && g.bulk) issue(next);  // every lane of the team has read F
      if constexpr (!RING) prefetch(next);
    }

    // ---- phi transform, exp(i A), inverse phi transform of the lane's two lines
    const int tp = min(4 * h + t, g.pairs - 1);  // theta beyond the grid: zero lines
    const long long e0 = (static_cast<long long>(izr) * a.n_rep + (g.phi_map ? __ldg(a.rep_of + ixy) : ixy)) * NPHI * g.pairs;
    const float4* et = g.table + e0 + tp;
    const __half2* em = g.mods + e0 + tp * G;
    auto apply = [&](auto p, float4 e4, uint32_t m2) {  // exp_mul_m on both lines
      const F2 m = f2(mod_lo(m2), mod_hi(m2)) * f2(5.9604644775390625e-8f);  // 2^-24
      const C2 e = c2(f2(e4.x, e4.y), f2(e4.z, e4.w));
      x[p] = cadd(x[p], cmul2(x[p], e, c2(m * (f2(1.0f) + e.x), m * e.y)));
    };
    if constexpr (RING) {
      constexpr int NB = NPHI / G;
      unsigned char* const ring = own + h * kBatches * kBatchBytes + lane * 16;
      auto request = [&](auto b) {
        constexpr int B = SPO_CV(b);
        unsigned char* const to = ring + (B % kBatches) * kBatchBytes;
        if (g.phi_map == nullptr) {
          static_for<0, G>([&](auto i) { copy16(to + SPO_CV(i) * 512, et + (B * G + SPO_CV(i)) * g.pairs); });
          copy16(to + G * 512, em + B * G * g.pairs);
        } else {
          const uint8_t* const map = g.phi_map + ixy * NPHI + B * G;
          uint32_t* const m = reinterpret_cast<uint32_t*>(to + G * 512);
          static_for<0, G>([&](auto i) {
            const int pm = __ldg(map + SPO_CV(i));
            copy16(to + SPO_CV(i) * 512, et + pm * g.pairs);
            m[SPO_CV(i)] = __ldg(reinterpret_cast<const uint32_t*>(em + (pm / G) * G * g.pairs + pm % G));
          });
        }
        copy_commit();
      };
      static_for<0, kBatches>([&](auto b) { request(b); });
      rdft<NPHI, +1>(x);
      static_for<0, NB>([&](auto b) {
        constexpr int B = SPO_CV(b);
        copy_wait<(NB - 1 - B < kBatches - 1 ? NB - 1 - B : kBatches - 1)>();
        const unsigned char* const from = ring + (B % kBatches) * kBatchBytes;
        const uint4 m = *reinterpret_cast<const uint4*>(from + G * 512);
        const uint32_t m2[4] = {m.x, m.y, m.z, m.w};
        static_for<0, G>([&](auto i) {
          apply(std::integral_constant<int, B * G + SPO_CV(i)>{}, *reinterpret_cast<const float4*>(from + SPO_CV(i) * 512), m2[SPO_CV(i)]);
        });
        if constexpr (B + kBatches < NB) request(std::integral_constant<int, B + kBatches>{});
      });
    } else {
      rdft<NPHI, +1>(x);
      // Two phi per batch, the next batch's loads in flight while one is applied. The empty asm statements tie a batch's
      // address to values of the batch before the last, so that the compiler does not collect all loads in front (and
      // spill the lines to make room for them).
      constexpr int NB = NPHI / 2;
      float4 w[2][2];
      uint32_t m2[2][2];
      auto load = [&](auto b) {
        constexpr int P = 2 * SPO_CV(b), U = SPO_CV(b) % 2;
        if (g.phi_map == nullptr) {
          const uint2 m = ld_stream2(em + (P / G) * G * g.pairs + P % G);
          m2[U][0] = m.x;
          m2[U][1] = m.y;
          w[U][0] = ld_stream4(et + P * g.pairs);
          w[U][1] = ld_stream4(et + (P + 1) * g.pairs);
        } else {
          const uint8_t* map = g.phi_map + ixy * NPHI;
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const int pm = __ldg(map + P + i);
            m2[U][i] = __ldg(reinterpret_cast<const uint32_t*>(em + (pm / G) * G * g.pairs + pm % G));
            w[U][i] = ld_stream4(et + pm * g.pairs);
          }
        }
      };
      asm volatile("" : "+l"(et), "+l"(em), "+l"(x[NPHI - 1].x.v));
      load(std::integral_constant<int, 0>{});
      static_for<0, NB>([&](auto b) {
        constexpr int B = SPO_CV(b), U = B % 2;
        if constexpr (B + 1 < NB) load(std::integral_constant<int, B + 1>{});
        apply(std::integral_constant<int, 2 * B>{}, w[U][0], m2[U][0]);
        apply(std::integral_constant<int, 2 * B + 1>{}, w[U][1], m2[U][1]);
        asm volatile("" : "+l"(et), "+l"(em), "+l"(x[2 * B + 1].y.v));
      });
    }
    rdft<NPHI, -1>(x);

    // ---- transposed contraction, rot(dt/2), store
    float2* const out = a.psi + static_cast<long long>(col) * n_rot;
    // (RING: the row in shared memory, if the item lies at one point, as in issue())
    const bool row = RING && g.bulk && (item * kCols) / n_xy == min(item * kCols + kCols - 1, g.n_cols - 1) / n_xy;
    const double2* const rot = row ? rot_row : g.rot + ir * n_rot;
    auto rot_at = [&](int irot) {
      if constexpr (RING) return rot[irot];
      else return __ldg(rot + irot);
    };
    auto finish = [&](int irot, double2 w, double re, double im) {
      out[irot] = make_float2(static_cast<float>(re * w.x - im * w.y), static_cast<float>(re * w.y + im * w.x));
    };
    // One slot: the warp's own theta in v[0..3], the other warp's in v[4..7].
    auto back = [&](int p, const double (&v)[4 * H]) {
      const int4 s = slots[p];
      const int nj = s.y & 0xffff;
#pragma unroll 1
      for (int jt = 0; 8 * jt < nj; ++jt) {
        const double* const m0 = mb + 32 * (s.w + (jt * H + h) * 2);
        const double* const m1 = mb + 32 * (s.w + (jt * H + H - 1 - h) * 2);
        const int j = 8 * jt + t;
        const double2 wa = rot_at(s.x + min(j, nj - 1)), wb = rot_at(s.x + min(j + 4, nj - 1));
        double r0 = 0, r1 = 0, q0 = 0, q1 = 0;
#pragma unroll
        for (int i = 0; i < 2 * H; ++i) {
          const double w = (i < 2 ? m0 : m1)[32 * (i % 2)];
          dmma(r0, r1, v[2 * i], w);
          dmma(q0, q1, v[2 * i + 1], w);
        }
        if (col_ok) {
          if (j < nj) finish(s.x + j, wa, r0, q0);
          if (j + 4 < nj) finish(s.x + j + 4, wb, r1, q1);
        }
      }
    };
    if constexpr (H == 1) {
      static_for<0, NPHI>([&](auto p) {
        float2 u, w;
        c2_split(x[p], u, w);
        const double v[4] = {u.x, u.y, w.x, w.y};
        back(SPO_CV(p), v);
      });
    } else {
      // Warp h takes the slots 2 q + h: it keeps its own theta of them and gets the other warp's through F.
      float4* const to = EX + (h ^ 1) * (NPHI / 2) * 32 + lane;
      const float4* const from = EX + h * (NPHI / 2) * 32 + lane;
      float4 mine[NPHI / 2];
      if (RING) team_sync<H>(bar_id);  // both warps have read their exp(i A) entries
      static_for<0, NPHI / 2>([&](auto q) {
        float2 e0, e1, o0, o1;
        c2_split(x[2 * SPO_CV(q)], e0, e1);
        c2_split(x[2 * SPO_CV(q) + 1], o0, o1);
        const float4 xe = make_float4(e0.x, e0.y, e1.x, e1.y), xo = make_float4(o0.x, o0.y, o1.x, o1.y);
        to[SPO_CV(q) * 32] = h == 0 ? xo : xe;
        mine[SPO_CV(q)] = h == 0 ? xe : xo;
      });
      team_sync<H>(bar_id);
      static_for<0, NPHI / 2>([&](auto q) {
        const float4 z = mine[SPO_CV(q)], y = from[SPO_CV(q) * 32];
        const double v[8] = {z.x, z.y, z.z, z.w, y.x, y.y, y.z, y.w};
        back(2 * SPO_CV(q) + h, v);
      });
      team_sync<H>(bar_id);
      // the zeros behind the columns again, then the next item's columns
      if (h == 0) F[c * fcs + n_rot + t] = make_float2(0.0f, 0.0f);
      if (next < g.n_items) issue(next);
    }
    if (H == 1 && !g.bulk) {
      __syncwarp();
      if (next < g.n_items) issue(next);
    }
    if (!g.bulk) team_sync<H>(bar_id);
  }
}

namespace pot5 {

// The instantiation for (nphi, H), or null (spo_pot5.cu, one translation unit per part).
using Kernel = void (*)(Pot5Args, int*);
template <int PART>
Kernel kernel_of_part(int nphi, int h);
template <> Kernel kernel_of_part<0>(int nphi, int h);
template <> Kernel kernel_of_part<1>(int nphi, int h);
template <> Kernel kernel_of_part<2>(int nphi, int h);
template <> Kernel kernel_of_part<3>(int nphi, int h);
template <> Kernel kernel_of_part<4>(int nphi, int h);
template <> Kernel kernel_of_part<5>(int nphi, int h);
inline Kernel kernel_for(int nphi, int h) {
  Kernel k = nullptr;
  for (Kernel (*part)(int, int) : {kernel_of_part<0>, kernel_of_part<1>, kernel_of_part<2>, kernel_of_part<3>,
                                   kernel_of_part<4>, kernel_of_part<5>})
    if (!k) k = part(nphi, h);
  return k;
}
// Dynamic shared memory of a block of `teams` teams: matrix fragments, slots, barriers, per team F and exchange.
inline std::size_t smem_bytes(int n_rot, int nphi, int h, int frags, int teams) {
  return 256u * static_cast<std::size_t>(frags) + sizeof(int4) * static_cast<std::size_t>(nphi) +
         8u * static_cast<std::size_t>((teams + 1) & ~1) + teams * team_bytes(n_rot, nphi, h);
}

}  // namespace pot5

// exp(i A) - 1 and the modulus corrections (exp_potential_kernel) in the order of potential5, from n_reps blocks of
// ntheta x nphi values of V, phi fastest.
static __global__ void exp_pairs_kernel(const double* __restrict__ v, float4* __restrict__ table, __half2* __restrict__ mods,
                                        long long n_reps, int n_theta, int n_phi, int pairs, int group, double dt) {
  const long long n = n_reps * n_phi * pairs;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int tp = static_cast<int>(i % pairs);
    const long long q = i / pairs;
    const int p = static_cast<int>(q % n_phi);
    const long long rep = q / n_phi;
    float2 g[2];
    __half m[2];
    for (int k = 0; k < 2; ++k) {
      const int th = 2 * tp + k;
      g[k] = make_float2(0.0f, 0.0f);
      m[k] = __float2half(0.0f);
      if (th < n_theta) exp_entry(v[(rep * n_theta + th) * n_phi + p], dt, g[k], m[k]);
    }
    table[i] = make_float4(g[0].x, g[1].x, g[0].y, g[1].y);
    mods[rep * n_phi * pairs + (p / group) * group * pairs + tp * group + p % group] = __halves2half2(m[0], m[1]);
  }
}

}  // namespace spo
