// Potential step of the interaction region, FP64 form, with both theta contractions on the FP64 tensor cores
// (mma.m8n8k4.f64; src/propagation/potential_operator.cpp:84-135, angular_transform.cpp:54-114).
//
// A team of 128 threads owns GROUPS = 2 / H groups of 8 (x, y) columns at a time (H = 2 for ntheta <= 16, 1 for
// ntheta <= 8), i.e. 128 phi lines (column, theta), one per thread; X[slot][column][theta] in shared memory:
//   - forward: X_m[c, theta] = sum_J F[c, J] M_m[theta, J], one warp per (phi slot, group): the columns are the rows of
//     the product and come straight from global memory (every value of psi is read once, 64 bytes per column and
//     fragment; the next slot's are in flight during the products), real and imaginary parts share the matrix;
//   - phi: every thread takes its line into registers: DFT, exp(i A), inverse DFT, back in place. exp(i A) is stored
//     [phi][theta] per (Z, r) point and representative, so that a warp reads whole rows;
//   - back: out[c, J] = sum_theta X[c, theta] M_m[theta, J], one warp per (slot, 8 values of J, group), times
//     rot(dt/2), stored 64 bytes per column.
// psi comes scaled by the absorbers and rot(dt/2) (the xy pass). The projection is projection_finalize_kernel's.
//
// What bounds it: on configuration 2 the FP64 pipe (shared by the tensor products and the transforms) needs ~150
// multiply-adds per value of psi with the padding of the fragments (2.1 ms), HBM 16.9 GB (2.6 ms). A register-tiled
// form on FMAs took 10.8 ms with 8 warps per SM: each term of its contractions loads its operands from shared memory.
// On Z 128, r 48, 12 x 12 (9.5 GB) the FMA form took 6.05 ms, this one with every load where its value is needed 3.77
// (long-scoreboard stalls 2.7 of 7.7 cycles per issue), with psi and exp(i A) a phase ahead 3.00 (3.2 TB/s).
#pragma once

#include "spo_pot5.cuh"

namespace spo {

namespace pot4d {
// Threads per block: a line takes 4 nphi registers.
constexpr int threads_of(int nphi) { return nphi > 20 ? 256 : nphi > 16 ? 384 : 512; }
constexpr int kTeam = 128;
// 256 threads leave a thread 255 registers: while the lines are not in registers they hold psi of the team's next item (the
// 8 tasks of a warp; with one theta tile and two column groups they would be 16).
constexpr bool ahead_of(int nphi, int h) { return threads_of(nphi) == 256 && h == 2; }
}  // namespace pot4d

struct Pot4dArgs {
  PotArgs<double> p;
  const double2* table;    // exp(i A): [(Z, r) point][representative][phi][theta]
  const double* frags;     // matrix fragments of 32 values: the forward ones, then the transposed ones
  int n_fwd, n_back;
  const int4* slots;       // per phi slot: first irot, J count, first forward fragment, first transposed fragment
  const int* fwd_tasks;    // slots with basis functions, longest first, then the empty ones
  const int2* back_tasks;  // (slot, J octet)
  int n_back_tasks;
  const double2* rot;      // (ir, irot): rot(dt/2)
  const uint8_t* phi_map;  // n_xy * nphi, or null (no symmetry)
  int n_cols, n_items;
};

#ifdef __CUDACC__

// Columns (e.g. column c's theta) of X: theta t of column c at position t ^ (4 (c & 1)), so that the 2 x 4 values of a
// quarter-warp's fragment access fall on distinct banks.
template <int NPHI, int H>
__global__ void __launch_bounds__(pot4d::threads_of(NPHI), 1) potential4_dmma_kernel(Pot4dArgs g) {
  using pot5::dmma;
  constexpr int GROUPS = 2 / H, COLS = 8 * GROUPS, NT = 8 * H;
  constexpr int SLOT = COLS * NT;  // 128 values per slot
  static_assert(SLOT == pot4d::kTeam, "one line per thread");
  const PotArgs<double>& a = g.p;
  const int n_rot = a.n_rot, n_xy = a.n_xy, nr = a.nr, i0 = a.initial_channel;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const int team = threadIdx.x / pot4d::kTeam, teams = blockDim.x / pot4d::kTeam;
  const int tid = threadIdx.x % pot4d::kTeam, warp = tid / 32, lane = tid % 32;
  constexpr bool AHEAD = pot4d::ahead_of(NPHI, H);
  double2* const X = reinterpret_cast<double2*>(smem_raw) + team * (NPHI * SLOT + n_rot);
  double2* const rot_row = X + NPHI * SLOT;  // rot(dt/2) at the item's r point
  double* const mats = reinterpret_cast<double*>(reinterpret_cast<double2*>(smem_raw) + teams * (NPHI * SLOT + n_rot));
  int4* const slots = reinterpret_cast<int4*>(mats + 32 * (g.n_fwd + g.n_back));
  int2* const tiles = reinterpret_cast<int2*>(slots + NPHI);
  int* const order = reinterpret_cast<int*>(tiles + g.n_back_tasks);
  for (int k = threadIdx.x; k < 32 * (g.n_fwd + g.n_back); k += blockDim.x) mats[k] = g.frags[k];
  for (int k = threadIdx.x; k < NPHI; k += blockDim.x) {
    slots[k] = g.slots[k];
    order[k] = g.fwd_tasks[k];
  }
  for (int k = threadIdx.x; k < g.n_back_tasks; k += blockDim.x) tiles[k] = g.back_tasks[k];
  __syncthreads();
  auto team_sync = [&] { asm volatile("barrier.cta.sync %0, 128;" ::"r"(1 + team) : "memory"); };
  const double* const mf = mats + lane;
  const double* const mb = mats + 32 * g.n_fwd + lane;
  const int c = lane >> 2, t = lane & 3, sw = 4 * (c & 1);
  // this thread's phi line
  const int line_c = tid / NT, line_t = tid % NT;
  const int line_at = line_c * NT + (line_t ^ (4 * (line_c & 1)));
  const int step = gridDim.x * teams;

  constexpr int TASKS = NPHI * GROUPS, MINE = (TASKS + 3) / 4;
  auto load = [&](int task, int col0, double2 (&u)[4], int4& s) {
    s = slots[order[task / GROUPS]];
    const int col = col0 + (task % GROUPS) * 8 + c;
    const double2* const p = a.psi + static_cast<long long>(min(col, g.n_cols - 1)) * n_rot;
#pragma unroll
    for (int k = 0; k < 4; ++k)
      u[k] = 4 * k < s.y ? p[min(s.x + 4 * k + t, n_rot - 1)] : make_double2(0.0, 0.0);
  };
  double2 mine[AHEAD ? MINE : 1][4] = {};
  auto load_mine = [&](int item) {
    static_for<0, AHEAD ? MINE : 0>([&](auto k) {
      int4 s;
      load(min(warp + 4 * SPO_CV(k), TASKS - 1), item * COLS, mine[SPO_CV(k)], s);
    });
  };

  int item = blockIdx.x * teams + team;
  if (AHEAD && item < g.n_items) load_mine(item);
  for (; item < g.n_items; item += step) {
    const int col0 = item * COLS;
    // the next item's columns and exp(i A) rows into L2
    {
      const int col = col0 + step * COLS + lane;
      if (warp == 0 && lane < COLS && item + step < g.n_items && col < g.n_cols) {
        const int izr = col / n_xy, ixy = col - izr * n_xy;
        const long long e = (static_cast<long long>(izr) * a.n_rep + (g.phi_map ? __ldg(a.rep_of + ixy) : ixy)) * NPHI * a.n_theta;
        pot5::prefetch_l2(g.table + e, static_cast<uint32_t>(NPHI * a.n_theta * sizeof(double2)));
        pot5::prefetch_l2(a.psi + static_cast<long long>(col) * n_rot, static_cast<uint32_t>(n_rot * sizeof(double2)));
      }
    }
    // the item's row of rot(dt/2), if it lies at one point
    const int izr0 = col0 / n_xy;
    const bool row = min(col0 + COLS - 1, g.n_cols - 1) / n_xy == izr0;
    if (row)
      for (int k = tid; k < n_rot; k += pot4d::kTeam) rot_row[k] = g.rot[(izr0 % nr) * n_rot + k];

    // ---- forward: tasks (slot, group)
    auto multiply = [&](int task, double2 (&u)[4], const int4& s) {
      const int slot = order[task / GROUPS], grp = task % GROUPS;
      const int col = col0 + grp * 8 + c;
      const int nj = s.y;
      // the specular wave into the initial channel (potential_operator.cpp:116-123)
      if (i0 >= s.x && i0 < s.x + nj && ((i0 - s.x) & 3) == t && col < g.n_cols) {
        const int izr = col / n_xy, ixy = col - izr * n_xy;
        const double2 v = cmul(g.rot[(izr % nr) * n_rot + i0], cmul(a.sp2sc[ixy], a.chi[izr]));
#pragma unroll
        for (int k = 0; k < 4; ++k)
          u[k] = cadd(u[k], k == (i0 - s.x) >> 2 ? v : make_double2(0.0, 0.0));
      }
      double r[H][2], q[H][2];
#pragma unroll
      for (int h = 0; h < H; ++h) r[h][0] = r[h][1] = q[h][0] = q[h][1] = 0.0;
      const double* m = mf + 32 * s.z;
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (4 * k < nj) {
#pragma unroll
          for (int h = 0; h < H; ++h) {
            const double w = m[32 * (k * H + h)];
            dmma(r[h][0], r[h][1], u[k].x, w);
            dmma(q[h][0], q[h][1], u[k].y, w);
          }
        }
      const double2* const p = a.psi + static_cast<long long>(min(col, g.n_cols - 1)) * n_rot;
#pragma unroll 1
      for (int k = 4; 4 * k < nj; ++k) {  // more than 16 J
        const int j = s.x + 4 * k + t;
        double2 v = p[min(j, n_rot - 1)];
        if (j == i0 && col < g.n_cols) {
          const int izr = col / n_xy, ixy = col - izr * n_xy;
          v = cadd(v, cmul(g.rot[(izr % nr) * n_rot + i0], cmul(a.sp2sc[ixy], a.chi[izr])));
        }
#pragma unroll
        for (int h = 0; h < H; ++h) {
          const double w = m[32 * (k * H + h)];
          dmma(r[h][0], r[h][1], v.x, w);
          dmma(q[h][0], q[h][1], v.y, w);
        }
      }
      double2* const x = X + slot * SLOT + (grp * 8 + c) * NT;
#pragma unroll
      for (int h = 0; h < H; ++h) {
        x[8 * h + (t ^ sw)] = make_double2(r[h][0], q[h][0]);
        x[8 * h + ((t + 4) ^ sw)] = make_double2(r[h][1], q[h][1]);
      }
    };
    if constexpr (AHEAD) {
      static_for<0, MINE>([&](auto k) {
        const int task = warp + 4 * SPO_CV(k);
        if (task < TASKS) multiply(task, mine[SPO_CV(k)], slots[order[task / GROUPS]]);
      });
    } else {  // the fragments of the next task requested before the products of this one
      double2 u[4] = {}, un[4] = {};
      int4 s, sn = make_int4(0, 0, 0, 0);
      load(warp, col0, u, s);
#pragma unroll 1
      for (int task = warp; task < TASKS; task += 4) {
        if (task + 4 < TASKS) load(task + 4, col0, un, sn);
        multiply(task, u, s);
        s = sn;
#pragma unroll
        for (int k = 0; k < 4; ++k) u[k] = un[k];
      }
    }
    team_sync();

    // ---- phi transform, exp(i A), inverse phi transform
    {
      const int col = col0 + line_c;
      if (col < g.n_cols && line_t < a.n_theta) {
        const int izr = col / n_xy, ixy = col - izr * n_xy;
        const double2* const e =
            g.table + (static_cast<long long>(izr) * a.n_rep + (g.phi_map ? __ldg(a.rep_of + ixy) : ixy)) * NPHI * a.n_theta + line_t;
        double2 x[NPHI];
        constexpr int EARLY = AHEAD ? NPHI / 2 : 0;  // entries requested before the transform
        double2 ex[EARLY > 0 ? EARLY : 1];
        if (g.phi_map == nullptr) static_for<0, EARLY>([&](auto p) { ex[p] = __ldg(e + SPO_CV(p) * a.n_theta); });
        static_for<0, NPHI>([&](auto p) { x[p] = X[SPO_CV(p) * SLOT + line_at]; });
        rdft<NPHI, +1>(x);
        if (g.phi_map == nullptr) {
          static_for<0, EARLY>([&](auto p) {
            x[p] = cmul(ex[p], x[p]);
            ex[p] = __ldg(e + (SPO_CV(p) + EARLY) * a.n_theta);
          });
          static_for<EARLY, 2 * EARLY>([&](auto p) { x[p] = cmul(ex[SPO_CV(p) - EARLY], x[p]); });
          static_for<2 * EARLY, NPHI>([&](auto p) { x[p] = cmul(__ldg(e + SPO_CV(p) * a.n_theta), x[p]); });
        } else {
          const uint8_t* const map = g.phi_map + ixy * NPHI;
          static_for<0, NPHI>([&](auto p) { x[p] = cmul(__ldg(e + __ldg(map + SPO_CV(p)) * a.n_theta), x[p]); });
        }
        rdft<NPHI, -1>(x);
        static_for<0, NPHI>([&](auto p) { X[SPO_CV(p) * SLOT + line_at] = x[p]; });
      }
    }
    team_sync();

    // ---- back: tasks (slot, 8 values of J, group); psi of the next item on its way
    if (AHEAD) load_mine(min(item + step, g.n_items - 1));  // (the last one's again: every value of `mine` is defined anew)
#pragma unroll 1
    for (int task = warp; task < g.n_back_tasks * GROUPS; task += 4) {
      const int2 tile = tiles[task / GROUPS];
      const int grp = task % GROUPS;
      const int4 s4 = slots[tile.x];
      const int col = col0 + grp * 8 + c;
      const int ir = (min(col, g.n_cols - 1) / n_xy) % nr;
      const int j = 8 * tile.y + t;
      const double2* const w = (row ? rot_row : g.rot + ir * n_rot) + s4.x;
      const double2 wa = w[min(j, s4.y - 1)], wb = w[min(j + 4, s4.y - 1)];
      const double2* const x = X + tile.x * SLOT + (grp * 8 + c) * NT;
      const double* const m = mb + 32 * (s4.w + tile.y * 2 * H);
      double r0 = 0, r1 = 0, q0 = 0, q1 = 0;
#pragma unroll
      for (int k = 0; k < 2 * H; ++k) {
        const double2 v = x[(8 * (k / 2)) + ((t + 4 * (k % 2)) ^ sw)];
        const double f = m[32 * k];
        dmma(r0, r1, v.x, f);
        dmma(q0, q1, v.y, f);
      }
      if (col < g.n_cols) {
        double2* const out = a.psi + static_cast<long long>(col) * n_rot + s4.x;
        if (j < s4.y) out[j] = cmul(wa, make_double2(r0, q0));
        if (j + 4 < s4.y) out[j + 4] = cmul(wb, make_double2(r1, q1));
      }
    }
    team_sync();  // X is read before the next item's forward products write it
  }
}

#endif  // __CUDACC__

namespace pot4d {
using Kernel = void (*)(Pot4dArgs);
template <int PART>
Kernel kernel_of_part(int nphi, int h);
template <> Kernel kernel_of_part<0>(int nphi, int h);
template <> Kernel kernel_of_part<1>(int nphi, int h);
template <> Kernel kernel_of_part<2>(int nphi, int h);
template <> Kernel kernel_of_part<3>(int nphi, int h);
inline Kernel kernel_for(int nphi, int h) {
  Kernel k = nullptr;
  for (Kernel (*part)(int, int) : {kernel_of_part<0>, kernel_of_part<1>, kernel_of_part<2>, kernel_of_part<3>})
    if (!k) k = part(nphi, h);
  return k;
}
inline std::size_t smem_bytes(int n_rot, int nphi, int frags, int n_back_tasks, int teams) {
  return (2048u * static_cast<std::size_t>(nphi) + 16u * static_cast<std::size_t>(n_rot)) * teams + 256u * static_cast<std::size_t>(frags) +
         (sizeof(int4) + sizeof(int)) * static_cast<std::size_t>(nphi) + sizeof(int2) * static_cast<std::size_t>(n_back_tasks);
}
}  // namespace pot4d

// exp(i A) (exp_potential_kernel) in the order of potential4_dmma_kernel, from n_reps blocks of ntheta x nphi values of V,
// phi fastest.
static __global__ void exp_rows_kernel(const double* __restrict__ v, double2* __restrict__ table, long long n_reps,
                                       int n_theta, int n_phi, double dt) {
  const long long n = n_reps * n_phi * n_theta;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int th = static_cast<int>(i % n_theta);
    const long long q = i / n_theta;
    double sn, cs;
    sincos(-v[(q / n_phi * n_theta + th) * n_phi + q % n_phi] * dt, &sn, &cs);
    table[i] = make_double2(cs, sn);
  }
}

}  // namespace spo
