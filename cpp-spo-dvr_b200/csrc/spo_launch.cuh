// Launchers of the register-DFT kernels and of the potential kernels (declared in spo_host.cuh), apart from the
// host class so that the kernel families compile in parallel (spo_launch.cu).
#pragma once

#include "spo_host.cuh"

namespace spo_host {

// ---------------------------------------------------------------------------------------------
// Launchers of the register-DFT kernels for the sizes they are instantiated for. Each returns
// false for other sizes; the caller then uses the general shared-memory Stockham kernels.
// ---------------------------------------------------------------------------------------------
// Sets a kernel's dynamic shared-memory limit once per device (the attribute is per device context).
template <typename K>
void allow_smem(K kernel, std::size_t bytes, unsigned long long& done_mask, const char* what) {
  int dev = 0;
  check_cuda(cudaGetDevice(&dev), "cudaGetDevice");
  if (dev < 64 && (done_mask >> dev & 1ull)) return;
  check_cuda(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes)), what);
  if (dev < 64) done_mask |= 1ull << dev;
}

// Blocks of a persistent kernel: the SMs times the blocks that fit on one (looked up once per kernel).
template <typename K>
long long persistent_blocks(K kernel, int threads, std::size_t smem, int& cached) {
  if (cached <= 0) {
    int dev = 0, sms = 0, per_sm = 0;
    check_cuda(cudaGetDevice(&dev), "cudaGetDevice");
    check_cuda(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev), "SM count");
    check_cuda(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem), "occupancy");
    cached = std::max(1, sms * per_sm);
  }
  return cached;
}

template <typename T, int N1, int N2, int TB>
bool launch_axis2_tb(const spo::Axis2Args<T>& a, long long outer, cudaStream_t stream) {
  constexpr int NS = N1 > N2 ? N1 : N2;
  constexpr int N = N1 * N2;
  // the tile, then the factors (mixed form: their parts, spo::fmul_t) and the twiddles (mixed form: and their low parts)
  const std::size_t smem =
      sizeof(spo::Vec<T>) * (static_cast<std::size_t>(N) * TB + (sizeof(T) == 4 ? spo::kFactorParts + 2 : 2) * N);
  static unsigned long long configured = 0;
  allow_smem(spo::axis2_kernel<T, N1, N2, TB>, smem, configured, "axis2 smem");
  if (a.persistent && a.window == 0) {
    static unsigned long long configured_p = 0;
    static int blocks_p = 0;
    allow_smem(spo::axis2p_kernel<T, N1, N2, TB>, smem, configured_p, "axis2p smem");
    const long long lane_blocks = (a.inner + TB - 1) / TB;
    const long long n_tiles = outer * lane_blocks;
    const long long grid = std::min(n_tiles, persistent_blocks(spo::axis2p_kernel<T, N1, N2, TB>, TB * NS, smem, blocks_p));
    spo::axis2p_kernel<T, N1, N2, TB><<<static_cast<unsigned>(grid), TB * NS, smem, stream>>>(a, lane_blocks, n_tiles);
    return true;
  }
  if constexpr (N2 == 2 * N1) {
    if (a.balanced && a.window == 0) {
      static unsigned long long configured_b = 0;
      allow_smem(spo::axis2b_kernel<T, N1, N2, TB>, smem, configured_b, "axis2b smem");
      const dim3 grid(static_cast<unsigned>((a.inner + TB - 1) / TB), static_cast<unsigned>(outer));
      spo::axis2b_kernel<T, N1, N2, TB><<<grid, TB * N1, smem, stream>>>(a);
      return true;
    }
  }
  if (a.window > 0) {  // lane windows: groups x ceil(window / TB) blocks
    spo::Axis2Args<T> w = a;
    w.blocks_per_group = static_cast<int>((a.window + TB - 1) / TB);
    const dim3 grid(static_cast<unsigned>(a.groups * w.blocks_per_group), static_cast<unsigned>(outer));
    spo::axis2_kernel<T, N1, N2, TB><<<grid, TB * NS, smem, stream>>>(w);
    return true;
  }
  const dim3 grid(static_cast<unsigned>((a.inner + TB - 1) / TB), static_cast<unsigned>(outer));
  spo::axis2_kernel<T, N1, N2, TB><<<grid, TB * NS, smem, stream>>>(a);
  return true;
}

// Tile width (batch lanes per block): 32 lanes when a line has at most 8 sub-rows; for more sub-rows
// 16 lanes by default, or 8 or 32 lanes as the autotuner chose.
template <typename T, int N1, int N2>
bool launch_axis2_n(const spo::Axis2Args<T>& a, long long outer, cudaStream_t stream) {
  constexpr int NS = N1 > N2 ? N1 : N2;
  if constexpr (NS <= 8) {
    return launch_axis2_tb<T, N1, N2, 32>(a, outer, stream);
  } else {
    if (a.tile == 8) return launch_axis2_tb<T, N1, N2, 8>(a, outer, stream);
    if (a.tile == 32) return launch_axis2_tb<T, N1, N2, 32>(a, outer, stream);
    return launch_axis2_tb<T, N1, N2, 16>(a, outer, stream);
  }
}

template <typename T, int N1, int N2, int LT>
bool launch_axis2_pfa_n(const spo::Axis2Args<T>& a, long long outer, cudaStream_t stream) {
  constexpr int TB = 32, N = N1 * N2;
  const std::size_t smem = sizeof(spo::Vec<T>) * (static_cast<std::size_t>(N) * TB + (sizeof(T) == 4 ? spo::kFactorParts : 1) * N);
  static unsigned long long configured = 0;
  allow_smem(spo::axis2pfa_kernel<T, N1, N2, TB, LT>, smem, configured, "axis2pfa smem");
  spo::Axis2Args<T> w = a;
  unsigned blocks_x;
  if (a.window > 0) {
    w.blocks_per_group = static_cast<int>((a.window + TB - 1) / TB);
    blocks_x = static_cast<unsigned>(a.groups * w.blocks_per_group);
  } else {
    blocks_x = static_cast<unsigned>((a.inner + TB - 1) / TB);
  }
  spo::axis2pfa_kernel<T, N1, N2, TB, LT><<<dim3(blocks_x, static_cast<unsigned>(outer)), TB * LT, smem, stream>>>(w);
  return true;
}
template <typename T>
bool launch_axis2_pfa(int n, const spo::Axis2Args<T>& a, long long outer, cudaStream_t stream) {
  switch (n) {
    case 24: return launch_axis2_pfa_n<T, 3, 8, 4>(a, outer, stream);
    case 40: return launch_axis2_pfa_n<T, 5, 8, 8>(a, outer, stream);
    case 48: return launch_axis2_pfa_n<T, 3, 16, 4>(a, outer, stream);
    case 56: return launch_axis2_pfa_n<T, 7, 8, 8>(a, outer, stream);
    case 80: return launch_axis2_pfa_n<T, 5, 16, 8>(a, outer, stream);
    case 112: return launch_axis2_pfa_n<T, 7, 16, 8>(a, outer, stream);
    default: return false;
  }
}

template <typename T>
bool launch_axis2(int n, const spo::Axis2Args<T>& a, long long outer, cudaStream_t stream) {
  if (a.factor_pfa && !a.persistent) return launch_axis2_pfa<T>(n, a, outer, stream);
  switch (n) {
    // N = N1 N2 with N2 >= N1: the first level, which streams the tile in from HBM, uses every thread.
    case 24: return launch_axis2_n<T, 4, 6>(a, outer, stream);
    case 32: return launch_axis2_n<T, 4, 8>(a, outer, stream);
    case 40: return launch_axis2_n<T, 5, 8>(a, outer, stream);
    case 48: return launch_axis2_n<T, 6, 8>(a, outer, stream);
    case 56: return launch_axis2_n<T, 7, 8>(a, outer, stream);
    case 64: return launch_axis2_n<T, 8, 8>(a, outer, stream);
    case 80: return launch_axis2_n<T, 8, 10>(a, outer, stream);
    case 96: return launch_axis2_n<T, 8, 12>(a, outer, stream);
    case 112: return launch_axis2_n<T, 7, 16>(a, outer, stream);
    case 128: return launch_axis2_n<T, 8, 16>(a, outer, stream);
    case 160: return launch_axis2_n<T, 10, 16>(a, outer, stream);
    case 176: return launch_axis2_n<T, 11, 16>(a, outer, stream);
    case 192: return launch_axis2_n<T, 12, 16>(a, outer, stream);
    case 224: return launch_axis2_n<T, 14, 16>(a, outer, stream);
    case 256: return launch_axis2_n<T, 16, 16>(a, outer, stream);
    default: return false;
  }
}
template <typename T, int NX, int NY, int TB>
void launch_xy2_tb(const spo::XyArgs<T>& a, long long n_zr, cudaStream_t stream) {
  constexpr int NS = NX > NY ? NX : NY;
  const std::size_t smem =
      sizeof(spo::Vec<T>) * (static_cast<std::size_t>(NX * NY) * TB + (sizeof(T) == 4 ? spo::kFactorParts : 1) * NX * NY);
  if (a.persistent) {
    static unsigned long long configured_p = 0;
    static int blocks_p = 0;
    allow_smem(spo::xy2p_kernel<T, NX, NY, TB>, smem, configured_p, "xy2p smem");
    const long long rot_tiles = (a.n_rot + TB - 1) / TB;
    const long long n_tiles = n_zr * rot_tiles;
    const long long grid = std::min(n_tiles, persistent_blocks(spo::xy2p_kernel<T, NX, NY, TB>, TB * NS, smem, blocks_p));
    spo::xy2p_kernel<T, NX, NY, TB><<<static_cast<unsigned>(grid), TB * NS, smem, stream>>>(a, rot_tiles, n_tiles);
    return;
  }
  static unsigned long long configured = 0;
  allow_smem(spo::xy2_kernel<T, NX, NY, TB>, smem, configured, "xy2 smem");
  const dim3 grid(static_cast<unsigned>((a.n_rot + TB - 1) / TB), static_cast<unsigned>(n_zr));
  spo::xy2_kernel<T, NX, NY, TB><<<grid, TB * NS, smem, stream>>>(a);
}

template <typename T, int NX, int NY>
void launch_xy2_n(const spo::XyArgs<T>& a, long long n_zr, cudaStream_t stream) {
  constexpr int NS = NX > NY ? NX : NY;
  if constexpr (NS <= 8) {
    launch_xy2_tb<T, NX, NY, 32>(a, n_zr, stream);
  } else {
    if (a.tile == 8) launch_xy2_tb<T, NX, NY, 8>(a, n_zr, stream);
    else if (a.tile == 32) launch_xy2_tb<T, NX, NY, 32>(a, n_zr, stream);
    else launch_xy2_tb<T, NX, NY, 16>(a, n_zr, stream);
  }
}

template <typename T>
bool launch_xy2(const spo::XyArgs<T>& a, long long n_zr, cudaStream_t stream) {
  if (a.nx != a.ny) return false;
  switch (a.nx) {
    case 2: launch_xy2_n<T, 2, 2>(a, n_zr, stream); return true;
    case 4: launch_xy2_n<T, 4, 4>(a, n_zr, stream); return true;
    case 6: launch_xy2_n<T, 6, 6>(a, n_zr, stream); return true;
    case 8: launch_xy2_n<T, 8, 8>(a, n_zr, stream); return true;
    case 12: launch_xy2_n<T, 12, 12>(a, n_zr, stream); return true;
    case 16: launch_xy2_n<T, 16, 16>(a, n_zr, stream); return true;
    default: return false;
  }
}

template <typename T, int NPHI, int CB>
void launch_pot2_n(const spo::Pot2Args<T>& a, unsigned blocks, std::size_t smem, cudaStream_t stream) {
  // The shared memory depends on the case's sizes, not only on the instantiation: allow the device's
  // maximum, so that every case with this instantiation can launch.
  static unsigned long long configured = 0;
  allow_smem(spo::potential2_kernel<T, NPHI, CB>, smem_optin_bytes(), configured, "potential2 smem");
  spo::potential2_kernel<T, NPHI, CB><<<blocks, 128, smem, stream>>>(a);
}

template <typename T, int NPHI>
void launch_pot2_phi(const spo::Pot2Args<T>& a, unsigned blocks, std::size_t smem, cudaStream_t stream) {
  switch (a.cb) {
    case 32: launch_pot2_n<T, NPHI, 32>(a, blocks, smem, stream); break;
    case 8: launch_pot2_n<T, NPHI, 8>(a, blocks, smem, stream); break;
    default: launch_pot2_n<T, NPHI, 4>(a, blocks, smem, stream); break;
  }
}

template <typename T>
void launch_pot2(int nphi, const spo::Pot2Args<T>& a, unsigned blocks, std::size_t smem, cudaStream_t stream) {
  switch (nphi) {
    case 6: launch_pot2_phi<T, 6>(a, blocks, smem, stream); break;
    case 8: launch_pot2_phi<T, 8>(a, blocks, smem, stream); break;
    case 10: launch_pot2_phi<T, 10>(a, blocks, smem, stream); break;
    case 12: launch_pot2_phi<T, 12>(a, blocks, smem, stream); break;
    case 16: launch_pot2_phi<T, 16>(a, blocks, smem, stream); break;
    case 20: launch_pot2_phi<T, 20>(a, blocks, smem, stream); break;
    case 24: launch_pot2_phi<T, 24>(a, blocks, smem, stream); break;
    case 28: launch_pot2_phi<T, 28>(a, blocks, smem, stream); break;
    case 30: launch_pot2_phi<T, 30>(a, blocks, smem, stream); break;
    case 32: launch_pot2_phi<T, 32>(a, blocks, smem, stream); break;
    default: break;
  }
}
template <typename T, int NPHI, int CB>
void launch_pot3_n(const spo::Pot2Args<T>& a, dim3 grid, unsigned threads, std::size_t smem, cudaStream_t stream) {
  static unsigned long long configured = 0;
  allow_smem(spo::potential3_kernel<T, NPHI, CB>, smem_optin_bytes(), configured, "potential3 smem");
  spo::potential3_kernel<T, NPHI, CB><<<grid, threads, smem, stream>>>(a);
}

template <typename T, int NPHI>
void launch_pot3_phi(const spo::Pot2Args<T>& a, dim3 grid, unsigned threads, std::size_t smem, cudaStream_t stream) {
  if (a.cb == 16) launch_pot3_n<T, NPHI, 16>(a, grid, threads, smem, stream);
  else launch_pot3_n<T, NPHI, 8>(a, grid, threads, smem, stream);
}

template <typename T>
void launch_pot3(int nphi, const spo::Pot2Args<T>& a, dim3 grid, unsigned threads, std::size_t smem,
                 cudaStream_t stream) {
  switch (nphi) {
    case 6: launch_pot3_phi<T, 6>(a, grid, threads, smem, stream); break;
    case 8: launch_pot3_phi<T, 8>(a, grid, threads, smem, stream); break;
    case 10: launch_pot3_phi<T, 10>(a, grid, threads, smem, stream); break;
    case 12: launch_pot3_phi<T, 12>(a, grid, threads, smem, stream); break;
    case 16: launch_pot3_phi<T, 16>(a, grid, threads, smem, stream); break;
    case 20: launch_pot3_phi<T, 20>(a, grid, threads, smem, stream); break;
    case 24: launch_pot3_phi<T, 24>(a, grid, threads, smem, stream); break;
    case 28: launch_pot3_phi<T, 28>(a, grid, threads, smem, stream); break;
    case 30: launch_pot3_phi<T, 30>(a, grid, threads, smem, stream); break;
    case 32: launch_pot3_phi<T, 32>(a, grid, threads, smem, stream); break;
    default: break;
  }
}

template <typename T>
Pot4Kernel<T> pot4_kernel_for(int nphi, int nt) {  // the mixed form's; FP64 has potential4_dmma_kernel
  if constexpr (sizeof(T) == 4) {
    if (nt == 16 && nphi == 32) return spo::potential4_kernel<T, 32, 16, 8>;
    if (nt == 16 && nphi == 16) return spo::potential4_kernel<T, 16, 16, 8>;
    if (nt == 8 && nphi == 16) return spo::potential4_kernel<T, 16, 8, 16>;
    if (nt == 8 && nphi == 32) return spo::potential4_kernel<T, 32, 8, 16>;
    if (nt == 4 && nphi == 8) return spo::potential4_kernel<T, 8, 4, 32>;
    if (nt == 4 && nphi == 12) return spo::potential4_kernel<T, 12, 4, 32>;  // C6v grids
  }
  return nullptr;
}

template <typename T>
using KinKernel = void (*)(spo::KinArgs<typename spo::KinStored<T>::type>);
template <typename T>
KinKernel<T> kin_kernel_for(int map, int n1, int n2) {  // kin_preferred, kin_preferred_xy, kin_wide_xy
  constexpr bool mixed = std::is_same_v<T, float>, fp64 = std::is_same_v<T, double>, wide = std::is_same_v<T, spo::Wide>;
  if constexpr (wide) {
    if (map == spo::kXy && n1 == 6 && n2 == 6) return spo::kin_kernel<T, spo::kXy, 6, 6>;
  } else if (map == spo::kTwiddle) {
    if constexpr (fp64)
      if (n1 == 8 && n2 == 8) return spo::kin_kernel<T, spo::kTwiddle, 8, 8>;
    if constexpr (mixed)
      if (n1 == 8 && n2 == 12) return spo::kin_kernel<T, spo::kTwiddle, 8, 12>;
    if (n1 == 8 && n2 == 16) return spo::kin_kernel<T, spo::kTwiddle, 8, 16>;
    if (n1 == 12 && n2 == 16) return spo::kin_kernel<T, spo::kTwiddle, 12, 16>;
    if (n1 == 16 && n2 == 16) return spo::kin_kernel<T, spo::kTwiddle, 16, 16>;
  } else if (map == spo::kPrime) {
    if (n1 == 3 && n2 == 16) return spo::kin_kernel<T, spo::kPrime, 3, 16>;
    if (n1 == 11 && n2 == 16) return spo::kin_kernel<T, spo::kPrime, 11, 16>;
    if constexpr (mixed)
      if (n1 == 5 && n2 == 32) return spo::kin_kernel<T, spo::kPrime, 5, 32>;
    if (n1 == 7 && n2 == 32) return spo::kin_kernel<T, spo::kPrime, 7, 32>;
  } else if (map == spo::kXy && n1 == n2) {
    if (n1 == 2) return spo::kin_kernel<T, spo::kXy, 2, 2>;
    if (n1 == 4) return spo::kin_kernel<T, spo::kXy, 4, 4>;
    if constexpr (fp64)
      if (n1 == 6) return spo::kin_kernel<T, spo::kXy, 6, 6>;
    if (n1 == 8) return spo::kin_kernel<T, spo::kXy, 8, 8>;
    if (n1 == 12) return spo::kin_kernel<T, spo::kXy, 12, 12>;
    if (n1 == 16) return spo::kin_kernel<T, spo::kXy, 16, 16>;
  }
  if constexpr (mixed) throw SpoError(SPO_ERR_STATE, "kin_kernel: no pair kernel of these sizes");
  else
    return map == spo::kTwiddle ? spo::kin_kernel<T, spo::kTwiddle, 0, 0>
           : map == spo::kPrime ? spo::kin_kernel<T, spo::kPrime, 0, 0>
           : map == spo::kXy    ? spo::kin_kernel<T, spo::kXy, 0, 0>
                                : spo::kin_kernel<T, spo::kXyShift, 0, 0>;
}

// Threads per line: the number that wastes the fewest thread slots over the two levels (N2 lines of N1 points, then N1 of
// N2) in whole warps, among those that keep about 14 warps per SM beside the tiles' shared memory.
template <typename T>
KinLaunch<typename spo::KinStored<T>::type> kin_configure(int map, int n1, int n2, bool unit, int lanes_per_tile, long long window) {
  KinLaunch<typename spo::KinStored<T>::type> l;
  l.lanes = spo::KinLine<T>::lanes;
  l.kernel = kin_kernel_for<T>(map, n1, n2);
  while ((spo::KinLine<T>::lanes << (l.log_lines + 1)) <= lanes_per_tile) ++l.log_lines;
  while (l.log_lines > 0 && (static_cast<long long>(spo::KinLine<T>::lanes) << (l.log_lines - 1)) >= window) --l.log_lines;
  const std::size_t n = static_cast<std::size_t>(n1) * n2;
  auto smem_of = [&](int log_lines) { return 16 * (spo::kin_words<T>(map, n1 * n2, unit) + (2 * n << log_lines)); };
  while (l.log_lines > 0 && smem_of(l.log_lines) > static_cast<std::size_t>(smem_optin_bytes())) --l.log_lines;
  const int lines = 1 << l.log_lines, limit = spo::kin_max_threads(std::max(n1, n2));
  l.smem = smem_of(l.log_lines);
  const double fit = std::floor((228 << 10) / static_cast<double>(l.smem + 1024));
  double best = 0.0;
  for (int nt = 1; nt <= std::max(n1, n2) && nt * lines <= limit; ++nt) {
    const int threads = (nt * lines + 31) / 32 * 32;
    const double warps = std::max(1.0, fit) * threads / 32;
    const double cost = static_cast<double>((n2 + nt - 1) / nt * n1 + (n1 + nt - 1) / nt * n2) * threads * std::max(1.0, 14.0 / warps);
    if (best == 0.0 || cost < 0.999 * best) {
      best = cost;
      l.threads = nt * lines;
    }
  }
  check_cuda(cudaFuncSetAttribute(l.kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem_optin_bytes())),
             "kin smem");
  int dev = 0, sms = 0, per_sm = 0;
  check_cuda(cudaGetDevice(&dev), "cudaGetDevice");
  check_cuda(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev), "SM count");
  check_cuda(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, l.kernel, l.threads, l.smem), "occupancy");
  l.blocks = static_cast<long long>(sms) * std::max(per_sm, 1);
  return l;
}

}  // namespace spo_host
