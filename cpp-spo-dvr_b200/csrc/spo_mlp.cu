// The learned potential (include/spo_mlp.h): a BF16 multilayer perceptron whose products run on the
// B200 tensor cores through tcgen05.mma, FP32 accumulators in tensor memory.
//
// One GEMM kernel serves the forward pass and both backward products: C[M x N] = A[M x K] B[N x K]^T
// with A and B BF16, K-major (row-major with K contiguous), K and N multiples of 64:
//   - a block of 128 threads owns 128 rows and 64 columns of C (tiles of 256 columns left the forward product of a
//     batch of 4096 on 32 blocks: 48 us, 4096 x 256 x 256); warp 0 allocates 64 tensor-memory columns;
//   - per K chunk of 64, the threads stage A (128 x 64) and B (64 x 64) in shared memory in the
//     canonical K-major layout without swizzle (8-row x 16-byte core matrices: K chunks LBO bytes
//     apart, 8-row groups SBO = 128 bytes apart), make the writes visible to the tensor core
//     (fence.proxy.async), and one thread issues four tcgen05.mma (M 128, N, K 16) and a
//     tcgen05.commit on the stage's mbarrier; two stages alternate, so chunk k + 1 is staged while
//     the tensor core multiplies chunk k (a stage is rewritten after its previous commit, bounded wait);
//   - epilogue: each warp reads its 32 accumulator lanes (tcgen05.ld 32x32b, 16 columns at a time)
//     and writes FP32, BF16, or bias + SiLU (pre-activation FP32, activation BF16, row-major and transposed);
//   - split K: blockIdx.y takes a share of the K chunks and writes its own FP32 partial, summed in a
//     fixed order afterwards (weight gradients, where K is the batch).
// Prediction on many points is one kernel (mlp_predict_kernel): a block keeps the activations of 128 points in shared
// memory through all layers.
// Everything else (output layer, loss, SiLU derivative, Adam) is plain SIMT, with fixed-order reductions so that a
// training run is repeatable. A training step of 4 layers is 23 launches and no wait for the host (losses are summed on
// the device and read once per epoch); as 60 launches with two waits it took 0.9 ms, 0.5 of them the products.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <memory>
#include <stdexcept>
#include <string>
#include <vector>

#include "../../include/spo_b200.h"
#include "spo_hostcopy.cuh"
#include "../../include/spo_mlp.h"

namespace {

using bf16 = __nv_bfloat16;

struct MlpError : std::runtime_error {
  int code;
  MlpError(int c, const std::string& m) : std::runtime_error(m), code(c) {}
};

void ck(cudaError_t e, const char* what) {
  if (e == cudaErrorMemoryAllocation) throw MlpError(SPO_ERR_OOM, std::string(what) + ": " + cudaGetErrorString(e));
  if (e != cudaSuccess) throw MlpError(SPO_ERR_DEVICE, std::string(what) + ": " + cudaGetErrorString(e));
}
void need(bool c, const std::string& m) {
  if (!c) throw MlpError(SPO_ERR_INVALID, m);
}

// ------------------------------------------------------------------------------------------------
// tcgen05 / mbarrier primitives
// ------------------------------------------------------------------------------------------------
namespace tc {

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
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
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void fence_before_sync() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after_sync() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// Warp-wide: allocates `cols` tensor-memory columns, the address written to *slot.
__device__ __forceinline__ void tmem_alloc(uint32_t* slot, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(slot)), "r"(cols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t addr, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(cols) : "memory");
}
// Shared-memory matrix descriptor, K-major without swizzle (version 1, base offset 0).
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  return static_cast<uint64_t>((addr >> 4) & 0x3FFFu) | (static_cast<uint64_t>((lbo_bytes >> 4) & 0x3FFFu) << 16) |
         (static_cast<uint64_t>((sbo_bytes >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}
// D[tmem] (+)= A[smem] B[smem]^T, BF16 inputs, FP32 accumulate (one thread issues).
__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                         uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}" ::"r"(tmem_d),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(0), "r"(0), "r"(0), "r"(0)
      : "memory");
}
// Arrives on the barrier, announcing `bytes` of asynchronous copies, and one such copy (global -> shared).
__device__ __forceinline__ void mbar_arrive_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile(
      "{\n\t.reg .b64 state;\n\t"
      "mbarrier.arrive.expect_tx.shared::cta.b64 state, [%0], %1;\n\t}" ::"r"(smem_addr(bar)),
      "r"(bytes)
      : "memory");
}
__device__ __forceinline__ void bulk_copy(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_addr(dst)),
               "l"(src), "r"(bytes), "r"(smem_addr(bar))
               : "memory");
}
// Arrives on the barrier when this thread's earlier tcgen05.mma have completed.
__device__ __forceinline__ void commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_addr(bar))
               : "memory");
}
// Warp-wide: 16 consecutive FP32 columns of the warp's 32 lanes (one lane per thread).
__device__ __forceinline__ void tmem_ld16(uint32_t addr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
      "%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(addr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

}  // namespace tc

enum Epilogue { kEpiF32 = 0, kEpiBf16 = 1, kEpiBiasSilu = 2 };

struct GemmArgs {
  const bf16* a;
  long long lda;
  const bf16* b;
  long long ldb;
  int m, n, k;
  int epi;
  float* c;  // kEpiF32 (split K: partial y at c + y * c_split_stride), kEpiBiasSilu: pre-activation
  long long ldc, c_split_stride;
  const float* bias;
  bf16* out16;  // kEpiBf16: the product; kEpiBiasSilu: the activation
  long long ld16;
  bf16* out16t;  // kEpiBiasSilu: the activation transposed (column c at c * ldt), or null
  long long ldt;
  int* error_flag;
  int poll_limit;  // polls before a wait gives up; those of a block that leaves take kWaitLimit
};

constexpr int kBM = 128, kBK = 64, kBN = 64;
constexpr std::size_t kStageBytes = static_cast<std::size_t>(kBM + kBN) * kBK * 2;  // one A and one B chunk
// Two stages, barriers: at most four blocks per SM, whose 64 tensor-memory columns each fit the SM's 512 together.
constexpr std::size_t kGemmLaunchSmem = 2 * kStageBytes + 64;
static_assert(5 * kGemmLaunchSmem > 228 * 1024, "four blocks per SM at most");

__device__ __forceinline__ float silu(float z) { return z / (1.0f + __expf(-z)); }

// Two stages: while the tensor core multiplies chunk k (stage k % 2), the threads stage chunk k + 1 in
// the other buffer, after the commit of chunk k - 1 (its previous user) has arrived.
__global__ void __launch_bounds__(128) gemm_tn_kernel(GemmArgs g) {
  extern __shared__ __align__(1024) unsigned char smem[];
  uint64_t* bar = reinterpret_cast<uint64_t*>(smem + 2 * kStageBytes);  // one per stage
  uint32_t* tslot = reinterpret_cast<uint32_t*>(bar + 2);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (warp == 0) tc::tmem_alloc(tslot, kBN);
  if (tid == 0) {
    tc::mbar_init(bar, 1);
    tc::mbar_init(bar + 1, 1);
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = *tslot;
  const int m0 = blockIdx.x * kBM, n0 = blockIdx.z * kBN;
  const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(kBN >> 3) << 17) |
                         (static_cast<uint32_t>(kBM >> 4) << 24);
  const int nk = g.k / kBK;
  const int kc_first = static_cast<int>(static_cast<long long>(nk) * blockIdx.y / gridDim.y);
  const int kc_last = static_cast<int>(static_cast<long long>(nk) * (blockIdx.y + 1) / gridDim.y);
  // A: core (r8, kc) at (kc * 16 + r8) * 128; B: core (r8, kc) at (kc * 8 + r8) * 128
  // All of a thread's 16-byte loads of a chunk are issued before the first is stored.
  auto stage = [&](int st, int kc) {
    unsigned char* As = smem + st * kStageBytes;
    unsigned char* Bs = As + kBM * kBK * 2;
    const int k0 = kc * kBK;
    constexpr int NA = kBM * 8 / 128, NB = kBN * 8 / 128;
    uint4 va[NA], vb[NB];
#pragma unroll
    for (int i = 0; i < NA; ++i) {
      const int p = tid + 128 * i, r = p >> 3, c = p & 7;
      va[i] = m0 + r < g.m ? *reinterpret_cast<const uint4*>(g.a + static_cast<long long>(m0 + r) * g.lda + k0 + 8 * c)
                           : make_uint4(0, 0, 0, 0);
    }
#pragma unroll
    for (int i = 0; i < NB; ++i) {
      const int p = tid + 128 * i, r = p >> 3, c = p & 7;
      vb[i] = *reinterpret_cast<const uint4*>(g.b + static_cast<long long>(n0 + r) * g.ldb + k0 + 8 * c);
    }
#pragma unroll
    for (int i = 0; i < NA; ++i) {
      const int p = tid + 128 * i, r = p >> 3, c = p & 7;
      *reinterpret_cast<uint4*>(As + (c * (kBM / 8) + (r >> 3)) * 128 + (r & 7) * 16) = va[i];
    }
#pragma unroll
    for (int i = 0; i < NB; ++i) {
      const int p = tid + 128 * i, r = p >> 3, c = p & 7;
      *reinterpret_cast<uint4*>(Bs + (c * (kBN / 8) + (r >> 3)) * 128 + (r & 7) * 16) = vb[i];
    }
    tc::fence_proxy_async();  // the generic writes, visible to the tensor core
  };
  uint32_t parity = 0;   // bit s: the phase parity of stage s's barrier
  uint32_t pending = 0;  // bit s: a commit on stage s's barrier not yet waited for
  bool failed = false;
  if (kc_first < kc_last) stage(0, kc_first);
  tc::fence_before_sync();
  __syncthreads();
  for (int kc = kc_first; kc < kc_last; ++kc) {
    const int st = (kc - kc_first) & 1;
    if (tid == 0) {
      tc::fence_after_sync();
      const uint32_t a0 = tc::smem_addr(smem + st * kStageBytes);
      const uint32_t b0 = a0 + kBM * kBK * 2;
#pragma unroll
      for (int s = 0; s < kBK / 16; ++s) {
        const uint64_t ad = tc::smem_desc(a0 + 2 * s * (kBM / 8) * 128, (kBM / 8) * 128, 128);
        const uint64_t bd = tc::smem_desc(b0 + 2 * s * (kBN / 8) * 128, (kBN / 8) * 128, 128);
        tc::mma_bf16(tmem, ad, bd, idesc, (kc > kc_first || s > 0) ? 1u : 0u);
      }
      tc::commit(bar + st);
    }
    pending |= 1u << st;
    if (kc + 1 < kc_last) {
      // the other stage's previous chunk (kc - 1) must be multiplied before it is overwritten
      bool ok = true;
      if (kc > kc_first) {
        ok = tc::mbar_wait(bar + (st ^ 1), parity >> (st ^ 1) & 1u, g.poll_limit);
        if (ok) {
          parity ^= 1u << (st ^ 1);
          pending &= ~(1u << (st ^ 1));
        }
      }
      if (__syncthreads_or(!ok)) {
        failed = true;
        break;
      }
      stage(st ^ 1, kc + 1);
    }
    tc::fence_before_sync();
    __syncthreads();
  }
  // The last chunk's commit: it arrives when every earlier tcgen05.mma of the issuing thread has
  // completed, so the accumulator is final (the second-to-last commit needs no wait of its own).
  if (!failed && kc_last > kc_first) {
    const int last = (kc_last - kc_first - 1) & 1;
    const bool ok = tc::mbar_wait(bar + last, parity >> last & 1u, g.poll_limit);
    if (ok) pending = 0;  // the last commit arrives after every earlier MMA of the issuing thread
    failed = __syncthreads_or(!ok) != 0;
  }
  tc::fence_after_sync();
  if (failed) {
    if (tid == 0) atomicExch(g.error_flag, 1);
    // bounded waits for the MMAs in flight, so that none still writes the accumulator when it is freed
    for (int k = 0; k < 2; ++k)
      if (pending >> k & 1u) tc::mbar_wait(bar + k, parity >> k & 1u);
  } else if (kc_last > kc_first) {
    const int row = m0 + warp * 32 + lane;
    for (int j = 0; j < kBN / 16; ++j) {
      const int col = n0 + j * 16;
      uint32_t r[16];
      tc::tmem_ld16(tmem + (static_cast<uint32_t>(warp * 32) << 16) + static_cast<uint32_t>(j * 16), r);
      if (row < g.m) {
        if (g.epi == kEpiF32) {
          float* dst = g.c + blockIdx.y * g.c_split_stride + static_cast<long long>(row) * g.ldc + col;
#pragma unroll
          for (int e = 0; e < 16; e += 4)
            *reinterpret_cast<float4*>(dst + e) = make_float4(__uint_as_float(r[e]), __uint_as_float(r[e + 1]),
                                                              __uint_as_float(r[e + 2]), __uint_as_float(r[e + 3]));
        } else if (g.epi == kEpiBf16) {
          bf16* dst = g.out16 + static_cast<long long>(row) * g.ld16 + col;
          __align__(16) bf16 v[16];
#pragma unroll
          for (int e = 0; e < 16; ++e) v[e] = __float2bfloat16_rn(__uint_as_float(r[e]));
          reinterpret_cast<uint4*>(dst)[0] = reinterpret_cast<const uint4*>(v)[0];
          reinterpret_cast<uint4*>(dst)[1] = reinterpret_cast<const uint4*>(v)[1];
        } else {
          float* zd = g.c + static_cast<long long>(row) * g.ldc + col;
          bf16* ad = g.out16 + static_cast<long long>(row) * g.ld16 + col;
          __align__(16) float z[16];
          __align__(16) bf16 v[16];
#pragma unroll
          for (int e = 0; e < 16; ++e) {
            z[e] = __uint_as_float(r[e]) + __ldg(g.bias + col + e);
            v[e] = __float2bfloat16_rn(silu(z[e]));
          }
#pragma unroll
          for (int e = 0; e < 4; ++e) reinterpret_cast<float4*>(zd)[e] = reinterpret_cast<const float4*>(z)[e];
          reinterpret_cast<uint4*>(ad)[0] = reinterpret_cast<const uint4*>(v)[0];
          reinterpret_cast<uint4*>(ad)[1] = reinterpret_cast<const uint4*>(v)[1];
          if (g.out16t)
#pragma unroll
            for (int e = 0; e < 16; ++e) g.out16t[(col + e) * g.ldt + row] = v[e];
        }
      }
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(tmem, kBN);
}

// ------------------------------------------------------------------------------------------------
// Prediction
// ------------------------------------------------------------------------------------------------
// y[i] = network(x[i]): a block of 128 threads takes tiles of 128 points through all layers. The activations stay in
// shared memory as the A operand (BF16, canonical layout), the accumulator in tensor memory, and the weights come in
// chunks of 32 inputs (packed in the B operand's layout by pack_weights_kernel) by bulk copies into three slots, two
// chunks ahead of the products; two blocks per SM, so that one's SiLU overlaps the other's products. The separate
// kernels (input rounding, one GEMM per layer with its pre-activations in FP32, output layer) moved 1.5 KB per point
// and layer through memory. Bound: the SiLU (two special-function operations per unit: 0.5 ms for 1e6 points of
// 4 x 256), then the weights from L2 (3.2 GB).
struct PredictArgs {
  const float* x;       // n x n_in
  long long n;
  int n_in, width, depth;
  const bf16* weights;  // chunk after chunk, layer after layer
  const float* bias;    // depth x width
  const float* wo;
  const float* bo;
  float* y;
  int* error_flag;
  int poll_limit;
};
constexpr int kPredictSlots = 3, kPredictChunk = 32;
constexpr std::size_t predict_smem(int width) {
  const std::size_t k = width > 64 ? width : 64;
  return 128 * k * 2 + kPredictSlots * static_cast<std::size_t>(width) * kPredictChunk * 2 + 64 + 64;
}

__global__ void __launch_bounds__(128) mlp_predict_kernel(PredictArgs g) {
  extern __shared__ __align__(1024) unsigned char smem[];
  const int width = g.width, n8 = width / 8;
  unsigned char* const A = smem;
  unsigned char* const W = smem + 128 * (width > 64 ? width : 64) * 2;
  const uint32_t chunk_bytes = static_cast<uint32_t>(width * kPredictChunk * 2);
  uint64_t* const full = reinterpret_cast<uint64_t*>(W + kPredictSlots * chunk_bytes);  // per slot: the chunk has arrived
  uint64_t* const empty = full + kPredictSlots;                                         // per slot: its products are done
  uint64_t* const done = empty + kPredictSlots;                                         // a layer's products are done
  uint32_t* const tslot = reinterpret_cast<uint32_t*>(done + 1);
  const int tid = threadIdx.x, warp = tid >> 5;
  if (warp == 0) tc::tmem_alloc(tslot, static_cast<uint32_t>(width));
  if (tid == 0)
    for (int k = 0; k < 2 * kPredictSlots + 1; ++k) tc::mbar_init(full + k, 1);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = *tslot;
  const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(width >> 3) << 17) |
                         (static_cast<uint32_t>(kBM >> 4) << 24);
  const long long tiles = (g.n + kBM - 1) / kBM;
  const int per_tile = 64 / kPredictChunk + (g.depth - 1) * (width / kPredictChunk);  // chunks
  const long long my_tiles = tiles > blockIdx.x ? (tiles - blockIdx.x + gridDim.x - 1) / gridDim.x : 0;
  const long long chunks = my_tiles * per_tile;
  // Thread 0: chunks requested and multiplied so far; chunk k is the k % per_tile-th of the weights, in slot k % 3.
  long long requested = 0, used = 0;
  uint32_t done_parity = 0;
  bool done_pending = false;  // thread 0: a commit on `done` not yet waited for
  bool failed = false;
  auto request = [&] {  // every slot whose products are done, in order; false when a wait gave up
    while (requested < chunks && requested < used + kPredictSlots) {
      const int slot = static_cast<int>(requested % kPredictSlots);
      if (requested >= kPredictSlots &&
          !tc::mbar_wait(empty + slot, static_cast<uint32_t>(requested / kPredictSlots - 1) & 1u, g.poll_limit))
        return false;
      tc::mbar_arrive_tx(full + slot, chunk_bytes);
      tc::bulk_copy(W + slot * chunk_bytes, reinterpret_cast<const unsigned char*>(g.weights) + (requested % per_tile) * chunk_bytes,
                    chunk_bytes, full + slot);
      ++requested;
    }
    return true;
  };
  if (tid == 0) request();
  for (long long tile = blockIdx.x; tile < tiles && !failed; tile += gridDim.x) {
    const long long row = tile * kBM + tid;
    {  // the point's features, rounded to BF16, zero-padded to 64
      const float* const x = g.x + row * g.n_in;
      for (int c = 0; c < 8; ++c) {
        __align__(16) bf16 v[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) v[e] = __float2bfloat16_rn(row < g.n && 8 * c + e < g.n_in ? x[8 * c + e] : 0.0f);
        *reinterpret_cast<uint4*>(A + (c * (kBM / 8) + (tid >> 3)) * 128 + (tid & 7) * 16) = *reinterpret_cast<const uint4*>(v);
      }
    }
    double out = 0.0;
    for (int l = 0; l < g.depth; ++l) {
      tc::fence_proxy_async();  // the activations, visible to the tensor core
      tc::fence_before_sync();
      __syncthreads();
      if (tid == 0) {
        tc::fence_after_sync();
        const int nc = (l == 0 ? 64 : width) / kPredictChunk;
        const uint32_t a0 = tc::smem_addr(A);
        bool ok = true;
        for (int c = 0; c < nc && ok; ++c) {
          const int slot = static_cast<int>(used % kPredictSlots);
          ok = tc::mbar_wait(full + slot, static_cast<uint32_t>(used / kPredictSlots) & 1u, g.poll_limit);
          if (!ok) break;
          const uint32_t b0 = tc::smem_addr(W + slot * chunk_bytes);
#pragma unroll
          for (int s = 0; s < kPredictChunk / 16; ++s) {
            const uint64_t ad = tc::smem_desc(a0 + (c * (kPredictChunk / 8) + 2 * s) * (kBM / 8) * 128, (kBM / 8) * 128, 128);
            const uint64_t bd = tc::smem_desc(b0 + 2 * s * n8 * 128, static_cast<uint32_t>(n8 * 128), 128);
            tc::mma_bf16(tmem, ad, bd, idesc, (c > 0 || s > 0) ? 1u : 0u);
          }
          tc::commit(empty + slot);
          ++used;
          if (c == nc - 1) {
            tc::commit(done);
            done_pending = true;
          }
          // the chunk after the next two, into the slot of the chunk before this one
          if (c + 1 < nc || l + 1 < g.depth || tile + gridDim.x < tiles) {
            const long long keep = used;
            used = keep - 1;  // this chunk's slot is not waited for yet
            ok = request();
            used = keep;
          }
        }
        if (!ok) atomicExch(g.error_flag, 1);
      }
      const bool ok = tc::mbar_wait(done, done_parity, g.poll_limit);
      if (__syncthreads_or(!ok)) {
        failed = true;
        break;
      }
      done_parity ^= 1u;
      done_pending = false;
      tc::fence_after_sync();
      // bias, SiLU, BF16: the next layer's A operand, or the output layer's sum
      const float* const bias = g.bias + l * width;
      for (int j = 0; j < width / 16; ++j) {
        uint32_t r[16];
        tc::tmem_ld16(tmem + (static_cast<uint32_t>(warp * 32) << 16) + static_cast<uint32_t>(j * 16), r);
        __align__(16) bf16 v[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) v[e] = __float2bfloat16_rn(silu(__uint_as_float(r[e]) + __ldg(bias + j * 16 + e)));
        if (l + 1 < g.depth) {
#pragma unroll
          for (int c = 0; c < 2; ++c)
            *reinterpret_cast<uint4*>(A + ((2 * j + c) * (kBM / 8) + (tid >> 3)) * 128 + (tid & 7) * 16) =
                reinterpret_cast<const uint4*>(v)[c];
        } else {
          float t[16];  // 16 columns as a tree, their sums in FP64
#pragma unroll
          for (int e = 0; e < 16; ++e) t[e] = __bfloat162float(v[e]) * __ldg(g.wo + j * 16 + e);
#pragma unroll
          for (int k = 8; k > 0; k /= 2)
#pragma unroll
            for (int e = 0; e < k; ++e) t[e] += t[e + k];
          out += t[0];
        }
      }
    }
    if (!failed && row < g.n) g.y[row] = static_cast<float>(out + g.bo[0]);
  }
  if (failed) {
    if (tid == 0) {
      atomicExch(g.error_flag, 1);
      // bounded waits for this block's copies and products in flight and all they arrive on, so that nothing reaches its
      // shared memory after the block has left
      for (long long k = used; k < requested; ++k)
        tc::mbar_wait(full + k % kPredictSlots, static_cast<uint32_t>(k / kPredictSlots) & 1u);
      for (long long k = used > kPredictSlots ? used - kPredictSlots : 0; k < used; ++k)
        tc::mbar_wait(empty + k % kPredictSlots, static_cast<uint32_t>(k / kPredictSlots) & 1u);
      if (done_pending) tc::mbar_wait(done, done_parity);
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(tmem, static_cast<uint32_t>(width));
}

// W (out x in, FP32) -> BF16 chunks of 32 inputs in the B operand's layout: core matrices of 8 outputs x 8 inputs, outputs
// adjacent (n8 = out / 8 of them), inputs n8 apart.
__global__ void pack_weights_kernel(const float* __restrict__ w, int out, int in, bf16* __restrict__ packed) {
  const int total = out * in, n8 = out / 8;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < total; t += gridDim.x * blockDim.x) {
    const int n = t / in, k = t - n * in;
    packed[(k / kPredictChunk) * out * kPredictChunk + (((k % kPredictChunk) / 8) * n8 + n / 8) * 64 + (n % 8) * 8 + k % 8] =
        __float2bfloat16_rn(w[t]);
  }
}

// ------------------------------------------------------------------------------------------------
// SIMT kernels
// ------------------------------------------------------------------------------------------------
// The batch: rows idx[i] (or i) of x (n x n_in, FP32) as BF16 rows of width w (zero-padded) and transposed, and of y.
__global__ void gather_kernel(const float* __restrict__ x, const float* __restrict__ y, int n_in, const long long* __restrict__ idx,
                              long long rows, int w, bf16* __restrict__ out, bf16* __restrict__ out_t, float* __restrict__ yb) {
  const long long total = rows * w, step = static_cast<long long>(gridDim.x) * blockDim.x;
  const long long first = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
  for (long long t = first; t < total; t += step) {
    const long long i = t / w;
    const int c = static_cast<int>(t - i * w);
    out[t] = __float2bfloat16_rn(c < n_in ? x[(idx ? idx[i] : i) * n_in + c] : 0.0f);
  }
  for (long long t = first; t < total; t += step) {
    const int c = static_cast<int>(t / rows);
    const long long i = t - c * rows;
    out_t[t] = __float2bfloat16_rn(c < n_in ? x[(idx ? idx[i] : i) * n_in + c] : 0.0f);
  }
  for (long long i = first; i < rows; i += step) yb[i] = y[idx ? idx[i] : i];
}

// The output layer, the error and the loss of a batch: out = sum_k a[i][k] w[k] + b, d[i] = 2 (out - y[i]) / rows, and per
// block of 64 rows the sum of its squared errors. One warp per row at a time, fixed order (lane-strided sums, then a fixed
// tree).
__global__ void __launch_bounds__(256) output_loss_kernel(const bf16* __restrict__ a, int w, const float* __restrict__ wo,
                                                          const float* __restrict__ bo, const float* __restrict__ y,
                                                          long long rows, float* __restrict__ d, double* __restrict__ block_sums) {
  __shared__ double part[8];
  const int warp = threadIdx.x / 32, lane = threadIdx.x & 31;
  double sq = 0.0;
#pragma unroll 2
  for (int r = 0; r < 8; ++r) {
    const long long row = blockIdx.x * 64ll + warp * 8 + r;
    if (row >= rows) break;
    float s = 0.0f;
    for (int k = lane; k < w; k += 32) s += __bfloat162float(a[row * w + k]) * wo[k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    const float e = s + bo[0] - y[row];
    if (lane == 0) d[row] = 2.0f * e / static_cast<float>(rows);
    sq += static_cast<double>(e) * e;
  }
  if (lane == 0) part[warp] = sq;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int k = 0; k < 8; ++k) t += part[k];
    block_sums[blockIdx.x] = t;
  }
}

// dz = g SiLU'(z) for a tile of 64 rows x 64 columns: BF16 row-major and transposed (the operands of the products) and the
// tile's column sums of dz (bias gradient). g is the BF16 gradient of the layer above, or for the last hidden layer (top)
// d[i] w_out[k]; there also the column sums of d[i] a[i][k] (output weights) and, in column tile 0, of d (output bias).
__global__ void __launch_bounds__(256) silu_backward_kernel(const bf16* __restrict__ g16, const float* __restrict__ d,
                                                            const float* __restrict__ wo, const bf16* __restrict__ a,
                                                            const float* __restrict__ z, long long rows, int w, bf16* __restrict__ dz16,
                                                            bf16* __restrict__ dzt, float* __restrict__ db, float* __restrict__ dwo,
                                                            float* __restrict__ dbo) {
  __shared__ bf16 tile[64][66];
  __shared__ float part[2][4][64];
  const int c = threadIdx.x % 64, q = threadIdx.x / 64;
  const int col = blockIdx.x * 64 + c;
  const long long r0 = blockIdx.y * 64ll;
  float sum = 0.0f, sum_wo = 0.0f;
#pragma unroll 4
  for (int k = 0; k < 16; ++k) {
    const long long i = r0 + q * 16 + k;
    const float zz = z[i * w + col];
    const float s = 1.0f / (1.0f + __expf(-zz));
    const float gv = g16 ? __bfloat162float(g16[i * w + col]) : d[i] * wo[col];
    const float v = gv * s * (1.0f + zz * (1.0f - s));
    const bf16 h = __float2bfloat16_rn(v);
    dz16[i * w + col] = h;
    tile[q * 16 + k][c] = h;
    sum += v;
    if (!g16) sum_wo += d[i] * __bfloat162float(a[i * w + col]);
  }
  part[0][q][c] = sum;
  part[1][q][c] = sum_wo;
  __syncthreads();
  if (q == 0) {
    db[blockIdx.y * static_cast<long long>(w) + col] = part[0][0][c] + part[0][1][c] + part[0][2][c] + part[0][3][c];
    if (!g16) dwo[blockIdx.y * static_cast<long long>(w) + col] = part[1][0][c] + part[1][1][c] + part[1][2][c] + part[1][3][c];
  }
  if (!g16 && blockIdx.x == 0 && threadIdx.x == 0) {
    float t = 0.0f;
    for (int k = 0; k < 64; ++k) t += d[r0 + k];
    dbo[blockIdx.y] = t;
  }
  for (int k = q; k < 64; k += 4) dzt[(blockIdx.x * 64ll + k) * rows + r0 + c] = tile[c][k];
}

// n values, `stride` apart, in a fixed order: 16 sums side by side, then a tree. One chain over up to 1024 partials of 64 rows
// lost 1.5e-5 of a sum of equal terms, where the sums over single rows before it had lost 3e-6; this one at most 34 x 2^-24.
__device__ __forceinline__ float sum_rows(const float* __restrict__ p, int n, long long stride) {
  float s[16] = {};
  int k = 0;
  for (; k + 15 < n; k += 16) {
#pragma unroll
    for (int i = 0; i < 16; ++i) s[i] += p[(k + i) * stride];
  }
  for (; k < n; ++k) s[0] += p[k * stride];
#pragma unroll
  for (int w = 8; w > 0; w /= 2)
#pragma unroll
    for (int i = 0; i < w; ++i) s[i] += s[i + w];
  return s[0];
}

// Sums of partials in order: weights (n_parts of nw), then biases (n_rows_parts of w); for the last hidden layer also the
// output layer's gradients and the loss (the block sums of output_loss_kernel over `rows`).
__global__ void sum_partials_kernel(const float* __restrict__ parts, int n_parts, long long nw, float* __restrict__ gw,
                                    const float* __restrict__ db, int n_row_parts, int w, float* __restrict__ gb,
                                    const float* __restrict__ dwo, float* __restrict__ gwo, const float* __restrict__ dbo,
                                    float* __restrict__ gbo, const double* __restrict__ loss_parts, int n_loss, long long rows,
                                    double* __restrict__ loss) {
  const long long total = nw + w + (dwo ? w + 2 : 0);
  for (long long t = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; t < total;
       t += static_cast<long long>(gridDim.x) * blockDim.x) {
    if (t < nw) {
      float s = 0.0f;
#pragma unroll 8
      for (int p = 0; p < n_parts; ++p) s += parts[p * nw + t];
      gw[t] = s;
    } else if (t < nw + 2 * w) {
      const bool hidden = t < nw + w;
      const int k = static_cast<int>(t - nw) - (hidden ? 0 : w);
      (hidden ? gb : gwo)[k] = sum_rows((hidden ? db : dwo) + k, n_row_parts, w);
    } else if (t == nw + 2 * w) {
      gbo[0] = sum_rows(dbo, n_row_parts, 1);
    } else {
      double s = 0.0;
#pragma unroll 8
      for (int p = 0; p < n_loss; ++p) s += loss_parts[p];
      loss[0] = s / static_cast<double>(rows);
    }
  }
}

// Adam on FP32 parameters, all tensors in one launch (blockIdx.y), with the BF16 copies of the weight matrices (rows x
// cols): row-major and transposed.
struct AdamTensor {
  float *p, *m, *v;
  const float* g;
  long long n;
  int cols;  // 0: no BF16 copies
  bf16 *wb, *wt;
};
constexpr int kAdamTensors = 18;  // 8 layers of W and b, the output layer's
struct AdamArgs {
  AdamTensor t[kAdamTensors];
};
// A step whose gradients are not complete (a bounded wait gave up) changes nothing, nor do the steps queued behind it.
__global__ void adam_kernel(const __grid_constant__ AdamArgs args, float lr, float b1, float b2, float c1, float c2, float eps,
                            const int* __restrict__ error_flag, long long* __restrict__ steps_done) {
  if (*error_flag != 0) return;
  if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) ++*steps_done;
  const AdamTensor& a = args.t[blockIdx.y];
  for (long long t = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; t < a.n;
       t += static_cast<long long>(gridDim.x) * blockDim.x) {
    const float gt = a.g[t];
    const float mt = b1 * a.m[t] + (1.0f - b1) * gt;
    const float vt = b2 * a.v[t] + (1.0f - b2) * gt * gt;
    a.m[t] = mt;
    a.v[t] = vt;
    const float p = a.p[t] - lr * (mt / c1) / (sqrtf(vt / c2) + eps);
    a.p[t] = p;
    if (a.cols > 0) {
      const int r = static_cast<int>(t / a.cols), c = static_cast<int>(t - static_cast<long long>(r) * a.cols);
      const bf16 h = __float2bfloat16_rn(p);
      a.wb[t] = h;
      a.wt[c * (a.n / a.cols) + r] = h;
    }
  }
}

// BF16 copies of a weight matrix W (rows x cols): row-major and transposed.
__global__ void weights_to_bf16_kernel(const float* __restrict__ w, int rows, int cols, bf16* __restrict__ wb,
                                       bf16* __restrict__ wt) {
  const long long total = static_cast<long long>(rows) * cols;
  for (long long t = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; t < total;
       t += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int r = static_cast<int>(t / cols), c = static_cast<int>(t - static_cast<long long>(r) * cols);
    const bf16 h = __float2bfloat16_rn(w[t]);
    wb[t] = h;
    wt[static_cast<long long>(c) * rows + r] = h;
  }
}

constexpr int kSplits = 32;  // K splits of the weight gradients

unsigned grid_for(long long n, int threads = 256) {
  return static_cast<unsigned>(std::min<long long>(std::max<long long>((n + threads - 1) / threads, 1), 148 * 16));
}

// ------------------------------------------------------------------------------------------------
// The network
// ------------------------------------------------------------------------------------------------
template <typename U>
struct DevBuf {
  U* p = nullptr;
  std::size_t n = 0;
  void alloc(std::size_t count) {
    free();
    ck(cudaMalloc(&p, sizeof(U) * std::max<std::size_t>(count, 1)), "cudaMalloc");
    n = count;
  }
  void free() {
    if (p) cudaFree(p);
    p = nullptr;
    n = 0;
  }
  ~DevBuf() { free(); }
};

struct Layer {
  int in, out;
  DevBuf<float> w, b, gw, gb, mw, vw, mb, vb;
  DevBuf<bf16> wb, wt;
};

}  // namespace

struct spo_mlp {
  std::string err;
  int device = 0;
  int n_in = 0, in_pad = 0, width = 0, depth = 0;
  cudaStream_t stream = nullptr;
  std::vector<std::unique_ptr<Layer>> layers;
  DevBuf<float> wo, bo, gwo, gbo, mwo, vwo, mbo, vbo;
  DevBuf<int> error_flag;
  // per-batch work space (capacity rows)
  long long cap = 0;
  DevBuf<bf16> x16, x16t;                  // rows x in_pad, and transposed
  std::vector<std::unique_ptr<DevBuf<float>>> z;           // per layer: rows x width (pre-activation)
  std::vector<std::unique_ptr<DevBuf<bf16>>> act, act_t;   // per layer: rows x width (activation), and transposed
  DevBuf<float> yb, d, db, dwo, dbo, partials;             // db, dwo, dbo: column sums per 64 rows
  DevBuf<double> loss_parts, loss;                         // per 64 rows; per step of an epoch
  DevBuf<bf16> g16, dz16, dzt;
  long long step = 0;             // of Adam; on the device those that were applied
  DevBuf<long long> steps_done;
  int poll_limit = tc::kWaitLimit;
  // Device memory for a call's points, kept for the next call: at most this much for a training set (which is given back
  // above it) and as much for the predictions' points, which go in chunks that fit: 2^20 points of up to 15 features, 258048
  // of 64. (Chunks of 2^20 whatever the features kept 268 MB.)
  static constexpr std::size_t kKeepBytes = 64ull << 20;
  long long predict_rows() const {
    const long long fit = static_cast<long long>(kKeepBytes / (sizeof(float) * (n_in + 1))) / kBM * kBM;
    return std::min(fit, 1ll << 20);
  }
  DevBuf<float> tx, ty;
  DevBuf<long long> tperm;
  void training_set(long long n, bool order) {
    if (tx.n < static_cast<std::size_t>(n * n_in)) tx.alloc(static_cast<std::size_t>(n * n_in));
    if (ty.n < static_cast<std::size_t>(n)) ty.alloc(static_cast<std::size_t>(n));
    if (order && tperm.n < static_cast<std::size_t>(n)) tperm.alloc(static_cast<std::size_t>(n));
  }
  struct TrainingSetKeeper {  // at the end of a call, also of one that failed
    spo_mlp* m;
    ~TrainingSetKeeper() { m->release_training_set(); }
  };
  void release_training_set() {
    if (sizeof(float) * (tx.n + ty.n) + sizeof(long long) * tperm.n <= kKeepBytes) return;
    tx.free();
    ty.free();
    tperm.free();
  }
  DevBuf<float> px, py, pbias;
  DevBuf<bf16> packed;
  int sms = 0;
  bool predict_ready = false;  // all of these are there
  spo_host::RawCopier copier;

  ~spo_mlp() {
    if (stream) cudaStreamDestroy(stream);
  }

  long long parameter_count() const {
    long long n = 0;
    for (const auto& l : layers) n += static_cast<long long>(l->in) * l->out + l->out;
    return n + width + 1;
  }

  void ensure_capacity(long long rows) {
    if (rows <= cap) return;
    cap = 0;  // until the last allocation has succeeded: a call after one that failed starts over
    const long long grown = ((rows + 127) / 128) * 128;
    x16.alloc(grown * in_pad);
    x16t.alloc(grown * in_pad);
    z.clear();
    act.clear();
    act_t.clear();
    for (int l = 0; l < depth; ++l) {
      z.push_back(std::make_unique<DevBuf<float>>());
      z.back()->alloc(grown * width);
      for (auto* v : {&act, &act_t}) {
        v->push_back(std::make_unique<DevBuf<bf16>>());
        v->back()->alloc(grown * width);
      }
    }
    yb.alloc(grown);
    d.alloc(grown);
    db.alloc(grown / 64 * width);
    dwo.alloc(grown / 64 * width);
    dbo.alloc(grown / 64);
    g16.alloc(grown * width);
    dz16.alloc(grown * width);
    dzt.alloc(grown * width);
    loss_parts.alloc(grown / 64);
    if (!loss.p) loss.alloc(1);
    cap = grown;
  }

  void refresh_bf16() {
    for (auto& l : layers)
      weights_to_bf16_kernel<<<grid_for(static_cast<long long>(l->in) * l->out), 256, 0, stream>>>(l->w.p, l->out, l->in,
                                                                                                   l->wb.p, l->wt.p);
    ck(cudaGetLastError(), "weights_to_bf16");
  }

  void gemm(const bf16* a, long long lda, const bf16* b, long long ldb, int m, int n, int k, int epi, float* c,
            long long ldc, const float* bias, bf16* out16, long long ld16, int splits = 1, long long split_stride = 0,
            bf16* out16t = nullptr, long long ldt = 0) {
    need(k % kBK == 0 && n % kBN == 0 && n > 0 && lda % 8 == 0 && ldb % 8 == 0, "gemm shape");
    GemmArgs g{a, lda, b, ldb, m, n, k, epi, c, ldc, split_stride, bias, out16, ld16, out16t, ldt, error_flag.p, poll_limit};
    const dim3 grid(static_cast<unsigned>((m + kBM - 1) / kBM), static_cast<unsigned>(splits), static_cast<unsigned>(n / kBN));
    gemm_tn_kernel<<<grid, 128, kGemmLaunchSmem, stream>>>(g);
    ck(cudaGetLastError(), "gemm launch");
  }

  // Forward pass of `rows` rows already in x16 / yb; the output layer's errors in d, the squared ones in loss_parts.
  void forward(long long rows) {
    const bf16* a = x16.p;
    int k = in_pad;
    for (int l = 0; l < depth; ++l) {
      Layer& L = *layers[l];
      gemm(a, k, L.wb.p, L.in, static_cast<int>(rows), width, k, kEpiBiasSilu, z[l]->p, width, L.b.p, act[l]->p, width, 1, 0,
           l + 1 < depth ? act_t[l]->p : nullptr, rows);
      a = act[l]->p;
      k = width;
    }
    output_loss_kernel<<<static_cast<unsigned>((rows + 63) / 64), 256, 0, stream>>>(act[depth - 1]->p, width, wo.p, bo.p, yb.p, rows,
                                                                                 d.p, loss_parts.p);
    ck(cudaGetLastError(), "output layer");
  }

  // All gradients for `rows` rows (a multiple of 64) after forward(); the mean squared error into loss[slot].
  void backward(long long rows, long long slot) {
    // split K so that the weight gradients (few tiles of C) fill the GPU; every split has its chunks of kBK rows
    const int splits = static_cast<int>(std::min<long long>(kSplits, rows / kBK));
    const int row_parts = static_cast<int>(rows / 64);
    for (int l = depth - 1; l >= 0; --l) {
      Layer& L = *layers[l];
      const bool top = l == depth - 1;
      silu_backward_kernel<<<dim3(static_cast<unsigned>(width / 64), static_cast<unsigned>(row_parts)), 256, 0, stream>>>(
          top ? nullptr : g16.p, d.p, wo.p, act[l]->p, z[l]->p, rows, width, dz16.p, dzt.p, db.p, dwo.p, dbo.p);
      ck(cudaGetLastError(), "silu backward");
      // gW = dz^T a_in : A = dz^T (width x rows), B = a_in^T (in x rows), K = rows
      const long long wsz = static_cast<long long>(L.out) * L.in;
      gemm(dzt.p, rows, l == 0 ? x16t.p : act_t[l - 1]->p, rows, L.out, L.in, static_cast<int>(rows), kEpiF32, partials.p, L.in,
           nullptr, nullptr, 0, splits, wsz);
      sum_partials_kernel<<<grid_for(wsz + 2 * width + 2), 256, 0, stream>>>(
          partials.p, splits, wsz, L.gw.p, db.p, row_parts, width, L.gb.p, top ? dwo.p : nullptr, gwo.p, dbo.p, gbo.p, loss_parts.p,
          static_cast<int>((rows + 63) / 64), rows, loss.p + slot);
      ck(cudaGetLastError(), "sum partials");
      if (l > 0)  // d a_in = dz W : A = dz (rows x width), B = W^T (in x width)
        gemm(dz16.p, width, L.wt.p, L.out, static_cast<int>(rows), L.in, width, kEpiBf16, nullptr, 0, nullptr, g16.p, L.in);
    }
  }

  void check_flag() {
    int f = 0;
    ck(cudaMemcpy(&f, error_flag.p, sizeof(int), cudaMemcpyDeviceToHost), "error flag");
    if (f) {
      ck(cudaMemcpy(&step, steps_done.p, sizeof step, cudaMemcpyDeviceToHost), "steps done");
      ck(cudaMemset(error_flag.p, 0, sizeof(int)), "error flag");
      throw MlpError(SPO_ERR_TIMEOUT, "mlp: a bounded wait for the tensor cores gave up");
    }
  }

  void load_rows(const float* x_dev, const float* y_dev, const long long* idx_dev, long long rows) {
    gather_kernel<<<grid_for(rows * in_pad), 256, 0, stream>>>(x_dev, y_dev, n_in, idx_dev, rows, in_pad, x16.p, x16t.p, yb.p);
    ck(cudaGetLastError(), "gather");
  }

  void adam(float lr) {
    ++step;
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    const float c1 = 1.0f - std::pow(b1, static_cast<float>(step)), c2 = 1.0f - std::pow(b2, static_cast<float>(step));
    AdamArgs args{};
    int n = 0;
    for (auto& l : layers) {
      args.t[n++] = {l->w.p, l->mw.p, l->vw.p, l->gw.p, static_cast<long long>(l->in) * l->out, l->in, l->wb.p, l->wt.p};
      args.t[n++] = {l->b.p, l->mb.p, l->vb.p, l->gb.p, l->out, 0, nullptr, nullptr};
    }
    args.t[n++] = {wo.p, mwo.p, vwo.p, gwo.p, width, 0, nullptr, nullptr};
    args.t[n++] = {bo.p, mbo.p, vbo.p, gbo.p, 1, 0, nullptr, nullptr};
    adam_kernel<<<dim3(64, static_cast<unsigned>(n)), 256, 0, stream>>>(args, lr, b1, b2, c1, c2, eps, error_flag.p, steps_done.p);
    ck(cudaGetLastError(), "adam");
  }

  // Parameter transfer in the documented order.
  template <typename F>
  void for_each_param(F&& f) {
    for (auto& l : layers) {
      f(l->w, l->gw, static_cast<long long>(l->in) * l->out);
      f(l->b, l->gb, l->out);
    }
    f(wo, gwo, width);
    f(bo, gbo, 1);
  }
};

namespace {
std::string g_mlp_error;

template <typename F>
int guarded_mlp(spo_mlp* m, F&& f) {
  if (!m) return SPO_ERR_INVALID;
  try {
    ck(cudaSetDevice(m->device), "cudaSetDevice");
    f();
    return SPO_OK;
  } catch (const MlpError& e) {
    m->err = e.what();
    return e.code;
  } catch (const std::exception& e) {
    m->err = e.what();
    return SPO_ERR_DEVICE;
  }
}

// splitmix64, for the initial weights and the batch order.
struct SplitMix {
  uint64_t s;
  uint64_t next() {
    uint64_t z = (s += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
  }
  double uniform() { return (next() >> 11) * (1.0 / 9007199254740992.0); }
};
}  // namespace

extern "C" {

const char* spo_mlp_last_error(const spo_mlp* m) { return m ? m->err.c_str() : g_mlp_error.c_str(); }

int spo_mlp_create(int n_in, int width, int depth, unsigned long long seed, int device, spo_mlp** out) {
  if (!out) return SPO_ERR_INVALID;
  *out = nullptr;
  auto m = std::make_unique<spo_mlp>();
  try {
    need(n_in >= 1 && n_in <= 64, "spo_mlp_create: n_in must be 1..64");
    need(width == 64 || width == 128 || width == 256, "spo_mlp_create: width must be 64, 128 or 256");
    need(depth >= 1 && depth <= 8, "spo_mlp_create: depth must be 1..8");
    m->device = device;
    ck(cudaSetDevice(device), "cudaSetDevice");
    int major = 0;
    ck(cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, device), "compute capability");
    need(major >= 10, "spo_mlp_create: needs an sm_100 device (tcgen05)");
    ck(cudaStreamCreateWithFlags(&m->stream, cudaStreamNonBlocking), "cudaStreamCreate");
    ck(cudaFuncSetAttribute(gemm_tn_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                            static_cast<int>(kGemmLaunchSmem)),
       "gemm smem");
    m->n_in = n_in;
    m->in_pad = 64;
    m->width = width;
    m->depth = depth;
    SplitMix rng{seed};
    auto init = [&](DevBuf<float>& buf, long long n, double scale) {
      std::vector<float> h(static_cast<std::size_t>(n));
      for (auto& v : h) v = static_cast<float>((2.0 * rng.uniform() - 1.0) * scale);
      buf.alloc(static_cast<std::size_t>(n));
      ck(cudaMemcpy(buf.p, h.data(), sizeof(float) * n, cudaMemcpyHostToDevice), "init");
    };
    auto zeros = [&](DevBuf<float>& buf, long long n) {
      buf.alloc(static_cast<std::size_t>(n));
      ck(cudaMemset(buf.p, 0, sizeof(float) * n), "init");
    };
    for (int l = 0; l < depth; ++l) {
      auto L = std::make_unique<Layer>();
      L->in = l == 0 ? m->in_pad : width;
      L->out = width;
      const long long nw = static_cast<long long>(L->in) * L->out;
      const int fan_in = l == 0 ? n_in : width;
      init(L->w, nw, 1.0 / std::sqrt(static_cast<double>(fan_in)));
      if (l == 0) {  // the padded input columns carry no weight
        std::vector<float> h(static_cast<std::size_t>(nw));
        ck(cudaMemcpy(h.data(), L->w.p, sizeof(float) * nw, cudaMemcpyDeviceToHost), "init");
        for (int r = 0; r < L->out; ++r)
          for (int c = n_in; c < L->in; ++c) h[static_cast<std::size_t>(r) * L->in + c] = 0.0f;
        ck(cudaMemcpy(L->w.p, h.data(), sizeof(float) * nw, cudaMemcpyHostToDevice), "init");
      }
      zeros(L->b, L->out);
      zeros(L->gw, nw);
      zeros(L->gb, L->out);
      zeros(L->mw, nw);
      zeros(L->vw, nw);
      zeros(L->mb, L->out);
      zeros(L->vb, L->out);
      L->wb.alloc(static_cast<std::size_t>(nw));
      L->wt.alloc(static_cast<std::size_t>(nw));
      m->layers.push_back(std::move(L));
    }
    init(m->wo, width, 1.0 / std::sqrt(static_cast<double>(width)));
    zeros(m->bo, 1);
    zeros(m->gwo, width);
    zeros(m->gbo, 1);
    zeros(m->mwo, width);
    zeros(m->vwo, width);
    zeros(m->mbo, 1);
    zeros(m->vbo, 1);
    m->error_flag.alloc(1);
    ck(cudaMemset(m->error_flag.p, 0, sizeof(int)), "error flag");
    m->steps_done.alloc(1);
    ck(cudaMemset(m->steps_done.p, 0, sizeof(long long)), "steps done");
    m->partials.alloc(static_cast<std::size_t>(kSplits) * width * std::max(width, m->in_pad));
    m->refresh_bf16();
    ck(cudaStreamSynchronize(m->stream), "create");
  } catch (const MlpError& e) {
    g_mlp_error = e.what();
    return e.code;
  } catch (const std::exception& e) {
    g_mlp_error = e.what();
    return SPO_ERR_DEVICE;
  }
  *out = m.release();
  return SPO_OK;
}

int spo_mlp_destroy(spo_mlp* m) {
  if (!m) return SPO_OK;
  cudaSetDevice(m->device);
  delete m;
  return SPO_OK;
}

int spo_mlp_parameter_count(const spo_mlp* m, long long* n) {
  if (!m || !n) return SPO_ERR_INVALID;
  *n = m->parameter_count();
  return SPO_OK;
}

int spo_mlp_input_width(const spo_mlp* m, int* n) {
  if (!m || !n) return SPO_ERR_INVALID;
  *n = m->in_pad;
  return SPO_OK;
}

int spo_mlp_get_parameters(spo_mlp* m, float* out) {
  return guarded_mlp(m, [&] {
    need(out != nullptr, "null pointer");
    long long off = 0;
    m->for_each_param([&](DevBuf<float>& p, DevBuf<float>&, long long n) {
      ck(cudaMemcpy(out + off, p.p, sizeof(float) * n, cudaMemcpyDeviceToHost), "get parameters");
      off += n;
    });
  });
}

int spo_mlp_set_parameters(spo_mlp* m, const float* in) {
  return guarded_mlp(m, [&] {
    need(in != nullptr, "null pointer");
    long long off = 0;
    m->for_each_param([&](DevBuf<float>& p, DevBuf<float>&, long long n) {
      ck(cudaMemcpy(p.p, in + off, sizeof(float) * n, cudaMemcpyHostToDevice), "set parameters");
      off += n;
    });
    m->refresh_bf16();
    ck(cudaStreamSynchronize(m->stream), "set parameters");
  });
}

int spo_mlp_predict(spo_mlp* m, const float* x, long long n, float* y) {
  return guarded_mlp(m, [&] {
    need(x && y && n > 0, "spo_mlp_predict: bad arguments");
    const long long most = std::min(n, m->predict_rows());
    if (m->px.n < static_cast<std::size_t>(most * m->n_in)) m->px.alloc(static_cast<std::size_t>(most * m->n_in));
    if (m->py.n < static_cast<std::size_t>(most)) m->py.alloc(static_cast<std::size_t>(most));
    if (!m->predict_ready) {
      std::size_t total = 0;
      for (const auto& l : m->layers) total += static_cast<std::size_t>(l->in) * l->out;
      m->packed.alloc(total);
      m->pbias.alloc(static_cast<std::size_t>(m->depth) * m->width);
      ck(cudaDeviceGetAttribute(&m->sms, cudaDevAttrMultiProcessorCount, m->device), "SM count");
      ck(cudaFuncSetAttribute(mlp_predict_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              static_cast<int>(predict_smem(256))), "predict smem");
      m->predict_ready = true;
    }
    std::size_t off = 0;
    for (int l = 0; l < m->depth; ++l) {
      const Layer& L = *m->layers[l];
      pack_weights_kernel<<<grid_for(static_cast<long long>(L.in) * L.out), 256, 0, m->stream>>>(L.w.p, L.out, L.in, m->packed.p + off);
      off += static_cast<std::size_t>(L.in) * L.out;
      ck(cudaMemcpyAsync(m->pbias.p + static_cast<std::size_t>(l) * m->width, L.b.p, sizeof(float) * m->width,
                         cudaMemcpyDeviceToDevice, m->stream), "biases");
    }
    ck(cudaGetLastError(), "pack weights");
    for (long long i0 = 0; i0 < n; i0 += most) {
      const long long rows = std::min(most, n - i0);
      const std::size_t in_bytes = sizeof(float) * static_cast<std::size_t>(rows * m->n_in), out_bytes = sizeof(float) * rows;
      if (m->copier.wanted(x, in_bytes, m->device))
        ck(m->copier.to_device(x + i0 * m->n_in, m->px.p, in_bytes, m->device), "upload");
      else
        ck(cudaMemcpyAsync(m->px.p, x + i0 * m->n_in, in_bytes, cudaMemcpyHostToDevice, m->stream), "upload");
      PredictArgs g{m->px.p, rows, m->n_in, m->width, m->depth, m->packed.p, m->pbias.p, m->wo.p, m->bo.p, m->py.p, m->error_flag.p, m->poll_limit};
      const long long tiles = (rows + kBM - 1) / kBM;
      mlp_predict_kernel<<<static_cast<unsigned>(std::min<long long>(tiles, 2ll * m->sms)), 128, predict_smem(m->width), m->stream>>>(g);
      ck(cudaGetLastError(), "predict launch");
      if (m->copier.wanted(y, out_bytes, m->device)) {
        ck(cudaStreamSynchronize(m->stream), "predict");
        ck(m->copier.to_host(m->py.p, y + i0, out_bytes, m->device), "download");
      } else {
        ck(cudaMemcpyAsync(y + i0, m->py.p, out_bytes, cudaMemcpyDeviceToHost, m->stream), "download");
        ck(cudaStreamSynchronize(m->stream), "predict");
      }
    }
    m->check_flag();
  });
}

int spo_mlp_test_wait_timeout(spo_mlp* m, int poll_limit) {
  if (!m) return SPO_ERR_INVALID;
  m->poll_limit = poll_limit < 0 ? tc::kWaitLimit : poll_limit;
  return SPO_OK;
}

int spo_mlp_gradients(spo_mlp* m, const float* x, const float* y, long long n, double* loss, float* grad) {
  return guarded_mlp(m, [&] {
    need(x && y && grad && n >= kBK && n <= 65536 && n % kBK == 0,
         "spo_mlp_gradients: n must be a multiple of 64, at most 65536");
    m->ensure_capacity(n);
    m->training_set(n, false);
    ck(cudaMemcpyAsync(m->tx.p, x, sizeof(float) * n * m->n_in, cudaMemcpyHostToDevice, m->stream), "upload");
    ck(cudaMemcpyAsync(m->ty.p, y, sizeof(float) * n, cudaMemcpyHostToDevice, m->stream), "upload");
    m->load_rows(m->tx.p, m->ty.p, nullptr, n);
    m->forward(n);
    m->backward(n, 0);
    double l = 0.0;
    ck(cudaMemcpyAsync(&l, m->loss.p, sizeof(double), cudaMemcpyDeviceToHost, m->stream), "loss");
    ck(cudaStreamSynchronize(m->stream), "gradients");
    m->check_flag();
    if (loss) *loss = l;
    long long off = 0;
    m->for_each_param([&](DevBuf<float>&, DevBuf<float>& g, long long cnt) {
      ck(cudaMemcpy(grad + off, g.p, sizeof(float) * cnt, cudaMemcpyDeviceToHost), "gradients");
      off += cnt;
    });
  });
}

int spo_mlp_train(spo_mlp* m, const float* x, const float* y, long long n, int epochs, int batch, float lr,
                  unsigned long long seed, double* last_epoch_loss) {
  return guarded_mlp(m, [&] {
    need(x && y && n >= batch && epochs > 0 && batch >= 128 && batch % 128 == 0 && batch <= 65536 && lr > 0.0f,
         "spo_mlp_train: bad arguments");
    m->ensure_capacity(batch);
    const spo_mlp::TrainingSetKeeper keeper{m};
    m->training_set(n, true);
    ck(cudaMemcpyAsync(m->tx.p, x, sizeof(float) * n * m->n_in, cudaMemcpyHostToDevice, m->stream), "upload");
    ck(cudaMemcpyAsync(m->ty.p, y, sizeof(float) * n, cudaMemcpyHostToDevice, m->stream), "upload");
    SplitMix rng{seed};
    std::vector<long long> order(static_cast<std::size_t>(n));
    const long long steps_per_epoch = n / batch;
    const long long total_steps = steps_per_epoch * epochs;
    if (m->loss.n < static_cast<std::size_t>(steps_per_epoch)) m->loss.alloc(static_cast<std::size_t>(steps_per_epoch));
    std::vector<double> losses(static_cast<std::size_t>(steps_per_epoch));
    long long t = 0;
    double epoch_loss = 0.0;
    for (int e = 0; e < epochs; ++e) {
      for (long long i = 0; i < n; ++i) order[i] = i;
      for (long long i = n - 1; i > 0; --i) std::swap(order[i], order[rng.next() % static_cast<uint64_t>(i + 1)]);
      ck(cudaMemcpyAsync(m->tperm.p, order.data(), sizeof(long long) * n, cudaMemcpyHostToDevice, m->stream), "order");
      for (long long s = 0; s < steps_per_epoch; ++s, ++t) {
        const double frac = static_cast<double>(t) / static_cast<double>(std::max<long long>(total_steps - 1, 1));
        const float rate = static_cast<float>(lr * (0.05 + 0.95 * 0.5 * (1.0 + std::cos(3.14159265358979 * frac))));
        m->load_rows(m->tx.p, m->ty.p, m->tperm.p + s * batch, batch);
        m->forward(batch);
        m->backward(batch, s);
        m->adam(rate);
      }
      ck(cudaMemcpyAsync(losses.data(), m->loss.p, sizeof(double) * steps_per_epoch, cudaMemcpyDeviceToHost, m->stream), "losses");
      ck(cudaStreamSynchronize(m->stream), "epoch");  // and before the next epoch's order is uploaded
      m->check_flag();
      epoch_loss = 0.0;
      for (const double v : losses) epoch_loss += v;
      epoch_loss /= static_cast<double>(steps_per_epoch);
    }
    ck(cudaStreamSynchronize(m->stream), "train");
    m->check_flag();
    if (last_epoch_loss) *last_epoch_loss = epoch_loss;
  });
}

}  // extern "C"
