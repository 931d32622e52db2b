// Diagnostic: how long the tensor pipe is held by the three products of the decode kernel.
//
// One CTA per SM; a converged warp (or a warp per product) issues through an elected lane, back to back and without any other work
// on the SM, the tcgen05.mma chains of a 128-token tile as the decode kernel shapes and issues them -- (1) K = X Bk: 8 x (M=128,
// N=128, K=16), both operands in shared memory; (2) S = K' Q~^T: 8 x (M=128, N=16, K=16), A in tensor memory; (3) O^T += XV^T P: 8 x
// (M=128, N=16, K=16), both operands in shared memory, A MN-major -- commits once (or behind every chain) and waits (bounded).
// The result is clock cycles per tile: a floor under the kernel's time per tile.
// It has no counterpart in the reference and touches no cache state.
#include <type_traits>

#include "dkv_common.cuh"

namespace dkv {

namespace {

constexpr uint32_t PROBE_SPIN = 1u << 22;
constexpr int PP_PITCH = 128 * 16 + 32;                       // chunks of the operand tiles, as in the decode kernel
constexpr int PP_A = 0, PP_B = PP_A + 16 * PP_PITCH, PP_V = PP_B + 32768, PP_Q = PP_V + 16 * PP_PITCH, PP_BAR = PP_Q + 12288;
constexpr int PROBE_SMEM = PP_BAR + 128;
static_assert(PP_B % 128 == 0 && PP_V % 128 == 0 && PP_Q % 128 == 0 && PP_BAR % 16 == 0, "operand tiles are aligned");

__device__ __forceinline__ uint32_t pp_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint64_t pp_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((addr >> 4) & 0x3FFF) | ((uint64_t)((lbo >> 4) & 0x3FFF) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3FFF) << 32) | (1ull << 46);
}
__device__ __forceinline__ void pp_mma_ss(uint32_t d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t acc) {
  asm volatile("{\n.reg .pred p, e;\nelect.sync _|e, 0xffffffff;\nsetp.ne.b32 p, %4, 0;\n@e tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}"
               ::"r"(d), "l"(da), "l"(db), "r"(idesc), "r"(acc) : "memory");
}
__device__ __forceinline__ void pp_mma_ts(uint32_t d, uint32_t a, uint64_t db, uint32_t idesc, uint32_t acc) {
  asm volatile("{\n.reg .pred p, e;\nelect.sync _|e, 0xffffffff;\nsetp.ne.b32 p, %4, 0;\n@e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}"
               ::"r"(d), "r"(a), "l"(db), "r"(idesc), "r"(acc) : "memory");
}
__device__ __forceinline__ void pp_commit(uint32_t bar) {
  asm volatile("{\n.reg .pred e;\nelect.sync _|e, 0xffffffff;\n@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}" ::"r"(bar) : "memory");
}

// MASK: 1 | 2 | 4 the products of warp 0; 8 product (3) from warp 1 beside it; 16 a commit behind every chain; 32 operands that are
// not zero; 64 a warp per product
template <int MASK>
__global__ void __launch_bounds__(128) pipe_probe_kernel(long long* cycles, int32_t* status, int tiles) {
  extern __shared__ __align__(1024) unsigned char pp_raw[];
  const uint32_t sA = pp_smem(pp_raw + PP_A), sB = pp_smem(pp_raw + PP_B);      // K operand tile, basis
  const uint32_t sV = pp_smem(pp_raw + PP_V), sQ = pp_smem(pp_raw + PP_Q);      // V operand tile, rotated queries / P
  const uint32_t bar = pp_smem(pp_raw + PP_BAR);                                // a barrier per warp, one per product's commits (never waited for)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(pp_raw + PP_BAR + 64);
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  for (int e = tid; e < PP_BAR / 16; e += blockDim.x) {
    // zero operands, or (mask bit 32) a non-trivial bit pattern: small bf16 values of both signs
    uint4 v = make_uint4(0, 0, 0, 0);
    if (MASK & 32) {
      const uint32_t h = (uint32_t)e * 2654435761u;
      v = make_uint4(0x3c003b00u ^ (h & 0x80ff80ffu), 0x3a803c80u ^ ((h >> 3) & 0x80ff80ffu), 0x3b403bc0u ^ ((h >> 7) & 0x80ff80ffu),
                     0x3c403a40u ^ ((h >> 11) & 0x80ff80ffu));
    }
    reinterpret_cast<uint4*>(pp_raw)[e] = v;
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(pp_smem(tmem_slot)), "r"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 0) {
    for (int i = 0; i < 6; ++i) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar + 8 * i));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tb = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  constexpr uint32_t id_k = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | ((128u >> 3) << 17) | ((128u >> 4) << 24);
  constexpr uint32_t id_s = (1u << 4) | (1u << 7) | (1u << 10) | ((16u >> 3) << 17) | ((128u >> 4) << 24);
  constexpr uint32_t id_o = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) | ((16u >> 3) << 17) | ((128u >> 4) << 24);
  // the chains of `products` for every tile; the warp's commit, its wait and the clock
  auto issue = [&](auto products) {
    constexpr int P = decltype(products)::value;
    const long long t0 = clock64();
    for (int r = 0; r < tiles; ++r) {
      if (P & 1) {      // (two accumulators; the third is product (2)'s operand)
#pragma unroll
        for (int ks = 0; ks < 8; ++ks)
          pp_mma_ss(tb + 128 * (r & 1), pp_desc(sA + ks * 2 * PP_PITCH, PP_PITCH, 128), pp_desc(sB + ks * 4096, 2048, 128), id_k, ks > 0);
        if (MASK & 16) pp_commit(bar + 24);
      }
      if (P & 2) {
#pragma unroll
        for (int ks = 0; ks < 8; ++ks)
          pp_mma_ts(tb + 448 + 16 * (r & 1), tb + 256 + 32 * (ks >> 1) + 8 * (ks & 1), pp_desc(sQ + ks * 2 * 272, 272, 128), id_s, ks > 0);
        if (MASK & 16) pp_commit(bar + 32);
      }
      if (P & 4) {
#pragma unroll
        for (int ks = 0; ks < 8; ++ks)
          pp_mma_ss(tb + 480 + 16 * (r & 1), pp_desc(sV + ks * 256, 128, PP_PITCH), pp_desc(sQ + ks * 256, 128, 0), id_o, 1);
        if (MASK & 16) pp_commit(bar + 40);
      }
    }
    pp_commit(bar + 8 * warp);
    bool ok = false;
    for (uint32_t it = 0; it < PROBE_SPIN && !ok; ++it) {
      uint32_t r;
      asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0,1,0,p;\n}"
                   : "=r"(r) : "r"(bar + 8 * warp), "r"(0u) : "memory");
      ok = __all_sync(0xffffffffu, r != 0);
    }
    const long long t1 = clock64();
    if ((tid & 31) == 0) {
      if (!ok) set_status(status, DKV_ST_TIMEOUT);
      cycles[(size_t)warp * gridDim.x + blockIdx.x] = t1 - t0;
    }
  };
  if (MASK & 64) {
    if (warp == 0) issue(std::integral_constant<int, 1>());
    if (warp == 1) issue(std::integral_constant<int, 2>());
    if (warp == 2) issue(std::integral_constant<int, 4>());
  } else {
    if (warp == 0) issue(std::integral_constant<int, (MASK & 7)>());
    if (warp == 1 && (MASK & 8)) issue(std::integral_constant<int, 4>());
  }
  __syncwarp();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tb), "r"(512));
  }
}

template <int MASK>
cudaError_t launch_probe(int n_cta, long long* cycles, int32_t* status, int tiles, cudaStream_t st) {
  cudaError_t e = cudaFuncSetAttribute(pipe_probe_kernel<MASK>, cudaFuncAttributeMaxDynamicSharedMemorySize, PROBE_SMEM);
  if (e == cudaSuccess) pipe_probe_kernel<MASK><<<n_cta, 128, PROBE_SMEM, st>>>(cycles, status, tiles);
  return e;
}

}  // namespace

}  // namespace dkv

using namespace dkv;

extern "C" int dkv_probe_tensor_pipe(int32_t products, int32_t tiles, int32_t n_cta, int64_t* cycles, int32_t* status,
                                     void* stream) {
  DKV_REQUIRE(((products >= 1 && products <= 7) || products == 11 || products == 23 || products == 39 || products == 43 || products == 71 || products == 103) && tiles >= 1 && tiles <= 100000 && n_cta >= 1 &&
                  n_cta <= 1024,
              DKV_E_ARG, "dkv_probe_tensor_pipe: products is a mask of 1|2|4 (or 11 = 1|2 from one warp with product "
                         "(3) from a second, 71 a warp per product), tiles in 1..100000, n_cta in 1..1024");
  DKV_REQUIRE(cycles != nullptr, DKV_E_ARG, "dkv_probe_tensor_pipe: null output");
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  long long* out = reinterpret_cast<long long*>(cycles);
  cudaError_t e = cudaSuccess;
  switch (products) {
    case 1: e = launch_probe<1>(n_cta, out, status, tiles, st); break;
    case 2: e = launch_probe<2>(n_cta, out, status, tiles, st); break;
    case 3: e = launch_probe<3>(n_cta, out, status, tiles, st); break;
    case 4: e = launch_probe<4>(n_cta, out, status, tiles, st); break;
    case 5: e = launch_probe<5>(n_cta, out, status, tiles, st); break;
    case 6: e = launch_probe<6>(n_cta, out, status, tiles, st); break;
    case 11: e = launch_probe<11>(n_cta, out, status, tiles, st); break;
    case 23: e = launch_probe<23>(n_cta, out, status, tiles, st); break;   // 7 with a commit behind every chain
    case 39: e = launch_probe<39>(n_cta, out, status, tiles, st); break;   // 7 over non-zero operands
    case 43: e = launch_probe<43>(n_cta, out, status, tiles, st); break;   // 11 over non-zero operands
    case 71: e = launch_probe<71>(n_cta, out, status, tiles, st); break;   // a warp per product
    case 103: e = launch_probe<103>(n_cta, out, status, tiles, st); break; // the same over non-zero operands
    default: e = launch_probe<7>(n_cta, out, status, tiles, st); break;
  }
  DKV_REQUIRE(e == cudaSuccess, DKV_E_CUDA, "dkv_probe_tensor_pipe: %s", cudaGetErrorString(e));
  DKV_CHECK_LAUNCH();
  return DKV_OK;
}
