// Cutoff gate: how many leading spectral coefficients of a token row are kept.
//   logits = b + x . W ; p = softmax(logits) ; c_j = p_0 + .. + p_j ;
//   length = #{ i < low_rank : c_{d-1-i} >= threshold }          (the kept set is a prefix: c is non-decreasing)
// Reference: kv_process_fused, src/dynakv/kernels/compressed_attention.py:84-119 (one side per call; the
// reference runs K and V rows through one concatenated softmax/cumsum call, which is row-wise anyway).
// Sums are fp32 whatever the storage type; with native_rounding the intermediate tensors are rounded to the storage
// type where the reference's torch ops materialise them.  Two kernels: the logits (8 rows per CTA, so that W is read
// once per 8 rows; the reduction is cut in chunks when there are few rows), then one warp per row for the rest.
#include <math.h>

#include <type_traits>

#include "dkv_common.cuh"
#include "dkv_tma.cuh"

namespace dkv {

constexpr int GATE_ROWS = 8;       // rows per CTA of the logits kernel
constexpr int GATE_MAX_DIM = 1024;
constexpr int GATE_TILE = 128;     // columns per CTA (one per thread) and reduction indices per chunk

// logits, split over column blocks (x), reduction chunks (y) and row tiles (z): part[y][row][col] =
// sum_{i in chunk y} x[row][i] * W[i][col].  fp32, i ascending.  With few rows (decode) the reduction is cut in
// d/128 chunks so that the d x d weight is read by many CTAs at once; the chunks are added in a fixed order by
// the second kernel, so the result does not depend on scheduling.
template <typename T>
__global__ void __launch_bounds__(GATE_TILE) gate_logits_kernel(dkv_gate_args p, int chunk_len, int stage_w) {
  __shared__ float xs[GATE_ROWS][GATE_MAX_DIM];
  extern __shared__ __align__(16) unsigned char gate_wtile[];   // [GATE_TILE][GATE_TILE] of T when stage_w
  const int d = p.dim, tid = threadIdx.x;
  const int col0 = blockIdx.x * GATE_TILE, col = col0 + tid;
  const int i0 = blockIdx.y * chunk_len, i1 = min(i0 + chunk_len, d);
  const int row0 = blockIdx.z * GATE_ROWS;
  const T* x = reinterpret_cast<const T*>(p.x);
  const T* w = reinterpret_cast<const T*>(p.w);
  if (stage_w) {
    // the whole 128 x 128 weight tile in one round of 16-byte async copies (one memory round trip instead of
    // one per group of rows); only used when the tile is complete and 16-byte aligned
    constexpr int PER_ROW = GATE_TILE * (int)sizeof(T) / 16;
    for (int e = tid; e < GATE_TILE * PER_ROW; e += GATE_TILE) {
      const int i = e / PER_ROW, c = e - i * PER_ROW;
      const unsigned dst = (unsigned)__cvta_generic_to_shared(gate_wtile + ((size_t)i * GATE_TILE) * sizeof(T) + c * 16);
      const unsigned char* src = reinterpret_cast<const unsigned char*>(w + (size_t)(i0 + i) * d + col0) + c * 16;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  for (int e = tid; e < GATE_ROWS * (i1 - i0); e += GATE_TILE) {
    const int r = e / (i1 - i0), i = e - r * (i1 - i0);
    xs[r][i] = (row0 + r < p.n_rows) ? to_f32(x[(size_t)(row0 + r) * p.x_stride + i0 + i]) : 0.f;
  }
  if (stage_w) asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  float acc[GATE_ROWS];
#pragma unroll
  for (int r = 0; r < GATE_ROWS; ++r) acc[r] = 0.f;
  if (col < d) {
    if (stage_w) {
      const T* wt = reinterpret_cast<const T*>(gate_wtile);
#pragma unroll 8
      for (int i = 0; i < GATE_TILE; ++i) {
        const float wv = to_f32(wt[i * GATE_TILE + tid]);
#pragma unroll
        for (int r = 0; r < GATE_ROWS; ++r) acc[r] = fmaf(xs[r][i], wv, acc[r]);
      }
    } else {
      int i = i0;
      for (; i + 8 <= i1; i += 8) {
        float wv[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) wv[u] = to_f32(w[(size_t)(i + u) * d + col]);   // 8 independent loads in flight
#pragma unroll
        for (int u = 0; u < 8; ++u)
#pragma unroll
          for (int r = 0; r < GATE_ROWS; ++r) acc[r] = fmaf(xs[r][i - i0 + u], wv[u], acc[r]);
      }
      for (; i < i1; ++i) {
        const float wv = to_f32(w[(size_t)i * d + col]);
#pragma unroll
        for (int r = 0; r < GATE_ROWS; ++r) acc[r] = fmaf(xs[r][i - i0], wv, acc[r]);
      }
    }
    float* part = reinterpret_cast<float*>(p.workspace) + (size_t)blockIdx.y * p.n_rows * d;
#pragma unroll
    for (int r = 0; r < GATE_ROWS; ++r)
      if (row0 + r < p.n_rows) part[(size_t)(row0 + r) * d + col] = acc[r];
  }
}

// The rest of a row, one warp per row, from its logits (in lg, shared memory) and this lane's partial maximum:
// softmax, running sum, count, optional masked copy.  Shared by the two-kernel path and the single-kernel path for
// narrow rows, so that both do the same arithmetic in the same order.
template <typename T>
__device__ __forceinline__ void gate_finish_row(const dkv_gate_args& p, int row, float* lg, float mx, int lane, bool native,
                                                float thr) {
  const int d = p.dim;
  mx = warp_max(mx);
  float z = 0.f;
  for (int j = lane; j < d; j += 32) {
    const float e = expf(lg[j] - mx);
    lg[j] = e;
    z += e;
  }
  z = warp_sum(z);
  __syncwarp();
  // lane l owns the contiguous columns [l*per, (l+1)*per): local sums, exclusive scan over lanes, then the walk
  const int per = (d + 31) / 32;
  const int j0 = min(lane * per, d), j1 = min(j0 + per, d);
  if (native) {   // softmax writes the probabilities in the storage type
    for (int j = lane; j < d; j += 32) lg[j] = to_f32(from_f32<T>(lg[j] / z));
    z = 1.f;
    __syncwarp();
  }
  float local = 0.f;
  for (int j = j0; j < j1; ++j) local += lg[j] / z;
  float incl = local;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const float t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  float run = incl - local;
  const int lo = d - min(max(p.low_rank, 0), d);   // only columns >= lo can count
  int cnt = 0;
  for (int j = j0; j < j1; ++j) {
    run += lg[j] / z;
    const float c = native ? to_f32(from_f32<T>(run)) : run;   // cumsum writes every running sum in the storage type
    if (j >= lo && c >= thr) ++cnt;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
  if (p.len_multiple > 1) cnt = min((cnt + p.len_multiple - 1) / p.len_multiple * p.len_multiple, d - d % p.len_multiple);
  if (lane == 0) p.lengths[row] = cnt;
  if (p.masked) {
    const T* x = reinterpret_cast<const T*>(p.x);
    T* out = reinterpret_cast<T*>(p.masked) + (size_t)row * p.masked_stride;
    const T* xr = x + (size_t)row * p.x_stride;
    for (int i = lane; i < d; i += 32) out[i] = i < cnt ? xr[i] : from_f32<T>(0.f);
  }
}

// one warp per row: logits = b + sum of the chunk partials, softmax, running sum, count
template <typename T>
__global__ void __launch_bounds__(256) gate_count_kernel(dkv_gate_args p, int n_chunks) {
  __shared__ float lg_s[8][GATE_MAX_DIM];
  const int d = p.dim, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int row = blockIdx.x * 8 + warp;
  if (row >= p.n_rows) return;
  const T* b = reinterpret_cast<const T*>(p.b);
  const bool native = p.native_rounding != 0 && sizeof(T) == 2;
  const float thr = native ? to_f32(from_f32<T>(p.threshold)) : p.threshold;   // the comparison converts the scalar
  const float* part = reinterpret_cast<const float*>(p.workspace);
  float* lg = lg_s[warp];
  float mx = -INFINITY;
  const size_t cstride = (size_t)p.n_rows * d;   // between the partials of consecutive chunks
  for (int jb = lane; jb < d; jb += 32 * 4) {
    // four columns at a time, all their partials loaded before the (fixed-order) additions
    float pv[4][8];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int j = jb + 32 * u;
#pragma unroll
      for (int c = 0; c < 8; ++c) pv[u][c] = (j < d && c < n_chunks) ? part[c * cstride + (size_t)row * d + j] : 0.f;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int j = jb + 32 * u;
      if (j < d) {
        float v = 0.f;
#pragma unroll
        for (int c = 0; c < 8; ++c) v += pv[u][c];
        v += to_f32(b[j]);
        if (native) v = to_f32(from_f32<T>(v));   // addmm writes the logits in the storage type
        lg[j] = v;
        mx = fmaxf(mx, v);
      }
    }
  }
  gate_finish_row<T>(p, row, lg, mx, lane, native, thr);
}

// Narrow rows (dim <= 128, the per-head decode shape), K and V sides in one launch: blockIdx.y picks the side, a
// CTA takes 8 rows; the logits go straight to shared memory (same fp32 sum, i ascending, as the two-kernel path
// with one reduction chunk), then one warp per row finishes as above.  Bound by latency: a 16-bit weight is fetched whole
// by asynchronous copies before anything else (512 rows a side of 128: 6.5 us, 19 with it read eight elements at a time).
template <typename T>
__global__ void __launch_bounds__(256) gate_small_kernel(dkv_gate_args pk, dkv_gate_args pv) {
  constexpr bool STAGED = sizeof(T) == 2;
  __shared__ __align__(16) T ws[STAGED ? GATE_TILE * GATE_TILE : 8];
  __shared__ __align__(16) float xs[8][GATE_TILE];
  __shared__ float lg_s[8][GATE_TILE];
  const dkv_gate_args& p = blockIdx.y ? pv : pk;
  const int d = p.dim, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int row0 = blockIdx.x * 8;
  const T* x = reinterpret_cast<const T*>(p.x);
  const T* w = reinterpret_cast<const T*>(p.w);
  const T* b = reinterpret_cast<const T*>(p.b);
  const bool native = p.native_rounding != 0 && sizeof(T) == 2;
  const float thr = native ? to_f32(from_f32<T>(p.threshold)) : p.threshold;
  const bool staged = STAGED && d % 8 == 0 && (reinterpret_cast<uintptr_t>(w) & 15) == 0;
  if (staged) {
    for (int e = tid; e < d * d / 8; e += 256)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(ws + 8 * e)), "l"(w + 8 * e) : "memory");
  }
  for (int e = tid; e < 8 * d; e += 256) {
    const int r = e / d, i = e - r * d;
    xs[r][i] = (row0 + r < p.n_rows) ? to_f32(x[(size_t)(row0 + r) * p.x_stride + i]) : 0.f;
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  {
    const int col = tid & (GATE_TILE - 1), rq = (tid >> 7) * 4;   // four rows per thread
    if (col < d) {
      float acc[4] = {0.f, 0.f, 0.f, 0.f};
      int i = 0;
      if (staged) {
#pragma unroll 4
        for (; i < d; i += 4) {
          float wv[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) wv[u] = to_f32(ws[(i + u) * d + col]);
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            const float4 xv = *reinterpret_cast<const float4*>(&xs[rq + r][i]);
            acc[r] = fmaf(xv.x, wv[0], acc[r]);
            acc[r] = fmaf(xv.y, wv[1], acc[r]);
            acc[r] = fmaf(xv.z, wv[2], acc[r]);
            acc[r] = fmaf(xv.w, wv[3], acc[r]);
          }
        }
      }
      for (; i + 8 <= d; i += 8) {
        float wv[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) wv[u] = to_f32(w[(size_t)(i + u) * d + col]);
#pragma unroll
        for (int u = 0; u < 8; ++u)
#pragma unroll
          for (int r = 0; r < 4; ++r) acc[r] = fmaf(xs[rq + r][i + u], wv[u], acc[r]);
      }
      for (; i < d; ++i) {
        const float wv = to_f32(w[(size_t)i * d + col]);
#pragma unroll
        for (int r = 0; r < 4; ++r) acc[r] = fmaf(xs[rq + r][i], wv, acc[r]);
      }
      const float bias = to_f32(b[col]);
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        float v = acc[r] + bias;
        if (native) v = to_f32(from_f32<T>(v));   // addmm writes the logits in the storage type
        lg_s[rq + r][col] = v;
      }
    }
  }
  __syncthreads();
  const int row = row0 + warp;
  if (row >= p.n_rows) return;
  float* lg = lg_s[warp];
  float mx = -INFINITY;
  for (int j = lane; j < d; j += 32) mx = fmaxf(mx, lg[j]);
  gate_finish_row<T>(p, row, lg, mx, lane, native, thr);
}

// ---- many 16-bit rows (a prompt): logits on the tensor core, then one warp per row with its columns in registers ----
//
// gate_gemm_kernel: logits = x W + b, of one side or of both in one launch.  Tiles of 128 rows x BN columns; the reduction
// runs over 64-wide stages, x as a K-major operand (boxes of 64 dims x 128 rows), W as it lies in memory, an MN-major
// operand (boxes of 64 columns x 64 dims), both by TMA in the 128-byte swizzle, as many stages in flight as shared memory
// holds.  One CTA per SM walks the tiles with two accumulators in tensor memory, so that a tile is read back and written
// while the next one is multiplied, and no wave is left half empty.  fp32 accumulation; the sum is rounded to the storage
// type only where the reference's addmm writes it (native rounding), and the logits then travel in that type (half the
// bytes).  Bound by the operands' way from L2 (48 KB per stage, ~45 bytes per SM and clock), before the tensor core: both
// sides of 8192 rows x 1024 take 36 us (2 x 21.6 with a CTA per tile, two stages and two CTAs an SM; 2 x 1161 on the CUDA
// cores); the products alone are 21 us.
constexpr int GG_ROWS = 128, GG_BK = 64, GG_RING = 192 * 1024, GG_THREADS = 192;
constexpr uint32_t GG_SPIN = 1u << 22;

__device__ __forceinline__ uint32_t gg_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ bool gg_wait(unsigned long long* bar, uint32_t parity) {
#pragma unroll 1
  for (uint32_t it = 0; it < GG_SPIN; ++it) {
    uint32_t r;
    asm volatile("{\n.reg .pred q;\nmbarrier.try_wait.parity.shared::cta.b64 q, [%1], %2;\nselp.u32 %0, 1, 0, q;\n}"
                 : "=r"(r) : "r"(gg_smem(bar)), "r"(parity) : "memory");
    if (r) return true;
  }
  return false;
}
__device__ __forceinline__ void gg_load(uint32_t dst, const CUtensorMap* map, int c0, int c1, unsigned long long* bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
               ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(gg_smem(bar)) : "memory");
}
// 128-byte swizzle descriptor: leading / stride byte offsets in 16-byte units
__device__ __forceinline__ uint64_t gg_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((addr >> 4) & 0x3FFF) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(sbo >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
template <typename T>
__device__ __forceinline__ uint32_t gg_pack(float lo, float hi) {
  if constexpr (std::is_same<T, __nv_bfloat16>::value) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
  } else {
    __half2 v = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
  }
}

template <typename T, int BN>
__global__ void __launch_bounds__(GG_THREADS) gate_gemm_kernel(const __grid_constant__ CUtensorMap map_xk, const __grid_constant__ CUtensorMap map_wk,
                                                               const __grid_constant__ CUtensorMap map_xv, const __grid_constant__ CUtensorMap map_wv,
                                                               const __grid_constant__ dkv_gate_args pk, const __grid_constant__ dkv_gate_args pv, int n_tiles) {
  constexpr int A_BYTES = GG_ROWS * GG_BK * 2, B_BYTES = BN * GG_BK * 2, STAGE = A_BYTES + B_BYTES, STAGES = GG_RING / STAGE;
  extern __shared__ unsigned char gg_raw[];
  // the swizzle is taken on absolute shared-memory addresses: tiles start on 1024-byte boundaries
  unsigned char* ring = gg_raw + ((1024u - (gg_smem(gg_raw) & 1023u)) & 1023u);
  __shared__ alignas(8) unsigned long long full[STAGES], empty[STAGES], acc_full[2], acc_empty[2];
  __shared__ uint32_t tmem_slot;
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const int n_k = pk.dim / GG_BK, cols = pk.dim / BN, per_side = cols * ((pk.n_rows + GG_ROWS - 1) / GG_ROWS);
  if (tid == 0) {
    for (int s = 0; s < STAGES; ++s) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(gg_smem(&full[s])));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(gg_smem(&empty[s])));
    }
    for (int s = 0; s < 2; ++s) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(gg_smem(&acc_full[s])));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(gg_smem(&acc_empty[s])), "n"(4));
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(gg_smem(&tmem_slot)), "r"(2 * BN));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_slot, 0);
  pdl_launch_dependents();
  if (warp == 0) {
    if (lane == 0) {
      bool ok = true;
      int s = 0;
      uint32_t turn = 0;      // rounds of the ring
      for (int t = blockIdx.x; t < n_tiles && ok; t += gridDim.x) {
        const int side = t >= per_side, u = t - side * per_side, n0 = (u % cols) * BN, row0 = (u / cols) * GG_ROWS;
        const CUtensorMap *mx = side ? &map_xv : &map_xk, *mw = side ? &map_wv : &map_wk;
        for (int k = 0; k < n_k; ++k) {
          if (turn > 0 && !(ok = gg_wait(&empty[s], (turn - 1) & 1))) break;
          const uint32_t a = gg_smem(ring) + s * STAGE, b = a + A_BYTES;
          asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(gg_smem(&full[s])), "r"(STAGE) : "memory");
          gg_load(a, mx, k * GG_BK, row0, &full[s]);
#pragma unroll
          for (int nb = 0; nb < BN / 64; ++nb) gg_load(b + nb * (64 * GG_BK * 2), mw, n0 + 64 * nb, k * GG_BK, &full[s]);
          if (++s == STAGES) { s = 0; ++turn; }
        }
      }
      if (!ok) {      // given up: reported, and the copies in flight waited for
        set_status(pk.status, DKV_ST_TIMEOUT);
        for (int i = 0; i < STAGES; ++i)
          if (i < s || turn > 0) gg_wait(&full[i], (i < s ? turn : turn - 1) & 1);
      }
    }
  } else if (warp == 1) {
    {     // a converged warp, whose elected lane's operands are known to be the same in all: both sides of 8192 rows x 1024 63.3 -> 61.5 us
      const uint32_t fmt = std::is_same<T, __nv_bfloat16>::value ? 1u : 0u;
      // D fp32, A K-major, B MN-major (bit 16), M = 128, N = BN
      const uint32_t idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | (1u << 16) | ((uint32_t)(BN >> 3) << 17) | ((128u >> 4) << 24);
      bool ok = true;
      int s = 0, j = 0;
      uint32_t turn = 0;
      for (int t = blockIdx.x; t < n_tiles && ok; t += gridDim.x, ++j) {
        if (j >= 2 && !(ok = __all_sync(0xffffffffu, gg_wait(&acc_empty[j & 1], (uint32_t)((j >> 1) - 1) & 1)))) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        for (int k = 0; k < n_k; ++k) {
          if (!(ok = __all_sync(0xffffffffu, gg_wait(&full[s], turn & 1)))) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t a = gg_smem(ring) + s * STAGE, b = a + A_BYTES;
#pragma unroll
          for (int ks = 0; ks < GG_BK / 16; ++ks) {
            // A: 8-row groups 1024 bytes apart, k-step 32 bytes on; B: 64-column blocks 64 * GG_BK * 2 bytes apart, groups of
            // 8 dims 1024 bytes apart, k-step two groups on
            const uint64_t da = gg_desc(a + 32 * ks, 16, 1024), db = gg_desc(b + 2048 * ks, 64 * GG_BK * 2, 1024);
            asm volatile("{\n.reg .pred q, e;\nelect.sync _|e, 0xffffffff;\nsetp.ne.b32 q, %4, 0;\n@e tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, q;\n}"
                         ::"r"(tmem + (j & 1) * BN), "l"(da), "l"(db), "r"(idesc), "r"(k + ks > 0 ? 1u : 0u) : "memory");
          }
          asm volatile("{\n.reg .pred e;\nelect.sync _|e, 0xffffffff;\n@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}" ::"r"(gg_smem(&empty[s])) : "memory");
          if (++s == STAGES) { s = 0; ++turn; }
        }
        if (ok) asm volatile("{\n.reg .pred e;\nelect.sync _|e, 0xffffffff;\n@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}" ::"r"(gg_smem(&acc_full[j & 1])) : "memory");
      }
      if (!ok) {      // given up: reported, and the products in flight waited for
        if (lane == 0) set_status(pk.status, DKV_ST_TIMEOUT);
        if (s > 0 || turn > 0) gg_wait(&empty[s > 0 ? s - 1 : STAGES - 1], (s > 0 ? turn : turn - 1) & 1);
      }
    }
  } else {
    const int quarter = warp & 3;         // the quarter of tensor memory that the warp may read
    unsigned char* const stage = ring + GG_RING + (warp - 2) * 4096;
    int j = 0;
    for (int t = blockIdx.x; t < n_tiles; t += gridDim.x, ++j) {
      const int side = t >= per_side, u = t - side * per_side, n0 = (u % cols) * BN, row = (u / cols) * GG_ROWS + 32 * quarter + lane;
      const dkv_gate_args& p = side ? pv : pk;
      const T* bias = reinterpret_cast<const T*>(p.b) + n0;
      const bool native = p.native_rounding != 0;
      if (!__all_sync(0xffffffffu, gg_wait(&acc_full[j & 1], (uint32_t)(j >> 1) & 1))) {
        if (lane == 0) set_status(p.status, DKV_ST_TIMEOUT);
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t lane_addr = tmem + (j & 1) * BN + ((uint32_t)(32 * quarter) << 16);
      // 32 columns of the thread's row at a time go through the warp's 4 KB of shared memory and leave as whole 128-byte
      // lines (16-byte pieces of 32 rows per store made the read-back as long as the products); 16-byte piece q of row r
      // lies at (q ^ r % 8) * 16 of the row
      const int row_base = row - lane;
      const size_t es = native ? sizeof(T) : sizeof(float), pitch = (size_t)p.dim * es;
      unsigned char* const out = reinterpret_cast<unsigned char*>(p.workspace) + (size_t)row_base * pitch + (size_t)n0 * es;
      auto flush = [&](int c) {        // 128 bytes of each row from column c on
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int r = 4 * i + (lane >> 3), q = lane & 7;
          if (row_base + r < p.n_rows)
            *reinterpret_cast<uint4*>(out + r * pitch + c * es + 16 * q) = *reinterpret_cast<const uint4*>(stage + r * 128 + ((q ^ (r & 7)) << 4));
        }
        __syncwarp();
      };
#pragma unroll 1
      for (int c = 0; c < BN; c += 32) {
        uint32_t r[32];
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n"
            "tcgen05.wait::ld.sync.aligned;"
            : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
              "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
              "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
              "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
            : "r"(lane_addr + c) : "memory");
        float v[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]) + to_f32(__ldg(bias + c + i));
        if (native) {      // two rounds make a line
          const int q0 = (c & 32) >> 3;
#pragma unroll
          for (int i = 0; i < 4; ++i)
            *reinterpret_cast<uint4*>(stage + lane * 128 + (((q0 + i) ^ (lane & 7)) << 4)) =
                make_uint4(gg_pack<T>(v[8 * i], v[8 * i + 1]), gg_pack<T>(v[8 * i + 2], v[8 * i + 3]),
                           gg_pack<T>(v[8 * i + 4], v[8 * i + 5]), gg_pack<T>(v[8 * i + 6], v[8 * i + 7]));
          if (c & 32) flush(c - 32);
        } else {
#pragma unroll
          for (int i = 0; i < 8; ++i)
            *reinterpret_cast<float4*>(stage + lane * 128 + ((i ^ (lane & 7)) << 4)) = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
          flush(c);
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(gg_smem(&acc_empty[j & 1])) : "memory");
    }
  }
  __syncwarp();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * BN));
  }
}

// The least float whose rounding to T reaches thr (itself a value of T): rounding is monotonic, so comparing an unrounded sum
// with this bound is comparing the rounded one with thr.  The bound is the middle between thr and the value of T below it,
// which rounds to thr when thr's last bit is even, or the float after it.  (Sums are not negative: bounds <= 0 stay.)
template <typename T>
__device__ __forceinline__ float rounded_bound(float thr) {
  if (!(thr > 0.f) || isinf(thr)) return thr;
  const T t = from_f32<T>(thr);
  uint16_t u = *reinterpret_cast<const uint16_t*>(&t);
  const bool even = (u & 1) == 0;
  --u;
  const float mid = 0.5f * (thr + to_f32(*reinterpret_cast<const T*>(&u)));     // exact
  return even ? mid : __uint_as_float(__float_as_uint(mid) + 1);
}
// a / b for y = 1 / b correctly rounded, two at a time: a quotient within one last place and two remainders (Markstein,
// "Computation of elementary functions on the IBM RISC System/6000 processor", 1990).  It is the result of the division as long
// as the remainders are exact, that is down to about a = 2^-102 for b in 1..1024; below (exponentials of logits 71 or more under the
// row's largest) it may be off in the last place, of terms too small to change a sum that holds the largest.
__device__ __forceinline__ float2 quotient2(float2 a, float2 neg_b, float2 y) {
  float2 q = __fmul2_rn(a, y);
  q = __ffma2_rn(__ffma2_rn(q, neg_b, a), y, q);
  return __ffma2_rn(__ffma2_rn(q, neg_b, a), y, q);
}

// gate_rows_kernel: softmax, running sum, count and masked copy of a row whose logits gate_gemm_kernel left in the
// workspace; lane l holds columns PER l .. PER l + PER - 1 in registers.  The work is one read of the logits, one of x
// and one write of the masked row; bound by the instructions of a row.  Both sides of 8192 rows x 1024, bf16: 2 x 98 us with
// the columns in (bank-conflicted) shared memory, 27 us in registers and one launch (1230 instructions a row, 0.69 of the issue
// slots), now 22: one reciprocal and exact remainders for the divisions by the row's sum, the bound compared instead of each
// sum rounded, roundings of pairs.  (Call with the logits: 61.5 -> 57.5 us.)
template <typename T, bool NATIVE, int PER>
__global__ void __launch_bounds__(256) gate_rows_kernel(const __grid_constant__ dkv_gate_args pk, const __grid_constant__ dkv_gate_args pv) {
  const dkv_gate_args& p = blockIdx.y ? pv : pk;
  const int lane = threadIdx.x & 31, row = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (row >= p.n_rows) return;
  pdl_wait();       // the logits come from gate_gemm_kernel
  constexpr int d = 32 * PER;
  // the comparison converts the scalar; cumsum writes every running sum in the storage type
  const float thr = NATIVE ? rounded_bound<T>(to_f32(from_f32<T>(p.threshold))) : p.threshold;
  float e[PER];
  if (NATIVE) {
    constexpr int W = PER < 8 ? PER : 8;           // columns of a load
    struct alignas(2 * W) Piece { T t[W]; };
    const Piece* src = reinterpret_cast<const Piece*>(reinterpret_cast<const T*>(p.workspace) + (size_t)row * d + PER * lane);
#pragma unroll
    for (int i = 0; i < PER / W; ++i) {
      const Piece v = src[i];
#pragma unroll
      for (int k = 0; k < W; ++k) e[W * i + k] = to_f32(v.t[k]);
    }
  } else {
    const float4* src = reinterpret_cast<const float4*>(reinterpret_cast<const float*>(p.workspace) + (size_t)row * d + PER * lane);
#pragma unroll
    for (int i = 0; i < PER / 4; ++i) {
      const float4 v = src[i];
      e[4 * i] = v.x; e[4 * i + 1] = v.y; e[4 * i + 2] = v.z; e[4 * i + 3] = v.w;
    }
  }
  float mx = e[0];
#pragma unroll
  for (int i = 1; i < PER; ++i) mx = fmaxf(mx, e[i]);
  mx = warp_max(mx);
  float z = 0.f;
#pragma unroll
  for (int i = 0; i < PER; ++i) { e[i] = expf(e[i] - mx); z += e[i]; }
  z = warp_sum(z);
  float local = 0.f;
  const float y = __frcp_rn(z);
#pragma unroll
  for (int i = 0; i < PER; i += 2) {
    const float2 q = quotient2(make_float2(e[i], e[i + 1]), make_float2(-z, -z), make_float2(y, y));
    e[i] = q.x;
    e[i + 1] = q.y;
    if (NATIVE) {      // softmax writes the probabilities in the storage type
      const uint32_t w = gg_pack<T>(q.x, q.y);
      const T* const t = reinterpret_cast<const T*>(&w);
      e[i] = to_f32(t[0]);
      e[i + 1] = to_f32(t[1]);
    }
    local += e[i];
    local += e[i + 1];
  }
  float incl = local;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const float t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  float run = incl - local;
  const int lo = d - min(max(p.low_rank, 0), d);   // only columns >= lo can count
  int below = 0;      // the lane's sums do not fall: those that do not reach the bound (or are no numbers) come first
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    run += e[i];
    below += !(run >= thr);
  }
  int cnt = PER - max(below, min(max(lo - PER * lane, 0), PER));
  cnt = __reduce_add_sync(0xffffffffu, cnt);
  if (p.len_multiple > 1) cnt = min((cnt + p.len_multiple - 1) / p.len_multiple * p.len_multiple, d - d % p.len_multiple);
  if (lane == 0) p.lengths[row] = cnt;
  if (p.masked) {
    const T* xr = reinterpret_cast<const T*>(p.x) + (size_t)row * p.x_stride;
    T* out = reinterpret_cast<T*>(p.masked) + (size_t)row * p.masked_stride;
    if (((reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(xr)) & 15) == 0) {
#pragma unroll
      for (int i0 = 0; i0 < d; i0 += 256) {
        const int i = i0 + 8 * lane;
        if (i >= d) break;
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (i < cnt) v = __ldcs(reinterpret_cast<const uint4*>(xr + i));
        if (i + 8 > cnt && i < cnt) {
          T* t = reinterpret_cast<T*>(&v);
#pragma unroll
          for (int k = 0; k < 8; ++k)
            if (i + k >= cnt) t[k] = from_f32<T>(0.f);
        }
        __stcs(reinterpret_cast<uint4*>(out + i), v);
      }
    } else {
      for (int i = lane; i < d; i += 32) out[i] = i < cnt ? xr[i] : from_f32<T>(0.f);
    }
  }
}

// The tensor-core path takes blocks of more than 64 rows (fewer: the reduction split over CTAs reads W at once) of 16-bit
// types whose width is a whole number of its column tiles and that TMA can address.
static bool gate_gemm_ok(const dkv_gate_args* a) {
  return a->dtype != DKV_F32 && a->n_rows > 64 && (a->dim == 128 || a->dim == 256 || a->dim == 512 || a->dim == 1024) &&
         (((uintptr_t)a->x | (uintptr_t)a->w | (uintptr_t)a->workspace) & 15) == 0 && a->x_stride % 8 == 0;
}

template <typename T, int BN>
static cudaError_t launch_gate_gemm(const dkv_gate_args* a, const dkv_gate_args* b, const CUtensorMap (&m)[4], int row_tiles, cudaStream_t st) {
  const int smem = GG_RING + 4 * 4096 + 1024, n_tiles = row_tiles * (a->dim / BN);
  const cudaError_t e = cudaFuncSetAttribute(gate_gemm_kernel<T, BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e == cudaSuccess) gate_gemm_kernel<T, BN><<<min(n_tiles, sm_count()), GG_THREADS, smem, st>>>(m[0], m[1], m[2], m[3], *a, *b, n_tiles);
  return e;
}
// one side (b == a), or two sides of one shape in one launch each
template <typename T>
static int gate_prompt(const dkv_gate_args* a, const dkv_gate_args* b) {
  cudaStream_t st = reinterpret_cast<cudaStream_t>(a->stream);
  const int sides = a == b ? 1 : 2;
  CUtensorMap m[4];
  for (int i = 0; i < 2; ++i) {
    const dkv_gate_args* s = i ? b : a;
    DKV_REQUIRE(tensor_map_16bit(&m[2 * i], s->dtype, s->x, (uint64_t)s->n_rows, (uint64_t)s->dim, (uint64_t)s->x_stride, GG_ROWS) &&
                    tensor_map_16bit(&m[2 * i + 1], s->dtype, s->w, (uint64_t)s->dim, (uint64_t)s->dim, (uint64_t)s->dim, GG_BK),
                DKV_E_CUDA, "dkv_gate_lengths: tensor map encoding failed");
  }
  // 256-column tiles (a quarter less through L2 per product) once they give every SM one; 256 x 256 ones, which leave no
  // second accumulator, were slower (39 against 36 us)
  const int row_tiles = sides * ((a->n_rows + GG_ROWS - 1) / GG_ROWS);
  const bool wide = a->dim % 256 == 0 && (long long)row_tiles * (a->dim / 256) >= sm_count();
  const cudaError_t e = wide ? launch_gate_gemm<T, 256>(a, b, m, row_tiles, st) : launch_gate_gemm<T, 128>(a, b, m, row_tiles, st);
  DKV_REQUIRE(e == cudaSuccess, DKV_E_CUDA, "dkv_gate_lengths: %s", cudaGetErrorString(e));
  DKV_CHECK_LAUNCH();
  const dim3 grid((a->n_rows + 7) / 8, sides);
  cudaError_t r = cudaSuccess;
#define ROWS(NAT)                                                                                       \
  do {                                                                                                  \
    if (a->dim == 128) r = launch_pdl(gate_rows_kernel<T, NAT, 4>, grid, dim3(256), 0, st, *a, *b);       \
    else if (a->dim == 256) r = launch_pdl(gate_rows_kernel<T, NAT, 8>, grid, dim3(256), 0, st, *a, *b);  \
    else if (a->dim == 512) r = launch_pdl(gate_rows_kernel<T, NAT, 16>, grid, dim3(256), 0, st, *a, *b); \
    else r = launch_pdl(gate_rows_kernel<T, NAT, 32>, grid, dim3(256), 0, st, *a, *b);                    \
  } while (0)
  if (a->native_rounding) ROWS(true); else ROWS(false);
#undef ROWS
  DKV_REQUIRE(r == cudaSuccess, DKV_E_CUDA, "dkv_gate_lengths: %s", cudaGetErrorString(r));
  DKV_CHECK_LAUNCH();
  return DKV_OK;
}

static int gate_chunks(const dkv_gate_args* a) {
  // few rows: cut the reduction so that d/128 x d/128 CTAs share the weight read; many rows: the row tiles
  // already fill the GPU
  return a->n_rows <= 64 ? (a->dim + GATE_TILE - 1) / GATE_TILE : 1;   // at most 8 (dim <= 1024)
}

}  // namespace dkv

extern "C" size_t dkv_gate_workspace_bytes(const dkv_gate_args* a) {
  if (a == nullptr || a->n_rows <= 0 || a->dim <= 0) return 0;
  return (size_t)dkv::gate_chunks(a) * (size_t)a->n_rows * (size_t)a->dim * sizeof(float);
}

static int check_gate(const dkv_gate_args* a) {
  using namespace dkv;
  DKV_REQUIRE(a != nullptr, DKV_E_ARG, "dkv_gate_lengths: null args");
  DKV_REQUIRE(a->dtype >= DKV_F32 && a->dtype <= DKV_BF16, DKV_E_ARG, "dkv_gate_lengths: bad dtype %d", a->dtype);
  DKV_REQUIRE(a->n_rows >= 0 && a->dim >= 1 && a->dim <= GATE_MAX_DIM, DKV_E_LIMIT,
              "dkv_gate_lengths: dim must be in 1..%d, got %d", GATE_MAX_DIM, a->dim);
  DKV_REQUIRE(a->x && a->w && a->b && a->lengths, DKV_E_ARG, "dkv_gate_lengths: null input");
  DKV_REQUIRE(a->x_stride >= a->dim && (!a->masked || a->masked_stride >= a->dim), DKV_E_ARG,
              "dkv_gate_lengths: row strides must be at least dim");
  DKV_REQUIRE(a->n_rows == 0 || (a->workspace != nullptr && a->workspace_bytes >= dkv_gate_workspace_bytes(a)), DKV_E_WORKSPACE,
              "dkv_gate_lengths: workspace too small: need %zu bytes, got %zu", dkv_gate_workspace_bytes(a), a->workspace_bytes);
  DKV_REQUIRE((a->n_rows + GATE_ROWS - 1) / GATE_ROWS <= 65535, DKV_E_LIMIT, "dkv_gate_lengths: at most %d rows per call", 65535 * GATE_ROWS);
  return DKV_OK;
}

extern "C" int dkv_gate_lengths(const dkv_gate_args* a) {
  using namespace dkv;
  if (int rc = check_gate(a)) return rc;
  if (a->n_rows == 0) return DKV_OK;
  if (gate_gemm_ok(a)) return a->dtype == DKV_F16 ? gate_prompt<__half>(a, a) : gate_prompt<__nv_bfloat16>(a, a);
  cudaStream_t st = reinterpret_cast<cudaStream_t>(a->stream);
  const int n_chunks = gate_chunks(a);
  const int chunk_len = n_chunks == 1 ? a->dim : GATE_TILE;
  dim3 grid((a->dim + GATE_TILE - 1) / GATE_TILE, n_chunks, (a->n_rows + GATE_ROWS - 1) / GATE_ROWS);
  const int cgrid = (a->n_rows + 7) / 8;
  // weight tiles are staged through shared memory when the reduction is chunked and every tile is whole and aligned
  const size_t esz = dtype_size(a->dtype);
  const int stage_w = (n_chunks > 1 && a->dim % GATE_TILE == 0 && ((uintptr_t)a->w & 15) == 0) ? 1 : 0;
  const size_t wsmem = stage_w ? (size_t)GATE_TILE * GATE_TILE * esz : 0;
#define LAUNCH(T)                                                                        \
  do {                                                                                   \
    if (wsmem > 0) /* static 32 KB + the tile exceed the default 48 KB */                \
      cudaFuncSetAttribute(gate_logits_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)wsmem); \
    gate_logits_kernel<T><<<grid, GATE_TILE, wsmem, st>>>(*a, chunk_len, stage_w);       \
    gate_count_kernel<T><<<cgrid, 256, 0, st>>>(*a, n_chunks);                           \
  } while (0)
  if (a->dtype == DKV_F32) LAUNCH(float);
  else if (a->dtype == DKV_F16) LAUNCH(__half);
  else LAUNCH(__nv_bfloat16);
#undef LAUNCH
  DKV_CHECK_LAUNCH();
  return DKV_OK;
}

extern "C" int dkv_gate_lengths_both(const dkv_gate_args* k, const dkv_gate_args* v) {
  using namespace dkv;
  if (int rc = check_gate(k)) return rc;
  if (int rc = check_gate(v)) return rc;
  // one shape and rounding, and scratch of their own: one launch of each kernel takes both sides
  if (k->n_rows > 0 && k->dtype == v->dtype && k->dim == v->dim && k->n_rows == v->n_rows && k->stream == v->stream &&
      k->native_rounding == v->native_rounding && k->workspace != v->workspace && gate_gemm_ok(k) && gate_gemm_ok(v))
    return k->dtype == DKV_F16 ? gate_prompt<__half>(k, v) : gate_prompt<__nv_bfloat16>(k, v);
  if (int rc = dkv_gate_lengths(k)) return rc;
  return dkv_gate_lengths(v);
}

extern "C" int dkv_gate_lengths_pair(const dkv_gate_args* k, const dkv_gate_args* v) {
  using namespace dkv;
  DKV_REQUIRE(k != nullptr && v != nullptr, DKV_E_ARG, "dkv_gate_lengths_pair: null args");
  DKV_REQUIRE(k->dtype == v->dtype && k->dim == v->dim && k->n_rows == v->n_rows && k->stream == v->stream, DKV_E_ARG,
              "dkv_gate_lengths_pair: the two sides must agree in dtype, dim, rows and stream");
  DKV_REQUIRE(k->dtype >= DKV_F32 && k->dtype <= DKV_BF16, DKV_E_ARG, "dkv_gate_lengths_pair: bad dtype %d", k->dtype);
  DKV_REQUIRE(k->n_rows >= 0 && k->dim >= 1 && k->dim <= GATE_TILE, DKV_E_LIMIT,
              "dkv_gate_lengths_pair: dim must be in 1..%d (wider rows: dkv_gate_lengths per side)", GATE_TILE);
  for (const dkv_gate_args* a : {k, v}) {
    DKV_REQUIRE(a->x && a->w && a->b && a->lengths, DKV_E_ARG, "dkv_gate_lengths_pair: null input");
    DKV_REQUIRE(a->x_stride >= a->dim && (!a->masked || a->masked_stride >= a->dim), DKV_E_ARG,
                "dkv_gate_lengths_pair: row strides must be at least dim");
  }
  if (k->n_rows == 0) return DKV_OK;
  DKV_REQUIRE((k->n_rows + 7) / 8 <= 2147483647 / 8, DKV_E_LIMIT, "dkv_gate_lengths_pair: too many rows");
  cudaStream_t st = reinterpret_cast<cudaStream_t>(k->stream);
  const dim3 grid((k->n_rows + 7) / 8, 2);
  if (k->dtype == DKV_F32) gate_small_kernel<float><<<grid, 256, 0, st>>>(*k, *v);
  else if (k->dtype == DKV_F16) gate_small_kernel<__half><<<grid, 256, 0, st>>>(*k, *v);
  else gate_small_kernel<__nv_bfloat16><<<grid, 256, 0, st>>>(*k, *v);
  DKV_CHECK_LAUNCH();
  return DKV_OK;
}
