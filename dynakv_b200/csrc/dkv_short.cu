// Short-cache decode attention over packed per-KV-head arenas (bf16 / fp16, D = 128, R <= 128, lengths multiples of 8):
// one cluster of CTAs per (batch row, KV head), one 128-token tile per CTA, result projected in-kernel.
//
// A short row is a chain of latencies, not work: 500 tokens are four tiles and 15 KB.  So a CTA takes one tile through its
// two products with all of its 512 threads and no pipeline -- a thread owns a quarter of a token's row in every step
// (gather, rotation, scores) -- and the tiles of a row run at the same time on the CTAs of a cluster, which merge their
// partial results in distributed shared memory and share the up-projection by query head.  (Rows of more tiles than the
// cluster has CTAs are walked with a running softmax.)  Everything that does not depend on the kernel before this one
// (basis, tensor memory, barriers) is set up before griddepcontrol.wait.
// Per launch in a chain (8 KV heads, bf16), against the warp-specialised pipeline of dkv_mma_decode.cu, one CTA per row:
// B = 1, 499 tokens 16.1 -> 10.7 us; B = 4, 1 token 12.1 -> 10.2, 499 tokens 16.3 -> 12.0; B = 64, 128 tokens 49.5 -> 32.1 (with a
// workspace such batches go through the split kernel).
//
// Reference math: src/dynakv/kernels/fused.py:28-142.
#include <math.h>

#include <type_traits>

#include "dkv_common.cuh"

namespace dkv {

namespace {

constexpr int SD = 128;                 // head_dim
constexpr int ST = 128;                 // tokens per tile
constexpr int STHREADS = 512;
constexpr int SHP = 4;                  // query heads per KV head
constexpr int SCLUSTER = 4;             // CTAs per row at most
// A routed call whose rows can be no longer is one launch of this kernel: two rounds of tiles per CTA at most.  Measured (us,
// against split and merge for all rows; 1, 2, 4, 8 KV heads and every batch that short_ok admits): 600 to 1024 tokens 13.7-15.4
// and 14.6-24, at 128 CTAs 15.1-16.0 and 15.5-15.8, 32 rows of one KV head 16.1-18.8 and 15.8; 1 row of 1400 tokens 18.6 and 15.1.
constexpr int SHORT_ALL_TOKENS = 1024;
constexpr uint32_t SSPIN = 1u << 22;
constexpr uint32_t S_TM_K = 0, S_TM_O = 128, S_TMEM_COLS = 256;

struct ShortSmem {
  alignas(128) unsigned char x[ST * 256];       // piece c (8 coefficients) of token t at c*2048 + t*16
  alignas(128) unsigned char v[ST * 256];
  alignas(128) unsigned char basis[128 * 256];  // Bk[r][d] at (r/8)*2048 + (d/8)*128 + (r%8)*16 + (d%8)*2
  alignas(128) unsigned char p[ST * 16];        // weights of token t at t*16: heads 0..3, then their remainders
  alignas(16) float q[SHP][SD];                 // scaled queries
  alignas(16) float part[3][ST][SHP];           // partial scores of a token's quarters 1..3 (two CTAs' memory just fits an SM)
  alignas(16) float lat[SHP][SD];               // this CTA's latent sums
  alignas(16) float ml[2][SHP];                 // its maxima and weight sums
  float ss[4][ST];
  float knw[SD];
  alignas(16) uint32_t phi[64];                 // turns per token, 2^-32
  float wmax[4][SHP], wsum[4][SHP];
  alignas(8) unsigned long long bar[3];
  uint32_t tmem;
};

static_assert(2 * (sizeof(ShortSmem) + 128 + 1024) <= 228 * 1024, "two CTAs per SM");

__device__ __forceinline__ uint32_t ss_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ bool ss_wait(unsigned long long* bar, uint32_t parity) {
#pragma unroll 1
  for (uint32_t it = 0; it < SSPIN; ++it) {
    uint32_t r;
    asm volatile("{\n.reg .pred q;\nmbarrier.try_wait.parity.shared::cta.b64 q, [%1], %2;\nselp.u32 %0, 1, 0, q;\n}"
                 : "=r"(r) : "r"(ss_addr(bar)), "r"(parity) : "memory");
    if (r) return true;
  }
  return false;
}
__device__ __forceinline__ uint64_t ss_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((addr >> 4) & 0x3FFF) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(sbo >> 4) << 32) | (1ull << 46);
}
// Called by a converged warp with operands that are the same in all lanes; an elected lane issues (in a branch of a single lane
// the operands are not known to be uniform: a decode step of 4 short rows through 32 layers 793 -> 733 us).
__device__ __forceinline__ void ss_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, bool acc) {
  asm volatile("{\n.reg .pred q, e;\nelect.sync _|e, 0xffffffff;\nsetp.ne.b32 q, %4, 0;\n@e tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, q;\n}"
               ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(acc ? 1u : 0u) : "memory");
}
__device__ __forceinline__ void ss_commit(unsigned long long* bar) {
  asm volatile("{\n.reg .pred e;\nelect.sync _|e, 0xffffffff;\n@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}" ::"r"(ss_addr(bar)) : "memory");
}
// columns c .. c+7 and c+64 .. c+71 of this thread's lane
__device__ __forceinline__ void ss_ld_pairs(float (&lo)[8], float (&hi)[8], uint32_t addr) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%16];\n"
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%8,%9,%10,%11,%12,%13,%14,%15}, [%17];\n"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(addr), "r"(addr + 64) : "memory");
#pragma unroll
  for (int i = 0; i < 8; ++i) { lo[i] = __uint_as_float(r[i]); hi[i] = __uint_as_float(r[8 + i]); }
}
// maximum over the warp (order-preserving map float <-> int)
__device__ __forceinline__ float redux_max(float v) {
  int i = __float_as_int(v);
  i ^= (i >> 31) & 0x7fffffff;
  i = __reduce_max_sync(0xffffffffu, i);
  return __int_as_float(i ^ ((i >> 31) & 0x7fffffff));
}
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ float dsmem_f32(const void* p, uint32_t rank) {
  uint32_t a;
  float v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(ss_addr(p)), "r"(rank));
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
  return v;
}
template <typename T>
__device__ __forceinline__ uint32_t ss_pack(float a, float b) {
  if constexpr (std::is_same<T, __nv_bfloat16>::value) {
    __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&v);
  } else {
    __half2 v = __floats2half2_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&v);
  }
}

template <typename T, bool KNORM>
__global__ void __launch_bounds__(STHREADS, 2) short_decode_kernel(dkv_attn_args p, float log_theta) {
  extern __shared__ unsigned char ss_raw[];
  ShortSmem& sm = *reinterpret_cast<ShortSmem*>(ss_raw + ((128u - (ss_addr(ss_raw) & 127u)) & 127u));
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;     // (the warp: known to be the same in all lanes)
  const int tok = tid & 127, quarter = tid >> 7;
  const int CS = (int)(gridDim.x / p.batch), rank = (int)cluster_rank();
  const int i_row = blockIdx.x / CS, g = blockIdx.y;
  const int G = p.n_q_heads / p.n_basis_groups, R = p.rank;

  // ---- set-up that reads only the bases: overlaps the end of the kernel before this one ----
  {
    const T* kup = reinterpret_cast<const T*>(p.k_up) + (size_t)g * R * SD;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int e = tid + u * STHREADS, r = e >> 4, d = e & 15;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;"
                   ::"r"(ss_addr(sm.basis + (r >> 3) * 2048 + d * 128 + (r & 7) * 16)), "l"(kup + (size_t)min(r, R - 1) * SD + 8 * d), "r"(r < R ? 16 : 0) : "memory");
    }
  }
  if (tid < 64) {
    const float f = expf(-((float)(2 * tid) / (float)SD) * log_theta);
    sm.phi[tid] = (uint32_t)(long long)llrint((double)f * 683565275.57643158978229477811035);   // 2^32 / (2 pi)
  }
  if (tid == 64) {
    for (int s = 0; s < 3; ++s) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(ss_addr(&sm.bar[s])));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 4) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(ss_addr(&sm.tmem)), "r"(S_TMEM_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (CS > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");     // all CTAs have started before any reads another's memory
  pdl_wait();
  const int b = p.batch_index ? p.batch_index[i_row] : i_row;
  const int a = b * p.arenas_per_batch + g;
  // the row's length, the query and the first tile's metadata are asked for together (columns below seq_len exist
  // whatever the row's length)
  int lk = 0, lv = 0, ok_ = 0, ov = 0;
  auto load_meta = [&](int s) {
    lk = lv = ok_ = ov = 0;
    if (s < p.seq_len) {
      lk = p.k.lens[(size_t)a * p.k.lens_stride_a + s];
      ok_ = p.k.offs[(size_t)a * p.k.offs_stride_a + s];
      lv = p.v.lens[(size_t)a * p.v.lens_stride_a + s];
      ov = p.v.offs[(size_t)a * p.v.offs_stride_a + s];
    }
  };
  load_meta(rank * ST + tok);
  float qv = 0.f;
  if (quarter < G) qv = to_f32((reinterpret_cast<const T*>(p.q) + (size_t)b * p.q_stride_b + (size_t)(g * G + quarter) * p.q_stride_h)[tok]);
  if (KNORM && tid < SD) sm.knw[tid] = p.k_norm_weight[tid];
  int n_tok = p.seq_len;
  if (p.seq_lens) n_tok = min(n_tok, max(p.seq_lens[b], 0));
  const bool mine = !row_routed_out(p, b);      // else the row belongs to the other kernel: nothing is written
  const int n_tile = mine ? (n_tok + ST - 1) / ST : 0;
  sm.q[quarter][tok] = qv * (rsqrtf((float)SD) * 1.4426950408889634f);      // softmax scale and log2(e) folded in
  float m_run[SHP], l_run[SHP], o_run[SHP];      // of all heads (o: latent `tok`), in the threads of quarter 0
#pragma unroll
  for (int h = 0; h < SHP; ++h) { m_run[h] = -INFINITY; l_run[h] = 0.f; o_run[h] = 0.f; }
  const uint32_t fmt = std::is_same<T, __nv_bfloat16>::value ? 1u : 0u;
  const uint32_t idesc_k = (1u << 4) | (fmt << 7) | (fmt << 10) | (1u << 16) | ((128u >> 3) << 17) | ((128u >> 4) << 24);
  const uint32_t idesc_o = (1u << 4) | (fmt << 7) | (fmt << 10) | (1u << 15) | (1u << 16) | ((16u >> 3) << 17) | ((128u >> 4) << 24);
  const bool v_vec = (reinterpret_cast<uintptr_t>(p.v_up) & 15) == 0;
  auto load_bv = [&]() {      // Bv takes the place of X: piece d/8 of row r at (d/8)*2048 + r*16
    const T* vup = reinterpret_cast<const T*>(p.v_up) + (size_t)g * R * SD;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int e = tid + u * STHREADS, r = e >> 4, d = e & 15;
      unsigned char* dst = sm.x + d * 2048 + r * 16;
      if (v_vec) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(ss_addr(dst)), "l"(vup + (size_t)min(r, R - 1) * SD + 8 * d), "r"(r < R ? 16 : 0) : "memory");
      } else {
        for (int k = 0; k < 8; ++k) reinterpret_cast<T*>(dst)[k] = r < R ? vup[(size_t)r * SD + 8 * d + k] : from_f32<T>(0.f);
      }
    }
  };
  bool ok = true;
  uint32_t phase = 0;
  for (int tile = rank; tile < n_tile; tile += CS, phase ^= 1u) {
    // ---- gather: this thread's quarter (four 16-byte pieces a side) of its token's rows, zeros past their ends ----
    const int s = tile * ST + tok;
    if (tile != rank) load_meta(s);
    if (s >= n_tok) lk = lv = ok_ = ov = 0;
    if (((lk | ok_) & 7) != 0 || (unsigned)lk > (unsigned)R || ok_ < 0 || (int64_t)ok_ + lk > p.k.flat_stride) {
      set_status(p.status, DKV_ST_BAD_LENGTH);       // breaks the layout contract: token dropped, call flagged
      lk = 0;
    }
    if (((lv | ov) & 7) != 0 || (unsigned)lv > (unsigned)R || ov < 0 || (int64_t)ov + lv > p.v.flat_stride) {
      set_status(p.status, DKV_ST_BAD_LENGTH);
      lv = 0;
    }
    const T* ksrc = reinterpret_cast<const T*>(p.k.flat) + (size_t)a * p.k.flat_stride + (lk > 0 ? ok_ : 0);
    const T* vsrc = reinterpret_cast<const T*>(p.v.flat) + (size_t)a * p.v.flat_stride + (lv > 0 ? ov : 0);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int c = quarter + 4 * u;        // pieces interleaved over the quarters: short rows keep all four busy
      asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;"
                   ::"r"(ss_addr(sm.x + c * 2048 + tok * 16)), "l"(ksrc + (8 * c < lk ? 8 * c : 0)), "r"(8 * c < lk ? 16 : 0) : "memory");
      asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;"
                   ::"r"(ss_addr(sm.v + c * 2048 + tok * 16)), "l"(vsrc + (8 * c < lv ? 8 * c : 0)), "r"(8 * c < lv ? 16 : 0) : "memory");
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = __shfl_sync(0xffffffffu, sm.tmem, 0);
    if (warp == 0) {
      // K = X Bk
#pragma unroll
      for (int ks = 0; ks < 8; ++ks)
        ss_mma(tmem + S_TM_K, ss_desc(ss_addr(sm.x) + ks * 4096, 2048, 128), ss_desc(ss_addr(sm.basis) + ks * 4096, 2048, 128), idesc_k, ks > 0);
      ss_commit(&sm.bar[0]);
    }
    __syncwarp();
    ok = ss_wait(&sm.bar[0], phase) && ok;
    __syncwarp();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (tile + CS >= n_tile) load_bv();      // last tile: X has been read
    // ---- [RMSNorm,] RoPE at the token's position, scores of this quarter's 16 pairs ----
    const uint32_t lane_addr = tmem + S_TM_K + ((uint32_t)(32 * (warp & 3)) << 16);
    float acc[SHP] = {0.f, 0.f, 0.f, 0.f}, ssq = 0.f;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int j0 = 16 * quarter + 8 * i;
      float lo[8], hi[8];
      ss_ld_pairs(lo, hi, lane_addr + j0);
      if (KNORM) {
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          ssq = fmaf(lo[e], lo[e], fmaf(hi[e], hi[e], ssq));
          lo[e] *= sm.knw[j0 + e];
          hi[e] *= sm.knw[64 + j0 + e];
        }
      }
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float ang = (float)(int)((uint32_t)s * sm.phi[j0 + e]) * 1.46291807926715968e-9f;      // 2 pi / 2^32
        const float sn = __sinf(ang), cs = __cosf(ang), l = lo[e], h = hi[e];
        lo[e] = l * cs - h * sn;
        hi[e] = h * cs + l * sn;
      }
#pragma unroll
      for (int h = 0; h < SHP; ++h) {
        const float4 q0 = *reinterpret_cast<const float4*>(&sm.q[h][j0]), q1 = *reinterpret_cast<const float4*>(&sm.q[h][j0 + 4]);
        const float4 q2 = *reinterpret_cast<const float4*>(&sm.q[h][64 + j0]), q3 = *reinterpret_cast<const float4*>(&sm.q[h][64 + j0 + 4]);
        float v0 = acc[h], v1 = 0.f;
        v0 = fmaf(q0.x, lo[0], v0); v0 = fmaf(q0.y, lo[1], v0); v0 = fmaf(q0.z, lo[2], v0); v0 = fmaf(q0.w, lo[3], v0);
        v1 = fmaf(q1.x, lo[4], v1); v1 = fmaf(q1.y, lo[5], v1); v1 = fmaf(q1.z, lo[6], v1); v1 = fmaf(q1.w, lo[7], v1);
        v0 = fmaf(q2.x, hi[0], v0); v0 = fmaf(q2.y, hi[1], v0); v0 = fmaf(q2.z, hi[2], v0); v0 = fmaf(q2.w, hi[3], v0);
        v1 = fmaf(q3.x, hi[4], v1); v1 = fmaf(q3.y, hi[5], v1); v1 = fmaf(q3.z, hi[6], v1); v1 = fmaf(q3.w, hi[7], v1);
        acc[h] = v0 + v1;
      }
    }
    if (quarter > 0) *reinterpret_cast<float4*>(sm.part[quarter - 1][tok]) = make_float4(acc[0], acc[1], acc[2], acc[3]);
    if (KNORM) sm.ss[quarter][tok] = ssq;
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    // ---- softmax weights of the tile, one thread per token ----
    float sc[SHP], m_tile[SHP];
    if (quarter == 0) {
      float rs = 1.f;
      if (KNORM) rs = rsqrtf((sm.ss[0][tok] + sm.ss[1][tok] + sm.ss[2][tok] + sm.ss[3][tok]) * (1.0f / SD) + p.k_norm_eps);
#pragma unroll
      for (int h = 0; h < SHP; ++h) {
        const float v = (acc[h] + sm.part[0][tok][h]) + (sm.part[1][tok][h] + sm.part[2][tok][h]);
        sc[h] = lk > 0 ? v * rs : -INFINITY;
        const float m = redux_max(sc[h]);
        if (lane == 0) sm.wmax[warp][h] = m;
      }
    }
    __syncthreads();
    if (quarter == 0) {
      float pr[SHP], rest[SHP];
#pragma unroll
      for (int h = 0; h < SHP; ++h) {
        m_tile[h] = fmaxf(fmaxf(sm.wmax[0][h], sm.wmax[1][h]), fmaxf(sm.wmax[2][h], sm.wmax[3][h]));
        pr[h] = m_tile[h] == -INFINITY ? 0.f : exp2f(sc[h] - m_tile[h]);
        sc[h] = pr[h];
        rest[h] = pr[h] - to_f32(from_f32<T>(pr[h]));
      }
      *reinterpret_cast<uint4*>(sm.p + tok * 16) = make_uint4(ss_pack<T>(pr[0], pr[1]), ss_pack<T>(pr[2], pr[3]), ss_pack<T>(rest[0], rest[1]), ss_pack<T>(rest[2], rest[3]));
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncthreads();
    if (warp == 0) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      // O^T = XV^T P: columns 0..3 values, 4..7 remainders, 8..15 alias them
#pragma unroll
      for (int ks = 0; ks < 8; ++ks)
        ss_mma(tmem + S_TM_O, ss_desc(ss_addr(sm.v) + ks * 256, 128, 2048), ss_desc(ss_addr(sm.p) + ks * 256, 128, 0), idesc_o, ks > 0);
      ss_commit(&sm.bar[1]);
    }
    if (quarter == 0) {        // the weights' sums, behind the product
#pragma unroll
      for (int h = 0; h < SHP; ++h) {
        const float l = warp_sum(sc[h]);
        if (lane == 0) sm.wsum[warp][h] = l;
      }
    }
    __syncwarp();
    ok = ss_wait(&sm.bar[1], phase) && ok;
    __syncwarp();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    float m_f[SHP];
    if (quarter == 0) {
      uint32_t r[8];
      asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\ntcgen05.wait::ld.sync.aligned;"
                   : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                   : "r"(tmem + S_TM_O + ((uint32_t)(32 * warp) << 16)) : "memory");
#pragma unroll
      for (int h = 0; h < SHP; ++h) {
        const float m_new = fmaxf(m_run[h], m_tile[h]);
        const float f0 = m_new == -INFINITY ? 0.f : exp2f(m_run[h] - m_new), f1 = m_new == -INFINITY ? 0.f : exp2f(m_tile[h] - m_new);
        m_f[h] = f1;
        l_run[h] *= f0;
        o_run[h] = o_run[h] * f0 + f1 * (__uint_as_float(r[h]) + __uint_as_float(r[4 + h]));
        m_run[h] = m_new;
      }
    }
    __syncthreads();
    if (quarter == 0) {
#pragma unroll
      for (int h = 0; h < SHP; ++h) l_run[h] += m_f[h] * ((sm.wsum[0][h] + sm.wsum[1][h]) + (sm.wsum[2][h] + sm.wsum[3][h]));
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    // (the next tile's first barrier orders its copies' results; its copies themselves overwrite tiles both products have read)
  }
  if (rank >= n_tile && n_tile > 0) load_bv();      // (a CTA without a tile still projects its heads)
  if (quarter == 0 && n_tile > 0) {
#pragma unroll
    for (int h = 0; h < SHP; ++h) {
      sm.lat[h][tok] = o_run[h];
      if (tid == 0) { sm.ml[0][h] = m_run[h]; sm.ml[1][h] = l_run[h]; }
    }
  }
  if (!ok && tid == 0) set_status(p.status, DKV_ST_TIMEOUT);
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  pdl_launch_dependents();
  if (CS > 1) {
    asm volatile("barrier.cluster.wait.aligned;" ::: "memory");        // of the arrive in the set-up
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
  // ---- heads rank, rank + CS, ...: merge the CTAs' latent sums and project through Bv ----
  if (mine) {
    const int nh = rank < G ? (G - rank + CS - 1) / CS : 0;
    auto out_of = [&](int k) {
      return reinterpret_cast<T*>(p.out) + (size_t)b * p.out_stride_b + (size_t)(g * G + rank + k * CS) * p.out_stride_h;
    };
    if (n_tile == 0) {      // row without tokens: zeros, flagged
      if (quarter < nh) out_of(quarter)[tok] = from_f32<T>(0.f);
      if (tid == 0) set_status(p.status, DKV_ST_EMPTY_ROW);
    } else if (nh > 0) {
      // merged latents of head rank + k CS as values (column k) and remainders (column 4 + k), one more product:
      // out^T = Bv^T lat, M = 128 dims
      if (quarter < SHP) {
        float lat = 0.f;
        if (quarter < nh) {
          const int h = rank + quarter * CS, nc = min(CS, n_tile);
          float M = -INFINITY, L = 0.f, v = 0.f, mc[SCLUSTER], lc[SCLUSTER], vc[SCLUSTER];
#pragma unroll
          for (int c = 0; c < SCLUSTER; ++c) {
            mc[c] = -INFINITY; lc[c] = 0.f; vc[c] = 0.f;
            if (c < nc) { mc[c] = dsmem_f32(&sm.ml[0][h], c); lc[c] = dsmem_f32(&sm.ml[1][h], c); vc[c] = dsmem_f32(&sm.lat[h][tok], c); }
            M = fmaxf(M, mc[c]);
          }
          if (M != -INFINITY)
#pragma unroll
            for (int c = 0; c < SCLUSTER; ++c) {
              const float f = exp2f(mc[c] - M);
              L = fmaf(f, lc[c], L);
              v = fmaf(f, vc[c], v);
            }
          if (L <= 0.f && tok == 0) set_status(p.status, DKV_ST_EMPTY_ROW);
          lat = L > 0.f ? v / L : 0.f;
        }
        const T hi = from_f32<T>(lat);
        reinterpret_cast<T*>(sm.p)[tok * 8 + quarter] = hi;
        reinterpret_cast<T*>(sm.p)[tok * 8 + 4 + quarter] = from_f32<T>(lat - to_f32(hi));
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncthreads();
      if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
        for (int ks = 0; ks < 8; ++ks)
          ss_mma(__shfl_sync(0xffffffffu, sm.tmem, 0) + S_TM_O, ss_desc(ss_addr(sm.x) + ks * 256, 128, 2048), ss_desc(ss_addr(sm.p) + ks * 256, 128, 0), idesc_o, ks > 0);
        ss_commit(&sm.bar[2]);
      }
      __syncwarp();
      const bool ok2 = ss_wait(&sm.bar[2], 0);
      __syncwarp();
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (quarter == 0) {
        uint32_t r[8];
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\ntcgen05.wait::ld.sync.aligned;"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                     : "r"(sm.tmem + S_TM_O + ((uint32_t)(32 * warp) << 16)) : "memory");
#pragma unroll
        for (int k = 0; k < SHP; ++k)
          if (k < nh) out_of(k)[tok] = from_f32<T>(__uint_as_float(r[k]) + __uint_as_float(r[4 + k]));
        if (!ok2 && tid == 0) set_status(p.status, DKV_ST_TIMEOUT);
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 4) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(sm.tmem), "r"(S_TMEM_COLS));
  }
  if (CS > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;\nbarrier.cluster.wait.aligned;" ::: "memory");     // nobody leaves while its sums are read
}

// CTAs per row: one per tile of the longest row that can come (a routed call sees no row at or past route_max_tokens), in
// powers of two
int short_cluster(const dkv_attn_args* a) {
  const int longest = a->route_max_tokens > 0 && a->route_max_tokens <= a->seq_len ? a->route_max_tokens - 1 : a->seq_len;
  const int tiles = (longest + ST - 1) / ST;
  return tiles > 2 ? SCLUSTER : tiles > 1 ? 2 : 1;
}

template <typename T, bool KNORM>
int launch_short(const dkv_attn_args* a) {
  const int cs = short_cluster(a);
  const int smem = (int)sizeof(ShortSmem) + 128;
  auto kern = short_decode_kernel<T, KNORM>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e == cudaSuccess) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(a->batch * cs), a->n_basis_groups);
    cfg.blockDim = dim3(STHREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = reinterpret_cast<cudaStream_t>(a->stream);
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = cs;
    at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = cs > 1 ? 2 : 1;
    e = cudaLaunchKernelEx(&cfg, kern, *a, (float)log((double)a->theta));
  }
  DKV_REQUIRE(e == cudaSuccess, DKV_E_CUDA, "launch of the short decode kernel failed: %s", cudaGetErrorString(e));
  DKV_CHECK_LAUNCH();
  return DKV_OK;
}

}  // namespace

// Whether a fused call takes this kernel: no row has more than one tile, or all of its CTAs have an SM of their own.  A tile
// costs a CTA here several times what it costs the pipeline of dkv_mma_decode.cu, so where CTAs of longer rows queue up the
// pipeline is faster (B = 16, 256 tokens, two CTAs per SM: 16.4 us here, 14.7 there; B = 64, 499 tokens: 172 and 65).
bool short_ok(const dkv_attn_args* a) {
  const int cs = short_cluster(a), n_sm = a->n_sm > 0 ? a->n_sm : sm_count();
  return cs == 1 || (long long)a->batch * a->n_basis_groups * cs <= n_sm;
}

// Whether a routed call leaves its rows to this kernel, also those at or past the switch point.  The policy's switch point
// decides with them: only while no row has more than twice the tiles of the longest row that it calls short (500: 1024 tokens,
// 64: 256) -- a caller with a low switch point asks for the long rows' kernel where this one would still be taken.
bool short_takes_all(const dkv_attn_args* a, int switch_tokens) {
  dkv_attn_args all = *a;
  all.route_min_tokens = all.route_max_tokens = 0;
  const int tiles = (a->seq_len + ST - 1) / ST, short_tiles = (int)(((long long)switch_tokens - 1 + ST - 1) / ST);
  return a->seq_len <= SHORT_ALL_TOKENS && tiles <= 2LL * short_tiles && short_ok(&all);
}

int short_fused(const dkv_attn_args* a) {
  if (a->batch == 0) return DKV_OK;
  if (a->dtype == DKV_BF16) return a->k_norm_weight ? launch_short<__nv_bfloat16, true>(a) : launch_short<__nv_bfloat16, false>(a);
  return a->k_norm_weight ? launch_short<__half, true>(a) : launch_short<__half, false>(a);
}

}  // namespace dkv
