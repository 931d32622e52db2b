// Attention over caches that the packed tensor-core kernel does not take: fp32, the joint latent row shared by all heads
// (rank up to 1024), any integer lengths, strided metadata.  Three kernels instead of one CTA per (row, query head):
//   1. scores, one CTA per (batch row, token tile, heads that share a basis and an arena): the tile's K is reconstructed once
//      for these query heads, rotated and multiplied with each of them; fp32 scores go to the workspace (or, for the score operator,
//      out in the query type);
//   2. latent sum, one CTA per (token slice, block of 128 latent coefficients, arena): the V rows are read once for all
//      heads of the arena; a slice leaves a partial record (m, l, latent accumulator) per head;
//   3. merge of a head's records and projection through Bv.
// 16-bit types reconstruct and accumulate on tcgen05: 128-token tiles, the ragged rows staged K-major in shared memory
// (a piece of 8 coefficients may start at any element, it is put together from two aligned 16-byte loads), the softmax
// weights as two 16-bit terms so that nothing is lost against fp32 weights.  fp32 stays on the FMA units.
// The first version (one CTA per (row, query head, slice), K reconstructed per query head on mma.sync) took 281 us on
// B = 2, S = 2048, R = 1024, 8 groups, bf16, and 13 us for the merge; the three took 25 (scores) + 13 (latent sums) + 7 us (merge),
// the call 48.0; 43.1 since a thread's pieces are asked for together and the V rows before the scores are waited for.
// fp32, B = 1, S = 256, 8 arenas: 131 us in one kernel of 32 CTAs, in three kernels 22.5, 19.1 since queries, basis
// rows and V are asked for ahead.
//
// Math (reference: src/dynakv/kernels/fused.py:28-142, two_stage.py:52-157, 211-281): as in dkv_generic.cu, which keeps
// the single-kernel path for callers without a workspace.
#include <math.h>

#include <numeric>
#include <type_traits>

#include "dkv_common.cuh"

namespace dkv {

namespace {

constexpr int TD = 128;                 // head_dim
constexpr int TS_TOK = 128;             // tokens per tile of the 16-bit kernels
constexpr int TS_THREADS = 256;
constexpr int TS_CHUNK = 64;            // coefficients per pipeline stage of the reconstruction
constexpr int TS_STAGES = 3;
constexpr int TS_STAGE_BYTES = TS_TOK * TS_CHUNK * 2;
constexpr int TS_HB = 8;                // query heads per pass of the score epilogue
constexpr int TF_TOK = 16;              // tokens per tile of the fp32 score kernel
constexpr int TF_SLICE = 32;            // token granularity of fp32 slices
constexpr uint32_t TS_SPIN = 1u << 22;

__device__ __forceinline__ uint32_t ts_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ bool ts_wait(unsigned long long* bar, uint32_t parity) {
  for (uint32_t it = 0; it < TS_SPIN; ++it) {
    uint32_t r;
    asm volatile("{\n.reg .pred q;\nmbarrier.try_wait.parity.shared::cta.b64 q, [%1], %2;\nselp.u32 %0, 1, 0, q;\n}"
                 : "=r"(r) : "r"(ts_smem(bar)), "r"(parity) : "memory");
    if (r) return true;
  }
  return false;
}
// unswizzled operand descriptor
__device__ __forceinline__ uint64_t ts_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((addr >> 4) & 0x3FFF) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(sbo >> 4) << 32) | (1ull << 46);
}
__device__ __forceinline__ void ts_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, bool acc) {
  asm volatile("{\n.reg .pred q;\nsetp.ne.b32 q, %4, 0;\ntcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, q;\n}"
               ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(acc ? 1u : 0u) : "memory");
}
__device__ __forceinline__ void ts_commit(unsigned long long* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(ts_smem(bar)) : "memory");
}
__device__ __forceinline__ void ts_ld8(float (&v)[8], uint32_t addr) {      // (the caller waits)
  uint32_t r[8];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\ntcgen05.wait::ld.sync.aligned;"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(addr) : "memory");
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}

// Elements e0 .. e0+7 of a row of `len` 16-bit elements (zeros past its end), whatever the row's alignment: a piece that
// does not start on a 16-byte boundary is cut out of two aligned blocks.  Only 16-byte blocks that hold an element of the
// row are touched.  Asking for the blocks and cutting the piece are two steps without a branch around the loads: in one
// function the pieces of a thread were read one after the other, a trip to memory each.
struct RawPiece {
  uint4 v0, v1;
  int shift, n;          // elements of v0 before the piece; elements of the piece that exist
};
__device__ __forceinline__ RawPiece ask_piece(const uint16_t* row, int e0, int len) {
  RawPiece r;
  r.n = min(max(len - e0, 0), 8);
  const uintptr_t a = reinterpret_cast<uintptr_t>(row + e0);
  const uint4* base = reinterpret_cast<const uint4*>(a & ~(uintptr_t)15);
  r.shift = (int)(a & 15) >> 1;
  r.v0 = r.v1 = make_uint4(0u, 0u, 0u, 0u);
  if (r.n > 0) r.v0 = __ldg(base);
  if (r.shift + r.n > 8) r.v1 = __ldg(base + 1);       // (only with r.n > 0: shift is at most 7)
  return r;
}
__device__ __forceinline__ uint4 cut_piece(const RawPiece& r) {
  uint32_t w[8] = {r.v0.x, r.v0.y, r.v0.z, r.v0.w, r.v1.x, r.v1.y, r.v1.z, r.v1.w};
  if (r.shift & 4) {
#pragma unroll
    for (int i = 0; i < 6; ++i) w[i] = w[i + 2];
  }
  if (r.shift & 2) {
#pragma unroll
    for (int i = 0; i < 5; ++i) w[i] = w[i + 1];
  }
  const uint32_t sel = (r.shift & 1) ? 0x5432u : 0x3210u;
  uint32_t t[4] = {__byte_perm(w[0], w[1], sel), __byte_perm(w[1], w[2], sel), __byte_perm(w[2], w[3], sel), __byte_perm(w[3], w[4], sel)};
#pragma unroll
  for (int i = 0; i < 4; ++i) t[i] = r.n >= 2 * i + 2 ? t[i] : (r.n == 2 * i + 1 ? t[i] & 0xffffu : 0u);
  return make_uint4(t[0], t[1], t[2], t[3]);
}

__device__ __forceinline__ int row_len(const dkv_attn_args& p, int b) {
  int s = p.seq_len;
  if (p.seq_lens) s = min(s, max(p.seq_lens[b], 0));
  return s;
}
// length and offset of token s of arena row a; a row outside its arena is dropped and flagged
__device__ __forceinline__ void token_meta(const dkv_attn_args& p, const dkv_side& sd, int a, int s, int& len, int& off) {
  len = sd.lens[(size_t)a * sd.lens_stride_a + (size_t)s * sd.lens_stride_s];
  off = sd.offs[(size_t)a * sd.offs_stride_a + (size_t)s * sd.offs_stride_s];
  len = min(max(len, 0), p.rank);
  if (off < 0 || (int64_t)off + len > sd.flat_stride) {
    set_status(p.status, DKV_ST_BAD_LENGTH);
    len = 0;
    off = 0;
  }
}

// Where the scores of (call row i, head h, token s) go.  The score kernels are given units in place of basis groups in
// p.n_basis_groups: consecutive query heads that share a basis and an arena, a basis group or an equal part of one.
struct ScoreSink {
  float* ws;             // fp32 workspace [batch, Hq, pitch], or NULL: out in the query type, masked as the reference does
  int64_t pitch;
  int per_basis;         // units of a basis group
};

// --------------------------------------------------------------- 1. scores, 16-bit types
struct ScoreSmem {
  alignas(128) unsigned char x[TS_STAGES][TS_STAGE_BYTES];       // piece c (8 coefficients) of token t at c*2048 + t*16
  alignas(128) unsigned char b[TS_STAGES][TS_STAGE_BYTES];       // basis rows [64][128]: (r/8)*2048 + (d/8)*128 + (r%8)*16
  alignas(16) float q[TS_HB][TD];
  alignas(16) float part[TS_HB][TS_TOK];
  float ss[2][TS_TOK];
  float knw[TD];
  uint32_t phi[64];
  int len[TS_TOK], off[TS_TOK];
  alignas(8) unsigned long long done[TS_STAGES];
  uint32_t tmem;
  int rmax;
};

// Bound by latency and staging: a CTA's products are 1 us of tensor pipe (R = 1024), its two operands 26 KB per 64
// coefficients.  Stages of 64 coefficients, three in flight: the next piece of X is on its way into registers and the next
// basis rows by cp.async while the current stage is multiplied.  The epilogue is fp32 (as before): two threads per token,
// each half of the rotation pairs, angles from integer phases (position * turns per token mod 1, exact in 32 bits).
template <typename T>
__global__ void __launch_bounds__(TS_THREADS) tile_scores_kernel(dkv_attn_args p, ScoreSink sink, float log_theta) {
  extern __shared__ unsigned char ts_raw[];
  ScoreSmem& sm = *reinterpret_cast<ScoreSmem*>(ts_raw + ((128u - (ts_smem(ts_raw) & 127u)) & 127u));
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int n_tile = (p.seq_len + TS_TOK - 1) / TS_TOK, i_row = blockIdx.x / n_tile, g = blockIdx.y, t0 = (blockIdx.x - i_row * n_tile) * TS_TOK;
  const int b = p.batch_index ? p.batch_index[i_row] : i_row;
  const int A = p.arenas_per_batch, Hq = p.n_q_heads, R = p.rank, G = Hq / p.n_basis_groups;
  if (sink.ws && row_routed_out(p, b)) return;
  const int t_end = sink.ws ? row_len(p, b) : p.seq_len;     // the operator writes every column
  if (t0 >= t_end) return;
  const int a = b * A + (g * G * A) / Hq;
  pdl_launch_dependents();      // the latent-sum kernel may set itself up meanwhile
  if (tid == 0) {
    sm.rmax = 0;
    for (int s = 0; s < TS_STAGES; ++s) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(ts_smem(&sm.done[s])));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(ts_smem(&sm.tmem)), "r"(128));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid < 64) {
    const float f = expf(-((float)(2 * tid) / (float)TD) * log_theta);
    sm.phi[tid] = (uint32_t)(long long)llrint((double)f * 683565275.57643158978229477811035);   // 2^32 / (2 pi)
  }
  if (p.k_norm_weight && tid >= 128) sm.knw[tid - 128] = p.k_norm_weight[tid - 128];
  __syncthreads();
  if (tid < TS_TOK) {
    int len = 0, off = 0;
    if (t0 + tid < t_end) token_meta(p, p.k, a, t0 + tid, len, off);
    sm.len[tid] = len;
    sm.off[tid] = off;
    const int mx = __reduce_max_sync(0xffffffffu, len);
    if (lane == 0) atomicMax(&sm.rmax, mx);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = sm.tmem;
  const int rmax = sm.rmax, n_chunk = (rmax + TS_CHUNK - 1) / TS_CHUNK;
  const T* flat = reinterpret_cast<const T*>(p.k.flat) + (size_t)a * p.k.flat_stride;
  const T* kup = reinterpret_cast<const T*>(p.k_up) + (size_t)(g / sink.per_basis) * R * TD;
  const bool b_vec = (reinterpret_cast<uintptr_t>(p.k_up) & 15) == 0;
  // X pieces of this thread: tokens (tid & 7) + 8 * (tid >> 5) + 64 u', pieces ((tid >> 3) & 3) + 4 u: eight lanes with
  // consecutive tokens write 128 consecutive bytes, four lanes read 64 consecutive bytes of a row
  const int x_t = (tid & 7) + 8 * warp, x_c = (tid >> 3) & 3;
  RawPiece xr[4];
  auto load_x = [&](int c) {
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int t = x_t + 64 * (u & 1), e = c * TS_CHUNK + 8 * (x_c + 4 * (u >> 1));
      xr[u] = ask_piece(reinterpret_cast<const uint16_t*>(flat) + sm.off[t], e, sm.len[t]);
    }
  };
  auto copy_b = [&](int c) {
    const int buf = c % TS_STAGES;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int e = tid + u * TS_THREADS, rr = e >> 4, d = e & 15, r = c * TS_CHUNK + rr;
      unsigned char* dst = sm.b[buf] + (rr >> 3) * 2048 + d * 128 + (rr & 7) * 16;
      if (b_vec) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(ts_smem(dst)), "l"(kup + (size_t)min(r, R - 1) * TD + 8 * d), "r"(r < R ? 16 : 0) : "memory");
      } else {
        __align__(16) T v[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] = r < R ? kup[(size_t)r * TD + 8 * d + k] : from_f32<T>(0.f);
        *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(v);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  const uint32_t fmt = std::is_same<T, __nv_bfloat16>::value ? 1u : 0u;
  const uint32_t idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | (1u << 16) | ((128u >> 3) << 17) | ((128u >> 4) << 24);
  bool ok = true;
  if (n_chunk > 0) {
    load_x(0);
    copy_b(0);
  }
  for (int c = 0; c < n_chunk; ++c) {
    const int buf = c % TS_STAGES;
    // (the products of stage c - 3, the last user of this buffer, were waited for in the round before)
#pragma unroll
    for (int u = 0; u < 4; ++u)
      *reinterpret_cast<uint4*>(sm.x[buf] + (x_c + 4 * (u >> 1)) * 2048 + (x_t + 64 * (u & 1)) * 16) = cut_piece(xr[u]);
    if (c + 1 < n_chunk) {
      if (c >= 2) ok = ts_wait(&sm.done[(c + 1) % TS_STAGES], (uint32_t)(((c - 2) / TS_STAGES) & 1)) && ok;
      load_x(c + 1);
      copy_b(c + 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    if (tid == 0) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const int ksteps = (min(TS_CHUNK, rmax - c * TS_CHUNK) + 15) >> 4;
      for (int ks = 0; ks < ksteps; ++ks)
        ts_mma(tmem, ts_desc(ts_smem(sm.x[buf]) + ks * 4096, 2048, 128), ts_desc(ts_smem(sm.b[buf]) + ks * 4096, 2048, 128), idesc, c + ks > 0);
      ts_commit(&sm.done[buf]);
    }
  }
  if (n_chunk > 0) ok = ts_wait(&sm.done[(n_chunk - 1) % TS_STAGES], (uint32_t)(((n_chunk - 1) / TS_STAGES) & 1)) && ok;
  ok = __syncthreads_and(ok) != 0;
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (!ok && tid == 0) set_status(p.status, DKV_ST_TIMEOUT);

  // ---- [RMSNorm,] RoPE, scores: thread = (token, half of the pairs) ----
  const int tok = tid & 127, half = tid >> 7, s = t0 + tok;
  const uint32_t lane_addr = tmem + ((uint32_t)(32 * (warp & 3)) << 16);
  const bool has_k = ok && n_chunk > 0;
  float rs = 1.f;
  if (p.k_norm_weight) {
    float ss = 0.f;
    if (has_k) {
#pragma unroll 1
      for (int i = 0; i < 8; ++i) {
        float v[8];
        ts_ld8(v, lane_addr + 64 * half + 8 * i);
#pragma unroll
        for (int e = 0; e < 8; ++e) ss = fmaf(v[e], v[e], ss);
      }
    }
    sm.ss[half][tok] = ss;
    __syncthreads();
    rs = rsqrtf((sm.ss[0][tok] + sm.ss[1][tok]) * (1.0f / TD) + p.k_norm_eps);
  }
  const float scale = rsqrtf((float)TD);
  for (int h0 = 0; h0 < G; h0 += TS_HB) {
    const int nh = min(TS_HB, G - h0);
    __syncthreads();
    for (int e = tid; e < nh * TD; e += TS_THREADS) {
      const T* qp = reinterpret_cast<const T*>(p.q) + (size_t)b * p.q_stride_b + (size_t)(g * G + h0 + (e >> 7)) * p.q_stride_h;
      sm.q[e >> 7][e & 127] = to_f32(qp[e & 127]);
    }
    __syncthreads();
    float acc[TS_HB];
#pragma unroll
    for (int h = 0; h < TS_HB; ++h) acc[h] = 0.f;
    if (has_k) {
#pragma unroll 1
      for (int i = 0; i < 4; ++i) {
        const int j0 = 32 * half + 8 * i;
        float lo[8], hi[8];
        ts_ld8(lo, lane_addr + j0);
        ts_ld8(hi, lane_addr + 64 + j0);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const float ang = (float)(int)((uint32_t)s * sm.phi[j0 + e]) * 1.46291807926715968e-9f;   // 2 pi / 2^32
          const float sn = __sinf(ang), cs = __cosf(ang);
          float l = lo[e], h = hi[e];
          if (p.k_norm_weight) {
            l = sm.knw[j0 + e] * (l * rs);
            h = sm.knw[64 + j0 + e] * (h * rs);
          }
          lo[e] = l * cs - h * sn;
          hi[e] = h * cs + l * sn;
        }
#pragma unroll
        for (int h = 0; h < TS_HB; ++h) {
          if (h < nh) {
            const float4 q0 = *reinterpret_cast<const float4*>(&sm.q[h][j0]), q1 = *reinterpret_cast<const float4*>(&sm.q[h][j0 + 4]);
            const float4 q2 = *reinterpret_cast<const float4*>(&sm.q[h][64 + j0]), q3 = *reinterpret_cast<const float4*>(&sm.q[h][64 + j0 + 4]);
            float v = acc[h];
            v = fmaf(q0.x, lo[0], v); v = fmaf(q0.y, lo[1], v); v = fmaf(q0.z, lo[2], v); v = fmaf(q0.w, lo[3], v);
            v = fmaf(q1.x, lo[4], v); v = fmaf(q1.y, lo[5], v); v = fmaf(q1.z, lo[6], v); v = fmaf(q1.w, lo[7], v);
            v = fmaf(q2.x, hi[0], v); v = fmaf(q2.y, hi[1], v); v = fmaf(q2.z, hi[2], v); v = fmaf(q2.w, hi[3], v);
            v = fmaf(q3.x, hi[4], v); v = fmaf(q3.y, hi[5], v); v = fmaf(q3.z, hi[6], v); v = fmaf(q3.w, hi[7], v);
            acc[h] = v;
          }
        }
      }
    }
    if (half == 1) {
#pragma unroll
      for (int h = 0; h < TS_HB; ++h) sm.part[h][tok] = acc[h];
    }
    __syncthreads();
    if (half == 0 && s < t_end) {
#pragma unroll
      for (int h = 0; h < TS_HB; ++h) {
        if (h < nh) {
          const float v = acc[h] + sm.part[h][tok];
          const int head = g * G + h0 + h;
          if (sink.ws) {
            sink.ws[((size_t)i_row * Hq + head) * sink.pitch + s] = sm.len[tok] > 0 ? v * scale : -INFINITY;
          } else {
            T* op = reinterpret_cast<T*>(p.out) + (size_t)b * p.out_stride_b + (size_t)head * p.out_stride_h;
            op[s] = from_f32<T>((sm.len[tok] > 0 ? v : -1.0e4f) * scale);
          }
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(128));
  }
}

}  // namespace

namespace {

// --------------------------------------------------------------- 2. latent sums of a slice
// Scores of a slice: fp32 workspace, or the operator's input in the query type (every token up to the row's length counts).
template <typename T>
struct ScoreSource {
  const float* ws;       // [batch, Hq, pitch]
  int64_t pitch;
  const T* in;           // [batch rows, Hq, S]
  int64_t sb, sh;
  __device__ __forceinline__ float get(int i_row, int b, int Hq, int head, int s) const {
    return ws ? ws[((size_t)i_row * Hq + head) * pitch + s] : to_f32(in[(size_t)b * sb + (size_t)head * sh + s]);
  }
};

// Maximum of each head's scores over tokens [t0, t1), one warp per head in turn; m_s[h] for heads head0 .. head0 + nh - 1.
template <typename T>
__device__ __forceinline__ void slice_maxima(const ScoreSource<T>& src, int i_row, int b, int Hq, int head0, int nh, int t0, int t1, float* m_s) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int h = warp; h < nh; h += TS_THREADS / 32) {
    float m = -INFINITY;
    for (int s = t0 + lane; s < t1; s += 32) m = fmaxf(m, src.get(i_row, b, Hq, head0 + h, s));
    m = warp_max(m);
    if (lane == 0) m_s[h] = m;
  }
}

template <int NH>
struct PvSmem {
  alignas(128) unsigned char v[2][TS_TOK * 256];        // piece c (8 latents) of token t at c*2048 + t*16
  alignas(128) unsigned char pt[2][TS_TOK * 4 * NH];    // weights: column n of token t at (n/8)*2048 + t*16 + (n%8)*2; columns NH.. are the remainders
  float m[NH], l[NH];
  int len[2][TS_TOK], off[2][TS_TOK];
  alignas(8) unsigned long long done[2];
  uint32_t tmem;
  int rmax[2];
};

// grid (batch x arenas x slices, latent blocks of 128 x head blocks).  Per 128-token tile: the V rows' pieces of this latent
// block staged as in the score kernel, weights exp(s - m) of NH heads as value + remainder, one chain of 8 k-steps
// M = 128 latents, N = 2 NH; two tiles in flight.
template <typename T, int NH>
__global__ void __launch_bounds__(TS_THREADS) tile_pv_kernel(dkv_attn_args p, ScoreSource<T> src, float* rec, int slice, int n_split, int r_blocks) {
  extern __shared__ unsigned char ts_raw[];
  PvSmem<NH>& sm = *reinterpret_cast<PvSmem<NH>*>(ts_raw + ((128u - (ts_smem(ts_raw) & 127u)) & 127u));
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int A = p.arenas_per_batch, Hq = p.n_q_heads, R = p.rank, HA = Hq / A;
  const int row_arena = blockIdx.x / n_split, sl = blockIdx.x - row_arena * n_split, i_row = row_arena / A, j = row_arena - i_row * A;
  const int rb = blockIdx.y % r_blocks, head0 = j * HA + (blockIdx.y / r_blocks) * NH, nh = min(NH, (j + 1) * HA - head0);
  // Behind the score kernel, which started when everything before it had ended, the rows' indices and lengths may be read
  // at once; the operator follows whatever the caller ran last -- an append, say, that moves seq_lens on.
  if (src.ws == nullptr) pdl_wait();
  const int b = p.batch_index ? p.batch_index[i_row] : i_row;
  if (row_routed_out(p, b)) return;
  pdl_launch_dependents();
  const int S = row_len(p, b), t0 = sl * slice, t1 = min(S, t0 + slice);
  float* my_rec = rec + (((size_t)i_row * Hq + head0) * n_split + sl) * (size_t)(2 + R);     // + h * n_split * (2 + R)
  const size_t rec_h = (size_t)n_split * (2 + R);
  if (t0 >= t1) {
    pdl_wait();
    if (rb == 0 && tid < nh) { my_rec[tid * rec_h] = -INFINITY; my_rec[tid * rec_h + 1] = 0.f; }
    return;
  }
  const int a = b * A + j;
  if (tid == 0) {
    for (int s = 0; s < 2; ++s) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(ts_smem(&sm.done[s])));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  constexpr int COLS = 2 * NH < 32 ? 32 : 2 * NH;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(ts_smem(&sm.tmem)), "r"(COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid < NH) sm.l[tid] = 0.f;
  for (int e = tid; e < 2 * TS_TOK * NH; e += TS_THREADS) reinterpret_cast<uint32_t*>(sm.pt)[e] = 0u;     // columns of heads that are not there
  const T* flat = reinterpret_cast<const T*>(p.v.flat) + (size_t)a * p.v.flat_stride;
  const uint32_t fmt = std::is_same<T, __nv_bfloat16>::value ? 1u : 0u;
  // D fp32, A = V^T (MN-major: bit 15), B = P (MN-major: bit 16), M = 128, N = 2 NH
  const uint32_t idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | (1u << 15) | (1u << 16) | ((uint32_t)((2 * NH) >> 3) << 17) | ((128u >> 4) << 24);
  const int x_t = (tid & 7) + 8 * warp, x_c = (tid >> 3) & 3;
  bool ok = true;
  int n_done = 0;
  for (int tt = t0; tt < t1; tt += TS_TOK) {
    const int buf = n_done & 1;
    if (n_done >= 2) ok = ts_wait(&sm.done[buf], (uint32_t)(((n_done - 2) >> 1) & 1)) && ok;
    const int par = ((tt - t0) / TS_TOK) & 1;      // (not buf, which an unused tile leaves to the next one, whose reset could overtake a reader)
    if (tid == 0) sm.rmax[par] = 0;
    __syncthreads();
    if (tid < TS_TOK) {
      int len = 0, off = 0;
      if (tt + tid < t1) token_meta(p, p.v, a, tt + tid, len, off);
      sm.len[buf][tid] = len;
      sm.off[buf][tid] = off;
      const int mx = __reduce_max_sync(0xffffffffu, len);
      if (lane == 0) atomicMax(&sm.rmax[par], mx);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    // The V rows are asked for before the weights are formed, the first tile's before the scores are waited for.
    const bool use = sm.rmax[par] > 128 * rb;
    RawPiece v[8];
    if (use) {
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int t = x_t + 64 * (u & 1);
        v[u] = ask_piece(reinterpret_cast<const uint16_t*>(flat) + sm.off[buf][t], 128 * rb + 8 * (x_c + 4 * (u >> 1)), sm.len[buf][t]);
      }
    }
    if (tt == t0) {
      pdl_wait();        // the scores (and, in a chain of layers, the workspace) are the kernel's before this one
      slice_maxima(src, i_row, b, Hq, head0, nh, t0, t1, sm.m);
      __syncthreads();
    }
    // weights: a warp takes a head at a time, four tokens per lane
    for (int h = warp; h < nh; h += TS_THREADS / 32) {
      const float m = sm.m[h];
      float l = 0.f;
#pragma unroll
      for (int u = 0; u < TS_TOK / 32; ++u) {
        const int t = lane + 32 * u, s = tt + t;
        const float sc = s < t1 ? src.get(i_row, b, Hq, head0 + h, s) : -INFINITY;
        const float pv = sc == -INFINITY ? 0.f : __expf(sc - m);
        l += pv;
        const T hi = from_f32<T>(pv);
        unsigned char* dst = sm.pt[buf] + (h >> 3) * 2048 + t * 16 + (h & 7) * 2;
        *reinterpret_cast<T*>(dst) = hi;
        *reinterpret_cast<T*>(dst + (NH >> 3) * 2048) = from_f32<T>(pv - to_f32(hi));
      }
      l = warp_sum(l);
      if (lane == 0) sm.l[h] += l;
    }
    if (use) {
#pragma unroll
      for (int u = 0; u < 8; ++u)
        *reinterpret_cast<uint4*>(sm.v[buf] + (x_c + 4 * (u >> 1)) * 2048 + (x_t + 64 * (u & 1)) * 16) = cut_piece(v[u]);
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncthreads();
      if (tid == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
        for (int ks = 0; ks < 8; ++ks)
          ts_mma(sm.tmem, ts_desc(ts_smem(sm.v[buf]) + ks * 256, 128, 2048), ts_desc(ts_smem(sm.pt[buf]) + ks * 256, 128, 2048), idesc, n_done > 0 || ks > 0);
        ts_commit(&sm.done[buf]);
      }
      ++n_done;
    }
  }
  if (n_done > 0) ok = ts_wait(&sm.done[(n_done - 1) & 1], (uint32_t)(((n_done - 1) >> 1) & 1)) && ok;
  ok = __syncthreads_and(ok) != 0;
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (!ok && tid == 0) set_status(p.status, DKV_ST_TIMEOUT);
  if (rb == 0 && tid < nh) { my_rec[tid * rec_h] = sm.m[tid]; my_rec[tid * rec_h + 1] = sm.l[tid]; }
  // thread = (latent, half of the heads)
  const uint32_t tmem = sm.tmem;
  const int r = 128 * rb + (tid & 127), half = tid >> 7;
  const uint32_t lane_addr = tmem + ((uint32_t)(32 * (warp & 3)) << 16);
#pragma unroll
  for (int h0 = 0; h0 < NH / 2; h0 += 8) {
    float v[8], w[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] = w[e] = 0.f;
    if (ok && n_done > 0) {
      ts_ld8(v, lane_addr + half * (NH / 2) + h0);
      ts_ld8(w, lane_addr + NH + half * (NH / 2) + h0);
    }
    if (r < R) {
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const int h = half * (NH / 2) + h0 + e;
        if (h < nh) my_rec[h * rec_h + 2 + r] = v[e] + w[e];
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(COLS));
  }
}

// --------------------------------------------------------------- fp32: the same two steps on the FMA units
// 16 tokens per CTA: thread = (dim, 8 tokens), coefficients staged transposed so that a load serves four tokens; the
// rotation's (cos, sin) once per CTA for all heads of the unit, exact sincosf as in the single-kernel path.
__global__ void __launch_bounds__(TS_THREADS) tile_scores_f32_kernel(dkv_attn_args p, ScoreSink sink, float log_theta) {
  __shared__ __align__(16) float x_s[TS_CHUNK][TF_TOK];
  __shared__ float k_s[TF_TOK][TD + 4];
  __shared__ float cs_s[TF_TOK][64], sn_s[TF_TOK][64];
  __shared__ float q_s[TS_HB][TD];
  __shared__ int len_s[TF_TOK], off_s[TF_TOK];
  __shared__ int rmax_s;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int n_tile = (p.seq_len + TF_TOK - 1) / TF_TOK, i_row = blockIdx.x / n_tile, g = blockIdx.y, t0 = (blockIdx.x - i_row * n_tile) * TF_TOK;
  const int b = p.batch_index ? p.batch_index[i_row] : i_row;
  const int A = p.arenas_per_batch, Hq = p.n_q_heads, R = p.rank, G = Hq / p.n_basis_groups;
  if (sink.ws && row_routed_out(p, b)) return;
  const int t_end = sink.ws ? row_len(p, b) : p.seq_len;
  if (t0 >= t_end) return;
  const int a = b * A + (g * G * A) / Hq;
  pdl_launch_dependents();
  // the queries of up to TS_HB heads are on their way from the start (asked for head by head they were a trip to memory each)
  auto ask_queries = [&](int h0) {
    const int n = min(TS_HB, G - h0) * TD;
    for (int e = tid; e < n; e += TS_THREADS) {
      const float* qp = reinterpret_cast<const float*>(p.q) + (size_t)b * p.q_stride_b + (size_t)(g * G + h0 + (e >> 7)) * p.q_stride_h + (e & 127);
      asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(ts_smem(&q_s[e >> 7][e & 127])), "l"(qp) : "memory");
    }
  };
  ask_queries(0);
  if (warp == 0) {
    int len = 0, off = 0;
    if (lane < TF_TOK) {
      if (t0 + lane < t_end) token_meta(p, p.k, a, t0 + lane, len, off);
      len_s[lane] = len;
      off_s[lane] = off;
    }
    const int mx = __reduce_max_sync(0xffffffffu, len);
    if (lane == 0) rmax_s = mx;
  }
  const int d = tid & 127, th = tid >> 7;
  const float* kup = reinterpret_cast<const float*>(p.k_up) + (size_t)(g / sink.per_basis) * R * TD;
  float w[16];           // the first basis rows too, before it is known how many are needed
#pragma unroll
  for (int u = 0; u < 16; ++u) w[u] = u < R ? __ldg(kup + (size_t)u * TD + d) : 0.f;
  for (int e = tid; e < TF_TOK * 64; e += TS_THREADS) {
    const int t = e >> 6, j = e & 63;
    sincosf((float)(t0 + t) * expf(-((float)(2 * j) / (float)TD) * log_theta), &sn_s[t][j], &cs_s[t][j]);
  }
  __syncthreads();
  const float* flat = reinterpret_cast<const float*>(p.k.flat) + (size_t)a * p.k.flat_stride;
  const int rmax = rmax_s;
  float acc[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) acc[i] = 0.f;
  for (int r0 = 0; r0 < rmax; r0 += TS_CHUNK) {
    const int nr = min(TS_CHUNK, rmax - r0);
    for (int e = tid; e < TS_CHUNK * TF_TOK; e += TS_THREADS) {
      const int t = e >> 6, r = e & 63;
      x_s[r][t] = r0 + r < len_s[t] ? flat[(size_t)off_s[t] + r0 + r] : 0.f;
    }
    __syncthreads();
#pragma unroll 1
    for (int rr = 0; rr < nr; rr += 16) {
      if (r0 + rr > 0) {
#pragma unroll
        for (int u = 0; u < 16; ++u) w[u] = r0 + rr + u < rmax ? __ldg(kup + (size_t)(r0 + rr + u) * TD + d) : 0.f;
      } else if (rmax < 16) {      // rows that no token of the tile reaches take no part, whatever they hold (here, where they have arrived)
#pragma unroll
        for (int u = 0; u < 16; ++u) w[u] = u < rmax ? w[u] : 0.f;
      }
#pragma unroll
      for (int u = 0; u < 16; ++u) {
        const float4 x0 = *reinterpret_cast<const float4*>(&x_s[rr + u][8 * th]), x1 = *reinterpret_cast<const float4*>(&x_s[rr + u][8 * th + 4]);
        acc[0] = fmaf(x0.x, w[u], acc[0]); acc[1] = fmaf(x0.y, w[u], acc[1]); acc[2] = fmaf(x0.z, w[u], acc[2]); acc[3] = fmaf(x0.w, w[u], acc[3]);
        acc[4] = fmaf(x1.x, w[u], acc[4]); acc[5] = fmaf(x1.y, w[u], acc[5]); acc[6] = fmaf(x1.z, w[u], acc[6]); acc[7] = fmaf(x1.w, w[u], acc[7]);
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) k_s[8 * th + i][d] = acc[i];
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  const float scale = rsqrtf((float)TD);
  // a warp rotates its two tokens in place, then multiplies them with every head
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int t = warp + 8 * u;
    float k0a = k_s[t][lane], k0b = k_s[t][lane + 32], k1a = k_s[t][lane + 64], k1b = k_s[t][lane + 96];
    if (p.k_norm_weight) {
      const float ss = warp_sum(k0a * k0a + k0b * k0b + k1a * k1a + k1b * k1b);
      const float rs = rsqrtf(ss * (1.0f / TD) + p.k_norm_eps);
      k0a = p.k_norm_weight[lane] * (k0a * rs);
      k0b = p.k_norm_weight[lane + 32] * (k0b * rs);
      k1a = p.k_norm_weight[lane + 64] * (k1a * rs);
      k1b = p.k_norm_weight[lane + 96] * (k1b * rs);
    }
    const float ca = cs_s[t][lane], sa = sn_s[t][lane], cb = cs_s[t][lane + 32], sb = sn_s[t][lane + 32];
    k_s[t][lane] = k0a * ca - k1a * sa;
    k_s[t][lane + 64] = k1a * ca + k0a * sa;
    k_s[t][lane + 32] = k0b * cb - k1b * sb;
    k_s[t][lane + 96] = k1b * cb + k0b * sb;
  }
  for (int h = 0; h < G; ++h) {
    const int head = g * G + h, hs = h % TS_HB;
    if (h > 0 && hs == 0) {
      __syncthreads();
      ask_queries(h);
      asm volatile("cp.async.wait_all;" ::: "memory");
      __syncthreads();
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int t = warp + 8 * u, s = t0 + t;
      float part = q_s[hs][lane] * k_s[t][lane] + q_s[hs][lane + 64] * k_s[t][lane + 64] + q_s[hs][lane + 32] * k_s[t][lane + 32] + q_s[hs][lane + 96] * k_s[t][lane + 96];
      part = warp_sum(part);
      if (lane == 0 && s < t_end) {
        if (sink.ws) sink.ws[((size_t)i_row * Hq + head) * sink.pitch + s] = len_s[t] > 0 ? part * scale : -INFINITY;
        else (reinterpret_cast<float*>(p.out) + (size_t)b * p.out_stride_b + (size_t)head * p.out_stride_h)[s] = (len_s[t] > 0 ? part : -1.0e4f) * scale;
      }
    }
  }
}

// thread = (latent of the block, every second token); NH heads accumulate per V element read
template <int NH>
__global__ void __launch_bounds__(TS_THREADS) tile_pv_f32_kernel(dkv_attn_args p, ScoreSource<float> src, float* rec, int slice, int n_split, int r_blocks) {
  __shared__ __align__(16) float p_s[TF_SLICE][NH];
  __shared__ float m_s[NH], l_s[NH], red[NH][128];
  __shared__ int len_s[TF_SLICE], off_s[TF_SLICE];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int A = p.arenas_per_batch, Hq = p.n_q_heads, R = p.rank, HA = Hq / A;
  const int row_arena = blockIdx.x / n_split, sl = blockIdx.x - row_arena * n_split, i_row = row_arena / A, j = row_arena - i_row * A;
  const int rb = blockIdx.y % r_blocks, head0 = j * HA + (blockIdx.y / r_blocks) * NH, nh = min(NH, (j + 1) * HA - head0);
  // Behind the score kernel, which started when everything before it had ended, the rows' indices and lengths may be read
  // at once; the operator follows whatever the caller ran last -- an append, say, that moves seq_lens on.
  if (src.ws == nullptr) pdl_wait();
  const int b = p.batch_index ? p.batch_index[i_row] : i_row;
  if (row_routed_out(p, b)) return;
  pdl_launch_dependents();
  const int S = row_len(p, b), t0 = sl * slice, t1 = min(S, t0 + slice);
  float* my_rec = rec + (((size_t)i_row * Hq + head0) * n_split + sl) * (size_t)(2 + R);
  const size_t rec_h = (size_t)n_split * (2 + R);
  if (t0 >= t1) {
    pdl_wait();
    if (rb == 0 && tid < nh) { my_rec[tid * rec_h] = -INFINITY; my_rec[tid * rec_h + 1] = 0.f; }
    return;
  }
  const int a = b * A + j;
  if (tid < NH) l_s[tid] = 0.f;
  const float* flat = reinterpret_cast<const float*>(p.v.flat) + (size_t)a * p.v.flat_stride;
  const int r = 128 * rb + (tid & 127), half = tid >> 7;
  float acc[NH];
#pragma unroll
  for (int h = 0; h < NH; ++h) acc[h] = 0.f;
  for (int tt = t0; tt < t1; tt += TF_SLICE) {
    __syncthreads();
    if (warp == 0) {
      int len = 0, off = 0;
      if (tt + lane < t1) token_meta(p, p.v, a, tt + lane, len, off);
      len_s[lane] = len;
      off_s[lane] = off;
    }
    __syncthreads();
    // V is asked for before the weights are formed, the first tile's before the scores are waited for
    float v[TF_SLICE / 2];
#pragma unroll
    for (int k = 0; k < TF_SLICE / 2; ++k) {
      const int t = half + 2 * k;
      v[k] = 0.f;
      if (r < len_s[t]) v[k] = __ldg(flat + (size_t)off_s[t] + r);
    }
    if (tt == t0) {
      pdl_wait();
      slice_maxima(src, i_row, b, Hq, head0, nh, t0, t1, m_s);
      __syncthreads();
    }
    for (int h = warp; h < NH; h += TS_THREADS / 32) {
      float pv = 0.f;
      if (h < nh && tt + lane < t1) {
        const float sc = src.get(i_row, b, Hq, head0 + h, tt + lane);
        pv = sc == -INFINITY ? 0.f : __expf(sc - m_s[h]);
      }
      p_s[lane][h] = pv;
      const float l = warp_sum(pv);
      if (lane == 0) l_s[h] += l;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < TF_SLICE / 2; ++k) {
#pragma unroll
      for (int h = 0; h < NH; h += 4) {
        const float4 w = *reinterpret_cast<const float4*>(&p_s[half + 2 * k][h]);
        acc[h] = fmaf(w.x, v[k], acc[h]);
        acc[h + 1] = fmaf(w.y, v[k], acc[h + 1]);
        acc[h + 2] = fmaf(w.z, v[k], acc[h + 2]);
        acc[h + 3] = fmaf(w.w, v[k], acc[h + 3]);
      }
    }
  }
  if (half == 1) {
#pragma unroll
    for (int h = 0; h < NH; ++h) red[h][tid & 127] = acc[h];
  }
  __syncthreads();
  if (rb == 0 && tid < nh) { my_rec[tid * rec_h] = m_s[tid]; my_rec[tid * rec_h + 1] = l_s[tid]; }
  if (half == 0 && r < R) {
#pragma unroll
    for (int h = 0; h < NH; ++h)
      if (h < nh) my_rec[h * rec_h + 2 + r] = acc[h] + red[h][tid];
  }
}

// --------------------------------------------------------------- 3. merge and projection
// grid (batch, Hq, RS), clusters of RS CTAs: each merges R / RS latent coefficients of the head's records and projects
// them; the CTAs' partial outputs meet in the first one's shared memory.  RS = 4 for long latents, where one CTA would read
// 256 KB of Bv alone (13 us; 8 us split).
template <typename T, bool OPERATOR>
__global__ void __launch_bounds__(TS_THREADS) tile_combine_kernel(dkv_attn_args p, const float* rec, int n_split) {
  __shared__ float lat_s[1024];
  __shared__ float w_s[64];
  __shared__ float red_s[16][TD];
  __shared__ float part_s[4][TD];
  __shared__ float L_s;
  const int tid = threadIdx.x, h = blockIdx.y, Hq = p.n_q_heads, R = p.rank, RS = gridDim.z, rs = blockIdx.z;
  const int b = p.batch_index ? p.batch_index[blockIdx.x] : blockIdx.x;
  if (row_routed_out(p, b)) return;      // (uniform over the cluster)
  if (RS > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");     // the others' shared memory is there once they have started
  const int g = h / (Hq / p.n_basis_groups);
  pdl_wait();
  const float* rec0 = rec + (((size_t)blockIdx.x * Hq + h) * n_split) * (size_t)(2 + R);
  if (tid < 32) {      // maxima and sums of up to 64 records, asked for at once
    float m[2], l[2], M, L = 0.f;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int k = tid + 32 * u;
      m[u] = k < n_split ? rec0[(size_t)k * (2 + R)] : -INFINITY;
      l[u] = k < n_split ? rec0[(size_t)k * (2 + R) + 1] : 0.f;
    }
    M = warp_max(fmaxf(m[0], m[1]));
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      // (a slice whose scores are all NaN leaves the maximum of no score and a sum that is NaN, which its weight takes on)
      const float w = l[u] != l[u] ? l[u] : m[u] == -INFINITY ? 0.f : __expf(m[u] - M);
      w_s[tid + 32 * u] = w;
      L = fmaf(w, l[u], L);
    }
    L = warp_sum(L);
    if (tid == 0) L_s = L;
  }
  __syncthreads();
  const float L = L_s;
  if (!OPERATOR && L <= 0.f && tid == 0 && rs == 0) set_status(p.status, DKV_ST_EMPTY_ROW);
  const float inv = OPERATOR ? 1.f / fmaxf(L, 1e-6f) : (L > 0.f ? 1.f / L : 0.f);
  const int rn = (R + RS - 1) / RS, r_lo = rs * rn, r_hi = min(R, r_lo + rn);
  for (int r = r_lo + tid; r < r_hi; r += TS_THREADS) {
    float v = 0.f;
    for (int k0 = 0; k0 < n_split; k0 += 8) {
      float x[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) x[k] = (k0 + k < n_split && w_s[k0 + k] != 0.f) ? rec0[(size_t)(k0 + k) * (2 + R) + 2 + r] : 0.f;
#pragma unroll
      for (int k = 0; k < 8; ++k)
        if (k0 + k < n_split) v = fmaf(w_s[k0 + k], x[k], v);
    }
    lat_s[r - r_lo] = v * inv;
  }
  __syncthreads();
  // projection: thread (rg, dg) takes rows rg, rg + 16, ... and the 8 output dims 8 dg .. 8 dg + 7
  const T* vup = reinterpret_cast<const T*>(p.v_up) + (size_t)g * R * TD;
  const int dg = tid & 15, rg = tid >> 4;
  const bool vec = (reinterpret_cast<uintptr_t>(p.v_up) & 15) == 0;
  float acc8[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) acc8[e] = 0.f;
#pragma unroll 8
  for (int r = r_lo + rg; r < r_hi; r += 16) {
    const float lr = lat_s[r - r_lo];
    __align__(16) T v[8];
    if (vec) {
#pragma unroll
      for (int k = 0; k < (int)sizeof(T) / 2; ++k)
        reinterpret_cast<uint4*>(v)[k] = __ldg(reinterpret_cast<const uint4*>(vup + (size_t)r * TD + 8 * dg) + k);
    } else {
#pragma unroll
      for (int e = 0; e < 8; ++e) v[e] = vup[(size_t)r * TD + 8 * dg + e];
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) acc8[e] = fmaf(lr, to_f32(v[e]), acc8[e]);
  }
#pragma unroll
  for (int e = 0; e < 8; ++e) red_s[rg][8 * dg + e] = acc8[e];
  __syncthreads();
  float o = 0.f;
  if (tid < TD) {
#pragma unroll
    for (int k = 0; k < 16; ++k) o += red_s[k][tid];
  }
  if (RS > 1) {
    asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
    if (tid < TD) {
      uint32_t dst;      // this CTA's row of the first CTA's part_s
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(dst) : "r"(ts_smem(&part_s[rs][tid])), "r"(0));
      asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(dst), "f"(o) : "memory");
    }
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (rs != 0) return;
    if (tid < TD) o = (part_s[0][tid] + part_s[1][tid]) + (part_s[2][tid] + part_s[3][tid]);
  }
  if (tid < TD) {
    T* op = reinterpret_cast<T*>(p.out) + (size_t)b * p.out_stride_b + (size_t)h * p.out_stride_h;
    op[tid] = from_f32<T>(o);
  }
}

// --------------------------------------------------------------- host side
int slice_tokens(const dkv_attn_args* a) {      // at most 64 slices of whole tiles
  const int unit = a->dtype == DKV_F32 ? TF_SLICE : TS_TOK;
  const int t = (a->seq_len + 63) / 64;
  return t <= unit ? unit : (t + unit - 1) / unit * unit;
}
int n_slices(const dkv_attn_args* a) {
  const int t = slice_tokens(a), n = (a->seq_len + t - 1) / t;
  return n < 1 ? 1 : n;
}
int64_t score_pitch(const dkv_attn_args* a) { return ((int64_t)a->seq_len + 3) / 4 * 4; }
size_t score_bytes(const dkv_attn_args* a) { return ((size_t)a->batch * a->n_q_heads * score_pitch(a) * sizeof(float) + 255) / 256 * 256; }
size_t record_bytes(const dkv_attn_args* a) { return (size_t)a->batch * a->n_q_heads * n_slices(a) * (size_t)(2 + a->rank) * sizeof(float); }

template <typename K>
int opt_in(K kern, int bytes) {
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  DKV_REQUIRE(e == cudaSuccess, DKV_E_CUDA, "shared memory of a tile kernel: %s", cudaGetErrorString(e));
  return DKV_OK;
}

int launch_scores(const dkv_attn_args* a, float* ws) {
  if (a->batch == 0 || a->seq_len == 0) return DKV_OK;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(a->stream);
  const float log_theta = (float)log((double)a->theta);
  const int heads = std::gcd(a->n_q_heads / a->n_basis_groups, a->n_q_heads / a->arenas_per_batch);
  dkv_attn_args u = *a;
  u.n_basis_groups = a->n_q_heads / heads;
  const ScoreSink sink{ws, score_pitch(a), u.n_basis_groups / a->n_basis_groups};
  const int tok = a->dtype == DKV_F32 ? TF_TOK : TS_TOK;
  const long long ctas = (long long)a->batch * ((a->seq_len + tok - 1) / tok);
  DKV_REQUIRE(ctas <= 2147483647LL, DKV_E_LIMIT, "too many tokens");
  const dim3 grid((unsigned)ctas, u.n_basis_groups);      // (n_q_heads <= 65535)
  const int smem = (int)sizeof(ScoreSmem) + 128;
  if (a->dtype == DKV_F32) {
    tile_scores_f32_kernel<<<grid, TS_THREADS, 0, st>>>(u, sink, log_theta);
  } else if (a->dtype == DKV_F16) {
    if (int rc = opt_in(tile_scores_kernel<__half>, smem)) return rc;
    tile_scores_kernel<__half><<<grid, TS_THREADS, smem, st>>>(u, sink, log_theta);
  } else {
    if (int rc = opt_in(tile_scores_kernel<__nv_bfloat16>, smem)) return rc;
    tile_scores_kernel<__nv_bfloat16><<<grid, TS_THREADS, smem, st>>>(u, sink, log_theta);
  }
  DKV_CHECK_LAUNCH();
  return DKV_OK;
}

template <typename T, int NH>
int launch_pv(const dkv_attn_args* a, const ScoreSource<T>& src, float* rec) {
  cudaStream_t st = reinterpret_cast<cudaStream_t>(a->stream);
  const int r_blocks = (a->rank + 127) / 128, heads = a->n_q_heads / a->arenas_per_batch, n_split = n_slices(a);
  const long long ctas = (long long)a->batch * a->arenas_per_batch * n_split;
  DKV_REQUIRE(ctas <= 2147483647LL && (long long)r_blocks * ((heads + NH - 1) / NH) <= 65535, DKV_E_LIMIT, "too many rows or heads");
  const dim3 grid((unsigned)ctas, r_blocks * ((heads + NH - 1) / NH));
  if constexpr (std::is_same<T, float>::value) {
    launch_pdl(tile_pv_f32_kernel<NH>, grid, dim3(TS_THREADS), 0, st, *a, src, rec, slice_tokens(a), n_split, r_blocks);
  } else {
    const int smem = (int)sizeof(PvSmem<NH>) + 128;
    if (int rc = opt_in(tile_pv_kernel<T, NH>, smem)) return rc;
    launch_pdl(tile_pv_kernel<T, NH>, grid, dim3(TS_THREADS), smem, st, *a, src, rec, slice_tokens(a), n_split, r_blocks);
  }
  DKV_CHECK_LAUNCH();
  return DKV_OK;
}

template <typename T, bool OPERATOR>
int launch_merge(const dkv_attn_args* a, const float* rec) {
  const int rs = a->rank >= 512 ? 4 : 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(a->batch, a->n_q_heads, rs);
  cfg.blockDim = dim3(TS_THREADS);
  cfg.stream = reinterpret_cast<cudaStream_t>(a->stream);
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = at[1].val.clusterDim.y = 1;
  at[1].val.clusterDim.z = rs;
  cfg.attrs = at;
  cfg.numAttrs = rs > 1 ? 2 : 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, tile_combine_kernel<T, OPERATOR>, *a, rec, n_slices(a));
  DKV_REQUIRE(e == cudaSuccess, DKV_E_CUDA, "launch of the merge kernel failed: %s", cudaGetErrorString(e));
  DKV_CHECK_LAUNCH();
  return DKV_OK;
}

template <typename T, bool OPERATOR>
int sum_and_merge(const dkv_attn_args* a, const ScoreSource<T>& src, float* rec) {
  // heads of an arena that share the V rows: 8 (fp32) or 16 per CTA, 32 for the joint row
  const int heads = a->n_q_heads / a->arenas_per_batch;
  constexpr int SMALL = std::is_same<T, float>::value ? 8 : 16;
  if (int rc = heads <= SMALL ? launch_pv<T, SMALL>(a, src, rec) : launch_pv<T, 32>(a, src, rec)) return rc;
  return launch_merge<T, OPERATOR>(a, rec);
}

template <typename T>
int attention(const dkv_attn_args* a) {
  float* scores = reinterpret_cast<float*>(a->workspace);
  float* rec = reinterpret_cast<float*>(reinterpret_cast<unsigned char*>(a->workspace) + score_bytes(a));
  if (int rc = launch_scores(a, scores)) return rc;
  return sum_and_merge<T, false>(a, ScoreSource<T>{scores, score_pitch(a), nullptr, 0, 0}, rec);
}

template <typename T>
int softmax_v(const dkv_attn_args* a, const void* scores, int64_t sb, int64_t sh) {
  return sum_and_merge<T, true>(a, ScoreSource<T>{nullptr, 0, reinterpret_cast<const T*>(scores), sb, sh}, reinterpret_cast<float*>(a->workspace));
}

}  // namespace

// the workspace of the attention (scores and records)
size_t tiles_workspace_bytes(const dkv_attn_args* a) {
  if (a->batch <= 0 || a->seq_len <= 0) return 0;
  return score_bytes(a) + record_bytes(a);
}
// Whether a call takes the tile kernels.  Small calls do not, where a chain of kernels costs more than the one-kernel path of
// dkv_generic.cu: a few tokens, and CTAs enough for every (row, head) at once.
static bool one_kernel_call(const dkv_attn_args* a, int tokens) {
  return a->seq_len <= tokens && (long long)a->batch * a->n_q_heads <= 4LL * sm_count();
}
// The attention, with its workspace: up to a tile of 32 tokens (measured, bf16: 8.7-13 us against 18-22 at up to 32 tokens,
// 19-20 against 18-23 at 48; B * Hq = 1024: 42-51 against 28), for fp32 at a rank up to 256 (1024: 57 against 41).
bool tiles_ok(const dkv_attn_args* a) {
  if (one_kernel_call(a, 32) && (a->dtype != DKV_F32 || a->rank <= 256)) return false;
  return a->batch > 0 && a->seq_len > 0 && a->workspace != nullptr && ((uintptr_t)a->workspace & 15) == 0 &&
         a->workspace_bytes >= record_bytes(a) + score_bytes(a);
}
// The scores alone, 32 heads: 16-bit types up to 32 tokens (rank 256: 6.2 us against 8.6, 48 tokens 9.7 against 8.4; rank 1024:
// 14.6 against 16.2, 48 tokens 25 against 17).  fp32 never (16 tokens, rank 256: 20.5 against 11).
bool tiles_scores_ok(const dkv_attn_args* a) { return a->dtype == DKV_F32 || !one_kernel_call(a, 32); }
// The softmax over given scores, 32 heads: 16-bit types up to 32 tokens (rank 256: 9 us against 13, 48 tokens 12.3-13.1 against
// 14; rank 1024: 15-16 against 14-17), fp32 up to 64 (rank 256: 9.4 against 13.5, 128 tokens 14.5 against 13.6; rank 1024: 16
// against 14-23).
static bool softmax_in_one_kernel(const dkv_attn_args* a) { return one_kernel_call(a, a->dtype == DKV_F32 ? 64 : 32); }
size_t tiles_softmax_workspace_bytes(const dkv_attn_args* a) {
  return a->batch <= 0 || a->seq_len <= 0 || softmax_in_one_kernel(a) ? 0 : record_bytes(a);
}
bool tiles_softmax_ok(const dkv_attn_args* a) {
  return !softmax_in_one_kernel(a) && a->batch > 0 && a->seq_len > 0 && a->workspace != nullptr && ((uintptr_t)a->workspace & 15) == 0 &&
         a->workspace_bytes >= record_bytes(a);
}
int tiles_scores(const dkv_attn_args* a) { return launch_scores(a, nullptr); }
int tiles_attention(const dkv_attn_args* a) {
  if (a->dtype == DKV_F32) return attention<float>(a);
  return a->dtype == DKV_F16 ? attention<__half>(a) : attention<__nv_bfloat16>(a);
}
int tiles_softmax_v(const dkv_attn_args* a, const void* scores, int64_t sb, int64_t sh) {
  if (a->dtype == DKV_F32) return softmax_v<float>(a, scores, sb, sh);
  return a->dtype == DKV_F16 ? softmax_v<__half>(a, scores, sb, sh) : softmax_v<__nv_bfloat16>(a, scores, sb, sh);
}

}  // namespace dkv
