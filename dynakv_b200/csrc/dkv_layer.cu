// The row operators between the GEMMs of a Llama-shaped decode step (dynakv_b200/runner.py).  As chains of elementwise
// torch kernels they were 45 launches and ~140 us per layer at 32 rows of 4096, more than the weight GEMMs; each chain is
// one kernel here with the same roundings at the same places.  All of them are bound by latency (a few hundred KB).  32 rows
// of 4096: a norm 4.9 us (12.7 with a row read 512 elements at a time), split 2.1 (5.2 with one CTA per row), silu 2.7,
// maximum of 128256 columns 11.6 (18.5 with one CTA per row, torch 42); the step of 4 layers 1.38 -> 0.73 ms.
#include <math.h>

#include "dkv_common.cuh"

namespace dkv {

namespace {

constexpr int LN_THREADS = 512, LN_MAX_DIM = 49152;  // the row in fp32 in shared memory

// h += y (when given; rounded to the storage type), x = round(h * rsqrt(mean(h^2) + eps)) * weight (rounded), and with a
// cutoff head the kept lengths 8 clamp(ceil(16 sigmoid(x . w_o + bias)), 1, 16) of the row, fp32 dot products: outputs
// 0 .. n_cut/2 - 1 go to len_k, the rest to len_v.  One CTA per row; a warp takes one output of the cutoff head at a time.
// Rows in 16-byte pieces (VEC), two of them per thread asked for at once with the weights and the first rows of the cutoff
// head, so that a row costs one trip to memory and not one per 512 elements.
template <typename T, bool VEC>
__global__ void __launch_bounds__(LN_THREADS) norm_rows_kernel(T* h, const T* y, const T* weight, float eps, T* x, int dim, const float* w_cut,
                                                               int n_cut, float bias, int32_t* len_k, int32_t* len_v) {
  extern __shared__ __align__(16) float xs[];
  __shared__ float red[LN_THREADS / 32];
  constexpr int E = VEC ? 16 / (int)sizeof(T) : 1, U = VEC ? 2 : 8;
  struct alignas(E * sizeof(T)) Piece { T v[E]; };
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, n = dim / E;
  const size_t base = (size_t)blockIdx.x * dim;
  Piece *hp = reinterpret_cast<Piece*>(h + base), *xp = reinterpret_cast<Piece*>(x + base);
  const Piece *yp = reinterpret_cast<const Piece*>(y + base), *wp = reinterpret_cast<const Piece*>(weight);
  Piece wt[U];
#pragma unroll
  for (int u = 0; u < U; ++u)
    if (tid + u * LN_THREADS < n) wt[u] = wp[tid + u * LN_THREADS];
  if (VEC && n_cut > 0)
    for (int o = warp; o < n_cut; o += LN_THREADS / 32)
      for (int i = 32 * lane; i < dim; i += 1024) asm volatile("prefetch.global.L2 [%0];" ::"l"(w_cut + (size_t)o * dim + i));
  float ss = 0.f;
  for (int i0 = tid; i0 < n; i0 += U * LN_THREADS) {
    Piece a[U], b[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = i0 + u * LN_THREADS;
      if (i < n) {
        a[u] = hp[i];
        if (y) b[u] = yp[i];
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = i0 + u * LN_THREADS;
      if (i < n) {
#pragma unroll
        for (int e = 0; e < E; ++e) {
          if (y) a[u].v[e] = from_f32<T>(to_f32(a[u].v[e]) + to_f32(b[u].v[e]));
          const float v = to_f32(a[u].v[e]);
          xs[i * E + e] = v;
          ss = fmaf(v, v, ss);
        }
        if (y) hp[i] = a[u];
      }
    }
  }
  ss = warp_sum(ss);
  if (lane == 0) red[warp] = ss;
  __syncthreads();
  float tot = 0.f;
#pragma unroll
  for (int w = 0; w < LN_THREADS / 32; ++w) tot += red[w];
  const float rs = rsqrtf(tot / (float)dim + eps);
  for (int i0 = tid; i0 < n; i0 += U * LN_THREADS) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = i0 + u * LN_THREADS;
      if (i < n) {
        const Piece w = i0 == tid ? wt[u] : wp[i];
        Piece r;
#pragma unroll
        for (int e = 0; e < E; ++e) {
          r.v[e] = from_f32<T>(to_f32(from_f32<T>(xs[i * E + e] * rs)) * to_f32(w.v[e]));
          xs[i * E + e] = to_f32(r.v[e]);
        }
        xp[i] = r;
      }
    }
  }
  if (n_cut == 0) return;
  __syncthreads();
  const bool vec = (dim & 3) == 0 && (reinterpret_cast<uintptr_t>(w_cut) & 15) == 0;
  for (int o = warp; o < n_cut; o += LN_THREADS / 32) {
    const float* w = w_cut + (size_t)o * dim;
    float s = 0.f;
    if (vec) {
#pragma unroll 8
      for (int i = 4 * lane; i < dim; i += 128) {
        const float4 v = __ldg(reinterpret_cast<const float4*>(w + i)), u = *reinterpret_cast<const float4*>(xs + i);
        s = fmaf(v.x, u.x, s); s = fmaf(v.y, u.y, s); s = fmaf(v.z, u.z, s); s = fmaf(v.w, u.w, s);
      }
    } else {
      for (int i = lane; i < dim; i += 32) s = fmaf(w[i], xs[i], s);
    }
    s = warp_sum(s) + bias;
    if (lane == 0) {
      const float score = 1.f / (1.f + expf(-s));
      const int r = 8 * (int)fminf(fmaxf(ceilf(16.f * score), 1.f), 16.f);
      const int half = n_cut / 2;
      if (o < half) len_k[(size_t)blockIdx.x * half + o] = r;
      else len_v[(size_t)blockIdx.x * half + o - half] = r;
    }
  }
}

// Row and four heads a CTA of a merged projection [q heads | k heads | v heads] x 128: q rotated by the row's position (rotate-half
// RoPE in fp32), k and v copied out; 64 threads a head.
template <typename T>
__global__ void __launch_bounds__(256) split_qkv_kernel(const T* qkv, int64_t stride, int n_q, int n_kv, const int32_t* pos, float log_theta, T* q, T* k, T* v) {
  const int row = blockIdx.x, j = threadIdx.x & 63, n = n_q + 2 * n_kv;
  const T* src = qkv + (size_t)row * stride;
  const float ang = (float)pos[row] * expf(-((float)(2 * j) / 128.f) * log_theta);
  float sn, cs;
  sincosf(ang, &sn, &cs);
  const int h = blockIdx.y * 4 + (threadIdx.x >> 6);
  if (h < n) {
    const T lo = src[h * 128 + j], hi = src[h * 128 + 64 + j];
    if (h < n_q) {
      T* o = q + ((size_t)row * n_q + h) * 128;
      const float l = to_f32(lo), u = to_f32(hi);
      o[j] = from_f32<T>(__fsub_rn(__fmul_rn(l, cs), __fmul_rn(u, sn)));        // products and sums rounded one by one, as torch does
      o[64 + j] = from_f32<T>(__fadd_rn(__fmul_rn(u, cs), __fmul_rn(l, sn)));
    } else {
      const int kv = h - n_q;
      T* o = kv < n_kv ? k + ((size_t)row * n_kv + kv) * 128 : v + ((size_t)row * n_kv + kv - n_kv) * 128;
      o[j] = lo;
      o[64 + j] = hi;
    }
  }
}

// out = round(silu(g)) * u (rounded) of a merged projection [g | u]
template <typename T>
__global__ void __launch_bounds__(256) silu_mul_kernel(const T* gu, int m, T* out) {
  const T* g = gu + (size_t)blockIdx.y * 2 * m;
  for (int i = (blockIdx.x * 256 + threadIdx.x) * 2; i < m; i += gridDim.x * 512) {
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      if (i + e < m) {
        const float x = to_f32(g[i + e]);
        const T s = from_f32<T>(x / (1.f + expf(-x)));
        out[(size_t)blockIdx.y * m + i + e] = from_f32<T>(to_f32(s) * to_f32(g[m + i + e]));
      }
    }
  }
}

// Index of the row's maximum (the first of equals; a NaN is above all numbers).  A cluster of up to eight CTAs per row, each
// takes a range of it; the CTAs' winners meet in the first CTA's memory.
constexpr int AM_THREADS = 512, AM_CLUSTER = 8;
template <typename T>
__global__ void __launch_bounds__(AM_THREADS) argmax_rows_kernel(const T* x, int64_t stride, int n, int64_t* out, int parts) {
  __shared__ float mv[AM_THREADS / 32], cv[AM_CLUSTER];
  __shared__ int mi[AM_THREADS / 32], ci[AM_CLUSTER];
  const int r = blockIdx.x / parts, part = blockIdx.x - r * parts;
  const T* row = x + (size_t)r * stride;
  asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");     // the first CTA's shared memory is there once it has started
  float best = -INFINITY;
  int at = n;
  auto take = [&](float v, int i) {
    if (v > best || (v != v && best == best) || ((v == best || (v != v && best != best)) && i < at)) { best = v; at = i; }
  };
  constexpr int E = 16 / (int)sizeof(T);
  const bool vec = (reinterpret_cast<uintptr_t>(row) & 15) == 0;
  const int nv = vec ? n / E : 0, per = (nv + parts - 1) / parts;
#pragma unroll 4
  for (int p = part * per + threadIdx.x; p < min(nv, (part + 1) * per); p += AM_THREADS) {
    const uint4 w = __ldg(reinterpret_cast<const uint4*>(row) + p);
    const T* t = reinterpret_cast<const T*>(&w);
#pragma unroll
    for (int e = 0; e < E; ++e) take(to_f32(t[e]), p * E + e);
  }
  for (int i = nv * E + part * AM_THREADS + threadIdx.x; i < n; i += parts * AM_THREADS) take(to_f32(row[i]), i);
  auto over_lanes = [&]() {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float v = __shfl_xor_sync(0xffffffffu, best, o);
      const int i = __shfl_xor_sync(0xffffffffu, at, o);
      take(v, i);
    }
  };
  over_lanes();
  if ((threadIdx.x & 31) == 0) { mv[threadIdx.x >> 5] = best; mi[threadIdx.x >> 5] = at; }
  __syncthreads();
  asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
  if (threadIdx.x < 32) {
    best = -INFINITY;
    at = n;
    if (threadIdx.x < AM_THREADS / 32) { best = mv[threadIdx.x]; at = mi[threadIdx.x]; }
    over_lanes();
    if (threadIdx.x == 0) {
      uint32_t v, i;
      asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(v) : "r"((uint32_t)__cvta_generic_to_shared(&cv[part])));
      asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(i) : "r"((uint32_t)__cvta_generic_to_shared(&ci[part])));
      asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(v), "f"(best) : "memory");
      asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(i), "r"(at) : "memory");
    }
  }
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  if (part == 0 && threadIdx.x == 0) {
    best = -INFINITY;
    at = n;
    for (int c = 0; c < parts; ++c) take(cv[c], ci[c]);
    out[r] = at < n ? at : 0;
  }
}

}  // namespace

}  // namespace dkv

using namespace dkv;

#define BY_TYPE(dtype, CALL)                         \
  do {                                               \
    if ((dtype) == DKV_F32) { using T = float; CALL; }           \
    else if ((dtype) == DKV_F16) { using T = __half; CALL; }     \
    else { using T = __nv_bfloat16; CALL; }          \
  } while (0)

extern "C" int dkv_norm_rows(const dkv_norm_args* a) {
  DKV_REQUIRE(a != nullptr && a->h && a->weight && a->x, DKV_E_ARG, "dkv_norm_rows: null argument");
  DKV_REQUIRE(a->dtype >= DKV_F32 && a->dtype <= DKV_BF16 && a->n_rows >= 0 && a->dim >= 1 && a->dim <= LN_MAX_DIM, DKV_E_ARG,
              "dkv_norm_rows: bad type or sizes (at most %d columns)", LN_MAX_DIM);
  DKV_REQUIRE(a->n_cut >= 0 && a->n_cut % 2 == 0 && (a->n_cut == 0 || (a->w_cut && a->len_k && a->len_v)), DKV_E_ARG, "dkv_norm_rows: bad cutoff head");
  if (a->n_rows == 0) return DKV_OK;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(a->stream);
  const int smem = a->dim * (int)sizeof(float);
  const uintptr_t at = (uintptr_t)a->h | (uintptr_t)a->y | (uintptr_t)a->weight | (uintptr_t)a->x;
  const bool vec = (at & 15) == 0 && a->dim % 8 == 0;     // 16-byte pieces, also from one row to the next
#define NORM(V)                                                                                                            \
  do {                                                                                                                     \
    if (smem > 32 * 1024) cudaFuncSetAttribute(norm_rows_kernel<T, V>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem); \
    norm_rows_kernel<T, V><<<a->n_rows, LN_THREADS, smem, st>>>((T*)a->h, (const T*)a->y, (const T*)a->weight, a->eps, (T*)a->x, a->dim, \
                                                                a->w_cut, a->n_cut, a->cut_bias, a->len_k, a->len_v);      \
  } while (0)
  BY_TYPE(a->dtype, if (vec) NORM(true); else NORM(false));
#undef NORM
  DKV_CHECK_LAUNCH();
  return DKV_OK;
}

extern "C" int dkv_split_qkv(int32_t dtype, int32_t n_rows, int32_t n_q_heads, int32_t n_kv_heads, const void* qkv, int64_t stride, const int32_t* positions,
                             float theta, void* q, void* k, void* v, void* stream) {
  DKV_REQUIRE(qkv && positions && q && k && v, DKV_E_ARG, "dkv_split_qkv: null argument");
  DKV_REQUIRE(dtype >= DKV_F32 && dtype <= DKV_BF16 && n_rows >= 0 && n_q_heads >= 1 && n_kv_heads >= 1 && n_q_heads <= 65536 && n_kv_heads <= 65536 && stride >= (n_q_heads + 2 * n_kv_heads) * 128,
              DKV_E_ARG, "dkv_split_qkv: bad type or sizes");
  if (n_rows == 0) return DKV_OK;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  BY_TYPE(dtype, (split_qkv_kernel<T><<<dim3(n_rows, (n_q_heads + 2 * n_kv_heads + 3) / 4), 256, 0, st>>>((const T*)qkv, stride, n_q_heads, n_kv_heads, positions, (float)log((double)theta), (T*)q, (T*)k, (T*)v)));
  DKV_CHECK_LAUNCH();
  return DKV_OK;
}

extern "C" int dkv_silu_mul(int32_t dtype, int32_t n_rows, int32_t m, const void* gu, void* out, void* stream) {
  DKV_REQUIRE(gu && out && dtype >= DKV_F32 && dtype <= DKV_BF16 && n_rows >= 0 && n_rows <= 65535 && m >= 1, DKV_E_ARG, "dkv_silu_mul: bad argument");
  if (n_rows == 0) return DKV_OK;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  BY_TYPE(dtype, (silu_mul_kernel<T><<<dim3((m + 511) / 512, n_rows), 256, 0, st>>>((const T*)gu, m, (T*)out)));
  DKV_CHECK_LAUNCH();
  return DKV_OK;
}

extern "C" int dkv_argmax_rows(int32_t dtype, int32_t n_rows, int32_t n, const void* x, int64_t stride, int64_t* out, void* stream) {
  DKV_REQUIRE(x && out && dtype >= DKV_F32 && dtype <= DKV_BF16 && n_rows >= 0 && n >= 1 && stride >= n, DKV_E_ARG, "dkv_argmax_rows: bad argument");
  if (n_rows == 0) return DKV_OK;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  // a CTA per 8192 columns or so, as many as a portable cluster has
  int parts = 1;
  while (parts < AM_CLUSTER && parts * 8192 < n) parts *= 2;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(n_rows * parts));
  cfg.blockDim = dim3(AM_THREADS);
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = parts;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  BY_TYPE(dtype, cudaLaunchKernelEx(&cfg, argmax_rows_kernel<T>, (const T*)x, stride, n, out, parts));
  DKV_CHECK_LAUNCH();
  return DKV_OK;
}
