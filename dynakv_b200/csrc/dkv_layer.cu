// The row operators between the GEMMs of a Llama-shaped decode step (dynakv_b200/runner.py).  As chains of elementwise
// torch kernels they were 45 launches and ~140 us per layer at 32 rows of 4096, more than the weight GEMMs; each chain is
// one kernel here with the same roundings at the same places.  All of them are bound by latency (a few hundred KB): the two
// norms 13 us each, split 5, silu 2.8, maximum of 128256 columns 18.5 (torch: 42); the step of 4 layers 1.33 -> 0.82 ms.
#include <math.h>

#include "dkv_common.cuh"

namespace dkv {

namespace {

constexpr int LN_THREADS = 512, LN_MAX_DIM = 49152;  // the row in fp32 in shared memory

// h += y (when given; rounded to the storage type), x = round(h * rsqrt(mean(h^2) + eps)) * weight (rounded), and with a
// cutoff head the kept lengths 8 clamp(ceil(16 sigmoid(x . w_o + bias)), 1, 16) of the row, fp32 dot products: outputs
// 0 .. n_cut/2 - 1 go to len_k, the rest to len_v.  One CTA per row; a warp takes one output of the cutoff head at a time.
template <typename T>
__global__ void __launch_bounds__(LN_THREADS) norm_rows_kernel(T* h, const T* y, const T* weight, float eps, T* x, int dim, const float* w_cut,
                                                               int n_cut, float bias, int32_t* len_k, int32_t* len_v) {
  extern __shared__ float xs[];
  __shared__ float red[LN_THREADS / 32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const size_t base = (size_t)blockIdx.x * dim;
  float ss = 0.f;
  for (int i = tid; i < dim; i += LN_THREADS) {
    float v = to_f32(h[base + i]);
    if (y) {
      const T r = from_f32<T>(v + to_f32(y[base + i]));
      h[base + i] = r;
      v = to_f32(r);
    }
    xs[i] = v;
    ss = fmaf(v, v, ss);
  }
  ss = warp_sum(ss);
  if (lane == 0) red[warp] = ss;
  __syncthreads();
  float tot = 0.f;
#pragma unroll
  for (int w = 0; w < LN_THREADS / 32; ++w) tot += red[w];
  const float rs = rsqrtf(tot / (float)dim + eps);
  for (int i = tid; i < dim; i += LN_THREADS) {
    const T r = from_f32<T>(to_f32(from_f32<T>(xs[i] * rs)) * to_f32(weight[i]));
    x[base + i] = r;
    xs[i] = to_f32(r);
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

// One CTA per row of a merged projection [q heads | k heads | v heads] x 128: q rotated by the row's position (rotate-half
// RoPE in fp32), k and v copied out; 64 threads a head.
template <typename T>
__global__ void __launch_bounds__(256) split_qkv_kernel(const T* qkv, int64_t stride, int n_q, int n_kv, const int32_t* pos, float log_theta, T* q, T* k, T* v) {
  const int row = blockIdx.x, j = threadIdx.x & 63, n = n_q + 2 * n_kv;
  const T* src = qkv + (size_t)row * stride;
  const float ang = (float)pos[row] * expf(-((float)(2 * j) / 128.f) * log_theta);
  float sn, cs;
  sincosf(ang, &sn, &cs);
  for (int h = threadIdx.x >> 6; h < n; h += 4) {
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

// index of the row's maximum (the first of equals), one CTA per row
template <typename T>
__global__ void __launch_bounds__(1024) argmax_rows_kernel(const T* x, int64_t stride, int n, int64_t* out) {
  __shared__ float mv[32];
  __shared__ int mi[32];
  const T* row = x + (size_t)blockIdx.x * stride;
  float best = -INFINITY;
  int at = n;
  auto take = [&](float v, int i) {
    if (v > best || (v != v && best == best) || ((v == best || (v != v && best != best)) && i < at)) { best = v; at = i; }  // a NaN is above all
  };
  constexpr int E = 16 / (int)sizeof(T);
  const bool vec = (reinterpret_cast<uintptr_t>(row) & 15) == 0;
  const int nv = vec ? n / E : 0;
#pragma unroll 4
  for (int p = threadIdx.x; p < nv; p += 1024) {
    const uint4 w = __ldg(reinterpret_cast<const uint4*>(row) + p);
    const T* t = reinterpret_cast<const T*>(&w);
#pragma unroll
    for (int e = 0; e < E; ++e) take(to_f32(t[e]), p * E + e);
  }
  for (int i = nv * E + threadIdx.x; i < n; i += 1024) take(to_f32(row[i]), i);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) take(__shfl_xor_sync(0xffffffffu, best, o), __shfl_xor_sync(0xffffffffu, at, o));
  if ((threadIdx.x & 31) == 0) { mv[threadIdx.x >> 5] = best; mi[threadIdx.x >> 5] = at; }
  __syncthreads();
  if (threadIdx.x < 32) {
    best = mv[threadIdx.x];
    at = mi[threadIdx.x];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) take(__shfl_xor_sync(0xffffffffu, best, o), __shfl_xor_sync(0xffffffffu, at, o));
    if (threadIdx.x == 0) out[blockIdx.x] = at < n ? at : 0;
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
  BY_TYPE(a->dtype, if (smem > 32 * 1024) cudaFuncSetAttribute(norm_rows_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
                    (norm_rows_kernel<T><<<a->n_rows, LN_THREADS, smem, st>>>(
                        (T*)a->h, (const T*)a->y, (const T*)a->weight, a->eps, (T*)a->x, a->dim, a->w_cut, a->n_cut, a->cut_bias, a->len_k, a->len_v)));
  DKV_CHECK_LAUNCH();
  return DKV_OK;
}

extern "C" int dkv_split_qkv(int32_t dtype, int32_t n_rows, int32_t n_q_heads, int32_t n_kv_heads, const void* qkv, int64_t stride, const int32_t* positions,
                             float theta, void* q, void* k, void* v, void* stream) {
  DKV_REQUIRE(qkv && positions && q && k && v, DKV_E_ARG, "dkv_split_qkv: null argument");
  DKV_REQUIRE(dtype >= DKV_F32 && dtype <= DKV_BF16 && n_rows >= 0 && n_q_heads >= 1 && n_kv_heads >= 1 && stride >= (n_q_heads + 2 * n_kv_heads) * 128,
              DKV_E_ARG, "dkv_split_qkv: bad type or sizes");
  if (n_rows == 0) return DKV_OK;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  BY_TYPE(dtype, (split_qkv_kernel<T><<<n_rows, 256, 0, st>>>((const T*)qkv, stride, n_q_heads, n_kv_heads, positions, (float)log((double)theta), (T*)q, (T*)k, (T*)v)));
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
  BY_TYPE(dtype, (argmax_rows_kernel<T><<<n_rows, 1024, 0, st>>>((const T*)x, stride, n, out)));
  DKV_CHECK_LAUNCH();
  return DKV_OK;
}
