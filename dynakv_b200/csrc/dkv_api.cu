// C-ABI entry points of the decode-attention paths and library-wide helpers.
#include <stdarg.h>
#include <string.h>

#include "dkv_common.cuh"

namespace dkv {

static thread_local char g_err[512] = "";

void set_error(const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof(g_err), fmt, ap);
  va_end(ap);
}

int sm_count() {
  static int cached[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
  if (cached[dev] == 0) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
    cached[dev] = n;
  }
  return cached[dev];
}

// implemented in dkv_generic.cu / dkv_tiles.cu / dkv_mma_decode.cu
int check_attn_args(const dkv_attn_args* a, const char* who, bool need_q, bool need_k, bool need_v);
int generic_attention(const dkv_attn_args* a);
size_t tiles_workspace_bytes(const dkv_attn_args* a);
bool mma_path_ok(const dkv_attn_args* a);
size_t mma_split_workspace_bytes(const dkv_attn_args* a);
int mma_fused(const dkv_attn_args* a);
bool short_ok(const dkv_attn_args* a);
bool short_takes_all(const dkv_attn_args* a, int switch_tokens);
int short_fused(const dkv_attn_args* a);
int mma_split(const dkv_attn_args* a);
int mma_combine(const dkv_attn_args* a);
int mma_two_stage_noalloc(const dkv_attn_args* a);

}  // namespace dkv

using namespace dkv;

extern "C" int dkv_version(void) { return DKV_VERSION; }

extern "C" const char* dkv_last_error(void) { return g_err; }

namespace dkv {
// Whether the fused entry is better off as split + merge.  One-kernel paths take whole rows and queue them up, the split grid
// cuts the same tiles evenly: better once the (row, KV head) pairs fill the SMs twice for the short kernel, of which two fit
// an SM (8 KV heads, 128 tokens: 32 rows 15.9 against 19.6 us, 64 rows 32 against 28.5), and once for the fused pipeline
// (499 tokens: 16 rows 17 against 20 us, 32 rows 32 against 26, 64 rows 65 against 40).
static bool fused_by_split(const dkv_attn_args* a) {
  const int n_sm = a->n_sm > 0 ? a->n_sm : sm_count();
  return (long long)a->batch * a->n_basis_groups > (short_ok(a) ? 2LL : 1LL) * n_sm;
}
// Kernels of a routed call on the packed path: 1 = the short kernel for rows of any length, 2 = split + merge for all rows, 3 = the
// short kernel for short rows and split + merge for the others.  A launch of a kernel whose rows are all someone else's costs
// 2 us, so all rows take one route (8 rows of 500 tokens: 18.0 us with three kernels, 15.1 with two) unless it would be less
// exact: the short kernel keeps scores in fp32 and weights as value and remainder, the pipeline, which is what short rows take in
// batches past short_ok, does what the split does.
static int routed_launches(const dkv_attn_args* a, int switch_tokens) {
  dkv_attn_args s = *a, all = *a;
  all.route_min_tokens = all.route_max_tokens = s.route_min_tokens = 0;
  s.route_max_tokens = switch_tokens;
  if (short_takes_all(&all, switch_tokens) && !fused_by_split(&all)) return 1;
  return !short_ok(&s) || fused_by_split(&s) ? 2 : 3;
}
}  // namespace dkv

extern "C" int dkv_fused_decode(const dkv_attn_args* a) {
  if (int rc = check_attn_args(a, "dkv_fused_decode", true, true, true)) return rc;
  if (mma_path_ok(a)) {
    if (fused_by_split(a) && a->workspace != nullptr && a->workspace_bytes >= mma_split_workspace_bytes(a) && ((uintptr_t)a->workspace & 15) == 0) {
      if (int rc = mma_split(a)) return rc;
      return mma_combine(a);
    }
    return short_ok(a) ? short_fused(a) : mma_fused(a);
  }
  return generic_attention(a);
}

extern "C" size_t dkv_split_workspace_bytes(const dkv_attn_args* a) {
  if (a == nullptr) return 0;
  if (!mma_path_ok(a)) return tiles_workspace_bytes(a);
  return mma_split_workspace_bytes(a);
}

extern "C" size_t dkv_fused_workspace_bytes(const dkv_attn_args* a) {
  if (a == nullptr) return 0;
  if (!mma_path_ok(a)) return tiles_workspace_bytes(a);
  return fused_by_split(a) ? mma_split_workspace_bytes(a) : 0;
}

extern "C" int dkv_split_decode(const dkv_attn_args* a) {
  if (int rc = check_attn_args(a, "dkv_split_decode", true, true, true)) return rc;
  DKV_REQUIRE(mma_path_ok(a), DKV_E_ARG,
              "dkv_split_decode: needs 16-bit elements, per-KV-head arenas, rank <= 128, lengths declared as "
              "multiples of 8 and 16-byte aligned arena rows; use dkv_two_stage_decode for other caches");
  return mma_split(a);
}

extern "C" int dkv_split_combine(const dkv_attn_args* a) {
  if (int rc = check_attn_args(a, "dkv_split_combine", false, false, false)) return rc;
  DKV_REQUIRE(a->v_up != nullptr, DKV_E_ARG, "dkv_split_combine: null v_up");
  DKV_REQUIRE(mma_path_ok(a), DKV_E_ARG, "dkv_split_combine: arguments do not describe a split-path call");
  return mma_combine(a);
}

extern "C" int dkv_two_stage_decode(const dkv_attn_args* a) {
  if (int rc = check_attn_args(a, "dkv_two_stage_decode", true, true, true)) return rc;
  if (!mma_path_ok(a)) return generic_attention(a);
  if (int rc = mma_split(a)) return rc;
  return mma_combine(a);
}

extern "C" int dkv_routed_decode(const dkv_attn_args* a, int32_t switch_tokens) {
  if (int rc = check_attn_args(a, "dkv_routed_decode", true, true, true)) return rc;
  DKV_REQUIRE(a->seq_lens != nullptr, DKV_E_ARG, "dkv_routed_decode: needs seq_lens");
  dkv_attn_args s = *a, l = *a;
  s.route_min_tokens = l.route_min_tokens = l.route_max_tokens = 0;
  if (switch_tokens <= 0) return dkv_two_stage_decode(&l);      // no row is short
  s.route_max_tokens = l.route_min_tokens = switch_tokens;
  if (mma_path_ok(a)) {
    const int n = routed_launches(a, switch_tokens);
    l.route_min_tokens = n < 3 ? 0 : switch_tokens;
    if (n == 1) return short_fused(&l);
    if (n == 2) return dkv_two_stage_decode(&l);
  }
  if (int rc = dkv_fused_decode(&s)) return rc;
  return dkv_two_stage_decode(&l);
}

extern "C" int dkv_routed_launches(const dkv_attn_args* a, int32_t switch_tokens) {
  if (a == nullptr || !mma_path_ok(a)) return 0;
  return switch_tokens > 0 ? routed_launches(a, switch_tokens) : 2;
}

extern "C" int dkv_two_stage_decode_noalloc(const dkv_attn_args* a) {
  if (int rc = check_attn_args(a, "dkv_two_stage_decode_noalloc", true, true, true)) return rc;
  return mma_two_stage_noalloc(a);
}
