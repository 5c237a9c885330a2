// Attention of a Qwen3 decode step over the paged cache: QK-norm, rotary embedding, K/V store and attention in one launch.
#include "attention_decode.cuh"

using namespace nqb200;

namespace {
template <typename T>
int run(const void* qkv, int64_t stride, const void* q_weight, const void* k_weight, const float* cos_sin, const int64_t* positions, const int64_t* slots,
        void* k_cache, void* v_cache, const int32_t* table, const int32_t* ctx, int64_t table_width, int64_t block_size, void* out, int64_t batch,
        int64_t heads, int64_t kv_heads, float scale, float eps, float* shares, cudaStream_t st) {
  attdec::Args<T> a = {};
  a.proj = (const T*)qkv; a.stride = stride; a.q_off = 0; a.k_off = heads * attdec::kDim; a.v_off = (heads + kv_heads) * attdec::kDim;
  a.k_cache = (T*)k_cache; a.v_cache = (T*)v_cache;
  a.table = table; a.table_width = (int)table_width; a.block_size = (int)block_size;
  a.last = ctx; a.last_shift = -1; a.rows = slots;
  a.heads = (int)heads; a.kv_heads = (int)kv_heads; a.chunk = 0;
  a.out = (T*)out; a.out_stride = heads * attdec::kDim; a.out_col = 0;
  a.scale = scale; a.out_scale = 1.f;
  a.shares = shares;
  a.cos_sin = cos_sin; a.positions = positions; a.q_weight = (const T*)q_weight; a.k_weight = (const T*)k_weight; a.eps = eps;
  return attdec::launch<true>(a, batch, table_width * block_size, false, st);
}
}  // namespace

static int attention(const void* qkv, int64_t row_stride, const void* q_weight, const void* k_weight, const float* cos_sin,
                     const int64_t* positions, const int64_t* slots, void* k_cache, void* v_cache, const int32_t* table, const int32_t* ctx,
                     int64_t table_width, int64_t block_size, void* out, int64_t batch, int64_t num_q_heads, int64_t num_kv_heads, int64_t head_dim,
                     float scale, float eps, int dtype, float* shares, void* stream) {
  if (batch < 0 || batch > 65535 || table_width <= 0 || table_width > INT32_MAX || block_size <= 0 || block_size > INT32_MAX ||
      !attdec::supported(num_q_heads, num_kv_heads, head_dim, head_dim) || row_stride < (num_q_heads + 2 * num_kv_heads) * head_dim || row_stride % 8 != 0)
    return NQB200_ERR_BAD_SHAPE;
  if (dtype != NQB200_F16 && dtype != NQB200_BF16) return NQB200_ERR_BAD_DTYPE;
  if (batch == 0) return NQB200_OK;
  if (!qkv || !q_weight || !k_weight || !cos_sin || !positions || !slots || !k_cache || !v_cache || !table || !ctx || !out) return NQB200_ERR_NULL_POINTER;
  if (!aligned16(qkv) || !aligned16(k_cache) || !aligned16(v_cache)) return NQB200_ERR_MISALIGNED;
  const auto go = dtype == NQB200_BF16 ? run<__nv_bfloat16> : run<__half>;
  return go(qkv, row_stride, q_weight, k_weight, cos_sin, positions, slots, k_cache, v_cache, table, ctx, table_width, block_size, out, batch, num_q_heads,
            num_kv_heads, scale, eps, shares, (cudaStream_t)stream);
}

extern "C" int nqb200_decode_attention(const void* qkv, int64_t row_stride, const void* q_weight, const void* k_weight, const float* cos_sin,
                                       const int64_t* positions, const int64_t* slots, void* k_cache, void* v_cache, const int32_t* table,
                                       const int32_t* ctx, int64_t table_width, int64_t block_size, void* out, int64_t batch, int64_t num_q_heads,
                                       int64_t num_kv_heads, int64_t head_dim, float scale, float eps, int dtype, void* stream) {
  return attention(qkv, row_stride, q_weight, k_weight, cos_sin, positions, slots, k_cache, v_cache, table, ctx, table_width, block_size, out, batch,
                   num_q_heads, num_kv_heads, head_dim, scale, eps, dtype, nullptr, stream);
}

extern "C" size_t nqb200_decode_attention_scratch_bytes(int64_t table_width, int64_t block_size, int64_t batch, int64_t num_q_heads, int64_t num_kv_heads) {
  if (batch <= 0 || batch > 65535 || table_width <= 0 || table_width > INT32_MAX || block_size <= 0 || block_size > INT32_MAX ||
      !attdec::supported(num_q_heads, num_kv_heads, attdec::kDim, attdec::kDim))
    return 0;
  const int64_t units = num_kv_heads * attdec::head_groups((int)num_q_heads, (int)num_kv_heads) * batch;
  return (size_t)attdec::share_floats(batch, (int)num_q_heads, attdec::split(units, table_width * block_size, true).parts) * sizeof(float);
}

extern "C" int nqb200_decode_attention_split(const void* qkv, int64_t row_stride, const void* q_weight, const void* k_weight, const float* cos_sin,
                                             const int64_t* positions, const int64_t* slots, void* k_cache, void* v_cache, const int32_t* table,
                                             const int32_t* ctx, int64_t table_width, int64_t block_size, void* out, int64_t batch, int64_t num_q_heads,
                                             int64_t num_kv_heads, int64_t head_dim, float scale, float eps, int dtype, void* scratch,
                                             size_t scratch_bytes, void* stream) {
  const size_t need = nqb200_decode_attention_scratch_bytes(table_width, block_size, batch, num_q_heads, num_kv_heads);
  if (need > 0 && (!scratch || scratch_bytes < need)) return NQB200_ERR_WORKSPACE;
  if (need > 0 && !aligned16(scratch)) return NQB200_ERR_MISALIGNED;
  return attention(qkv, row_stride, q_weight, k_weight, cos_sin, positions, slots, k_cache, v_cache, table, ctx, table_width, block_size, out, batch,
                   num_q_heads, num_kv_heads, head_dim, scale, eps, dtype, need > 0 ? (float*)scratch : nullptr, stream);
}
