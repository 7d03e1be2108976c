// C-ABI entry of the prefill branch of the reference's Attention.forward (nanovllm/layers/attention.py:64-70,
// flash_attn_varlen_func with an optional block_table).  The kernel is the persistent tcgen05 / TMEM / TMA attention of fa_tc.cuh,
// launched from prefill_fa.cu; this file validates arguments and forwards.
#include "common.cuh"

int b200_prefill_fa_launch(b200_ctx* ctx, int layer, const void* q, int64_t q_stride0, const void* k, int64_t k_stride0,
                           const void* v, int64_t v_stride0, const int32_t* cu_q, const int32_t* cu_k,
                           const int32_t* block_tables, int bt_stride, void* out, int64_t out_stride0, int total_q,
                           int num_seqs, int max_seqlen_q, int num_q_heads, int num_kv_heads, float scale,
                           const int32_t* slot_mapping, int num_slots, cudaStream_t stream);

extern "C" int b200_paged_prefill(b200_ctx* ctx, int layer, const void* q, int64_t q_stride0,
                                  const void* k, int64_t k_stride0, const void* v,
                                  int64_t v_stride0, const int32_t* cu_seqlens_q,
                                  const int32_t* cu_seqlens_k, const int32_t* block_tables,
                                  int bt_stride, void* out, int64_t out_stride0, int total_q,
                                  int num_seqs, int max_seqlen_q, int max_seqlen_k,
                                  int num_q_heads, int num_kv_heads, float scale, void* stream) {
    (void)max_seqlen_k;
    if (!ctx || !q || !out || !cu_seqlens_q || !cu_seqlens_k || num_seqs < 0 || total_q < 0) return B200_EINVAL;
    if (num_kv_heads <= 0 || num_q_heads % num_kv_heads) return B200_EINVAL;
    if (total_q == 0 || num_seqs == 0 || max_seqlen_q <= 0) return B200_OK;
    if ((q_stride0 % 8) || (out_stride0 % 8) || ((uintptr_t)q & 15) || ((uintptr_t)out & 15)) return B200_EINVAL;
    if (block_tables) {
        if (!ctx->k_base) return B200_ENOTBOUND;
        if (layer < 0 || layer >= ctx->layers || num_kv_heads != ctx->num_kv_heads) return B200_EINVAL;
    } else {
        if (!k || !v || (k_stride0 % 8) || (v_stride0 % 8) || ((uintptr_t)k & 15) || ((uintptr_t)v & 15)) return B200_EINVAL;
    }
    return b200_prefill_fa_launch(ctx, layer, q, q_stride0, k, k_stride0, v, v_stride0, cu_seqlens_q, cu_seqlens_k, block_tables, bt_stride,
                                  out, out_stride0, total_q, num_seqs, max_seqlen_q, num_q_heads, num_kv_heads, scale,
                                  nullptr, 0, static_cast<cudaStream_t>(stream));
}

// Packed prompts whose K / V rows go into the cache on the way, copied by the kernel's idle warps under the products.
extern "C" int b200_paged_prefill_store(b200_ctx* ctx, int layer, const void* q, int64_t q_stride0, const void* k, int64_t k_stride0, const void* v,
                                        int64_t v_stride0, const int32_t* slot_mapping, int num_slots, const int32_t* cu_seqlens_q,
                                        const int32_t* cu_seqlens_k, void* out, int64_t out_stride0, int total_q, int num_seqs, int max_seqlen_q,
                                        int num_q_heads, int num_kv_heads, float scale, void* stream) {
    if (!ctx || !q || !k || !v || !out || !slot_mapping || !cu_seqlens_q || !cu_seqlens_k || num_seqs < 0 || total_q < 0 || num_slots < 0) return B200_EINVAL;
    if (!ctx->k_base) return B200_ENOTBOUND;
    if (layer < 0 || layer >= ctx->layers || num_kv_heads != ctx->num_kv_heads || num_kv_heads <= 0 || num_q_heads % num_kv_heads) return B200_EINVAL;
    const uintptr_t kp = reinterpret_cast<uintptr_t>(k), vp = reinterpret_cast<uintptr_t>(v);
    if (q_stride0 % 8 || out_stride0 % 8 || k_stride0 % 8 || v_stride0 % 8 || k_stride0 < 0 || v_stride0 < 0 ||
        ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(out) | kp | vp) & 15))
        return B200_EUNSUPPORTED;
    if (total_q == 0 || num_seqs == 0 || max_seqlen_q <= 0 || num_slots == 0) return B200_EUNSUPPORTED;          // no launch to ride in
    // rows that lie in the cache themselves are read after the scatter, not beside it
    const uintptr_t bytes = (uintptr_t)ctx->layers * ctx->layer_elems() * 2, row = (uintptr_t)num_kv_heads * B200_HEAD_DIM;
    const uintptr_t k_end = kp + ((uintptr_t)(num_slots - 1) * k_stride0 + row) * 2, v_end = vp + ((uintptr_t)(num_slots - 1) * v_stride0 + row) * 2;
    for (uintptr_t base : {reinterpret_cast<uintptr_t>(ctx->k_base), reinterpret_cast<uintptr_t>(ctx->v_base)})
        if ((kp < base + bytes && base < k_end) || (vp < base + bytes && base < v_end)) return B200_EUNSUPPORTED;
    return b200_prefill_fa_launch(ctx, layer, q, q_stride0, k, k_stride0, v, v_stride0, cu_seqlens_q, cu_seqlens_k, nullptr, 0, out, out_stride0, total_q,
                                  num_seqs, max_seqlen_q, num_q_heads, num_kv_heads, scale, slot_mapping, num_slots, static_cast<cudaStream_t>(stream));
}
