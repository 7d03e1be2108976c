// Prompt attention of the paged grouped-query path (reference nanovllm/layers/attention.py:64-70, flash_attn_varlen_func with an optional
// block table): the persistent tcgen05 kernel of fa_tc.cuh over packed projections or head-major pages, bottom-right aligned causal mask.
#include "fa_tc.cuh"

using namespace b200fa;

// Called from b200_paged_prefill (prefill_attn.cu), which has validated the arguments.  Returns B200_EUNSUPPORTED if TMA descriptors cannot be built.
int b200_prefill_fa_launch(b200_ctx* ctx, int layer, const void* q, int64_t q_stride0, const void* k, int64_t k_stride0,
                           const void* v, int64_t v_stride0, const int32_t* cu_q, const int32_t* cu_k,
                           const int32_t* block_tables, int bt_stride, void* out, int64_t out_stride0, int total_q,
                           int num_seqs, int max_seqlen_q, int num_q_heads, int num_kv_heads, float scale,
                           const int32_t* slot_mapping, int num_slots, cudaStream_t stream) {
    constexpr int D = B200_HEAD_DIM;
    CUtensorMap tq, tk, tv;
    if (!make_map(&tq, q, (uint64_t)num_q_heads * D, (uint64_t)total_q, (uint64_t)q_stride0, BM)) return B200_EUNSUPPORTED;
    FaParams p = {};
    p.cu_q = cu_q;
    p.cu_k = cu_k;
    p.block_tables = block_tables;
    p.bt_stride = bt_stride;
    p.num_seqs = num_seqs;
    p.hq = num_q_heads;
    p.hkv = num_kv_heads;
    p.q_col_step = D;
    p.scale_log2 = scale * LOG2E;
    p.lag = 8.0f;
    p.out = out;
    p.out_stride = out_stride0;
    p.out_scale = 1.0f;
    p.block_size = p.box_rows = BN;
    if (block_tables) {
        const uint64_t rows = (uint64_t)ctx->layers * ctx->num_blocks * ctx->num_kv_heads * ctx->block_size;
        if (rows >= (1ull << 31)) return B200_EUNSUPPORTED;
        p.block_size = ctx->block_size;
        p.box_rows = ctx->block_size < BN ? ctx->block_size : BN;
        p.head_rows = ctx->block_size;
        p.page_rows = (int64_t)ctx->block_size * ctx->num_kv_heads;
        p.row0 = (int64_t)layer * ctx->num_blocks * p.page_rows;
        if (!make_map(&tk, ctx->k_base, D, rows, D, p.box_rows) || !make_map(&tv, ctx->v_base, D, rows, D, p.box_rows)) return B200_EUNSUPPORTED;
    } else {                             // packed: K / V rows are the step's own tokens
        p.k_col_step = p.v_col_step = D;
        if (!make_map(&tk, k, (uint64_t)num_kv_heads * D, (uint64_t)total_q, (uint64_t)k_stride0, BN) ||
            !make_map(&tv, v, (uint64_t)num_kv_heads * D, (uint64_t)total_q, (uint64_t)v_stride0, BN))
            return B200_EUNSUPPORTED;
    }
    if (slot_mapping) {                  // rows, and the layer's cache rows, are named by 32 bits
        if (block_tables || scale <= 0.f || ctx->num_blocks * ctx->num_kv_heads * ctx->block_size >= (1ll << 31) || (int64_t)num_slots * num_kv_heads >= (1ll << 31) - 256)
            return B200_EUNSUPPORTED;
        p.st_slots = slot_mapping;
        p.st_k = static_cast<const __nv_bfloat16*>(k);
        p.st_v = static_cast<const __nv_bfloat16*>(v);
        p.st_k_stride = k_stride0;
        p.st_v_stride = v_stride0;
        p.st_kc = ctx->k_layer(layer);
        p.st_vc = ctx->v_layer(layer);
        p.st_rows = num_slots * num_kv_heads;
        p.st_shift = ctx->block_shift;
    }
    // An even head group: the item's two tiles are two heads that share every K and V tile.  Else (groups of 1, 3, ..): 256 rows of one head.
    const bool pair = (num_q_heads / num_kv_heads) % 2 == 0;
    if (slot_mapping)
        return pair ? fa_launch<D, true, false, true>(p, tq, tk, tv, tk, total_q, max_seqlen_q, stream)
                    : fa_launch<D, false, false, true>(p, tq, tk, tv, tk, total_q, max_seqlen_q, stream);
    if (scale > 0.f)
        return pair ? fa_launch<D, true, false>(p, tq, tk, tv, tk, total_q, max_seqlen_q, stream) : fa_launch<D, false, false>(p, tq, tk, tv, tk, total_q, max_seqlen_q, stream);
    return pair ? fa_launch<D, true, true>(p, tq, tk, tv, tk, total_q, max_seqlen_q, stream) : fa_launch<D, false, true>(p, tq, tk, tv, tk, total_q, max_seqlen_q, stream);
}
