// Single-token paged decode attention of small steps (reference nanovllm/layers/attention.py:71-74).
//
// A step of a few sequences is bound by latency, not by HBM: the stream-K kernel (decode_attn.cu) prefixes the whole batch, gives each warp
// eight chunks that pass through a two-deep ring one after the other, and merges through global memory with a counter (15-20 us whatever the
// bytes).  Here a CTA belongs to one (sequence, kv head): its eight warps take 16-token chunks in turn, straight from global memory into
// registers (16 loads of 16 bytes per lane in flight, the next chunk's already asked for), meet in shared memory, and the CTAs of a cluster that
// share a long context exchange their partials through distributed shared memory.  No workspace, no atomics, one launch; the order of every
// sum is fixed by the shape.
//
// The walk over a context's chunks is decode_walk.cuh's; FUSED takes the raw qkv projection (q/k-norm, RoPE and the KV append happen here).  Wider head groups than GW heads take several CTAs per kv head (K and V then come from L2).
#include "decode_walk.cuh"

using namespace b200dec;

namespace {

__device__ __forceinline__ void cluster_sync() { asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory"); }
__device__ __forceinline__ float ld_cluster(const float* p, uint32_t rank) {
    uint32_t remote;
    float v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(smem_u32(p)), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(remote) : "memory");
    return v;
}

// GW: query heads of this CTA.  grid = (splits of a context, hkv * (G / GW), batch), cluster = (splits, 1, 1).
template <int GW, bool FUSED>
__global__ void __launch_bounds__(SW * 32, 1) paged_decode_small_kernel(const DecodeParams p, int G) {
    B200_PDL_TRIGGER();
    constexpr int D = B200_HEAD_DIM;
    __shared__ float sh_o[SW][GW][D];              // each warp's unnormalised result
    __shared__ float sh_ml[SW][GW][2];
    __shared__ float red_o[GW][D];                 // this CTA's
    __shared__ float red_ml[GW][2];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, hw = lane >> 4, j = lane & 15;
    const int splits = gridDim.x, rank = blockIdx.x, subs = G / GW;
    const int kvh = blockIdx.y / subs, head0 = kvh * G + (blockIdx.y % subs) * GW, b = blockIdx.z;
    const bool writer = blockIdx.y % subs == 0;    // of the CTAs that share a kv head, the one that appends
    // metadata is uploaded before the step: read while the kernels in front drain
    const int ctx = max(p.context_lens[b], 0);
    const int old = FUSED ? max(ctx - 1, 0) : ctx; // tokens that are in the cache
    const int n = (old + CHUNK - 1) / CHUNK, c0 = (int)((int64_t)n * rank / splits), c1 = (int)((int64_t)n * (rank + 1) / splits);
    const int32_t* bt = p.block_tables + (int64_t)b * p.bt_stride;
    const int mask = (1 << p.block_shift) - 1;
    auto row_of = [&](int ck) -> int64_t {         // first cache row of a chunk (a chunk lies inside one page)
        const int tok = ck * CHUNK;
        return (((int64_t)bt[tok >> p.block_shift] * p.hkv + kvh) << p.block_shift) + (tok & mask);
    };
    int64_t row = c0 + warp < c1 ? row_of(c0 + warp) : 0;
    B200_PDL_WAIT();

    const WalkLane wl(lane);
    auto load = [&](int ck, int64_t at, uint4 (&k)[8], uint4 (&v)[8]) {
        walk_load(wl, p.k_layer, at, old - ck * CHUNK, k);
        walk_load(wl, p.v_layer, at, old - ck * CHUNK, v);
    };
    uint4 kr[8], vr[8];
    if (c0 + warp < c1) load(c0 + warp, row, kr, vr);

    // ---- queries ----
    float qw[8], kw[8], cosr[8], sinr[8];
    const __nv_bfloat16* qrow = p.q + (int64_t)b * p.q_stride + j * 8;
    if (FUSED) {
        unpack8(*reinterpret_cast<const uint4*>(p.q_norm_w + j * 8), qw);
        unpack8(*reinterpret_cast<const uint4*>(p.k_norm_w + j * 8), kw);
        const float* cs = p.cos_sin + (int64_t)old * D + (j & 7) * 8;
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            cosr[e] = cs[e];
            sinr[e] = cs[64 + e];
        }
    }
    WalkState<GW> st;
#pragma unroll
    for (int g = 0; g < GW; ++g) {
        unpack8(*reinterpret_cast<const uint4*>(qrow + (head0 + g) * D), st.q[g]);
        if (FUSED) walk_norm_rope(wl, st.q[g], qw, cosr, sinr, p.eps);
    }
    st.begin(p.scale_log2);

#pragma unroll 1
    for (int ck = c0 + warp; ck < c1; ck += SW) {
        uint4 kn[8], vn[8];
        if (ck + SW < c1) load(ck + SW, row_of(ck + SW), kn, vn);
        st.chunk(wl, kr, vr, old - ck * CHUNK);
#pragma unroll
        for (int it = 0; it < 8; ++it) {
            kr[it] = kn[it];
            vr[it] = vn[it];
        }
    }
    if (FUSED && ctx > 0 && rank == splits - 1 && warp == SW - 1) {          // the step's own token
        float kn[8], vn[8];
        const uint4 v_raw = *reinterpret_cast<const uint4*>(qrow + (p.hkv * G + p.hkv + kvh) * D);
        unpack8(*reinterpret_cast<const uint4*>(qrow + (p.hkv * G + kvh) * D), kn);
        unpack8(v_raw, vn);
        walk_norm_rope(wl, kn, kw, cosr, sinr, p.eps);
        if (hw == 0 && writer) {
            const int64_t at = (((int64_t)bt[old >> p.block_shift] * p.hkv + kvh) << p.block_shift) + (old & mask);
            *reinterpret_cast<uint4*>(p.k_layer_w + at * D + j * 8) = pack8(kn);
            *reinterpret_cast<uint4*>(p.v_layer_w + at * D + j * 8) = v_raw;
        }
        st.own(wl, kn, vn);
    }
    // ---- the warps of this CTA meet ----
    st.leave(wl, sh_o[warp], sh_ml[warp]);
    __syncthreads();
    auto store = [&](int g, int d, float v) { p.out[(int64_t)b * p.out_stride + (head0 + g) * D + d] = __float2bfloat16_rn(v); };
    for (int i = tid; i < GW * D; i += SW * 32) {
        const int g = i / D, d = i % D;
        float M, L, a;
        walk_meet(sh_o, sh_ml, g, d, M, L, a);
        if (splits == 1) {
            store(g, d, L > 0.f ? a / L : 0.f);
        } else {
            red_o[g][d] = a;
            if (d == 0) {
                red_ml[g][0] = M;
                red_ml[g][1] = L;
            }
        }
    }
    if (splits == 1) return;
    // ---- the CTAs of the cluster meet: each writes its share of the columns ----
    cluster_sync();
    for (int i = rank * (SW * 32) + tid; i < GW * D; i += splits * SW * 32) {
        const int g = i / D, d = i % D;
        float ms[8], M = -INFINITY, L = 0.f, a = 0.f;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            ms[c] = c < splits ? ld_cluster(&red_ml[g][0], c) : -INFINITY;
            M = fmaxf(M, ms[c]);
        }
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            if (c >= splits || ms[c] == -INFINITY) continue;
            const float f = fast_exp2(ms[c] - M);
            L = fmaf(f, ld_cluster(&red_ml[g][1], c), L);
            a = fmaf(f, ld_cluster(&red_o[g][d], c), a);
        }
        store(g, d, L > 0.f ? a / L : 0.f);
    }
    cluster_sync();                                // nobody leaves while its partials are being read
}

template <int GW, bool FUSED>
int launch_small(b200_ctx* ctx, const DecodeParams& prm, int G, int splits, cudaStream_t stream) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(splits, prm.hkv * (G / GW), prm.batch);
    cfg.blockDim = dim3(SW * 32);
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    int na = 0;
    if (splits > 1) {
        attr[na].id = cudaLaunchAttributeClusterDimension;
        attr[na].val.clusterDim = {(unsigned)splits, 1, 1};
        ++na;
    }
#ifdef B200_PDL
    if (!b200_tls_pdl_off()) {
        attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[na].val.programmaticStreamSerializationAllowed = 1;
        ++na;
    }
#endif
    cfg.attrs = attr;
    cfg.numAttrs = na;
    cudaLaunchKernelEx(&cfg, paged_decode_small_kernel<GW, FUSED>, prm, G);
    return b200_launch_status(ctx);
}

}  // namespace

// CTAs along a context (1, 2, 4 or 8: the cluster), or 0: a step for the stream-K kernels.
//
// Taken while every (sequence, kv head) has a CTA of its own in one wave and no warp can get more than MAX_CHUNKS chunks, whatever the contexts
// are (bounded by the table's width; the lengths are on the device).  A chunk takes a warp about 0.75 us (twice that with four heads), so the
// longest context allowed ends no later than the stream-K kernels do on the smallest step.  A captured step's tables are as wide as the longest
// sequence the engine may hold, so that length decides there: with 8 kv heads in groups of two, 1 and 2 rows take this kernel up to 16384 tokens, 4 rows
// up to 8192, 8 up to 4096, 9-18 up to 2048.  Measured (whole captured Qwen3-0.6B step, us, here / stream-K): 1 row 980 / 1323, 4 rows 1040 / 1330, 16
// rows with tables of 1024 tokens 1195 / 1362; beyond the bound (the operator alone) 16 rows of 600-8192 tokens 78 / 52, with 32 heads 112 / 56.
static int small_splits(const b200_ctx* ctx, int batch, int G, int bt_stride) {
    const int GW = G >= 4 ? 4 : G, ctas = batch * ctx->num_kv_heads * (G / GW), MAX_CHUNKS = GW == 4 ? 4 : 16;
    if (ctas > ctx->sm_count) return 0;
    int splits = 1;
    while (splits < 8 && ctas * splits * 2 <= ctx->sm_count) splits *= 2;
    const int64_t chunks = ((int64_t)bt_stride << ctx->block_shift) / CHUNK;
    return chunks > (int64_t)MAX_CHUNKS * SW * splits ? 0 : splits;
}

extern "C" int b200_decode_small_splits(const b200_ctx* ctx, int batch, int num_q_heads, int bt_stride) {
    if (!ctx || batch <= 0 || bt_stride < 0 || num_q_heads <= 0) return B200_EINVAL;
    if (!ctx->k_base) return B200_ENOTBOUND;
    const int G = num_q_heads % ctx->num_kv_heads ? 0 : num_q_heads / ctx->num_kv_heads;
    if (G != 1 && G != 2 && G != 4 && G != 8) return B200_EUNSUPPORTED;
    return small_splits(ctx, batch, G, bt_stride);
}

// Called from decode_common() in decode_attn.cu; B200_EUNSUPPORTED: a step for the stream-K kernels.
int b200_decode_small_launch(b200_ctx* ctx, const DecodeParams& prm, int G, bool fused, cudaStream_t stream) {
    const int GW = G >= 4 ? 4 : G, splits = small_splits(ctx, prm.batch, G, prm.bt_stride);
    if (splits == 0) return B200_EUNSUPPORTED;
    if (fused) return GW == 1 ? launch_small<1, true>(ctx, prm, G, splits, stream) : launch_small<2, true>(ctx, prm, G, splits, stream);
    switch (GW) {
        case 1: return launch_small<1, false>(ctx, prm, G, splits, stream);
        case 2: return launch_small<2, false>(ctx, prm, G, splits, stream);
        default: return launch_small<4, false>(ctx, prm, G, splits, stream);
    }
}
