// Prompt portions of the hybrid decoders' attention layers on the persistent tcgen05 kernel (fa_tc.cuh).
//
//   windowed grouped-query attention : queries from the projection, keys and values from token-major cache rows through the page table
//   latent attention                 : keys and values of every head formed from the cached latents first.  Per (head, query, key) the
//                                      products are then 192 + 128 wide instead of the 576 + 512 of attention over the latents themselves
//                                      (rank 512), which pays from a few tens of queries per sequence on.
#include "mix_common.cuh"
#include "fa_tc.cuh"

using namespace b200fa;

namespace {

// Rows of a cache are read by page: the map covers every row a page id can name.
constexpr uint64_t ANY_ROWS = (1ull << 31) - 1;

// Pages the kernel's boxes can follow: a block of 64 keys is whole pages, or lies inside one.
bool pages_ok(int block_size) { return block_size % BN == 0 || (block_size >= 8 && BN % block_size == 0); }

// The last rows of every sequence, one sequence after the other: out[i] for i in [cu_rows[s], cu_rows[s + 1]) are the cached rows of that many tokens at the
// end of sequence s.  A warp per row, 16-byte pieces.
__global__ void __launch_bounds__(256) latent_gather_kernel(const uint4* __restrict__ cache, int pieces, const int32_t* __restrict__ block_tables, int bt_stride,
                                                            int block_size, const int32_t* __restrict__ cu_k, const int32_t* __restrict__ cu_rows, int num_seqs,
                                                            uint4* __restrict__ out, int out_rows) {
    B200_PDL_SYNC();
    const int i = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (i >= out_rows || i >= cu_rows[num_seqs]) return;
    int s = 0;                                                           // the last sequence that begins at or before row i
    for (int hi = num_seqs; hi - s > 1;) {
        const int mid = (s + hi) >> 1;
        if (cu_rows[mid] <= i) s = mid;
        else hi = mid;
    }
    const int j = cu_k[s + 1] - cu_k[s] - (cu_rows[s + 1] - i);          // token of the sequence
    const int page = block_tables[(int64_t)s * bt_stride + j / block_size];
    const uint4* src = cache + ((int64_t)page * block_size + j % block_size) * pieces;
    uint4* dst = out + (int64_t)i * pieces;
    for (int c = lane; c < pieces; c += 32) dst[c] = page < 0 ? make_uint4(0, 0, 0, 0) : src[c];
}

// cu_rows[s] = sum over the sequences before s of the keys that some query of theirs sees: all up to `window` - 1 before the first query.  One CTA.
__global__ void __launch_bounds__(1024) latent_visible_kernel(const int32_t* __restrict__ cu_q, const int32_t* __restrict__ cu_k, int num_seqs, int window,
                                                              int32_t* __restrict__ cu_rows) {
    B200_PDL_SYNC();
    __shared__ int sums[32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    int at = 0;
    for (int s0 = 0; s0 < num_seqs; s0 += 1024) {
        const int s = s0 + tid;
        int len = 0;
        if (s < num_seqs) {
            const int n = cu_q[s + 1] - cu_q[s];
            len = n > 0 ? (int)min((int64_t)(cu_k[s + 1] - cu_k[s]), (int64_t)n + window - 1) : 0;      // any window, up to the largest int
        }
        int inc = len;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += v;
        }
        if (lane == 31) sums[warp] = inc;
        __syncthreads();
        if (warp == 0) {
            int v = sums[lane];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int u = __shfl_up_sync(0xffffffffu, v, o);
                if (lane >= o) v += u;
            }
            sums[lane] = v;
        }
        __syncthreads();
        if (s < num_seqs) cu_rows[s] = at + inc - len + (warp ? sums[warp - 1] : 0);
        at += sums[31];
        __syncthreads();
    }
    if (tid == 0) cu_rows[num_seqs] = at;
}

// The rotated part of every head's query, in place: a thread per V pairs (V = 4: 16-byte (layout 0) or 8-byte (layout 1) accesses; a pair per thread
// took 24.6 us for 8192 tokens x 16 heads of 64 columns, 17 MB read and written).  layout 0: pairs (2i, 2i + 1), 1: (i, i + dims / 2).
template <int V>
__global__ void __launch_bounds__(256) latent_rotate_kernel(__nv_bfloat16* q, int64_t tok_stride, int head_stride, const float* __restrict__ cos_sin, int dims,
                                                            const int64_t* __restrict__ positions, int n, int heads, int layout) {
    B200_PDL_SYNC();
    const int half = dims / 2, per = half / V;
    const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
    if (i >= (int64_t)n * heads * per) return;
    const int c = (int)(i % per) * V, h = (int)(i / per % heads), t = (int)(i / per / heads);
    __nv_bfloat16* x = q + t * tok_stride + (int64_t)h * head_stride;
    const float* cs = cos_sin + positions[t] * dims;
    float u[V], v[V];
    if constexpr (V == 4) {
        const float4 co = *reinterpret_cast<const float4*>(cs + c), si = *reinterpret_cast<const float4*>(cs + half + c);
        const float cc[4] = {co.x, co.y, co.z, co.w}, ss[4] = {si.x, si.y, si.z, si.w};
        if (layout) {
            uint2 *lo = reinterpret_cast<uint2*>(x + c), *hi = reinterpret_cast<uint2*>(x + c + half);
            const uint2 a = *lo, b = *hi;
            const float fa[4] = {bf16lo(a.x), bf16hi(a.x), bf16lo(a.y), bf16hi(a.y)}, fb[4] = {bf16lo(b.x), bf16hi(b.x), bf16lo(b.y), bf16hi(b.y)};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                u[k] = fa[k] * cc[k] - fb[k] * ss[k];
                v[k] = fb[k] * cc[k] + fa[k] * ss[k];
            }
            *lo = make_uint2(pack_bf16x2(u[0], u[1]), pack_bf16x2(u[2], u[3]));
            *hi = make_uint2(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]));
        } else {
            uint4* at = reinterpret_cast<uint4*>(x + 2 * c);
            float f[8];
            unpack8(*at, f);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const float a = f[2 * k], b = f[2 * k + 1];
                f[2 * k] = a * cc[k] - b * ss[k];
                f[2 * k + 1] = b * cc[k] + a * ss[k];
            }
            *at = pack8(f);
        }
    } else {
        const int e0 = layout ? c : 2 * c, e1 = layout ? c + half : 2 * c + 1;
        u[0] = __bfloat162float(x[e0]);
        v[0] = __bfloat162float(x[e1]);
        x[e0] = __float2bfloat16_rn(u[0] * cs[c] - v[0] * cs[half + c]);
        x[e1] = __float2bfloat16_rn(v[0] * cs[c] + u[0] * cs[half + c]);
    }
}

}  // namespace

// Called from b200m_window_attention, which has validated the arguments.
int b200m_window_prompt(const void* q, int64_t q_stride, const void* cache, int row_elems, int v_off, const int32_t* block_tables, int bt_stride, int block_size,
                        const int32_t* cu_q, const int32_t* cu_k, const float* slopes, int window, int chunk, const float* sinks, const void* gate,
                        int64_t gate_stride, int gate_elems, float out_scale, void* out, int64_t out_stride, bool out_f32, int total_q, int num_seqs, int max_q,
                        int heads, int kv_heads, float scale, cudaStream_t stream) {
    constexpr int D = 128;
    const uintptr_t bases = reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(cache) | reinterpret_cast<uintptr_t>(out) |
                            (gate && gate_elems ? reinterpret_cast<uintptr_t>(gate) : 0);
    if (bases % 16 || q_stride % 8 || row_elems % 8 || v_off % 8 || out_stride % (out_f32 ? 4 : 8) || (gate && gate_elems && gate_stride % 8) || !pages_ok(block_size))
        return B200_EUNSUPPORTED;
    const int box = block_size < BN ? block_size : BN;
    CUtensorMap tq, tk;
    if (!make_map(&tq, q, (uint64_t)heads * D, (uint64_t)total_q, (uint64_t)q_stride, BM) ||
        !make_map(&tk, cache, (uint64_t)row_elems, ANY_ROWS, (uint64_t)row_elems, box))
        return B200_EUNSUPPORTED;
    FaParams p = {};
    p.cu_q = cu_q;
    p.cu_k = cu_k;
    p.block_tables = block_tables;
    p.bt_stride = bt_stride;
    p.num_seqs = num_seqs;
    p.hq = heads;
    p.hkv = kv_heads;
    p.q_col_step = p.k_col_step = p.v_col_step = D;
    p.v_col0 = v_off;
    p.block_size = block_size;
    p.box_rows = box;
    p.page_rows = block_size;
    p.scale_log2 = scale * LOG2E;
    p.lag = 0.f;                         // as the mma.sync forms of these layers
    p.slopes = slopes;
    p.sinks = sinks;
    p.window = window;
    p.chunk = chunk;
    p.out = out;
    p.out_stride = out_stride;
    p.out_f32 = out_f32;
    p.out_scale = out_scale;
    p.gate = static_cast<const __nv_bfloat16*>(gate);
    p.gate_stride = gate_stride;
    p.gate_elems = gate_elems;
    const bool pair = heads / kv_heads % 2 == 0, plain = !slopes && scale > 0.f;
    if (pair) return plain ? fa_launch<D, true, false>(p, tq, tk, tk, tk, total_q, max_q, stream) : fa_launch<D, true, true>(p, tq, tk, tk, tk, total_q, max_q, stream);
    return plain ? fa_launch<D, false, false>(p, tq, tk, tk, tk, total_q, max_q, stream) : fa_launch<D, false, true>(p, tq, tk, tk, tk, total_q, max_q, stream);
}

extern "C" int b200m_latent_visible(const int32_t* cu_q, const int32_t* cu_k, int num_seqs, int window, int32_t* cu_rows, void* stream) {
    if (!cu_q || !cu_k || !cu_rows || num_seqs < 0 || window <= 0) return B200_EINVAL;
    B200_LAUNCH((latent_visible_kernel), 1, 1024, 0, static_cast<cudaStream_t>(stream), cu_q, cu_k, num_seqs, window, cu_rows);
    return b200_launch_status(nullptr);
}

extern "C" int b200m_latent_gather(const void* cache, int row_elems, const int32_t* block_tables, int bt_stride, int block_size, const int32_t* cu_k, const int32_t* cu_rows,
                                   int num_seqs, void* out, int out_rows, void* stream) {
    if (!cache || !block_tables || !cu_k || !cu_rows || !out || row_elems <= 0 || block_size <= 0 || num_seqs < 0 || out_rows < 0) return B200_EINVAL;
    if (row_elems % 8 || (reinterpret_cast<uintptr_t>(cache) | reinterpret_cast<uintptr_t>(out)) % 16) return B200_EUNSUPPORTED;
    if (num_seqs == 0 || out_rows == 0) return B200_OK;
    B200_LAUNCH((latent_gather_kernel), (out_rows + 7) / 8, 256, 0, static_cast<cudaStream_t>(stream), static_cast<const uint4*>(cache), row_elems / 8, block_tables,
                bt_stride, block_size, cu_k, cu_rows, num_seqs, static_cast<uint4*>(out), out_rows);
    return b200_launch_status(nullptr);
}

extern "C" int b200m_latent_rotate(void* q, int64_t tok_stride, int head_stride, const float* cos_sin, int rope_dims, const int64_t* positions, int n, int heads,
                                   int layout, void* stream) {
    if (!q || !cos_sin || !positions || n < 0 || heads <= 0 || rope_dims < 0 || rope_dims % 2) return B200_EINVAL;
    if (n == 0 || rope_dims == 0) return B200_OK;
    auto go = [&](auto kernel, int per) {
        const int64_t total = (int64_t)n * heads * (rope_dims / 2 / per);
        B200_LAUNCH((kernel), dim3((unsigned)((total + 255) / 256)), 256, 0, static_cast<cudaStream_t>(stream), static_cast<__nv_bfloat16*>(q), tok_stride, head_stride, cos_sin,
                    rope_dims, positions, n, heads, layout);
    };
    if (rope_dims % 8 == 0 && tok_stride % 8 == 0 && head_stride % 8 == 0 && (reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(cos_sin)) % 16 == 0)
        go(latent_rotate_kernel<4>, 4);
    else
        go(latent_rotate_kernel<1>, 1);
    return b200_launch_status(nullptr);
}

extern "C" int b200m_latent_prompt(const void* q, int64_t q_stride, const void* keys, const void* values, int64_t kv_stride, const void* rows, int row_elems, int rank,
                                   int total_k, const int32_t* cu_q, const int32_t* cu_k, const float* sink, void* out, int64_t out_stride, int total_q, int num_seqs, int max_q,
                                   int heads, int dim, int rot_dim, int vdim, float scale, int window, void* stream) {
    if (!q || !keys || !values || !rows || !cu_q || !cu_k || !out || total_q < 0 || num_seqs < 0 || heads <= 0 || rank <= 0 || total_k < 0) return B200_EINVAL;
    const uintptr_t bases = reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(keys) | reinterpret_cast<uintptr_t>(values) |
                            reinterpret_cast<uintptr_t>(rows) | reinterpret_cast<uintptr_t>(out);
    if (dim != 128 || rot_dim != 64 || vdim != 128 || scale <= 0.f || bases % 16 || q_stride % 8 || out_stride % 8 || kv_stride % 8 || row_elems % 8 || rank % 8) return B200_EUNSUPPORTED;
    if (total_q == 0 || num_seqs == 0 || max_q <= 0) return B200_OK;
    CUtensorMap tq, tk, tv, tr;
    if (!make_map(&tq, q, (uint64_t)heads * 192, (uint64_t)total_q, (uint64_t)q_stride, BM) || !make_map(&tk, keys, (uint64_t)heads * 128, (uint64_t)total_k, (uint64_t)kv_stride, BN) ||
        !make_map(&tv, values, (uint64_t)heads * 128, (uint64_t)total_k, (uint64_t)kv_stride, BN) || !make_map(&tr, rows, (uint64_t)row_elems, (uint64_t)total_k, (uint64_t)row_elems, BN))
        return B200_EUNSUPPORTED;
    FaParams p = {};
    p.cu_q = cu_q;
    p.cu_k = cu_k;
    p.num_seqs = num_seqs;
    p.hq = p.hkv = heads;
    p.q_col_step = 192;
    p.k_col_step = p.v_col_step = 128;
    p.k2_col = rank;
    p.block_size = p.box_rows = BN;
    p.scale_log2 = scale * LOG2E;
    p.lag = 0.f;                         // as the mma.sync forms of these layers
    p.sinks = sink;
    p.window = window;
    p.out = out;
    p.out_stride = out_stride;
    p.out_scale = 1.0f;
    return fa_launch<192, false, false>(p, tq, tk, tv, tr, total_q, max_q, static_cast<cudaStream_t>(stream));
}
