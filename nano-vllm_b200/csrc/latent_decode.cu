// Latent attention of single-token steps on the 5th-generation tensor cores (bf16, up to 16 heads, latents of 256 or 512 columns beside a rotated
// key part of 64; latent_attn.cu has the definition and the general forms).
//
// Every cached row is read once for all heads, so the step is HBM-bound (226 MB for 64 sequences of 3072 tokens at rank 512: 35 us); what matters
// is to keep loads in flight.  One CTA per SM takes an equal share of the step's 64-key tiles, whatever the lengths (a share may begin and end
// inside a sequence; each (CTA, sequence) leaves an unnormalised partial that latent_fold_kernel sums in a fixed order).  Roles (224 threads):
//
//   warp 4       TMA: a tile as units of 128 columns (two swizzled [64 keys][64] pieces, 16 KB), eleven slots, and the rotated part (8 KB), two slots
//   warp 5       tcgen05.mma with the KEYS as rows and the heads as columns (N = 16): S^T = K Q^T, one tile ahead of the softmax.  M = 128 all the same: the rows behind the 64
//                keys are whatever lies there, and nobody reads their results
//   warp 6       O^T (128 latent columns at a time) += C^T P (N = 32) with the same staged rows as MN-major operand; nothing is padded to 128 heads
//   warps 0-3    thread = key (warps 0 and 1): 16 scores from TMEM, eight of them handed to warps 2 and 3; exp2 against a reference maximum per head that moves only when a
//                score passes it by 2^8 (then O^T's columns are scaled), P to shared memory; row sums stay per thread until the end of a share
//
// P goes in as two bf16 terms, the rounded weight and what it left, side by side as 32 columns: the product is bound by its 128 rows, and a reference
// that lags behind the maximum would otherwise have a row's largest weights rounded where 2^0 is exact (one term: 0.00453 from 64 bits on 64 rows of
// 2048-4096 tokens, the former kernel 0.00447).
//
// What bounds it: a tile's units come free when its products are done, and what is asked for then comes 1.8 us later; in between lie scores, softmax and products.  128-key tiles
// left 1.2 of them in the ring and took 6.6 us each (70 us in all).  64-key tiles alone gained nothing: small products cost their thread 40-80 cycles each
// whatever their size, 52 a tile in one warp 2.2 us; two warps issue them in 1.6 us a tile, which is the memory's rate.  Queries are staged with all their loads in flight: one
// after the other they took 6 us a share.  Layer of the size above 110.0 -> 94.1 us, 128 sequences of 100-2000 tokens 122 -> 103, rank 256 82 -> 76; one sequence of 4096 (its
// 64 shares folded by four groups of threads) 57 -> 49.  Asking for tiles in L2 further
// ahead, whole rows at a time, made all of it slower (104).
#include "mix_common.cuh"
#include "tc_common.cuh"

namespace {

using namespace b200tc;

constexpr int KEYS = 64, NH = 16, UNITS = 11, ROTS = 2, THREADS = 224, SEQ_CAP = 1024, SHARES = 512;      // SHARES: most CTAs of a launch
constexpr uint32_t PIECE = KEYS * 128, UNIT = 2 * PIECE;              // [64 keys][64 columns]; two of them
constexpr uint32_t QPIECE = NH * 128;                                 // [16 heads][64 columns]
constexpr uint32_t OFF_ROT = UNITS * UNIT;                            // the rotated parts' ring
constexpr uint32_t OFF_Q = OFF_ROT + ROTS * PIECE;                    // up to 9 pieces
constexpr uint32_t OFF_P = OFF_Q + 9 * QPIECE;                        // a PPIECE for tiles of even number, one for the others
constexpr uint32_t PPIECE = 2 * QPIECE;                               // [16 heads: weights, 16 heads: what they left][64 keys]
constexpr uint32_t OFF_SC = OFF_P + 2 * PPIECE;                       // float4[2 tiles][2][64 keys]: scores of heads 8 to 15
constexpr uint32_t OFF_RED = OFF_SC + 2 * KEYS * 32;                     // float[4][16] per-warp maxima / sums, float[16] reference maxima, float[16] factors
constexpr uint32_t OFF_CUM = OFF_RED + 6 * NH * 4;                    // int[SEQ_CAP + 1] tiles before each sequence
constexpr uint32_t OFF_BAR = (OFF_CUM + (SEQ_CAP + 1) * 4 + 7) / 8 * 8;
constexpr uint32_t SMEM = OFF_BAR + 320;
// per unit, per rotated part, per tile of even and odd number (scores, P, products: two tiles are under way), queries
constexpr uint32_t B_FULL = 0, B_EMPTY = UNITS, B_RFULL = 2 * UNITS, B_REMPTY = B_RFULL + ROTS, B_S = B_REMPTY + ROTS, B_PV = B_S + 2, B_P = B_PV + 2, B_Q = B_P + 2, B_COUNT = B_Q + 1;
constexpr float THRESHOLD = 8.0f, LOG2E = 1.4426950408889634f;

struct LatentParams {
    const __nv_bfloat16* q_lat;                                       // [H, n, rank]
    const __nv_bfloat16* q_raw;
    int64_t q_tok_stride;
    int q_head_stride, q_rot_off;
    const int32_t* block_tables;
    int bt_stride, block_size, box_rows;
    const int32_t* ctx_lens;
    const float* sink;
    const float* cos_sin;
    int rope_dims, layout, n, H, rank, window;
    float scale_log2;
    float* part;                                                      // slot (CTA + sequence): [H][rank] results, then [H][2] (maximum, sum)
    int64_t slot;                                                     // floats per slot, a multiple of four (the results are read 16 bytes at a time)
    __nv_bfloat16* out;                                               // [H, n, rank]
    uint32_t* report;                                                 // host word for waits that gave up: results of such a launch are undefined
};

// Key tiles of a sequence: from the one that holds the first visible key.
__device__ __forceinline__ int first_tile(const LatentParams& p, int ctx) { return p.window > 0 && ctx > p.window ? (ctx - p.window) / KEYS : 0; }
__device__ __forceinline__ int tile_count(const LatentParams& p, int ctx) { return ctx > 0 ? (ctx + KEYS - 1) / KEYS - first_tile(p, ctx) : 0; }

// cum[s] = tiles of the sequences before s; returns all (one warp).
__device__ __forceinline__ int prefix_tiles(const LatentParams& p, int* cum, int lane) {
    int at = 0;
    for (int s0 = 0; s0 < p.n; s0 += 32) {
        const int s = s0 + lane, t = s < p.n ? tile_count(p, p.ctx_lens[s]) : 0;
        int inc = t;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += v;
        }
        if (s < p.n) cum[s] = at + inc - t;
        at += __shfl_sync(0xffffffffu, inc, 31);
    }
    if (lane == 0) cum[p.n] = at;
    return at;
}

// Whether v holds for any of the 128 softmax threads (a meeting of theirs).
__device__ __forceinline__ bool any_of_128(bool v) {
    int any;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %1, 0;\n\tbar.red.or.pred q, 2, 128, p;\n\tselp.b32 %0, 1, 0, q;\n\t}" : "=r"(any) : "r"((int)v) : "memory");
    return any != 0;
}
__device__ __forceinline__ int find_seq(const int* cum, int n, int tile) {       // the sequence that owns a tile
    int lo = 0, hi = n;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (cum[mid] <= tile) lo = mid;
        else hi = mid;
    }
    while (cum[lo + 1] == cum[lo]) ++lo;                              // cannot pass the end: the tile exists
    return lo;
}

__global__ void __launch_bounds__(THREADS, 1) latent_decode_kernel(const __grid_constant__ CUtensorMap tm, const __grid_constant__ LatentParams p) {
    extern __shared__ __align__(1024) uint8_t smem[];
    const uint32_t base = smem_u32(smem), bars = base + OFF_BAR, dead = bars + B_COUNT * 8 + 4;
    auto bar = [&](uint32_t i) { return bars + i * 8; };
    volatile uint32_t* words = reinterpret_cast<volatile uint32_t*>(smem + OFF_BAR + B_COUNT * 8);        // TMEM, dead, warps 0-3 leave
    int* cum = reinterpret_cast<int*>(smem + OFF_CUM);
    float* red = reinterpret_cast<float*>(smem + OFF_RED);
    float *m_ref = red + 4 * NH, *factor = m_ref + NH;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int pieces = p.rank / 64, pairs = p.rank / 128;
    if (tid == 0) {
        for (uint32_t i = 0; i < B_COUNT; ++i) mbar_init(bar(i), i >= B_P ? 128 : 1);
        mbar_fence_init();
        words[1] = words[2] = 0;
    }
    if (warp == 5) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(bars + B_COUNT * 8), "r"(256u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 128) asm volatile("prefetch.tensormap [%0];" ::"l"(&tm) : "memory");
    B200_PDL_TRIGGER();
    B200_PDL_WAIT();                                                  // a kernel in front may have written the lengths
    if (warp == 0) prefix_tiles(p, cum, lane);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = words[0], tmem_o = tmem + 32;               // S^T at 0 and 16, O^T block b at 32 + 32 b
    const int total = cum[p.n];
    const int t_begin = (int)((int64_t)total * blockIdx.x / gridDim.x), t_end = (int)((int64_t)total * (blockIdx.x + 1) / gridDim.x);

    if (warp < 4) {
        // ---- softmax, queries, partial results ----
        const uint32_t lanes = (uint32_t)(warp * 32) << 16;
        uint32_t g = 0;                                               // tiles so far
        bool alive = true;                                            // of this warp: no wait of its own gave up
        for (int t = t_begin; t < t_end;) {
            const int s = find_seq(cum, p.n, t), seg_end = min(t_end, cum[s + 1]), seg_begin = t, ctx = p.ctx_lens[s];
            const int tile0 = first_tile(p, ctx) - cum[s], lo = p.window > 0 ? ctx - p.window : 0;
            // queries -> shared memory as K-major operand: 16 head rows, pieces of 64 columns; rows past H are zero
            {
                const int c = tid % 8, h = tid / 8;                   // a thread's 16 bytes of every piece, all asked for at once
                const bool there = h < p.H;
                uint8_t* q0 = smem + OFF_Q + h * 128 + ((c ^ (h & 7)) << 4);
                const uint4* src = reinterpret_cast<const uint4*>(p.q_lat + ((int64_t)(there ? h : 0) * p.n + s) * p.rank) + c;
                uint4 v[8];
#pragma unroll
                for (int k = 0; k < 8; ++k) v[k] = there && k < pieces ? src[k * 8] : make_uint4(0, 0, 0, 0);
                uint4 rot = make_uint4(0, 0, 0, 0);
                if (there) {
                    const __nv_bfloat16* x = p.q_raw + s * p.q_tok_stride + (int64_t)h * p.q_head_stride + p.q_rot_off;
                    const float* cs = p.cos_sin + (int64_t)(ctx - 1) * p.rope_dims;
                    const int half = p.rope_dims / 2;
                    float f[8];
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        const int d = c * 8 + e;
                        if (d >= p.rope_dims) {
                            f[e] = __bfloat162float(x[d]);
                            continue;
                        }
                        const int m = p.layout ? (d < half ? d : d - half) : d >> 1;
                        const bool second = p.layout ? d >= half : (d & 1);
                        const float u = __bfloat162float(x[p.layout ? m : 2 * m]), w = __bfloat162float(x[p.layout ? m + half : 2 * m + 1]);
                        f[e] = second ? w * cs[m] + u * cs[half + m] : u * cs[m] - w * cs[half + m];
                    }
                    rot = pack8(f);
                }
#pragma unroll
                for (int k = 0; k < 8; ++k)
                    if (k < pieces) *reinterpret_cast<uint4*>(q0 + k * QPIECE) = v[k];
                *reinterpret_cast<uint4*>(q0 + pieces * QPIECE) = rot;
            }
            if (tid < NH) m_ref[tid] = -INFINITY;
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar(B_Q)) : "memory");
            asm volatile("bar.sync 1, 128;" ::: "memory");
            constexpr int HH = NH / 2;                                // heads of a thread's weights: warps 0 and 1 have the first ones, 2 and 3 the others
            const int h0 = warp < 2 ? 0 : HH, col = tid & (KEYS - 1);
            float l[HH];
#pragma unroll
            for (int h = 0; h < HH; ++h) l[h] = 0.f;
            for (; t < seg_end; ++t, ++g) {
                const int key = (t + tile0) * KEYS + col;
                float4* handed = reinterpret_cast<float4*>(smem + OFF_SC) + (g & 1) * 2 * KEYS + col;
                float sc[NH];
                if (warp < 2) {                                       // keys are TMEM lanes 0 to 63: theirs
                    alive = alive && bounded_wait(bar(B_S + (g & 1)), (g >> 1) & 1, dead, p.report);
                    tc_fence_after();
                    uint32_t r[NH];
                    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n\ttcgen05.wait::ld.sync.aligned;"
                                 : TC_R8(r, 0), TC_R8(r, 8)
                                 : "r"(tmem + lanes + (g & 1) * NH)
                                 : "memory");
                    const bool seen = key < ctx && key >= lo;
#pragma unroll
                    for (int h = 0; h < NH; ++h) sc[h] = seen ? __uint_as_float(r[h]) * p.scale_log2 : -INFINITY;
                    handed[0] = make_float4(sc[HH], sc[HH + 1], sc[HH + 2], sc[HH + 3]);
                    handed[KEYS] = make_float4(sc[HH + 4], sc[HH + 5], sc[HH + 6], sc[HH + 7]);
                } else {
#pragma unroll
                    for (int h = 0; h < NH; ++h) sc[h] = -INFINITY;
                }
                bool grow = !alive;
#pragma unroll
                for (int h = 0; h < NH; ++h) grow |= sc[h] > m_ref[h] + THRESHOLD;
                if (!alive) words[2] = 1;
                if (any_of_128(grow)) {
                    if (words[2]) goto leave;                         // all four warps or none: they meet at barriers
#pragma unroll
                    for (int h = 0; h < NH; ++h) {
                        const float m = warp_max(sc[h]);
                        if (lane == 0) red[warp * NH + h] = m;
                    }
                    asm volatile("bar.sync 1, 128;" ::: "memory");
                    if (tid < NH) {
                        const float m = fmaxf(fmaxf(red[tid], red[NH + tid]), fmaxf(red[2 * NH + tid], red[3 * NH + tid])), was = m_ref[tid];
                        const bool up = m > was + THRESHOLD;
                        factor[tid] = up ? fast_exp2(was - m) : 1.0f;
                        if (up) m_ref[tid] = m;
                    }
                    asm volatile("bar.sync 1, 128;" ::: "memory");
#pragma unroll
                    for (int h = 0; h < HH; ++h) l[h] *= factor[h0 + h];
                    if (t > seg_begin) {                              // O^T holds the share's tiles before this one once their products are done
                        alive = bounded_wait(bar(B_PV + ((g - 1) & 1)), ((g - 1) >> 1) & 1, dead, p.report);
                        tc_fence_after();
                        for (int b = 0; b < pairs; ++b) {
                            float r[2 * NH];
                            tmem_ld32(tmem_o + lanes + b * 2 * NH, r);
#pragma unroll
                            for (int h = 0; h < 2 * NH; ++h) r[h] *= factor[h % NH];
                            tmem_st32(tmem_o + lanes + b * 2 * NH, r);
                        }
                    }
                }
                if (warp >= 2) {
                    const float4 x = handed[0], y = handed[KEYS];
                    sc[0] = x.x, sc[1] = x.y, sc[2] = x.z, sc[3] = x.w, sc[4] = y.x, sc[5] = y.y, sc[6] = y.z, sc[7] = y.w;
                }
                if (g > 1) alive = alive && bounded_wait(bar(B_PV + (g & 1)), ((g - 2) >> 1) & 1, dead, p.report);          // P of two tiles ago has been read
                if (!alive) continue;                                 // leaves at the next meeting
                uint8_t* pp = smem + OFF_P + (g & 1) * PPIECE + h0 * 128 + (col & 7) * 2;
#pragma unroll
                for (int h = 0; h < HH; ++h) {
                    const float m = m_ref[h0 + h], pv = m == -INFINITY ? 0.f : fast_exp2(sc[h] - m);
                    l[h] += pv;
                    const __nv_bfloat16 hi = __float2bfloat16_rn(pv);
                    uint8_t* at = pp + h * 128 + (((col >> 3) ^ h) << 4);                // h0 + h and h: the same row of eight
                    *reinterpret_cast<__nv_bfloat16*>(at) = hi;
                    *reinterpret_cast<__nv_bfloat16*>(at + QPIECE) = __float2bfloat16_rn(pv - __bfloat162float(hi));
                }
                if (warp < 2 && key >= ctx) {                         // a row past the context may hold anything, and 0 * NaN would poison the sum
                    const uint32_t u0 = g * pairs;
                    for (int k = 0; k < pieces; ++k) {
                        uint8_t* x = smem + (u0 + (k >> 1)) % UNITS * UNIT + (k & 1) * PIECE + tid * 128;
#pragma unroll
                        for (int c = 0; c < 8; ++c) *reinterpret_cast<uint4*>(x + c * 16) = make_uint4(0, 0, 0, 0);
                    }
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                tc_fence_before();
                asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar(B_P + (g & 1))) : "memory");
            }
            // ---- this share's part of the sequence ----
            alive = alive && bounded_wait(bar(B_PV + ((g - 1) & 1)), ((g - 1) >> 1) & 1, dead, p.report);
            if (any_of_128(!alive)) goto leave;
            tc_fence_after();
            float* dst = p.part + (int64_t)(blockIdx.x + s) * p.slot;
            for (int b = 0; b < pairs; ++b) {
                float r[2 * NH];
                tmem_ld32(tmem_o + lanes + b * 2 * NH, r);
#pragma unroll
                for (int h = 0; h < NH; ++h)
                    if (h < p.H) dst[(int64_t)h * p.rank + b * 128 + tid] = r[h] + r[NH + h];
            }
            tc_fence_before();
#pragma unroll
            for (int h = 0; h < HH; ++h) {
                const float v = warp_sum(l[h]);
                if (lane == 0) red[(warp & 1) * NH + h0 + h] = v;
            }
            asm volatile("bar.sync 1, 128;" ::: "memory");
            if (tid < p.H) {
                dst[(int64_t)p.H * p.rank + 2 * tid] = m_ref[tid];
                dst[(int64_t)p.H * p.rank + 2 * tid + 1] = red[tid] + red[NH + tid];
            }
            asm volatile("bar.sync 1, 128;" ::: "memory");
        }
    } else if (warp == 4) {
        // ---- loads (the whole warp: a lane per page box) ----
        uint32_t u = 0, g = 0;
        const int boxes = KEYS / p.box_rows;
        for (int t = t_begin; t < t_end;) {
            const int s = find_seq(cum, p.n, t), seg_end = min(t_end, cum[s + 1]), ctx = p.ctx_lens[s], tile0 = first_tile(p, ctx) - cum[s];
            for (; t < seg_end; ++t, ++g) {
                int row = 0;
                if (lane < boxes) {
                    const int key = (t + tile0) * KEYS + lane * p.box_rows;
                    const int page = key < ctx ? p.block_tables[(int64_t)s * p.bt_stride + key / p.block_size] : -1;
                    row = page < 0 ? -p.box_rows : page * p.block_size + key % p.block_size;      // no page: outside the map, zeros
                }
                for (int k = 0; k < pairs; ++k, ++u) {
                    const uint32_t slot = u % UNITS;
                    if (!bounded_wait(bar(B_EMPTY + slot), ((u / UNITS) & 1) ^ 1, dead, p.report)) goto leave;
                    if (lane == 0) mbar_expect_tx(bar(B_FULL + slot), UNIT);
                    __syncwarp();
                    if (lane < boxes)
                        for (int h = 0; h < 2; ++h)
                            tma_load_2d(base + slot * UNIT + h * PIECE + lane * p.box_rows * 128, &tm, bar(B_FULL + slot), k * 128 + h * 64, row);
                    __syncwarp();
                }
                const uint32_t slot = g % ROTS;
                if (!bounded_wait(bar(B_REMPTY + slot), ((g / ROTS) & 1) ^ 1, dead, p.report)) goto leave;
                if (lane == 0) mbar_expect_tx(bar(B_RFULL + slot), PIECE);
                __syncwarp();
                if (lane < boxes) tma_load_2d(base + OFF_ROT + slot * PIECE + lane * p.box_rows * 128, &tm, bar(B_RFULL + slot), p.rank, row);
                __syncwarp();
            }
        }
    } else if (warp == 5) {
        // ---- scores: products of 128 rows, 64 keys and what lies behind them in shared memory, whose results nobody reads ----
        const bool leader = elect_one();
        constexpr uint32_t IDESC = make_idesc(128, NH, false);
        const uint64_t kd0 = make_desc(base, 16, 1024), qd0 = make_desc(base + OFF_Q, 16, 1024);
        uint32_t g = 0, u = 0, segs = 0;
        for (int t = t_begin; t < t_end; ++segs) {
            const int s = find_seq(cum, p.n, t), seg_end = min(t_end, cum[s + 1]);
            if (!bounded_wait(bar(B_Q), segs & 1, dead, p.report)) goto leave;
            for (; t < seg_end; ++t, ++g) {
                const uint32_t d = tmem + (g & 1) * NH;
                if (g > 1 && !bounded_wait(bar(B_P + (g & 1)), ((g - 2) >> 1) & 1, dead, p.report)) goto leave;           // scores of two tiles ago have been read
                for (int k = 0; k < pairs; ++k, ++u) {
                    const uint32_t slot = u % UNITS;
                    if (!bounded_wait(bar(B_FULL + slot), (u / UNITS) & 1, dead, p.report)) goto leave;
                    tc_fence_after();
                    if (leader) {
                        const uint64_t kd = kd0 + slot * (UNIT / 16), qd = qd0 + k * (2 * QPIECE / 16);
                        tc_mma(d, kd, qd, IDESC, k > 0);
#pragma unroll
                        for (int q = 1; q < 8; ++q) tc_mma(d, kd + (q >> 2) * (PIECE / 16) + (q & 3) * 2, qd + (q >> 2) * (QPIECE / 16) + (q & 3) * 2, IDESC, 1);
                    }
                }
                const uint32_t slot = g % ROTS;
                if (!bounded_wait(bar(B_RFULL + slot), (g / ROTS) & 1, dead, p.report)) goto leave;
                tc_fence_after();
                if (leader) {
                    const uint64_t kd = kd0 + (OFF_ROT + slot * PIECE) / 16, qd = qd0 + pairs * (2 * QPIECE / 16);
#pragma unroll
                    for (int q = 0; q < 4; ++q) tc_mma(d, kd + q * 2, qd + q * 2, IDESC, 1);
                    tc_commit(bar(B_REMPTY + slot));
                    tc_commit(bar(B_S + (g & 1)));
                }
            }
        }
    } else {
        // ---- weights times latents ----
        const bool leader = elect_one();
        constexpr uint32_t IDESC = make_idesc(128, 2 * NH, false) | (1u << 15);          // latents: MN-major
        const uint64_t vd0 = make_desc(base, PIECE, 1024), pd0 = make_desc(base + OFF_P, 16, 1024);
        uint32_t g = 0, u = 0;
        for (int t = t_begin; t < t_end;) {
            const int s = find_seq(cum, p.n, t), seg_end = min(t_end, cum[s + 1]), seg_begin = t;
            for (; t < seg_end; ++t, ++g) {
                if (!bounded_wait(bar(B_P + (g & 1)), (g >> 1) & 1, dead, p.report)) goto leave;
                tc_fence_after();
                const uint64_t pd = pd0 + (g & 1) * (PPIECE / 16);
                for (int b = 0; b < pairs; ++b, ++u) {
                    const uint32_t slot = u % UNITS, d = tmem_o + b * 2 * NH;
                    if (leader) {
                        const uint64_t vd = vd0 + slot * (UNIT / 16);
                        tc_mma(d, vd, pd, IDESC, t > seg_begin);
#pragma unroll
                        for (int q = 1; q < KEYS / 16; ++q) tc_mma(d, vd + q * (2048 / 16), pd + q * 2, IDESC, 1);
                        tc_commit(bar(B_EMPTY + slot));
                    }
                }
                if (leader) tc_commit(bar(B_PV + (g & 1)));
            }
        }
    }
leave:
    __syncwarp();
    if (words[1])                                                     // gave up: let copies that are still in flight land first
        for (int i = 0; i < 1000; ++i) __nanosleep(1000);
    tc_fence_before();
    __syncthreads();
    if (warp == 5) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(256u) : "memory");
}

// out[h, s, :] = sum over the shares that hold part of sequence s, in a fixed order; the sink counts once.  grid (n, H), a thread per four columns, GROUPS of 128 threads with every
// GROUPS-th share each.  The shares' factors are formed first, side by side, so that the sum's loads do not wait for one another (a long sequence alone has a share per CTA).
template <int GROUPS>
__global__ void __launch_bounds__(128 * GROUPS) latent_fold_kernel(const LatentParams p, int ctas) {
    B200_PDL_TRIGGER();
    __shared__ int cum[SEQ_CAP + 1];
    __shared__ float fac[SHARES], red[4];
    __shared__ float4 sums[GROUPS > 1 ? GROUPS - 1 : 1][128];
    const int s = blockIdx.x, h = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    B200_PDL_WAIT();
    if (tid < 32) prefix_tiles(p, cum, tid);
    __syncthreads();
    const int64_t total = cum[p.n];
    const int t0 = cum[s], t1 = cum[s + 1];
    if (t0 == t1) return;
    // CTA c owns tiles [total c / ctas, total (c + 1) / ctas): the owners of the first and the last tile
    const int c0 = (int)((((int64_t)t0 + 1) * ctas - 1) / total), n = (int)(((int64_t)t1 * ctas - 1) / total) - c0 + 1;
    const float* part = p.part + (c0 + s) * p.slot;
    const float* ml = part + (int64_t)p.H * p.rank + 2 * h;
    const float sink = p.sink ? p.sink[h] * LOG2E : -INFINITY;
    // with fewer tiles than CTAs some of them have no share: nothing was written to their slots
    auto owns = [&](int c) { return total * (c0 + c) / ctas < total * (c0 + c + 1) / ctas; };
    float M = sink, L = 0.f;
    if (warp < 4) {
        for (int c = tid; c < n; c += 128)
            if (owns(c)) M = fmaxf(M, ml[c * p.slot]);
        M = warp_max(M);
        if (lane == 0) red[warp] = M;
    }
    __syncthreads();
    M = fmaxf(fmaxf(red[0], red[1]), fmaxf(red[2], red[3]));
    __syncthreads();
    if (warp < 4) {
        for (int c = tid; c < n; c += 128) {
            const float m = owns(c) ? ml[c * p.slot] : -INFINITY, f = m == -INFINITY ? 0.f : fast_exp2(m - M);
            fac[c] = f;
            if (f > 0.f) L = fmaf(f, ml[c * p.slot + 1], L);
        }
        L = warp_sum(L);
        if (lane == 0) red[warp] = L;
    }
    __syncthreads();
    L = red[0] + red[1] + red[2] + red[3] + (p.sink ? fast_exp2(sink - M) : 0.f);
    const int col = (tid & 127) * 4, group = tid >> 7;
    const bool has = col < p.rank;
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
    if (has) {
#pragma unroll 8
        for (int c = group; c < n; c += GROUPS) {
            const float f = fac[c];
            if (f == 0.f) continue;
            const float4 v = *reinterpret_cast<const float4*>(part + c * p.slot + (int64_t)h * p.rank + col);
            a.x = fmaf(f, v.x, a.x);
            a.y = fmaf(f, v.y, a.y);
            a.z = fmaf(f, v.z, a.z);
            a.w = fmaf(f, v.w, a.w);
        }
    }
    if (GROUPS > 1) {
        if (group) sums[group - 1][tid & 127] = a;
        __syncthreads();
        if (group) return;
#pragma unroll
        for (int i = 0; i < GROUPS - 1; ++i) {
            const float4 v = sums[i][tid];
            a.x += v.x, a.y += v.y, a.z += v.z, a.w += v.w;
        }
    }
    if (!has) return;
    const float inv = L > 0.f ? 1.0f / L : 0.f;
    *reinterpret_cast<uint2*>(p.out + ((int64_t)h * p.n + s) * p.rank + col) = make_uint2(pack_bf16x2(a.x * inv, a.y * inv), pack_bf16x2(a.z * inv, a.w * inv));
}

// Floats of a slot.
int64_t slot_floats(int heads, int rank) { return ((int64_t)heads * (rank + 2) + 3) / 4 * 4; }

}  // namespace

extern "C" size_t b200m_latent_decode_workspace_bytes(int n, int num_heads, int rank) {
    int dev = 0, sms = 0;
    if (n <= 0 || num_heads <= 0 || rank <= 0 || cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
    return (size_t)(sms + n) * slot_floats(num_heads, rank) * sizeof(float);
}

extern "C" int b200m_latent_decode(const void* q_lat, const void* q_raw, int64_t q_tok_stride, int q_head_stride, int q_rot_off, const void* cache, const int32_t* block_tables,
                                   int bt_stride, int block_size, const int32_t* ctx_lens, const float* sink, const float* cos_sin, int rope_dims, void* out, int n,
                                   int num_heads, int rank, int rot_dim, float scale, int window, int layout, void* workspace, size_t workspace_bytes, void* stream) {
    if (!q_lat || !q_raw || !cache || !block_tables || !ctx_lens || !cos_sin || !out || !workspace || n < 0 || num_heads <= 0 || rank <= 0 || block_size <= 0) return B200_EINVAL;
    if (rope_dims < 0 || rope_dims > rot_dim || (rope_dims & 1)) return B200_EINVAL;
    const uintptr_t bases = reinterpret_cast<uintptr_t>(q_lat) | reinterpret_cast<uintptr_t>(cache) | reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(workspace);
    if (rot_dim != 64 || (rank != 256 && rank != 512) || num_heads > NH || n > SEQ_CAP || bases % 16 || scale <= 0.f ||
        !(block_size % 128 == 0 || (block_size >= 8 && 128 % block_size == 0)))
        return B200_EUNSUPPORTED;
    if (n == 0) return B200_OK;
    int dev = 0, sms = 0;
    B200_CUDA_CHECK((b200_ctx*)nullptr, cudaGetDevice(&dev));
    B200_CUDA_CHECK((b200_ctx*)nullptr, cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    if (sms > SHARES) sms = SHARES;
    if (workspace_bytes < (size_t)(sms + n) * slot_floats(num_heads, rank) * sizeof(float)) return B200_EWORKSPACE;
    CUtensorMap tm;
    const int box = block_size < KEYS ? block_size : KEYS;
    if (!make_map(&tm, cache, (uint64_t)(rank + rot_dim), (1ull << 31) - 1, (uint64_t)(rank + rot_dim), box)) return B200_EUNSUPPORTED;       // rows are named by page
    LatentParams p = {static_cast<const __nv_bfloat16*>(q_lat), static_cast<const __nv_bfloat16*>(q_raw), q_tok_stride, q_head_stride, q_rot_off, block_tables, bt_stride,
                      block_size, box, ctx_lens, sink, cos_sin, rope_dims, layout, n, num_heads, rank, window, scale * LOG2E, static_cast<float*>(workspace), slot_floats(num_heads, rank),
                      static_cast<__nv_bfloat16*>(out), nullptr};
    if (const int rc = b200wait::launch_word(&p.report); rc != B200_OK) return rc;
    static B200SmemOptIn opt;
    B200_CUDA_CHECK((b200_ctx*)nullptr, opt.ensure(latent_decode_kernel, SMEM));
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    B200_LAUNCH((latent_decode_kernel), dim3(sms), THREADS, SMEM, st, tm, p);
    // Few sequences have many shares each: one of 4096 tokens 64 of them
    if (n <= 16) B200_LAUNCH((latent_fold_kernel<4>), dim3(n, num_heads), 512, 0, st, p, sms);
    else B200_LAUNCH((latent_fold_kernel<1>), dim3(n, num_heads), 128, 0, st, p, sms);
    return b200_launch_status(nullptr);
}
