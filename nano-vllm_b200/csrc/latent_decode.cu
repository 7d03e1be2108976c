// Latent attention of single-token steps on the 5th-generation tensor cores (bf16, up to 16 heads, latents of 256 or 512 columns beside a rotated
// key part of 64; latent_attn.cu has the definition and the general forms).
//
// Every cached row is read once for all heads, so the step is HBM-bound (226 MB for 64 sequences of 3072 tokens at rank 512: 35 us); what matters
// is to keep loads in flight.  One CTA per SM takes an equal share of the step's 128-key tiles, whatever the lengths (a share may begin and end
// inside a sequence; each (CTA, sequence) leaves an unnormalised partial that latent_fold_kernel sums in a fixed order).  Roles (192 threads):
//
//   warp 4       TMA: a tile as units of 128 columns (two swizzled [128 keys][64] pieces, 32 KB) and the rotated part (16 KB), six slots in flight
//   warp 5       tcgen05.mma with the KEYS as rows (M = 128) and the heads as columns (N = 16): S^T = K Q^T, then O^T (128 latent columns at a time)
//                += C^T P (N = 32) with the same staged rows as MN-major operand; both results are a few TMEM columns, so nothing is padded to 128 heads
//   warps 0-3    thread = key: 16 scores from TMEM, exp2 against a reference maximum per head that moves only when a score passes it by 2^8 (then
//                O^T's columns are scaled), P to shared memory; row sums stay per thread until the end of a share
//
// P goes in as two bf16 terms, the rounded weight and what it left, side by side as 32 columns: the product is bound by its 128 rows, and a reference
// that lags behind the maximum would otherwise have a row's largest weights rounded where 2^0 is exact (one term: 0.00453 from 64 bits on 64 rows of
// 2048-4096 tokens, the former kernel 0.00447).
//
// The mma.sync form this replaces for these sizes staged 64-key tiles with one tile in flight and read every row twice (output columns in two halves):
// 224 us + 14 us merge at the size above.
#include "mix_common.cuh"
#include "tc_common.cuh"

namespace {

using namespace b200tc;

constexpr int KEYS = 128, NH = 16, UNITS = 6, THREADS = 192, SEQ_CAP = 1024, SHARES = 512;      // SHARES: most CTAs of a launch
constexpr uint32_t PIECE = KEYS * 128, UNIT = 2 * PIECE;              // [128 keys][64 columns]
constexpr uint32_t QPIECE = NH * 128;                                 // [16 heads][64 columns]
constexpr uint32_t OFF_Q = UNITS * UNIT;                              // up to 9 pieces
constexpr uint32_t OFF_P = OFF_Q + 9 * QPIECE;                        // two PPIECEs
constexpr uint32_t PPIECE = 2 * QPIECE;                               // [16 heads: weights, 16 heads: what they left][64 keys]
constexpr uint32_t OFF_RED = OFF_P + 2 * PPIECE;                      // float[4][16] per-warp maxima / sums, float[16] reference maxima, float[16] factors
constexpr uint32_t OFF_CUM = OFF_RED + 6 * NH * 4;                    // int[SEQ_CAP + 1] tiles before each sequence
constexpr uint32_t OFF_BAR = (OFF_CUM + (SEQ_CAP + 1) * 4 + 7) / 8 * 8;
constexpr uint32_t SMEM = OFF_BAR + 192;
constexpr uint32_t B_FULL = 0, B_EMPTY = UNITS, B_S = 2 * UNITS, B_PV = B_S + 1, B_P = B_PV + 1, B_Q = B_P + 1, B_COUNT = B_Q + 1;
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
    const int pieces = p.rank / 64, pairs = p.rank / 128, units = pairs + 1;
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
    const uint32_t tmem = words[0], tmem_o = tmem + 32;               // S^T at 0, O^T block b at 32 + 32 b
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
            for (int i = tid; i < NH * (pieces + 1) * 8; i += 128) {
                const int c = i % 8, h = i / 8 % NH, k = i / (8 * NH);
                uint4 v = make_uint4(0, 0, 0, 0);
                if (h < p.H) {
                    if (k < pieces) {
                        v = *reinterpret_cast<const uint4*>(p.q_lat + ((int64_t)h * p.n + s) * p.rank + k * 64 + c * 8);
                    } else {
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
                        v = pack8(f);
                    }
                }
                *reinterpret_cast<uint4*>(smem + OFF_Q + k * QPIECE + h * 128 + ((c ^ (h & 7)) << 4)) = v;
            }
            if (tid < NH) m_ref[tid] = -INFINITY;
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar(B_Q)) : "memory");
            asm volatile("bar.sync 1, 128;" ::: "memory");
            float l[NH];
#pragma unroll
            for (int h = 0; h < NH; ++h) l[h] = 0.f;
            for (; t < seg_end; ++t, ++g) {
                const int key = (t + tile0) * KEYS + tid;
                alive = alive && bounded_wait(bar(B_S), g & 1, dead, p.report);
                tc_fence_after();
                float sc[NH];
                {
                    uint32_t r[NH];
                    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n\ttcgen05.wait::ld.sync.aligned;"
                                 : TC_R8(r, 0), TC_R8(r, 8)
                                 : "r"(tmem + lanes)
                                 : "memory");
                    const bool seen = key < ctx && key >= lo;
#pragma unroll
                    for (int h = 0; h < NH; ++h) sc[h] = seen ? __uint_as_float(r[h]) * p.scale_log2 : -INFINITY;
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
                    for (int h = 0; h < NH; ++h) l[h] *= factor[h];
                    if (t > seg_begin) {                              // O^T holds the share's tiles before this one once their products are done
                        alive = bounded_wait(bar(B_PV), (g - 1) & 1, dead, p.report);
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
                if (g > 0) alive = alive && bounded_wait(bar(B_PV), (g - 1) & 1, dead, p.report);          // P has been read
                if (!alive) continue;                                 // leaves at the next meeting
                uint8_t* pp = smem + OFF_P + (tid >> 6) * PPIECE + (tid & 7) * 2;
#pragma unroll
                for (int h = 0; h < NH; ++h) {
                    const float pv = m_ref[h] == -INFINITY ? 0.f : fast_exp2(sc[h] - m_ref[h]);
                    l[h] += pv;
                    const __nv_bfloat16 hi = __float2bfloat16_rn(pv);
                    uint8_t* at = pp + h * 128 + ((((tid & 63) >> 3) ^ (h & 7)) << 4);
                    *reinterpret_cast<__nv_bfloat16*>(at) = hi;
                    *reinterpret_cast<__nv_bfloat16*>(at + QPIECE) = __float2bfloat16_rn(pv - __bfloat162float(hi));
                }
                if (key >= ctx) {                                     // a row past the context may hold anything, and 0 * NaN would poison the sum
                    const uint32_t u0 = g * units;
                    for (int k = 0; k < pieces; ++k) {
                        uint8_t* x = smem + (u0 + (k >> 1)) % UNITS * UNIT + (k & 1) * PIECE + tid * 128;
#pragma unroll
                        for (int c = 0; c < 8; ++c) *reinterpret_cast<uint4*>(x + c * 16) = make_uint4(0, 0, 0, 0);
                    }
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                tc_fence_before();
                asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar(B_P)) : "memory");
            }
            // ---- this share's part of the sequence ----
            alive = alive && bounded_wait(bar(B_PV), (g - 1) & 1, dead, p.report);
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
            for (int h = 0; h < NH; ++h) {
                const float v = warp_sum(l[h]);
                if (lane == 0) red[warp * NH + h] = v;
            }
            asm volatile("bar.sync 1, 128;" ::: "memory");
            if (tid < p.H) {
                dst[(int64_t)p.H * p.rank + 2 * tid] = m_ref[tid];
                dst[(int64_t)p.H * p.rank + 2 * tid + 1] = red[tid] + red[NH + tid] + red[2 * NH + tid] + red[3 * NH + tid];
            }
            asm volatile("bar.sync 1, 128;" ::: "memory");
        }
    } else if (warp == 4) {
        // ---- loads (the whole warp: a lane per page box) ----
        uint32_t u = 0;
        const int boxes = KEYS / p.box_rows;
        for (int t = t_begin; t < t_end;) {
            const int s = find_seq(cum, p.n, t), seg_end = min(t_end, cum[s + 1]), ctx = p.ctx_lens[s], tile0 = first_tile(p, ctx) - cum[s];
            for (; t < seg_end; ++t) {
                int row = 0;
                if (lane < boxes) {
                    const int key = (t + tile0) * KEYS + lane * p.box_rows;
                    const int page = key < ctx ? p.block_tables[(int64_t)s * p.bt_stride + key / p.block_size] : -1;
                    row = page < 0 ? -p.box_rows : page * p.block_size + key % p.block_size;      // no page: outside the map, zeros
                }
                for (int k = 0; k < units; ++k, ++u) {
                    const uint32_t slot = u % UNITS;
                    if (!bounded_wait(bar(B_EMPTY + slot), ((u / UNITS) & 1) ^ 1, dead, p.report)) goto leave;
                    if (lane == 0) mbar_expect_tx(bar(B_FULL + slot), k < pairs ? UNIT : PIECE);
                    __syncwarp();
                    if (lane < boxes)
                        for (int h = 0; h < (k < pairs ? 2 : 1); ++h)
                            tma_load_2d(base + slot * UNIT + h * PIECE + lane * p.box_rows * 128, &tm, bar(B_FULL + slot), k * 128 + h * 64, row);
                    __syncwarp();
                }
            }
        }
    } else {
        // ---- products ----
        const bool leader = elect_one();
        constexpr uint32_t IDESC_S = make_idesc(KEYS, NH, false), IDESC_O = make_idesc(128, 2 * NH, false) | (1u << 15);      // A of the second: MN-major
        const uint64_t kd0 = make_desc(base, 16, 1024), qd0 = make_desc(base + OFF_Q, 16, 1024), vd0 = make_desc(base, PIECE, 1024), pd0 = make_desc(base + OFF_P, 16, 1024);
        uint32_t g = 0, u = 0, segs = 0;
        for (int t = t_begin; t < t_end; ++segs) {
            const int s = find_seq(cum, p.n, t), seg_end = min(t_end, cum[s + 1]), seg_begin = t;
            if (!bounded_wait(bar(B_Q), segs & 1, dead, p.report)) goto leave;
            for (; t < seg_end; ++t, ++g, u += units) {
                for (int k = 0; k < units; ++k) {
                    const uint32_t slot = (u + k) % UNITS;
                    if (!bounded_wait(bar(B_FULL + slot), ((u + k) / UNITS) & 1, dead, p.report)) goto leave;
                    tc_fence_after();
                    if (leader) {
                        const uint64_t kd = kd0 + slot * (UNIT / 16), qd = qd0 + k * (2 * QPIECE / 16);
#pragma unroll
                        for (int q = 0; q < 8; ++q) {
                            if (q >= 4 && k == pairs) break;
                            tc_mma(tmem, kd + (q >> 2) * (PIECE / 16) + (q & 3) * 2, qd + (q >> 2) * (QPIECE / 16) + (q & 3) * 2, IDESC_S, k > 0 || q > 0);
                        }
                        if (k == pairs) {
                            tc_commit(bar(B_EMPTY + slot));
                            tc_commit(bar(B_S));
                        }
                    }
                }
                if (!bounded_wait(bar(B_P), g & 1, dead, p.report)) goto leave;
                tc_fence_after();
                if (leader) {
                    for (int b = 0; b < pairs; ++b) {
                        const uint32_t slot = (u + b) % UNITS;
                        const uint64_t vd = vd0 + slot * (UNIT / 16);
#pragma unroll
                        for (int q = 0; q < KEYS / 16; ++q)
                            tc_mma(tmem_o + b * 2 * NH, vd + q * (2048 / 16), pd0 + (q >> 2) * (PPIECE / 16) + (q & 3) * 2, IDESC_O, t > seg_begin || q > 0);
                        tc_commit(bar(B_EMPTY + slot));
                    }
                    tc_commit(bar(B_PV));
                }
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

// out[h, s, :] = sum over the shares that hold part of sequence s, in their order; the sink counts once.  grid (n, H), a thread per four columns.  The
// shares' factors are formed first, side by side, so that the sum's loads do not wait for one another (a long sequence alone has a share per CTA).
__global__ void __launch_bounds__(128) latent_fold_kernel(const LatentParams p, int ctas) {
    B200_PDL_TRIGGER();
    __shared__ int cum[SEQ_CAP + 1];
    __shared__ float fac[SHARES], red[4];
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
    float M = sink;
    for (int c = tid; c < n; c += 128)
        if (owns(c)) M = fmaxf(M, ml[c * p.slot]);
    M = warp_max(M);
    if (lane == 0) red[warp] = M;
    __syncthreads();
    M = fmaxf(fmaxf(red[0], red[1]), fmaxf(red[2], red[3]));
    __syncthreads();
    float L = 0.f;
    for (int c = tid; c < n; c += 128) {
        const float m = owns(c) ? ml[c * p.slot] : -INFINITY, f = m == -INFINITY ? 0.f : fast_exp2(m - M);
        fac[c] = f;
        if (f > 0.f) L = fmaf(f, ml[c * p.slot + 1], L);
    }
    L = warp_sum(L);
    if (lane == 0) red[warp] = L;
    __syncthreads();
    L = red[0] + red[1] + red[2] + red[3] + (p.sink ? fast_exp2(sink - M) : 0.f);
    const int col = tid * 4;
    if (col >= p.rank) return;
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
    for (int c = 0; c < n; ++c) {
        const float f = fac[c];
        if (f == 0.f) continue;
        const float4 v = *reinterpret_cast<const float4*>(part + c * p.slot + (int64_t)h * p.rank + col);
        a.x = fmaf(f, v.x, a.x);
        a.y = fmaf(f, v.y, a.y);
        a.z = fmaf(f, v.z, a.z);
        a.w = fmaf(f, v.w, a.w);
    }
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
        !(block_size % KEYS == 0 || (block_size >= 8 && KEYS % block_size == 0)))
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
    B200_LAUNCH((latent_fold_kernel), dim3(n, num_heads), 128, 0, st, p, sms);
    return b200_launch_status(nullptr);
}
