// Grouped expert GEMMs on the 5th-generation tensor cores (bf16 operands, fp32 accumulation).
//
// The rows of each expert's run come in 64-row tiles (moe_align).  Two kernels share the work by how many rows an expert has:
//
//   moe_rows_kernel    many rows: persistent, one CTA per SM.  An item is up to two consecutive tiles of one expert (M = 128 rows) times
//                      256 rows of its weights (N = 256; with the gated activation 128 gate rows and the 128 matching up rows), K in
//                      stages of 64 through a 4-deep TMA ring, two accumulators in TMEM so that an item's results are written while the
//                      next one multiplies.
//                      Bound by the L2 -> shared-memory path: 48 KB per 2 M multiply-adds, 94 B per cycle and SM at the tensor cores' full
//                      rate.  128 x 256 tiles rather than 64 x 128 (the mma.sync form) halve that traffic.
//   moe_stream_kernel  few rows: HBM-bound, every weight is read once.  An item is 128 weight rows (M; gated: 64 gate + 64 up) times one tile of 64 rows (N).
//                      Two CTAs per SM walk the items with a ring each, so that the next item's weights are on their way while one's results are written; a CTA
//                      per item, three per SM, left a short second turn (512 items on 444 places) and its ramp-up.  Weights do not depend on the kernel in front: the
//                      first stages of them are asked for before it has ended (MoeParams.early).  Whole layer, us, before / after: 64 tokens 84.9 / 76.8, 256 90.4 / 82.1,
//                      gated 64 108.5 / 100.1, 200 116.0 / 106.4, of width 1024 1 token 45.5 / 43.3, 64 57.2 / 53.8.  More of them asked into L2 ahead of the ring made it slower (87).
//
// Both read grouped rows: the experts' inputs are gathered (and weighted) by a copy in front.  Gathering them inside, four rows per TMA
// gather instruction, took 383 us where the copy and the box loads take 23 + 158 (8192 tokens, width 2048, gate | up), and 89 us against 4.5 + 42 on 64 tokens.
// Padding rows (-1) hold anything and are never written: a result row depends on its own input row alone.
#include "mix_common.cuh"
#include "tc_common.cuh"

namespace {

using namespace b200tc;

constexpr int TILE = 64;                          // rows per tile of moe_align
constexpr uint32_t ROW_B = 128;                   // bytes of a staged row: 64 bf16

struct MoeParams {
    const int32_t* sorted_rows;                   // [max_tiles * 64] pair index or -1
    const int32_t* tile_expert;
    const int32_t* num_tiles;
    int max_tiles;
    int N, K, n_out, act;                         // weight rows per expert, output columns; act 0 none, 1 relu^2, 2 gated SiLU
    void* C;
    int out_f32;
    int early;                                    // few rows: the kernel in front lets this one begin only when all before itself has ended, so that what the
                                                  // grouping wrote may be read, and weights, before that kernel has ended
    uint32_t* report;                             // host word for waits that gave up: results of such a launch are undefined
};

__device__ __forceinline__ float moe_act1(float v) {
    v = fmaxf(v, 0.f);
    return v * v;
}

// ---- many rows -----------------------------------------------------------------------------------------------------------------
constexpr int R_STAGES = 4, R_THREADS = 192, R_TILES = 2048;      // warps 0-3 results, 4 loads, 5 products; most tiles of a launch
constexpr uint32_t R_A = 128 * ROW_B, R_W = 256 * ROW_B, R_STAGE = R_A + R_W;
constexpr uint32_t R_OFF_LIST = R_STAGES * R_STAGE;               // uint32[R_TILES]: tile expert, then first tile of each pair | two << 31
constexpr uint32_t R_OFF_BAR = R_OFF_LIST + R_TILES * 4;          // full[S], empty[S], acc_full[2], acc_empty[2], TMEM slot, dead, pairs
constexpr uint32_t R_SMEM = R_OFF_BAR + 128;

__global__ void __launch_bounds__(R_THREADS, 1) moe_rows_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_w, const MoeParams p) {
    extern __shared__ __align__(1024) uint8_t smem[];
    const uint32_t base = smem_u32(smem), bars = base + R_OFF_BAR;
    const uint32_t full = bars, empty = bars + R_STAGES * 8, acc_full = empty + R_STAGES * 8, acc_empty = acc_full + 16, slot = acc_empty + 16, dead = slot + 4;
    volatile uint32_t* words = reinterpret_cast<volatile uint32_t*>(smem + R_OFF_BAR + R_STAGES * 16 + 32);      // TMEM, dead, pairs
    uint32_t* list = reinterpret_cast<uint32_t*>(smem + R_OFF_LIST);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        for (int i = 0; i < 2 * R_STAGES + 2; ++i) mbar_init(bars + i * 8, 1);
        for (int i = 0; i < 2; ++i) mbar_init(acc_empty + i * 8, 128);
        mbar_fence_init();
        words[1] = 0;
    }
    if (warp == 5) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    B200_PDL_SYNC();
    const int tiles = min(p.num_tiles[0], p.max_tiles);
    for (int i = tid; i < tiles; i += R_THREADS) list[i] = (uint32_t)p.tile_expert[i];
    __syncthreads();
    if (warp == 0) {                              // pairs of tiles, in place: an entry lands at or before the tile it starts at
        uint32_t before = 0xffffffffu, begin = 0, count = 0;             // expert of the tile before this chunk, first tile of its run, pairs so far
        for (int c = 0; c < tiles; c += 32) {
            const int i = c + lane;
            const uint32_t e = i < tiles ? list[i] : 0xfffffffeu;
            uint32_t prev = __shfl_up_sync(0xffffffffu, e, 1), next = __shfl_down_sync(0xffffffffu, e, 1);
            if (lane == 0) prev = before;
            if (lane == 31) next = i + 1 < tiles ? list[i + 1] : 0xfffffffeu;
            const uint32_t firsts = __ballot_sync(0xffffffffu, e != prev) & (0xffffffffu >> (31 - lane));
            const uint32_t run = firsts ? c + 31 - __clz(firsts) : begin;
            const bool start = i < tiles && ((i - run) & 1) == 0;
            const uint32_t starts = __ballot_sync(0xffffffffu, start);
            __syncwarp();
            if (start) list[count + __popc(starts & ((1u << lane) - 1))] = (uint32_t)i | (next == e ? 1u << 31 : 0u);
            before = __shfl_sync(0xffffffffu, e, 31);
            begin = __shfl_sync(0xffffffffu, run, 31);
            count += __popc(starts);
            __syncwarp();
        }
        if (lane == 0) words[2] = count;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = words[0];
    const bool gated = p.act == 2;
    const int half = p.N >> 1, cols = gated ? 128 : 256;                 // output columns of an item
    const int nblk = p.n_out / cols, items = (int)words[2] * nblk, ksteps = (p.K + 63) / 64;

    if (warp < 4) {
        // ---- results: a thread per row ----
        uint32_t n = 0;
        for (int i = blockIdx.x; i < items; i += gridDim.x, ++n) {
            const uint32_t ent = list[i / nblk], b = n & 1;
            const int c0 = i % nblk * cols;
            const int64_t row = (int64_t)(ent & 0x7fffffffu) * TILE + tid;
            const int pair = tid < TILE || (ent >> 31) ? p.sorted_rows[row] : -1;
            if (!bounded_wait(acc_full + b * 8, (n >> 1) & 1, dead, p.report)) goto leave;
            tc_fence_after();
            const uint32_t acc = tmem + b * 256 + ((uint32_t)(warp * 32) << 16);
#pragma unroll 1
            for (int c = 0; c < cols; c += 32) {
                __syncwarp();
                float v[32];
                tmem_ld32(acc + c, v);
                if (gated) {
                    float u[32];
                    tmem_ld32(acc + 128 + c, u);
#pragma unroll
                    for (int k = 0; k < 32; ++k) v[k] = siluf_(v[k]) * u[k];
                } else {
#pragma unroll
                    for (int k = 0; k < 32; ++k) v[k] = p.act == 1 ? moe_act1(v[k]) : v[k];
                }
                if (pair < 0) continue;
                if (p.out_f32) {
                    float* d = static_cast<float*>(p.C) + row * p.n_out + c0 + c;
#pragma unroll
                    for (int k = 0; k < 4; ++k) st_256(d + k * 8, reinterpret_cast<const uint32_t*>(v) + k * 8);
                } else {
                    uint32_t pk[16];
#pragma unroll
                    for (int k = 0; k < 16; ++k) pk[k] = pack_bf16x2(v[2 * k], v[2 * k + 1]);
                    __nv_bfloat16* d = static_cast<__nv_bfloat16*>(p.C) + row * p.n_out + c0 + c;
                    st_256(d, pk);
                    st_256(d + 16, pk + 8);
                }
            }
            tc_fence_before();
            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(acc_empty + b * 8) : "memory");
        }
    } else if (warp == 4) {
        // ---- loads ----
        uint32_t s = 0, ph = 1;
        for (int i = blockIdx.x; i < items; i += gridDim.x) {
            const int tile = list[i / nblk] & 0x7fffffffu, w0 = p.tile_expert[tile] * p.N + i % nblk * cols;
            for (int k = 0; k < ksteps; ++k) {
                if (!bounded_wait(empty + s * 8, ph, dead, p.report)) goto leave;
                if (lane == 0) {
                    const uint32_t dst = base + s * R_STAGE, bar = full + s * 8;
                    mbar_expect_tx(bar, R_STAGE);
                    tma_load_2d(dst, &tm_a, bar, k * 64, tile * TILE);
                    tma_load_2d(dst + R_A, &tm_w, bar, k * 64, w0);
                    tma_load_2d(dst + R_A + R_W / 2, &tm_w, bar, k * 64, w0 + (gated ? half : 128));
                }
                if (++s == R_STAGES) {
                    s = 0;
                    ph ^= 1;
                }
            }
        }
    } else {
        // ---- products ----
        const bool leader = elect_one();
        const uint64_t ad0 = make_desc(base, 16, 1024), wd0 = make_desc(base + R_A, 16, 1024);
        constexpr uint32_t IDESC = make_idesc(128, 256, false);
        uint32_t s = 0, ph = 0, n = 0;
        for (int i = blockIdx.x; i < items; i += gridDim.x, ++n) {
            const uint32_t b = n & 1;
            if (!bounded_wait(acc_empty + b * 8, ((n >> 1) & 1) ^ 1, dead, p.report)) goto leave;
            tc_fence_after();
            for (int k = 0; k < ksteps; ++k) {
                if (!bounded_wait(full + s * 8, ph, dead, p.report)) goto leave;
                tc_fence_after();
                if (leader) {
                    const uint64_t ad = ad0 + s * (R_STAGE / 16), wd = wd0 + s * (R_STAGE / 16);
#pragma unroll
                    for (int q = 0; q < 4; ++q) tc_mma(tmem + b * 256, ad + q * 2, wd + q * 2, IDESC, k > 0 || q > 0);
                    tc_commit(empty + s * 8);
                    if (k + 1 == ksteps) tc_commit(acc_full + b * 8);
                }
                if (++s == R_STAGES) {
                    s = 0;
                    ph ^= 1;
                }
            }
        }
    }
leave:
    __syncwarp();
    if (words[1])                                 // gave up: let copies that are still in flight land first
        for (int i = 0; i < 1000; ++i) __nanosleep(1000);
    tc_fence_before();
    __syncthreads();
    if (warp == 5) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
}

// ---- few rows ------------------------------------------------------------------------------------------------------------------
constexpr int S_STAGES = 4, S_THREADS = 192;      // warps 0-3 results, 4 loads, 5 products
constexpr uint32_t S_W = 128 * ROW_B, S_T = TILE * ROW_B, S_STAGE = S_W + S_T;
constexpr uint32_t S_OFF_BAR = S_STAGES * S_STAGE;                // full[S], empty[S], acc_full[2], acc_empty[2], TMEM, dead
constexpr uint32_t S_OFF_SRC = S_OFF_BAR + 128;                   // int[2][64] pair of each row
constexpr uint32_t S_OFF_SWAP = S_OFF_SRC + 2 * TILE * 4;         // gated: float[2][64 rows of W][16 + 1 rows], halves that change hands
constexpr uint32_t S_SMEM = S_OFF_SWAP + 2 * 64 * 17 * 4;         // 105 KB: two CTAs per SM

__global__ void __launch_bounds__(S_THREADS, 2) moe_stream_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_w, const MoeParams p) {
    extern __shared__ __align__(1024) uint8_t smem[];
    const uint32_t base = smem_u32(smem), full = base + S_OFF_BAR, empty = full + S_STAGES * 8, acc_full = empty + S_STAGES * 8, acc_empty = acc_full + 16, slot = acc_empty + 16, dead = slot + 4;
    volatile uint32_t* words = reinterpret_cast<volatile uint32_t*>(smem + S_OFF_BAR + S_STAGES * 16 + 32);      // TMEM, dead
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (!p.early) B200_PDL_WAIT();
    const bool gated = p.act == 2;
    const int half = p.N >> 1, cols = gated ? 64 : 128, nblk = p.n_out / cols, ksteps = (p.K + 63) / 64;
    const int items = min(p.num_tiles[0], p.max_tiles) * nblk;
    if ((int)blockIdx.x >= items) {               // this grid ends behind the kernel in front also where no CTA has an item (no token with an expert of its own)
        if (p.early) B200_PDL_WAIT();
        return;
    }
    if (tid == 0) {
        for (int i = 0; i < 2 * S_STAGES + 2; ++i) mbar_init(full + i * 8, 1);
        for (int i = 0; i < 2; ++i) mbar_init(acc_empty + i * 8, 128);
        mbar_fence_init();
        words[1] = 0;
    }
    if (warp == 5) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot), "r"(128u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = words[0];
    if (warp == 4) {
        // ---- loads ----
        const int steps = ((items - 1 - (int)blockIdx.x) / (int)gridDim.x + 1) * ksteps, begun = min(S_STAGES, steps);
        auto row_of = [&](int i) { return p.tile_expert[i / nblk] * p.N + i % nblk * cols; };
        auto weights = [&](int w0, int k, int s) {
            const uint32_t dst = base + s * S_STAGE, bar = full + s * 8;
            mbar_expect_tx(bar, S_STAGE);
            tma_load_2d(dst, &tm_w, bar, k * 64, w0);
            tma_load_2d(dst + S_W / 2, &tm_w, bar, k * 64, w0 + (gated ? half : 64));
        };
        if (lane == 0) {
            int w0 = 0;
            for (int q = 0, i = blockIdx.x, k = 0; q < begun; ++q) {
                if (k == 0) w0 = row_of(i);
                weights(w0, k, q);
                if (++k == ksteps) {
                    k = 0;
                    i += gridDim.x;
                }
            }
        }
        __syncwarp();
        if (p.early) B200_PDL_WAIT();
        B200_PDL_TRIGGER();                       // all that this kernel waited for has ended: the next one may count on it
        uint32_t s = 0, ph = 1;
        for (int i = blockIdx.x, q = 0; i < items; i += gridDim.x) {
            const int w0 = row_of(i), row = i / nblk * TILE;
            for (int k = 0; k < ksteps; ++k, ++q) {
                if (!bounded_wait(empty + s * 8, ph, dead, p.report)) goto leave;
                if (lane == 0) {
                    if (q >= begun) weights(w0, k, s);
                    tma_load_2d(base + s * S_STAGE + S_W, &tm_a, full + s * 8, k * 64, row);
                }
                if (++s == S_STAGES) {
                    s = 0;
                    ph ^= 1;
                }
            }
        }
    } else if (warp == 5) {
        // ---- products ----
        if (p.early) B200_PDL_WAIT();
        B200_PDL_TRIGGER();
        const bool leader = elect_one();
        const uint64_t wd0 = make_desc(base, 16, 1024), td0 = make_desc(base + S_W, 16, 1024);
        constexpr uint32_t IDESC = make_idesc(128, TILE, false);
        uint32_t s = 0, ph = 0, n = 0;
        for (int i = blockIdx.x; i < items; i += gridDim.x, ++n) {
            const uint32_t b = n & 1;
            if (!bounded_wait(acc_empty + b * 8, ((n >> 1) & 1) ^ 1, dead, p.report)) goto leave;
            tc_fence_after();
            for (int k = 0; k < ksteps; ++k) {
                if (!bounded_wait(full + s * 8, ph, dead, p.report)) goto leave;
                tc_fence_after();
                if (leader) {
                    const uint64_t wd = wd0 + s * (S_STAGE / 16), td = td0 + s * (S_STAGE / 16);
#pragma unroll
                    for (int q = 0; q < 4; ++q) tc_mma(tmem + b * TILE, wd + q * 2, td + q * 2, IDESC, k > 0 || q > 0);
                    tc_commit(empty + s * 8);
                    if (k + 1 == ksteps) tc_commit(acc_full + b * 8);
                }
                if (++s == S_STAGES) {
                    s = 0;
                    ph ^= 1;
                }
            }
        }
    } else {
        // ---- results: a thread per row of W, an output column ----
        if (p.early) B200_PDL_WAIT();
        B200_PDL_TRIGGER();
        float* swap = reinterpret_cast<float*>(smem + S_OFF_SWAP);
        uint32_t n = 0;
        for (int i = blockIdx.x; i < items; i += gridDim.x, ++n) {
            const uint32_t b = n & 1;
            const int tile = i / nblk, col = i % nblk * cols + (gated ? tid & 63 : tid);
            int* src = reinterpret_cast<int*>(smem + S_OFF_SRC) + b * TILE;
            if (tid < TILE) src[tid] = p.sorted_rows[tile * TILE + tid];
            const bool ok = bounded_wait(acc_full + b * 8, (n >> 1) & 1, dead, p.report);
            int all;                              // whether all four warps go on, and their rows' pairs are there
            asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %1, 0;\n\tbar.red.and.pred q, 1, 128, p;\n\tselp.b32 %0, 1, 0, q;\n\t}" : "=r"(all) : "r"((int)ok) : "memory");
            if (!all) goto leave;
            tc_fence_after();
            const uint32_t acc = tmem + b * TILE + ((uint32_t)(warp * 32) << 16);
#pragma unroll 1
            for (int h = 0; h < 2; ++h) {
                __syncwarp();
                float v[32];
                tmem_ld32(acc + h * 32, v);
                auto put = [&](int k, float x) {
                    const int r = h * 32 + k;
                    if (src[r] < 0) return;
                    const int64_t at = ((int64_t)tile * TILE + r) * p.n_out + col;
                    if (p.out_f32) static_cast<float*>(p.C)[at] = x;
                    else static_cast<__nv_bfloat16*>(p.C)[at] = __float2bfloat16_rn(x);
                };
                if (!gated) {
#pragma unroll
                    for (int k = 0; k < 32; ++k) put(k, p.act == 1 ? moe_act1(v[k]) : v[k]);
                    continue;
                }
                // rows 64 to 127 are the up half: warps 0 and 1 get it of 16 rows and hand over the gate half of the other 16 to warps 2 and 3
                const bool low = warp < 2;
                float *mine = swap + (low ? 64 * 17 : 0) + (tid & 63) * 17, *theirs = swap + (low ? 0 : 64 * 17) + (tid & 63) * 17;
#pragma unroll
                for (int k = 0; k < 16; ++k) mine[k] = low ? v[16 + k] : v[k];
                asm volatile("bar.sync 1, 128;" ::: "memory");
#pragma unroll
                for (int k = 0; k < 16; ++k) {
                    const int at = low ? k : 16 + k;
                    if (src[h * 32 + at] < 0) continue;       // no activation for rows without a pair, of a few tokens most of a tile's (width 1024, 1 token: 48.2 us the layer with it)
                    const float other = theirs[k];
                    put(at, siluf_(low ? v[k] : other) * (low ? other : v[16 + k]));
                }
                asm volatile("bar.sync 1, 128;" ::: "memory");
            }
            tc_fence_before();
            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(acc_empty + b * 8) : "memory");
        }
    }
leave:
    __syncwarp();
    if (words[1])                                 // gave up: let copies that are still in flight land first
        for (int i = 0; i < 1000; ++i) __nanosleep(1000);
    tc_fence_before();
    __syncthreads();
    if (warp == 5) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(128u) : "memory");
}

// The experts' inputs in grouped order: out[i] = A[pair / top] (times wgt[pair], rounded) for every grouped row i with a pair.  A warp per row.
__global__ void __launch_bounds__(256) moe_gather_kernel(const __nv_bfloat16* __restrict__ A, int64_t a_stride, const int32_t* __restrict__ sorted_rows,
                                                         const float* __restrict__ wgt, int top, const int32_t* __restrict__ num_tiles, int rows, int pieces,
                                                         __nv_bfloat16* __restrict__ out) {
    B200_PDL_WAIT();                              // first this: who begins early behind this kernel reads what the one in front of it has written
    B200_PDL_TRIGGER();
    const int i = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (i >= rows || i >= num_tiles[0] * TILE) return;
    const int pair = sorted_rows[i];
    if (pair < 0) return;
    const uint4* src = reinterpret_cast<const uint4*>(A + (int64_t)(pair / top) * a_stride);
    uint4* dst = reinterpret_cast<uint4*>(out) + (int64_t)i * pieces;
    const float w = wgt ? wgt[pair] : 1.0f;
#pragma unroll 4
    for (int c = lane; c < pieces; c += 32) {
        uint4 v = src[c];
        if (wgt) {
            float f[8];
            unpack8(v, f);
#pragma unroll
            for (int k = 0; k < 8; ++k) f[k] *= w;
            v = pack8(f);
        }
        dst[c] = v;
    }
}

}  // namespace

extern "C" int b200m_moe_gather(const void* A, int64_t a_stride, const int32_t* sorted_rows, const float* wgt, int top, const int32_t* num_tiles, int max_tiles, int K,
                                void* out, void* stream) {
    if (!A || !sorted_rows || !num_tiles || !out || top <= 0 || max_tiles < 0 || K <= 0) return B200_EINVAL;
    if (K % 8 || a_stride % 8 || (reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(out)) % 16) return B200_EUNSUPPORTED;
    if (max_tiles == 0) return B200_OK;
    B200_LAUNCH((moe_gather_kernel), dim3(max_tiles * (TILE / 8)), 256, 0, static_cast<cudaStream_t>(stream), static_cast<const __nv_bfloat16*>(A), a_stride, sorted_rows,
                wgt, top, num_tiles, max_tiles * TILE, K / 8, static_cast<__nv_bfloat16*>(out));
    return b200_launch_status(nullptr);
}

// Called from b200m_moe_gemm, which has validated the arguments (bf16).  rows_per_expert: about how many rows an expert has; 0: not
// known, and A may be shorter than its tiles.  early: see MoeParams.  B200_EUNSUPPORTED: that, and shapes these kernels do not tile (in particular a last block of weight rows that would reach into the next expert's, or
// past the last one's).
int b200m_moe_gemm_tc(const void* A, int64_t a_stride, const int32_t* sorted_rows, const int32_t* tile_expert, const int32_t* num_tiles, int max_tiles, const void* W, int N, int K,
                      void* C, int out_f32, int act, int rows_per_expert, int early, cudaStream_t stream) {
    constexpr uint64_t ANY_ROWS = (1ull << 31) - 1;              // weight rows are named by expert: whole blocks of existing ones
    // Above STREAM_ROWS rows an expert is two or more tiles, whose weights the streaming kernel reads once per tile.  Measured (width 2048, 32 experts,
    // whole layer, us, streaming / many rows): 32 rows 128 / 135, 70 rows 193 / 200 (gated), 87 rows 179 / 154, 102 rows 257 / 234 (gated).
    constexpr int STREAM_ROWS = 64;
    const bool stream_form = rows_per_expert <= STREAM_ROWS;
    const int n_out = act == 2 ? N / 2 : N, cols = (act == 2 ? 64 : 128) * (stream_form ? 1 : 2);
    const uintptr_t bases = reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(W);
    if (rows_per_expert <= 0 || K % 8 || a_stride % 8 || bases % 16 || reinterpret_cast<uintptr_t>(C) % 32 || n_out % cols || max_tiles > (stream_form ? 65535 : R_TILES)) return B200_EUNSUPPORTED;
    MoeParams p = {sorted_rows, tile_expert, num_tiles, max_tiles, N, K, n_out, act, C, out_f32, early, nullptr};
    if (const int rc = b200wait::launch_word(&p.report); rc != B200_OK) return rc;
    CUtensorMap ta, tw;
    if (!make_map(&ta, A, (uint64_t)K, (uint64_t)max_tiles * TILE, (uint64_t)a_stride, stream_form ? TILE : 128) ||
        !make_map(&tw, W, (uint64_t)K, ANY_ROWS, (uint64_t)K, stream_form ? 64 : 128))
        return B200_EUNSUPPORTED;
    static B200SmemOptIn opt_rows, opt_stream;
    int dev = 0, sms = 0;
    B200_CUDA_CHECK((b200_ctx*)nullptr, cudaGetDevice(&dev));
    B200_CUDA_CHECK((b200_ctx*)nullptr, cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const int64_t bound = (int64_t)max_tiles * (n_out / cols);
    if (stream_form) {
        B200_CUDA_CHECK((b200_ctx*)nullptr, opt_stream.ensure(moe_stream_kernel, S_SMEM));
        B200_LAUNCH((moe_stream_kernel), dim3((unsigned)(bound < 2 * sms ? bound : 2 * sms)), S_THREADS, S_SMEM, stream, ta, tw, p);
        return b200_launch_status(nullptr);
    }
    B200_CUDA_CHECK((b200_ctx*)nullptr, opt_rows.ensure(moe_rows_kernel, R_SMEM));
    B200_LAUNCH((moe_rows_kernel), dim3((unsigned)(bound < sms ? bound : sms)), R_THREADS, R_SMEM, stream, ta, tw, p);
    return b200_launch_status(nullptr);
}

// ---- everything between the router's choice and the block's result, one call -------------------------------------------------------
namespace {

struct ExpertsSpace {
    int cap;                                      // rows of the grouped buffers
    size_t sorted, pos, tile, num, counts, grouped, inter, bytes;
};
ExpertsSpace experts_space(int64_t pairs, int experts, int K, int inter) {
    ExpertsSpace s;
    const int64_t cap = (pairs + (int64_t)experts * (TILE - 1) + TILE - 1) / TILE * TILE;
    s.cap = cap < (1ll << 31) ? (int)cap : 0;
    size_t at = 0;
    auto take = [&](size_t bytes) {
        const size_t p = at;
        at += (bytes + 255) / 256 * 256;
        return p;
    };
    s.sorted = take(4 * cap);
    s.pos = take(4 * pairs);
    s.tile = take(4 * (cap / TILE));
    s.num = take(4);
    s.counts = take(8 * (size_t)experts);
    s.grouped = take(2 * (size_t)cap * K);
    s.inter = take(2 * (size_t)cap * inter);
    s.bytes = at;
    return s;
}

}  // namespace

extern "C" size_t b200m_moe_experts_workspace_bytes(int64_t pairs, int num_experts, int K, int inter) {
    if (pairs < 0 || num_experts <= 0 || K <= 0 || inter <= 0) return 0;
    return experts_space(pairs, num_experts, K, inter).bytes;
}

extern "C" int b200m_moe_experts(const void* A, int64_t a_stride, const int32_t* idx, const float* wgt, int weigh_inputs, int n, int top, int num_experts,
                                 const void* W_in, int N, int K, int act, const void* W_out, int width, const void* shared, const float* gate_logit, int64_t gate_ld,
                                 const float* ident, float* out, float* rows, int rows_cap, void* workspace, size_t workspace_bytes, void* stream) {
    if (!A || !idx || !wgt || !W_in || !W_out || !out || !rows || !workspace || n < 0 || top <= 0 || num_experts <= 0 || N <= 0 || K <= 0 || width <= 0 || act < 0 || act > 2 ||
        (act == 2 && N % 2))
        return B200_EINVAL;
    if (n == 0) return B200_OK;
    const int inter = act == 2 ? N / 2 : N;
    const int64_t pairs = (int64_t)n * top;
    const ExpertsSpace s = experts_space(pairs, num_experts, K, inter);
    if (s.cap == 0 || pairs >= (1ll << 31)) return B200_EUNSUPPORTED;
    if (workspace_bytes < s.bytes || reinterpret_cast<uintptr_t>(workspace) % 256 || rows_cap < s.cap || reinterpret_cast<uintptr_t>(rows) % 256) return B200_EWORKSPACE;
    uint8_t* ws = static_cast<uint8_t*>(workspace);
    int32_t *sorted = reinterpret_cast<int32_t*>(ws + s.sorted), *pos = reinterpret_cast<int32_t*>(ws + s.pos), *tile = reinterpret_cast<int32_t*>(ws + s.tile),
            *num = reinterpret_cast<int32_t*>(ws + s.num), *counts = reinterpret_cast<int32_t*>(ws + s.counts);
    const int tiles = s.cap / TILE;
    const int64_t per = pairs / num_experts;
    const int hint = (per < 1 ? 1 : per > (1 << 22) ? 1 << 22 : (int)per) << 8;
    const float* in_wgt = weigh_inputs ? wgt : nullptr;
    int rc = b200m_moe_align(idx, (int)pairs, num_experts, sorted, s.cap, pos, tile, num, counts, stream);
    if (rc != B200_OK) return rc;
    // grouped inputs for the tcgen05 forms; weight blocks they do not tile: gathered inside the general form
    rc = N % 256 == 0 ? b200m_moe_gather(A, a_stride, sorted, in_wgt, top, num, tiles, K, ws + s.grouped, stream) : B200_EUNSUPPORTED;
    // The tcgen05 forms themselves, which may begin early here: in front of the first is the gather, in front of the second the first, and both let go only behind their own wait
    bool first = false;
    if (rc == B200_OK) {
        rc = b200m_moe_gemm_tc(ws + s.grouped, K, sorted, tile, num, tiles, W_in, N, K, ws + s.inter, 0, act, hint >> 8, 1, static_cast<cudaStream_t>(stream));
        first = rc == B200_OK;
        if (rc == B200_EUNSUPPORTED) rc = b200m_moe_gemm(ws + s.grouped, K, sorted, nullptr, top, 0, tile, num, tiles, W_in, N, K, ws + s.inter, 0, act | hint, 0, stream);
    } else if (rc == B200_EUNSUPPORTED) {
        rc = b200m_moe_gemm(A, a_stride, sorted, in_wgt, top, 1, tile, num, tiles, W_in, N, K, ws + s.inter, 0, act, 0, stream);
    }
    if (rc != B200_OK) return rc;
    rc = first ? b200m_moe_gemm_tc(ws + s.inter, inter, sorted, tile, num, tiles, W_out, width, inter, rows, 1, 0, hint >> 8, 1, static_cast<cudaStream_t>(stream)) : B200_EUNSUPPORTED;
    if (rc == B200_EUNSUPPORTED) rc = b200m_moe_gemm(ws + s.inter, inter, sorted, nullptr, top, 0, tile, num, tiles, W_out, width, inter, rows, 1, hint, 0, stream);
    if (rc != B200_OK) return rc;
    return b200m_moe_combine(rows, pos, top, shared, gate_logit, gate_ld, weigh_inputs ? nullptr : wgt, ident, out, n, width, 0, stream);
}
