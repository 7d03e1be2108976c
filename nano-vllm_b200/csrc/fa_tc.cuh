// Causal attention of prompt portions on the 5th-generation tensor cores: one persistent, warp-specialised kernel for every
// key/value source this framework has (packed projections, head-major pages, token-major cache rows).
//
// A CTA walks a list of work items; an item is TWO tiles of 128 query rows that share their keys: the same rows of two query heads of one
// kv head (PAIR_HEADS), or 256 consecutive rows of one head.  Keys come in blocks of 64.  Roles (512 threads):
//
//   warps 0-3, 4-7   softmax of tile 0 / tile 1: thread = query row; S row from TMEM, scale / bias / mask, running maximum, exp2, P (bf16)
//                    back into the TMEM columns of S; O is rescaled in TMEM when a row's maximum grows by more than FaParams::lag (log2)
//   warps 8-11       results: O / l from TMEM to memory while the softmax warps are at the next item; zeroes V rows past the last key
//   warps 12, 13     tcgen05.mma of tile 0 / tile 1: S_t = Q_t K^T (both operands in shared memory), O_t += P_t V (P from TMEM, V an MN-major
//                    operand); one warp for both tiles was bound by the instructions around its products (2490 cycles per 64 keys)
//   warp 14          TMA: Q of the next items, K and V blocks through two rings of slots
//
// TMEM (512 columns): S / P of each tile twice (4 x 64), O of each tile (2 x 128).  A tile's products come in the order PV(j) QK(j+2):
// scores are two blocks ahead, so a softmax warp finds its next block's scores ready and waits for the products of the block it just left only
// to rescale O.  The walk does not stop at the end of an item: with two Q buffers the next items' first scores follow the last blocks of the
// present one.
//
// What bounds it: per step (64 keys, both tiles) the products take 2 x (384 + 256) cycles (QK^T reads 48 KB of shared memory at 128 B per
// cycle, PV 2 M multiply-adds) and 16384 exponentials 1024 on the special-function unit (16 per cycle); a step measures 1700-1800 cycles,
// most of it the softmax warps' instructions.  128-key blocks with one S per tile read less but put softmax, PV and QK of a tile in one
// chain: 1950 cycles per 64 keys.  A quarter to a half of the exponentials by a polynomial on the multiply-add pipe shortened the step to
// 1650 cycles and the time by nothing (the clock gave way).  Items are dealt out longest first (causal tiles late in a sequence see the
// most keys), every other round from the far end, so CTAs finish together.  One call at a time on a cool GPU, us of the layer: 4 x 2048 tokens of latent attention 303 -> 285, one
// prompt of 4096 239 -> 201, 3 of 500-1500 behind 1000 others in a window 165 -> 148, packed prompts of 1000-4000 193 -> 177.  Back to back at the power limit's clock: 4 x 2048 of
// latent attention 331 -> 317; windows (6 of 500-2200, 288 -> 282), 28 short packed prompts and long portions within 2 %, no more than runs of one side differ.
#pragma once
#include "tc_common.cuh"

// A copy per library (B200_LIB): kernels, and the record of their shared-memory opt-in, must not be merged across libraries of one process (a
// template's static is one object for all of them).
namespace b200fa {
inline namespace B200_LIB {

using namespace b200tc;

constexpr int BM = 128;                 // query rows per tile
constexpr int BN = 64;                  // keys per block
constexpr int DV = 128;                 // columns of a value row
constexpr int THREADS = 512;
constexpr int ITEM_CAP = 96;            // items per CTA (more items: more CTAs)
constexpr int LEVELS_CAP = 8192;        // row blocks per sequence that the longest-first order covers (its counters lie where Q will be)
constexpr float LOG2E = 1.4426950408889634f;

struct FaParams {
    const int32_t* cu_q;
    const int32_t* cu_k;
    const int32_t* block_tables;        // null: keys of sequence s are rows cu_k[s] .. of the K / V maps
    int bt_stride;
    int num_seqs, max_rb;               // sequences; most row blocks of one sequence
    int hq, hkv, hp;                    // query heads, kv heads, head items (hq / 2 or hq)
    int q_col_step;                     // columns from one head of Q to the next
    int k_col_step, v_col0, v_col_step; // columns of kv head h: h * step (+ v_col0)
    int k2_col;                         // 192-wide heads: first column of the last 64 key elements, shared by the heads, in their own map
    int block_size, box_rows;           // paged: rows of a page, rows per TMA box
    int64_t row0, page_rows, head_rows; // paged row = row0 + page * page_rows + kvh * head_rows + row in page
    float scale_log2;
    // How far (log2) a row's maximum may pass the reference its weights are formed against.  Above 0 spares most rescaling of O, but the row's largest
    // weights are then rounded to bf16 where 2^0 is exact, which peaked rows feel: scores of deviation 1 / 2 / 5 over 2048 keys are 0.0016 / 0.0016 /
    // 0.0012 from 64 bits at 8, and 0.0015 / 0.0009 / 0.0004 at 0.
    float lag;
    const float* slopes;                // per head, or null: score -= slope * (query position - key position)
    const float* sinks;                 // per head, or null: score of an extra term without a value
    int window, chunk;                  // visible keys: the last `window`, or those of the query's own chunk (0: all)
    void* out;                          // bf16 (or fp32) [rows, out_stride], head h at column h * DV
    int64_t out_stride;
    int out_f32;
    float out_scale;
    const __nv_bfloat16* gate;          // or null: result times sigmoid(gate), one per head or one per element
    int64_t gate_stride;
    int gate_elems;
    uint32_t* report;                   // host word for waits that gave up: results of such a launch are undefined
    // or null: rows of K and V (DV columns each, row r: token r / hkv, head r % hkv) that go into pages of 2^st_shift slots
    const int32_t* st_slots;            // per token, < 0: not stored
    const __nv_bfloat16 *st_k, *st_v;
    int64_t st_k_stride, st_v_stride;
    __nv_bfloat16 *st_kc, *st_vc;
    int st_rows, st_shift;
};

// The copy of this CTA's share of the rows, a part at a time by whichever warp is free (a counter in shared memory deals them out): half a warp per row, all loads of a
// part before its stores.  (A rotation by single rows, and loads under a condition, ran one row after the other: 283 us for 848 rows; one warp alone took 85.)
struct FaCopy {
    static constexpr int PAIRS = 8, ROWS = 2 * PAIRS;         // rows of a part
    int end, begin, row, slot;            // of the share; first row of the part this warp has next (end: none), slot of this lane's row in it

    __device__ __forceinline__ void next(const FaParams& p, int* counter, int lane) {
        int i = 0;
        if (lane == 0) i = atomicAdd(counter, 1);
        row = min(begin + ROWS * __shfl_sync(0xffffffffu, i, 0), end);
        slot = lane < ROWS && row + lane < end ? p.st_slots[(row + lane) / p.hkv] : -1;
    }
    __device__ __forceinline__ void start(const FaParams& p, int* counter, int lane) {
        begin = (int)((int64_t)p.st_rows * blockIdx.x / gridDim.x);
        end = (int)((int64_t)p.st_rows * (blockIdx.x + 1) / gridDim.x);
        next(p, counter, lane);
    }
    __device__ __forceinline__ bool part(const FaParams& p, int* counter, int lane) {
        if (row >= end) return false;
        const int in = min(row + lane, end - 1);                         // past the end: a row of this share once more, stored nowhere
        const int half = lane >> 4, col = (lane & 15) * 8;
        const int tok = in / p.hkv, head = in - tok * p.hkv;
        const int to = slot < 0 ? -1 : (((slot >> p.st_shift) * p.hkv + head) << p.st_shift) + (slot & ((1 << p.st_shift) - 1));
        next(p, counter, lane);
        uint4 k[PAIRS], v[PAIRS];
        int dst[PAIRS];
#pragma unroll
        for (int j = 0; j < PAIRS; ++j) {
            const int from = 2 * j + half;
            dst[j] = __shfl_sync(0xffffffffu, to, from);
            const int t = __shfl_sync(0xffffffffu, tok, from), h = __shfl_sync(0xffffffffu, head, from);
            k[j] = *reinterpret_cast<const uint4*>(p.st_k + t * p.st_k_stride + h * DV + col);
            v[j] = *reinterpret_cast<const uint4*>(p.st_v + t * p.st_v_stride + h * DV + col);
        }
#pragma unroll
        for (int j = 0; j < PAIRS; ++j)
            if (dst[j] >= 0) {
                *reinterpret_cast<uint4*>(p.st_kc + (int64_t)dst[j] * DV + col) = k[j];
                *reinterpret_cast<uint4*>(p.st_vc + (int64_t)dst[j] * DV + col) = v[j];
            }
        __syncwarp();
        return true;
    }
};

template <int DQK>
struct FaSmem {
    static constexpr int kQBufs = DQK <= 128 ? 2 : 1;                    // wider heads: one Q buffer, the walk refills at item borders
    static constexpr int kSlots = 3;                                     // K blocks, and V blocks, in flight
    static constexpr uint32_t kQSub = BM * 128;                          // one [128][64] piece of a Q tile
    static constexpr uint32_t kQTile = (DQK / 64) * kQSub;
    static constexpr uint32_t kKSub = BN * 128;
    static constexpr uint32_t kKBytes = (DQK / 64) * kKSub;
    static constexpr uint32_t kVBytes = (DV / 64) * kKSub;
    static constexpr uint32_t kOffK = kQBufs * 2 * kQTile;
    static constexpr uint32_t kOffV = kOffK + kSlots * kKBytes;
    static constexpr uint32_t kOffL = kOffV + kSlots * kVBytes;          // float[2][128] row sums
    static constexpr uint32_t kOffList = kOffL + 2 * BM * 4;             // int4[ITEM_CAP]
    static constexpr uint32_t kOffBar = kOffList + ITEM_CAP * 16;
    static constexpr uint32_t kTotal = kOffBar + 320;
    static_assert(kTotal <= 227 * 1024, "shared memory");
};
// barriers (8 bytes each): index of the first of each kind
constexpr uint32_t NSLOT = 3;
constexpr uint32_t B_QFULL = 0, B_KFULL = 2, B_VFULL = B_KFULL + NSLOT, B_S = B_VFULL + NSLOT /* [tile][buffer] */, B_PV = B_S + 4, B_O = B_PV + 2, B_VRAW = B_O + 2,
                   B_QEMPTY = B_VRAW + 1 /* from here on 2 arrivals each: the two MMA warps */, B_KEMPTY = B_QEMPTY + 2, B_VEMPTY = B_KEMPTY + NSLOT,
                   B_P = B_VEMPTY + NSLOT /* [tile][buffer]; from here on 128 arrivals each */, B_L = B_P + 4, B_OFREE = B_L + 2, B_VFIX = B_OFREE + 2,
                   B_COUNT = B_VFIX + 1;
constexpr uint32_t BAR_TMEM = B_COUNT * 8, BAR_DEAD = BAR_TMEM + 4, BAR_COPY = BAR_DEAD + 4;      // tcgen05.alloc result; set when a wait gave up; parts dealt out
static_assert(BAR_COPY + 4 <= 320, "barrier area");

__device__ __forceinline__ void fa_arrive(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }

__device__ __forceinline__ void tc_mma_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}\n" ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// 32 consecutive columns of this thread's lane, without the wait
__device__ __forceinline__ void tmem_ld32n(uint32_t taddr, float* v) {
    uint32_t* r = reinterpret_cast<uint32_t*>(v);
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,"
        "%28,%29,%30,%31}, [%32];\n\t"
        : TC_R8(r, 0), TC_R8(r, 8), TC_R8(r, 16), TC_R8(r, 24)
        : "r"(taddr));
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_st32u(uint32_t taddr, const uint32_t* v) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,"
        "%27,%28,%29,%30,%31,%32};" ::"r"(taddr),
        TC_I8(v, 0), TC_I8(v, 8), TC_I8(v, 16), TC_I8(v, 24)
        : "memory");
}

// Two fp32 operations in one instruction.
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    float2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;"
        : "=l"(reinterpret_cast<uint64_t&>(d))
        : "l"(reinterpret_cast<uint64_t&>(a)), "l"(reinterpret_cast<uint64_t&>(b)), "l"(reinterpret_cast<uint64_t&>(c)));
    return d;
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
    float2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(reinterpret_cast<uint64_t&>(d)) : "l"(reinterpret_cast<uint64_t&>(a)), "l"(reinterpret_cast<uint64_t&>(b)));
    return d;
}
__device__ __forceinline__ float2 both(float v) { return make_float2(v, v); }
__device__ __forceinline__ float max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
// One work item.  Its list entry: (sequence, row block | head item << 20, key blocks of tile 0 | of tile 1 << 16, first block | "the last
// block reaches past the keys" << 31).
struct FaItem {
    int seq, head0, kvh;
    int q0, len_q, k0, len_k, off;
    int r0[2];                          // first query row of each tile
    int n[2];                           // key blocks of each tile (0: no such tile)
    int nmax, j_lo;                     // blocks walked, first block
};

template <bool PAIR_HEADS>
__device__ __forceinline__ int4 fa_entry(const FaParams& p, int seq, int rb, int hp) {
    constexpr int RT = PAIR_HEADS ? BM : 2 * BM;
    const int len_q = p.cu_q[seq + 1] - p.cu_q[seq], len_k = p.cu_k[seq + 1] - p.cu_k[seq], off = len_k - len_q;
    const int pos0 = rb * RT + off;                                      // position of the item's first row
    int lo = 0;
    if (p.chunk > 0) lo = pos0 > 0 ? pos0 / p.chunk * p.chunk : 0;
    else if (p.window > 0) lo = pos0 - p.window + 1;
    const int j_lo = lo > 0 ? lo / BN : 0;
    int n[2];
#pragma unroll
    for (int t = 0; t < 2; ++t) {
        const int r0 = rb * RT + (PAIR_HEADS ? 0 : t * BM);
        int end = r0 + BM + off;
        end = end < len_k ? end : len_k;
        const int k = (end + BN - 1) / BN - j_lo;
        n[t] = r0 < len_q ? (k > 1 ? k : 1) : 0;                         // a tile without visible keys walks one masked block: its result is 0
    }
    const int nmax = n[0] > n[1] ? n[0] : n[1];
    return make_int4(seq, rb | hp << 20, n[0] | n[1] << 16, j_lo | ((j_lo + nmax) * BN > len_k ? 1 << 31 : 0));
}
template <bool PAIR_HEADS>
__device__ __forceinline__ FaItem fa_item(const FaParams& p, const int4* list, int e) {
    FaItem it;
    const int4 v = list[e];
    it.seq = v.x;
    it.q0 = p.cu_q[it.seq];
    it.len_q = p.cu_q[it.seq + 1] - it.q0;
    it.k0 = p.cu_k[it.seq];
    it.len_k = p.cu_k[it.seq + 1] - it.k0;
    it.off = it.len_k - it.len_q;
    it.head0 = (v.y >> 20) * (PAIR_HEADS ? 2 : 1);
    it.kvh = it.head0 / (p.hq / p.hkv);
    it.r0[0] = (v.y & 0xfffff) * (PAIR_HEADS ? BM : 2 * BM);
    it.r0[1] = it.r0[0] + (PAIR_HEADS ? 0 : BM);
    it.n[0] = v.z & 0xffff;
    it.n[1] = (int)((uint32_t)v.z >> 16);
    it.nmax = it.n[0] > it.n[1] ? it.n[0] : it.n[1];
    it.j_lo = v.w & 0x7fffffff;
    return it;
}
// A slot of a ring of NSLOT and the parity of its use.
struct FaSlot {
    uint32_t i = 0, ph = 0;
    __device__ __forceinline__ void next() {
        if (++i == NSLOT) {
            i = 0;
            ph ^= 1;
        }
    }
};

// GENERAL: scores with a distance bias, or a scale that is not positive.  STORE: warps 8-11, between items, and 15 scatter the step's K and V rows into their pages.
template <int DQK, bool PAIR_HEADS, bool GENERAL, bool STORE>
__global__ void __launch_bounds__(THREADS, 1)
fa_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v,
          const __grid_constant__ CUtensorMap tm_k2, const __grid_constant__ FaParams p) {
    using L = FaSmem<DQK>;
    constexpr uint32_t IDESC_QK = make_idesc(BM, BN, false), IDESC_PV = make_idesc(BM, DV, true);
    constexpr int RT = PAIR_HEADS ? BM : 2 * BM;
    extern __shared__ __align__(1024) uint8_t smem[];
    const uint32_t base = smem_u32(smem);
    const uint32_t bars = base + L::kOffBar, dead = bars + BAR_DEAD;
    auto bar = [&](uint32_t i) { return bars + i * 8; };
    auto fa_wait = [&](uint32_t b, uint32_t parity) { return bounded_wait(b, parity, dead, p.report); };
    auto lane_wait = [&](uint32_t b, uint32_t parity) { return bounded_wait_as<false>(b, parity, dead, p.report); };
    int4* list = reinterpret_cast<int4*>(smem + L::kOffList);
    int* parts = reinterpret_cast<int*>(smem + L::kOffBar + BAR_COPY);
    float* lbuf = reinterpret_cast<float*>(smem + L::kOffL);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

    if (tid == 0) {
        for (uint32_t i = 0; i < B_COUNT; ++i) mbar_init(bar(i), i >= B_P ? 128 : i >= B_QEMPTY ? 2 : 1);
        mbar_fence_init();
        *reinterpret_cast<volatile uint32_t*>(smem + L::kOffBar + BAR_DEAD) = 0;
        if (STORE) *reinterpret_cast<volatile int*>(smem + L::kOffBar + BAR_COPY) = 0;
    }
    if (warp == 12) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(bars + BAR_TMEM), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid >= 448 && tid < 451) {
        const CUtensorMap* m = tid == 448 ? &tm_q : tid == 449 ? &tm_k : &tm_v;
        asm volatile("prefetch.tensormap [%0];" ::"l"(m) : "memory");
    }
    B200_PDL_SYNC();
    // ---- this CTA's items: all (sequence, row block) pairs, last row blocks first, head items innermost ----
    int* level = reinterpret_cast<int*>(smem);                           // level[b]: sequences with more than b row blocks
    const bool sorted = p.max_rb <= LEVELS_CAP;
    int total = 0;
    if (sorted) {
        for (int b = tid; b < p.max_rb; b += THREADS) level[b] = 0;
        __syncthreads();
        for (int s = tid; s < p.num_seqs; s += THREADS) {
            int nb = (p.cu_q[s + 1] - p.cu_q[s] + RT - 1) / RT;
            nb = nb < p.max_rb ? nb : p.max_rb;
            for (int b = 0; b < nb; ++b) atomicAdd(&level[b], 1);
        }
        __syncthreads();
    }
    {
        int64_t tiles = 0;
        if (sorted) for (int b = 0; b < p.max_rb; ++b) tiles += level[b];
        else for (int s = 0; s < p.num_seqs; ++s) tiles += (p.cu_q[s + 1] - p.cu_q[s] + RT - 1) / RT;
        total = (int)(tiles * p.hp);
    }
    // A CTA's items are early and late ones of their rounds in turn (each round from the same end gave the first CTAs 1.05 to 1.3 times the mean's work)
    auto place = [&](int round) { return round & 1 ? (int)gridDim.x - 1 - (int)blockIdx.x : (int)blockIdx.x; };
    int n_items = total / (int)gridDim.x;
    n_items += place(n_items) < total - n_items * (int)gridDim.x;
    n_items = n_items < ITEM_CAP ? n_items : ITEM_CAP;                   // cannot bind while total_q covers the sequences
    if (tid < n_items) {
        const int i = tid * (int)gridDim.x + place(tid);
        int w = i / p.hp, seq = 0, rb = 0;
        if (sorted) {
            rb = p.max_rb - 1;
            while (w >= level[rb]) w -= level[rb--];
            for (;; ++seq)
                if ((p.cu_q[seq + 1] - p.cu_q[seq] + RT - 1) / RT > rb && w-- == 0) break;
        } else {
            for (;; ++seq) {
                const int nb = (p.cu_q[seq + 1] - p.cu_q[seq] + RT - 1) / RT;
                if (w < nb) break;
                w -= nb;
            }
            rb = (p.cu_q[seq + 1] - p.cu_q[seq] + RT - 1) / RT - 1 - w;
        }
        list[tid] = fa_entry<PAIR_HEADS>(p, seq, rb, i % p.hp);
    }
    tc_fence_before();
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");         // the counters' bytes go to the TMA next
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(smem + L::kOffBar + BAR_TMEM);
    const uint32_t tmem_o = tmem + 256;                                  // S_t / P_t at t * 128 + buffer * 64, O_t at 256 + t * 128

    if (warp < 8) {
        // ---- softmax ------------------------------------------------------------------------------------------------------
        const int t = warp >> 2, r = tid & 127;
        const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
        const uint32_t ts0 = tmem + t * 128 + lane_base, to = tmem_o + t * 128 + lane_base;
        uint32_t blk = 0, items = 0;                                     // blocks and items of this tile so far
        for (int e = 0; e < n_items; ++e) {
            const FaItem it = fa_item<PAIR_HEADS>(p, list, e);
            const int n = it.n[t];
            if (n == 0) continue;
            const int head = it.head0 + (PAIR_HEADS ? t : 0);
            const int pos = it.r0[t] + r + it.off;                       // this row's position
            int lo = 0;
            if (p.chunk > 0) lo = pos > 0 ? pos / p.chunk * p.chunk : 0;
            else if (p.window > 0) lo = pos - p.window + 1;
            // extreme positions of the warp's rows: blocks inside them need no mask
            const int wpos = it.r0[t] + (warp & 3) * 32 + it.off;
            int wlo = 0;                                                 // largest lower bound among the warp's rows
            if (p.chunk > 0) wlo = wpos + 31 > 0 ? (wpos + 31) / p.chunk * p.chunk : 0;
            else if (p.window > 0) wlo = wpos + 31 - p.window + 1;
            const float slope = GENERAL && p.slopes ? p.slopes[head] * LOG2E : 0.f;
            float m_ref = -INFINITY, l_sum = 0.f;
            if (p.sinks) {
                m_ref = p.sinks[head] * LOG2E;
                l_sum = 1.0f;
            }
            for (int j = 0; j < n; ++j, ++blk) {
                const int key0 = (it.j_lo + j) * BN;
                const uint32_t b = blk & 1, ts = ts0 + b * BN;
                if (!fa_wait(bar(B_S + t * 2 + b), (blk >> 1) & 1)) goto leave;
                tc_fence_after();
                float s[BN];
                tmem_ld32n(ts, s);
                tmem_ld32n(ts + 32, s + 32);
                tmem_wait_ld();
                // GENERAL: scores in log2 units with their bias, before the maximum.  Else (scale > 0, no bias) the scale rides in the exponent's
                // multiply-add.
                if (GENERAL) {
                    const float b0 = slope * (float)(key0 - pos);
#pragma unroll
                    for (int c = 0; c < BN; c += 2) {
                        const float2 v = fma2(make_float2(s[c], s[c + 1]), both(p.scale_log2), make_float2(fmaf(slope, (float)c, b0), fmaf(slope, (float)(c + 1), b0)));
                        s[c] = v.x;
                        s[c + 1] = v.y;
                    }
                }
                if (key0 + BN > it.len_k || key0 + BN - 1 > wpos) {      // keys after this row's position, or past the last one
                    const int hi = (pos < it.len_k ? pos : it.len_k - 1) - key0;
#pragma unroll
                    for (int c = 0; c < BN; ++c) s[c] = c <= hi ? s[c] : -INFINITY;
                }
                if (key0 < wlo) {                                        // keys before the window or chunk
                    const int lo_c = lo - key0;
#pragma unroll
                    for (int c = 0; c < BN; ++c) s[c] = c >= lo_c ? s[c] : -INFINITY;
                }
                float mx[4] = {max3(s[0], s[1], s[2]), max3(s[3], s[4], s[5]), max3(s[6], s[7], s[8]), max3(s[9], s[10], s[11])};
#pragma unroll
                for (int c = 12; c + 7 < BN; c += 8) {
#pragma unroll
                    for (int k = 0; k < 4; ++k) mx[k] = max3(mx[k], s[c + 2 * k], s[c + 2 * k + 1]);
                }
                mx[0] = max3(mx[0], s[BN - 4], s[BN - 3]);
                mx[1] = max3(mx[1], s[BN - 2], s[BN - 1]);
                float m_new = max3(fmaxf(mx[0], mx[1]), mx[2], mx[3]);
                if (!GENERAL) m_new *= p.scale_log2;
                const bool grow = m_new > m_ref + p.lag;                 // m_ref = -inf: the first block with a visible key
                if (__any_sync(0xffffffffu, grow)) {
                    const float m_upd = grow ? m_new : m_ref;
                    const float f = m_ref == m_upd ? 1.0f : fast_exp2(m_ref - m_upd);
                    m_ref = m_upd;
                    l_sum *= f;
                    if (j > 0) {                                         // O holds the blocks before this one once their products are done
                        if (!fa_wait(bar(B_PV + t), (blk - 1) & 1)) goto leave;
                        tc_fence_after();
#pragma unroll 1
                        for (int c = 0; c < DV; c += 32) {
                            float o[32];
                            tmem_ld32n(to + c, o);
                            tmem_wait_ld();
#pragma unroll
                            for (int k = 0; k < 32; ++k) o[k] *= f;
                            tmem_st32u(to + c, reinterpret_cast<const uint32_t*>(o));
                        }
                        tmem_wait_st();
                    }
                }
                const float m_use = m_ref == -INFINITY ? 0.f : m_ref;
                const float2 nm2 = both(-m_use), sc2 = both(p.scale_log2);
                float2 acc0 = both(0.f), acc1 = both(0.f);
                uint32_t pk[BN / 2];
#pragma unroll
                for (int c = 0; c < BN; c += 4) {
                    float2 x = GENERAL ? add2(make_float2(s[c], s[c + 1]), nm2) : fma2(make_float2(s[c], s[c + 1]), sc2, nm2);
                    float2 y = GENERAL ? add2(make_float2(s[c + 2], s[c + 3]), nm2) : fma2(make_float2(s[c + 2], s[c + 3]), sc2, nm2);
                    x.x = fast_exp2(x.x);
                    x.y = fast_exp2(x.y);
                    y.x = fast_exp2(y.x);
                    y.y = fast_exp2(y.y);
                    acc0 = add2(acc0, x);
                    acc1 = add2(acc1, y);
                    pk[c / 2] = pack_bf16x2(x.x, x.y);
                    pk[c / 2 + 1] = pack_bf16x2(y.x, y.y);
                }
                tmem_st32u(ts, pk);
                l_sum += (acc0.x + acc0.y) + (acc1.x + acc1.y);
                tmem_wait_st();
                tc_fence_before();
                fa_arrive(bar(B_P + t * 2 + b));
            }
            if (!fa_wait(bar(B_OFREE + t), (items & 1) ^ 1)) goto leave;     // the sums of the item before have been read
            lbuf[t * BM + r] = l_sum;
            fa_arrive(bar(B_L + t));
            ++items;
        }
    } else if (warp < 12) {
        // ---- results ------------------------------------------------------------------------------------------------------
        const int r = tid & 127;
        const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
        uint32_t items[2] = {0, 0}, fixes = 0;
        FaSlot vs;
        FaCopy copy;
        if (STORE) copy.start(p, parts, lane);
        const bool wide = (reinterpret_cast<uintptr_t>(p.out) & 31) == 0 && (p.out_stride & 15) == 0;      // 32-byte stores: whole sectors
        for (int e = 0; e < n_items; ++e) {
            const FaItem it = fa_item<PAIR_HEADS>(p, list, e);
            const int last = (it.j_lo + it.nmax) * BN;
            for (int k = 1; k < it.nmax; ++k) vs.next();                 // the slot of the item's last V block
            if (last > it.len_k) {
                // The last block reaches past the sequence's keys: those V rows are not its own (stale page rows, the next sequence of a
                // packed batch, perhaps NaN).  Their P is exactly 0, but 0 * NaN would poison the sum: zero the staged rows (a whole
                // 128-byte row is swizzle-agnostic).
                if (!fa_wait(bar(B_VRAW), fixes & 1)) goto leave;  // an MMA warp has seen it land
                ++fixes;
                int first = it.len_k - (last - BN);
                first = first > 0 ? first : 0;
                uint8_t* v = smem + L::kOffV + vs.i * L::kVBytes;
                for (int i = r; i < (BN - first) * (DV / 8); i += 128) {
                    const int row = first + i / (DV / 8), c = i % (DV / 8);
                    *reinterpret_cast<uint4*>(v + (c >> 3) * L::kKSub + row * 128 + ((c & 7) << 4)) = make_uint4(0, 0, 0, 0);
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                fa_arrive(bar(B_VFIX));
            }
            vs.next();
#pragma unroll
            for (int t = 0; t < 2; ++t) {
                if (it.n[t] == 0) continue;
                const int head = it.head0 + (PAIR_HEADS ? t : 0), row = it.r0[t] + r;
                const bool valid = row < it.len_q;
                const int64_t grow = it.q0 + (valid ? row : 0);
                if (!fa_wait(bar(B_L + t), items[t] & 1)) goto leave;
                const float l = lbuf[t * BM + r];
                float f = l > 0.f ? p.out_scale / l : 0.f;
                if (p.gate && !p.gate_elems && valid) f *= 1.0f / (1.0f + expf(-__bfloat162float(p.gate[grow * p.gate_stride + head])));
                if (!fa_wait(bar(B_O + t), items[t] & 1)) goto leave;
                tc_fence_after();
                if (!p.out_f32 && !(p.gate && p.gate_elems)) {
                    // the usual result: all of O into registers, so that the next item's products can start, then the stores
                    uint32_t pk[DV / 2];
#pragma unroll
                    for (int q4 = 0; q4 < DV / 32; ++q4) {
                        float o[32];
                        tmem_ld32(tmem_o + t * 128 + lane_base + q4 * 32, o);
#pragma unroll
                        for (int k = 0; k < 16; ++k) pk[q4 * 16 + k] = pack_bf16x2(o[2 * k] * f, o[2 * k + 1] * f);
                    }
                    tc_fence_before();
                    fa_arrive(bar(B_OFREE + t));
                    if (valid) {
                        __nv_bfloat16* d = static_cast<__nv_bfloat16*>(p.out) + grow * p.out_stride + (int64_t)head * DV;
                        if (wide) {
#pragma unroll
                            for (int k = 0; k < DV / 16; ++k) st_256(d + k * 16, pk + k * 8);
                        } else {
#pragma unroll
                            for (int k = 0; k < DV / 8; ++k) *reinterpret_cast<uint4*>(d + k * 8) = make_uint4(pk[4 * k], pk[4 * k + 1], pk[4 * k + 2], pk[4 * k + 3]);
                        }
                    }
                    ++items[t];
                    continue;
                }
#pragma unroll 1
                for (int q4 = 0; q4 < DV / 32; ++q4) {
                    __syncwarp();
                    float o[32];
                    tmem_ld32(tmem_o + t * 128 + lane_base + q4 * 32, o);
                    if (!valid) continue;
                    const int64_t col = (int64_t)head * DV + q4 * 32;
#pragma unroll
                    for (int c8 = 0; c8 < 4; ++c8) {
                        float v[8];
#pragma unroll
                        for (int k = 0; k < 8; ++k) v[k] = o[c8 * 8 + k] * f;
                        if (p.gate && p.gate_elems) {
                            float g[8];
                            unpack8(*reinterpret_cast<const uint4*>(p.gate + grow * p.gate_stride + col + c8 * 8), g);
#pragma unroll
                            for (int k = 0; k < 8; ++k) v[k] *= 1.0f / (1.0f + expf(-g[k]));
                        }
                        if (p.out_f32) {
                            float* d = static_cast<float*>(p.out) + grow * p.out_stride + col + c8 * 8;
                            *reinterpret_cast<float4*>(d) = make_float4(v[0], v[1], v[2], v[3]);
                            *reinterpret_cast<float4*>(d + 4) = make_float4(v[4], v[5], v[6], v[7]);
                        } else {
                            *reinterpret_cast<uint4*>(static_cast<__nv_bfloat16*>(p.out) + grow * p.out_stride + col + c8 * 8) = pack8(v);
                        }
                    }
                }
                tc_fence_before();
                fa_arrive(bar(B_OFREE + t));
                ++items[t];
            }
            if (STORE) copy.part(p, parts, lane);                        // while the next item's products run
        }
        if (STORE) while (copy.part(p, parts, lane)) {}
    } else if (warp < 14) {
        // ---- products of one tile (all lanes walk and wait, one issues) -------------------------------------------------------
        const int t = warp - 12;
        const bool leader = elect_one();
        const uint64_t qd0 = make_desc(base + t * L::kQTile, 16, 1024), kd0 = make_desc(base + L::kOffK, 16, 1024), vd0 = make_desc(base + L::kOffV, L::kKSub, 1024);
        const uint32_t ts = tmem + t * 128, to = tmem_o + t * 128;
        // the scores' walk runs ahead of the products' walk: its item, block and K slot
        int la_n = 0, la_max = 0, la_e = 0, la_j = 0;
        uint32_t sbuf = 0, pbuf = 0, pph = 0, oph = 1, fixes = 0;
        FaSlot ks, vs;
        auto la_load = [&]() {
            const int z = list[la_e].z, n0 = z & 0xffff, n1 = (int)((uint32_t)z >> 16);
            la_n = t ? n1 : n0;
            la_max = max(n0, n1);
        };
        if (n_items > 0) la_load();
        auto qk = [&]() -> bool {                                        // S = Q K^T into the buffer whose P went two blocks ago
            const uint32_t qb = la_e % L::kQBufs;
            if (la_j == 0 && !lane_wait(bar(B_QFULL + qb), (la_e / L::kQBufs) & 1)) return false;
            if (!lane_wait(bar(B_KFULL + ks.i), ks.ph)) return false;
            tc_fence_after();
            const bool mine = la_j < la_n;
            if (leader) {
                if (mine) {
                    const uint64_t qd = qd0 + qb * (2 * L::kQTile / 16), kd = kd0 + ks.i * (L::kKBytes / 16);
#pragma unroll
                    for (int k = 0; k < DQK / 16; ++k)
                        tc_mma(ts + sbuf * BN, qd + ((k >> 2) * L::kQSub + (k & 3) * 32) / 16, kd + ((k >> 2) * L::kKSub + (k & 3) * 32) / 16, IDESC_QK, k > 0);
                    tc_commit(bar(B_S + t * 2 + sbuf));
                }
                tc_commit(bar(B_KEMPTY + ks.i));
                if (la_j + 1 == la_max) tc_commit(bar(B_QEMPTY + qb));
            }
            if (mine) sbuf ^= 1;
            ks.next();
            if (++la_j == la_max) {
                la_j = 0;
                if (++la_e < n_items) la_load();
            }
            return true;
        };
        for (int e = 0; e < n_items; ++e) {
            const int4 w = list[e];
            const int n0 = w.z & 0xffff, n1 = (int)((uint32_t)w.z >> 16), n = t ? n1 : n0, nmax = max(n0, n1);
            if (e == 0 || L::kQBufs == 1)                                // fill: the first two blocks' scores
                for (int k = 0; k < 2 && la_e < n_items && (L::kQBufs > 1 || la_e == e); ++k)
                    if (!qk()) goto leave;
            for (int j = 0; j < nmax; ++j) {
                if (!lane_wait(bar(B_VFULL + vs.i), vs.ph)) goto leave;
                if (w.w < 0 && j + 1 == nmax) {
                    if (t == 0 && leader) fa_arrive(bar(B_VRAW));
                    if (!lane_wait(bar(B_VFIX), fixes & 1)) goto leave;
                    ++fixes;
                }
                if (j < n) {
                    if (!lane_wait(bar(B_P + t * 2 + pbuf), pph)) goto leave;
                    if (j == 0) {                                        // the results of the item before have been read out
                        if (!lane_wait(bar(B_OFREE + t), oph)) goto leave;
                        oph ^= 1;
                    }
                    tc_fence_after();
                    if (leader) {
                        const uint64_t vd = vd0 + vs.i * (L::kVBytes / 16);
#pragma unroll
                        for (int k = 0; k < BN / 16; ++k) tc_mma_ts(to, ts + pbuf * BN + k * 8, vd + k * (2048 / 16), IDESC_PV, k > 0 || j > 0);
                        tc_commit(bar(B_PV + t));
                        if (j + 1 == n) tc_commit(bar(B_O + t));
                    }
                    pbuf ^= 1;
                    pph ^= pbuf ^ 1;
                }
                if (leader) tc_commit(bar(B_VEMPTY + vs.i));
                vs.next();
                if (la_e < n_items && (L::kQBufs > 1 || la_e == e) && !qk()) goto leave;
            }
        }
    } else if (warp == 14) {
        // ---- loads (the whole warp: a lane per page box) -----------------------------------------------------------------------
        FaSlot sl;                                                       // K and V blocks alternate: one position for both rings
        const int boxes = p.block_tables ? BN / p.box_rows : 1;
        auto load_q = [&](int e) -> bool {
            const FaItem it = fa_item<PAIR_HEADS>(p, list, e);
            const uint32_t qb = e % L::kQBufs;
            if (!fa_wait(bar(B_QEMPTY + qb), ((e / L::kQBufs) & 1) ^ 1)) return false;
            if (lane == 0) {
                mbar_expect_tx(bar(B_QFULL + qb), ((it.n[0] > 0) + (it.n[1] > 0)) * L::kQTile);
                for (int t = 0; t < 2; ++t)
                    if (it.n[t])
                        for (int h = 0; h < DQK / 64; ++h)
                            tma_load_2d(base + (qb * 2 + t) * L::kQTile + h * L::kQSub, &tm_q, bar(B_QFULL + qb), (it.head0 + (PAIR_HEADS ? t : 0)) * p.q_col_step + h * 64,
                                        it.q0 + it.r0[t]);
            }
            __syncwarp();
            return true;
        };
        if (n_items > 0 && !load_q(0)) goto leave;
        for (int e = 0; e < n_items; ++e) {
            const FaItem it = fa_item<PAIR_HEADS>(p, list, e);
            if (L::kQBufs == 1 && e > 0 && !load_q(e)) goto leave;
            // with two buffers the next item's Q is asked for early in this one, once its buffer's last reader (the item before) is done:
            // that is when the third K slot of this item has come free
            const int ask = it.nmax > 2 ? 2 : it.nmax - 1;
            for (int j = 0; j < it.nmax; ++j) {
                const int key0 = (it.j_lo + j) * BN;
                int row = it.k0 + key0;
                if (p.block_tables && lane < boxes) {
                    const int key = key0 + lane * p.box_rows;
                    const int page = key < it.len_k ? p.block_tables[(int64_t)it.seq * p.bt_stride + key / p.block_size] : -1;
                    // no page (below a window, past the keys): a box outside the map, which reads as zeros
                    row = page < 0 ? -p.box_rows : (int)(p.row0 + page * p.page_rows + it.kvh * p.head_rows + key % p.block_size);
                }
                if (!fa_wait(bar(B_KEMPTY + sl.i), sl.ph ^ 1)) goto leave;
                if (lane == 0) mbar_expect_tx(bar(B_KFULL + sl.i), L::kKBytes);
                __syncwarp();
                if (lane < boxes)
                    for (int h = 0; h < DQK / 64; ++h) {
                        const uint32_t dst = base + L::kOffK + sl.i * L::kKBytes + lane * p.box_rows * 128 + h * L::kKSub;
                        if (h < 2) tma_load_2d(dst, &tm_k, bar(B_KFULL + sl.i), it.kvh * p.k_col_step + h * 64, row);
                        else tma_load_2d(dst, &tm_k2, bar(B_KFULL + sl.i), p.k2_col, row);         // the key part all heads share
                    }
                if (!fa_wait(bar(B_VEMPTY + sl.i), sl.ph ^ 1)) goto leave;
                if (lane == 0) mbar_expect_tx(bar(B_VFULL + sl.i), L::kVBytes);
                __syncwarp();
                if (lane < boxes)
                    for (int h = 0; h < DV / 64; ++h)
                        tma_load_2d(base + L::kOffV + sl.i * L::kVBytes + lane * p.box_rows * 128 + h * L::kKSub, &tm_v, bar(B_VFULL + sl.i), p.v_col0 + it.kvh * p.v_col_step + h * 64, row);
                __syncwarp();
                sl.next();
                if (L::kQBufs > 1 && j == ask && e + 1 < n_items && !load_q(e + 1)) goto leave;
            }
        }
    } else if (STORE) {
        FaCopy copy;
        copy.start(p, parts, lane);
        while (copy.part(p, parts, lane)) {}
    }
leave:
    __syncwarp();
    if (*reinterpret_cast<volatile uint32_t*>(smem + L::kOffBar + BAR_DEAD))      // gave up: let copies that are still in flight land first
        for (int i = 0; i < 1000; ++i) __nanosleep(1000);
    tc_fence_before();
    __syncthreads();
    if (warp == 12) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
}

// Launch; the caller has filled everything but hp / max_rb and built the maps (box of Q: 64 x 128, of K and V: 64 x box_rows or 64 x BN;
// tk2 is only read with 192-wide heads).
template <int DQK, bool PAIR_HEADS, bool GENERAL, bool STORE = false>
int fa_launch(FaParams& p, const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& tk2, int total_q, int max_seqlen_q,
              cudaStream_t stream) {
    constexpr int RT = PAIR_HEADS ? BM : 2 * BM;
    p.hp = PAIR_HEADS ? p.hq / 2 : p.hq;
    p.max_rb = (max_seqlen_q + RT - 1) / RT;
    if (const int rc = b200wait::launch_word(&p.report); rc != B200_OK) return rc;
    if (p.hp >= 2048 || p.max_rb >= (1 << 20)) return B200_EUNSUPPORTED;
    static B200SmemOptIn optin;
    B200_CUDA_CHECK((b200_ctx*)nullptr, optin.ensure(fa_kernel<DQK, PAIR_HEADS, GENERAL, STORE>, FaSmem<DQK>::kTotal));
    int dev = 0, sms = 0;
    B200_CUDA_CHECK((b200_ctx*)nullptr, cudaGetDevice(&dev));
    B200_CUDA_CHECK((b200_ctx*)nullptr, cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const int64_t bound = (int64_t)p.hp * (total_q / RT + p.num_seqs);
    if (bound > (1ll << 30)) return B200_EUNSUPPORTED;
    int64_t grid = bound < sms ? bound : sms;
    if ((bound + grid - 1) / grid > ITEM_CAP) grid = (bound + ITEM_CAP - 1) / ITEM_CAP;
    B200_LAUNCH((fa_kernel<DQK, PAIR_HEADS, GENERAL, STORE>), dim3((unsigned)grid), THREADS, (FaSmem<DQK>::kTotal), stream, tq, tk, tv, tk2, p);
    return b200_launch_status(nullptr);
}

}  // inline namespace
}  // namespace b200fa
