// All layers of a decode step of up to 8 rows as ONE kernel: embedding, per layer qkv_proj, paged attention, o_proj, gate_up_proj + SiluAndMul,
// down_proj with the norms between them (reference models/qwen3.py:146-175), and the final norm.
//
// What bounds such a step: its weights (31 MB a layer at hidden 1024) stream in 5 us, but a layer is a chain of five products that each need all of the one
// before.  As five launches each link cost 4-5 us: launch, ramp-up, loads of x behind the dependency wait, drain.  Here every SM has one CTA for the
// whole step, and a link is one exchange through L2 plus the products' own chain, 3.1 us in all at 1 row and 3.4 at 4 (433 and 470 us for the 140 of 28 layers, contexts of 60 tokens):
//   * Weights: a warp of each CTA copies the CTA's tiles of all layers, in the order of their use, into a ring in shared memory; it never waits for the exchanges, only for
//     free slots.  A tile is 8 rows of W, the 8-column side of mma.sync; the rows of x are the other side.  (One tcgen05 tile is 128 rows: with so few the
//     tensor rate is idle either way.)  A chain of 64 products takes 1600 cycles with one accumulator, the launches' order; two would
//     be shorter and no less exact, with other roundings than theirs.
//   * Exchange: a result travels as 8 bytes, two bf16 (or one fp32) and the layer's number + 1, stored and loaded whole; who needs it polls for the number.  No
//     barrier, no fence, no second trip for the data.  The buffers start as zeros.  Each is used again in every layer: whoever writes it has, through the
//     chain of products, waited for everybody who read it the layer before (each reader publishes something afterwards that all of the next writers need; a CTA
//     without tiles of the wide products reads no norms' inputs).  One way takes 0.36 us between two CTAs, 1.3-1.6 us as 148 of them ask for the same lines.
//   * Keys and values of the cache do not depend on the step: a warp's first chunks are on their way to L2 a layer ahead, the others two chunks ahead.  Contexts are cut over
//     CTAs as in decode_small.cu; the first CTA of a context adds the parts up.
//   * The residual stream stays in shared memory, a copy per CTA: every CTA forms the norms for itself.
//   * A warp's own chain of instructions is half of a link's time (27 % of the issue slots at 4 rows of 1024 tokens, nothing else busy), so they are counted: loads without branches, no spilled register (with 28 KB
//     of L1 beside the ring each reload is a trip to L2: 500 bytes of them made the step 1.4 times as long).
// Every sum has the order of the launches it replaces (linear_rows.cu, decode_small.cu): the results are theirs bit for bit.  Captured Qwen3-0.6B step, contexts of 100-1024
// tokens, us, those launches / this kernel: 1 row 590 / 493, 2 rows 737 / 508, 4 rows 672 / 567, 8 rows 746 / 676; contexts of 16-64 tokens, 1 row 582 / 490.  16 rows took 979
// / 1160 (twice the exchange and the chunks of a warp one after the other), so they keep their launches.  Long contexts: at sr_splits.
// CTAs wait for one another: launched cooperatively, one per SM.  Waits are bounded (wait_report.cuh).
#include "decode_walk.cuh"
#include "tc_common.cuh"

using namespace b200dec;

bool b200_decode_forced_mma();                      // decode_attn.cu

namespace {

using b200tc::mbar_try;

constexpr int SR_WARPS = SW;                       // compute warps; of another warpgroup one copies weights
constexpr int SR_THREADS = (SR_WARPS + 4) * 32;    // 168 registers each at launch, 64512 in all: 24 for the copying warpgroup, 240 for the two that compute
constexpr int SR_COLS = 1024;                      // k columns of a ring slot
constexpr int SR_PITCH = SR_COLS + 8;              // elements: rows start 16 bytes further in the banks each
constexpr int SR_SLOT = 8 * SR_PITCH * 2;
constexpr int SR_HIDDEN = 1024;                    // widest residual stream
constexpr int SR_K = 3 * SR_COLS;                  // widest input of o_proj and down_proj
constexpr int SR_MAX_LAYERS = 64;
constexpr int SR_MAX_CHUNKS = 128;                 // of one CTA's part of a context
// Chunks a warp has on their way to L2, of the next layer and along its walk (there is no second pair of registers for the next chunk).  Four of the next layer and none along the walk
// cost from the fifth chunk on what memory takes to answer (8 rows of 4096 tokens, without the LM head, us: 1260 for the launches' 1202); 4 and 4 1167, 4 and 2 1143, 4 and 6 1259, 2 and 2
// 1110, asked for in front of the scores, and 1088 behind the values' loads.
constexpr int SR_AHEAD = 2;

constexpr int SR_SLOTS = 10;
constexpr int SR_ROWS = 8;                         // one side of mma.sync

__host__ __device__ constexpr int sr_part(int gw) { return gw * (1 + B200_HEAD_DIM / 2); }     // pairs of units of a CTA's part of a context
static_assert(7 * sr_part(2) <= 4 * SR_WARPS * 32 && 7 * sr_part(2) * 8 <= 8 * SR_PITCH * 2, "parts of a context");

template <int GW>
struct SrSmem {
    static constexpr int kRing = 0;
    static constexpr int kX = SR_SLOTS * SR_SLOT;                                  // normed rows
    static constexpr int kRes = kX + SR_ROWS * SR_PITCH * 2;                            // residual rows
    static constexpr int kNorm = kRes + SR_ROWS * SR_HIDDEN * 2;                        // two layers' norm weights
    static constexpr int kNormBytes = 2 * SR_HIDDEN * 2 + 2 * B200_HEAD_DIM * 2;
    static constexpr int kRed = kNorm + 2 * kNormBytes;
    static constexpr int kSums = kRed + SR_WARPS * 32 * 8;                             // rows' sums of squares
    static constexpr int kO = kSums + SR_ROWS * 16;
    static constexpr int kMl = kO + SW * GW * B200_HEAD_DIM * 4;
    static constexpr int kQ = kMl + SW * GW * 2 * 4;                                   // queries, the step's own key and value
    static constexpr int kPages = kQ + (GW + 2) * B200_HEAD_DIM * 4;
    static constexpr int kBars = kPages + SR_MAX_CHUNKS * 4;                           // full, empty per slot; norm full, norm empty per layer parity; dead
    static constexpr int kTotal = kBars + (2 * SR_SLOTS + 4) * 8 + 16;
};
static_assert(SrSmem<2>::kTotal <= 227 * 1024, "shared memory");

struct SrLayer {
    const __nv_bfloat16 *qkv, *o, *gate_up, *down, *ln1, *ln2, *q_norm, *k_norm;
};
struct SrParams {
    SrLayer layer[SR_MAX_LAYERS];
    const int64_t* ids;
    const __nv_bfloat16* embed;
    int64_t vocab;
    const __nv_bfloat16* final_norm;
    const float* cos_sin;
    const int32_t* block_tables;
    const int32_t* context_lens;
    __nv_bfloat16 *k_base, *v_base, *out;
    int64_t layer_elems;
    uint8_t *xq, *xpart, *xt, *xo, *xa, *xd;                // exchange buffers: qkv, parts of a context, attention, o, act, down
    uint32_t* report;
    int layers, rows, hidden, inter, hq, hkv, bt_stride, block_shift, splits;
    float eps, scale_log2;
};

// ---- the exchange: 8 bytes {value, tag} ----------------------------------------------------------------------------------
__device__ __forceinline__ void put(uint8_t* p, uint32_t value, uint32_t tag) {
    asm volatile("{\n\t.reg .b64 u;\n\tmov.b64 u, {%1, %2};\n\tst.relaxed.gpu.global.b64 [%0], u;\n\t}" ::"l"(p), "r"(value), "r"(tag) : "memory");
}
// two units next to each other; each is whole by itself.  Zero when both have come
__device__ __forceinline__ uint32_t get2(const uint8_t* p, uint32_t tag, uint32_t& v0, uint32_t& v1) {
    uint32_t t0, t1;
    asm volatile("{\n\t.reg .b64 a, b;\n\tld.relaxed.gpu.global.v2.b64 {a, b}, [%4];\n\tmov.b64 {%0, %1}, a;\n\tmov.b64 {%2, %3}, b;\n\t}"
                 : "=r"(v0), "=r"(t0), "=r"(v1), "=r"(t1)
                 : "l"(p)
                 : "memory");
    return (t0 ^ tag) | (t1 ^ tag);
}
// ... where `on`, else zeros; not a branch: loads that follow one another go out together
__device__ __forceinline__ uint32_t get2_if(const uint8_t* p, uint32_t tag, uint32_t& v0, uint32_t& v1, bool on) {
    uint32_t t0, t1;
    asm volatile("{\n\t.reg .pred w;\n\t.reg .b64 a, b;\n\tsetp.ne.u32 w, %5, 0;\n\tmov.b64 a, 0;\n\tmov.b64 b, 0;\n\t@w ld.relaxed.gpu.global.v2.b64 {a, b}, [%4];\n\t"
                 "mov.b64 {%0, %1}, a;\n\tmov.b64 {%2, %3}, b;\n\t}"
                 : "=r"(v0), "=r"(t0), "=r"(v1), "=r"(t1)
                 : "l"(p), "r"((uint32_t)on)
                 : "memory");
    return on ? (t0 ^ tag) | (t1 ^ tag) : 0u;
}

// A warp's waits: true when one is to end unanswered, after so many looks (seconds) or because some wait of this CTA gave up.  No call: what its callers' registers would
// cost is paid in every layer.
struct Patience {
    uint32_t dead, *report;
    uint32_t n = 0;
    __device__ __forceinline__ bool over(uint32_t limit) {
        if (++n & 63) return false;
        uint32_t d;
        asm volatile("ld.volatile.shared.u32 %0, [%1];" : "=r"(d) : "r"(dead) : "memory");
        if (n >= limit && !d && (threadIdx.x & 31) == 0) {
            asm volatile("st.volatile.shared.u32 [%0], %1;" ::"r"(dead), "r"(1u) : "memory");
            *static_cast<volatile uint32_t*>(report) = 1 + *static_cast<volatile uint32_t*>(report);    // two at once may count as one: the word has moved all the same
            __threadfence_system();
        }
        return __any_sync(0xffffffffu, d || n >= limit);
    }
};
constexpr uint32_t SR_POLLS = 1u << 22, SR_TESTS = 1u << 26;             // of a third of a microsecond and more; of some ten nanoseconds
__device__ __forceinline__ bool wait(uint32_t bar, uint32_t parity, uint32_t dead, uint32_t* report) {
    Patience patience{dead, report};
    uint32_t ok;
    do {
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.b32 %0, 1, 0, p;\n\t}" : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
        ok = __all_sync(0xffffffffu, ok);
    } while (!ok && !patience.over(SR_TESTS));
    return ok;
}
// N pairs of units per lane: pair i at at(i) where use(i), which is the same for all lanes (ALL: always).  `one` >= 0: that pair of the warp's is waited for first, by one lane, another
// one in each CTA; for what all 148 CTAs wait for (the norms' inputs) that is faster, everything else is asked for at once (first one pair everywhere: 1 row 512 us a step, 4
// rows 594, 8 rows 717; nowhere 500, 578, 705; for the norms alone 494, 576, 698).
template <int N, bool ALL, typename At, typename Use>
__device__ __forceinline__ void get_pairs(uint32_t (&v)[N][2], At at, Use use, uint32_t tag, uint32_t dead, uint32_t* report, int one = -1) {
    Patience patience{dead, report};
    uint32_t a, b, bad;
    if (one >= 0) {
        const bool asks = (threadIdx.x & 31) == (blockIdx.x & 31);
        do bad = get2_if(at(one), tag, a, b, asks);
        while (__any_sync(0xffffffffu, bad) && !patience.over(SR_POLLS));
    }
    do {
        bad = 0;
#pragma unroll
        for (int i = 0; i < N; ++i) bad |= ALL ? get2(at(i), tag, v[i][0], v[i][1]) : get2_if(at(i), tag, v[i][0], v[i][1], use(i));
    } while (__any_sync(0xffffffffu, bad) && !patience.over(SR_POLLS));
}

__device__ __forceinline__ void mma_x(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldsm4(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void compute_sync() { asm volatile("bar.sync 1, 256;" ::: "memory"); }      // the compute warps
__device__ __forceinline__ void arrive(uint32_t bar, int count) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(count) : "memory"); }

// Tiles t = first, first + grid, ... of n: how many
__device__ __forceinline__ int tiles_of(int n, int first, int grid) { return first < n ? (n - 1 - first) / grid + 1 : 0; }

// GW: query heads per kv head.
template <int GW>
__global__ void __launch_bounds__(SR_THREADS, 1) step_rows_kernel(const __grid_constant__ SrParams p) {
    using L = SrSmem<GW>;
    constexpr int D = B200_HEAD_DIM, SLOTS = SR_SLOTS, PART = sr_part(GW);
    extern __shared__ __align__(128) unsigned char sm[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, q = lane & 3, cta = blockIdx.x, grid = gridDim.x;
    const int rows = p.rows, hidden = p.hidden, q_size = p.hq * D, n_qkv = (p.hq + 2 * p.hkv) * D, inter = p.inter;
    const uint32_t ring = smem_u32(sm + L::kRing), full = smem_u32(sm + L::kBars), empty = full + SLOTS * 8, nfull = empty + SLOTS * 8, nempty = nfull + 16, dead = nempty + 16;
    if (tid == 0) {
#pragma unroll 1
        for (int i = 0; i < SLOTS; ++i) mbar_init(full + i * 8, 1), mbar_init(empty + i * 8, SR_WARPS);
#pragma unroll 1
        for (int i = 0; i < 2; ++i) mbar_init(nfull + i * 8, 1), mbar_init(nempty + i * 8, 1);
        *reinterpret_cast<uint32_t*>(sm + L::kBars + (2 * SLOTS + 4) * 8) = 0;
        mbar_fence_init();
    }
    __syncthreads();
    // This CTA's tiles: of the wide products from the front, of the narrow ones from the back, so that no CTA has the most of both
    const int back = grid - 1 - cta;
    const int n1 = tiles_of(n_qkv / 8, cta, grid), n4 = tiles_of(inter / 4, cta, grid), n3 = tiles_of(hidden / 8, back, grid);     // n3: of o_proj, and of down_proj

    if (warp >= SR_WARPS) {                        // ---- weights, in the order of their use ----
        asm volatile("setmaxnreg.dec.sync.aligned.u32 24;");
        if (warp > SR_WARPS) return;
        const uint64_t policy = l2_policy_evict_first();                 // read once a step: what waits in L2 for its use are keys and values
        uint32_t it = 0;
        bool alive = true;
        int l = 0;
        auto issue = [&](const __nv_bfloat16* row0, const __nv_bfloat16* row4, int64_t stride, int cols) {   // rows 0-3 and 4-7 of a tile, from row0 and row4 on
            const int s = it % SLOTS;
            if (it >= SLOTS) alive = alive && wait(empty + s * 8, (it / SLOTS - 1) & 1, dead, p.report);
            if (!alive) return;
            if (lane == 0) mbar_expect_tx(full + s * 8, 8 * cols * 2);
            __syncwarp();
            if (lane < 8) bulk_g2s_hint(ring + s * SR_SLOT + lane * SR_PITCH * 2, (lane < 4 ? row0 : row4) + (lane & 3) * stride, cols * 2, full + s * 8, policy);
            ++it;
        };
#pragma unroll 1
        for (; l < p.layers && alive; ++l) {
            const SrLayer& w = p.layer[l];
            const uint32_t bar = nfull + (l & 1) * 8, dst = smem_u32(sm + L::kNorm) + (l & 1) * L::kNormBytes;
            if (l >= 2) alive = wait(nempty + (l & 1) * 8, ((l >> 1) - 1) & 1, dead, p.report);
            if (!alive) break;
            if (lane == 0) {
                mbar_expect_tx(bar, 2 * hidden * 2 + 2 * D * 2);
                bulk_g2s(dst, w.ln1, hidden * 2, bar);
                bulk_g2s(dst + SR_HIDDEN * 2, w.ln2, hidden * 2, bar);
                bulk_g2s(dst + 2 * SR_HIDDEN * 2, w.q_norm, D * 2, bar);
                bulk_g2s(dst + 2 * SR_HIDDEN * 2 + D * 2, w.k_norm, D * 2, bar);
            }
            __syncwarp();
#pragma unroll 1
            for (int m = 0; m < 4; ++m) {          // qkv, o, gate_up (4 gate rows, 4 up rows), down
                const __nv_bfloat16* base = m == 0 ? w.qkv : m == 1 ? w.o : m == 2 ? w.gate_up : w.down;
                const int k = m == 1 ? q_size : m == 3 ? inter : hidden, per = m == 2 ? 4 : 8;
                const int tiles = (m == 0 ? n_qkv : m == 2 ? inter : hidden) / per;
                const int64_t up = (int64_t)(m == 2 ? inter : 4) * k;
#pragma unroll 1
                for (int t = m & 1 ? back : cta; t < tiles; t += grid) {
                    const __nv_bfloat16* row = base + (int64_t)t * per * k;
#pragma unroll 1
                    for (int c = 0; c < k; c += SR_COLS) issue(row + c, row + up + c, k, min(SR_COLS, k - c));
                }
            }
        }
        if (!alive) {                              // nobody waits for them any more: the copies in flight still have to land in this CTA's memory
            uint64_t t0, t1;
            asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t0));
            auto land = [&](uint32_t b, uint32_t parity) {
                do asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t1));
                while (!mbar_try(b, parity) && t1 - t0 < 2000000000ull);
            };
#pragma unroll 1
            for (uint32_t i = it > SLOTS ? it - SLOTS : 0; i < it; ++i) land(full + i % SLOTS * 8, i / SLOTS & 1);
#pragma unroll 1
            for (int i = max(l - 2, 0); i < l; ++i) land(nfull + (i & 1) * 8, i >> 1 & 1);
            if (l < p.layers && it > 0) land(nfull + (l & 1) * 8, l >> 1 & 1);
        }
        return;
    }

    asm volatile("setmaxnreg.inc.sync.aligned.u32 240;");
    // ---- what stays the same over the layers ----
    const int split = rows <= 2 ? 2 : rows <= 4 ? 1 : 0;                                // 1 << split warps per row in the norms
    const bool wide = n1 || n4;                    // has tiles of the wide products: needs the norms
    uint4* res = reinterpret_cast<uint4*>(sm + L::kRes);                               // [row][hidden / 8]
    unsigned char* xs = sm + L::kX;
    const float per_hidden = 1.0f / (float)hidden; // a power of two: exact
    const int pieces = hidden / 8, xrow = (hidden + 8) * 2;
    float2(*red)[32] = reinterpret_cast<float2(*)[32]>(sm + L::kRed);
    float(*sums)[4] = reinterpret_cast<float(*)[4]>(sm + L::kSums);
    auto& sh_o = *reinterpret_cast<float(*)[SW][GW][D]>(sm + L::kO);
    auto& sh_ml = *reinterpret_cast<float(*)[SW][GW][2]>(sm + L::kMl);
    auto& sh_q = *reinterpret_cast<float(*)[GW + 2][D]>(sm + L::kQ);
    int* pages = reinterpret_cast<int*>(sm + L::kPages);
    uint32_t item = 0;                             // ring items used up so far
    // attention: this CTA's part (rank of splits) of a (sequence, kv head)
    const WalkLane wl(lane);
    const int unit = cta / p.splits, rank = cta % p.splits, b = unit / p.hkv, kvh = unit % p.hkv;
    const bool attends = unit < rows * p.hkv;
    int ctx = 0, old = 0, c0 = 0, c1 = 0;
    const int mask = (1 << p.block_shift) - 1;
    if (attends) {
        ctx = min(max(p.context_lens[b], 0), p.bt_stride << p.block_shift);
        old = max(ctx - 1, 0);
        const int n = (old + CHUNK - 1) / CHUNK;
        c0 = (int)((int64_t)n * rank / p.splits), c1 = min((int)((int64_t)n * (rank + 1) / p.splits), c0 + SR_MAX_CHUNKS);
#pragma unroll 1
        for (int i = tid; i < c1 - c0; i += SR_WARPS * 32) pages[i] = p.block_tables[(int64_t)b * p.bt_stride + ((c0 + i) * CHUNK >> p.block_shift)];
    }
    if (wide) {
#pragma unroll 1
        for (int t = warp; t < rows; t += SR_WARPS) {                                  // an id that is not a token embeds to zeros
            const int64_t id = p.ids[t];
            const bool ok = id >= 0 && id < p.vocab;
            const uint4* src = reinterpret_cast<const uint4*>(p.embed + (ok ? id : 0) * hidden);
#pragma unroll 1
            for (int c = lane; c < pieces; c += 32) res[t * pieces + c] = ok ? src[c] : make_uint4(0, 0, 0, 0);
        }
    }
    compute_sync();
    auto row_of = [&](int ck) -> int64_t { return (((int64_t)pages[ck - c0] * p.hkv + kvh) << p.block_shift) + (ck * CHUNK & mask); };   // first cache row of a chunk
    const int64_t own_row = attends && ctx > 0 ? (((int64_t)p.block_tables[(int64_t)b * p.bt_stride + (old >> p.block_shift)] * p.hkv + kvh) << p.block_shift) + (old & mask) : -1;
    auto to_l2 = [&](const __nv_bfloat16* k_layer, const __nv_bfloat16* v_layer, int ck) {             // a chunk's 32 lines of 128 bytes of keys, and of values
        const int64_t r = ck < c1 ? row_of(ck) : -1;
        if (r < 0) return;
        asm volatile("prefetch.global.L2 [%0];" ::"l"(k_layer + r * D + lane * 64));
        asm volatile("prefetch.global.L2 [%0];" ::"l"(v_layer + r * D + lane * 64));
    };
    auto load_chunk = [&](const __nv_bfloat16* layer, int ck, uint4 (&x)[8]) {
        const int64_t at = ck < c1 ? row_of(ck) : -1;                                  // behind the last chunk, or on an absent page: zeros
        walk_load(wl, layer, at, at < 0 ? 0 : old - ck * CHUNK, x);
    };

    // rmsnorm(residual + what `add` brings) * w -> dst rows (pitch in bytes); the residual becomes bf16 of the sum.  1 << split warps share a row, whose columns are four
    // pieces of 8 a lane; their sums of squares are added in the norm kernels' order.
    auto norm = [&](const uint8_t* add, uint32_t tag, const uint4* w4, bool one_sum, int split, unsigned char* dst, int pitch) {
        const int t = warp >> split, part = warp & ((1 << split) - 1);
        const bool row = t < rows;
        auto mine = [&](int i) { return row && i >> (2 - split) == part && i * 32 < pieces; };
        float f[4][8], ss[4] = {0.f, 0.f, 0.f, 0.f};
        uint32_t v[8][2];
        if (add && mine(part << (2 - split))) {
            const uint8_t* at = add + (t * (hidden / 2) + lane * 4) * 8;
            get_pairs<8, false>(v, [&](int i) { return at + (i >> 1) * 1024 + (i & 1) * 16; }, [&](int i) { return mine(i >> 1); }, tag, dead, p.report, part << (3 - split));
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (!mine(i)) continue;
            unpack8(res[t * pieces + lane + 32 * i], f[i]);
            if (add) {
                float e[8];
                unpack8(make_uint4(v[2 * i][0], v[2 * i][1], v[2 * i + 1][0], v[2 * i + 1][1]), e);
#pragma unroll
                for (int k = 0; k < 8; ++k) f[i][k] += e[k];
            }
            float s = one_sum ? ss[0] : ss[i];
#pragma unroll
            for (int e = 0; e < 8; ++e) s = fmaf(f[i][e], f[i][e], s);
            if (one_sum) ss[0] = s;
            else ss[i] = s;
        }
        if (split == 0) {
#pragma unroll
            for (int i = 0; i < 4; ++i) ss[i] = warp_sum(ss[i]);
        } else {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                if (i >> (2 - split) != part) continue;
                ss[i] = warp_sum(ss[i]);
                if (lane == 0 && row) sums[t][i] = ss[i];
            }
            compute_sync();
#pragma unroll
            for (int i = 0; i < 4; ++i) ss[i] = row ? sums[t][i] : 0.f;
        }
        const float rstd = 1.0f / sqrtf((ss[0] + ss[1] + ss[2] + ss[3]) * per_hidden + p.eps);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (!mine(i)) continue;
            const int c = lane + 32 * i;
            if (add) res[t * pieces + c] = pack8(f[i]);
            float w[8];
            unpack8(w4[c], w);
#pragma unroll
            for (int e = 0; e < 8; ++e) f[i][e] = __fmul_rn(__fmul_rn(f[i][e], rstd), w[e]);
            reinterpret_cast<uint4*>(dst + t * pitch)[c] = pack8(f[i]);
        }
    };

    // One chain of products over hidden columns: xs times the tile in ring slot s (a warp)
    auto wide_chain = [&](uint32_t slot, float (&acc)[4]) {
        const uint32_t wa = slot + (lane & 7) * SR_PITCH * 2 + (lane >> 3) * 16, xa = smem_u32(xs) + (lane & 7) * xrow + (lane >> 3) * 16;
        uint32_t w[4][4], x[4][4];                 // four steps of 32: three are on their way while one's products run
        auto load = [&](int c, int u) { ldsm4(wa + u * 64, w[c]), ldsm4(xa + u * 64, x[c]); };
        auto products = [&](int c) {
            mma_x(acc, x[c][0], 0u, x[c][1], 0u, w[c][0], w[c][1]);
            mma_x(acc, x[c][2], 0u, x[c][3], 0u, w[c][2], w[c][3]);
        };
        const int steps = hidden / 32;             // a multiple of four
#pragma unroll
        for (int c = 0; c < 3; ++c) load(c, c);
#pragma unroll 1
        for (int u = 0; u < steps; u += 4) {
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                if (u + c + 3 < steps) load((c + 3) & 3, u + c + 3);
                products(c);
            }
        }
    };

    // One tile of a product with hidden outputs: eight chains, a warp each, over k / 8 columns.  The first weights are in registers when x comes, straight from its
    // exchange buffer, whose blocks of 16 columns hold the units of the mma's operand in a lane's order: [block][row of 8][unit 0 4 1 5 2 6 3 7].
    auto narrow = [&](auto THOUSANDS, const uint8_t* x, uint32_t tag, uint8_t* out, int t) {
        constexpr int slots = decltype(THOUSANDS)::value, steps = slots * SR_COLS / 128, kw = slots * SR_COLS / 8;       // 16-column steps of a chain
#pragma unroll 1
        for (int s = 0; s < slots; ++s) wait(full + (item + s) % SLOTS * 8, (item + s) / SLOTS & 1, dead, p.report);
        const uint32_t wa = ring + (lane & 7) * SR_PITCH * 2 + (lane >> 3) * 16;
        uint32_t w[4][4], v[steps][2];
        auto load = [&](int i) {                                                        // 32 columns: within a slot
            const int col = warp * kw + i * 32;
            ldsm4(wa + (item + col / SR_COLS) % SLOTS * SR_SLOT + col % SR_COLS * 2, w[i & 3]);
        };
#pragma unroll
        for (int i = 0; i < 4; ++i) load(i);
        // rows that do not exist are some row's values, and not stored
        const uint8_t* at = x + ((warp * steps * SR_ROWS + min(g, rows - 1)) * 8 + 2 * q) * 8;
        get_pairs<steps, true>(v, [&](int i) { return at + i * (SR_ROWS * 64); }, [](int) { return true; }, tag, dead, p.report);
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int i = 0; i < steps / 2; ++i) {
            mma_x(acc, v[2 * i][0], 0u, v[2 * i][1], 0u, w[i & 3][0], w[i & 3][1]);
            mma_x(acc, v[2 * i + 1][0], 0u, v[2 * i + 1][1], 0u, w[i & 3][2], w[i & 3][3]);
            if (i + 4 < steps / 2) load(i + 4);
        }
        if (lane == 0) {
#pragma unroll 1
            for (int s = 0; s < slots; ++s) arrive(empty + (item + s) % SLOTS * 8, 1);
        }
        red[warp][lane] = make_float2(acc[0], acc[1]);
        compute_sync();
        if (warp == 0) {
            float2 sum = make_float2(0.f, 0.f);
#pragma unroll
            for (int i = 0; i < SR_WARPS; ++i) {
                const float2 a = red[i][lane];
                sum.x += a.x, sum.y += a.y;
            }
            if (g < rows) put(out + ((int64_t)g * (hidden / 2) + t * 4 + q) * 8, pack_bf16x2(sum.x, sum.y), tag);
        }
        item += slots;
    };
    auto narrow_tiles = [&](const uint8_t* x, int k, uint32_t tag, uint8_t* out) {
#pragma unroll 1
        for (int t = back; t < hidden / 8; t += grid) {
            if (t != back) compute_sync();         // red[] has been read
            if (k == 2 * SR_COLS) narrow(std::integral_constant<int, 2>{}, x, tag, out, t);
            else if (k == 3 * SR_COLS) narrow(std::integral_constant<int, 3>{}, x, tag, out, t);
            else narrow(std::integral_constant<int, 1>{}, x, tag, out, t);
        }
    };
    // where a pair of columns (2 u, 2 u + 1) of a row sits in such a buffer
    auto unit_of = [&](uint8_t* x, int row, int u) { return x + (((u >> 3) * SR_ROWS + row) * 8 + ((u & 3) * 2 + (u >> 2 & 1))) * 8; };

    // Layer by layer, in two halves: norm, a wide product, (attention,) a narrow one.  One layer on, the final norm.
#pragma unroll 1
    for (int step = 0; step <= 2 * p.layers; ++step) {
        const int l = step >> 1;
        const bool second = step & 1, last = l == p.layers;
        const uint32_t tag = l + 1;
        if (last && cta) break;
        const unsigned char* nw = sm + L::kNorm + (l & 1) * L::kNormBytes;
        if (!second && !last) wait(nfull + (l & 1) * 8, l >> 1 & 1, dead, p.report);
        if (wide) {
            const int n = second ? n4 : n1;
            const uint32_t s0 = (item + warp) % SLOTS;
            if (!last && warp < n) wait(full + s0 * 8, (item + warp) / SLOTS & 1, dead, p.report);
            // residual + down_proj (or, second, o_proj)
            norm(second ? p.xo : l ? p.xd : nullptr, second ? tag : tag - 1, last ? reinterpret_cast<const uint4*>(p.final_norm) : reinterpret_cast<const uint4*>(nw + (second ? SR_HIDDEN * 2 : 0)),
                 step == 0, step ? split : 0, last ? reinterpret_cast<unsigned char*>(p.out) : xs, last ? hidden * 2 : xrow);
            if (last) break;
            compute_sync();
            if (warp < n) {                        // at most a tile a warp
                float acc[4] = {0.f, 0.f, 0.f, 0.f};
                wide_chain(ring + s0 * SR_SLOT, acc);
                const int t = cta + warp * grid;
                uint8_t* to = p.xq + ((int64_t)g * (n_qkv / 2) + t * 4 + q) * 8;
                if (second) {                      // lanes q = 0, 1 of a row have four gate columns, q = 2, 3 the up columns
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const float z = round_bf16(acc[e]), u = __shfl_xor_sync(0xffffffffu, z, 2);
                        acc[e] = __fmul_rn(z / (1.0f + expf(-z)), u);
                    }
                    to = unit_of(p.xa, g, t * 2 + q);
                }
                if (g < rows && !(second && q >= 2)) put(to, pack_bf16x2(acc[0], acc[1]), tag);
                __syncwarp();
                if (lane == 0) arrive(empty + s0 * 8, SR_WARPS);
            }
            item += n;
        } else if (!last) {
            compute_sync();                        // for the norm weights, which attention reads too
        }
        if (second && tid == 0) arrive(nempty + (l & 1) * 8, 1);
        if (!second && attends) {
            const int j = wl.j;
            const __nv_bfloat16 *k_layer = p.k_base + l * p.layer_elems, *v_layer = p.v_base + l * p.layer_elems;
            uint4 kr[8], vr[8];                    // no second pair of registers for the next chunk: it is in L2
            load_chunk(k_layer, c0 + warp, kr);
            load_chunk(v_layer, c0 + warp, vr);
            WalkState<GW> st;
            {                                      // a warp per query head, one for the key, one for the value
                float f[8];
                if (warp < GW + 2) {
                    const int head = warp < GW ? kvh * GW + warp : p.hq + (warp - GW) * p.hkv + kvh;
                    const uint8_t* at = p.xq + ((int64_t)b * (n_qkv / 2) + head * (D / 2) + j * 4) * 8;
                    float cosr[8], sinr[8], nw8[8];
                    const float4* cs = reinterpret_cast<const float4*>(p.cos_sin + (int64_t)old * D + (j & 7) * 8);
                    const float4 ca = cs[0], cb = cs[1], sa = cs[16], sb = cs[17];
                    cosr[0] = ca.x, cosr[1] = ca.y, cosr[2] = ca.z, cosr[3] = ca.w, cosr[4] = cb.x, cosr[5] = cb.y, cosr[6] = cb.z, cosr[7] = cb.w;
                    sinr[0] = sa.x, sinr[1] = sa.y, sinr[2] = sa.z, sinr[3] = sa.w, sinr[4] = sb.x, sinr[5] = sb.y, sinr[6] = sb.z, sinr[7] = sb.w;
                    uint32_t v[2][2];
                    get_pairs<2, true>(v, [&](int i) { return at + i * 16; }, [](int) { return true; }, tag, dead, p.report);
                    const uint4 raw = make_uint4(v[0][0], v[0][1], v[1][0], v[1][1]);
                    unpack8(raw, f);
                    if (warp <= GW) {
                        unpack8(reinterpret_cast<const uint4*>(nw + 2 * SR_HIDDEN * 2 + (warp == GW ? D * 2 : 0))[j], nw8);
                        walk_norm_rope(wl, f, nw8, cosr, sinr, p.eps);
                    }
                    if (wl.hw == 0) {
                        *reinterpret_cast<float4*>(&sh_q[warp][j * 8]) = make_float4(f[0], f[1], f[2], f[3]);
                        *reinterpret_cast<float4*>(&sh_q[warp][j * 8 + 4]) = make_float4(f[4], f[5], f[6], f[7]);
                        // the step's own token, appended by the context's last CTA
                        if (warp >= GW && rank == p.splits - 1 && own_row >= 0)
                            *reinterpret_cast<uint4*>((warp == GW ? p.k_base : p.v_base) + l * p.layer_elems + own_row * D + j * 8) = warp == GW ? pack8(f) : raw;
                    }
                }
                compute_sync();
            }
            auto fetch = [&](int r, float (&f)[8]) {
                const float4 a = *reinterpret_cast<const float4*>(&sh_q[r][j * 8]), b4 = *reinterpret_cast<const float4*>(&sh_q[r][j * 8 + 4]);
                f[0] = a.x, f[1] = a.y, f[2] = a.z, f[3] = a.w, f[4] = b4.x, f[5] = b4.y, f[6] = b4.z, f[7] = b4.w;
            };
#pragma unroll
            for (int h = 0; h < GW; ++h) fetch(h, st.q[h]);
            st.begin(p.scale_log2);
#pragma unroll 1
            for (int ck = c0 + warp; ck < c1; ck += SW) {
                float acc[GW][8];
                st.scores(kr, acc);
                load_chunk(k_layer, ck + SW, kr);
                st.values(wl, acc, vr, old - ck * CHUNK);
                load_chunk(v_layer, ck + SW, vr);
                to_l2(k_layer, v_layer, ck + SR_AHEAD * SW);
            }
            if (ctx > 0 && rank == p.splits - 1 && warp == SW - 1) {                   // the step's own token
                float kn[8], vn[8];
                fetch(GW, kn);
                fetch(GW + 1, vn);
                st.own(wl, kn, vn);
            }
            st.leave(wl, sh_o[warp], sh_ml[warp]);
            compute_sync();
            float M = 0.f, S = 0.f, a = 0.f;
            const int h = tid / D, d = tid % D;
            const bool mine = tid < GW * D;        // whole warps
            if (mine) walk_meet<GW>(sh_o, sh_ml, h, d, M, S, a);
            uint8_t* part = p.xpart + (int64_t)cta * PART * 16;                        // GW pairs (max, sum), then the results
            if (rank) {                            // to the first CTA of this context
                if (mine) {
                    put(part + (GW * 2 + tid) * 8, __float_as_uint(a), tag);
                    if (d < 2) put(part + (h * 2 + d) * 8, __float_as_uint(d ? S : M), tag);
                }
            } else {
                if (p.splits > 1) {
                    // all pairs of the other parts, four a thread, into shared memory (xs is not in use); then in order, as decode_small.cu adds them
                    float2* got = reinterpret_cast<float2*>(xs);
                    const int pairs = (p.splits - 1) * PART;
                    uint32_t v[4][2];
                    get_pairs<4, false>(v, [&](int i) { return part + (PART + min(tid + i * SR_WARPS * 32, pairs - 1)) * 16; }, [&](int i) { return i * SR_WARPS * 32 < pairs; }, tag, dead, p.report);
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        if (tid + i * SR_WARPS * 32 < pairs) got[tid + i * SR_WARPS * 32] = make_float2(__uint_as_float(v[i][0]), __uint_as_float(v[i][1]));
                    compute_sync();
                    if (mine) {
                        const float m0 = M, s0 = S, a0 = a;
#pragma unroll 1
                        for (int c = 0; c < p.splits - 1; ++c) M = fmaxf(M, got[c * PART + h].x);
                        S = 0.f, a = 0.f;
#pragma unroll 1
                        for (int c = 0; c < p.splits; ++c) {
                            const float2 ms = c ? got[(c - 1) * PART + h] : make_float2(m0, s0);
                            if (ms.x == -INFINITY) continue;
                            const float f = fast_exp2(ms.x - M), o = c ? reinterpret_cast<const float*>(got + (c - 1) * PART + GW)[tid] : a0;
                            S = fmaf(f, ms.y, S);
                            a = fmaf(f, o, a);
                        }
                    }
                }
                if (mine) {
                    const float y = S > 0.f ? a / S : 0.f, y1 = __shfl_xor_sync(0xffffffffu, y, 1);
                    if (!(d & 1)) put(unit_of(p.xt, b, ((kvh * GW + h) * D + d) / 2), pack_bf16x2(y, y1), tag);
                }
            }
        }
        if (n3) {
            compute_sync();                        // the narrow product before has read red[]
            narrow_tiles(second ? p.xa : p.xt, second ? inter : q_size, tag, second ? p.xd : p.xo);
        }
        if (second && attends && l + 1 < p.layers) {                                   // the next layer's keys and values, while the others finish this one
                const __nv_bfloat16 *k_next = p.k_base + (l + 1) * p.layer_elems, *v_next = p.v_base + (l + 1) * p.layer_elems;
#pragma unroll 1
                for (int i = 0, ck = c0 + warp; i < SR_AHEAD && ck < c1; ++i, ck += SW) to_l2(k_next, v_next, ck);
        }
    }
}

struct SrLayout {
    size_t q, part, t, o, a, d, total;
};
SrLayout sr_layout(int sm_count, int rows, int hidden, int inter, int hq, int hkv) {
    SrLayout w;
    size_t at = 0;
    auto take = [&](size_t units) {
        const size_t here = at;
        at += (units * 8 + 255) / 256 * 256;
        return here;
    };
    w.q = take((size_t)rows * (hq + 2 * hkv) * B200_HEAD_DIM / 2);
    w.part = take((size_t)sm_count * sr_part(hq / hkv) * 2);
    w.t = take((size_t)SR_ROWS * hq * B200_HEAD_DIM / 2);
    w.o = take((size_t)rows * hidden / 2);
    w.a = take((size_t)SR_ROWS * inter / 2);
    w.d = take((size_t)rows * hidden / 2);
    w.total = at;
    return w;
}

// Splits of a context, 0 where the step is not this kernel's.  What it takes: one CTA per (sequence, kv head) and split (decode_small.cu's rule, whose sums it repeats), at most a tile
// of the wide products per warp and of the narrow ones per CTA, ring slots that are full.  Up to that rule's longest contexts this kernel is the faster one.  Captured Qwen3-0.6B step without
// the LM head, tables of the widest such context, every row of the length named, us, launches / here: 1 row of 1024 tokens 577 / 460, 4096 678 / 600, 16384 1054 / 1032; 4 rows of 1024 673 / 554,
// 4096 890 / 787, 8192 1184 / 1075; 8 rows of 1024 762 / 648, 2048 910 / 793, 4096 1201 / 1088; rows of a k-th of that each (least gain) 6 rows up to 4096 1073 / 1050.  Hidden 512 with 8 over 8
// or 8 over 4 heads, 1024 with 24 over 12: 1.01 to 1.6 times at every length up to theirs.
int sr_splits(const b200_ctx* ctx, int rows, int layers, int hidden, int inter, int hq, int bt_stride) {
    if (b200_decode_forced_mma()) return 0;
    if (!ctx->k_base || rows <= 0 || rows > SR_ROWS || layers <= 0 || layers > SR_MAX_LAYERS || layers > ctx->layers || hq <= 0 || ctx->num_kv_heads <= 0) return 0;
    const int hkv = ctx->num_kv_heads, G = hq % hkv ? 0 : hq / hkv;
    if (G != 1 && G != 2) return 0;
    if (hidden <= 0 || hidden % 512 || hidden > SR_HIDDEN || inter <= 0 || inter % SR_COLS || inter > SR_K || hq * B200_HEAD_DIM % SR_COLS || hq * B200_HEAD_DIM > SR_K) return 0;
    if (hidden / 8 > ctx->sm_count || ((hq + 2 * hkv) * B200_HEAD_DIM / 8 - 1) / ctx->sm_count >= SR_WARPS || (inter / 4 - 1) / ctx->sm_count >= SR_WARPS) return 0;
    const int splits = b200_decode_small_splits(ctx, rows, hq, bt_stride);
    return splits > 0 ? splits : 0;
}

template <int GW>
int sr_launch(b200_ctx* ctx, const SrParams& p, cudaStream_t st) {
    static B200SmemOptIn optin;
    B200_CUDA_CHECK(ctx, optin.ensure(step_rows_kernel<GW>, SrSmem<GW>::kTotal));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ctx->sm_count);
    cfg.blockDim = dim3(SR_THREADS);
    cfg.dynamicSmemBytes = SrSmem<GW>::kTotal;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;   // all CTAs resident: they wait for one another
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    B200_CUDA_CHECK(ctx, cudaLaunchKernelEx(&cfg, step_rows_kernel<GW>, p));
    return b200_launch_status(ctx);
}

}  // namespace

extern "C" size_t b200_step_rows_workspace_bytes(const b200_ctx* ctx, int rows, int layers, int hidden, int inter, int num_q_heads, int bt_stride) {
    if (!ctx || sr_splits(ctx, rows, layers, hidden, inter, num_q_heads, bt_stride) == 0) return 0;
    return sr_layout(ctx->sm_count, rows, hidden, inter, num_q_heads, ctx->num_kv_heads).total;
}

extern "C" int b200_step_rows(b200_ctx* ctx, const void* const* weights, int layers, const int64_t* ids, const void* embed, int64_t vocab, const void* final_norm,
                              const float* cos_sin, float eps, const int32_t* block_tables, int bt_stride, const int32_t* context_lens, void* out, int rows, int hidden,
                              int inter, int num_q_heads, float scale, void* workspace, size_t workspace_bytes, void* stream) {
    if (!ctx || !weights || !ids || !embed || vocab <= 0 || !final_norm || !cos_sin || !block_tables || !context_lens || !out || !workspace) return B200_EINVAL;
    if (!ctx->k_base) return B200_ENOTBOUND;
    const int splits = sr_splits(ctx, rows, layers, hidden, inter, num_q_heads, bt_stride);
    if (splits == 0) return B200_EUNSUPPORTED;
    const SrLayout w = sr_layout(ctx->sm_count, rows, hidden, inter, num_q_heads, ctx->num_kv_heads);
    if (workspace_bytes < w.total) return B200_EWORKSPACE;
    uintptr_t low = reinterpret_cast<uintptr_t>(embed) | reinterpret_cast<uintptr_t>(final_norm) | reinterpret_cast<uintptr_t>(cos_sin) | reinterpret_cast<uintptr_t>(out) |
                    reinterpret_cast<uintptr_t>(workspace);
    SrParams p = {};
    for (int l = 0; l < layers; ++l) {
        const __nv_bfloat16* v[8];
        for (int i = 0; i < 8; ++i) {
            v[i] = static_cast<const __nv_bfloat16*>(weights[l * 8 + i]);
            if (!v[i]) return B200_EINVAL;
            low |= reinterpret_cast<uintptr_t>(v[i]);
        }
        p.layer[l] = {v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7]};
    }
    if (low & 15) return B200_EUNSUPPORTED;
    uint8_t* ws = static_cast<uint8_t*>(workspace);
    p.ids = ids;
    p.embed = static_cast<const __nv_bfloat16*>(embed);
    p.vocab = vocab;
    p.final_norm = static_cast<const __nv_bfloat16*>(final_norm);
    p.cos_sin = cos_sin;
    p.block_tables = block_tables;
    p.context_lens = context_lens;
    p.k_base = ctx->k_base;
    p.v_base = ctx->v_base;
    p.out = static_cast<__nv_bfloat16*>(out);
    p.layer_elems = (int64_t)ctx->layer_elems();
    p.xq = ws + w.q, p.xpart = ws + w.part, p.xt = ws + w.t, p.xo = ws + w.o, p.xa = ws + w.a, p.xd = ws + w.d;
    p.layers = layers, p.rows = rows, p.hidden = hidden, p.inter = inter, p.hq = num_q_heads, p.hkv = ctx->num_kv_heads;
    p.bt_stride = bt_stride, p.block_shift = ctx->block_shift, p.splits = splits;
    p.eps = eps, p.scale_log2 = scale * 1.4426950408889634f;
    if (const int rc = b200wait::launch_word(&p.report); rc != B200_OK) return rc;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    B200_CUDA_CHECK(ctx, cudaMemsetAsync(workspace, 0, w.total, st));
    const int G = num_q_heads / ctx->num_kv_heads;
    return G == 1 ? sr_launch<1>(ctx, p, st) : sr_launch<2>(ctx, p, st);
}
