// Linear layers of the smallest steps (up to 16 rows), y = x W^T, with the residual add + RMSNorm in front and SiluAndMul behind fused in.
//
// What bounds them: a step of a few rows streams every weight once (31 MB and 5 us a layer at hidden 1024), but as separate kernels (library or tcgen05
// products, partial sums, add + norm, activation) a layer took seven launches of 4-5 us besides attention, each a chain of wait -> fill -> products ->
// drain.  So: four launches, each with its whole share of the weights asked for before it waits for the kernel in front.
//   * Weights go to shared memory by asynchronous copies, all asked for at the start; they are then the 16-row side of mma.sync, rows of x its 8-column
//     side (one or two tiles).  One tcgen05 tile is 128 rows: with so few the tensor rate is idle either way.
//   * The add + norm in front is formed by every CTA for itself, a warp per row of x: 2 x 2 KB a row out of L2 instead of a launch.  One CTA writes the
//     new residual, to a buffer of its own (the others still read the old one).
//   * A sum in parts (o_proj and down_proj) has a warp per part; they meet in shared memory, in order.  Spreading the parts over a cluster of two CTAs, so that
//     128 SMs and not 64 load weights, was 0.4 us a product slower: the weights are there before the rows anyway, and the cluster meets twice.
// Results are those of the launches they replace, bit for bit, not only their rounding points (the projection to bf16, the residual sum to bf16, the normed
// row to bf16, gate and up to bf16): a chain of m16n8k16 products over ascending k gives what the tcgen05 kernel and the library's give, so a sum
// of `splits` chains is b200_linear's with that many partials, one chain the library's, and the norm adds its squares in the norm kernels' order.
// A chain of 64 products costs 0.7 us that eight warps with an eighth of k each would not take.
#include "common.cuh"

namespace {

constexpr int RL_TILE = 16;                                         // W rows of a tile
__host__ __device__ constexpr int rl_warps(int nt) { return 8 * nt; }   // a warp per row of x: the norm's loads of a row are one round trip
constexpr size_t RL_SMEM_MAX = 210 * 1024;

struct RowsParams {
    const __nv_bfloat16* x;                // [rows, k]; with norm: the residual stream
    int64_t x_stride;
    const __nv_bfloat16* add;              // norm: the projection to add first, or null
    int64_t add_stride;
    __nv_bfloat16* residual_out;           // norm with add: x + add, contiguous
    const __nv_bfloat16* norm_w;           // or null: x as it is
    float eps;
    const __nv_bfloat16* w;                // [n, k]; SILU: [2 n, k], gate rows then up rows
    __nv_bfloat16* out;                    // [rows, n]
    int64_t out_stride;
    int rows, n, k, chains, prefetch;       // chains: of a CTA, equal parts of its k
    int one_sum;                            // norm: a lane's squares in one sum (else one for each of four pieces, as 128 threads add them)
};

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void mma_w(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldsm4(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
// MT: 16-row tiles of W of a CTA; NT: 8-row tiles of x; grid = n / (16 MT) (SILU: n / (8 MT)).  A warp has one chain of one tile of
// W and of x: p.chains * MT * NT <= 8 NT of them.  HOLD: rows of up to 1024 columns, which the norm keeps in registers (else it reads them twice).  Few enough
// registers and bytes that CTAs of this kernel and of its neighbours share an SM, so that all of gate_up's weights can be on their way while
// o_proj runs: with the weights in registers instead (118 registers, two CTAs) the Qwen3-0.6B step of 4 rows took 50 us more.
template <int MT, int NT, bool NORM, bool SILU, bool HOLD>
__global__ void __launch_bounds__(rl_warps(NT) * 32, 4 / NT) linear_rows_kernel(const RowsParams p) {
    constexpr int RL_WARPS = rl_warps(NT);
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    extern __shared__ __align__(16) unsigned char rl_smem[];
    __shared__ __align__(16) float4 red[RL_WARPS][32];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, q = lane & 3;
    const int tile = blockIdx.x, kw = p.k / p.chains, row = p.k + 8;               // k of a chain; rows in shared memory start 16 bytes further in the banks each
    __nv_bfloat16 *ws = reinterpret_cast<__nv_bfloat16*>(rl_smem), *xs = ws + MT * RL_TILE * row, *ns = xs + NT * 8 * row;
    if (!p.prefetch) asm volatile("griddepcontrol.wait;" ::: "memory");
    if constexpr (NORM) {                                                          // its weights first, a group of their own
        for (int c = tid; c < p.k / 8; c += RL_WARPS * 32) cp_async16(smem_u32(ns + c * 8), p.norm_w + c * 8);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    {
        const int per = p.k / 8;                                                   // 16-byte pieces of a row of W
        for (int r = warp; r < MT * RL_TILE; r += RL_WARPS) {
            const int m = tile * MT + r / RL_TILE, i = r % RL_TILE;
            const int64_t wr = SILU ? (i < 8 ? m * 8 + i : p.n + m * 8 + i - 8) : m * RL_TILE + i;      // rows 8-15 of a tile: the up rows, or the next ones
            const __nv_bfloat16* src = p.w + wr * p.k;
            const uint32_t dst = smem_u32(ws + r * row);
#pragma unroll 4
            for (int c = lane; c < per; c += 32) cp_async16(dst + c * 16, src + c * 8);
        }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    if constexpr (NORM) {
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
    // ---- x into shared memory ----
    if constexpr (NORM) {
        const int pieces = p.k / 8;
        const bool add = p.add != nullptr, keep = add && tile == 0;
        if (warp < p.rows) {                                                       // a warp per row of x
            const int t = warp;
            const uint4 *xr = reinterpret_cast<const uint4*>(p.x + t * p.x_stride), *ar = reinterpret_cast<const uint4*>(p.add + t * p.add_stride);
            uint4* ro = reinterpret_cast<uint4*>(p.residual_out + (int64_t)t * p.k);
            uint4 a[4], b[4];
            auto load = [&](int c0) {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int c = c0 + 32 * i;
                    a[i] = c < pieces ? xr[c] : make_uint4(0, 0, 0, 0);
                    b[i] = add && c < pieces ? ar[c] : make_uint4(0, 0, 0, 0);
                }
            };
            auto piece = [&](int i, float (&f)[8]) {
                float e[8];
                unpack8(a[i], f);
                unpack8(b[i], e);                                                  // zeros without an addend
#pragma unroll
                for (int k = 0; k < 8; ++k) f[k] += e[k];
            };
            float ss[4] = {0.f, 0.f, 0.f, 0.f};
            for (int c0 = lane; c0 < pieces; c0 += 128) {
                load(c0);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    float f[8];
                    piece(i, f);
                    float s = p.one_sum ? ss[0] : ss[i];
#pragma unroll
                    for (int e = 0; e < 8; ++e) s = fmaf(f[e], f[e], s);
                    if (p.one_sum) ss[0] = s;
                    else ss[i] = s;
                    const int c = c0 + 32 * i;
                    if (keep && c < pieces) ro[c] = pack8(f);
                }
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) ss[i] = warp_sum(ss[i]);
            const float rstd = 1.0f / sqrtf((ss[0] + ss[1] + ss[2] + ss[3]) / (float)p.k + p.eps);
            for (int c0 = lane; c0 < pieces; c0 += 128) {
                if constexpr (!HOLD) load(c0);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int c = c0 + 32 * i;
                    if (c >= pieces) continue;
                    float f[8], w[8];
                    piece(i, f);
                    unpack8(reinterpret_cast<const uint4*>(ns)[c], w);
#pragma unroll
                    for (int e = 0; e < 8; ++e) f[e] = __fmul_rn(__fmul_rn(f[e], rstd), w[e]);
                    reinterpret_cast<uint4*>(xs + t * row)[c] = pack8(f);
                }
            }
        }
    } else {
        const int pieces = p.k / 8;
        for (int t = warp; t < p.rows; t += RL_WARPS) {
            const uint4* src = reinterpret_cast<const uint4*>(p.x + t * p.x_stride);
            uint4* dst = reinterpret_cast<uint4*>(xs + t * row);
#pragma unroll 4
            for (int c = lane; c < pieces; c += 32) dst[c] = src[c];
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    // ---- products.  Columns of x rows that do not exist hold whatever shared memory held and are not stored ----
    const int chain = warp / (MT * NT), m = warp / NT % MT, nt = warp % NT;
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    if (chain < p.chains) {
        const uint32_t wa = smem_u32(ws + (m * RL_TILE + (lane & 15)) * row + chain * kw + (lane >> 4) * 8);
        const uint32_t xa = smem_u32(xs + (nt * 8 + (lane & 7)) * row + chain * kw + (lane >> 3) * 8);
        uint32_t a[2][2][4], b[2][4];                                              // two steps of 32: one is loaded while the other's products run
        auto load = [&](int c, int u) { ldsm4(wa + u * 64, a[c][0]), ldsm4(wa + u * 64 + 32, a[c][1]), ldsm4(xa + u * 64, b[c]); };
        auto products = [&](int c) {
            mma_w(acc, a[c][0][0], a[c][0][1], a[c][0][2], a[c][0][3], b[c][0], b[c][1]);
            mma_w(acc, a[c][1][0], a[c][1][1], a[c][1][2], a[c][1][3], b[c][2], b[c][3]);
        };
        const int steps = kw / 32;                                                 // even
        load(0, 0);
#pragma unroll 2
        for (int u = 0; u < steps; u += 2) {
            load(1, u + 1);
            products(0);
            if (u + 2 < steps) load(0, u + 2);
            products(1);
        }
    }
    float4 sum = make_float4(acc[0], acc[1], acc[2], acc[3]);
    if (p.chains > 1) {                                                            // 0 + first + second + ...: the order of the partials' kernel
        red[warp][lane] = sum;
        __syncthreads();
        sum = make_float4(0.f, 0.f, 0.f, 0.f);
        if (chain == 0)
            for (int i = 0; i < p.chains; ++i) {
                const float4 v = red[i * MT * NT + warp][lane];
                sum.x += v.x, sum.y += v.y, sum.z += v.z, sum.w += v.w;
            }
    }
    if (chain) return;
    const int mt = tile * MT + m;
    // a lane holds rows g and g + 8 of the tile for x rows 2 q and 2 q + 1
    const float s0[2] = {sum.x, sum.y}, s1[2] = {sum.z, sum.w};
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        const int t = nt * 8 + 2 * q + e;
        if (t >= p.rows) continue;
        __nv_bfloat16* o = p.out + t * p.out_stride;
        if constexpr (SILU) {
            const float z = round_bf16(s0[e]), u = round_bf16(s1[e]);
            o[mt * 8 + g] = __float2bfloat16_rn(__fmul_rn(z / (1.0f + expf(-z)), u));
        } else {
            o[mt * RL_TILE + g] = __float2bfloat16_rn(s0[e]);
            o[mt * RL_TILE + 8 + g] = __float2bfloat16_rn(s1[e]);
        }
    }
}

template <int MT, int NT, bool NORM, bool SILU, bool HOLD>
int rl_launch(const RowsParams& p, size_t smem, bool pdl, cudaStream_t st) {
    static B200SmemOptIn opt;
    if (opt.ensure(linear_rows_kernel<MT, NT, NORM, SILU, HOLD>, RL_SMEM_MAX) != cudaSuccess) return B200_ECUDA;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(p.n / (MT * (SILU ? 8 : RL_TILE)));
    cfg.blockDim = dim3(rl_warps(NT) * 32);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = pdl ? 1 : 0;
    if (cudaLaunchKernelEx(&cfg, linear_rows_kernel<MT, NT, NORM, SILU, HOLD>, p) != cudaSuccess) return B200_ECUDA;
    return b200_launch_status(nullptr);
}

}  // namespace

extern "C" int b200_linear_rows(const void* x, int64_t x_stride, const void* add, int64_t add_stride, void* residual_out, const void* norm_w, float eps,
                                const void* w, void* out, int64_t out_stride, int rows, int n, int k, int splits, int silu, int flags, void* stream) {
    if (!x || !w || !out || rows < 0 || n <= 0 || k <= 0 || splits <= 0) return B200_EINVAL;
    if (add && (!norm_w || !residual_out || residual_out == x || residual_out == add)) return B200_EINVAL;
    if (rows > 16 || splits > 8 || k % (64 * splits) || n % (silu ? 8 : RL_TILE) || x_stride % 8 || add_stride % 8 || out_stride < n) return B200_EUNSUPPORTED;
    if ((silu && !norm_w) || (norm_w && splits != 1)) return B200_EUNSUPPORTED;
    const uintptr_t a16 = reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(add) | reinterpret_cast<uintptr_t>(residual_out) | reinterpret_cast<uintptr_t>(norm_w);
    if ((a16 & 15) || (reinterpret_cast<uintptr_t>(w) & 15)) return B200_EUNSUPPORTED;
    const int tiles = n / (silu ? 8 : RL_TILE), nt = rows > 8 ? 2 : 1;
    // Tiles of a CTA with the norm in front, which each CTA forms for itself: several, where half of the SMs still get one (weights are there before the rows, so
    // fewer CTAs cost little).  Step of 1 / 4 / 8 / 16 rows in us: one tile 581 / 686 / 839 / 1095, two 581 / 681 / 778 / 1028, four 591 / 670 / 749 / 984.
    const int want = rows >= 4 && tiles % 4 == 0 && tiles / 4 >= 64 ? 4 : tiles % 2 == 0 && tiles / 2 >= 64 ? 2 : 1;
    const int mt = norm_w && k <= 1024 ? want : 1;
    const size_t smem = (size_t)(mt * RL_TILE + nt * 8) * (k + 8) * 2 + (norm_w ? (size_t)k * 2 : 0);
    if (smem > RL_SMEM_MAX) return B200_EUNSUPPORTED;
    if (rows == 0) return B200_OK;
    using bf = __nv_bfloat16;
    const RowsParams p{static_cast<const bf*>(x), x_stride, static_cast<const bf*>(add), add_stride, static_cast<bf*>(residual_out), static_cast<const bf*>(norm_w), eps,
                       static_cast<const bf*>(w), static_cast<bf*>(out), out_stride, rows, n, k, splits, flags & 1,
                       !add && (k == 256 || k == 512 || k == 1024 || k == 2048)};             // rows that b200_rmsnorm gives a warp
    const bool pdl = (flags & 1) != 0;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (!norm_w) return nt == 2 ? rl_launch<1, 2, false, false, false>(p, smem, pdl, st) : rl_launch<1, 1, false, false, false>(p, smem, pdl, st);
#define RL_GO(MT, NT, HOLD) (silu ? rl_launch<MT, NT, true, true, HOLD>(p, smem, pdl, st) : rl_launch<MT, NT, true, false, HOLD>(p, smem, pdl, st))
    if (mt == 4) return nt == 2 ? RL_GO(4, 2, true) : RL_GO(4, 1, true);
    if (mt == 2) return nt == 2 ? RL_GO(2, 2, true) : RL_GO(2, 1, true);
    if (k <= 1024) return nt == 2 ? RL_GO(1, 2, true) : RL_GO(1, 1, true);
    return nt == 2 ? RL_GO(1, 2, false) : RL_GO(1, 1, false);
#undef RL_GO
}
