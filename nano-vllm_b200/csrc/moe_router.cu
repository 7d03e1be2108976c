// Router logits: out[t, e] = sum_k x[t, k] w[e, k] (+ bias[e]) in fp32 on the fp32 pipe, x in fp32 or bf16 (exact as fp32), for the few dozen outputs of a router.
//
// Bound by the fp32 pipe on a prompt step (8192 x 40 x 2048: 22 us of multiply-adds, 10 us of reading x; measured 46) and by latency on a decode step (64 rows:
// 6).  The library's fp32 product took 70 us of the former and, with the copy of x to fp32 in front, 23 us of the latter.  A third stage of the copies
// changed nothing.  Here a CTA has 32 tokens and up to 40 outputs and its warps an
// eighth of every 128 columns, so that a lane holds 4 x 10 sums (pairs over k for the two-wide multiply-add): 14 shared-memory reads of 16 bytes feed 80 of
// them.  Large steps: 64 tokens and 8 x 10 sums (18 reads feed 160).  Small steps spread k over a cluster.  Every sum has a fixed order: lanes over ascending k, then warps, then the CTAs of the cluster.
// More than 40 outputs read x again for every 40: from some hundred tiles on the library is faster (142 us against 130 for 8192 x 128 x 2048), and the caller's rule sends those there.
#include "mma_common.cuh"

namespace {

constexpr int RO_K = 128, RO_THREADS = 256, RO_WARPS = 8;

__device__ __forceinline__ uint64_t ro_fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ uint64_t ro_pack(float lo, float hi) {
    uint64_t d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
    return d;
}
__device__ __forceinline__ ulonglong2 ro_quad(const float* p) { return *reinterpret_cast<const ulonglong2*>(p); }
__device__ __forceinline__ ulonglong2 ro_quad(const __nv_bfloat16* p) {
    const uint2 v = *reinterpret_cast<const uint2*>(p);
    return make_ulonglong2(ro_pack(bf16lo(v.x), bf16hi(v.x)), ro_pack(bf16lo(v.y), bf16hi(v.y)));
}

template <typename T, int NT, int NE>
struct RoSmem {                                             // two stages of (x rows, w rows), rows 16 bytes longer than their data: eight rows, eight bank groups
    static constexpr int XROW = RO_K * (int)sizeof(T) + 16, WROW = RO_K * 4 + 16, RO_TOK = 8 * NT, X = RO_TOK * XROW, STAGE = X + 4 * NE * WROW;
    static constexpr int RED = RO_WARPS * RO_TOK * 4 * NE * 4;              // afterwards: the warps' sums
    static constexpr int BYTES = 2 * STAGE > RED ? 2 * STAGE : RED;
};

// grid (cluster CTAs along k, token tiles, tiles of 4 NE outputs)
template <typename T, int NT, int NE>
__global__ void __launch_bounds__(RO_THREADS, NT * NE > 40 ? 1 : 2) moe_router_kernel(const T* __restrict__ x, int64_t x_stride, const float* __restrict__ w,
                                                                   const float* __restrict__ bias, float* __restrict__ out, int n, int E, int K, int kc) {
    B200_PDL_SYNC();
    using SM = RoSmem<T, NT, NE>;
    constexpr int RO_TOK = SM::RO_TOK;
    extern __shared__ __align__(16) unsigned char ro_smem[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, tg = lane & 7, eg = lane >> 3;
    const int t0 = blockIdx.y * RO_TOK, e0 = blockIdx.z * 4 * NE, k_begin = blockIdx.x * kc, k_end = min(K, k_begin + kc);
    const uint32_t base = smem_u32(ro_smem);
    auto fetch = [&](int k0, int st) {                      // rows and columns past the end: zeros
        constexpr int XP = RO_K * (int)sizeof(T) / 16, PER = 16 / (int)sizeof(T);
#pragma unroll
        for (int i = 0; i < RO_TOK * XP / RO_THREADS; ++i) {
            const int e = tid + RO_THREADS * i, r = e / XP, p = e % XP, k = k0 + p * PER;
            const bool in = t0 + r < n && k < k_end;
            wm_cp16(base + st * SM::STAGE + r * SM::XROW + p * 16, in ? x + (int64_t)(t0 + r) * x_stride + k : x, in ? 16 : 0);
        }
#pragma unroll
        for (int i = 0; i < (4 * NE * 32 + RO_THREADS - 1) / RO_THREADS; ++i) {
            const int e = tid + RO_THREADS * i, r = e >> 5, p = e & 31, k = k0 + p * 4;
            if (r >= 4 * NE) break;
            const bool in = e0 + r < E && k < k_end;
            wm_cp16(base + st * SM::STAGE + SM::X + r * SM::WROW + p * 16, in ? w + (int64_t)(e0 + r) * K + k : w, in ? 16 : 0);
        }
        wm_commit();
    };
    uint64_t acc[NT][NE];
#pragma unroll
    for (int i = 0; i < NT; ++i)
#pragma unroll
        for (int j = 0; j < NE; ++j) acc[i][j] = 0;
    fetch(k_begin, 0);
    for (int k0 = k_begin, st = 0; k0 < k_end; k0 += RO_K, st ^= 1) {
        if (k0 + RO_K < k_end) {
            fetch(k0 + RO_K, st ^ 1);
            wm_wait<1>();
        } else {
            wm_wait<0>();
        }
        __syncthreads();
        const unsigned char *xs = ro_smem + st * SM::STAGE + tg * SM::XROW + warp * 16 * sizeof(T), *ws = ro_smem + st * SM::STAGE + SM::X + eg * SM::WROW + warp * 64;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            ulonglong2 xv[NT];
#pragma unroll
            for (int i = 0; i < NT; ++i) xv[i] = ro_quad(reinterpret_cast<const T*>(xs + 8 * i * SM::XROW) + 4 * q);
#pragma unroll
            for (int j = 0; j < NE; ++j) {
                const ulonglong2 wv = ro_quad(reinterpret_cast<const float*>(ws + 4 * j * SM::WROW) + 4 * q);
#pragma unroll
                for (int i = 0; i < NT; ++i) acc[i][j] = ro_fma2(xv[i].y, wv.y, ro_fma2(xv[i].x, wv.x, acc[i][j]));
            }
        }
        __syncthreads();
    }
    float* red = reinterpret_cast<float*>(ro_smem);         // [warp][token][output]
#pragma unroll
    for (int i = 0; i < NT; ++i)
#pragma unroll
        for (int j = 0; j < NE; ++j) {
            const float2 f = *reinterpret_cast<const float2*>(&acc[i][j]);
            red[(warp * RO_TOK + tg + 8 * i) * (4 * NE) + eg + 4 * j] = f.x + f.y;
        }
    __syncthreads();
    constexpr int ALL = RO_TOK * 4 * NE, OWN = (ALL + RO_THREADS - 1) / RO_THREADS;
    float sum[OWN];
#pragma unroll
    for (int i = 0; i < OWN; ++i) {
        sum[i] = 0.f;
        if (ALL % RO_THREADS && tid + RO_THREADS * i >= ALL) break;
#pragma unroll
        for (int v = 0; v < RO_WARPS; ++v) sum[i] += red[v * ALL + tid + RO_THREADS * i];
    }
    if (gridDim.x > 1) {
        __syncthreads();
#pragma unroll
        for (int i = 0; i < OWN; ++i)
            if (tid + RO_THREADS * i < ALL) red[tid + RO_THREADS * i] = sum[i];
        asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
        // a CTA adds its share of the outputs over the cluster
        const int rank = blockIdx.x, ctas = gridDim.x;
        for (int e = rank * RO_THREADS + tid; e < ALL; e += ctas * RO_THREADS) {
            float v = 0.f;
            for (int r = 0; r < ctas; ++r) {
                uint32_t from;
                float f;
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(from) : "r"(smem_u32(red + e)), "r"(r));
                asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(f) : "r"(from) : "memory");
                v += f;
            }
            const int t = t0 + e / (4 * NE), o = e0 + e % (4 * NE);
            if (t < n && o < E) out[(int64_t)t * E + o] = bias ? v + bias[o] : v;
        }
        asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");       // nobody leaves while its sums are being read
        return;
    }
#pragma unroll
    for (int i = 0; i < OWN; ++i) {
        const int e = tid + RO_THREADS * i, t = t0 + e / (4 * NE), o = e0 + e % (4 * NE);
        if (e < ALL && t < n && o < E) out[(int64_t)t * E + o] = bias ? sum[i] + bias[o] : sum[i];
    }
}

template <typename T, int NT, int NE>
int launch_router(const void* x, int64_t x_stride, const float* w, const float* bias, float* out, int n, int E, int K, cudaStream_t st) {
    using SM = RoSmem<T, NT, NE>;
    const int tok = (n + SM::RO_TOK - 1) / SM::RO_TOK, outs = (E + 4 * NE - 1) / (4 * NE), steps = (K + RO_K - 1) / RO_K;
    // k over a cluster while the tiles leave SMs idle
    int ctas = 1;
    while (ctas < 8 && (int64_t)tok * outs * ctas * 2 <= 148 && steps >= ctas * 2) ctas *= 2;
    const int per = (steps + ctas - 1) / ctas, kc = per * RO_K;
    ctas = (steps + per - 1) / per;                         // nobody without columns: such a CTA would not wait for its first copies before its sums take their place
    static B200SmemOptIn opt;
    if (opt.ensure(moe_router_kernel<T, NT, NE>, SM::BYTES) != cudaSuccess) return B200_ECUDA;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ctas, tok, outs);
    cfg.blockDim = dim3(RO_THREADS);
    cfg.dynamicSmemBytes = SM::BYTES;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim = {(unsigned)ctas, 1, 1};
    cfg.attrs = attr;
    cfg.numAttrs = 1;
#ifdef B200_PDL
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.numAttrs = b200_tls_pdl_off() ? 1 : 2;
#endif
    cudaLaunchKernelEx(&cfg, moe_router_kernel<T, NT, NE>, static_cast<const T*>(x), x_stride, w, bias, out, n, E, K, kc);
    return b200_launch_status(nullptr);
}

}  // namespace

extern "C" int b200m_moe_logits(const void* x, int64_t x_stride, const float* w, const float* bias, float* out, int n, int num_outputs, int K, int is32,
                                void* stream) {
    if (!x || !w || !out || n < 0 || num_outputs <= 0 || K <= 0) return B200_EINVAL;
    if (K % 8 || x_stride % 8 || ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w)) & 15)) return B200_EUNSUPPORTED;
    if ((n + 31) / 32 > 65535 || num_outputs > 1024) return B200_EUNSUPPORTED;
    if (n == 0) return B200_OK;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    // tiles of 20 outputs where they waste less than tiles of 40; of 64 tokens where those still give most SMs one (8192 x 40 x 2048: 46 us against 48)
    const bool narrow = (num_outputs + 19) / 20 * 20 < (num_outputs + 39) / 40 * 40, large = (int64_t)(n + 63) / 64 * ((num_outputs + 39) / 40) >= 100;
    B200M_DISPATCH(is32, if (narrow) return (launch_router<T, 4, 5>(x, x_stride, w, bias, out, n, num_outputs, K, st));
                   return (large ? launch_router<T, 8, 10>(x, x_stride, w, bias, out, n, num_outputs, K, st)
                                 : launch_router<T, 4, 10>(x, x_stride, w, bias, out, n, num_outputs, K, st)));
    return B200_EUNSUPPORTED;
}
