// The delta rule with a decay per (head, key channel) over prompt portions, sixteen tokens at a time on the tensor cores (bf16 activations):
//     S <- diag(g) S;  u = beta (v - S^T k);  S <- S + k u^T;  o = scale * S^T q          per head S [dim, vdim] fp32, q and k of unit norm, g <= 1
// With P_t = g_1 ... g_t and R_t = g_(t+1) ... g_16 the products of a chunk's decays (per channel) and S the state before it,
//     A_ts = sum_c k_tc (g_(s+1) ... g_t)_c k_sc  (s < t),   B_ts likewise with q_t  (s <= t),   T = (1 + diag(beta) A)^-1 diag(beta)
//     W = T (P k),  Q = P q - B W;   U = T V - W S,   o = scale * ((B T) V + Q S),   S <- P_16 S + (R k)^T U
// which is the token-by-token recurrence regrouped: only products of decays, never quotients, so no decay is too strong for it.  Rows of W and Q and
// entries of T and B T are at most one: each is the answer of a chain of contractions to a unit input.
//
// Two kernels.  The first has a block per (chunk, head), all chunks at once, and a thread per channel: decays, A and B (products of keys and queries with
// the decays from a place between the two tokens, see below), T by forward substitution, W and Q.  The second walks a sequence's chunks, three products
// each: a CTA owns 64 value columns of a head, two consumer warps 16 of them, with S^T as product accumulators in registers that are the next
// product's left operand as they are; two warps copy the chunks ahead.
//
// Precision: an operand of a product is fp32 split into two fp16 numbers (11 + 11 bits; both rounded to nearest, so the pair carries 22 to 23
// bits), scaled by powers of two into fp16's range -- per value column for S and U, by 2^14 for what is at most one -- and three of
// the four partial products are taken (the fourth is below 2^-22).  Against tf32 pairs this halves the tensor work (m16n8k16 at the price of
// m16n8k8).  V is bf16 as it is, T and B T are three bf16 numbers each.  S itself is fp32 and sees one fused multiply-add per chunk.  Against
// float64 the whole is 1e-7 to 3e-6 of the results' norm off, mostly less than the fp32-pipe form of recurrent_mix.cu (1e-7 to 6e-6).
//
// Measured on a B200, 16 heads of 128 x 128, both kernels together against that form: 4 x 2048 tokens 351 us (137 + 214) against 676, 1 x 4096 486 against
// 1331, 16 x 1000 691 against 1127, 12 x 600 321 against 551, 16 x 64 60 against 92, 16 x 16 29 against 35.
#include "mma_common.cuh"
#include "state_common.cuh"

#include <cuda_fp16.h>

namespace {

constexpr int CD_L = 16, CD_D = 128, CD_VC = 64, CD_STAGES = 4;
constexpr float CD_UP = 16384.f;                       // 2^14: scale of operands that are at most one
// Workspace of one (chunk, head), a stage of the walk as it lies in shared memory: W, Q, R k as fp16 pairs (high rows, low rows), a row of sixteen tokens
// per channel; T and B T as three bf16 matrices [16][16] each, a row per token; P_16 in fp32.  Tokens of a channel's row (and the rows of T and B T) stand
// in the order 0 1 8 9 2 3 10 11 ..., which is how a product's accumulators hold them.  The two 16-byte pieces of a row change places every four
// rows, so that a piece of eight rows lies in eight bank groups.
constexpr int CW_ROWS = CD_D * CD_L * 2, CW_W = 0, CW_Q = 2 * CW_ROWS, CW_R = 4 * CW_ROWS, CW_MAT = CD_L * CD_L * 2, CW_T = 6 * CW_ROWS,
              CW_BT = CW_T + 3 * CW_MAT, CW_P = CW_BT + 3 * CW_MAT, CW_BYTES = CW_P + CD_D * 4;
__device__ __forceinline__ uint32_t row_swz(int row, int piece) { return row * (CD_L * 2) + ((piece ^ ((row >> 2) & 1)) << 4); }        // rows of sixteen
__device__ __forceinline__ uint32_t val_swz(int row, int piece) { return row * (CD_VC * 2) + ((piece ^ (row & 7)) << 4); }               // rows of 64
__device__ __forceinline__ uint32_t raw_swz(int row, int piece) { return row * (CD_D * 2) + ((piece ^ (row & 7)) << 4); }                // rows of 128
__device__ __forceinline__ uint32_t mat_row(int row, int col) { return row_swz(row, col >> 3) + (col & 7) * 2; }
__device__ __forceinline__ constexpr int place_of(int token) { return token < 8 ? 4 * (token >> 1) + (token & 1) : 4 * ((token - 8) >> 1) + 2 + (token & 1); }
__device__ __forceinline__ int token_at(int place) { return 2 * (place >> 2) + (place & 1) + 8 * ((place >> 1) & 1); }

__device__ __forceinline__ uint64_t cd_fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ uint64_t cd_mul2(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ uint64_t cd_pack(float lo, float hi) {
    uint64_t d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
    return d;
}
__device__ __forceinline__ uint64_t cd_add2(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ float2 cd_two(uint64_t v) {
    float2 f;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
    return f;
}
__device__ __forceinline__ float cd_sum(uint64_t v) {
    const float2 f = cd_two(v);
    return f.x + f.y;
}
// a pair of floats -> fp16 pairs: their roundings, and what these leave (exact before its own rounding)
__device__ __forceinline__ void split_f16(uint64_t v, uint32_t& hi, uint32_t& lo) {
    const float2 f = cd_two(v);
    asm("{\n\t.reg .b16 a, b, m;\n\t.reg .f32 x, y;\n\t"
        "cvt.rn.f16x2.f32 %0, %3, %2;\n\t"
        "mov.b32 {a, b}, %0;\n\tmov.b16 m, 0xBC00;\n\t"
        "fma.rn.f32.f16 x, a, m, %2;\n\tfma.rn.f32.f16 y, b, m, %3;\n\t"
        "cvt.rn.f16x2.f32 %1, y, x;\n\t}"
        : "=&r"(hi), "=r"(lo)
        : "f"(f.x), "f"(f.y));
}
// exp(rate softplus(x)), c = rate * log2(e): softplus(x) = max(x, 0) + log1p(exp(-|x|)), log1p(y) / y over [0, 1] and 2^f over [-1/2, 1/2] as series
// whose coefficients are weighted least-squares fits taken to equal ripples (relative errors below 3e-8 and 2e-9).  2^f is 1 + f Q(f), so that a
// decay next to one is rounded once: the power unit's last bits would add up over a sequence.  As close as expf and log1pf give it, in half of
// their instructions.  Below 2^-126 it stays there.
__device__ __forceinline__ float decay_fit(float x, float c) {
    constexpr float L[9] = {0.99999994f, -0.499994934f, 0.333190978f, -0.24842982f, 0.191060051f, -0.136632428f, 0.0782259107f, -0.0295052137f, 0.00523268804f};
    constexpr float Q[6] = {0.69314718f, 0.240226477f, 0.0555033237f, 0.00961843692f, 0.00133988948f, 0.000153534871f}, MAGIC = 12582912.f;
    float y, m, w;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(fminf(fabsf(x), 80.f) * -1.44269502f));
    float p = L[8];
#pragma unroll
    for (int i = 7; i >= 0; --i) p = fmaf(p, y, L[i]);
    asm("max.NaN.f32 %0, %1, 0f00000000;" : "=f"(m) : "f"(x));
    asm("max.NaN.f32 %0, %1, 0fC2FC0000;" : "=f"(w) : "f"(fmaf(p, y, m) * c));                      // -126
    const float n = w + MAGIC, f = w - (n - MAGIC);
    float q = Q[5];
#pragma unroll
    for (int i = 4; i >= 0; --i) q = fmaf(q, f, Q[i]);
    return fmaf(q, f, 1.f) * __uint_as_float(__float_as_uint(n) * 0x800000u + 0x3f800000u);
}
__device__ __forceinline__ void mma_f16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// the same from zero
__device__ __forceinline__ void mma_f16_new(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}

// ---- first kernel: decays, A, B, T, W, Q ------------------------------------------------------------------------------------------------
// A_ts and B_ts need the decays between s and t.  Pairs of tokens are taken by the largest of four levels (half blocks of 8, 4, 2, 1 tokens) whose middle
// parts them: with the middle m, k_t and q_t take g_m ... g_t, k_s takes g_(s+1) ... g_(m-1), all at most one, and a level is one product of
// [8 k rows, 8 q rows] with [8 k rows].  Bound by the instruction rate (about 2200 per thread, half an instruction per cycle
// and scheduler).  A form with a warp per (chunk, head) and the sums on the fp32 pipe, 8500 instructions of straight-line code, spent two thirds of its
// time waiting for instructions: 153 us where this one takes 137.
constexpr int CP_THREADS = 128;
struct CpSmem {
    static constexpr int RAW_K = 0, RAW_Q = CD_L * CD_D * 2, A = 2 * RAW_Q, B = A + CD_L * CD_L * 4, T = B + CD_L * CD_L * 4,
                         MAT = T + CD_L * CD_L * 4,                          // T high, low, -B T high, low (fp16), rows of tokens
                         NORM = MAT + 4 * CW_MAT,                            // normalisers of k, of q, strengths
                         FACT = NORM + 3 * CD_L * 4, FROW = CD_D * 16,       // [two levels][k left, q left, k right][high, low]: rows of eight tokens per channel
                         PK = FACT, PQ = PK + 2 * CW_ROWS, PQ_STRIDE = 18,   // in their place: P k (fp16 pairs), P q (fp32)
                         BYTES = FACT + 12 * FROW;
    static_assert(PQ + CD_D * PQ_STRIDE * 4 <= BYTES, "");
};
// A channel's factors of a level: places 2 i and 2 i + 1 of its eight left and eight right tokens
template <int T>
__device__ __forceinline__ float cd_at(const uint64_t (&v)[CD_L / 2]) {
    const float2 f = cd_two(v[T / 2]);
    return T & 1 ? f.y : f.x;
}
template <int LEVEL, int I>
__device__ __forceinline__ void level_pair(const uint64_t (&g)[CD_L / 2], const uint64_t (&k)[CD_L / 2], const uint64_t (&q)[CD_L / 2], float& p,
                                           float (&R)[8], uint32_t (&rw)[24]) {
    constexpr int N = 8 >> LEVEL, A0 = 2 * I, A1 = 2 * I + 1, L0 = A0 / N * 2 * N + N + A0 % N, L1 = A1 / N * 2 * N + N + A1 % N, R0 = L0 - N, R1 = L1 - N;
    const float l0 = A0 % N == 0 ? cd_at<L0>(g) : p * cd_at<L0>(g), l1 = A1 % N == 0 ? cd_at<L1>(g) : l0 * cd_at<L1>(g);
    p = l1;
    const uint64_t l = cd_pack(l0, l1);
    split_f16(cd_mul2(cd_pack(cd_at<L0>(k), cd_at<L1>(k)), l), rw[I], rw[4 + I]);
    split_f16(cd_mul2(cd_pack(cd_at<L0>(q), cd_at<L1>(q)), l), rw[8 + I], rw[12 + I]);
    if constexpr (N == 1) split_f16(cd_pack(cd_at<R0>(k), cd_at<R1>(k)), rw[16 + I], rw[20 + I]);
    else split_f16(cd_mul2(cd_pack(cd_at<R0>(k), cd_at<R1>(k)), cd_pack(R[A0], R[A1])), rw[16 + I], rw[20 + I]);
}
template <int LEVEL, int A>
__device__ __forceinline__ void level_right(const uint64_t (&g)[CD_L / 2], float (&R)[8]) {             // from the last place to the first
    constexpr int N = 8 >> LEVEL, T = A / N * 2 * N + A % N;
    if constexpr (A % N == N - 1) R[A] = 1.f;
    else R[A] = R[A + 1] * cd_at<T + 1>(g);
    if constexpr (A > 0) level_right<LEVEL, A - 1>(g, R);
}
template <int LEVEL>
__device__ __forceinline__ void level_factors(const uint64_t (&g)[CD_L / 2], const uint64_t (&k)[CD_L / 2], const uint64_t (&q)[CD_L / 2], unsigned char* to) {
    uint32_t rw[24];                                        // k left high, low; q left; k right
    float R[8], p = 1.f;
    level_right<LEVEL, 7>(g, R);
    level_pair<LEVEL, 0>(g, k, q, p, R, rw);
    level_pair<LEVEL, 1>(g, k, q, p, R, rw);
    level_pair<LEVEL, 2>(g, k, q, p, R, rw);
    level_pair<LEVEL, 3>(g, k, q, p, R, rw);
#pragma unroll
    for (int i = 0; i < 6; ++i)
        *reinterpret_cast<uint4*>(to + i * (CD_D * 16)) = make_uint4(rw[4 * i], rw[4 * i + 1], rw[4 * i + 2], rw[4 * i + 3]);
}
__global__ void __launch_bounds__(CP_THREADS, 4) channel_delta_prepare_kernel(
    const __nv_bfloat16* __restrict__ x, int64_t stride, int q_off, int k_off, const __nv_bfloat16* __restrict__ write_in, int64_t write_stride,
    const float* __restrict__ decay_in, int64_t decay_stride, const float* __restrict__ rate, const float* __restrict__ bias, float sign,
    const int32_t* __restrict__ cu_q, unsigned char* __restrict__ ws, int H, int G, int dim, int first, int chunks) {
    B200_PDL_SYNC();
    using SM = CpSmem;
    extern __shared__ __align__(128) unsigned char cp_smem[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, gq = lane >> 2, t4 = lane & 3, s = blockIdx.y;
    const int h = blockIdx.x % H, c = blockIdx.x / H;
    const int q0 = cu_q[s], qlen = cu_q[s + 1] - q0, t0 = (first + c) * CD_L;
    if (t0 >= qlen) return;
    const int len = min(CD_L, qlen - t0);
    const uint32_t sbase = smem_u32(cp_smem);
    const __nv_bfloat16* qp = x + (int64_t)(q0 + t0) * stride + q_off + (int64_t)(h / (H / G)) * dim;
    const __nv_bfloat16* kp = qp + (k_off - q_off);
    float* A = reinterpret_cast<float*>(cp_smem + SM::A);
    float* B = reinterpret_cast<float*>(cp_smem + SM::B);
    float* T = reinterpret_cast<float*>(cp_smem + SM::T);
    float* norm = reinterpret_cast<float*>(cp_smem + SM::NORM);
#pragma unroll
    for (int i = 0; i < 2; ++i) {                           // rows past the end and channels past dim: zeros
        const int e = tid + CP_THREADS * i, r = e >> 4, p = e & 15;
        const bool in = r < len && p * 8 < dim;
        wm_cp16(sbase + SM::RAW_K + raw_swz(r, p), in ? kp + r * stride + p * 8 : x, in ? 16 : 0);
        wm_cp16(sbase + SM::RAW_Q + raw_swz(r, p), in ? qp + r * stride + p * 8 : x, in ? 16 : 0);
    }
    wm_commit();
    uint64_t g[CD_L / 2];                                   // this channel's decays, tokens 2 i and 2 i + 1
    {
        const bool in = tid < dim;
        const float* gp = decay_in + (int64_t)(q0 + t0) * decay_stride + (int64_t)h * dim + (in ? tid : 0);
        float z[CD_L];
#pragma unroll
        for (int t = 0; t < CD_L; ++t) z[t] = gp[min(t, len - 1) * (int)decay_stride];      // (a step's sixteen rows are within 2^31 elements: the launch)
        const float c = rate[h] * 1.44269502f, b = sign * bias[(int64_t)h * dim + (in ? tid : 0)];
        if (tid < CD_L) norm[2 * CD_L + tid] = tid < len ? sigmoidf_(__bfloat162float(write_in[(int64_t)(q0 + t0 + tid) * write_stride + h])) : 0.f;
        reinterpret_cast<float4*>(A)[tid] = make_float4(0.f, 0.f, 0.f, 0.f);            // A and B: zeros above their diagonals
#pragma unroll
        for (int t = 0; t < CD_L; ++t) z[t] = decay_fit(fmaf(sign, z[t], b), c);
        if (len < CD_L) {                                   // behind the end nothing decays, and keys and queries are zeros
#pragma unroll
            for (int t = 0; t < CD_L; ++t) z[t] = t < len ? z[t] : 1.f;
        }
#pragma unroll
        for (int i = 0; i < CD_L / 2; ++i) g[i] = cd_pack(z[2 * i], z[2 * i + 1]);
    }
    wm_wait<0>();
    __syncthreads();
    // k.k, q.q, q.k of every token: the diagonals of three products of the rows as they are
    const int ar = lane & 15, br = (lane & 7) + ((lane >> 4) << 3), bp = (lane >> 3) & 1;
    if (warp < 3) {
        const uint32_t ra = sbase + (warp == 0 ? SM::RAW_K : SM::RAW_Q), rb = sbase + (warp == 1 ? SM::RAW_Q : SM::RAW_K);
        float D[2][4];
#pragma unroll
        for (int i = 0; i < 2; ++i) D[i][0] = D[i][1] = D[i][2] = D[i][3] = 0.f;
#pragma unroll
        for (int kk = 0; kk < CD_D / 16; ++kk) {
            uint32_t a[4], b[4];
            wm_ldsm(ra + raw_swz(ar, kk * 2 + (lane >> 4)), a[0], a[1], a[2], a[3]);
            wm_ldsm(rb + raw_swz(br, kk * 2 + bp), b[0], b[1], b[2], b[3]);
            wm_mma(D[0], a[0], a[1], a[2], a[3], b[0], b[1]);
            wm_mma(D[1], a[0], a[1], a[2], a[3], b[2], b[3]);
        }
        if (t4 == gq >> 1) {                                // places (gq, gq) and (gq + 8, gq + 8)
            const float lo = gq & 1 ? D[0][1] : D[0][0], hi = gq & 1 ? D[1][3] : D[1][2];
            if (warp < 2) {
                norm[warp * CD_L + gq] = 1.0f / sqrtf(lo + 1e-6f);
                norm[warp * CD_L + gq + 8] = 1.0f / sqrtf(hi + 1e-6f);
            } else {
                B[gq * (CD_L + 1)] = lo, B[(gq + 8) * (CD_L + 1)] = hi;
            }
        }
    }
    __syncthreads();
    if (tid < CD_L) B[tid * (CD_L + 1)] *= norm[tid] * norm[CD_L + tid];
    uint64_t k[CD_L / 2], q[CD_L / 2];                      // unit rows' entries of this channel, times 2^14
#pragma unroll
    for (int i = 0; i < CD_L / 2; ++i) {
        float v[4];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const uint32_t at = raw_swz(2 * i + e, tid >> 3) + (tid & 7) * 2;
            v[e] = __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(cp_smem + SM::RAW_K + at));
            v[2 + e] = __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(cp_smem + SM::RAW_Q + at));
        }
        const uint64_t up = cd_pack(CD_UP, CD_UP);
        k[i] = cd_mul2(cd_pack(v[0], v[1]), cd_mul2(*reinterpret_cast<const uint64_t*>(norm + 2 * i), up));
        q[i] = cd_mul2(cd_pack(v[2], v[3]), cd_mul2(*reinterpret_cast<const uint64_t*>(norm + CD_L + 2 * i), up));
    }
    // two levels at a time: a warp has half of the channels of one, and its sums meet the other half's in A and B (two additions onto zero)
    auto level_sums = [&](int n) {
        const uint32_t f = sbase + SM::FACT + (warp >> 1) * 6 * SM::FROW + (warp & 1) * (CD_D / 2) * 16;
        const int m = lane >> 3, r8 = lane & 7;             // which of four 8 x 8 tiles this lane's address is for
        float D[4], E[4];
#pragma unroll
        for (int kk = 0; kk < CD_D / 32; ++kk) {
            uint32_t ah[4], al[4], b[4];
            const uint32_t ra = f + (m & 1) * 2 * SM::FROW + (kk * 16 + (m >> 1) * 8 + r8) * 16;
            wm_ldsm_t(ra, ah[0], ah[1], ah[2], ah[3]);
            wm_ldsm_t(ra + SM::FROW, al[0], al[1], al[2], al[3]);
            wm_ldsm_t(f + 4 * SM::FROW + (m >> 1) * SM::FROW + (kk * 16 + (m & 1) * 8 + r8) * 16, b[0], b[1], b[2], b[3]);
            if (kk == 0) mma_f16_new(D, ah, b[0], b[1]), mma_f16_new(E, al, b[0], b[1]);
            else mma_f16(D, ah, b[0], b[1]), mma_f16(E, al, b[0], b[1]);
            mma_f16(E, ah, b[2], b[3]);
        }
        const int sh = 31 - __clz(n), t = ((gq >> sh) << (sh + 1)) + n + (gq & (n - 1));
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int j = 2 * t4 + e;
            if (gq >> sh == j >> sh) {
                const int at = t * CD_L + ((j >> sh) << (sh + 1)) + (j & (n - 1));
                atomicAdd(A + at, (D[e] + E[e]) * (1.f / (CD_UP * CD_UP)));
                atomicAdd(B + at, (D[2 + e] + E[2 + e]) * (1.f / (CD_UP * CD_UP)));
            }
        }
    };
    level_factors<0>(g, k, q, cp_smem + SM::FACT + tid * 16);
    level_factors<1>(g, k, q, cp_smem + SM::FACT + 6 * SM::FROW + tid * 16);
    __syncthreads();
    level_sums(8 >> (warp >> 1));
    __syncthreads();
    level_factors<2>(g, k, q, cp_smem + SM::FACT + tid * 16);
    level_factors<3>(g, k, q, cp_smem + SM::FACT + 6 * SM::FROW + tid * 16);
    __syncthreads();
    level_sums(2 >> (warp >> 1));
    __syncthreads();
    unsigned char* wp = ws + (((int64_t)s * chunks + c) * H + h) * (int64_t)CW_BYTES;
    if (warp == 0) {
        // a lane has a column of T.  Places above the diagonal stay zero; a row takes the entries up to its own token alone
        const int j = lane & (CD_L - 1);
        float y[CD_L];
#pragma unroll
        for (int t = 0; t < CD_L; ++t) {
            float a[CD_L], acc0 = 0.f, acc1 = 0.f;
#pragma unroll
            for (int i = 0; i < t; i += 4) {
                const float4 v = *reinterpret_cast<const float4*>(A + t * CD_L + i);
                a[i] = v.x, a[i + 1] = v.y, a[i + 2] = v.z, a[i + 3] = v.w;
            }
#pragma unroll
            for (int i = 0; i < t; i += 2) {
                acc0 = fmaf(a[i], y[i], acc0);
                if (i + 1 < t) acc1 = fmaf(a[i + 1], y[i + 1], acc1);
            }
            y[t] = t >= j ? norm[2 * CD_L + t] * ((t == j ? 1.f : 0.f) - (acc0 + acc1)) : 0.f;
            if (lane < CD_L) T[t * CD_L + j] = y[t];
        }
    }
    bool clean;
    {
        uint64_t upto[CD_L / 2];                            // products of the decays up to a token
        uint32_t pk[2 * CD_L / 2], rk[2 * CD_L / 2];
        float p = 1.f;
        uint64_t zero = 0;
#pragma unroll
        for (int i = 0; i < CD_L / 2; ++i) {
            const float2 f = cd_two(g[i]);
            const float a = p * f.x;
            p = a * f.y;
            upto[i] = cd_pack(a, p);
            const uint64_t v = cd_mul2(upto[i], k[i]);
            zero = cd_fma2(v, 0ull, zero);
            split_f16(v, pk[i], pk[CD_L / 2 + i]);
            *reinterpret_cast<uint64_t*>(cp_smem + SM::PQ + tid * (SM::PQ_STRIDE * 4) + i * 8) = cd_mul2(upto[i], q[i]);
        }
        clean = cd_sum(zero) == 0.f;
        *reinterpret_cast<float*>(wp + CW_P + tid * 4) = p;
        p = 1.f;
#pragma unroll
        for (int i = CD_L / 2 - 1; i >= 0; --i) {           // tokens 2 i and 2 i + 1 side by side: place 4 i, or 4 (i - 4) + 2
            const float2 f = cd_two(g[i]);
            const float a = p * f.y;
            const int w = i < 4 ? 2 * i : 2 * (i - 4) + 1;
            split_f16(cd_mul2(cd_pack(a, p), k[i]), rk[w], rk[CD_L / 2 + w]);
            p = a * f.x;
        }
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int w = 8 * m + 4 * i;
                *reinterpret_cast<uint4*>(cp_smem + SM::PK + m * CW_ROWS + row_swz(tid, i)) = make_uint4(pk[w], pk[w + 1], pk[w + 2], pk[w + 3]);
                *reinterpret_cast<uint4*>(wp + CW_R + m * CW_ROWS + row_swz(tid, i)) = make_uint4(rk[w], rk[w + 1], rk[w + 2], rk[w + 3]);
            }
    }
    clean = __syncthreads_and(clean);
    {   // two neighbours of a row of T and of B T each
        const int t = tid >> 3, j = (tid & 7) * 2, place = place_of(t);
        const uint64_t tv = *reinterpret_cast<const uint64_t*>(T + t * CD_L + j);
        uint64_t bt = 0;
#pragma unroll
        for (int i = 0; i < CD_L; i += 4) {
            const float4 b = *reinterpret_cast<const float4*>(B + t * CD_L + i);
            const float bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (i + e <= t) bt = cd_fma2(cd_pack(bv[e], bv[e]), *reinterpret_cast<const uint64_t*>(T + (i + e) * CD_L + j), bt);
        }
#pragma unroll
        for (int w = 0; w < 2; ++w) {
            const uint64_t v = w ? bt : tv;
            float2 f = cd_two(v);
            const uint32_t row = mat_row(t, j), to = mat_row(place, j);
#pragma unroll
            for (int m = 0; m < 3; ++m) {
                const uint32_t b = pack_bf16x2(f.x, f.y);
                *reinterpret_cast<uint32_t*>(wp + (w ? CW_BT : CW_T) + m * CW_MAT + to) = b;
                f.x -= bf16lo(b), f.y -= bf16hi(b);
            }
            const float up = w ? -CD_UP : CD_UP;
            uint32_t hi, lo;
            split_f16(cd_mul2(v, cd_pack(up, up)), hi, lo);
            *reinterpret_cast<uint32_t*>(cp_smem + SM::MAT + 2 * w * CW_MAT + row) = hi;
            *reinterpret_cast<uint32_t*>(cp_smem + SM::MAT + (2 * w + 1) * CW_MAT + row) = lo;
        }
        if (!clean) {
            *reinterpret_cast<uint64_t*>(cp_smem + SM::RAW_K + (t * CD_L + j) * 4) = tv;         // for the rows one by one, below
            *reinterpret_cast<uint64_t*>(cp_smem + SM::RAW_Q + (t * CD_L + j) * 4) = bt;
        }
    }
    __syncthreads();
    // W^T = (P k)^T T^T and Q^T = (P q)^T - (P k)^T (B T)^T, [32 channels of this warp] x [16 tokens]
    uint32_t mt[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) wm_ldsm(sbase + SM::MAT + i * CW_MAT + row_swz(br, bp), mt[i][0], mt[i][1], mt[i][2], mt[i][3]);
#pragma unroll
    for (int m = 0; m < 2; ++m) {
        const int c0 = warp * 32 + m * 16;
        uint32_t ah[4], al[4];
        wm_ldsm(sbase + SM::PK + row_swz(c0 + ar, lane >> 4), ah[0], ah[1], ah[2], ah[3]);
        wm_ldsm(sbase + SM::PK + CW_ROWS + row_swz(c0 + ar, lane >> 4), al[0], al[1], al[2], al[3]);
        float W[2][4], Q[2][4];                             // channels gq, gq + 8; tokens 8 i + 2 t4, + 1
        const float* pq = reinterpret_cast<const float*>(cp_smem + SM::PQ) + (c0 + gq) * SM::PQ_STRIDE + 2 * t4;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
#pragma unroll
            for (int e = 0; e < 4; ++e) Q[i][e] = pq[(e >> 1) * 8 * SM::PQ_STRIDE + 8 * i + (e & 1)] * CD_UP;
            mma_f16_new(W[i], al, mt[0][2 * i], mt[0][2 * i + 1]);
            mma_f16(W[i], ah, mt[1][2 * i], mt[1][2 * i + 1]);
            mma_f16(W[i], ah, mt[0][2 * i], mt[0][2 * i + 1]);
            mma_f16(Q[i], al, mt[2][2 * i], mt[2][2 * i + 1]);
            mma_f16(Q[i], ah, mt[3][2 * i], mt[3][2 * i + 1]);
            mma_f16(Q[i], ah, mt[2][2 * i], mt[2][2 * i + 1]);
        }
        if (!clean) {
            // a key or a decay that is no number: a token's row takes the tokens up to its own alone (its products with the zeros above would not)
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int t = 8 * i + 2 * t4 + (e & 1), ch = c0 + gq + 8 * (e >> 1);
                    float w = 0.f, v = reinterpret_cast<const float*>(cp_smem + SM::PQ)[ch * SM::PQ_STRIDE + t] * CD_UP;
#pragma unroll 1
                    for (int j = 0; j <= t; ++j) {
                        const unsigned char* at = cp_smem + SM::PK + row_swz(ch, j >> 3) + (j & 7) * 2;
                        const float f = __half2float(*reinterpret_cast<const __half*>(at)) + __half2float(*reinterpret_cast<const __half*>(at + CW_ROWS));
                        w = fmaf(reinterpret_cast<const float*>(cp_smem + SM::RAW_K)[t * CD_L + j] * CD_UP, f, w);
                        v = fmaf(reinterpret_cast<const float*>(cp_smem + SM::RAW_Q)[t * CD_L + j] * -CD_UP, f, v);
                    }
                    W[i][e] = w, Q[i][e] = v;
                }
        }
        const uint64_t down = cd_pack(1.f / CD_UP, 1.f / CD_UP);
#pragma unroll
        for (int r = 0; r < 2; ++r) {                       // tokens 2 t4, + 1, 8 + 2 t4, + 1 side by side: the order of the workspace
            unsigned char* d = wp + row_swz(c0 + gq + 8 * r, t4 >> 1) + (t4 & 1) * 8;
            uint2 hi, lo;
            split_f16(cd_mul2(cd_pack(W[0][2 * r], W[0][2 * r + 1]), down), hi.x, lo.x);
            split_f16(cd_mul2(cd_pack(W[1][2 * r], W[1][2 * r + 1]), down), hi.y, lo.y);
            *reinterpret_cast<uint2*>(d + CW_W) = hi;
            *reinterpret_cast<uint2*>(d + CW_W + CW_ROWS) = lo;
            split_f16(cd_mul2(cd_pack(Q[0][2 * r], Q[0][2 * r + 1]), down), hi.x, lo.x);
            split_f16(cd_mul2(cd_pack(Q[1][2 * r], Q[1][2 * r + 1]), down), hi.y, lo.y);
            *reinterpret_cast<uint2*>(d + CW_Q) = hi;
            *reinterpret_cast<uint2*>(d + CW_Q + CW_ROWS) = lo;
        }
    }
}

// ---- second kernel: the walk over the chunks --------------------------------------------------------------------------------------------
struct CdSmem {                                             // stages of (a chunk's workspace, its V), the halves' partial sums
    static constexpr int V = CW_BYTES, STAGE = V + CD_L * CD_VC * 2, XCH = CD_STAGES * STAGE, BYTES = XCH + 8 * 32 * 14 * 4;
};
// Named barriers: a chunk is there (per pair of consumer warps and parity, so that pairs drift apart and fill each other's waits), a chunk of a parity
// is done with, the two halves of a pair of consumers
constexpr int CD_FULL = 0, CD_EMPTY = 8, CD_HALVES = 10;
template <int COUNT>
__device__ __forceinline__ void cd_sync(int id) { asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(COUNT) : "memory"); }
template <int COUNT>
__device__ __forceinline__ void cd_arrive(int id) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "n"(COUNT) : "memory"); }

// powers of two for values of at most v: `up` brings them below 2^15, `down` undoes it and CD_UP.  Below 2^-97 the scale stays.
struct Pow2 {
    float up, down;
};
__device__ __forceinline__ Pow2 pow2_of(float v) {
    const uint32_t e = max(__float_as_uint(v) >> 23, 30u);
    return {__uint_as_float((268u - e) << 23), __uint_as_float((e - 28u) << 23)};
}
__device__ __forceinline__ float quad_max(float m) {
    m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 1));
    return fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 2));
}

// Eight consumer warps: warp 2 p + hf holds 16 value columns (p) and 64 of the channels (hf), so that two warps per scheduler hide each other's waits;
// a pair adds its two halves of W S and of Q S through shared memory.  Two copying warps, two chunks ahead.  Bound by the consumers' chain per chunk (tensor
// cores 45 % busy): 1.67 us a chunk.  One warp per 16 columns and all channels 4.0 us; scaling keys and queries here instead of W and Q in the first
// kernel, 2.1 us.
constexpr int CD_THREADS = 320;
__global__ void __launch_bounds__(CD_THREADS, 1) channel_delta_chunks_kernel(
    const __nv_bfloat16* __restrict__ x, int64_t stride, int v_off, const unsigned char* __restrict__ ws, float* __restrict__ state,
    const int32_t* __restrict__ state_slots, const int32_t* __restrict__ cu_q, const int32_t* __restrict__ cu_k, float* __restrict__ out, int H, int dim,
    int vdim, float q_scale, int first, int chunks) {
    B200_PDL_SYNC();
    using SM = CdSmem;
    extern __shared__ __align__(128) unsigned char cd_smem[];
    const int h = blockIdx.x, s = blockIdx.y, col0 = blockIdx.z * CD_VC, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const SeqSpan sp = seq_span(cu_q, cu_k, nullptr, s);
    const int nch = min(chunks, (sp.qlen + CD_L - 1) / CD_L - first);       // this launch's chunks
    if (nch <= 0) return;
    const uint32_t sbase = smem_u32(cd_smem);
    const int row0 = sp.q0 + first * CD_L, rows = sp.qlen - first * CD_L;   // its tokens (and the later launches')
    if (warp >= 8) {
        const int pt = threadIdx.x & 63;
        const unsigned char* wp = ws + ((int64_t)s * chunks * H + h) * (int64_t)CW_BYTES + pt * 16;
        const __nv_bfloat16* vp = x + (int64_t)row0 * stride + v_off + (int64_t)h * vdim + col0 + (pt & 7) * 8;
        const bool v_in = col0 + (pt & 7) * 8 < vdim;
        auto fetch = [&](int c) {
            if (c < nch) {
                const uint32_t d = sbase + (c & (CD_STAGES - 1)) * SM::STAGE;
                const unsigned char* wc = wp + (int64_t)c * H * CW_BYTES;
                static_assert(CW_BYTES % 1024 == 512, "whole rounds of 64 pieces and half a one");
#pragma unroll 9
                for (int i = 0; i < CW_BYTES / 1024; ++i) wm_cp16(d + pt * 16 + i * 1024, wc + i * 1024, 16);
                if (pt < 32) wm_cp16(d + pt * 16 + CW_BYTES / 1024 * 1024, wc + CW_BYTES / 1024 * 1024, 16);
#pragma unroll
                for (int i = 0; i < 2; ++i) {               // rows past the end and columns past vdim: zeros
                    const int r = (pt >> 3) + 8 * i;
                    const bool have = v_in && c * CD_L + r < rows;
                    wm_cp16(d + SM::V + val_swz(r, pt & 7), have ? vp + (int64_t)(c * CD_L + r) * stride : x, have ? 16 : 0);
                }
            }
            wm_commit();
        };
        fetch(0);
        fetch(1);
        for (int c = 0; c < nch; ++c) {
            if (c >= 2) cd_sync<320>(CD_EMPTY + (c & 1));   // all are done with chunk c - 2, whose stage chunk c + 2 takes
            fetch(c + 2);
            wm_wait<2>();                                   // this thread's part of chunk c
#pragma unroll
            for (int i = 0; i < 4; ++i) cd_arrive<128>(CD_FULL + 2 * i + (c & 1));
        }
        return;
    }
    // ---- consumers ----
    const int hf = warp & 1, vw = warp >> 1, gq = lane >> 2, t4 = lane & 3, vrow = col0 + vw * 16 + gq;
    constexpr int NT = CD_D / 16, KT = CD_D / 32;           // 8-column tiles and 16-deep steps of this half's 64 channels
    const int ch0 = hf * (CD_D / 2);
    float* stp = state + ((int64_t)state_slots[s] * H + h) * vdim * dim + ch0;
    const bool has_hist = first > 0 || sp.klen - sp.qlen > 0, live = col0 + vw * 16 < vdim;
    const int br = (lane & 7) + ((lane >> 4) << 3), kr = (lane & 7) + (((lane >> 3) & 1) << 3), bp = (lane >> 3) & 1;
    float* mine = reinterpret_cast<float*>(cd_smem + SM::XCH) + warp * (32 * 14) + lane;
    const float* other = reinterpret_cast<const float*>(cd_smem + SM::XCH) + (warp ^ 1) * (32 * 14) + lane;
    uint64_t S[NT][2];                                      // rows gq, gq + 8 of the pair's 16 value columns, channels ch0 + n * 8 + 2 t4, + 1
    float m0 = 0.f, m1 = 0.f;                               // largest magnitude of either row over all channels (a NaN need not count: its row is lost)
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
            float2 f = make_float2(0.f, 0.f);
            if (has_hist && vrow + 8 * hh < vdim && ch0 + n * 8 < dim) f = *reinterpret_cast<const float2*>(stp + (int64_t)(vrow + 8 * hh) * dim + n * 8 + 2 * t4);
            S[n][hh] = cd_pack(f.x, f.y);
            float& m = hh ? m1 : m0;
            m = fmaxf(m, fmaxf(fabsf(f.x), fabsf(f.y)));
        }
    mine[12 * 32] = m0 = quad_max(m0), mine[13 * 32] = m1 = quad_max(m1);
    if (live) cd_sync<64>(CD_HALVES + vw);
    m0 = fmaxf(m0, other[12 * 32]), m1 = fmaxf(m1, other[13 * 32]);
    // V^T [16 columns x 16 tokens] (as loaded) times a lower triangular matrix of the stage, by multiply-adds over the places on and below its diagonal
    // alone: for chunks whose V holds an infinity or a NaN, which a product with the zeros above would carry to earlier tokens
    auto triangle = [&](const unsigned char* mat, const uint32_t (&va)[4], float (&Y)[2][4]) {
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e) Y[i][e] = 0.f;
#pragma unroll 1
        for (int i = 0; i < CD_L; ++i) {
            const int from = (lane & ~3) | ((i & 7) >> 1);
            const uint32_t a = __shfl_sync(0xffffffffu, i < 8 ? va[0] : va[2], from), b = __shfl_sync(0xffffffffu, i < 8 ? va[1] : va[3], from);
            const float x0 = i & 1 ? bf16hi(a) : bf16lo(a), x1 = i & 1 ? bf16hi(b) : bf16lo(b);
#pragma unroll
            for (int jj = 0; jj < 2; ++jj)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int place = jj * 8 + 2 * t4 + e;
                    if (i <= token_at(place)) {
                        const __nv_bfloat16* p = reinterpret_cast<const __nv_bfloat16*>(mat + mat_row(place, i));
                        const float f = __bfloat162float(p[0]) + (__bfloat162float(p[CW_MAT / 2]) + __bfloat162float(p[CW_MAT]));
                        Y[jj][e] = fmaf(f, x0, Y[jj][e]);
                        Y[jj][2 + e] = fmaf(f, x1, Y[jj][2 + e]);
                    }
                }
        }
    };
    for (int c = 0; c < nch; ++c) {
        const unsigned char* sm = cd_smem + (c & (CD_STAGES - 1)) * SM::STAGE;
        const uint32_t sb = sbase + (c & (CD_STAGES - 1)) * SM::STAGE;
        const Pow2 s0 = pow2_of(m0), s1 = pow2_of(m1);
        // S as fp16 pairs, the left operand of W S and Q S
        uint32_t ah[KT][4], al[KT][4];
#pragma unroll
        for (int kk = 0; kk < KT; ++kk)
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                split_f16(cd_mul2(S[2 * kk + i][0], cd_pack(s0.up, s0.up)), ah[kk][2 * i], al[kk][2 * i]);
                split_f16(cd_mul2(S[2 * kk + i][1], cd_pack(s1.up, s1.up)), ah[kk][2 * i + 1], al[kk][2 * i + 1]);
            }
        cd_sync<128>(CD_FULL + 2 * vw + (c & 1));
        if (live) {
            // this half's part of rows [16 tokens] x S: the large product apart from the two small ones
            auto rows_times_state = [&](int at, float (&R)[2][4]) {
                float P[2][4], Q[2][4];
#pragma unroll
                for (int kk = 0; kk < KT; ++kk) {
                    uint32_t b[4], d[4];
                    wm_ldsm_t(sb + at + row_swz(ch0 + kk * 16 + kr, lane >> 4), b[0], b[1], b[2], b[3]);
                    wm_ldsm_t(sb + at + CW_ROWS + row_swz(ch0 + kk * 16 + kr, lane >> 4), d[0], d[1], d[2], d[3]);
#pragma unroll
                    for (int i = 0; i < 2; ++i) kk ? mma_f16(Q[i], al[kk], b[2 * i], b[2 * i + 1]) : mma_f16_new(Q[i], al[kk], b[2 * i], b[2 * i + 1]);
#pragma unroll
                    for (int i = 0; i < 2; ++i) kk ? mma_f16(P[i], ah[kk], b[2 * i], b[2 * i + 1]) : mma_f16_new(P[i], ah[kk], b[2 * i], b[2 * i + 1]);
#pragma unroll
                    for (int i = 0; i < 2; ++i) mma_f16(Q[i], ah[kk], d[2 * i], d[2 * i + 1]);
                }
#pragma unroll
                for (int i = 0; i < 2; ++i)
#pragma unroll
                    for (int e = 0; e < 4; ++e) R[i][e] = P[i][e] + Q[i][e];
            };
            uint32_t va[4];
            wm_ldsm_t(sb + SM::V + val_swz(br, vw * 2 + bp), va[0], va[1], va[2], va[3]);
            float U[2][4], O[2][4], Y[2][4];
            rows_times_state(CW_W, U);
            // T V by the first half of the channels, (B T) V by both (a tile of eight tokens each is used): small terms first
            auto times_values = [&](int mat, float (&D)[2][4]) {
                uint32_t b[4];
#pragma unroll
                for (int i = 0; i < 2; ++i) D[i][0] = D[i][1] = D[i][2] = D[i][3] = 0.f;
#pragma unroll
                for (int m = 2; m >= 0; --m) {
                    wm_ldsm(sb + mat + m * CW_MAT + row_swz(br, bp), b[0], b[1], b[2], b[3]);
#pragma unroll
                    for (int i = 0; i < 2; ++i) wm_mma(D[i], va[0], va[1], va[2], va[3], b[2 * i], b[2 * i + 1]);
                }
            };
            uint32_t odd = 0;                               // an exponent of ones carries into the sign's place
#pragma unroll
            for (int i = 0; i < 4; ++i) odd |= (va[i] & 0x7f807f80u) + 0x00800080u;
            const bool whole = __all_sync(0xffffffffu, !(odd & 0x80008000u));
            if (hf == 0) {
                times_values(CW_T, Y);
                if (!whole) triangle(sm + CW_T, va, Y);
#pragma unroll
                for (int i = 0; i < 2; ++i)
#pragma unroll
                    for (int e = 0; e < 4; ++e) mine[(4 * i + e) * 32] = U[i][e] = fmaf(-(e < 2 ? s0.down : s1.down), U[i][e], Y[i][e]);
            } else {
#pragma unroll
                for (int i = 0; i < 2; ++i)
#pragma unroll
                    for (int e = 0; e < 4; ++e) mine[(4 * i + e) * 32] = U[i][e] = -(e < 2 ? s0.down : s1.down) * U[i][e];
            }
            // |U| <= 16 max |V| + sqrt(128) max |S|: rows of W and entries of T are at most one
            const float v0 = quad_max(fmaxf(fmaxf(fabsf(bf16lo(va[0])), fabsf(bf16hi(va[0]))), fmaxf(fabsf(bf16lo(va[2])), fabsf(bf16hi(va[2])))));
            const float v1 = quad_max(fmaxf(fmaxf(fabsf(bf16lo(va[1])), fabsf(bf16hi(va[1]))), fmaxf(fabsf(bf16lo(va[3])), fabsf(bf16hi(va[3])))));
            const Pow2 p0 = pow2_of(fmaf(16.f, v0, 12.f * m0)), p1 = pow2_of(fmaf(16.f, v1, 12.f * m1));
            cd_sync<64>(CD_HALVES + vw);
            uint32_t xh[4], xl[4];
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int e = 0; e < 4; e += 2) {
                    const uint64_t u = cd_add2(cd_pack(U[i][e], U[i][e + 1]), cd_pack(other[(4 * i + e) * 32], other[(4 * i + e + 1) * 32]));
                    split_f16(cd_mul2(u, e ? cd_pack(p1.up, p1.up) : cd_pack(p0.up, p0.up)), xh[2 * i + e / 2], xl[2 * i + e / 2]);
                }
            // S^T <- P_16 S^T + U^T (R k)
            float D[NT][4];
            uint32_t b[NT / 2][4], d[NT / 2][4];
#pragma unroll
            for (int n = 0; n < NT; n += 2) wm_ldsm(sb + CW_R + row_swz(ch0 + n * 8 + br, bp), b[n / 2][0], b[n / 2][1], b[n / 2][2], b[n / 2][3]);
#pragma unroll
            for (int n = 0; n < NT; n += 2)
                wm_ldsm(sb + CW_R + CW_ROWS + row_swz(ch0 + n * 8 + br, bp), d[n / 2][0], d[n / 2][1], d[n / 2][2], d[n / 2][3]);
#pragma unroll
            for (int n = 0; n < NT; ++n) mma_f16_new(D[n], xl, b[n / 2][2 * (n & 1)], b[n / 2][2 * (n & 1) + 1]);
#pragma unroll
            for (int n = 0; n < NT; ++n) mma_f16(D[n], xh, d[n / 2][2 * (n & 1)], d[n / 2][2 * (n & 1) + 1]);
#pragma unroll
            for (int n = 0; n < NT; ++n) mma_f16(D[n], xh, b[n / 2][2 * (n & 1)], b[n / 2][2 * (n & 1) + 1]);
            rows_times_state(CW_Q, O);
            times_values(CW_BT, Y);
            if (!whole) triangle(sm + CW_BT, va, Y);
            // the half's tile of the output: its own sums and the other half's
#pragma unroll
            for (int e = 0; e < 4; ++e) mine[(8 + e) * 32] = hf ? O[0][e] : O[1][e];
            m0 = m1 = 0.f;
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                const uint64_t g = *reinterpret_cast<const uint64_t*>(sm + CW_P + (ch0 + n * 8 + 2 * t4) * 4);
                S[n][0] = cd_fma2(g, S[n][0], cd_mul2(cd_pack(D[n][0], D[n][1]), cd_pack(p0.down, p0.down)));
                S[n][1] = cd_fma2(g, S[n][1], cd_mul2(cd_pack(D[n][2], D[n][3]), cd_pack(p1.down, p1.down)));
                const float2 u = cd_two(S[n][0]), v = cd_two(S[n][1]);
                m0 = fmaxf(m0, fmaxf(fabsf(u.x), fabsf(u.y)));
                m1 = fmaxf(m1, fmaxf(fabsf(v.x), fabsf(v.y)));
            }
            mine[12 * 32] = m0 = quad_max(m0), mine[13 * 32] = m1 = quad_max(m1);
            cd_sync<64>(CD_HALVES + vw);
            const float w0 = s0.down * q_scale, w1 = s1.down * q_scale;
            m0 = fmaxf(m0, other[12 * 32]), m1 = fmaxf(m1, other[13 * 32]);
            const int t = c * CD_L + token_at(hf * 8 + 2 * t4);             // the lane's places 2 t4 and 2 t4 + 1 of the tile are neighbours
            float* op = out + ((int64_t)(row0 + t) * H + h) * vdim + vrow;
#pragma unroll
            for (int e = 0; e < 4; ++e) {                   // token t + (e & 1), column gq or gq + 8
                const float o = fmaf((hf ? O[1][e] : O[0][e]) + other[(8 + e) * 32], e < 2 ? w0 : w1, (hf ? Y[1][e] : Y[0][e]) * q_scale);
                if (t + (e & 1) < rows && vrow + 8 * (e >> 1) < vdim) op[(int64_t)(e & 1) * H * vdim + 8 * (e >> 1)] = o;
            }
        }
        if (c + 2 < nch) cd_arrive<320>(CD_EMPTY + (c & 1));
    }
    if (live) {
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int hh = 0; hh < 2; ++hh)
                if (vrow + 8 * hh < vdim && ch0 + n * 8 < dim)
                    *reinterpret_cast<uint64_t*>(stp + (int64_t)(vrow + 8 * hh) * dim + n * 8 + 2 * t4) = S[n][hh];
    }
}

// Chunks of every sequence that a launch pair handles: what a workspace of WS_BOUND bytes holds, but at least one
constexpr int64_t WS_BOUND = 256ll << 20;
int64_t chunks_per_launch(int num_seqs, int max_q, int num_heads) {
    const int64_t all = ((int64_t)max_q + CD_L - 1) / CD_L, fit = WS_BOUND / ((int64_t)num_seqs * num_heads * CW_BYTES);
    return all < fit ? all : fit > 0 ? fit : 1;
}

}  // namespace

extern "C" size_t b200m_channel_delta_workspace_bytes(int num_seqs, int max_q, int num_heads) {
    if (max_q <= 0 || num_seqs <= 0 || num_heads <= 0) return (size_t)WS_BOUND;
    return (size_t)chunks_per_launch(num_seqs, max_q, num_heads) * num_seqs * (size_t)num_heads * CW_BYTES;
}

extern "C" int b200m_channel_delta_prompts(const void* x, int64_t stride, int q_off, int k_off, int v_off, const void* write_in, int64_t write_stride,
                                           const float* decay_in, int64_t decay_stride, const float* rate, const float* decay_bias, float decay_sign,
                                           float* state, const int32_t* state_slots, const int32_t* cu_q, const int32_t* cu_k, float* out, int n,
                                           int num_seqs, int max_q, int num_heads, int num_kv_heads, int dim, int vdim, float q_scale, void* workspace,
                                           size_t workspace_bytes, void* stream) {
    if (!x || !write_in || !decay_in || !state || !state_slots || !out || !rate || !decay_bias || !cu_q || !cu_k) return B200_EINVAL;
    if (num_heads <= 0 || num_kv_heads <= 0 || num_heads % num_kv_heads || dim <= 0 || vdim <= 0) return B200_EINVAL;
    if (decay_stride < (int64_t)num_heads * dim || n < 0 || max_q < 0) return B200_EINVAL;
    if (dim > CD_D || dim % 8 || vdim % 8 || stride % 8 || q_off % 8 || k_off % 8 || v_off % 8 || decay_stride % 4) return B200_EUNSUPPORTED;
    for (const void* p : {x, static_cast<const void*>(decay_in), static_cast<const void*>(decay_bias), static_cast<const void*>(state),
                          static_cast<const void*>(workspace)})
        if (reinterpret_cast<uintptr_t>(p) % 16) return B200_EUNSUPPORTED;
    if (num_seqs <= 0 || n == 0 || max_q == 0) return B200_OK;
    if (num_seqs > 65535 || decay_stride > (1 << 27) || (vdim + CD_VC - 1) / CD_VC > 65535) return B200_EUNSUPPORTED;
    if (!workspace || workspace_bytes < b200m_channel_delta_workspace_bytes(num_seqs, max_q, num_heads)) return B200_EINVAL;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const __nv_bfloat16* xb = static_cast<const __nv_bfloat16*>(x);
    unsigned char* ws = static_cast<unsigned char*>(workspace);
    const int all = (max_q + CD_L - 1) / CD_L, chunks = (int)chunks_per_launch(num_seqs, max_q, num_heads);
    const int64_t blocks = (int64_t)num_heads * chunks;
    if (blocks > 0x7fffffff) return B200_EUNSUPPORTED;
    static B200SmemOptIn opt, opt_prepare;
    if (opt.ensure(channel_delta_chunks_kernel, CdSmem::BYTES) != cudaSuccess) return B200_ECUDA;
    if (opt_prepare.ensure(channel_delta_prepare_kernel, CpSmem::BYTES) != cudaSuccess) return B200_ECUDA;
    for (int first = 0; first < all; first += chunks) {
        B200_LAUNCH((channel_delta_prepare_kernel), dim3((unsigned)blocks, num_seqs), CP_THREADS, CpSmem::BYTES, st, xb, stride, q_off,
                    k_off, static_cast<const __nv_bfloat16*>(write_in), write_stride, decay_in, decay_stride, rate, decay_bias, decay_sign, cu_q, ws,
                    num_heads, num_kv_heads, dim, first, chunks);
        if (const int rc = b200_launch_status(nullptr); rc != B200_OK) return rc;
        B200_LAUNCH((channel_delta_chunks_kernel), dim3(num_heads, num_seqs, (vdim + CD_VC - 1) / CD_VC), CD_THREADS, CdSmem::BYTES, st, xb, stride, v_off,
                    static_cast<const unsigned char*>(ws), state, state_slots, cu_q, cu_k, out, num_heads, dim, vdim, q_scale, first, chunks);
        if (const int rc = b200_launch_status(nullptr); rc != B200_OK) return rc;
    }
    return B200_OK;
}
