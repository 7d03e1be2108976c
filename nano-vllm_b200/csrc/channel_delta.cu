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
// Precision: an operand of a product is fp32 in three bf16 terms (3 x 8 bits: nothing is lost) and six of the nine partial products are taken (the others are
// below 2^-26), the largest ones apart and added outside the tensor cores, which cut sums off where the fp32 pipe rounds.  V is bf16 as it is.  S itself is fp32.
// No scales: bf16 has fp32's range, so a state or a read-out that strong decays have made small keeps its bits.  Against float64 the results are 0.9e-7 to 3.1e-7
// of their norm off and the state 0.5e-7 to 3.7e-7, the fp32-pipe form of recurrent_mix.cu 1.0e-7 to 18.5e-7 and 0.8e-7 to 23e-7.  (That one is closer, 0.8e-7 for 1.0e-7,
// where strong decays leave a state of a token or two: keys are rounded once more here.)  With fp16 pairs, 22 bits and half of the products, it was 1.2e-7 to 3.5e-7, and
// nothing was left of a state below 2^-25 of one; both kernels together took 350 us where these take 447.
//
// Measured on a B200, 16 heads of 128 x 128, both kernels together against that form: 4 x 2048 tokens 447 us against 669, 1 x 4096 634 against
// 1314, 16 x 1000 872 against 1127, 12 x 600 408 against 544, 16 x 64 71 against 84, 1 x 2048 beside 511 single tokens 870 against 1130.  With the workspace laid out as
// sequences x longest portion, and a launch pair for what of that fitted 256 MiB, that last step was 128 pairs of nearly empty grids and took 6.7 ms.
#include "mma_common.cuh"
#include "state_common.cuh"

namespace {

constexpr int CD_L = 16, CD_D = 128, CD_VC = 64, CD_STAGES = 4;
// Workspace of one (chunk, head), a stage of the walk as it lies in shared memory: W, Q, R k in three bf16 terms each (rows of the first, of the second, of the
// third), a row of sixteen tokens per channel; T and B T as three bf16 matrices [16][16] each, a row per token; P_16 in fp32.  Tokens of a channel's row (and the rows of T and B T) stand
// in the order 0 1 8 9 2 3 10 11 ..., which is how a product's accumulators hold them.  The two 16-byte pieces of a row change places every four
// rows, so that a piece of eight rows lies in eight bank groups.
constexpr int CW_ROWS = CD_D * CD_L * 2, CW_W = 0, CW_Q = 3 * CW_ROWS, CW_R = 6 * CW_ROWS, CW_MAT = CD_L * CD_L * 2, CW_T = 9 * CW_ROWS,
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
__device__ __forceinline__ void add4(float (&a)[4], const float (&b)[4]) {
#pragma unroll
    for (int e = 0; e < 4; e += 2) {
        const float2 f = cd_two(cd_add2(cd_pack(a[e], a[e + 1]), cd_pack(b[e], b[e + 1])));
        a[e] = f.x, a[e + 1] = f.y;
    }
}
__device__ __forceinline__ float cd_sum(uint64_t v) {
    const float2 f = cd_two(v);
    return f.x + f.y;
}
// Rows of the workspace (a row: a chunk, all heads).  Sequence s has those from here on, a place that needs no sum over the sequences in front of it:
// ceil(l / 16) <= floor((q + l) / 16) - floor(q / 16) + 1, so n / 16 + sequences rows hold every step of n tokens, whatever its lengths.
__device__ __forceinline__ int chunk_row(int q0, int s) { return q0 / CD_L + s; }
// The sequence that a row is of (-1: none), 128 at a time by a whole warp
__device__ __forceinline__ int row_sequence(const int32_t* __restrict__ cu_q, int num_seqs, int row, int lane) {
    int upto = 0;
    for (int s0 = 0; s0 < num_seqs; s0 += 128) {
        int start[4], have = 0;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int s = s0 + 32 * i + lane;
            start[i] = s < num_seqs ? chunk_row(cu_q[s], s) : 0x7fffffff;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) have += __popc(__ballot_sync(0xffffffffu, start[i] <= row));
        upto += have;
        if (have < 128) break;
    }
    return upto - 1;
}
// a pair of floats -> three bf16 terms each: their roundings, the roundings of what these leave, and the rest.  3 x 8 bits: nothing is lost
__device__ __forceinline__ void split3(uint64_t v, uint32_t& a, uint32_t& b, uint32_t& c) {
    const float2 f = cd_two(v);
    asm("{\n\t.reg .b16 s, t, m;\n\t.reg .f32 x, y;\n\tmov.b16 m, 0xBF80;\n\t"
        "cvt.rn.bf16x2.f32 %0, %4, %3;\n\tmov.b32 {s, t}, %0;\n\t"
        "fma.rn.f32.bf16 x, s, m, %3;\n\tfma.rn.f32.bf16 y, t, m, %4;\n\t"
        "cvt.rn.bf16x2.f32 %1, y, x;\n\tmov.b32 {s, t}, %1;\n\t"
        "fma.rn.f32.bf16 x, s, m, x;\n\tfma.rn.f32.bf16 y, t, m, y;\n\t"
        "cvt.rn.bf16x2.f32 %2, y, x;\n\t}"
        : "=&r"(a), "=&r"(b), "=r"(c)
        : "f"(f.x), "f"(f.y));
}
// exp(rate softplus(x)), rate <= 0: softplus(x) = max(x, 0) + log1p(exp(-|x|)), log1p(y) / y over [0, 1] and (2^f - 1) / f over [-1/2, 1/2] as polynomials
// (weighted least squares, reweighted until the ripples are equal (Lawson); coefficients rounded one by one, the rest fitted again; the first of log1p is
// one).  Off by 3.3e-8 of log1p(y) and 3e-9 of 2^f, before fp32's own rounding.  The exponent is reduced in two parts (Cody and Waite).  2^f is 1 + f (...), so
// that a decay next to one is rounded once: the power unit's last bits add up over a sequence.  Over |x| <= 100 and rates of -1e-3 to -16 no further from
// float64 than expf and log1pf (rate -400: 1.5 times).  Below 2^-126: zero.
__device__ __forceinline__ float decay_fit(float x, float rate) {
    constexpr float L[9] = {1.f, -0.49999648f, 0.3332133f, -0.24857217f, 0.19153848f, -0.13754188f, 0.07920883f, -0.0300683f, 0.0053654225f};
    constexpr float Q[6] = {0.6931472f, 0.24022648f, 0.0555036f, 0.009618506f, 0.0013390806f, 0.00015326463f};
    constexpr float MAGIC = 12582912.f, LOG2E = 1.44269502f, LOG2E_REST = 1.92596299e-8f;           // 1.5 x 2^23; log2(e) in two parts
    float y, m, r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(fminf(fabsf(x), 80.f) * -LOG2E));
    float p = L[8];
#pragma unroll
    for (int i = 7; i >= 0; --i) p = fmaf(p, y, L[i]);
    asm("max.NaN.f32 %0, %1, 0f00000000;" : "=f"(m) : "f"(x));
    const float v = fmaf(p, y, m) * rate;
    asm("max.NaN.f32 %0, %1, 0fC2AEAC4F;" : "=f"(r) : "f"(v));                                      // -126 ln 2
    const float n = fmaf(r, LOG2E, MAGIC), k = n - MAGIC, f = fmaf(r, LOG2E_REST, fmaf(r, LOG2E, -k));
    float q = Q[5];
#pragma unroll
    for (int i = 4; i >= 0; --i) q = fmaf(q, f, Q[i]);
    return v < -87.33654f ? 0.f : fmaf(q, f, 1.f) * __uint_as_float(__float_as_uint(n) * 0x800000u + 0x3f800000u);
}
__device__ __forceinline__ void mma_bf(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// the same from zero
__device__ __forceinline__ void mma_bf_new(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}
// the five small partial products of two operands of three terms each, from the smallest; `fresh`: from zero
__device__ __forceinline__ void mma_rest(float (&c)[4], const uint32_t (&a)[3][4], const uint32_t (&b)[3][2], bool fresh) {
    if (fresh) mma_bf_new(c, a[2], b[0][0], b[0][1]);
    else mma_bf(c, a[2], b[0][0], b[0][1]);
    mma_bf(c, a[0], b[2][0], b[2][1]);
    mma_bf(c, a[1], b[1][0], b[1][1]);
    mma_bf(c, a[1], b[0][0], b[0][1]);
    mma_bf(c, a[0], b[1][0], b[1][1]);
}

// ---- first kernel: decays, A, B, T, W, Q ------------------------------------------------------------------------------------------------
// A_ts and B_ts need the decays between s and t.  Pairs of tokens are taken by the largest of four levels (half blocks of 8, 4, 2, 1 tokens) whose middle
// parts them: with the middle m, k_t and q_t take g_m ... g_t, k_s takes g_(s+1) ... g_(m-1), all at most one, and a level is one product of
// [8 k rows, 8 q rows] with [8 k rows].  Bound by its instructions (2880 a thread, 0.53 per cycle and scheduler): 161 us for
// 8192 tokens of 16 heads (operands as fp16 pairs 137).
constexpr int CP_THREADS = 128;
struct CpSmem {
    static constexpr int RAW_K = 0, RAW_Q = CD_L * CD_D * 2, A = 2 * RAW_Q, B = A + CD_L * CD_L * 4, T = B + CD_L * CD_L * 4,
                         MAT = T + CD_L * CD_L * 4,                          // T, -B T in three bf16 terms, rows of tokens
                         NORM = MAT + 6 * CW_MAT,                            // normalisers of k, of q, strengths
                         FACT = NORM + 3 * CD_L * 4, FROW = CD_D * 16,       // [two levels][k left, q left, k right][term]: rows of eight tokens per channel
                         PK = FACT, PQ = PK + 3 * CW_ROWS, PQ_STRIDE = 18,   // in their place: P k in three terms, P q (fp32)
                         BYTES = FACT + 18 * FROW;
    static_assert(PQ + CD_D * PQ_STRIDE * 4 <= BYTES, "");
};
// A channel's factors of a level: places 2 i and 2 i + 1 of its eight left and eight right tokens
template <int T>
__device__ __forceinline__ float cd_at(const uint64_t (&v)[CD_L / 2]) {
    const float2 f = cd_two(v[T / 2]);
    return T & 1 ? f.y : f.x;
}
template <int LEVEL, int A>
__device__ __forceinline__ void level_left(const uint64_t (&g)[CD_L / 2], float (&l)[8]) {              // from the first place to the last
    constexpr int N = 8 >> LEVEL, T = A / N * 2 * N + N + A % N;
    if constexpr (A % N == 0) l[A] = cd_at<T>(g);
    else l[A] = l[A - 1] * cd_at<T>(g);
    if constexpr (A < 7) level_left<LEVEL, A + 1>(g, l);
}
template <int LEVEL, int A>
__device__ __forceinline__ void level_right(const uint64_t (&g)[CD_L / 2], float (&R)[8]) {             // from the last place to the first
    constexpr int N = 8 >> LEVEL, T = A / N * 2 * N + A % N;
    if constexpr (A % N == N - 1) R[A] = 1.f;
    else R[A] = R[A + 1] * cd_at<T + 1>(g);
    if constexpr (A > 0) level_right<LEVEL, A - 1>(g, R);
}
// the eight entries of v that a level's left (or right) tokens have, times f, in three terms
template <int LEVEL, bool LEFT, int I>
__device__ __forceinline__ void level_pair(const uint64_t (&v)[CD_L / 2], const float (&f)[8], uint32_t (&w)[3][4]) {
    constexpr int N = 8 >> LEVEL, UP = LEFT ? N : 0, A0 = 2 * I, A1 = A0 + 1, T0 = A0 / N * 2 * N + UP + A0 % N, T1 = A1 / N * 2 * N + UP + A1 % N;
    uint64_t e = cd_pack(cd_at<T0>(v), cd_at<T1>(v));
    if constexpr (LEFT || N > 1) e = cd_mul2(e, cd_pack(f[A0], f[A1]));              // (single tokens to the right: factors of one)
    split3(e, w[0][I], w[1][I], w[2][I]);
    if constexpr (I < 3) level_pair<LEVEL, LEFT, I + 1>(v, f, w);
}
template <int LEVEL, bool LEFT>
__device__ __forceinline__ void level_rows(const uint64_t (&v)[CD_L / 2], const float (&f)[8], unsigned char* to) {
    uint32_t w[3][4];
    level_pair<LEVEL, LEFT, 0>(v, f, w);
#pragma unroll
    for (int i = 0; i < 3; ++i) *reinterpret_cast<uint4*>(to + i * (CD_D * 16)) = make_uint4(w[i][0], w[i][1], w[i][2], w[i][3]);
}
template <int LEVEL>
__device__ __forceinline__ void level_factors(const uint64_t (&g)[CD_L / 2], const uint64_t (&k)[CD_L / 2], const uint64_t (&q)[CD_L / 2], unsigned char* to) {
    float f[8];
    level_left<LEVEL, 0>(g, f);
    level_rows<LEVEL, true>(k, f, to);
    level_rows<LEVEL, true>(q, f, to + 3 * CD_D * 16);
    level_right<LEVEL, 7>(g, f);
    level_rows<LEVEL, false>(k, f, to + 6 * CD_D * 16);
}
__global__ void __launch_bounds__(CP_THREADS, 4) channel_delta_prepare_kernel(
    const __nv_bfloat16* __restrict__ x, int64_t stride, int q_off, int k_off, const __nv_bfloat16* __restrict__ write_in, int64_t write_stride,
    const float* __restrict__ decay_in, int64_t decay_stride, const float* __restrict__ rate, const float* __restrict__ bias, float sign,
    const int32_t* __restrict__ cu_q, unsigned char* __restrict__ ws, int num_seqs, int H, int G, int dim, int first_row) {
    B200_PDL_SYNC();
    using SM = CpSmem;
    extern __shared__ __align__(128) unsigned char cp_smem[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, gq = lane >> 2, t4 = lane & 3;
    const int h = blockIdx.x % H, row = first_row + blockIdx.x / H, s = row_sequence(cu_q, num_seqs, row, lane);
    if (s < 0) return;
    const int q0 = cu_q[s], qlen = cu_q[s + 1] - q0, t0 = (row - chunk_row(q0, s)) * CD_L;
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
        const float rt = rate[h], b = sign * bias[(int64_t)h * dim + (in ? tid : 0)];
        if (tid < CD_L) norm[2 * CD_L + tid] = tid < len ? sigmoidf_(__bfloat162float(write_in[(int64_t)(q0 + t0 + tid) * write_stride + h])) : 0.f;
        reinterpret_cast<float4*>(A)[tid] = make_float4(0.f, 0.f, 0.f, 0.f);            // A and B: zeros above their diagonals
#pragma unroll
        for (int t = 0; t < CD_L; ++t) z[t] = decay_fit(fmaf(sign, z[t], b), rt);
        if (len < CD_L) {                                   // behind the end nothing decays, and keys and queries are zeros
#pragma unroll
            for (int t = 0; t < CD_L; ++t) z[t] = t < len ? z[t] : 1.f;
        }
#pragma unroll
        for (int i = 0; i < CD_L / 2; ++i) g[i] = cd_pack(z[2 * i], z[2 * i + 1]);
    }
    wm_wait<0>();
    __syncthreads();
    // k.k and q.q of every token: the diagonals of two products of the rows as they are.  k.q on the fp32 pipe, eight threads a token: where its terms cancel, a
    // product that cuts them off at the largest one is several times further off
    const int ar = lane & 15, br = (lane & 7) + ((lane >> 4) << 3), bp = (lane >> 3) & 1;
    {
        const int r = tid >> 3;
        float sum[2] = {0.f, 0.f};
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            float f[8], e[8];
            unpack8(*reinterpret_cast<const uint4*>(cp_smem + SM::RAW_K + raw_swz(r, (tid & 7) + 8 * i)), f);
            unpack8(*reinterpret_cast<const uint4*>(cp_smem + SM::RAW_Q + raw_swz(r, (tid & 7) + 8 * i)), e);
#pragma unroll
            for (int j = 0; j < 8; ++j) sum[i] = fmaf(f[j], e[j], sum[i]);
        }
        float v = sum[0] + sum[1];
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if ((tid & 7) == 0) B[r * (CD_L + 1)] = v;
    }
    if (warp < 2) {
        const uint32_t ra = sbase + (warp == 0 ? SM::RAW_K : SM::RAW_Q);
        float lo = 0.f, hi = 0.f;                           // places (gq, gq) and (gq + 8, gq + 8), of the lanes with t4 == gq / 2
#pragma unroll
        for (int kk = 0; kk < CD_D / 16; ++kk) {            // sixteen channels a product, the eight added here: a product's own sums are cut off, not rounded
            uint32_t a[4], b[4];
            float D[2][4] = {};
            wm_ldsm(ra + raw_swz(ar, kk * 2 + (lane >> 4)), a[0], a[1], a[2], a[3]);
            wm_ldsm(ra + raw_swz(br, kk * 2 + bp), b[0], b[1], b[2], b[3]);
            wm_mma(D[0], a[0], a[1], a[2], a[3], b[0], b[1]);
            wm_mma(D[1], a[0], a[1], a[2], a[3], b[2], b[3]);
            lo += gq & 1 ? D[0][1] : D[0][0];
            hi += gq & 1 ? D[1][3] : D[1][2];
        }
        if (t4 == gq >> 1) {
            norm[warp * CD_L + gq] = 1.0f / sqrtf(lo + 1e-6f);
            norm[warp * CD_L + gq + 8] = 1.0f / sqrtf(hi + 1e-6f);
        }
    }
    __syncthreads();
    if (tid < CD_L) B[tid * (CD_L + 1)] *= norm[tid] * norm[CD_L + tid];
    uint64_t k[CD_L / 2], q[CD_L / 2];                      // unit rows' entries of this channel
#pragma unroll
    for (int i = 0; i < CD_L / 2; ++i) {
        float v[4];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const uint32_t at = raw_swz(2 * i + e, tid >> 3) + (tid & 7) * 2;
            v[e] = __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(cp_smem + SM::RAW_K + at));
            v[2 + e] = __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(cp_smem + SM::RAW_Q + at));
        }
        k[i] = cd_mul2(cd_pack(v[0], v[1]), *reinterpret_cast<const uint64_t*>(norm + 2 * i));
        q[i] = cd_mul2(cd_pack(v[2], v[3]), *reinterpret_cast<const uint64_t*>(norm + CD_L + 2 * i));
    }
    // two levels at a time: a warp has half of the channels of one, and its sums meet the other half's in A and B (two additions onto zero)
    auto level_sums = [&](int n) {
        const uint32_t f = sbase + SM::FACT + (warp >> 1) * 9 * SM::FROW + (warp & 1) * (CD_D / 2) * 16;
        const int m = lane >> 3, r8 = lane & 7;             // which of four 8 x 8 tiles this lane's address is for
        float D[4], E[4];
#pragma unroll
        for (int kk = 0; kk < CD_D / 32; ++kk) {
            uint32_t a[3][4], b[3][2], skip[2];
            const uint32_t ra = f + (m & 1) * 3 * SM::FROW + (kk * 16 + (m >> 1) * 8 + r8) * 16, rb = f + 6 * SM::FROW + (kk * 16 + (m & 1) * 8 + r8) * 16;
#pragma unroll
            for (int i = 0; i < 3; ++i) wm_ldsm_t(ra + i * SM::FROW, a[i][0], a[i][1], a[i][2], a[i][3]);
            wm_ldsm_t(rb + (m >> 1) * SM::FROW, b[0][0], b[0][1], b[1][0], b[1][1]);
            wm_ldsm_t(rb + 2 * SM::FROW, b[2][0], b[2][1], skip[0], skip[1]);
            float P[4];
            mma_bf_new(kk ? P : D, a[0], b[0][0], b[0][1]);
            mma_rest(E, a, b, kk == 0);
            if (kk) add4(D, P);
        }
        const int sh = 31 - __clz(n), t = ((gq >> sh) << (sh + 1)) + n + (gq & (n - 1));
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int j = 2 * t4 + e;
            if (gq >> sh == j >> sh) {
                const int at = t * CD_L + ((j >> sh) << (sh + 1)) + (j & (n - 1));
                atomicAdd(A + at, D[e] + E[e]);
                atomicAdd(B + at, D[2 + e] + E[2 + e]);
            }
        }
    };
    level_factors<0>(g, k, q, cp_smem + SM::FACT + tid * 16);
    level_factors<1>(g, k, q, cp_smem + SM::FACT + 9 * SM::FROW + tid * 16);
    __syncthreads();
    level_sums(8 >> (warp >> 1));
    __syncthreads();
    level_factors<2>(g, k, q, cp_smem + SM::FACT + tid * 16);
    level_factors<3>(g, k, q, cp_smem + SM::FACT + 9 * SM::FROW + tid * 16);
    __syncthreads();
    level_sums(2 >> (warp >> 1));
    __syncthreads();
    unsigned char* wp = ws + (int64_t)blockIdx.x * CW_BYTES;
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
        uint32_t w[3][CD_L / 2];
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
            split3(v, w[0][i], w[1][i], w[2][i]);
            *reinterpret_cast<uint64_t*>(cp_smem + SM::PQ + tid * (SM::PQ_STRIDE * 4) + i * 8) = cd_mul2(upto[i], q[i]);
        }
        clean = cd_sum(zero) == 0.f;
        *reinterpret_cast<float*>(wp + CW_P + tid * 4) = p;
        auto rows = [&](unsigned char* to) {
#pragma unroll
            for (int m = 0; m < 3; ++m)
#pragma unroll
                for (int i = 0; i < 2; ++i)
                    *reinterpret_cast<uint4*>(to + m * CW_ROWS + row_swz(tid, i)) = make_uint4(w[m][4 * i], w[m][4 * i + 1], w[m][4 * i + 2], w[m][4 * i + 3]);
        };
        rows(cp_smem + SM::PK);
        p = 1.f;
#pragma unroll
        for (int i = CD_L / 2 - 1; i >= 0; --i) {           // tokens 2 i and 2 i + 1 side by side: place 4 i, or 4 (i - 4) + 2
            const float2 f = cd_two(g[i]);
            const float a = p * f.y;
            const int at = i < 4 ? 2 * i : 2 * (i - 4) + 1;
            split3(cd_mul2(cd_pack(a, p), k[i]), w[0][at], w[1][at], w[2][at]);
            p = a * f.x;
        }
        rows(wp + CW_R);
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
            const uint32_t row = mat_row(t, j), to = mat_row(place, j);
            uint32_t b[3];
            split3(v, b[0], b[1], b[2]);
#pragma unroll
            for (int m = 0; m < 3; ++m) {
                *reinterpret_cast<uint32_t*>(wp + (w ? CW_BT : CW_T) + m * CW_MAT + to) = b[m];
                *reinterpret_cast<uint32_t*>(cp_smem + SM::MAT + (3 * w + m) * CW_MAT + row) = w ? b[m] ^ 0x80008000u : b[m];       // -B T
            }
        }
        if (!clean) {
            *reinterpret_cast<uint64_t*>(cp_smem + SM::RAW_K + (t * CD_L + j) * 4) = tv;         // for the rows one by one, below
            *reinterpret_cast<uint64_t*>(cp_smem + SM::RAW_Q + (t * CD_L + j) * 4) = bt;
        }
    }
    __syncthreads();
    // W^T = (P k)^T T^T and Q^T = (P q)^T - (P k)^T (B T)^T, [32 channels of this warp] x [16 tokens]
    uint32_t tb[2][2][3][2];                                // [T, -B T][tile of eight tokens][term]
#pragma unroll
    for (int i = 0; i < 6; ++i)
        wm_ldsm(sbase + SM::MAT + i * CW_MAT + row_swz(br, bp), tb[i / 3][0][i % 3][0], tb[i / 3][0][i % 3][1], tb[i / 3][1][i % 3][0], tb[i / 3][1][i % 3][1]);
#pragma unroll
    for (int m = 0; m < 2; ++m) {
        const int c0 = warp * 32 + m * 16;
        uint32_t a[3][4];
#pragma unroll
        for (int i = 0; i < 3; ++i) wm_ldsm(sbase + SM::PK + i * CW_ROWS + row_swz(c0 + ar, lane >> 4), a[i][0], a[i][1], a[i][2], a[i][3]);
        float W[2][4], Q[2][4];                             // channels gq, gq + 8; tokens 8 i + 2 t4, + 1
        const float* pq = reinterpret_cast<const float*>(cp_smem + SM::PQ) + (c0 + gq) * SM::PQ_STRIDE + 2 * t4;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
#pragma unroll
            for (int e = 0; e < 4; ++e) Q[i][e] = pq[(e >> 1) * 8 * SM::PQ_STRIDE + 8 * i + (e & 1)];
            float P[4], R[4];                               // the large products and the small ones apart, added here
            mma_bf_new(P, a[0], tb[0][i][0][0], tb[0][i][0][1]);
            mma_rest(W[i], a, tb[0][i], true);
            add4(W[i], P);
            mma_bf_new(P, a[0], tb[1][i][0][0], tb[1][i][0][1]);
            mma_rest(R, a, tb[1][i], true);
            add4(P, R);
            add4(Q[i], P);
        }
        if (!clean) {
            // a key or a decay that is no number: a token's row takes the tokens up to its own alone (its products with the zeros above would not)
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int t = 8 * i + 2 * t4 + (e & 1), ch = c0 + gq + 8 * (e >> 1);
                    float w = 0.f, v = reinterpret_cast<const float*>(cp_smem + SM::PQ)[ch * SM::PQ_STRIDE + t];
#pragma unroll 1
                    for (int j = 0; j <= t; ++j) {
                        const unsigned char* at = cp_smem + SM::PK + row_swz(ch, j >> 3) + (j & 7) * 2;
                        const __nv_bfloat16* term = reinterpret_cast<const __nv_bfloat16*>(at);
                        const float f = __bfloat162float(term[0]) + (__bfloat162float(term[CW_ROWS / 2]) + __bfloat162float(term[CW_ROWS]));
                        w = fmaf(reinterpret_cast<const float*>(cp_smem + SM::RAW_K)[t * CD_L + j], f, w);
                        v = fmaf(-reinterpret_cast<const float*>(cp_smem + SM::RAW_Q)[t * CD_L + j], f, v);
                    }
                    W[i][e] = w, Q[i][e] = v;
                }
        }
#pragma unroll
        for (int r = 0; r < 2; ++r) {                       // tokens 2 t4, + 1, 8 + 2 t4, + 1 side by side: the order of the workspace
            unsigned char* d = wp + row_swz(c0 + gq + 8 * r, t4 >> 1) + (t4 & 1) * 8;
#pragma unroll
            for (int w = 0; w < 2; ++w) {
                const float(&v)[2][4] = w ? Q : W;
                uint2 o[3];
                split3(cd_pack(v[0][2 * r], v[0][2 * r + 1]), o[0].x, o[1].x, o[2].x);
                split3(cd_pack(v[1][2 * r], v[1][2 * r + 1]), o[0].y, o[1].y, o[2].y);
#pragma unroll
                for (int i = 0; i < 3; ++i) *reinterpret_cast<uint2*>(d + (w ? CW_Q : CW_W) + i * CW_ROWS) = o[i];
            }
        }
    }
}

// ---- second kernel: the walk over the chunks --------------------------------------------------------------------------------------------
struct CdSmem {                                             // stages of (a chunk's workspace, its V), the halves' partial sums of two chunks
    static constexpr int V = CW_BYTES, STAGE = V + CD_L * CD_VC * 2, XCH = CD_STAGES * STAGE, HALF = 32 * 12, BYTES = XCH + 2 * 8 * HALF * 4;
};
// Named barriers: a chunk is there (per pair of consumer warps and parity, so that pairs drift apart and fill each other's waits), a chunk of a parity
// is done with, the two halves of a pair of consumers
constexpr int CD_FULL = 0, CD_EMPTY = 8, CD_HALVES = 10;
template <int COUNT>
__device__ __forceinline__ void cd_sync(int id) { asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(COUNT) : "memory"); }
template <int COUNT>
__device__ __forceinline__ void cd_arrive(int id) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "n"(COUNT) : "memory"); }

// Eight consumer warps: warp 2 p + hf holds 16 value columns (p) and 64 of the channels (hf), so that two warps per scheduler hide each other's waits;
// a pair adds its two halves of W S and of Q S through shared memory.  Two copying warps, two chunks ahead.  Bound by the consumers' chain per chunk and
// the tensor pipe (63 % busy): 2.2 us of 156 products (fp16 pairs: 84 products, 1.67 us, of one warp per 16 columns and all channels 4.0).
constexpr int CD_THREADS = 320;
__global__ void __launch_bounds__(CD_THREADS, 1) channel_delta_chunks_kernel(
    const __nv_bfloat16* __restrict__ x, int64_t stride, int v_off, const unsigned char* __restrict__ ws, float* __restrict__ state,
    const int32_t* __restrict__ state_slots, const int32_t* __restrict__ cu_q, const int32_t* __restrict__ cu_k, float* __restrict__ out, int H, int dim,
    int vdim, float q_scale, int first_row, int rows_here) {
    B200_PDL_SYNC();
    using SM = CdSmem;
    extern __shared__ __align__(128) unsigned char cd_smem[];
    const int h = blockIdx.x, s = blockIdx.y, col0 = blockIdx.z * CD_VC, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const SeqSpan sp = seq_span(cu_q, cu_k, nullptr, s);
    const int row = chunk_row(sp.q0, s), first = max(0, first_row - row);   // first of this launch's chunks
    const int nch = min((sp.qlen + CD_L - 1) / CD_L, first_row + rows_here - row) - first;
    if (nch <= 0) return;
    const uint32_t sbase = smem_u32(cd_smem);
    const int row0 = sp.q0 + first * CD_L, rows = sp.qlen - first * CD_L;   // its tokens (and the later launches')
    if (warp >= 8) {
        const int pt = threadIdx.x & 63;
        const unsigned char* wp = ws + ((int64_t)(row + first - first_row) * H + h) * CW_BYTES + pt * 16;
        const __nv_bfloat16* vp = x + (int64_t)row0 * stride + v_off + (int64_t)h * vdim + col0 + (pt & 7) * 8;
        const bool v_in = col0 + (pt & 7) * 8 < vdim;
        auto fetch = [&](int c) {
            if (c < nch) {
                const uint32_t d = sbase + (c & (CD_STAGES - 1)) * SM::STAGE;
                const unsigned char* wc = wp + (int64_t)c * H * CW_BYTES;
                static_assert(CW_BYTES % 1024 == 512, "whole rounds of 64 pieces and half a one");
#pragma unroll 13
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
    float* sums = reinterpret_cast<float*>(cd_smem + SM::XCH) + lane;
    uint64_t S[NT][2];                                      // rows gq, gq + 8 of the pair's 16 value columns, channels ch0 + n * 8 + 2 t4, + 1
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
            float2 f = make_float2(0.f, 0.f);
            if (has_hist && vrow + 8 * hh < vdim && ch0 + n * 8 < dim) f = *reinterpret_cast<const float2*>(stp + (int64_t)(vrow + 8 * hh) * dim + n * 8 + 2 * t4);
            S[n][hh] = cd_pack(f.x, f.y);
        }
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
        float* mine = sums + ((c & 1) * 8 + warp) * SM::HALF;
        const float* other = sums + ((c & 1) * 8 + (warp ^ 1)) * SM::HALF;
        uint32_t a[KT][3][4];                               // S in three terms, the left operand of W S and Q S
#pragma unroll
        for (int kk = 0; kk < KT; ++kk)
#pragma unroll
            for (int i = 0; i < 4; ++i) split3(S[2 * kk + i / 2][i & 1], a[kk][0][i], a[kk][1][i], a[kk][2][i]);
        cd_sync<128>(CD_FULL + 2 * vw + (c & 1));
        if (live) {
            // this half's part of rows [16 tokens] x S: the large products each from zero and added here, the small ones apart
            auto rows_times_state = [&](int at, float (&R)[2][4]) {
                float X[2][4];
#pragma unroll
                for (int kk = 0; kk < KT; ++kk) {
                    uint32_t b[2][3][2];                    // [tile of eight tokens][term]
#pragma unroll
                    for (int m = 0; m < 3; ++m)
                        wm_ldsm_t(sb + at + m * CW_ROWS + row_swz(ch0 + kk * 16 + kr, lane >> 4), b[0][m][0], b[0][m][1], b[1][m][0], b[1][m][1]);
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        float P[4];
                        mma_bf_new(kk ? P : R[i], a[kk][0], b[i][0][0], b[i][0][1]);
                        mma_rest(X[i], a[kk], b[i], kk == 0);
                        if (kk) add4(R[i], P);
                    }
                }
#pragma unroll
                for (int i = 0; i < 2; ++i) add4(R[i], X[i]);
            };
            uint32_t va[4];
            wm_ldsm_t(sb + SM::V + val_swz(br, vw * 2 + bp), va[0], va[1], va[2], va[3]);
            float U[2][4], O[2][4], Y[2][4];
            rows_times_state(CW_W, U);
            // T V by the first half of the channels, (B T) V by both (a tile of eight tokens each is used): small terms first
            auto times_values = [&](int mat, float (&D)[2][4]) {
                uint32_t b[4];
#pragma unroll
                for (int m = 2; m >= 0; --m) {
                    float P[2][4] = {};
                    wm_ldsm(sb + mat + m * CW_MAT + row_swz(br, bp), b[0], b[1], b[2], b[3]);
#pragma unroll
                    for (int i = 0; i < 2; ++i) wm_mma(P[i], va[0], va[1], va[2], va[3], b[2 * i], b[2 * i + 1]);
#pragma unroll
                    for (int i = 0; i < 2; ++i)
                        if (m < 2) add4(D[i], P[i]);
                        else D[i][0] = P[i][0], D[i][1] = P[i][1], D[i][2] = P[i][2], D[i][3] = P[i][3];
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
                    for (int e = 0; e < 4; ++e) mine[(4 * i + e) * 32] = U[i][e] = Y[i][e] - U[i][e];
            } else {
#pragma unroll
                for (int i = 0; i < 2; ++i)
#pragma unroll
                    for (int e = 0; e < 4; ++e) mine[(4 * i + e) * 32] = U[i][e] = -U[i][e];
            }
            // the half's tile of the output: its own sums and the other half's
            rows_times_state(CW_Q, O);
            times_values(CW_BT, Y);
            if (!whole) triangle(sm + CW_BT, va, Y);
#pragma unroll
            for (int e = 0; e < 4; ++e) mine[(8 + e) * 32] = hf ? O[0][e] : O[1][e];
            cd_sync<64>(CD_HALVES + vw);                    // (the chunk after the next writes here again: both have read by then)
            uint32_t x[3][4];
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int e = 0; e < 4; e += 2) {
                    const uint64_t u = cd_add2(cd_pack(U[i][e], U[i][e + 1]), cd_pack(other[(4 * i + e) * 32], other[(4 * i + e + 1) * 32]));
                    split3(u, x[0][2 * i + e / 2], x[1][2 * i + e / 2], x[2][2 * i + e / 2]);
                }
            // S^T <- P_16 S^T + U^T (R k), channels n * 8 .. + 15 at a time
#pragma unroll
            for (int n = 0; n < NT; n += 2) {
                uint32_t b[2][3][2];
                float D[2][4];
#pragma unroll
                for (int m = 0; m < 3; ++m)
                    wm_ldsm(sb + CW_R + m * CW_ROWS + row_swz(ch0 + n * 8 + br, bp), b[0][m][0], b[0][m][1], b[1][m][0], b[1][m][1]);
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    float P[4];
                    mma_bf_new(P, x[0], b[i][0][0], b[i][0][1]);
                    mma_rest(D[i], x, b[i], true);
                    const uint64_t g = *reinterpret_cast<const uint64_t*>(sm + CW_P + (ch0 + (n + i) * 8 + 2 * t4) * 4);
                    S[n + i][0] = cd_add2(cd_fma2(g, S[n + i][0], cd_pack(D[i][0], D[i][1])), cd_pack(P[0], P[1]));
                    S[n + i][1] = cd_add2(cd_fma2(g, S[n + i][1], cd_pack(D[i][2], D[i][3])), cd_pack(P[2], P[3]));
                }
            }
            const int t = c * CD_L + token_at(hf * 8 + 2 * t4);             // the lane's places 2 t4 and 2 t4 + 1 of the tile are neighbours
            float* op = out + ((int64_t)(row0 + t) * H + h) * vdim + vrow;
#pragma unroll
            for (int e = 0; e < 4; ++e) {                   // token t + (e & 1), column gq or gq + 8
                const float o = ((hf ? O[1][e] : O[0][e]) + other[(8 + e) * 32] + (hf ? Y[1][e] : Y[0][e])) * q_scale;
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

}  // namespace

extern "C" size_t b200m_channel_delta_workspace_bytes(int n, int num_seqs, int num_heads) {
    if (n < 0 || num_seqs < 0 || num_heads <= 0) return 0;
    return ((size_t)(n / CD_L) + (size_t)num_seqs) * (size_t)num_heads * CW_BYTES;
}

extern "C" int b200m_channel_delta_prompts(const void* x, int64_t stride, int q_off, int k_off, int v_off, const void* write_in, int64_t write_stride,
                                           const float* decay_in, int64_t decay_stride, const float* rate, const float* decay_bias, float decay_sign,
                                           float* state, const int32_t* state_slots, const int32_t* cu_q, const int32_t* cu_k, float* out, int n,
                                           int num_seqs, int num_heads, int num_kv_heads, int dim, int vdim, float q_scale, void* workspace,
                                           size_t workspace_bytes, void* stream) {
    if (!x || !write_in || !decay_in || !state || !state_slots || !out || !rate || !decay_bias || !cu_q || !cu_k) return B200_EINVAL;
    if (num_heads <= 0 || num_kv_heads <= 0 || num_heads % num_kv_heads || dim <= 0 || vdim <= 0) return B200_EINVAL;
    if (decay_stride < (int64_t)num_heads * dim || n < 0) return B200_EINVAL;
    if (dim > CD_D || dim % 8 || vdim % 8 || stride % 8 || q_off % 8 || k_off % 8 || v_off % 8 || decay_stride % 4) return B200_EUNSUPPORTED;
    for (const void* p : {x, static_cast<const void*>(decay_in), static_cast<const void*>(decay_bias), static_cast<const void*>(state),
                          static_cast<const void*>(workspace)})
        if (reinterpret_cast<uintptr_t>(p) % 16) return B200_EUNSUPPORTED;
    if (num_seqs <= 0 || n == 0) return B200_OK;
    if (num_seqs > 65535 || decay_stride > (1 << 27) || (vdim + CD_VC - 1) / CD_VC > 65535) return B200_EUNSUPPORTED;
    const int64_t all = (int64_t)(n / CD_L) + num_seqs, fit = (int64_t)(workspace_bytes / ((size_t)num_heads * CW_BYTES));
    const int rows = (int)(all < fit ? all : fit);                                          // of a launch pair
    if (!workspace || rows <= 0) return B200_EINVAL;
    if ((int64_t)num_heads * rows > 0x7fffffff || all > 0x7fffffff - rows) return B200_EUNSUPPORTED;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const __nv_bfloat16* xb = static_cast<const __nv_bfloat16*>(x);
    unsigned char* ws = static_cast<unsigned char*>(workspace);
    static B200SmemOptIn opt, opt_prepare;
    if (opt.ensure(channel_delta_chunks_kernel, CdSmem::BYTES) != cudaSuccess) return B200_ECUDA;
    if (opt_prepare.ensure(channel_delta_prepare_kernel, CpSmem::BYTES) != cudaSuccess) return B200_ECUDA;
    for (int first = 0; first < all; first += rows) {
        const int here = (int)(all - first < rows ? all - first : rows);
        B200_LAUNCH((channel_delta_prepare_kernel), (unsigned)(num_heads * here), CP_THREADS, CpSmem::BYTES, st, xb, stride, q_off,
                    k_off, static_cast<const __nv_bfloat16*>(write_in), write_stride, decay_in, decay_stride, rate, decay_bias, decay_sign, cu_q, ws,
                    num_seqs, num_heads, num_kv_heads, dim, first);
        if (const int rc = b200_launch_status(nullptr); rc != B200_OK) return rc;
        B200_LAUNCH((channel_delta_chunks_kernel), dim3(num_heads, num_seqs, (vdim + CD_VC - 1) / CD_VC), CD_THREADS, CdSmem::BYTES, st, xb, stride, v_off,
                    static_cast<const unsigned char*>(ws), state, state_slots, cu_q, cu_k, out, num_heads, dim, vdim, q_scale, first, here);
        if (const int rc = b200_launch_status(nullptr); rc != B200_OK) return rc;
    }
    return B200_OK;
}
