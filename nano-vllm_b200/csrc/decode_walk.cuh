// Single-token attention of one (sequence, kv head) by the warps of a CTA, as the kernels for steps of a few rows do it (decode_small.cu, step_rows.cu).
//
// A warp takes chunks of 16 tokens straight from global memory into registers (16 loads of 16 bytes per lane), half a warp per token, 16 lanes x 8 dims,
// fp32 on the FMA pipe; the warps meet in shared memory.  The order of every sum is fixed here, so that both kernels give the same bits.
#pragma once
#include "decode_common.cuh"

namespace b200dec {

constexpr int SW = 8;                              // warps that share a context

struct WalkLane {
    int lane, hw, j;                               // half of the warp (even or odd tokens), dim slice
    __device__ __forceinline__ explicit WalkLane(int l) : lane(l), hw(l >> 4), j(l & 15) {}
};

// Keys or values of a chunk of `valid` tokens whose first cache row is `row`; rows past the context: zeros, nothing is read.
__device__ __forceinline__ void walk_load(const WalkLane& w, const __nv_bfloat16* layer, int64_t row, int valid, uint4 (&x)[8]) {
    const uint4* s = reinterpret_cast<const uint4*>(layer + row * B200_HEAD_DIM) + w.j;
#pragma unroll
    for (int it = 0; it < 8; ++it) {
        const int t = 2 * it + w.hw;
        x[it] = t < valid ? s[t * (B200_HEAD_DIM / 8)] : make_uint4(0, 0, 0, 0);
    }
}

// RMS norm -> bf16 -> NeoX rotation -> bf16, as qknorm_rope_store_kernel
__device__ __forceinline__ void walk_norm_rope(const WalkLane& wl, float (&x)[8], const float (&w)[8], const float (&cosr)[8], const float (&sinr)[8], float eps) {
    float ss = 0.f;
#pragma unroll
    for (int e = 0; e < 8; ++e) ss = fmaf(x[e], x[e], ss);
#pragma unroll
    for (int o2 = 8; o2 > 0; o2 >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o2);
    const float rstd = 1.0f / sqrtf(ss / (float)B200_HEAD_DIM + eps);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        const float y = round_bf16(__fmul_rn(__fmul_rn(x[e], rstd), w[e]));
        const float other = __shfl_xor_sync(0xffffffffu, y, 8);              // element d +- 64
        const float r = (wl.j < 8) ? __fsub_rn(__fmul_rn(y, cosr[e]), __fmul_rn(other, sinr[e]))
                                   : __fadd_rn(__fmul_rn(y, cosr[e]), __fmul_rn(other, sinr[e]));
        x[e] = round_bf16(r);
    }
}

// What a warp has of GW heads: queries (scaled), running maximum, sum and unnormalised result.
template <int GW>
struct WalkState {
    float q[GW][8], o[GW][8], m[GW], l[GW];

    __device__ __forceinline__ void begin(float scale_log2) {
#pragma unroll
        for (int g = 0; g < GW; ++g) {
            m[g] = -INFINITY;
            l[g] = 0.f;
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                q[g][e] *= scale_log2;
                o[g][e] = 0.f;
            }
        }
    }

    // One chunk; `left`: tokens of the context from this chunk's first on (at least 1).
    __device__ __forceinline__ void chunk(const WalkLane& w, const uint4 (&kr)[8], const uint4 (&vr)[8], int left) {
        float acc[GW][8];
        scores(kr, acc);
        values(w, acc, vr, left);
    }
    // ... and its two halves: this lane's dim slice of every token's scores; the softmax and the weighted values
    __device__ __forceinline__ void scores(const uint4 (&kr)[8], float (&acc)[GW][8]) const {
#pragma unroll
        for (int it = 0; it < 8; ++it) {
            float kf[8];
            unpack8(kr[it], kf);
#pragma unroll
            for (int g = 0; g < GW; ++g) {
                float a = q[g][0] * kf[0];
#pragma unroll
                for (int e = 1; e < 8; ++e) a = fmaf(q[g][e], kf[e], a);
                acc[g][it] = a;
            }
        }
    }
    __device__ __forceinline__ void values(const WalkLane& w, float (&acc)[GW][8], const uint4 (&vr)[8], int left) {
        const int j = w.j;
        // the score of token 2 * my_it + hw ends up in this lane (and its neighbour j ^ 1)
        const int my_it = ((j >> 3) & 1) * 4 + ((j >> 2) & 1) * 2 + ((j >> 1) & 1);
        const bool ok = 2 * my_it + w.hw < left;
        float pv[GW];
#pragma unroll
        for (int g = 0; g < GW; ++g) {             // sum over the 16 dim slices, scattering tokens over lanes: 8 -> 4 -> 2 -> 1 values
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                const float send = (j & 8) ? acc[g][x] : acc[g][x + 4], keep = (j & 8) ? acc[g][x + 4] : acc[g][x];
                acc[g][x] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
            }
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                const float send = (j & 4) ? acc[g][x] : acc[g][x + 2], keep = (j & 4) ? acc[g][x + 2] : acc[g][x];
                acc[g][x] = keep + __shfl_xor_sync(0xffffffffu, send, 4);
            }
            const float send = (j & 2) ? acc[g][0] : acc[g][1], keep = (j & 2) ? acc[g][1] : acc[g][0];
            float s = keep + __shfl_xor_sync(0xffffffffu, send, 2);
            s += __shfl_xor_sync(0xffffffffu, s, 1);
            s = ok ? s : -INFINITY;
            const float m_new = fmaxf(m[g], warp_max(s));                    // a chunk holds at least one token
            const float alpha = fast_exp2(m[g] - m_new);
            pv[g] = fast_exp2(s - m_new);
            m[g] = m_new;
            l[g] = l[g] * alpha + ((j & 1) ? 0.f : pv[g]);
#pragma unroll
            for (int e = 0; e < 8; ++e) o[g][e] *= alpha;
        }
        // token 2 it + hw sits in lanes whose bits (8, 4, 2) spell it: fetch each weight from there
#pragma unroll
        for (int it = 0; it < 8; ++it) {
            float vf[8];
            unpack8(vr[it], vf);
#pragma unroll
            for (int g = 0; g < GW; ++g) {
                const float p = __shfl_sync(0xffffffffu, pv[g], (w.lane & 16) | ((it & 4) << 1) | ((it & 2) << 1) | ((it & 1) << 1));
#pragma unroll
                for (int e = 0; e < 8; ++e) o[g][e] = fmaf(p, vf[e], o[g][e]);
            }
        }
    }

    // The step's own token, which is not in the cache yet (one warp of the context's).
    __device__ __forceinline__ void own(const WalkLane& w, const float (&kn)[8], const float (&vn)[8]) {
#pragma unroll
        for (int g = 0; g < GW; ++g) {
            float s = q[g][0] * kn[0];
#pragma unroll
            for (int e = 1; e < 8; ++e) s = fmaf(q[g][e], kn[e], s);
#pragma unroll
            for (int o2 = 8; o2 > 0; o2 >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o2);
            const float m_new = fmaxf(m[g], s), alpha = fast_exp2(m[g] - m_new), pn = fast_exp2(s - m_new);
            m[g] = m_new;
            l[g] = l[g] * alpha + (w.lane == 0 ? pn : 0.f);
            const float p = w.hw == 0 ? pn : 0.f;  // the halves' results are summed below
#pragma unroll
            for (int e = 0; e < 8; ++e) o[g][e] = fmaf(p, vn[e], o[g][e] * alpha);
        }
    }

    // This warp's part into shared memory, where the warps of the CTA meet.
    __device__ __forceinline__ void leave(const WalkLane& w, float (&sh_o)[GW][B200_HEAD_DIM], float (&sh_ml)[GW][2]) {
#pragma unroll
        for (int g = 0; g < GW; ++g) {
            l[g] = warp_sum(l[g]);
#pragma unroll
            for (int e = 0; e < 8; ++e) o[g][e] += __shfl_xor_sync(0xffffffffu, o[g][e], 16);
            if (w.hw == 0) {
                *reinterpret_cast<float4*>(&sh_o[g][w.j * 8]) = make_float4(o[g][0], o[g][1], o[g][2], o[g][3]);
                *reinterpret_cast<float4*>(&sh_o[g][w.j * 8 + 4]) = make_float4(o[g][4], o[g][5], o[g][6], o[g][7]);
            }
            if (w.lane == 0) {
                sh_ml[g][0] = m[g];
                sh_ml[g][1] = l[g];
            }
        }
    }
};

// Column d of head g over the warps' parts: maximum, sum, unnormalised result.
template <int GW>
__device__ __forceinline__ void walk_meet(const float (&sh_o)[SW][GW][B200_HEAD_DIM], const float (&sh_ml)[SW][GW][2], int g, int d, float& M, float& L, float& a) {
    M = -INFINITY;
    L = 0.f;
    a = 0.f;
#pragma unroll
    for (int w = 0; w < SW; ++w) M = fmaxf(M, sh_ml[w][g][0]);
#pragma unroll
    for (int w = 0; w < SW; ++w) {
        const float f = sh_ml[w][g][0] == -INFINITY ? 0.f : fast_exp2(sh_ml[w][g][0] - M);
        L = fmaf(f, sh_ml[w][g][1], L);
        a = fmaf(f, sh_o[w][g][d], a);
    }
}

}  // namespace b200dec
