// The operator for a handful of tokens: decoding with a carried state, sequences of a few tokens.
//
// What bounds it: the fp32 state, 16 KB in and 16 KB out per (sequence, head) at K = 64, against 640 bytes of token data;
// at one token the call is a copy of the state with a rank-one update on the way.  So no chunk, no tensor core and no
// tile: one CTA per (sequence, head), the state in registers from its first load to its last store, the token recurrence
//     S = exp(g_t) (.) S + k_t v_t^T ,   o_t = scale q_t^T S
// in fp32.  Warp w owns value columns 8 w .. 8 w + 7 of all key rows -- two lanes share the 32-byte sector of a row, so that
// every load and store moves whole sectors, and no warp waits for another -- and completes the read-out's sum over the
// rows with a 5-shuffle butterfly.
// Measured at B32 H12 K64, one token, state in and out: 5.7 us a call in a graph of 24 calls whose states no cache holds (12.6 MB each:
// 1.9 us at the copy rate), against 20.4 us of kernel for a chunk of which 63 rows are padding.
#pragma once

#include "gla_device.cuh"

namespace gla {

constexpr int kStepThreads = 256;
// Token by token costs about 0.3 us per token; a one-chunk sequence costs the chunk kernel 12 us alone on its SM and more
// when SMs take several.  Measured (us, this kernel / chunk kernel): 96 heads 10.8 / 12.3 at 24 tokens, 14.4 / 12.3 at 32;
// 384 heads 16.5 / 23.5 and 20.5 / 22.6; 1152 heads 36.9 / 51.3 and 45.5 / 49.2.
constexpr int kStepMaxTokens = 24;
constexpr int kStepBlock = 16;

struct StepParams {
    const __half *q, *k, *v, *g;
    __half* o;
    const float* s0;
    float* sT;
    uint32_t* ctrl;               // status words of the workspace: this path has no wait that could expire
    long long q_s[3], k_s[3], v_s[3], g_s[3], o_s[3];      // element strides (batch, token, head)
    int T, H, Hc, Wc, rev;        // scan order as in Params
    float scale, inv_norm;
};

template <int K>
__global__ void __launch_bounds__(kStepThreads) gla_step_kernel(const __grid_constant__ StepParams P) {
    constexpr int R = K / 16;                              // rows per lane: (lane >> 1) + 16 i
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    const int b = blockIdx.x / P.H, h = blockIdx.x - b * P.H;
    const int row0 = l >> 1, col = 8 * w + 4 * (l & 1);
    pdl_release();
    pdl_wait();
    if (blockIdx.x == 0 && threadIdx.x < 4) P.ctrl[threadIdx.x] = 0u;

    const size_t soff = static_cast<size_t>(blockIdx.x) * K * 64 + static_cast<size_t>(row0) * 64 + col;
    float4 S[R];
#pragma unroll
    for (int i = 0; i < R; ++i)
        S[i] = P.s0 != nullptr ? *reinterpret_cast<const float4*>(P.s0 + soff + i * 1024) : make_float4(0.f, 0.f, 0.f, 0.f);

    // Token data goes through shared memory kStepBlock tokens at a time, as fp32 factors: with the loads one token ahead of
    // their use instead, a token cost an L2 round trip (680 cycles).
    __shared__ __align__(16) float sq[kStepBlock][K], sk[kStepBlock][K], sa[kStepBlock][K], sv[kStepBlock][64];
    const __half* src[4] = {P.q + b * P.q_s[0] + h * P.q_s[2], P.k + b * P.k_s[0] + h * P.k_s[2],
                            P.g + b * P.g_s[0] + h * P.g_s[2], P.v + b * P.v_s[0] + h * P.v_s[2]};
    __half* o = P.o + b * P.o_s[0] + h * P.o_s[2];
    auto token = [&](int p) -> long long {
        const int u = P.rev ? P.T - 1 - p : p;
        if (P.Wc == 1) return u;
        const int c = u / P.Hc;
        return static_cast<long long>(u - c * P.Hc) * P.Wc + c;
    };
    auto stage = [&](int p0, int n) {                       // 16-byte vectors: K/8 of q, k, g and 8 of v per token
        constexpr int kVec = K / 8, kPer = 3 * kVec + 8;
        for (int e = threadIdx.x; e < n * kPer; e += kStepThreads) {
            const int p = e / kPer, i = e - p * kPer;
            const long long t = token(p0 + p);
            const int which = i < kVec ? 0 : i < 2 * kVec ? 1 : i < 3 * kVec ? 2 : 3;
            const int c8 = 8 * (i - which * kVec);
            const long long st = which == 0 ? P.q_s[1] : which == 1 ? P.k_s[1] : which == 2 ? P.g_s[1] : P.v_s[1];
            const __half* from = which == 0 ? src[0] : which == 1 ? src[1] : which == 2 ? src[2] : src[3];
            const uint4 r = *reinterpret_cast<const uint4*>(from + t * st + c8);
            const uint32_t u[4] = {r.x, r.y, r.z, r.w};
            float f[8];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float2 x = unpack_half2(u[j]);
                f[2 * j] = x.x; f[2 * j + 1] = x.y;
            }
            if (which == 2) {
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    if (P.inv_norm > 0.f) f[j] = __half2float(__float2half_rn(logsigmoid_f(f[j]) * P.inv_norm));  // fp16 log gates, as in the chunk kernel
                    f[j] = ex2(f[j] * 1.4426950408889634f);
                }
            }
            float* to = which == 0 ? &sq[p][c8] : which == 1 ? &sk[p][c8] : which == 2 ? &sa[p][c8] : &sv[p][c8];
            reinterpret_cast<float4*>(to)[0] = make_float4(f[0], f[1], f[2], f[3]);
            reinterpret_cast<float4*>(to)[1] = make_float4(f[4], f[5], f[6], f[7]);
        }
    };
    auto one_token = [&](int p, int pb) {
        float qf[R], kf[R], a[R];
#pragma unroll
        for (int i = 0; i < R; ++i) {
            qf[i] = sq[pb][row0 + 16 * i];
            kf[i] = sk[pb][row0 + 16 * i];
            a[i] = sa[pb][row0 + 16 * i];
        }
        const float4 vf = *reinterpret_cast<const float4*>(&sv[pb][col]);
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int i = 0; i < R; ++i) {
            S[i].x = fmaf(a[i], S[i].x, kf[i] * vf.x);
            S[i].y = fmaf(a[i], S[i].y, kf[i] * vf.y);
            S[i].z = fmaf(a[i], S[i].z, kf[i] * vf.z);
            S[i].w = fmaf(a[i], S[i].w, kf[i] * vf.w);
            acc.x = fmaf(qf[i], S[i].x, acc.x);
            acc.y = fmaf(qf[i], S[i].y, acc.y);
            acc.z = fmaf(qf[i], S[i].z, acc.z);
            acc.w = fmaf(qf[i], S[i].w, acc.w);
        }
        // sum over the 16 lanes of one column group (lane bits 1..4), halving the values kept at the first two exchanges
        const bool b4 = (l & 16) != 0, b3 = (l & 8) != 0;
        float x = b4 ? acc.z : acc.x, y = b4 ? acc.w : acc.y;
        x += __shfl_xor_sync(0xffffffffu, b4 ? acc.x : acc.z, 16);
        y += __shfl_xor_sync(0xffffffffu, b4 ? acc.y : acc.w, 16);
        float s = b3 ? y : x;
        s += __shfl_xor_sync(0xffffffffu, b3 ? x : y, 8);
        s += __shfl_xor_sync(0xffffffffu, s, 4);
        s += __shfl_xor_sync(0xffffffffu, s, 2);
        if ((l & 6) == 0) o[token(p) * P.o_s[1] + col + (b4 ? 2 : 0) + (b3 ? 1 : 0)] = __float2half_rn(s * P.scale);
    };
    for (int p0 = 0; p0 < P.T; p0 += kStepBlock) {
        const int n = min(kStepBlock, P.T - p0);
        if (p0 > 0) __syncthreads();
        stage(p0, n);
        __syncthreads();
        // four tokens at a time: their read-out sums do not depend on one another, only the state does
        int pb = 0;
        for (; pb + 4 <= n; pb += 4) {
#pragma unroll
            for (int j = 0; j < 4; ++j) one_token(p0 + pb + j, pb + j);
        }
        for (; pb < n; ++pb) one_token(p0 + pb, pb);
    }
    if (P.sT != nullptr) {
#pragma unroll
        for (int i = 0; i < R; ++i) *reinterpret_cast<float4*>(P.sT + soff + i * 1024) = S[i];
    }
}

}  // namespace gla
