// Gradient of the gated-linear-attention operator, chunk by chunk on the tensor cores.
//
//   forward    S_t = exp(g_t) S_{t-1} + k_t v_t^T ,  o_t = scale q_t^T S_t
//   gradient   dS_t = exp(g_{t+1}) dS_{t+1} + scale q_t do_t^T
//              dq_t = scale S_t do_t     dk_t = dS_t v_t     dv_t = dS_t^T k_t
//              dg_t = sum_{s >= t} (q_s dq_s - k_s dk_s)   (+ the final state's term at the last token)
//
// The reference trains through the third-party FLA operator (engine/gtr/backbone/vit_adapter.py:441,560-568); its
// own CUDA extension has no gradient.
//
// With G the inclusive gate sum inside a 64-token chunk, G_L its last value, R = G_L / 2 per channel, S the state at the
// chunk's start and dS the state gradient at its end:
//   qt = q e^(G-R)    kt = k e^(R-G)    St = e^R S    dSt = e^(G_L-R) dS    P = tril(qt kt^T)    dP = tril(do v^T)
//   dq = scale e^(G-R) (do St^T + dP kt)        dk = e^(R-G) (v dSt^T + scale dP^T qt)
//   dv = kt dSt + scale P^T do                  dS at the chunk's start = e^R (dSt + scale qt^T do)
//   dg_t = sum over the chunk's tokens s >= t of (q_s dq_s - k_s dk_s)  +  sum_v S_end dS   (S_end: state after the chunk)
// The last line closes the sum over all later tokens with two states at hand: no pass over the sequence is needed for dg.
//
// Precision.  The gradient is fp32 arithmetic on fp16 inputs, as a token recurrence in fp32 would be: every operand of the
// tensor cores that is not an input itself (qt, kt, P, dP, St, dSt) is the sum of two fp16 tiles, high and low part, and a
// product of two such operands is three MMAs (high high, high low, low high) into one fp32 accumulator: 22 bits.  Each
// operand carries a power-of-two scale of its own per chunk, taken from the largest magnitudes of the tiles at hand, that
// puts it where fp16 has both parts normal, so neither tiny nor huge gradients lose bits.  Measured against the float64
// recurrence: dg 1e-6 relative, the same as the token-by-token kernels these replace.
// A chunk in which some channel decays by more than 2^(2 kBwdRefLimit) has no common reference that keeps both operands in
// range; its products within the chunk are computed pair by pair in fp32 from gate differences, and the factors of what lies outside
// it from sums of gates that run one way each (bwd_wide_chunk).
//
// Measured (B200): B4 H12 T6400 K64 191 us (states 54, chunks 143) against 1080 us for three recurrent sweeps in fp32, whose
// bound was the FMA pipe (500 us); B8 H6 T1600 64 against 285.  HBM alone would take about 115 us at 6.5 TB/s (96 KB per
// chunk and head in the chunk kernel, 56 KB in the states'); what is left is the latency of the chunk's five dependent
// tensor-core round trips with two CTAs per SM.
//
// Two kernels.  gla_bwd_state_kernel walks the segments of every sequence and leaves the local state after every chunk
// (forward) and the local state gradient of a segment (backward); gla_bwd_chunk_kernel chains the segments' totals into its
// own start, then walks its segment backwards and emits everything.  Several CTAs share an SM and hide one another's
// tensor-core and memory latencies; the work of one chunk stays in one CTA.
#pragma once
#include <cuda_fp16.h>
#include <cstdint>

#include "gla_tiles.cuh"

namespace gla {

constexpr float kBwdFar = 1e30f;          // log2: stands for the decay by a gate of -inf, finite so that differences are too
constexpr float kBwdRefLimit = 8.f;       // log2: qt and kt carry factors up to 2^8, see bwd_scale() for the room they have

struct BwdParams {
    __half *dq, *dk, *dv;                 // contiguous [B,T,H,K|64], as q, k, v, g, do (which come through tensor maps)
    float* dg;            // [B,T,H,K] fp32, or null when dg_half is set
    __half* dg_half;
    const float* h0;      // [B,H,K,64] or null
    const float* dht;     // [B,H,K,64] or null
    float* dh0;           // [B,H,K,64] or null
    // States in scratch lie in the order of the threads that hold them: float4 e of thread t at [e][t].
    float* chunk_state;   // scratch [B*H][NT][4096]: forward state after a chunk, from a zero state at its segment's start
    float* chunk_decay;   // scratch [B*H][NT][64]: log2 decay from the segment's start to the chunk's end
    float* seg_grad;      // scratch [B*H][nseg][4096]: state gradient at a segment's start, from zero at its end
    float* seg_decay;     // scratch [B*H][nseg][64]: log2 decay over the segment
    uint32_t* ctrl;       // [1] status: a bounded wait expired
    uint32_t wait_limit_us;
    int B, T, H, NT;
    int nseg, cps;        // segments per sequence, chunks per segment
    int Hc, Wc, rev;      // scan order as in Params
    int sectors;          // dq, dk, dv and dg start on 32-byte boundaries
    float scale;
};

// ------------------------------------------------------------------------------------------ operands and scales
// a pair as a high and a low fp16 part
__device__ __forceinline__ void bwd_split(float2 x, uint32_t& h, uint32_t& l) {
    h = pack_half2(x.x, x.y);
    const float2 d = fma2(unpack_half2(h), make_float2(-1.f, -1.f), x);
    l = pack_half2(d.x, d.y);
}
// x[0..15] * f as a high and a low fp16 part, one row piece of two tiles
__device__ __forceinline__ void bwd_put_split(uint32_t hi, uint32_t lo, uint32_t row, uint32_t unit, const float* x, float f = 1.f) {
    uint32_t h[8], l[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) bwd_split(mul2(pair_of(x, i), two(f)), h[i], l[i]);
    put16(hi, row, unit, h);
    put16(lo, row, unit, l);
}
// in[0..15] * 2^(x * mul + add) likewise: the gated operands
__device__ __forceinline__ void bwd_put_gated(uint32_t hi, uint32_t lo, uint32_t row, uint32_t unit, const uint32_t* in, const float* x,
                                              float mul, float add) {
    uint32_t h[8], l[8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
        bwd_split(mul2(unpack_half2(in[i]), ex2_2(fma2(pair_of(x, i), two(mul), two(add)))), h[i], l[i]);
    put16(hi, row, unit, h);
    put16(lo, row, unit, l);
}

// largest |x| of 16 packed halves, as the bits of a half2 (both halves)
__device__ __forceinline__ uint32_t bwd_max16(const uint32_t* r) {
    __half2 m = __habs2(*reinterpret_cast<const __half2*>(&r[0]));
#pragma unroll
    for (int i = 1; i < 8; ++i) m = __hmax2(m, __habs2(*reinterpret_cast<const __half2*>(&r[i])));
    return *reinterpret_cast<uint32_t*>(&m);
}
__device__ __forceinline__ float bwd_half_max(uint32_t m) {
    const float2 f = unpack_half2(m);
    return fmaxf(f.x, f.y);
}
// the power of two that brings m to [2^(to-1), 2^to); 1 for zero and for what is not finite
__device__ __forceinline__ float bwd_scale(float m, int to) {
    const int e = static_cast<int>(__float_as_uint(m) >> 23);     // biased exponent: m in [2^(e-127), 2^(e-126))
    if (e == 0 || e == 255) return 1.f;
    return __uint_as_float(static_cast<uint32_t>(min(max(127 + to - 1 - (e - 127), 1), 254)) << 23);
}
__device__ __forceinline__ float bwd_log2(float f) { return static_cast<float>(static_cast<int>(__float_as_uint(f) >> 23) - 127); }  // of a power of two
__device__ __forceinline__ float bwd_inverse(float f) { return __uint_as_float((254u << 23) - __float_as_uint(f)); }   // of a power of two

// ------------------------------------------------------------------------------------------ segments' states
//   S after every chunk of a segment, from zero at its start:   S' = 2^G_L S + (k 2^(G_L-G))^T v
//   dS at a segment's start, from zero at its end, as a sum over the chunks in the same order, D their decay so far:
//                                                               dS' = dS + 2^D scale (q 2^G)^T do
// Both in one walk, so that the gates are read once, the two products share a chunk's round trips, and the blocks are as many as
// the gradient's, two to an SM in one wave (walks of their own, three to an SM, left the SMs idle for a third of the
// time).  Bound by memory, then by latency: a chunk is two dependent MMA round trips and two block barriers, the next chunk's
// tiles in flight meanwhile.
struct BwdStateSmem {
    static constexpr int kStage = 5 * kTileBytes;                                      // k, v, g, q, do
    static constexpr int kLowQ = 2 * kStage, kAfter = kLowQ + kTileBytes, kUpTo = kAfter + kTileBytes, kMisc = kUpTo + kTileBytes;
    static constexpr int kBytes = kMisc + 1024 + 1024;                                 // misc, alignment
};
struct BwdStateMisc {
    uint64_t full[2], bar_x, bar_inc, bar_fix;
    uint32_t tmem, gave_up;
    uint32_t reset;                   // the chunk has a gate of -inf
    uint32_t top[2][8];               // per warp: largest |k|, |q|, as half2 bits
    alignas(16) float gl[2][64];      // log2 decay of the chunk per channel
};
static_assert(sizeof(BwdStateMisc) <= 1024, "misc block too large");
enum { BWD_AFTER = 0, BWD_UP_TO = 1, BWD_INC_S = 2, BWD_INC_DS = 3 };

template <int K>
__global__ void __launch_bounds__(kComputeThreads, 2) gla_bwd_state_kernel(const __grid_constant__ Maps maps, const __grid_constant__ BwdParams P) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw), base = (raw + 1023u) & ~1023u;
    uint8_t* base_ptr = smem_raw + (base - raw);
    BwdStateMisc& M = *reinterpret_cast<BwdStateMisc*>(base_ptr + BwdStateSmem::kMisc);
    const int tid = threadIdx.x, w = tid >> 5, l = tid & 31;
    const int bh = blockIdx.x / P.nseg, seg = blockIdx.x - bh * P.nseg;
    const int first = seg * P.cps, n = min(P.cps, P.NT - first);
    const bool grad = seg > 0;                                     // nothing before the first segment needs its gradient
    const int b = bh / P.H, h = bh - b * P.H;
    const bool rev = P.rev != 0;

    if (tid == 0) {
        mbar_init(smem_u32(&M.full[0]), 1);
        mbar_init(smem_u32(&M.full[1]), 1);
        mbar_init(smem_u32(&M.bar_x), 1);
        mbar_init(smem_u32(&M.bar_inc), 1);
        mbar_init(smem_u32(&M.bar_fix), 1);
        M.gave_up = M.reset = 0u;
        fence_mbar_init();
    }
    if (w == 0) {
        tmem_alloc(smem_u32(&M.tmem), 128);
        tmem_relinquish();
    }
    // log factor of a row: the gates after it (k), its own and those before it (q), along the scan
    const uint32_t after = base + BwdStateSmem::kAfter, up_to = base + BwdStateSmem::kUpTo, low_q = base + BwdStateSmem::kLowQ;
    fill_constant(after, [&](uint32_t r, uint32_t s) { return (rev ? s < r : s > r) ? 1.f : 0.f; });
    fill_constant(up_to, [&](uint32_t r, uint32_t s) { return (rev ? s >= r : s <= r) ? 1.f : 0.f; });
    fence_proxy_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    pdl_wait();
    if (blockIdx.x == 0 && tid < 2) P.ctrl[tid] = 0u;
    const uint32_t tmem = M.tmem;
    auto load = [&](int i) {
        const uint32_t s = base + (i & 1) * BwdStateSmem::kStage, bar = smem_u32(&M.full[i & 1]);
        const Scan order{P.T, P.Hc, P.rev};
        const int tensors[3] = {TG, TK, TV}, others[2] = {TQ, TO};
        const uint32_t tiles[3] = {s + 2 * kTileBytes, s, s + kTileBytes}, other_tiles[2] = {s + 3 * kTileBytes, s + 4 * kTileBytes};
        mbar_arrive_expect_tx(bar, (grad ? 5 : 3) * kTileBytes);
        load_chunk(maps, order, first + i, b, h, 0, P.Hc, bar, tensors, tiles, l2_policy_normal());
        if (grad) load_chunk(maps, order, first + i, b, h, 0, P.Hc, bar, others, other_tiles, l2_policy_normal());
    };
    auto gate_sums = [&](int i) {          // of chunk i, as soon as it has landed
        const uint32_t tg = base + (i & 1) * BwdStateSmem::kStage + 2 * kTileBytes;
        wait_bar(P, M.full[i & 1], (i >> 1) & 1, M.gave_up);
        tc_fence_after();
        tile_mma<0, 1>(acc_slot(tmem, BWD_AFTER), after, tg, false);
        if (grad) tile_mma<0, 1>(acc_slot(tmem, BWD_UP_TO), up_to, tg, false);
        umma_commit(smem_u32(&M.bar_x));
    };
    if (w == 0 && elect_one()) {
        load(0);
        if (n > 1) load(1);
        gate_sums(0);
    }
    __syncwarp();

    const uint32_t row = 16u * (w & 3) + (l & 15u), c0 = 32u * (w >> 2) + 16u * (static_cast<uint32_t>(l) >> 4), u0 = c0 >> 3;
    float S[16], dS[16], total = 0.f;          // a state row piece each: channel `row`, columns c0 .. +15
    uint32_t fixes = 0;
#pragma unroll
    for (int e = 0; e < 16; ++e) S[e] = dS[e] = 0.f;
    const size_t cslot = static_cast<size_t>(bh) * P.NT;

    for (int i = 0; i < n; ++i) {
        const int st = i & 1;
        const uint32_t tk = base + st * BwdStateSmem::kStage, tv = tk + kTileBytes, tg = tv + kTileBytes, tq = tg + kTileBytes,
                       tdo = tq + kTileBytes;
        if (i == n - 1) pdl_release();
        wait_bar(P, M.full[st], (i >> 1) & 1, M.gave_up);
        uint32_t k[8], q[8];
        row16(tk, row, u0, k);
        const uint32_t mk = __reduce_max_sync(0xffffffffu, __float_as_uint(bwd_half_max(bwd_max16(k))));
        uint32_t mq = 0u;
        if (grad) {
            row16(tq, row, u0, q);
            mq = __reduce_max_sync(0xffffffffu, __float_as_uint(bwd_half_max(bwd_max16(q))));
        }
        if (l == 0) { M.top[0][w] = mk; M.top[1][w] = mq; }
        wait_bar(P, M.bar_x, i & 1, M.gave_up);
        tc_fence_after();
        float x[16], y[16];
        acc_read(tmem, BWD_AFTER, w, x);
        if (grad) acc_read(tmem, BWD_UP_TO, w, y);
        tmem_ld_wait();
        auto chunk_decay = [&] {                                    // all gates after the first row + its own
            uint32_t gr[8];
            row16(tg, row, u0, gr);
            bool lost = false;
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const float2 gf = unpack_half2(gr[e]);
                const float2 s = mul2(make_float2(x[2 * e] + gf.x, x[2 * e + 1] + gf.y), two(kLog2e));
                M.gl[st][c0 + 2 * e] = s.x;
                M.gl[st][c0 + 2 * e + 1] = s.y;
                lost = lost || !(s.x > -3e38f) || !(s.y > -3e38f);
            }
            return lost;
        };
        const bool first_row = row == (rev ? 63u : 0u);
        if (first_row && chunk_decay()) M.reset = 1u;
        __syncthreads();                                            // every warp's maxima are there
        if (M.reset != 0u) {                                        // 0 x -inf is no sum: once more from the lowest finite gate
            uint32_t gr[8];
            row16(tg, row, u0, gr);
#pragma unroll
            for (int e = 0; e < 8; ++e) gr[e] = hmax2_nan(gr[e], 0xfbfffbffu);      // -65504
            put16(tg, row, u0, gr);
            fence_proxy_async_smem();
            tc_fence_before();
            __syncthreads();
            if (tid == 0) M.reset = 0u;
            if (w == 0 && elect_one()) {
                tc_fence_after();
                tile_mma<0, 1>(acc_slot(tmem, BWD_AFTER), after, tg, false);
                if (grad) tile_mma<0, 1>(acc_slot(tmem, BWD_UP_TO), up_to, tg, false);
                umma_commit(smem_u32(&M.bar_fix));
            }
            __syncwarp();
            wait_bar(P, M.bar_fix, fixes & 1u, M.gave_up);
            ++fixes;
            tc_fence_after();
            acc_read(tmem, BWD_AFTER, w, x);
            if (grad) acc_read(tmem, BWD_UP_TO, w, y);
            tmem_ld_wait();
            if (first_row) chunk_decay();
        }
        uint32_t top_k = M.top[0][0], top_q = M.top[1][0];
#pragma unroll
        for (int j = 1; j < 8; ++j) { top_k = max(top_k, M.top[0][j]); top_q = max(top_q, M.top[1][j]); }
        const float fk = bwd_scale(__uint_as_float(top_k), 15), fq = bwd_scale(__uint_as_float(top_q), 15);
        bwd_put_gated(tk, tg, row, u0, k, x, kLog2e, bwd_log2(fk));            // the gates have been read: the low part's tile
        if (grad) bwd_put_gated(tq, low_q, row, u0, q, y, kLog2e, bwd_log2(fq));
        fence_proxy_async_smem();
        tc_fence_before();
        __syncthreads();
        if (w == 0 && elect_one()) {
            tc_fence_after();
            tile_mma<1, 1>(acc_slot(tmem, BWD_INC_S), tk, tv, false);
            tile_mma<1, 1>(acc_slot(tmem, BWD_INC_S), tg, tv, true);
            if (grad) {
                tile_mma<1, 1>(acc_slot(tmem, BWD_INC_DS), tq, tdo, false);
                tile_mma<1, 1>(acc_slot(tmem, BWD_INC_DS), low_q, tdo, true);
            }
            umma_commit(smem_u32(&M.bar_inc));
        }
        const float gl = M.gl[st][row], decay = ex2(gl), ck = bwd_inverse(fk), cq = P.scale * bwd_inverse(fq) * ex2(total);
        total += gl;
        wait_bar(P, M.bar_inc, i & 1, M.gave_up);
        tc_fence_after();
        if (w == 0 && elect_one()) {                                // this chunk's stage is free, and so are its gate sums
            if (i + 2 < n) load(i + 2);
            if (i + 1 < n) gate_sums(i + 1);
        }
        __syncwarp();
        acc_read(tmem, BWD_INC_S, w, x);
        if (grad) acc_read(tmem, BWD_INC_DS, w, y);
        tmem_ld_wait();
        tc_fence_before();
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const float2 s = fma2(two(decay), pair_of(S, e), mul2(two(ck), pair_of(x, e)));
            S[2 * e] = s.x; S[2 * e + 1] = s.y;
        }
        const size_t at = cslot + first + i;
        float4* dst = reinterpret_cast<float4*>(P.chunk_state + at * 4096) + tid;
#pragma unroll
        for (int e = 0; e < 4; ++e) dst[e * kComputeThreads] = make_float4(S[4 * e], S[4 * e + 1], S[4 * e + 2], S[4 * e + 3]);
        if (c0 == 0) P.chunk_decay[at * 64 + row] = total;
        if (grad) {
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const float2 s = fma2(two(cq), pair_of(y, e), pair_of(dS, e));
                dS[2 * e] = s.x; dS[2 * e + 1] = s.y;
            }
        }
    }
    if (grad) {
        const size_t at = static_cast<size_t>(bh) * P.nseg + seg;
        float4* dst = reinterpret_cast<float4*>(P.seg_grad + at * 4096) + tid;
#pragma unroll
        for (int e = 0; e < 4; ++e) dst[e * kComputeThreads] = make_float4(dS[4 * e], dS[4 * e + 1], dS[4 * e + 2], dS[4 * e + 3]);
        if (c0 == 0) P.seg_decay[at * 64 + row] = total;
    }
    tc_fence_before();
    __syncthreads();
    if (tid == 0 && M.gave_up) P.chunk_decay[(cslot + first + n - 1) * 64] = __uint_as_float(kTimedOut);
    if (w == 0) tmem_dealloc(tmem, 128);
}

// ------------------------------------------------------------------------------------------ the gradient
struct BwdChunkSmem {
    static constexpr int kG = 0, kQ = kTileBytes, kK = 2 * kTileBytes, kV = 3 * kTileBytes, kDo = 4 * kTileBytes;
    static constexpr int kQl = 5 * kTileBytes, kKl = 6 * kTileBytes;
    // four tiles, used in turn for St and dSt, for P and dP (high and low parts each), and, as 64 x 64 fp32, for the terms of dg
    static constexpr int kR = 7 * kTileBytes, kMat = 11 * kTileBytes;
    static constexpr int kS0 = 12 * kTileBytes;                       // the state the segment starts from, fp32, each thread's own piece
    static constexpr int kMisc = 14 * kTileBytes;
    // no slack: dynamic shared memory starts on a 1024-byte boundary when a kernel has no other (checked at run time), and two
    // CTAs of 113 KB fill an SM
    static constexpr int kBytes = kMisc + 1024;
};
struct BwdChunkMisc {
    uint64_t full, bar_x, bar_a, bar_s, bar_o;
    uint32_t tmem;
    // per chunk: largest |q|, |k|, |v|, |do|, |S|, |dS| as float bits, and whether the chunk needs the pair-by-pair path
    uint32_t top[2][8];
    alignas(16) float vec[64];        // log2: half the chunk's total decay per channel
    alignas(16) float decay[64];      // log2 decay from the segment's start to the chunk's start
};
static_assert(sizeof(BwdChunkMisc) <= 1024, "misc block too large");
enum { BWD_BAR_COMPUTE = 1, BWD_BAR_GATED = 2, BWD_BAR_STATES = 3, BWD_BAR_SCORES = 4, BWD_BAR_READ = 5 };     // named barriers
enum { BWD_X = 0, BWD_P = 1, BWD_DP = 2, BWD_DQ_S = 3, BWD_DK_S = 4, BWD_DV_S = 5, BWD_INC = 6, BWD_DQ_I = 7 };

// a 64 x 64 fp32 tile whose 16-byte units are permuted by the row, so that both row pieces and columns are read without
// bank conflicts
__device__ __forceinline__ uint32_t bwd_f32(uint32_t tile, uint32_t row, uint32_t col) {
    return tile + row * 256u + ((((col >> 2) ^ row) & 15u) << 4) + ((col & 3u) << 2);
}
__device__ __forceinline__ void bwd_f32_put16(uint32_t tile, uint32_t row, uint32_t c0, const float* x) {
#pragma unroll
    for (uint32_t e = 0; e < 4; ++e) st_shared_f4(bwd_f32(tile, row, c0 + 4 * e), x[4 * e], x[4 * e + 1], x[4 * e + 2], x[4 * e + 3]);
}
__device__ __forceinline__ void bwd_f32_row16(uint32_t tile, uint32_t row, uint32_t c0, float* x) {
#pragma unroll
    for (uint32_t e = 0; e < 4; ++e) {
        const float4 v = ld_shared_f4(bwd_f32(tile, row, c0 + 4 * e));
        x[4 * e] = v.x; x[4 * e + 1] = v.y; x[4 * e + 2] = v.z; x[4 * e + 3] = v.w;
    }
}

// e^gate of 8 channels (unit u) of a row, fp32: their halves lie 128 bytes apart, so that the eight lanes of a row read without conflicts
__device__ __forceinline__ uint32_t bwd_decay(uint32_t tile, uint32_t row, uint32_t u, uint32_t half) {
    return tile + row * 256u + 128u * half + 16u * u;
}

// A chunk with a strong decay, pair by pair in fp32: P (scaled by fq fk, into its accumulator), and the part of dq and dk that
// comes from within the chunk (into BWD_DQ_I and BWD_DP, complete); q and k are then rewritten with the references 0 and G_L,
// whose exponents are never positive.
// A pair's factors are the running product of the decays between its tokens, which are taken once per token and channel: with an
// exponential per pair and channel the special-function unit alone was busy for 17 thousand cycles a chunk.  Eight neighbouring
// lanes, 8 channels each, share tokens r and 63 - r, so that all of them have 65 pairs to walk; what bounds it now is the shared memory
// they read.  A sequence of nothing but such chunks, with an exponential per pair / now: B4 H12 T6400 976 / 640 us, B8 H6 T1600 300 / 198,
// B32 H12 T2048 2490 / 1600, B8 H3 T1600 K = 32 185 / 126 (ordinary ones 189, 64, 475, 43).
// Out of line.  Its loads ahead are as many as registers allow: with fewer in use the compiler spilt some of the ordinary chunk's around
// the call (3 to 6 percent there).
__device__ __noinline__ void bwd_wide_chunk(uint32_t base, float* vec, uint32_t tmem, float fq, float fk, float scale,
                                            bool rev) {
    const int tid = threadIdx.x, w = tid >> 5, l = tid & 31;
    const uint32_t row = 16u * (w & 3) + (l & 15u), c0 = 32u * (w >> 2) + 16u * (static_cast<uint32_t>(l) >> 4), u0 = c0 >> 3;
    const uint32_t tg = base + BwdChunkSmem::kG, tq = base + BwdChunkSmem::kQ, tk = base + BwdChunkSmem::kK;
    const uint32_t dp = base + BwdChunkSmem::kR, out = dp + 2 * kTileBytes;
    const uint32_t decays = base + BwdChunkSmem::kQl;      // until the low parts of q and k go there
    static_assert(BwdChunkSmem::kKl == BwdChunkSmem::kQl + kTileBytes, "the decays take both tiles");
    auto sync = [] { named_bar_sync(BWD_BAR_COMPUTE, kComputeThreads); };
    auto at = [&](int t) { return static_cast<uint32_t>(rev ? 63 - t : t); };     // row of the chunk's t-th token
    {
        uint32_t g[8];
        row16(tg, row, u0, g);
#pragma unroll
        for (uint32_t e = 0; e < 4; ++e) {
            const float2 a = ex2_2(mul2(unpack_half2(g[2 * e]), two(kLog2e))), b = ex2_2(mul2(unpack_half2(g[2 * e + 1]), two(kLog2e)));
            st_shared_f4(bwd_decay(decays, row, u0 + (e >> 1), e & 1u), a.x, a.y, b.x, b.y);
        }
        float x[16];
        acc_read(tmem, BWD_DP, w, x);
        tmem_ld_wait();
        bwd_f32_put16(dp, row, c0, x);
    }
    sync();
    const int r = tid >> 3;
    const uint32_t u = tid & 7u;
    float2 acc[4], F[4];
    auto start = [&] {
#pragma unroll
        for (int e = 0; e < 4; ++e) { acc[e] = two(0.f); F[e] = two(1.f); }
    };
    auto decay = [&](uint32_t row_t) {                     // F times the decays of a token
        const float4 a = ld_shared_f4(bwd_decay(decays, row_t, u, 0)), b = ld_shared_f4(bwd_decay(decays, row_t, u, 1));
        F[0] = mul2(F[0], make_float2(a.x, a.y)); F[1] = mul2(F[1], make_float2(a.z, a.w));
        F[2] = mul2(F[2], make_float2(b.x, b.y)); F[3] = mul2(F[3], make_float2(b.z, b.w));
    };
    auto unit = [&](uint32_t tile, uint32_t row_t, float2* v) {
        const uint4 h = ld_shared_v4(sw_unit(tile, row_t, u));
        v[0] = unpack_half2(h.x); v[1] = unpack_half2(h.y); v[2] = unpack_half2(h.z); v[3] = unpack_half2(h.w);
    };
    auto put = [&](int t) {
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[e] = mul2(acc[e], two(scale));
        st_shared_f4(bwd_f32(out, at(t), 8u * u), acc[0].x, acc[0].y, acc[1].x, acc[1].y);
        st_shared_f4(bwd_f32(out, at(t), 8u * u + 4u), acc[2].x, acc[2].y, acc[3].x, acc[3].y);
    };
    auto take = [&](uint32_t tile, int slot) {             // a whole array into an accumulator
        float x[16];
        bwd_f32_row16(tile, row, c0, x);
        acc_write(tmem, slot, w, x);
    };
    // dk: the queries from each key onwards.  A warp's four pairs of tokens go as far as the longest of them.
#pragma unroll 1
    for (int second = 0; second < 2; ++second) {
        const int j = second ? 63 - r : r, steps = second ? r | 3 : 63 - (r & ~3);
        start();
#pragma unroll 4
        for (int s = 0; s <= steps; ++s) {
            const int t = min(j + s, 63);
            if (s > 0) decay(at(t));
            float2 v[4];
            unit(tq, at(t), v);
            const float d = j + s <= 63 ? ld_shared_f(bwd_f32(dp, at(t), at(j))) : 0.f;
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[e] = fma2(two(d), mul2(v[e], F[e]), acc[e]);
        }
        put(j);
    }
    sync();
    take(out, BWD_DP);
    sync();
    // dq, and P in the place of dP: the keys from each query backwards, eight at a time, whose sums over the eight lanes end with one lane
    // each
#pragma unroll 1
    for (int second = 0; second < 2; ++second) {
        const int i = second ? 63 - r : r, steps = second ? 63 - (r & ~3) : r | 3;
        float2 q[4];
        unit(tq, at(i), q);
        start();
#pragma unroll 1
        for (int s0 = 0; s0 <= steps; s0 += 8) {
            float sum[8];
            uint4 h[8];
            float d[8];
            float4 f[2][2];
#pragma unroll
            for (int s = 0; s < 8; ++s) {
                const int j = max(i - s0 - s, 0);
                h[s] = ld_shared_v4(sw_unit(tk, at(j), u));
                d[s] = s0 + s <= i ? ld_shared_f(bwd_f32(dp, at(i), at(j))) : 0.f;
            }
#pragma unroll
            for (int s = 0; s < 8; ++s) {
                if (s % 2 == 0) {
#pragma unroll
                    for (int t = 0; t < 2; ++t) {
                        const uint32_t row_t = at(max(i - s0 - s - t, 0));
                        f[t][0] = ld_shared_f4(bwd_decay(decays, row_t, u, 0));
                        f[t][1] = ld_shared_f4(bwd_decay(decays, row_t, u, 1));
                    }
                }
                float2 v[4] = {unpack_half2(h[s].x), unpack_half2(h[s].y), unpack_half2(h[s].z), unpack_half2(h[s].w)};
                float2 dot = two(0.f);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    v[e] = mul2(v[e], F[e]);
                    dot = fma2(q[e], v[e], dot);
                    acc[e] = fma2(two(d[s]), v[e], acc[e]);
                }
                sum[s] = dot.x + dot.y;
                const float4 fa = f[s % 2][0], fb = f[s % 2][1];
                F[0] = mul2(F[0], make_float2(fa.x, fa.y)); F[1] = mul2(F[1], make_float2(fa.z, fa.w));
                F[2] = mul2(F[2], make_float2(fb.x, fb.y)); F[3] = mul2(F[3], make_float2(fb.z, fb.w));
            }
#pragma unroll
            for (int m = 4; m > 0; m >>= 1) {
                const bool upper = (u & m) != 0;
#pragma unroll
                for (int e = 0; e < m; ++e) {
                    const float give = upper ? sum[e] : sum[e + m], keep = upper ? sum[e + m] : sum[e];
                    sum[e] = keep + __shfl_xor_sync(0xffffffffu, give, m);
                }
            }
            const int j = i - s0 - static_cast<int>(u);    // keys after the query are masked later
            if (j >= 0) st_shared_f(bwd_f32(dp, at(i), at(j)), sum[0] * fq * fk);
        }
        put(i);
    }
    sync();
    take(dp, BWD_P);
    take(out, BWD_DQ_I);
    // The factors of what lies outside the chunk, e^G for q and e^(G_L-G) for k, from sums that run one way each.  X and the chunk's middle
    // would lose what a hard reset leaves of them (at gates of -1000 the fourth digit, at -60000 all), and a gate of -inf has no X.
    sync();
    const uint32_t sums = decays;                          // [4][64]: of 16 tokens each
    {
        const uint32_t c = tid & 63u;
        const int first = 16 * (tid >> 6);
        float g[16], run = 0.f;
#pragma unroll
        for (int t = 0; t < 16; ++t) g[t] = __half2float(__ushort_as_half(ld_shared_u16(tg + sw_f16(at(first + t), c))));
#pragma unroll
        for (int t = 0; t < 16; ++t) st_shared_f(bwd_f32(dp, at(first + t), c), run += g[t]);
        st_shared_f(sums + 256u * (tid >> 6) + 4u * c, run);
        run = 0.f;
#pragma unroll
        for (int t = 15; t >= 0; --t) {
            st_shared_f(bwd_f32(out, at(first + t), c), run);
            run += g[t];
        }
    }
    sync();
    float x[16], y[16];
    bwd_f32_row16(dp, row, c0, x);
    bwd_f32_row16(out, row, c0, y);
    const uint32_t quarter = (rev ? 63u - row : row) >> 4;
#pragma unroll
    for (uint32_t j = 0; j < 4; ++j) {
#pragma unroll
        for (uint32_t e = 0; e < 4; ++e) {
            const float4 v = ld_shared_f4(sums + 256u * j + 4u * c0 + 16u * e);
            const float z[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                if (j < quarter) x[4 * e + i] += z[i];
                if (j > quarter) y[4 * e + i] += z[i];
            }
        }
    }
    if (tid < 64) {
        float half = 0.f;
#pragma unroll
        for (uint32_t j = 0; j < 4; ++j) half += ld_shared_f(sums + 256u * j + 4u * tid);
        half *= 0.5f * kLog2e;
        vec[tid] = half < -2.f * kBwdFar ? -2.f * kBwdFar : half;
    }
    sync();
    uint32_t in[8];
    row16(tq, row, u0, in);
    bwd_put_gated(tq, base + BwdChunkSmem::kQl, row, u0, in, x, kLog2e, bwd_log2(fq));
    row16(tk, row, u0, in);
    bwd_put_gated(tk, base + BwdChunkSmem::kKl, row, u0, in, y, kLog2e, bwd_log2(fk));
    // for the outputs: the smaller of the two, which one it is in its last bit; the other is G_L less this one
#pragma unroll
    for (int e = 0; e < 16; ++e) {
        const bool after = fabsf(y[e]) < fabsf(x[e]);
        float v = kLog2e * (after ? y[e] : x[e]);
        v = v < -kBwdFar ? -kBwdFar : v;
        x[e] = __uint_as_float((__float_as_uint(v) & ~1u) | (after ? 1u : 0u));
    }
    acc_write(tmem, BWD_X, w, x);
    tmem_st_wait();
}

constexpr int kBwdChunkThreads = kComputeThreads + 32;       // eight compute warps, one that issues MMAs and copies

// Per chunk (walked from the segment's last to its first), compute warps | issuing warp:
//   tiles landed:  maxima of the tiles and states    | X = G - G_L/2 and dP = do v^T
//   St, dSt as split operands                        | do St^T, v dSt^T
//   qt, kt as split operands                         | P = qt kt^T, qt^T do, kt dSt
//   P, dP masked, as split operands                  | P^T do, dP kt, dP^T qt
//   dS to the chunk's start                          | next chunk's copies once those have run
//   outputs; dg                                      |
// The compute warps hand operands over with an arrival and never wait for one another to do so.
template <int K>
__global__ void __launch_bounds__(kBwdChunkThreads, 2) gla_bwd_chunk_kernel(const __grid_constant__ Maps maps, const __grid_constant__ BwdParams P) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t base = smem_u32(smem_raw);
    uint8_t* base_ptr = smem_raw;
    if ((base & 1023u) != 0u) {                                        // never with this kernel's shared memory, see kBytes
        if (threadIdx.x == 0) atomicCAS(P.ctrl + 1, 0u, static_cast<uint32_t>(WHERE_MBAR));
        return;
    }
    BwdChunkMisc& M = *reinterpret_cast<BwdChunkMisc*>(base_ptr + BwdChunkSmem::kMisc);
    const int tid = threadIdx.x, w = tid >> 5, l = tid & 31;
    const int bh = blockIdx.x / P.nseg, seg = blockIdx.x - bh * P.nseg;
    const int first = seg * P.cps, n = min(P.cps, P.NT - first);
    const int b = bh / P.H, h = bh - b * P.H;
    const bool rev = P.rev != 0;
    const size_t cslot = static_cast<size_t>(bh) * P.NT;
    const uint32_t tg = base + BwdChunkSmem::kG, tq = base + BwdChunkSmem::kQ, tk = base + BwdChunkSmem::kK, tv = base + BwdChunkSmem::kV,
                   tdo = base + BwdChunkSmem::kDo, ql = base + BwdChunkSmem::kQl, kl = base + BwdChunkSmem::kKl,
                   r0 = base + BwdChunkSmem::kR, r1 = r0 + kTileBytes, r2 = r1 + kTileBytes, r3 = r2 + kTileBytes;

    if (tid == 0) {
        mbar_init(smem_u32(&M.full), 1);
        mbar_init(smem_u32(&M.bar_x), 1);
        mbar_init(smem_u32(&M.bar_a), 1);
        mbar_init(smem_u32(&M.bar_s), 1);
        mbar_init(smem_u32(&M.bar_o), 1);
        fence_mbar_init();
    }
    if (w == 0) {
        tmem_alloc(smem_u32(&M.tmem), 256);
        tmem_relinquish();
    }
    fill_constant(base + BwdChunkSmem::kMat, [&](uint32_t r, uint32_t s) { return (rev ? s >= r : s <= r) ? 0.5f : -0.5f; });      // G - G_L / 2
    if (tid < 16) M.top[tid >> 3][tid & 7] = 0u;
    fence_proxy_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    pdl_wait();
    const uint32_t tmem = M.tmem;

    if (w == kComputeThreads / 32) {
        // ==================================================================== issuing warp
        const uint32_t sx = acc_slot(tmem, BWD_X), sp = acc_slot(tmem, BWD_P), sdp = acc_slot(tmem, BWD_DP), sdq = acc_slot(tmem, BWD_DQ_S),
                       sdk = acc_slot(tmem, BWD_DK_S), sdv = acc_slot(tmem, BWD_DV_S), sinc = acc_slot(tmem, BWD_INC), sdqi = acc_slot(tmem, BWD_DQ_I);
        // chunk i's tiles, and the state after chunk i - 1 (relative to the segment's start) into r2, r3
        auto load = [&](int i) {
            const uint32_t bar = smem_u32(&M.full);
            mbar_arrive_expect_tx(bar, i > 0 ? 7 * kTileBytes + 256 : 5 * kTileBytes);
            const int tensors[5] = {TG, TO, TV, TQ, TK};
            const uint32_t tiles[5] = {tg, tdo, tv, tq, tk};
            load_chunk(maps, Scan{P.T, P.Hc, P.rev}, first + i, b, h, 0, P.Hc, bar, tensors, tiles, l2_policy_normal());
            if (i > 0) {
                bulk_load(r2, P.chunk_state + (cslot + first + i - 1) * 4096, 2 * kTileBytes, bar);
                bulk_load(smem_u32(M.decay), P.chunk_decay + (cslot + first + i - 1) * 64, 256, bar);
            }
        };
        if (elect_one()) load(n - 1);
        __syncwarp();
        for (int i = n - 1, it = 0; i >= 0; --i, ++it) {
            const uint32_t ph = it & 1;
            wait_bar(P, M.full, ph);
            if (it > 0) named_bar_sync(BWD_BAR_READ, kBwdChunkThreads);            // the previous chunk's accumulators are read
            tc_fence_after();
            if (elect_one()) {
                tile_mma<0, 1>(sx, base + BwdChunkSmem::kMat, tg, false);
                tile_mma<0, 0>(sdp, tdo, tv, false);
                umma_commit(smem_u32(&M.bar_x));
            }
            named_bar_sync(BWD_BAR_STATES, kBwdChunkThreads);
            tc_fence_after();
            const bool wide = M.top[i & 1][6] != 0u;
            if (elect_one()) {
                tile_mma<0, 0>(sdq, tdo, r0, false);
                tile_mma<0, 0>(sdq, tdo, r1, true);
                tile_mma<0, 0>(sdk, tv, r2, false);
                tile_mma<0, 0>(sdk, tv, r3, true);
            }
            named_bar_sync(BWD_BAR_GATED, kBwdChunkThreads);
            tc_fence_after();
            if (elect_one()) {
                if (!wide) {
                    tile_mma<0, 0>(sp, tq, tk, false);
                    tile_mma<0, 0>(sp, tq, kl, true);
                    tile_mma<0, 0>(sp, ql, tk, true);
                }
                umma_commit(smem_u32(&M.bar_a));
                tile_mma<1, 1>(sinc, tq, tdo, false);
                tile_mma<1, 1>(sinc, ql, tdo, true);
                tile_mma<0, 1>(sdv, tk, r2, false);
                tile_mma<0, 1>(sdv, tk, r3, true);
                tile_mma<0, 1>(sdv, kl, r2, true);
                umma_commit(smem_u32(&M.bar_s));
            }
            named_bar_sync(BWD_BAR_SCORES, kBwdChunkThreads);
            tc_fence_after();
            if (elect_one()) {
                const uint32_t dv = wide ? sp : sdp;
                tile_mma<1, 1>(dv, r0, tdo, false);
                tile_mma<1, 1>(dv, r1, tdo, true);
                if (!wide) {
                    tile_mma<0, 1>(sdqi, r2, tk, false);
                    tile_mma<0, 1>(sdqi, r2, kl, true);
                    tile_mma<0, 1>(sdqi, r3, tk, true);
                    tile_mma<1, 1>(sp, r2, tq, false);
                    tile_mma<1, 1>(sp, r2, ql, true);
                    tile_mma<1, 1>(sp, r3, tq, true);
                }
                umma_commit(smem_u32(&M.bar_o));
            }
            __syncwarp();
            wait_bar(P, M.bar_o, ph);
            if (i > 0 && elect_one()) load(i - 1);
            __syncwarp();
        }
    } else {
        // ==================================================================== compute warps
        // This thread's piece of every 64 x 64 array: row `row`, columns c0 .. c0 + 15.  A row is a token (scores, gradients) or
        // a key channel (states).
        const uint32_t row = 16u * (w & 3) + (l & 15u), c0 = 32u * (w >> 2) + 16u * (static_cast<uint32_t>(l) >> 4), u0 = c0 >> 3;
        const bool real_row = row < K;
        auto sync = [] { named_bar_sync(BWD_BAR_COMPUTE, kComputeThreads); };
        auto hand_over = [](uint32_t id) {                   // operands written by this thread may be read by the tensor core
            fence_proxy_async_smem();
            tc_fence_before();
            named_bar_arrive(id, kBwdChunkThreads);
        };
        float dS[16];                 // the state gradient at the end of the current chunk
        const uint32_t s0_at = base + BwdChunkSmem::kS0 + 16u * tid;           // float4 e of this thread 4096 bytes apart
        auto own = [&](uint32_t at, float* x) {
#pragma unroll
            for (uint32_t e = 0; e < 4; ++e) {
                const float4 v = ld_shared_f4(at + 16u * kComputeThreads * e);
                x[4 * e] = v.x; x[4 * e + 1] = v.y; x[4 * e + 2] = v.z; x[4 * e + 3] = v.w;
            }
        };
        auto get = [&](const float* src, int step, float* x) {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float4 v = __ldcg(reinterpret_cast<const float4*>(src) + e * step);
                x[4 * e] = v.x; x[4 * e + 1] = v.y; x[4 * e + 2] = v.z; x[4 * e + 3] = v.w;
            }
        };
        auto chain = [&](float* x, float f, const float* y) {                // x = f x + y
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const float2 z = fma2(two(f), pair_of(x, e), pair_of(y, e));
                x[2 * e] = z.x; x[2 * e + 1] = z.y;
            }
        };
        const size_t state_off = (static_cast<size_t>(bh) * K + row) * 64 + c0;
        {
            float S0[16];
#pragma unroll
            for (int e = 0; e < 16; ++e) S0[e] = dS[e] = 0.f;
            if (P.h0 != nullptr && real_row) get(P.h0 + state_off, 1, S0);
            if (P.dht != nullptr && real_row) get(P.dht + state_off, 1, dS);
#pragma unroll 2
            for (int j = 0; j < seg; ++j) {
                const size_t at = cslot + static_cast<size_t>(j + 1) * P.cps - 1;
                float y[16];
                get(P.chunk_state + at * 4096 + 4 * tid, kComputeThreads, y);
                chain(S0, ex2(__ldcg(P.chunk_decay + at * 64 + row)), y);
            }
#pragma unroll 2
            for (int j = P.nseg - 1; j > seg; --j) {
                const size_t at = static_cast<size_t>(bh) * P.nseg + j;
                float y[16];
                get(P.seg_grad + at * 4096 + 4 * tid, kComputeThreads, y);
                chain(dS, ex2(__ldcg(P.seg_decay + at * 64 + row)), y);
            }
#pragma unroll
            for (uint32_t e = 0; e < 4; ++e) st_shared_f4(s0_at + 16u * kComputeThreads * e, S0[4 * e], S0[4 * e + 1], S0[4 * e + 2], S0[4 * e + 3]);
            // did a wait run out where the segment's states were made?
            if (c0 == 0 && __float_as_uint(__ldcg(P.chunk_decay + (cslot + first + n - 1) * 64 + row)) == kTimedOut) report_timeout(P);
            float later = 0.f;
            if (P.dht != nullptr || seg + 1 < P.nseg) {                  // dS is not zero at the segment's end
                float y[16];
                const size_t at = cslot + first + n - 1;
                get(P.chunk_state + at * 4096 + 4 * tid, kComputeThreads, y);
                chain(S0, ex2(__ldcg(P.chunk_decay + at * 64 + row)), y);          // now the state after the segment
#pragma unroll
                for (int e = 0; e < 16; ++e) later = fmaf(S0[e], dS[e], later);
                later += __shfl_xor_sync(0xffffffffu, later, 16);
            }
            // halves of the sum, per channel, by way of a tile that is not in use yet
            if (l < 16) asm volatile("st.shared.f32 [%0], %1;" ::"r"(kl + 256u * (w >> 2) + 4u * row), "f"(later) : "memory");
        }
        sync();
        float later = ld_shared_f(kl + 4u * (tid & 63)) + ld_shared_f(kl + 256u + 4u * (tid & 63));         // dg's share of all later tokens, channel tid & 63
        const uint32_t decay_at = smem_u32(M.decay);
        // 16 halves: 32 bytes, in one store where the caller's tensors allow it (whole sectors: 164 -> 153 us)
        auto put_row = [&](void* to, const uint32_t* r) {
            if (P.sectors) st_global_v8(to, r);
            else {
                reinterpret_cast<uint4*>(to)[0] = make_uint4(r[0], r[1], r[2], r[3]);
                reinterpret_cast<uint4*>(to)[1] = make_uint4(r[4], r[5], r[6], r[7]);
            }
        };
        const uint32_t last_row = rev ? 0u : 63u;
        const int above = 32 * (w >> 2) - 16 * (w & 3);                  // first column - first row of this warp's piece
        const bool on_diagonal = above == 0 || above == -16;
        const bool beyond = rev ? above < -16 : above > 0;               // wholly on the masked side of the diagonal

        for (int i = n - 1, it = 0; i >= 0; --i, ++it) {
            const int p = i & 1;
            const uint32_t ph = it & 1;
            wait_bar(P, M.full, ph);
            uint32_t qr[8], kr[8];
            float S[16], x[16];
            own(s0_at, S);
            if (i > 0) {
                own(r2 + 16u * tid, x);
                chain(S, ex2(ld_shared_f(decay_at + 4u * row)), x);
            }
            row16(tq, row, u0, qr);
            row16(tk, row, u0, kr);
            {
                float m[6];
                uint32_t t[8];
                m[0] = bwd_half_max(bwd_max16(qr));
                m[1] = bwd_half_max(bwd_max16(kr));
                row16(tv, row, u0, t);
                m[2] = bwd_half_max(bwd_max16(t));
                row16(tdo, row, u0, t);
                m[3] = bwd_half_max(bwd_max16(t));
                m[4] = m[5] = 0.f;
#pragma unroll
                for (int e = 0; e < 16; ++e) {
                    m[4] = fmaxf(m[4], fabsf(S[e]));
                    m[5] = fmaxf(m[5], fabsf(dS[e]));
                }
                uint32_t mine = 0u;
#pragma unroll
                for (int j = 0; j < 6; ++j) {
                    const uint32_t r = __reduce_max_sync(0xffffffffu, __float_as_uint(m[j]));
                    if (l == j) mine = r;
                }
                if (l < 6) atomicMax(&M.top[p][l], mine);
            }
            wait_bar(P, M.bar_x, ph);
            tc_fence_after();
            acc_read(tmem, BWD_X, w, x);
            tmem_ld_wait();
            if (row == last_row) {                                      // X of the last row is half the chunk's decay
                bool far = false;
#pragma unroll
                for (int e = 0; e < 16; ++e) {
                    const float half_decay = x[e] * kLog2e;
                    M.vec[c0 + e] = half_decay;
                    far = far || !(-half_decay <= kBwdRefLimit);
                }
                if (far) M.top[p][6] = 1u;
            }
            sync();                                                     // maxima, decay and the wide flag are complete
            const float fq = bwd_scale(__uint_as_float(M.top[p][0]), 6), fk = bwd_scale(__uint_as_float(M.top[p][1]), 6);
            const float fp = 0.125f, fd = bwd_scale(__uint_as_float(M.top[p][2]), 5) * bwd_scale(__uint_as_float(M.top[p][3]), 4);
            const float fS = bwd_scale(__uint_as_float(M.top[p][4]), 15), fdS = bwd_scale(__uint_as_float(M.top[p][5]), 15);
            const bool wide = M.top[p][6] != 0u;
            if (wide) {
                // out of line, and what registers hold across the call waits in accumulators that are not in use yet: the ordinary
                // chunk must not pay for it with spills (the SM's shared memory leaves no L1 to catch them)
                acc_write(tmem, BWD_DQ_S, w, dS);
                acc_write(tmem, BWD_DK_S, w, S);
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    x[e] = __uint_as_float(qr[e]);
                    x[8 + e] = __uint_as_float(kr[e]);
                }
                acc_write(tmem, BWD_DV_S, w, x);
                tmem_st_wait();
                bwd_wide_chunk(base, M.vec, tmem, fq, fk, P.scale, rev);
                sync();
                acc_read(tmem, BWD_DQ_S, w, dS);
                acc_read(tmem, BWD_DK_S, w, S);
                acc_read(tmem, BWD_DV_S, w, x);
                tmem_ld_wait();
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    qr[e] = __float_as_uint(x[e]);
                    kr[e] = __float_as_uint(x[8 + e]);
                }
            }
            const float half_decay = M.vec[row], eR = ex2(half_decay);
            bwd_put_split(r0, r1, row, u0, S, (wide ? 1.f : eR) * fS);
            bwd_put_split(r2, r3, row, u0, dS, (wide ? 1.f : eR) * fdS);
            hand_over(BWD_BAR_STATES);
            if (!wide) {
                acc_read(tmem, BWD_X, w, x);
                tmem_ld_wait();
                bwd_put_gated(tq, ql, row, u0, qr, x, kLog2e, bwd_log2(fq));
                bwd_put_gated(tk, kl, row, u0, kr, x, -kLog2e, bwd_log2(fk));
            }
            hand_over(BWD_BAR_GATED);
            // ---- within the chunk: P and dP, causal, as split operands
            wait_bar(P, M.bar_a, ph);
            tc_fence_after();
            if (!beyond) {
                float y[16];
                acc_read(tmem, BWD_P, w, x);
                acc_read(tmem, BWD_DP, w, y);                           // (of no use in a wide chunk)
                tmem_ld_wait();
                if (on_diagonal) {
                    const int lim = static_cast<int>(row) - static_cast<int>(c0);
#pragma unroll
                    for (int e = 0; e < 16; ++e) {
                        const bool keep = rev ? e >= lim : e <= lim;
                        x[e] = keep ? x[e] : 0.f;
                        y[e] = keep ? y[e] : 0.f;
                    }
                }
                bwd_put_split(r0, r1, row, u0, x, fp);                  // St has been read since bar_a, dSt will have with bar_s
                wait_bar(P, M.bar_s, ph);
                bwd_put_split(r2, r3, row, u0, y, fd);
            } else {
                const uint32_t z[8] = {0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
                put16(r0, row, u0, z); put16(r1, row, u0, z);
                wait_bar(P, M.bar_s, ph);
                put16(r2, row, u0, z); put16(r3, row, u0, z);
            }
            hand_over(BWD_BAR_SCORES);
            // ---- the state gradient moves to the chunk's start
            if (tid < 8) M.top[p ^ 1][tid] = 0u;
            acc_read(tmem, BWD_INC, w, x);
            tmem_ld_wait();
            {
                const float keep = eR * eR, c = (wide ? 1.f : eR) * P.scale * bwd_inverse(fq);
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    const float2 z = fma2(two(keep), pair_of(dS, e), mul2(two(c), pair_of(x, e)));
                    dS[2 * e] = z.x; dS[2 * e + 1] = z.y;
                }
            }
            const int tok = scan_token(P, P.T, (first + i) * kChunk + (rev ? 63 - static_cast<int>(row) : static_cast<int>(row)));
            const bool live = tok >= 0 && c0 < K;
            const long long at = (static_cast<long long>(b) * P.T + max(tok, 0)) * P.H + h;          // in units of one head's row
            wait_bar(P, M.bar_o, ph);
            tc_fence_after();
            // ---- outputs, read eight columns at a time, written as whole 32-byte sectors
            const int slot_dv = wide ? BWD_P : BWD_DP, slot_dk = wide ? BWD_DP : BWD_P;
            {
                float a[8], y[8], g[8], D[16];
                uint32_t o[8];
                // one of dk, dq: gate factor 2^(sign X) (in a wide chunk e^(G_L-G) or e^G, for the state part alone) times the sum of
                // state part and chunk part
                auto finish = [&](int slot_s, int slot_i, float cs, float ci, float sign, const uint32_t* in, __half* out) {
#pragma unroll
                    for (int hf = 0; hf < 2; ++hf) {
                        acc_read8(tmem, slot_s, w, 8 * hf, a);
                        acc_read8(tmem, slot_i, w, 8 * hf, y);
                        acc_read8(tmem, BWD_X, w, 8 * hf, g);
                        tmem_ld_wait();
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            float2 z;
                            if (!wide) {
                                z = fma2(two(cs), pair_of(a, e), mul2(two(ci), pair_of(y, e)));
                                z = mul2(z, ex2_2(mul2(pair_of(g, e), two(sign * kLog2e))));
                            } else {
                                auto factor = [&](int i) {                    // see the end of bwd_wide_chunk
                                    const bool after = (__float_as_uint(g[i]) & 1u) != 0u;
                                    return ex2(after == (sign < 0.f) ? g[i] : 2.f * M.vec[c0 + 8 * hf + i] - g[i]);
                                };
                                z = fma2(mul2(pair_of(a, e), two(cs)), make_float2(factor(2 * e), factor(2 * e + 1)), pair_of(y, e));
                            }
                            const int at2 = 4 * hf + e;
                            o[at2] = pack_half2(z.x, z.y);
                            const float2 f = unpack_half2(sign > 0.f ? in[at2] : in[at2] ^ 0x80008000u);
                            z = sign > 0.f ? fma2(f, z, pair_of(D, at2)) : mul2(f, z);
                            D[2 * at2] = z.x; D[2 * at2 + 1] = z.y;
                        }
                    }
                    if (live) put_row(out + at * K + c0, o);
                };
                finish(BWD_DK_S, slot_dk, bwd_inverse(fdS), P.scale * bwd_inverse(fd) * bwd_inverse(fq), -1.f, kr, P.dk);
                finish(BWD_DQ_S, BWD_DQ_I, P.scale * bwd_inverse(fS), P.scale * bwd_inverse(fd) * bwd_inverse(fk), 1.f, qr, P.dq);
                bwd_f32_put16(r0, row, c0, D);
                const float2 cs = two(bwd_inverse(fk) * bwd_inverse(fdS)), ci = two(P.scale * bwd_inverse(fq) * bwd_inverse(fk) * 8.f);      // 8 = 1 / fp
#pragma unroll
                for (int hf = 0; hf < 2; ++hf) {
                    acc_read8(tmem, BWD_DV_S, w, 8 * hf, a);
                    acc_read8(tmem, slot_dv, w, 8 * hf, y);
                    tmem_ld_wait();
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const float2 z = fma2(cs, pair_of(a, e), mul2(ci, pair_of(y, e)));
                        o[4 * hf + e] = pack_half2(z.x, z.y);
                    }
                }
                if (tok >= 0) put_row(P.dv + at * 64 + c0, o);
            }
            tc_fence_before();
            if (i > 0) named_bar_arrive(BWD_BAR_READ, kBwdChunkThreads);
            sync();
            // ---- dg: sums of the terms of the tokens at and after each token, a quarter of the rows per thread and channel, handed
            // back to the rows' owners in place
            {
                const uint32_t c = tid & 63u, q4 = static_cast<uint32_t>(tid) >> 6;
                float t[16], run = 0.f;
                if (!rev) {
#pragma unroll
                    for (int r = 15; r >= 0; --r) t[r] = run += ld_shared_f(bwd_f32(r0, 16u * q4 + r, c));
                } else {
#pragma unroll
                    for (int r = 0; r < 16; ++r) t[r] = run += ld_shared_f(bwd_f32(r0, 16u * q4 + r, c));
                }
                const uint32_t part = kl + 4u * c;                      // [4][64] sums of 16 rows
                asm volatile("st.shared.f32 [%0], %1;" ::"r"(part + 256u * q4), "f"(run) : "memory");
                sync();
                float add = later;
#pragma unroll
                for (uint32_t j = 0; j < 4; ++j) {
                    const float s = ld_shared_f(part + 256u * j);
                    add += (rev ? j < q4 : j > q4) ? s : 0.f;
                    later += s;
                }
#pragma unroll
                for (int r = 0; r < 16; ++r)
                    asm volatile("st.shared.f32 [%0], %1;" ::"r"(bwd_f32(r0, 16u * q4 + r, c)), "f"(t[r] + add) : "memory");
                sync();
                bwd_f32_row16(r0, row, c0, t);
                if (live) {
                    uint32_t o[8];
                    if (P.dg_half != nullptr) {
#pragma unroll
                        for (int e = 0; e < 8; ++e) o[e] = pack_half2(t[2 * e], t[2 * e + 1]);
                        put_row(P.dg_half + at * K + c0, o);
                    } else {
#pragma unroll
                        for (int m = 0; m < 2; ++m) {
#pragma unroll
                            for (int e = 0; e < 8; ++e) o[e] = __float_as_uint(t[8 * m + e]);
                            put_row(P.dg + at * K + c0 + 8 * m, o);
                        }
                    }
                }
            }
        }
        if (P.dh0 != nullptr && seg == 0 && real_row) {
            float4* dst = reinterpret_cast<float4*>(P.dh0 + state_off);
#pragma unroll
            for (int e = 0; e < 4; ++e) dst[e] = make_float4(dS[4 * e], dS[4 * e + 1], dS[4 * e + 2], dS[4 * e + 3]);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (w == 0) tmem_dealloc(tmem, 256);
}

}  // namespace gla
