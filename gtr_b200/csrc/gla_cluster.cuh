// The forward for a few short sequences: one launch, a thread-block cluster per sequence, every chunk on the way at once.
//
// What bounds such calls is not work but steps that wait for one another: the two kernels of gla_kernel.cuh pay two launches, load k, g and v
// and sum their gates twice, and each span reads the increments of all spans before it out of L2; the persistent kernel of gla_block.cuh walks four
// chunks twice and looks for its start state segment by segment.  Here a CTA has one to three chunks, four warps to each, and a sequence's
// CTAs are a cluster that exchanges states through its shared memories:
//   1. every chunk by itself: gate sums, gated operands, its state increment k~^T v (as in gla_kernel.cuh)
//   2. each CTA owns some rows of the 64 x 64 state: increments and decays are sent to the owners of their rows
//   3. an owner walks its rows through all chunks in registers and sends every chunk its rows of the fp16 start state; before that the
//      chunks' scores are made, while increments are on their way
//   4. outputs
// What is sent goes by bulk copies (factors by st.async) whose bytes the receiver's barriers count; a cluster barrier opens and one closes the exchange.
//
// B1 H6 T1600 14.1 -> 7.9 us, B3 H3 T1050 K = 32 with states 15.9 -> 8.9, the block's call at B1 H3 T1600 28 -> 11.4 (and no launch that clears flags).  Of some 11
// thousand cycles after the predecessor has ended (one image) 1.4 pass until the tiles are there, 0.5 for gate sums, 0.6 for k~, 2.0 until the increment
// is there (q~ meanwhile), 2.4 until all have arrived (scores meanwhile), 1.5 for the walk, 1.5 until the start state is there, 1.4 for the outputs.
// Tried on the way: increments and start states by plain stores to the other CTAs (16 bytes a lane, rows apart: 10 bytes a cycle; 8.6 us), start states by
// st.async (a barrier update for every lane's 8 bytes: 8.0) or by stores and a releasing arrival (8.8), copies sent by one warp (8.9), increments staged
// apart from k so that they leave before q~ and the scores (7.4 against 7.3, row order), tiles asked for by four warps (columns 0.1 better, rows 0.1 worse).
//
// kBlock: the arithmetic of the persistent kernel, to the bit, for the backbone's blocks (gla_block.cuh has the reason).  A sequence has the
// equal segments of that kernel's plan: increments in the form of its pre-pass (k 2^(G_L-G)) are summed to a segment's aggregate, its start state is chained
// from those before it, and within it the state goes on in the scale of the next chunk's reference; segments times rows are walked side by side, by twelve
// warps whatever the chunks (with four to a chunk B2 H3 T1024 took 9.8 us, 9.2).  That kernel adds up aggregates down to the first segment whose
// inclusive state happens to be there; here always down to the first segment.
#pragma once

#include "gla_kernel.cuh"

namespace gla {

constexpr int kClusterGroups = 3;                          // chunks per CTA, at most
constexpr int kClusterThreads = kFwdThreads * kClusterGroups;
constexpr int kClusterMax = 16;                            // CTAs per cluster, at most (more than eight have to be asked for)

struct ClusterPlan {
    int size, groups;    // CTAs per sequence, chunks per CTA
    int rows;            // rows of the state that a CTA owns
    int round;           // chunks at a time: all, or as many as the cluster holds
    int ns, cps;         // kBlock: segments, chunks per segment
};

struct ClusterSmem {
    // of each chunk: q, k, g, v as in OutSmem, its start state (until then the pre-pass's form of k and the exact path's scores), the scores; the increment on its way
    // to the owners takes the place of k and g, the one in the pre-pass's form has a place of its own
    static constexpr int kA = 5 * kTileBytes, kInc = OutSmem::kK, kIncA = 6 * kTileBytes;
    static_assert(OutSmem::kG == OutSmem::kK + kTileBytes, "an increment is fp32");
    static constexpr int kMiscBytes = 3 * 1024;
    int group, mat, in_u, in_a, in_f, misc, bytes;
    __host__ __device__ ClusterSmem(bool block, int groups, int NT, int rows) {
        group = (block ? 8 : 6) * kTileBytes;
        mat = groups * group;
        const int starts = (NT * rows * 128 + 1023) / 1024 * 1024, mats = (block ? 2 : 1) * kTileBytes;
        misc = mat + (starts > mats ? starts : mats);      // [chunk][row] start states, in the place of the matrices
        in_u = misc + kMiscBytes;                          // [chunk][row][64] increments
        in_a = in_u + NT * rows * 256;                     // increments in the pre-pass's form
        in_f = in_a + (block ? NT * rows * 256 : 0);       // [chunk][row] factors
        bytes = in_f + NT * rows * 16 + 1024;              // + alignment
    }
};
struct ClusterMisc {
    uint64_t full[kClusterGroups], raw[kClusterGroups], again[kClusterGroups], bar_x[kClusterGroups], bar_inc[kClusterGroups], bar_p[kClusterGroups], bar_a[kClusterGroups],
        bar_o[kClusterGroups], start[kClusterGroups], inbox;
    uint32_t tmem, gave_up;
    uint32_t wide[kClusterGroups];
    alignas(16) float vec[kClusterGroups][64];             // log2: half the chunk's total decay per channel
    alignas(16) float gl[kClusterGroups][64];              // log2: all of it, from the pre-pass's sums
    CausalMasks causal;
    alignas(16) uint32_t weight[kClusterGroups][32];
};
static_assert(sizeof(ClusterMisc) <= ClusterSmem::kMiscBytes, "misc block too large");

__device__ __forceinline__ uint32_t cluster_address(uint32_t a, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
// from this CTA's shared memory to another's, whose barrier counts the bytes
__device__ __forceinline__ void cluster_copy(uint32_t dst, uint32_t src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst), "r"(src), "r"(bytes), "r"(bar) : "memory");
}
// 16 bytes of registers likewise
__device__ __forceinline__ void cluster_send(uint32_t dst, float x, float y, float z, float w, uint32_t bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];"
                 ::"r"(dst), "f"(x), "f"(y), "f"(z), "f"(w), "r"(bar) : "memory");
}
// by whole warps: lanes that have left a wait one after the other come together first
__device__ __forceinline__ void cluster_arrive() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_arrive_relaxed() {       // no writes to be seen
    __syncwarp();
    asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
    __syncwarp();
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float2 ld_shared_f2(uint32_t a) {
    float2 v;
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ void st_shared_f2(uint32_t a, float2 v) {
    asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(a), "f"(v.x), "f"(v.y) : "memory");
}
// logits_to_log_gates with the persistent kernel's rounding: the normaliser divides the rounded log sigmoid
__device__ __forceinline__ void block_log_gates(const HalfRow& at, uint32_t tile, float inv_norm, bool real_row) {
    uint32_t r[16];
    at.get(tile, r);
#pragma unroll
    for (int e = 0; e < 16; ++e) {
        const float2 n = mul2(unpack_half2(r[e] & 0x7fff7fffu), two(-kLog2e));
        const float2 lg = make_float2(lg2(1.f + ex2(n.x)), lg2(1.f + ex2(n.y)));
        const float2 v = mul2(fma2(lg, two(-0.6931471805599453f), unpack_half2(hmin2_zero(r[e]))), two(inv_norm));
        r[e] = real_row ? pack_half2_sat(v.x, v.y) : 0u;
    }
    at.put(tile, r);
    fence_proxy_async_smem();
}

// The four warps of a chunk.  (A barrier's number in a register makes a block reserve all sixteen, which leaves room for no second block on the SM.)
__device__ __forceinline__ void group_sync(int grp) {
    if (grp == 0) named_bar_sync(1, kFwdThreads);
    else if (grp == 1) named_bar_sync(2, kFwdThreads);
    else named_bar_sync(3, kFwdThreads);
}
__device__ __forceinline__ bool group_or(int grp, bool x) {
    return grp == 0 ? named_bar_or<1>(kFwdThreads, x) : grp == 1 ? named_bar_or<2>(kFwdThreads, x) : named_bar_or<3>(kFwdThreads, x);
}

template <bool kGated, bool kLogits, bool kBlock, bool kRounds>
__global__ void __launch_bounds__(kClusterThreads) gla_cluster_kernel(const __grid_constant__ Maps maps, const __grid_constant__ Params P,
                                                                      const __grid_constant__ ClusterPlan C) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw), base = (raw + 1023u) & ~1023u;
    const ClusterSmem lay(kBlock, C.groups, kRounds ? C.round : P.NT, C.rows);
    ClusterMisc& M = *reinterpret_cast<ClusterMisc*>(smem_raw + (base - raw) + lay.misc);
    const int tid = threadIdx.x, grp = __shfl_sync(0xffffffffu, tid >> 7, 0), w = __shfl_sync(0xffffffffu, (tid >> 5) & 3, 0), l = tid & 31;
    const int seq = blockIdx.x / C.size, rank = blockIdx.x - seq * C.size, b = seq / P.H, h = seq - b * P.H;
    const int place = rank * C.groups + grp;               // the group's chunk in every round
    const bool mine_first = grp < C.groups && place < P.NT, rev = P.rev != 0;      // (warps beyond the groups help with the walk)
    const uint32_t own = base + grp * lay.group, tq = own + OutSmem::kQ, tk = own + OutSmem::kK, tg = own + OutSmem::kG, tv = own + OutSmem::kV,
                   s16 = own + OutSmem::kS16, ta = own + ClusterSmem::kA, mat = base + lay.mat;
    const int first = rank * C.rows, owned = max(min(C.rows, 64 - first), 0);       // rows of the state
    auto wait = [&](uint64_t& bar, uint32_t parity) { wait_bar(P, bar, parity, M.gave_up); };
    auto sync = [&] { group_sync(grp); };
    if (tid == 0) {
        for (int i = 0; i < kClusterGroups; ++i)
            for (uint64_t* bar : {M.full, M.raw, M.again, M.bar_x, M.bar_inc, M.bar_p, M.bar_a, M.bar_o}) mbar_init(smem_u32(bar + i), 1);
        for (int i = 0; i < kClusterGroups; ++i) mbar_init(smem_u32(&M.start[i]), 1);
        mbar_init(smem_u32(&M.inbox), 1);
        fence_mbar_init();
        for (int i = 0; i < kClusterGroups; ++i) mbar_arrive_expect_tx(smem_u32(&M.start[i]), kTileBytes);
        mbar_arrive_expect_tx(smem_u32(&M.inbox), owned * ((kRounds ? C.round : P.NT) * 272 + (kBlock ? (C.ns - 1) * C.cps * 256 : 0)));
        M.gave_up = 0u;
    }
    fill_constant(mat, [&](uint32_t r, uint32_t s) { return (rev ? s >= r : s <= r) ? 0.5f : -0.5f; });        // G - G_L / 2
    if (kBlock) fill_constant(mat + kTileBytes, [&](uint32_t r, uint32_t s) { return (rev ? s >= r : s <= r) ? 0.f : -1.f; });       // G - G_L
    M.causal.fill(rev);
    fence_proxy_async_smem();
    __syncthreads();
    cluster_arrive();                                       // nothing is sent to a CTA that has not begun
    pdl_wait();
    if (blockIdx.x == 0 && tid == 0) clear_alone(P.ctrl, P.clear);
    auto load = [&](int chunk) {
        const int tensors[4] = {TG, TK, TQ, TV};
        const uint32_t tiles[4] = {tg, tk, tq, tv};
        mbar_arrive_expect_tx(smem_u32(&M.full[grp]), 4 * kTileBytes);
        load_chunk(maps, Scan{P.T, P.Hc, P.rev}, chunk, b, h, 0, P.Hc, smem_u32(&M.full[grp]), tensors, tiles, l2_policy_stream());
    };
    if (mine_first && w == 0 && elect_one()) load(place);
    // (another kernel's blocks may not have their tensor memory before this one waits for them)
    const uint32_t columns = C.groups == 3 ? 512u : 128u * C.groups;
    if (tid >= 32 && tid < 64) {
        tmem_alloc(smem_u32(&M.tmem), columns);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = M.tmem + 128u * grp;
    pdl_release();

    const uint32_t half = static_cast<uint32_t>(l) >> 4, row = 16u * w + (l & 15u), c0 = 32u * half;
    const HalfRow at(own, row, half);
    const float hk = 0.5f * P.q_exp, hq = P.q_exp - hk;     // k's and q's share of the output scale (log2)
    // kRounds: a sequence longer than the cluster holds goes in rounds.  The owners keep their rows of the state, a chunk's tiles come in when its place is done
    // with the last ones, a cluster barrier lies between, and each barrier is used once a round.
    uint32_t raws = 0, agains = 0, ps = 0;                  // how often their barriers have been used
    float4 carry = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int at0 = 0, turn = 0;; at0 += C.round, ++turn) {
    const uint32_t ph = kRounds ? turn & 1 : 0;
    const int NT = kRounds ? min(C.round, P.NT - at0) : P.NT, chunk = kRounds ? at0 + place : place, left = kRounds ? P.NT - at0 - NT : 0;      // left: for later rounds
    const bool live = grp < C.groups && place < NT, opening = !kRounds || turn == 0;
    const int tok = live ? scan_token(P, P.T, chunk * kChunk + (rev ? 63 - static_cast<int>(row) : static_cast<int>(row))) : -1;
    const __half* gate_row_at = P.gate;
    __half* const op = P.o + b * P.o_s[0] + max(tok, 0) * P.o_s[1] + h * P.o_s[2] + c0;
    uint32_t weight = 0u;
    if (kGated && w == 0 && opening) weight = __ldg(reinterpret_cast<const uint32_t*>(P.rms_w) + l);
    uint32_t r[16];
    float x[32];
    if (live) {
        if (kGated && tok >= 0) {
            gate_row_at = P.gate + b * P.gate_s[0] + tok * P.gate_s[1] + h * P.gate_s[2] + c0;
            prefetch_l2(gate_row_at);
        }
        const bool pre = kBlock && chunk < (C.ns - 1) * C.cps;       // the chunk's segment has an aggregate
        // ---- gate sums, gated operands
        wait(M.full[grp], ph);
        if (kLogits) {
            if (kBlock) block_log_gates(at, OutSmem::kG, P.inv_norm, tok >= 0);
            else logits_to_log_gates(at, OutSmem::kG, P.inv_norm, tok >= 0);
            sync();
        }
        if (w == 0 && elect_one()) {
            tc_fence_after();
            tile_mma<0, 1>(acc_slot(tmem, ACC_X), mat, tg, false);
            if (pre) tile_mma<0, 1>(acc_slot(tmem, ACC_S), mat + kTileBytes, tg, false);
            umma_commit(smem_u32(&M.bar_x[grp]));
        }
        __syncwarp();
        uint32_t k[16];
        at.get(OutSmem::kK, k);
        if (kGated && w == 0 && opening) M.weight[grp][l] = weight;
        wait(M.bar_x[grp], ph);
        tc_fence_after();
        if (kBlock && pre) {
            half_row_read(tmem, ACC_S, w, x);
            tmem_ld_wait();
            if (row == (rev ? 63u : 0u)) {                  // the first row along the scan: G_L = own gate - x
                at.get(OutSmem::kG, r);
#pragma unroll
                for (int e = 0; e < 16; ++e) {
                    const float2 gf = unpack_half2(r[e]);
                    M.gl[grp][c0 + 2 * e] = (gf.x - x[2 * e]) * kLog2e;
                    M.gl[grp][c0 + 2 * e + 1] = (gf.y - x[2 * e + 1]) * kLog2e;
                }
            }
#pragma unroll
            for (int e = 0; e < 16; ++e) {
                const float2 f = ex2_2(mul2(pair_of(x, e), two(-kLog2e)));
                r[e] = hmul2_u32(k[e], pack_half2(f.x, f.y));
            }
            at.put(OutSmem::kS16, r);
        }
        half_row_read(tmem, ACC_X, w, x);
        tmem_ld_wait();
        if (w == (rev ? 0 : 3)) {                           // the warp that holds the last row: X there is G_L / 2
            bool far = false;
            if (row == (rev ? 0u : 63u)) {
                float least = 0.f;
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    const float2 a = mul2(pair_of(x, 2 * e), two(kLog2e)), c = mul2(pair_of(x, 2 * e + 1), two(kLog2e));
                    *reinterpret_cast<float4*>(&M.vec[grp][c0 + 4 * e]) = make_float4(a.x, a.y, c.x, c.y);
                    least = fminf(least, fminf(fminf(a.x, a.y), fminf(c.x, c.y)));
                }
                far = least < -kRefLimit;
            }
            far = __any_sync(0xffffffffu, far);
            if (l == 0) M.wide[grp] = far ? 1u : 0u;
        }
        auto gate_row = [&](uint32_t* v, uint32_t tile, float sign, float add) {
#pragma unroll
            for (int e = 0; e < 16; ++e) {
                const float2 f = ex2_2(fma2(pair_of(x, e), two(sign * kLog2e), two(add)));
                v[e] = hmul2_u32(v[e], pack_half2(f.x, f.y));
            }
            at.put(tile, v);
        };
        gate_row(k, OutSmem::kK, -1.f, hk);
        fence_proxy_async_smem();
        tc_fence_before();
        sync();
        const bool wide = M.wide[grp] != 0u;
        if (kBlock && pre && w == 0 && elect_one()) {
            tc_fence_after();
            tile_mma<1, 1>(acc_slot(tmem, ACC_S), s16, tv, false);
            umma_commit(smem_u32(&M.bar_a[grp]));
        }
        if (wide) {                                         // see gla_out_kernel
            if (kBlock && pre) wait(M.bar_a[grp], 0);       // the scores go where its operand is
            if (w == 0 && elect_one()) {                    // the raw q and k once more
                const int tensors[2] = {TK, TQ};
                const uint32_t tiles[2] = {tk, tq};
                mbar_arrive_expect_tx(smem_u32(&M.raw[grp]), 2 * kTileBytes);
                load_chunk(maps, Scan{P.T, P.Hc, P.rev}, chunk, b, h, 0, P.Hc, smem_u32(&M.raw[grp]), tensors, tiles, l2_policy_stream());
            }
            __syncwarp();
            wait(M.raw[grp], raws++ & 1u);
            if (group_or(grp, !(M.vec[grp][tid & 63] > -kExtreme))) {
                at.get(OutSmem::kG, r);
#pragma unroll
                for (int e = 0; e < 16; ++e) r[e] = hmax2_nan(r[e], kHardest);
                at.put(OutSmem::kG, r);
                fence_proxy_async_smem();
                tc_fence_before();
                sync();
                if (w == 0 && elect_one()) {
                    tc_fence_after();
                    tile_mma<0, 1>(acc_slot(tmem, ACC_X), mat, tg, false);
                    umma_commit(smem_u32(&M.again[grp]));
                }
                __syncwarp();
                wait(M.again[grp], agains++ & 1u);
                tc_fence_after();
                half_row_read(tmem, ACC_X, w, x);
                tmem_ld_wait();
                if (row == (rev ? 0u : 63u)) {
#pragma unroll
                    for (int e = 0; e < 32; ++e) M.vec[grp][c0 + e] = x[e] * kLog2e;
                }
                sync();
            }
            gate_wide_chunk(own, ClusterSmem::kA, M.vec[grp], tmem, rev, P.q_exp, P.q_mul, tid & (kFwdThreads - 1), sync);
            fence_proxy_async_smem();
            tc_fence_before();
            sync();
        }
        if (w == 0 && elect_one()) {
            tc_fence_after();
            tile_mma<1, 1>(acc_slot(tmem, ACC_INC), tk, tv, false);
            umma_commit(smem_u32(&M.bar_inc[grp]));
        }
        __syncwarp();
        if (!wide) {                                        // q~ while the increment is made
            at.get(OutSmem::kQ, r);
            gate_row(r, OutSmem::kQ, 1.f, hq);
            fence_proxy_async_smem();
            sync();
            if (w == 0 && elect_one()) {
                tile_mma<0, 0>(acc_slot(tmem, ACC_P), tq, tk, false);
                umma_commit(smem_u32(&M.bar_p[grp]));
            }
            __syncwarp();
        }
        // ---- the chunk's increment and decay, to the owners of their rows
        const float v = M.vec[grp][row];
        auto stage = [&](uint32_t to) {
#pragma unroll
            for (uint32_t e = 0; e < 8; ++e)
                st_shared_f4(own + to + row * 256u + half * 128u + ((e ^ (row & 7u)) << 4), x[4 * e], x[4 * e + 1], x[4 * e + 2], x[4 * e + 3]);
        };
        if (opening) cluster_wait();                        // every CTA has begun
        auto copy = [&](uint32_t from, int inbox) {         // a lane has an owner, a warp every fourth (a lane's copy goes out after another's)
            const int who = w + 4 * l, at_row = who * C.rows, n = min(C.rows, 64 - at_row);
            if (who < C.size && n > 0)
                cluster_copy(cluster_address(base + inbox + place * C.rows * 256, who), own + from + at_row * 256, n * 256, cluster_address(smem_u32(&M.inbox), who));
            __syncwarp();
        };
        if (half == 0u) {
            const uint32_t who = row / static_cast<uint32_t>(C.rows), to = cluster_address(base + lay.in_f + (place * C.rows + row - who * C.rows) * 16u, who),
                           bar = cluster_address(smem_u32(&M.inbox), who);
            if (kBlock) cluster_send(to, v, pre ? M.gl[grp][row] : 0.f, wide ? 1.f : 0.f, 0.f, bar);
            else cluster_send(to, ex2(2.f * v), ex2(wide ? hk : v + hk), 0.f, 0.f, bar);
        }
        __syncwarp();
        if (kBlock && pre) {
            wait(M.bar_a[grp], 0);
            tc_fence_after();
            half_row_read(tmem, ACC_S, w, x);
            tmem_ld_wait();
            stage(ClusterSmem::kIncA);
            fence_proxy_async_smem();
            sync();
            copy(ClusterSmem::kIncA, lay.in_a);
        }
        wait(M.bar_inc[grp], ph);
        tc_fence_after();
        half_row_read(tmem, ACC_INC, w, x);
        tmem_ld_wait();
        if (!kBlock) {
            const float c = ex2(wide ? -hk : v - hk);
#pragma unroll
            for (int e = 0; e < 16; ++e) {
                const float2 u = mul2(two(c), pair_of(x, e));
                x[2 * e] = u.x; x[2 * e + 1] = u.y;
            }
        }
        if (!wide) wait(M.bar_p[grp], ps++ & 1u);           // k~ has been read
        stage(ClusterSmem::kInc);
        fence_proxy_async_smem();
        sync();
        copy(ClusterSmem::kInc, lay.in_u);
        // ---- meanwhile the scores: causal, as an fp16 tile, and their share of the outputs
        if (!wide) {
            half_row_read(tmem, ACC_P, w, x);
            tmem_ld_wait();
            CausalRow(M.causal, w, l, rev).mask(w, x, r);
            at.put(ClusterSmem::kA, r);
        }
        fence_proxy_async_smem();
        tc_fence_before();
        sync();
        if (w == 0 && elect_one()) {
            tc_fence_after();
            tile_mma<0, 1>(acc_slot(tmem, ACC_P), ta, tv, false);
        }
        __syncwarp();
    } else if (opening) {
        cluster_wait();
    }
    wait(M.inbox, ph);

    // ---- the owned rows through all chunks, four columns a thread; 16 lanes have a row
    const int mine = owned * 16;
    const uint32_t step = C.rows * 256u;                    // from a chunk's increments to the next one's
    uint32_t srow, inc, to;                                 // of a unit: row of the state, its increments, its place in a chunk's start state
    size_t state_at;
    auto unit = [&](int u) {
        const uint32_t pos = u >> 4, j = u & 15, col = 4u * j;
        srow = first + pos;
        inc = base + lay.in_u + pos * 256u + (((j & 7u) ^ (srow & 7u)) << 4) + ((j & 8u) << 4);
        to = mat + pos * 128u + (sw_f16(srow, col) & 127u);         // (every chunk of this CTA has its gate sums)
        state_at = (static_cast<size_t>(seq) * P.K + srow) * kD + col;
    };
    auto give = [&](int c, float4 s) {                      // a piece of a start state
        asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(to + c * C.rows * 128u), "r"(pack_half2(s.x, s.y)), "r"(pack_half2(s.z, s.w)) : "memory");
    };
    auto initial = [&] {
        return P.s0 != nullptr && srow < static_cast<uint32_t>(P.K) ? __ldg(reinterpret_cast<const float4*>(P.s0 + state_at)) : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    auto final = [&](float4 s) {
        if (P.sT != nullptr && srow < static_cast<uint32_t>(P.K)) *reinterpret_cast<float4*>(P.sT + state_at) = s;
    };
    auto times = [](float f, float4 a) {
        const float2 x = mul2(two(f), make_float2(a.x, a.y)), y = mul2(two(f), make_float2(a.z, a.w));
        return make_float4(x.x, x.y, y.x, y.y);
    };
    auto plus = [](float f, float4 a, float4 c) {           // f a + c
        const float2 x = fma2(two(f), make_float2(a.x, a.y), make_float2(c.x, c.y)), y = fma2(two(f), make_float2(a.z, a.w), make_float2(c.z, c.w));
        return make_float4(x.x, x.y, y.x, y.y);
    };
    constexpr int kAhead = 5;                               // chunks whose loads go ahead together
    if (!kBlock) {
        for (int u = tid; u < mine; u += blockDim.x) {
            unit(u);
            const uint32_t fac = base + lay.in_f + (u >> 4) * 16u, fac_step = C.rows * 16u;
            float4 S = opening ? initial() : carry;
            for (int c0 = 0; c0 < NT; c0 += kAhead) {
                float2 f[kAhead];
                float4 d[kAhead];
#pragma unroll
                for (int i = 0; i < kAhead; ++i)
                    if (c0 + i < NT) {
                        f[i] = ld_shared_f2(fac + (c0 + i) * fac_step);
                        d[i] = ld_shared_f4(inc + (c0 + i) * step);
                    }
#pragma unroll
                for (int i = 0; i < kAhead; ++i)
                    if (c0 + i < NT) {
                        give(c0 + i, times(f[i].y, S));
                        S = plus(f[i].x, S, d[i]);
                    }
            }
            if (kRounds && left > 0) carry = S;             // (a row's unit a thread, then)
            else final(S);
        }
    } else {
        // segments times units, a warp always in one segment (what is left over of it does the last unit again)
        const uint32_t agg_at = lay.in_a - lay.in_u, fac_step = C.rows * 16u;
        const int across = (mine + 31) >> 5, warps = blockDim.x >> 5;
        auto pairs = [&](int segments, auto work) {
            if (mine == 0) return;
            int s = 0, at_warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
            while (true) {
                while (at_warp >= across) { at_warp -= across; ++s; }
                if (s >= segments) break;
                const int u = min(32 * at_warp + l, mine - 1);
                unit(u);
                work(s, base + lay.in_f + 16u * (u >> 4) + s * C.cps * fac_step);
                at_warp += warps;
            }
        };
        // the aggregates, each left with its segment's first chunk, and what the segment decays by
        pairs(C.ns - 1, [&](int s, uint32_t fac) {
            const uint32_t at = inc + agg_at + s * C.cps * step;
            float4 A = make_float4(0.f, 0.f, 0.f, 0.f);
            float sum = 0.f;
            for (int c0 = C.cps - 1; c0 >= 0; c0 -= kAhead) {
                float f[kAhead];
                float4 d[kAhead];
#pragma unroll
                for (int i = 0; i < kAhead; ++i)
                    if (c0 >= i) {
                        f[i] = ld_shared_f(fac + (c0 - i) * fac_step + 4u);
                        d[i] = ld_shared_f4(at + (c0 - i) * step);
                    }
#pragma unroll
                for (int i = 0; i < kAhead; ++i)
                    if (c0 >= i) {
                        const float4 t = times(ex2(sum), d[i]);
                        A = make_float4(__fadd_rn(A.x, t.x), __fadd_rn(A.y, t.y), __fadd_rn(A.z, t.z), __fadd_rn(A.w, t.w));       // two roundings: not one multiply-add
                        sum += f[i];
                    }
            }
            if (s == 0 && P.s0 != nullptr) A = plus(ex2(sum), initial(), A);
            st_shared_f4(at, A.x, A.y, A.z, A.w);
            st_shared_f(fac + 12u, sum);
        });
        __syncthreads();
        pairs(C.ns, [&](int s, uint32_t fac) {
            float4 S = s == 0 ? initial() : make_float4(0.f, 0.f, 0.f, 0.f);
            float dlog = 0.f;
            for (int s0 = s - 1; s0 >= 0; s0 -= kAhead) {
                float f[kAhead];
                float4 d[kAhead];
#pragma unroll
                for (int i = 0; i < kAhead; ++i)
                    if (s0 >= i) {
                        f[i] = ld_shared_f(fac + (s0 - i - s) * C.cps * fac_step + 12u);
                        d[i] = ld_shared_f4(inc + agg_at + (s0 - i) * C.cps * step);
                    }
#pragma unroll
                for (int i = 0; i < kAhead; ++i)
                    if (s0 >= i) {
                        S = plus(ex2(dlog), d[i], S);
                        dlog += f[i];
                    }
            }
            const int from = s * C.cps, n = min(C.cps, P.NT - from);
            auto reference = [&](float4 f) { return f.z != 0.f ? hk : f.x + hk; };
            float4 f = ld_shared_f4(fac);
            S = times(ex2(reference(f)), S);
            for (int c0 = 0; c0 < n; c0 += kAhead) {
                float4 next[kAhead], d[kAhead];
#pragma unroll
                for (int i = 0; i < kAhead; ++i)
                    if (c0 + i < n) {
                        if (c0 + i + 1 < n) next[i] = ld_shared_f4(fac + (c0 + i + 1) * fac_step);
                        d[i] = ld_shared_f4(inc + (from + c0 + i) * step);
                    }
#pragma unroll
                for (int i = 0; i < kAhead; ++i)
                    if (c0 + i < n) {
                        give(from + c0 + i, S);
                        const bool wide = f.z != 0.f;
                        const float rq = c0 + i + 1 < n ? reference(next[i]) : 0.f;
                        const float ta = wide ? 2.f * f.x - hk : f.x - hk, tb = wide ? -hk : f.x - hk;
                        S = plus(ex2(rq + ta), S, times(ex2(rq + tb), d[i]));
                        f = next[i];
                    }
            }
            if (s == C.ns - 1) final(S);
        });
    }
    fence_proxy_async_smem();
    __syncthreads();
    if (kRounds && left > 0 && tid == 0) mbar_arrive_expect_tx(smem_u32(&M.inbox), owned * min(C.round, left) * 272);
    {
        const int warps = blockDim.x >> 5, c = (tid >> 5) + warps * l, who = c / C.groups, g = c - who * C.groups;
        static_assert(kClusterMax * kClusterGroups <= 32 * 4, "a lane for every chunk");
        if (c < NT && owned > 0)
            cluster_copy(cluster_address(base + g * lay.group + OutSmem::kS16 + first * 128, who), mat + c * C.rows * 128, owned * 128,
                         cluster_address(smem_u32(&M.start[g]), who));
        __syncwarp();
    }
    uint4 gate[4];
    if (kGated && tok >= 0) {
        const uint4* gp = reinterpret_cast<const uint4*>(gate_row_at);
#pragma unroll
        for (int m = 0; m < 4; ++m) gate[m] = __ldg(gp + m);
    }

    // ---- outputs
    if (live) {
        if (w == 0) {
            wait(M.start[grp], ph);
            if (elect_one()) {
                if (kRounds && place < left) mbar_arrive_expect_tx(smem_u32(&M.start[grp]), kTileBytes);
                tc_fence_after();
                tile_mma<0, 1>(acc_slot(tmem, ACC_P), tq, s16, true);
                umma_commit(smem_u32(&M.bar_o[grp]));
            }
            __syncwarp();
        }
        wait(M.bar_o[grp], ph);
        if (kRounds) cluster_arrive();
        else cluster_arrive_relaxed();                      // every owner has what this chunk sent, and this chunk what they sent
        if (kRounds && place < left && w == 0) {
            if (elect_one()) load(chunk + C.round);
            __syncwarp();
        }
        tc_fence_after();
        half_row_read(tmem, ACC_P, w, x);
        tmem_ld_wait();
        float mul = P.o_mul;
        if (kGated) {
            // y = o * rsqrt(mean(o^2) + eps) * w * silu(gate): the two lanes of a row share its sum of squares
            float2 s2[2] = {two(0.f), two(0.f)};
#pragma unroll
            for (int e = 0; e < 16; ++e) s2[e & 1] = fma2(pair_of(x, e), pair_of(x, e), s2[e & 1]);
            float ss = (s2[0].x + s2[0].y) + (s2[1].x + s2[1].y);
            ss += __shfl_xor_sync(0xffffffffu, ss, 16);
            mul *= rsqrtf(ss * (P.o_mul * P.o_mul) * (1.f / kD) + P.rms_eps);
        }
        if (tok >= 0) {
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                uint4 wv = make_uint4(0u, 0u, 0u, 0u);
                if (kGated) wv = ld_shared_v4(smem_u32(M.weight[grp]) + 2u * c0 + 16u * m);
                const uint32_t gu[4] = {gate[m].x, gate[m].y, gate[m].z, gate[m].w}, wu[4] = {wv.x, wv.y, wv.z, wv.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    float2 y = pair_of(x + 8 * m, e);
                    if (kGated) {
                        const float2 hg = mul2(unpack_half2(gu[e]), two(0.5f)), silu = fma2(hg, tanh_2(hg), hg);             // silu = h + h tanh h
                        if (kBlock) y = mul2(y, mul2(mul2(two(mul), unpack_half2(wu[e])), silu));
                        else y = mul2(mul2(mul2(y, two(mul)), unpack_half2(wu[e])), silu);
                    } else {
                        y = mul2(y, two(mul));
                    }
                    r[4 * m + e] = pack_half2(y.x, y.y);
                }
            }
            if (P.sectors) {
                st_global_v8(op, r);
                st_global_v8(op + 16, r + 8);
            } else {
#pragma unroll
                for (int m = 0; m < 4; ++m) reinterpret_cast<uint4*>(op)[m] = make_uint4(r[4 * m], r[4 * m + 1], r[4 * m + 2], r[4 * m + 3]);
            }
        }
    } else if (kRounds) {
        cluster_arrive();
    } else {
        cluster_arrive_relaxed();
    }
    tc_fence_before();
    __syncthreads();
    cluster_wait();                                         // nothing is read from this CTA any more
    if (!kRounds || left == 0) break;
    fill_constant(mat, [&](uint32_t r, uint32_t s) { return (rev ? s >= r : s <= r) ? 0.5f : -0.5f; });        // where start states were
    fence_proxy_async_smem();
    __syncthreads();
    tc_fence_after();
    }
    if (tid == 0) {
        if (M.gave_up) report_alone(P, P.clear);
        if (blockIdx.x == 0) P.ctrl[0] = 0u;
    }
    if (tid >= 32 && tid < 64) tmem_dealloc(M.tmem, columns);
}

}  // namespace gla
