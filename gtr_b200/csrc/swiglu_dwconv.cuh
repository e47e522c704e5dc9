// Spatial SwiGLU middle step in one pass over memory:
//     out[b, r, c, :] = silu(gate[b, r, c, :]) * (bias + sum_{dr,dc in -1..1} w[dr, dc, :] * y[b, r+dr, c+dc, :])
// on tokens kept in their [B, L = hg*wg, C] layout (zero padding at the grid border).  Replaces, for the deploy
// form of the reference's SpatialSwiGLU (engine/gtr/backbone/vit_adapter_spatial_swiglu.py:50-60), the chain
// view/permute -> cuDNN depthwise 3x3 conv -> permute/reshape -> silu -> multiply and the layout copies around it.
//
// HBM-bound: gate and y are read once, out is written once (3 * 2 bytes per element).
#pragma once

#include <cuda_fp16.h>
#include <cstdint>

#include "gla_device.cuh"

namespace gla {

__device__ __forceinline__ void dw_unpack8(const uint4& v, float* x) {
    const __half2* h = reinterpret_cast<const __half2*>(&v);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 f = __half22float2(h[i]);
        x[2 * i] = f.x;
        x[2 * i + 1] = f.y;
    }
}

// to[0..7] = w[0..7] * y[0..7] + from[0..7] with the fp16 operands taken as they are: fma.rn.f32.f16 multiplies two fp16 values
// and accumulates in fp32 in one instruction (exact product, one rounding), so the taps cost no conversions.
__device__ __forceinline__ void dw_fma2(float* to, uint32_t w, uint32_t y, const float* from) {
    asm("{\n\t.reg .b16 wl, wh, yl, yh;\n\t"
        "mov.b32 {wl, wh}, %2;\n\tmov.b32 {yl, yh}, %3;\n\t"
        "fma.rn.f32.f16 %0, wl, yl, %4;\n\tfma.rn.f32.f16 %1, wh, yh, %5;\n\t}"
        : "=f"(to[0]), "=f"(to[1])
        : "r"(w), "r"(y), "f"(from[0]), "f"(from[1]));
}
__device__ __forceinline__ void dw_fma8(float* to, const uint4& wv, const uint4& yv, const float* from) {
    dw_fma2(to, wv.x, yv.x, from);
    dw_fma2(to + 2, wv.y, yv.y, from + 2);
    dw_fma2(to + 4, wv.z, yv.z, from + 4);
    dw_fma2(to + 6, wv.w, yv.w, from + 6);
}

// A CTA per SM with a ring of three stages.  A stage holds, for a slab of 64 channels, a y tile of up to 256 outputs (16 x 16 where
// the grid is a multiple of that; of several images where one tile takes a whole grid) plus its one-cell halo, the gate tile, and the slab's weights and bias, filled by four
// TMA copies (cells outside the grid and channels past C read as zero), so that 150 KB per SM are in flight while 16
// warps work on a stage.  Neighbouring blocks are neighbouring slabs of a tile, so that what is in flight at one time is
// whole cells.  Memory does not serve all SMs equally: a CTA that is done with its block takes over one that has not been
// launched (a cluster launch control request, in flight with the copies); with equal ranges SMs were idle for an eighth of
// the time.  A thread owns 8 channels and a strip of 4 outputs, its 3 x 3 window sliding along the strip out of shared
// memory; 8 threads cover the 128 bytes a cell has in a slab.  At 8 x 64 x 128 cells of 3072 channels 202 us, 6.0 TB/s
// (blocks that each loaded a tile and then worked on it: 254 us; this ring with equal ranges: 256 us).
constexpr int kDwSlab = 64, kDwStages = 3, kDwRun = 4;
constexpr int kDwStrips = 64, kDwCells = 18 * 18;                                    // at most, of a tile and with its halo
constexpr int kDwYBytes = kDwCells * kDwSlab * 2, kDwGateBytes = kDwStrips * kDwRun * kDwSlab * 2;
constexpr int kDwWeights = kDwYBytes + kDwGateBytes, kDwBias = kDwWeights + 9 * kDwSlab * 2;
constexpr int kDwStageBytes = kDwBias + kDwSlab * 2;                                 // 75,520: a multiple of 128
constexpr int kDwThreads = kDwStrips * (kDwSlab / 8);                                // 512: 128 registers each
constexpr int kDwSmem = kDwStages * kDwStageBytes + 128 + 128;                       // control words, alignment

struct DwMaps { CUtensorMap y, gate, weight, bias; };

__device__ __forceinline__ void dw_load4(uint32_t dst, const CUtensorMap* m, uint32_t bar, int c0, int c1, int c2, int c3,
                                         uint64_t policy) {
    asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.L2::cache_hint [%0], "
                 "[%1, {%3, %4, %5, %6}], [%2], %7;"
                 ::"r"(dst), "l"(reinterpret_cast<uint64_t>(m)), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "l"(policy) : "memory");
}
__device__ __forceinline__ void dw_load2(uint32_t dst, const CUtensorMap* m, uint32_t bar, int c0) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
                 ::"r"(dst), "l"(reinterpret_cast<uint64_t>(m)), "r"(bar), "r"(c0), "r"(0) : "memory");
}
// Asks for a block of the grid that has not been launched; the 16-byte answer arrives on `bar`.
__device__ __forceinline__ void dw_ask(uint32_t answer, uint32_t bar) {
    fence_proxy_async_smem();            // the answer before it has been read
    mbar_arrive_expect_tx(bar, 16);
    asm volatile("clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];"
                 ::"r"(answer), "r"(bar) : "memory");
}
__device__ __forceinline__ int dw_answer(uint32_t answer) {       // the block, or -1: none is left
    uint32_t got, x;
    asm volatile("{\n\t.reg .pred p;\n\t.reg .b128 h;\n\tld.shared.b128 h, [%2];\n\t"
                 "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, h;\n\tselp.u32 %0, 1, 0, p;\n\tmov.u32 %1, 0;\n\t"
                 "@p clusterlaunchcontrol.query_cancel.get_first_ctaid::x.b32.b128 %1, h;\n\t}"
                 : "=r"(got), "=r"(x) : "r"(answer) : "memory");
    return got ? static_cast<int>(x) : -1;
}
// Set when a wait of this kernel ran out anywhere on the device, until it is read (gla_b200_swiglu_status): the call has no scratch that
// could hold a word of its own.
__device__ uint32_t g_dw_status;
constexpr uint32_t kDwWaitUs = 2000000;
// Waits here are for copies, for warps of the same CTA and for the launch control's answers.  False after the limit, or as soon as
// another wait of this CTA (which sets its shared `flag`) has given up: the CTA then leaves, its outputs are undefined and the status says so.
__device__ __forceinline__ bool dw_wait(uint32_t bar, uint32_t parity, uint32_t flag, uint32_t limit_us = kDwWaitUs) {
    for (int n = 0; n < 64; ++n)
        if (mbar_try_wait(bar, parity)) return true;
    const uint32_t t0 = globaltimer_1024ns();
    while (ld_shared_u32(flag) == 0u) {
        for (int n = 0; n < 64; ++n)
            if (mbar_try_wait(bar, parity)) return true;
        if (globaltimer_1024ns() - t0 > limit_us) {
            st_shared_u32(flag, 1u);
            atomicExch(&g_dw_status, 1u);
        }
    }
    return false;
}
// One thread waits for a barrier that nobody arrives at.
__global__ void dw_timeout_selftest_kernel(uint32_t limit_us) {
    __shared__ uint64_t bar;
    __shared__ uint32_t flag;
    mbar_init(smem_u32(&bar), 1);
    flag = 0u;
    fence_mbar_init();
    dw_wait(smem_u32(&bar), 0, smem_u32(&flag), limit_us);
}

__global__ void __launch_bounds__(kDwThreads, 1) swiglu_dwconv_kernel(const __grid_constant__ DwMaps maps, __half* __restrict__ out,
                                                                      bool biased, int images, int rows, int strips, int B, int hg, int wg, int C) {
    extern __shared__ uint8_t dw_smem[];
    const uint32_t base = (smem_u32(dw_smem) + 127u) & ~127u, control = base + kDwStages * kDwStageBytes;
    const int tid = threadIdx.x;
    const int cols = strips * kDwRun, tiles_c = (wg + cols - 1) / cols, tiles_r = (hg + rows - 1) / rows;
    const int slabs = (C + kDwSlab - 1) / kDwSlab;
    // control words: the answer, a stage's item (-1: none is left), barriers, a flag
    auto item_of = [&](int s) { return control + 16u + 4u * s; };
    auto full = [&](int s) { return control + 32u + 8u * s; };
    auto empty = [&](int s) { return control + 32u + 8u * (kDwStages + s); };
    const uint32_t answered = control + 32u + 16u * kDwStages, gave_up = answered + 8u;
    if (tid == 0) {
        for (int s = 0; s < kDwStages; ++s) {
            mbar_init(full(s), 1);
            mbar_init(empty(s), kDwThreads / 32);
        }
        mbar_init(answered, 1);
        st_shared_u32(gave_up, 0u);
        fence_mbar_init();
    }
    __syncthreads();
    pdl_wait();
    const uint32_t bytes = (images * ((rows + 2) * (cols + 2) + rows * cols) + 9 + (biased ? 1 : 0)) * kDwSlab * 2u;
    // thread 0 fills the stages in turn, two items ahead of the work, and asks for the item after each
    int to_fill = 0;
    uint32_t fill_turn = 0, asked = 0;
    bool more = true;
    auto fill = [&](int item) {
        const int s = to_fill;
        if (!dw_wait(empty(s), (fill_turn & 1u) ^ 1u, gave_up)) { more = false; return; }       // the stage may still be read
        asm volatile("st.shared.b32 [%0], %1;" ::"r"(item_of(s)), "r"(item) : "memory");
        if (item < 0) {
            more = false;
            mbar_arrive(full(s));
            return;
        }
        const int slab = item % slabs, tile = item / slabs;
        const int tc = tile % tiles_c, rest = tile / tiles_c, tr = rest % tiles_r, b = rest / tiles_r * images;
        const uint32_t to = base + s * kDwStageBytes;
        mbar_arrive_expect_tx(full(s), bytes);
        dw_load4(to, &maps.y, full(s), slab * kDwSlab, tc * cols - 1, tr * rows - 1, b, l2_policy_normal());
        dw_load4(to + kDwYBytes, &maps.gate, full(s), slab * kDwSlab, tc * cols, tr * rows, b, l2_policy_stream());
        dw_load2(to + kDwWeights, &maps.weight, full(s), slab * kDwSlab);
        if (biased) dw_load2(to + kDwBias, &maps.bias, full(s), slab * kDwSlab);
        if (++to_fill == kDwStages) { to_fill = 0; ++fill_turn; }
        dw_ask(control, answered);
    };
    auto fill_next = [&] {
        if (!more) return;
        if (!dw_wait(answered, asked & 1u, gave_up)) { more = false; return; }
        ++asked;
        fill(dw_answer(control));
    };
    if (tid == 0) {
        fill(static_cast<int>(blockIdx.x));
        fill_next();
    }
    const int ci = tid & 7, tall = (tid >> 3) / strips, image = tall / rows, trow = tall - image * rows, tcol = (tid >> 3) % strips * kDwRun;
    const uint32_t line = (cols + 2) * 128u, y_at = (tall + 2 * image) * line + tcol * 128u + 16u * ci;
    const uint32_t gate_at = kDwYBytes + (tall * cols + tcol) * 128u + 16u * ci;
    const int CG = C >> 3;
    uint32_t turn = 0;
    for (int s = 0;;) {
        if (tid == 0) fill_next();
        __syncwarp();
        if (!dw_wait(full(s), turn & 1u, gave_up)) break;
        int item;
        asm volatile("ld.shared.b32 %0, [%1];" : "=r"(item) : "r"(item_of(s)) : "memory");
        if (item < 0) break;
        const int slab = item % slabs, tile = item / slabs, cg = slab * (kDwSlab / 8) + ci;
        const int tc = tile % tiles_c, rest = tile / tiles_c, tr = rest % tiles_r, b = rest / tiles_r * images + image;
        const int r = tr * rows + trow, c = tc * cols + tcol;
        const uint32_t stage = base + s * kDwStageBytes;
        if (image < images && b < B && r < hg && c < wg && cg < CG) {
            uint4 wv[9];
#pragma unroll
            for (int k = 0; k < 9; ++k) wv[k] = ld_shared_v4(stage + kDwWeights + 128u * k + 16u * ci);
            float bv[8] = {};
            if (biased) dw_unpack8(ld_shared_v4(stage + kDwBias + 16u * ci), bv);
            uint4 win[3][3];                 // win[column slot][row]; the columns change roles by renaming
#pragma unroll
            for (int rr = 0; rr < 3; ++rr) {
                win[0][rr] = ld_shared_v4(stage + y_at + rr * line);
                win[1][rr] = ld_shared_v4(stage + y_at + rr * line + 128u);
            }
            uint4* to = reinterpret_cast<uint4*>(out) + ((static_cast<long long>(b) * hg + r) * wg + c) * CG + cg;
#pragma unroll
            for (int j = 0; j < kDwRun; ++j) {
                const int sl = j % 3, sm = (j + 1) % 3, sn = (j + 2) % 3;     // left, middle, new column slots
#pragma unroll
                for (int rr = 0; rr < 3; ++rr) win[sn][rr] = ld_shared_v4(stage + y_at + rr * line + (j + 2) * 128u);
                float g[8], acc[8];
                dw_unpack8(ld_shared_v4(stage + gate_at + 128u * j), g);
#pragma unroll
                for (int rr = 0; rr < 3; ++rr) {
                    dw_fma8(acc, wv[3 * rr + 0], win[sl][rr], rr == 0 ? bv : acc);
                    dw_fma8(acc, wv[3 * rr + 1], win[sm][rr], acc);
                    dw_fma8(acc, wv[3 * rr + 2], win[sn][rr], acc);
                }
                uint4 o;
                __half2* oh = reinterpret_cast<__half2*>(&o);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float2 h = mul2(two(0.5f), pair_of(g, e));       // silu(x) = h + h * tanh(h), h = x / 2
                    const float2 z = mul2(fma2(h, tanh_2(h), h), pair_of(acc, e));
                    oh[e] = __floats2half2_rn(z.x, z.y);
                }
                if (c + j < wg) __stcs(to + static_cast<long long>(j) * CG, o);
            }
        }
        __syncwarp();
        if ((tid & 31) == 0) mbar_arrive(empty(s));
        if (++s == kDwStages) { s = 0; ++turn; }
    }
    if (tid == 0 && ld_shared_u32(gave_up) != 0u) {           // what this CTA still has under way must land before its memory is given back
        st_shared_u32(gave_up, 0u);
        const uint32_t filled = fill_turn * kDwStages + to_fill;
        for (uint32_t s = 0; s < kDwStages; ++s) {
            const uint32_t n = (filled + kDwStages - 1 - s) / kDwStages;
            if (n > 0 && !dw_wait(full(s), (n - 1) & 1u, gave_up)) return;
        }
        if (filled > asked) dw_wait(answered, asked & 1u, gave_up);
    }
}

// LayerNorm over rows of D fp16 values (D a multiple of 8, D <= 2048), affine, fp32 statistics: one warp per kRows rows, held
// in registers as they came between the mean, the variance and the output pass, so that x is read once and y written
// once.  HBM-bound: what matters is the bytes in flight, so the rows stay packed (as floats they took the registers of half
// the warps) and, where there are rows enough, a warp asks for two at once: 32768 rows of 768 27.9 -> 18.5 us, 5.4 TB/s;
// of 2048 (one row a warp) 68.9 -> 45.3 us.
// kVec = 16-byte vectors per lane and row, chosen by the host from D: a narrow row must not pay for the registers of the
// widest one.
constexpr int kLnMaxVec = 8;

// y may alias x (in-place use): x is read with plain loads and neither pointer is declared restrict.
template <int kVec, int kRows>
__global__ void __launch_bounds__(256) layernorm_rows_kernel(const __half* x, const __half* __restrict__ w,
                                                             const __half* __restrict__ b, __half* y,
                                                             long long rows, int D, float eps) {
    const long long row = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) / 32 * kRows;
    const int lane = threadIdx.x & 31;
    if (row >= rows) return;
    pdl_wait();
    const int nvec = D >> 3;
    const uint4* x4 = reinterpret_cast<const uint4*>(x) + row * nvec;
    uint4 in[kRows][kVec];
#pragma unroll
    for (int r = 0; r < kRows; ++r)
#pragma unroll
        for (int k = 0; k < kVec; ++k)
            in[r][k] = row + r < rows && lane + 32 * k < nvec ? x4[static_cast<long long>(r) * nvec + lane + 32 * k] : make_uint4(0u, 0u, 0u, 0u);
    float mean[kRows], rstd[kRows];
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
        float sum = 0.f;
#pragma unroll
        for (int k = 0; k < kVec; ++k) {
            if (lane + 32 * k < nvec) {
                float v[8];
                dw_unpack8(in[r][k], v);
#pragma unroll
                for (int e = 0; e < 8; ++e) sum += v[e];
            }
        }
        mean[r] = sum;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int r = 0; r < kRows; ++r) mean[r] += __shfl_xor_sync(0xffffffffu, mean[r], o);
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
        mean[r] = mean[r] / static_cast<float>(D);
        float sq = 0.f;
#pragma unroll
        for (int k = 0; k < kVec; ++k) {
            if (lane + 32 * k < nvec) {
                float v[8];
                dw_unpack8(in[r][k], v);
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    const float d = v[e] - mean[r];
                    sq = fmaf(d, d, sq);
                }
            }
        }
        rstd[r] = sq;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int r = 0; r < kRows; ++r) rstd[r] += __shfl_xor_sync(0xffffffffu, rstd[r], o);
#pragma unroll
    for (int r = 0; r < kRows; ++r) rstd[r] = rsqrtf(rstd[r] / static_cast<float>(D) + eps);
    uint4* y4 = reinterpret_cast<uint4*>(y) + row * nvec;
#pragma unroll
    for (int k = 0; k < kVec; ++k) {
        const int i = lane + 32 * k;
        if (i < nvec) {
            float wv[8], bv[8];
            dw_unpack8(__ldg(reinterpret_cast<const uint4*>(w) + i), wv);
            if (b != nullptr) dw_unpack8(__ldg(reinterpret_cast<const uint4*>(b) + i), bv);
#pragma unroll
            for (int r = 0; r < kRows; ++r) {
                float v[8];
                dw_unpack8(in[r][k], v);
                uint4 o;
                __half2* oh = reinterpret_cast<__half2*>(&o);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float a0 = (v[2 * e] - mean[r]) * rstd[r] * wv[2 * e] + (b != nullptr ? bv[2 * e] : 0.f);
                    const float a1 = (v[2 * e + 1] - mean[r]) * rstd[r] * wv[2 * e + 1] + (b != nullptr ? bv[2 * e + 1] : 0.f);
                    oh[e] = __floats2half2_rn(a0, a1);
                }
                if (row + r < rows) y4[static_cast<long long>(r) * nvec + i] = o;
            }
        }
    }
}

}  // namespace gla
