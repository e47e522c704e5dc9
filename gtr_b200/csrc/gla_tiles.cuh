// What the operator's kernels and its gradient's share: the tensors as tiles, the walk over a scan's boxes, tensor-memory
// accumulators of one chunk, bounded waits.
//
// Every kernel works on 64-token chunks of one (batch, head) as [64 x 64] fp16 tiles with rows of 128 bytes and the 128-byte
// XOR swizzle, the layout both TMA and the UMMA descriptors use.  Scan orders are folded into the tile coordinates: a tile holds
// its tokens in the order they lie in memory along the scan's columns, and a reversed scan's chunk is mirrored (its first
// token is row 63).
#pragma once

#include <type_traits>

#include "gla_device.cuh"

namespace gla {

constexpr int kChunk = 64;
constexpr int kD = 64;                    // V, and the widest K
constexpr int kTileBytes = kChunk * 128;  // one fp16 [64 x 64] tile
constexpr int kStageBytes = 4 * kTileBytes;
constexpr int kComputeThreads = 256;
constexpr float kLog2e = 1.4426950408889634f;

// tensor ids inside Maps
enum { TQ = 0, TK = 1, TG = 2, TV = 3, TO = 4, kNumTensors = 5 };
constexpr int kNumBoxes = 4;              // box heights 64, 16, 4, 1 rows

// Where the j-th of `parts` nearly equal parts of n things begins, floor(j n / parts), from n = parts * len + rest: no product
// leaves 32 bits while there are at most kMaxParts of them.
constexpr int kMaxParts = 65535;
__host__ __device__ constexpr int part_begin(int j, int len, int rest, int parts) {
    return j * len + static_cast<int>(static_cast<uint32_t>(j) * static_cast<uint32_t>(rest) / static_cast<uint32_t>(parts));
}

struct Maps {
    CUtensorMap m[kNumTensors][kNumBoxes];
};

enum { WHERE_MBAR = 1, WHERE_LOOKBACK = 2 };

// Bounded waits.  On expiry, or once another wait of its group has given up, a wait returns without its barrier, so that all warps keep
// following the protocol and the kernel drains and exits; its result is then undefined and the status word ctrl[1] says so.
template <class Gave, class Give>
__device__ __forceinline__ void bounded_wait(uint64_t& bar, uint32_t parity, uint32_t limit_us, Gave gave_up, Give give_up) {
    const uint32_t b = smem_u32(&bar);
    for (int n = 0; n < 8; ++n)
        if (mbar_try_wait(b, parity)) return;
    const uint32_t t0 = globaltimer_1024ns();             // 32 bits: registers are scarce where this is inlined
    for (uint32_t n = 1;; ++n) {
        if (mbar_try_wait(b, parity)) return;
        if ((n & 63u) != 0u) continue;
        if (gave_up()) return;
        if (globaltimer_1024ns() - t0 > limit_us) { give_up(); return; }
    }
}
template <class P_t>
__device__ __forceinline__ void report_timeout(const P_t& P) { atomicCAS(P.ctrl + 1, 0u, static_cast<uint32_t>(WHERE_MBAR)); }

// For a kernel that starts with the status word cleared, by the kernel before it in the stream: its group is the launch.
template <class P_t>
__device__ __forceinline__ void wait_bar(const P_t& P, uint64_t& bar, uint32_t parity) {
    bounded_wait(bar, parity, P.wait_limit_us, [&] { return *reinterpret_cast<volatile uint32_t*>(P.ctrl + 1) != 0u; }, [&] { report_timeout(P); });
}
// For the first kernel of a call, whose block 0 clears the word (what lies there is an earlier call's, or never was written): its
// group is the block, by a flag in shared memory.  Where a second kernel follows, this one leaves kTimedOut in place of a decay, which
// the second one reports; no arithmetic makes a NaN of these bits.
template <class P_t>
__device__ __forceinline__ void wait_bar(const P_t& P, uint64_t& bar, uint32_t parity, uint32_t& flag) {
    volatile uint32_t* f = &flag;
    bounded_wait(bar, parity, P.wait_limit_us, [&] { return *f != 0u; }, [&] { *f = 1u; });
}
constexpr uint32_t kTimedOut = 0x7fc0deadu;
// A kernel that is first and last: block 0 clears the word when it starts and says so with a number of the launch in ctrl[0], which it
// takes back when it leaves (the launch may be replayed); a block that has given up reports when it has seen that number.  Not
// seeing it for as long as a wait may take means that block 0 has long left.
__device__ __forceinline__ void clear_alone(uint32_t* ctrl, uint32_t launch) {
    volatile uint32_t* c = ctrl;
    c[1] = 0u;
    __threadfence();
    c[0] = launch;
}
template <class P_t>
__device__ __forceinline__ void report_alone(const P_t& P, uint32_t launch) {
    volatile uint32_t* c = P.ctrl;
    const uint32_t t0 = globaltimer_1024ns();
    while (c[0] != launch && globaltimer_1024ns() - t0 <= max(P.wait_limit_us, 10000u)) {}
    __threadfence();
    report_timeout(P);
}

// Enumerates the TMA boxes that cover one chunk of the scan: f(box_id, r, c, smem_row) with (r, c) the row inside the
// column and the column where the box starts.
struct BoxWalker {
    int u_lo;     // scan position of the chunk's first row (may be negative for the ragged chunk of a reversed scan)
    int c, r;     // column and row inside the column of max(u_lo, 0)
    template <class P_t>
    __device__ __forceinline__ BoxWalker(const P_t& P, int p0) {
        u_lo = P.rev ? (P.T - p0 - kChunk) : p0;
        const int u0 = max(u_lo, 0);
        c = u0 / P.Hc;
        r = u0 - c * P.Hc;
    }
    // boxes over the rows the sequence has
    template <class P_t, class F>
    __device__ __forceinline__ void for_each(const P_t& P, F f) const {
        int u0 = max(u_lo, 0);
        const int u1 = min(u_lo + kChunk, P.T);
        int cc = c, rr = r;
        while (u0 < u1) {
            int len = min(P.Hc - rr, u1 - u0);
            while (len > 0) {
                const int id = len >= 64 ? 0 : len >= 16 ? 1 : len >= 4 ? 2 : 3;
                const int R = 64 >> (2 * id);
                f(id, rr, cc, u0 - u_lo);
                rr += R;
                u0 += R;
                len -= R;
            }
            if (rr >= P.Hc) { rr = 0; ++cc; }
        }
    }
    // boxes over the rows of the tile the sequence does not have (loads only): placed out of bounds, the copy
    // engine fills them with zeros.  f(box_id, smem_row)
    template <class P_t, class F>
    __device__ __forceinline__ void for_each_missing(const P_t& P, F f) const {
        int row = u_lo < 0 ? 0 : min(u_lo + kChunk, P.T) - u_lo;        // first missing tile row
        int len = u_lo < 0 ? -u_lo : kChunk - row;
        while (len > 0) {
            const int id = len >= 16 ? 1 : len >= 4 ? 2 : 3;
            const int R = 64 >> (2 * id);
            f(id, row);
            row += R;
            len -= R;
        }
    }
};

__device__ __forceinline__ uint32_t sw_f16(uint32_t row, uint32_t col) {     // col in fp16 elements
    return row * 128u + ((((col >> 3) ^ row) & 7u) << 4) + ((col & 7u) << 1);
}
// address of 16-byte unit `unit` of row `row` in a swizzled tile
__device__ __forceinline__ uint32_t sw_unit(uint32_t tile, uint32_t row, uint32_t unit) {
    return tile + row * 128u + (((unit ^ row) & 7u) << 4);
}
__device__ __forceinline__ uint32_t hmul2_u32(uint32_t a, uint32_t b) {
    __half2 r = __hmul2(*reinterpret_cast<__half2*>(&a), *reinterpret_cast<__half2*>(&b));
    return *reinterpret_cast<uint32_t*>(&r);
}

__device__ __forceinline__ uint32_t hmin2_zero(uint32_t a) {
    __half2 r = __hmin2(*reinterpret_cast<__half2*>(&a), __half2half2(__ushort_as_half(0)));
    return *reinterpret_cast<uint32_t*>(&r);
}

// the larger of each; NaN stays
__device__ __forceinline__ uint32_t hmax2_nan(uint32_t a, uint32_t b) {
    __half2 r = __hmax2_nan(*reinterpret_cast<__half2*>(&a), *reinterpret_cast<__half2*>(&b));
    return *reinterpret_cast<uint32_t*>(&r);
}

// One M = 64 accumulator per slot: 64 columns, lanes 0-15 (even slots) or 16-31 (odd) of every quadrant.
__device__ __forceinline__ uint32_t acc_slot(uint32_t tmem, int slot) {
    return tmem + (static_cast<uint32_t>(16 * (slot & 1)) << 16) + 64u * static_cast<uint32_t>(slot >> 1);
}
// 16 columns of one accumulator row: lanes 0-15 of warp w columns 32 (w / 4) .. +15 of rows 16 (w % 4) + lane, lanes 16-31
// columns +16 .. +31 of the same rows.
__device__ __forceinline__ void acc_read(uint32_t tmem, int slot, int w, float* x) {
    const uint32_t a = acc_slot(tmem, slot) + (static_cast<uint32_t>(32 * (w & 3)) << 16) + 32u * static_cast<uint32_t>(w >> 2);
    uint32_t* r = reinterpret_cast<uint32_t*>(x);
    asm volatile(
        "tcgen05.ld.sync.aligned.16x32bx2.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16], 16;"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(a)
        : "memory");
}
// columns `off` .. +7 of the same piece
__device__ __forceinline__ void acc_read8(uint32_t tmem, int slot, int w, uint32_t off, float* x) {
    const uint32_t a = acc_slot(tmem, slot) + (static_cast<uint32_t>(32 * (w & 3)) << 16) + 32u * static_cast<uint32_t>(w >> 2) + off;
    uint32_t* r = reinterpret_cast<uint32_t*>(x);
    asm volatile("tcgen05.ld.sync.aligned.16x32bx2.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8], 16;"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(a)
                 : "memory");
}
__device__ __forceinline__ void acc_write(uint32_t tmem, int slot, int w, const float* x) {
    const uint32_t a = acc_slot(tmem, slot) + (static_cast<uint32_t>(32 * (w & 3)) << 16) + 32u * static_cast<uint32_t>(w >> 2);
    const uint32_t* r = reinterpret_cast<const uint32_t*>(x);
    asm volatile(
        "tcgen05.st.sync.aligned.16x32bx2.x16.b32 [%0], 16, "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
        ::"r"(a), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
          "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}

// D (+)= A B over K = 64 from two swizzled tiles; kA / kB: 1 when the tile's rows are the contraction index.
template <uint32_t kA, uint32_t kB>
__device__ __forceinline__ void tile_mma(uint32_t d, uint32_t a, uint32_t b, bool accumulate) {
    constexpr uint32_t id = umma_idesc(FMT_F16, kA, kB, 64, 64);
    const uint64_t da = umma_desc_sw128(a, 8192), db = umma_desc_sw128(b, 8192);
#pragma unroll
    for (uint32_t ks = 0; ks < 4; ++ks)
        umma_f16(d, da + ks * (kA ? 128u : 2u), db + ks * (kB ? 128u : 2u), id, (accumulate || ks > 0) ? 1u : 0u);
}

// 16 columns of one row of a swizzled fp16 tile as they lie there
__device__ __forceinline__ void row16(uint32_t tile, uint32_t row, uint32_t unit, uint32_t* r) {
    const uint4 a = ld_shared_v4(sw_unit(tile, row, unit)), b = ld_shared_v4(sw_unit(tile, row, unit + 1));
    r[0] = a.x; r[1] = a.y; r[2] = a.z; r[3] = a.w; r[4] = b.x; r[5] = b.y; r[6] = b.z; r[7] = b.w;
}
__device__ __forceinline__ void put16(uint32_t tile, uint32_t row, uint32_t unit, const uint32_t* r) {
    st_shared_v4(sw_unit(tile, row, unit), r[0], r[1], r[2], r[3]);
    st_shared_v4(sw_unit(tile, row, unit + 1), r[4], r[5], r[6], r[7]);
}
// A [64 x 64] constant operand of the gate-sum MMA (K-major): entry (r, s) = value(r, s), 16 bytes at a time
template <class F>
__device__ __forceinline__ void fill_constant(uint32_t tile, F value) {
    for (uint32_t e = threadIdx.x; e < 512u; e += blockDim.x) {
        const uint32_t r = e >> 3, s = (e & 7u) * 8u;
        uint32_t v[4];
#pragma unroll
        for (uint32_t i = 0; i < 4; ++i) v[i] = pack_half2(value(r, s + 2 * i), value(r, s + 2 * i + 1));
        st_shared_v4(sw_unit(tile, r, e & 7u), v[0], v[1], v[2], v[3]);
    }
}

// Masks of 16 scores, as fp16 pairs: on the diagonal by the row within its group of 16; all kept; none kept.  (Comparing rows and columns
// pair by pair was 870 cycles of a chunk's chain on an SM of its own, this is 250.)
struct CausalMasks {
    alignas(16) uint32_t m[18][8];
    // by 128 threads or more, without a loop: in calls of one chunk a block a general one was up to a tenth of the call (1200 x 1 chunk 21.4 us, 18.8)
    __device__ __forceinline__ void fill(bool rev) {
        const int e = threadIdx.x, t = e >> 3, c = 2 * (e & 7);
        if (e < 16 * 8) m[t][e & 7] = ((rev ? c >= t : c <= t) ? 0xffffu : 0u) | ((rev ? c + 1 >= t : c + 1 <= t) ? 0xffff0000u : 0u);
        if (e < 2 * 8) m[16 + t][e & 7] = t == 0 ? 0xffffffffu : 0u;
    }
};
// Those of the half row of scores that lane l of the w-th warp of four holds: of its two groups of 16 keys, the one of the warp's parity lies on
// the diagonal where the half row crosses it; what lies on the near side is kept whole, the rest dropped.
struct CausalRow {
    uint32_t at, beside;
    __device__ __forceinline__ CausalRow(const CausalMasks& masks, int w, int l, bool rev) {
        const int side = (l >> 4) - (w >> 1);              // 0: the half row crosses the diagonal; otherwise on which side it lies
        const bool near = rev ? side > 0 : side < 0;
        at = smem_u32(masks.m[side == 0 ? l & 15 : near ? 16 : 17]);
        beside = near || (side == 0 && ((w & 1) != 0) != rev) ? 0xffffffffu : 0u;
    }
    __device__ __forceinline__ void mask(int w, const float* x, uint32_t* r) const {
        const uint4 a = ld_shared_v4(at), b = ld_shared_v4(at + 16u);
        const uint32_t m[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
        auto group = [&](int first, bool diagonal) {
#pragma unroll
            for (int e = 0; e < 8; ++e) r[(first >> 1) + e] = pack_half2(x[first + 2 * e], x[first + 2 * e + 1]) & (diagonal ? m[e] : beside);
        };
        if (w & 1) { group(0, false); group(16, true); }
        else { group(0, true); group(16, false); }
    }
};

struct Scan { int T, Hc, rev; };          // what the walk over the boxes needs to know; `T` is the sequence's own length

// One chunk of kN tensors into tiles.  Rows past the sequence are filled with zeros, channels a K = 32 head does not have too.
// `tok0`: first row of the sequence when sequences are packed into one (`rows`: all rows there are).  `policy`: L2 eviction
// priority.
template <int kN>
__device__ __forceinline__ void load_chunk(const Maps& maps, const Scan& S, int chunk, int b, int h, int tok0, int rows, uint32_t bar,
                                           const int (&tensors)[kN], const uint32_t (&tiles)[kN], uint64_t policy) {
    const BoxWalker bw(S, chunk * kChunk);
    bw.for_each(S, [&](int id, int r, int c, int row) {
#pragma unroll
        for (int i = 0; i < kN; ++i) tma_load_5d_hint(tiles[i] + 128u * row, &maps.m[tensors[i]][id], bar, 0, h, r + tok0, c, b, policy);
    });
    bw.for_each_missing(S, [&](int id, int row) {
#pragma unroll
        for (int i = 0; i < kN; ++i) tma_load_5d(tiles[i] + 128u * row, &maps.m[tensors[i]][id], bar, 0, h, rows, 0, b);
    });
}
__device__ __forceinline__ void named_bar_arrive(uint32_t id, uint32_t threads) {
    asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}

// The token at scan position p of a sequence, or -1 past its end.
template <class P_t>
__device__ __forceinline__ int scan_token(const P_t& P, int T, int p) {
    if (p >= T) return -1;
    const int u = P.rev ? T - 1 - p : p;
    if (P.Wc == 1) return u;
    const int c = u / P.Hc;
    return (u - c * P.Hc) * P.Wc + c;
}

}  // namespace gla
