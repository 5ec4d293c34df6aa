// Q4 GEMV over M = 1 .. 8 rows of x for rows of any whole number of 256-column chunks (512 with groups of 128): the
// small-batch GEMM at every such width, and the single-row GEMV at the widths q4_gemv_mma.cuh is not built for. Dot
// products on the tensor cores with the operand formats of that kernel (nibbles as bf16 subnormals, activations scaled
// by a power of two), in the same order within a window: a batch row equals the same vector run alone bit for bit at 1024,
// 2048 and 4096 columns, and wherever one row of x runs on this kernel too (not at 8192 and 12288 columns, which the other
// kernel adds up window by window within a warp, nor where one row runs on the FMA pipe).
//
// What is different from that kernel, and why:
//   * A row's groups are dealt out to the 16 consumer warps one by one instead of in sixteenths of a fixed width, so K
//     need not be a power of two (2560 columns, groups of 64: 2 or 3 groups per warp).
//   * Rows longer than 4096 columns are split over the CTAs of a cluster, each holding the activations of its window in
//     registers for the whole launch; the windows' sums meet in the first CTA's shared memory (distributed shared memory,
//     added in window order). A block that walked the windows itself would read all of x (196 KB at 8 x 12288, as much
//     as its share of the weights), and would leave the chip in ceil(rows / 16 / 148) x windows steps instead of
//     ceil(rows / 16 / (148 / windows)).
//   * A second reducer warp: adding the 16 warps' sums of 8 columns and storing them took one warp longer than the stream
//     takes for a stage (151936 x 4096, M = 8: 72.9 us with one, 56.0 with two = 6.25 TB/s; 65.3 before this kernel).
//   * A stage is ONE tiled TMA copy of 16 rows x the window as 128-byte columns (3-D map: 128 bytes, rows, chunks) plus
//     one per 32 groups for the scale/bias pairs, both with the 128-byte swizzle. With rows back to back in shared
//     memory the eight lane groups of a warp read their scale/bias words from the same bank; swizzled, neither these reads
//     nor the rows' fragments meet a conflict, without padding.
//   * One row of x has instantiations of its own (ONE): the redundant work of eight equal columns, most of all every quad
//     converting the whole slice of x, made a short launch up to 0.9 us slower than the FMA-pipe kernels had been
//     (257 x 7168: 2.76 us there, 3.84 with it, 2.92 without; gate/up 2048 x 5120 6.10, 7.33, 6.37; 9216 x 2560 10.4, 9.45, 8.17).
//
// Bound: a long stream by HBM (above); a short launch by its start (x: 64 KB per SM at 8 x 4096, then ~300 instructions a
// lane to turn it into fragments) and by whole stages per SM. Measured before (row windows or the FMA pipe) and now, M = 8:
// 12288 x 4096 10.3 -> 8.3 us, 4096 x 4096 6.4 -> 4.6, 4096 x 12288 with the residual 63.7 -> 9.2, M = 5: 9216 x 2560
// 28.5 -> 5.0, 2560 x 9216 27.2 -> 6.9; M = 1: 6144 x 2560 5.6 -> 3.7, 4096 x 17408 24.6 -> 10.4. Groups of 32 hold eight groups'
// offsets and words per lane and spill 80 - 136 bytes at M > 1 (12288 x 4096, M = 8: 14.5 -> 11.9 us).
//
// Structure: 16 consumer warps, one producer, two reducers per block, one block per SM. Every mbarrier wait is bounded.
#pragma once
#include <cuda.h>

#include "q4_gemv_mma.cuh"

namespace tessl {
namespace q4b {

using q4k::lds32;
using q4k::map_to_cta;
using q4k::mbar_arrive;
using q4k::mbar_expect_tx;
using q4k::mbar_init;
using q4k::mbar_try;
using q4k::mbar_wait;
using q4k::smem_u32;
using q4k::tma_load_2d;
using q4k::tma_load_3d;
using q4m::lds64;
using q4m::mma_bf16;

constexpr int kConsumers = 16;
constexpr int kReducers = 2;
constexpr int kThreads = (kConsumers + 1 + kReducers) * 32;
constexpr uint32_t kRows = 16;                         // weight rows per stage = MMA M
constexpr uint32_t kChunkCols = 256;                   // columns of a 128-byte swizzle row
constexpr uint32_t kBoxBytes = kRows * 128;            // one chunk of packed rows, or 32 groups of scale/bias pairs
constexpr uint32_t kPartBytes = kConsumers * kRows * 8 * 4;
constexpr uint32_t kMailSlots = 4, kMailBytes = kRows * 8 * 4;  // a window's sums of one stage
constexpr uint32_t kMaxWindows = 8;                    // portable cluster size
constexpr uint32_t kWindowCols = 4096;                 // 8 words of 8 nibbles per lane and row

struct Seg {
    void *out;           // [m, rows]
    const float *resid;  // [m, rows] or null
    uint32_t rows;
    uint32_t rb_begin;   // first row block of this bank within the launch
};

struct Params {
    const uint16_t *x;  // bf16 [m, cols]
    Seg seg[3];
    uint32_t *status;
    uint32_t nseg, cols, m, group_shift;
    uint32_t units;     // cols in units of whole chunks and whole quads of groups; window c is [c units / nwin, (c + 1) units / nwin)
    uint32_t unit_cols;
    uint32_t nwin;      // windows = CTAs per cluster
    uint32_t chunks;    // chunks per copy (the widest window's)
    uint32_t sb_boxes;  // 32-group copies of scale/bias pairs per stage
    uint32_t stages, total_rb;
    uint32_t rb_step_lo, rb_step_hi;  // row blocks per cluster, 32.32 fixed point (see q4_gemv_mma.cuh)
    int epi, out_bf16;
};

/// Packed rows and scale/bias pairs of every bank of the launch (a gate/up pair: banks 0 and 1).
struct Maps {
    CUtensorMap w[3], sb[3];
};
__device__ __forceinline__ void mbar_arrive_remote(uint32_t cluster_addr)
{
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
/// Bounded wait for an arrival from another CTA of the cluster.
__device__ __forceinline__ bool mbar_wait_cluster(uint32_t bar, uint32_t parity, volatile int *abort_flag)
{
    const long long t0 = clock64();
    for (uint32_t i = 1;; ++i) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\tselp.b32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(bar), "r"(parity)
            : "memory");
        if (done) return true;
        if ((i & 63u) == 0) {
            if (*abort_flag) return false;
            if (clock64() - t0 > 4000000000ll) {
                *abort_flag = 1;
                return false;
            }
        }
    }
}

/// 4 bytes into another CTA's shared memory; completes 4 bytes on that CTA's barrier.
__device__ __forceinline__ void st_async4(uint32_t cluster_addr, float v, uint32_t cluster_bar)
{
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.f32 [%0], %1, [%2];" ::"r"(cluster_addr), "f"(v), "r"(cluster_bar)
                 : "memory");
}

/// 16 bytes into another CTA's shared memory; completes 16 bytes on that CTA's barrier.
__device__ __forceinline__ void st_async16(uint32_t cluster_addr, const float (&v)[4], uint32_t cluster_bar)
{
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1,%2,%3,%4}, [%5];" ::"r"(cluster_addr),
                 "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "r"(cluster_bar)
                 : "memory");
}

/// WPG: words of one lane per quantization group (G / 32). NGS: groups of the busiest warp (a warp has NGS or NGS - 1;
/// EVEN: every warp has NGS in every window, so its scale/bias words are aligned vectors and no group needs a test).
/// NB: banks per row block (2 = a gate/up pair and one row of x: MMA rows 0-7 are gate rows, 8-15 the same rows of up).
/// ONE: one row of x. The 8 columns of an MMA then hold the same vector, and what a batch does per column is done once: a
/// warp converts its slice of x together (a lane a word of 8 columns, through shared memory) instead of every quad for itself,
/// the lanes of a quad share the fold (lane t the group classes t), the reducers add one column. Same roundings, same bits.
template <int WPG, int NGS, bool EVEN, int NB, bool ONE>
__global__ void __launch_bounds__(kThreads, 1) q4_batch_mma_kernel(const __grid_constant__ Maps maps, const __grid_constant__ Params p)
{
    asm volatile("griddepcontrol.launch_dependents;");
    constexpr int SW = WPG * NGS;
    constexpr uint32_t G = 32 * WPG;
    constexpr uint32_t RPB = kRows / NB;        // rows per bank and stage
    constexpr uint32_t kBox = RPB * 128;        // one chunk, or 32 groups of pairs, of one bank
    static_assert(NB == 1 || ONE, "a pair of banks meets one row of x");
    extern __shared__ uint8_t smem_raw[];
    __shared__ int abort_flag;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t nwin = p.nwin;
    const uint32_t win = nwin == 1 ? 0u : blockIdx.x % nwin;  // the rank within the cluster
    const uint32_t cluster = nwin == 1 ? blockIdx.x : blockIdx.x / nwin;
    const uint32_t col0 = win * p.units / nwin * p.unit_cols, col1 = (win + 1) * p.units / nwin * p.unit_cols;

    const uint32_t S = p.stages;
    const uint32_t ring = (smem_u32(smem_raw) + 1023u) & ~1023u;  // the swizzle is a function of the address
    const uint32_t off_sb = p.chunks * kBoxBytes, off_part = off_sb + p.sb_boxes * kBoxBytes;
    const uint32_t stage_bytes = off_part + kPartBytes;
    const uint32_t mail = ring + S * stage_bytes;
    const uint32_t bars = mail + kMailSlots * (nwin - 1) * kMailBytes;
    auto full = [&](uint32_t s) { return bars + 8 * s; };
    auto empty = [&](uint32_t s) { return bars + 8 * (S + s); };
    auto done = [&](uint32_t s) { return bars + 8 * (2 * S + s); };
    const uint32_t xbar = bars + 24 * S;  // consumers: x is in registers (the producer holds the ring's tail for it)
    auto mail_full = [&](uint32_t s) { return xbar + 8 + 8 * s; };                // the first CTA's: the other windows' sums are here
    auto mail_empty = [&](uint32_t s) { return xbar + 8 + 8 * (kMailSlots + s); };  // the others': the slot has been read

    auto rb_at = [&](uint32_t b) { return min(__umulhi(b, p.rb_step_lo) + b * p.rb_step_hi, p.total_rb); };
    const uint32_t rb_lo = rb_at(cluster);
    const uint32_t n_local = rb_at(cluster + 1) - rb_lo;

    if (warp == kConsumers) {
        if (lane == 0) abort_flag = 0;
        if ((uint32_t)lane <= 3 * S) mbar_init(bars + 8 * lane, (uint32_t)lane < 2 * S ? 1u : (uint32_t)kConsumers);
        if (nwin > 1 && (uint32_t)lane < 2 * kMailSlots) mbar_init(mail_full(lane), 1u);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        asm volatile("bar.arrive 2, %0;" ::"n"(kThreads) : "memory");
    } else {
        asm volatile("bar.sync 2, %0;" ::"n"(kThreads) : "memory");
    }
    // Every CTA's barriers are set up before another CTA signals them: everybody arrives here, the reducers wait for it
    // before their first exchange, the others where the block ends.
    if (nwin > 1) asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    volatile int *abortp = &abort_flag;
    auto fail = [&](uint32_t role, uint32_t where) {
        *abortp = 1;
        if (*(volatile uint32_t *)p.status == 0)
            *(volatile uint32_t *)p.status = (0x60u << 24) | (role << 20) | (where & 0xfffffu);
    };

    if (warp == kConsumers) {
        // ------------------------------------------------ producer ---
        if (lane == 0) {
            const uint32_t bytes = (p.chunks + p.sb_boxes) * kBoxBytes;  // whole boxes: parts outside the bank are zero-filled and count
            uint32_t sg = 0;
            const int chunk0 = (int)(col0 / kChunkCols), group0 = (int)(col0 >> p.group_shift);
            const uint32_t hold_from = n_local == 3 ? 2u : q4m::kHoldFrom;  // see q4_gemv_mma.cuh
            uint32_t s = 0, ph = 0, issued = 0;
            for (uint32_t j = 0; j < n_local; ++j) {
                if (!mbar_wait(empty(s), ph ^ 1u, abortp, 64)) {
                    fail(1, j);
                    break;
                }
                if (j == hold_from && n_local <= q4m::kHoldMaxStages && !mbar_wait(xbar, 0, abortp, 64)) {
                    fail(1, j);
                    break;
                }
                const uint32_t st = ring + s * stage_bytes;
                while (sg + 1 < p.nseg && rb_lo + j >= p.seg[sg + 1].rb_begin) ++sg;
                const int row0 = (int)((rb_lo + j - p.seg[sg].rb_begin) * RPB);
                mbar_expect_tx(full(s), bytes);
#pragma unroll
                for (uint32_t b = 0; b < NB; ++b) {
                    tma_load_3d(st + b * p.chunks * kBox, &maps.w[sg + b], 0, row0, chunk0, full(s));
                    for (uint32_t i = 0; i < p.sb_boxes; ++i)
                        tma_load_2d(st + off_sb + (b * p.sb_boxes + i) * kBox, &maps.sb[sg + b], group0 + 32 * (int)i, row0, full(s));
                }
                ++issued;
                if (++s == S) s = 0, ph ^= 1u;
            }
            // After a timeout elsewhere copies may still be in flight: give the last ring a bounded chance to land.
            if (*abortp) {
                for (uint32_t i = issued > S ? issued - S : 0; i < issued; ++i) {
                    const long long t0 = clock64();
                    while (!mbar_try(full(i % S), (i / S) & 1u))
                        if (clock64() - t0 > 4000000000ll) break;
                }
            }
        }
        __syncwarp();
    } else if (warp > kConsumers) {
        // ------------------------------------------------ reducer ---
        asm volatile("griddepcontrol.wait;" ::: "memory");  // y and resid belong to the stream's order
        if (nwin > 1) asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
        // lane l: row l / 2 of the stage, batch columns 4 (l % 2) .. + 3; one row of x: lanes 0 .. 15 a row each
        constexpr int NC = ONE ? 1 : 4;
        constexpr uint32_t kMail = ONE ? kRows * 4 : kMailBytes;  // bytes of a window's sums of one stage
        const uint32_t r = ONE ? (uint32_t)lane & 15u : (uint32_t)lane >> 1, c0 = ONE ? 0u : (lane & 1) * 4;
        const uint32_t lead_mail = nwin > 1 ? map_to_cta(mail, 0) : 0u, lead_full = nwin > 1 ? map_to_cta(mail_full(0), 0) : 0u;
        const uint32_t q0 = (uint32_t)warp - kConsumers - 1;
        uint32_t s = q0, ph = 0;  // S >= kReducers
        for (uint32_t j = q0; j < n_local; j += kReducers) {
            const uint32_t slot = j % kMailSlots, mph = (j / kMailSlots) & 1u;
            uint32_t sg = 0;
            while (sg + 1 < p.nseg && rb_lo + j >= p.seg[sg + 1].rb_begin) ++sg;
            const uint32_t rows = p.seg[sg].rows;
            const uint32_t row = (rb_lo + j - p.seg[sg].rb_begin) * RPB + r;  // NB = 2: lanes of r < 8
            const bool live = row < rows && r < RPB && (!ONE || lane < 16);
            float rv[NC] = {};
            if (p.epi == q4k::EPI_ADD_RESID && win == 0 && live) {
#pragma unroll
                for (int c = 0; c < NC; ++c)
                    if (ONE || c0 + c < p.m) rv[c] = *(volatile const float *)(p.seg[sg].resid + (size_t)(c0 + c) * rows + row);
            }
            if (!mbar_wait(done(s), ph, abortp, 32)) {
                if (lane == 0) fail(3, j);
                break;
            }
            const uint32_t part = ring + s * stage_bytes + off_part;
            float v[NC] = {};
#pragma unroll
            for (int w = 0; w < kConsumers; ++w) {
                if constexpr (ONE) {
                    v[0] += __uint_as_float(lds32(part + w * 512 + r * 4));
                } else {
                    const uint4 q = q4k::lds128(part + ((w * 16 + r) * 8 + c0) * 4);
                    v[0] += __uint_as_float(q.x), v[1] += __uint_as_float(q.y);
                    v[2] += __uint_as_float(q.z), v[3] += __uint_as_float(q.w);
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(empty(s));  // partial sums read: the stage may be refilled
            if (nwin > 1) {
                if (win != 0) {
                    if (!mbar_wait_cluster(mail_empty(slot), mph ^ 1u, abortp)) {
                        if (lane == 0) fail(4, j);
                        break;
                    }
                    const uint32_t to = lead_mail + (slot * (nwin - 1) + win - 1) * kMailBytes;
                    if constexpr (ONE) {
                        if (lane < 16) st_async4(to + lane * 4, v[0], lead_full + 8 * slot);
                    } else {
                        st_async16(to + lane * 16, v, lead_full + 8 * slot);
                    }
                } else {
                    if (lane == 0) mbar_expect_tx(mail_full(slot), (nwin - 1) * kMail);
                    if (!mbar_wait_cluster(mail_full(slot), mph, abortp)) {
                        if (lane == 0) fail(5, j);
                        break;
                    }
                    for (uint32_t w = 0; w + 1 < nwin; ++w) {
                        const uint32_t from = mail + (slot * (nwin - 1) + w) * kMailBytes;
                        if constexpr (ONE) {
                            v[0] += __uint_as_float(lds32(from + r * 4));
                        } else {
                            const uint4 q = q4k::lds128(from + lane * 16);
                            v[0] += __uint_as_float(q.x), v[1] += __uint_as_float(q.y);
                            v[2] += __uint_as_float(q.z), v[3] += __uint_as_float(q.w);
                        }
                    }
                    __syncwarp();
                    if ((uint32_t)lane + 1 < nwin) mbar_arrive_remote(map_to_cta(mail_empty(slot), lane + 1));
                }
            }
            if constexpr (NB == 2) {
                const float up = __shfl_down_sync(0xffffffffu, v[0], 8);  // row r + 8
                v[0] = (p.epi == q4k::EPI_GATE_UP_GELU ? dev::gelu_pytorch_tanh(v[0]) : dev::silu(v[0])) * up;
            }
            if (win == 0 && live) {
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    if (ONE || c0 + c < p.m) {
                        const size_t idx = (size_t)(c0 + c) * rows + row;
                        float o = v[c];
                        if (p.epi == q4k::EPI_ADD_RESID) o = o + rv[c];
                        if (p.out_bf16) {
                            static_cast<uint16_t *>(p.seg[sg].out)[idx] = dev::f32_to_bf16_store(o);
                        } else {
                            static_cast<float *>(p.seg[sg].out)[idx] = o;
                        }
                    }
                }
            }
            s += kReducers;
            if (s >= S) s -= S, ph ^= 1u;
        }
    } else {
        // ------------------------------------------------ consumers ---
        const uint32_t g = lane >> 2, t = lane & 3;
        // Logical warp: the four warps of an SM sub-partition (warp % 4) take neighbouring slices, so that slices of NGS
        // and NGS - 1 groups, which alternate, are spread evenly over the sub-partitions.
        const uint32_t lw = ((uint32_t)warp & 3u) * 4 + ((uint32_t)warp >> 2);
        const uint32_t gw = (col1 - col0) >> p.group_shift;
        const uint32_t g_lo = lw * gw / kConsumers;
        const bool whole = (lw + 1) * gw / kConsumers - g_lo == (uint32_t)NGS;  // this warp has an NGS-th group
        asm volatile("griddepcontrol.wait;" ::: "memory");  // x is written by the preceding kernel
        // B fragments, group sums and the power-of-two scaling of the activations: as in q4_gemv_mma.cuh
        uint32_t xb[SW][4];
        constexpr int NQ = (NGS + 3) / 4;
        // Group sums and multipliers of this lane's outputs, which are batch columns 2 t and 2 t + 1 (they live in quads 2 t and
        // 2 t + 1). One row of x: the sums of the groups that this lane folds, t, t + 4, ...
        float xs0[ONE ? NQ : NGS], xs1[ONE ? 1 : NGS];
        float cw0, cw1 = 0.0f;
        if constexpr (ONE) {
            const uint32_t words = (whole ? NGS : NGS - 1) * 4 * WPG;  // of 8 columns: lane L takes word L
            const uint32_t xst = ring + off_part + lw * 512;  // staged in this warp's place for the sums of the first stage
            uint4 v = make_uint4(0u, 0u, 0u, 0u);
            if ((uint32_t)lane < words) v = dev::ld_after_wait16(p.x + col0 + g_lo * G + 8 * lane);
            const uint32_t amax2 = __vmaxu2(__vmaxu2(v.x & 0x7fff7fffu, v.y & 0x7fff7fffu), __vmaxu2(v.z & 0x7fff7fffu, v.w & 0x7fff7fffu));
            const dev::XScale xsc = dev::x_scale(__reduce_max_sync(0xffffffffu, max(amax2 & 0xffffu, amax2 >> 16)));
            cw0 = xsc.undo;
            uint32_t f[4];
            dev::x_fragment(v, xsc, f);
            asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(xst + lane * 16), "r"(f[0]), "r"(f[1]), "r"(f[2]), "r"(f[3]) : "memory");
            // the sum of a group: over the words of a lane t in turn, then over the four t, as for a batch
            const float a = (dev::bf16_lo(v.x) + dev::bf16_hi(v.x)) + (dev::bf16_lo(v.y) + dev::bf16_hi(v.y));
            const float b = (dev::bf16_lo(v.z) + dev::bf16_hi(v.z)) + (dev::bf16_lo(v.w) + dev::bf16_hi(v.w));
            float part = a + b;
#pragma unroll
            for (int u = 1; u < WPG; ++u) part += __shfl_down_sync(0xffffffffu, a, u), part += __shfl_down_sync(0xffffffffu, b, u);
            part += __shfl_xor_sync(0xffffffffu, part, WPG);
            part += __shfl_xor_sync(0xffffffffu, part, 2 * WPG);  // valid in the lanes of words u = 0
            part = dev::scaled_sum(part, xsc);
#pragma unroll
            for (int q = 0; q < NQ; ++q) xs0[q] = __shfl_sync(0xffffffffu, part, ((4 * q + t) * 4 * WPG) & 31u);
            __syncwarp();
#pragma unroll
            for (int jj = 0; jj < NGS; ++jj) {
#pragma unroll
                for (int u = 0; u < WPG; ++u) {
                    const uint4 w = q4k::lds128(xst + ((jj * 4 + t) * WPG + u) * 16);
                    xb[jj * WPG + u][0] = w.x, xb[jj * WPG + u][1] = w.y, xb[jj * WPG + u][2] = w.z, xb[jj * WPG + u][3] = w.w;
                }
            }
            __syncwarp();  // the staged copy is read: the place may take the sums
        } else {
            float xs[NGS];
            const uint16_t *xrow = p.x + (size_t)min(g, p.m - 1) * p.cols + col0;
#pragma unroll
            for (int jj = 0; jj < NGS; ++jj) {
#pragma unroll
                for (int u = 0; u < WPG; ++u) {
                    const uint32_t k = (g_lo + jj) * G + t * (G / 4) + 8 * u;
                    uint4 v = make_uint4(0u, 0u, 0u, 0u);
                    if (EVEN || jj < NGS - 1 || whole) v = dev::ld_after_wait16(xrow + k);
                    xb[jj * WPG + u][0] = v.x, xb[jj * WPG + u][1] = v.y, xb[jj * WPG + u][2] = v.z, xb[jj * WPG + u][3] = v.w;
                }
            }
            uint32_t amax2 = 0;  // two 16-bit maxima
#pragma unroll
            for (int i = 0; i < SW; ++i) {
#pragma unroll
                for (int c = 0; c < 4; ++c) amax2 = __vmaxu2(amax2, xb[i][c] & 0x7fff7fffu);
            }
            uint32_t amax = max(amax2 & 0xffffu, amax2 >> 16);
            amax = max(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
            amax = max(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
            const dev::XScale xsc = dev::x_scale(amax);
#pragma unroll
            for (int jj = 0; jj < NGS; ++jj) {
                float part = 0.0f;
#pragma unroll
                for (int u = 0; u < WPG; ++u) {
                    uint32_t(&f)[4] = xb[jj * WPG + u];
                    const uint4 v = make_uint4(f[0], f[1], f[2], f[3]);
                    part += (dev::bf16_lo(v.x) + dev::bf16_hi(v.x)) + (dev::bf16_lo(v.y) + dev::bf16_hi(v.y));
                    part += (dev::bf16_lo(v.z) + dev::bf16_hi(v.z)) + (dev::bf16_lo(v.w) + dev::bf16_hi(v.w));
                    dev::x_fragment(v, xsc, f);
                }
                part += __shfl_xor_sync(0xffffffffu, part, 1);
                part += __shfl_xor_sync(0xffffffffu, part, 2);
                xs[jj] = dev::scaled_sum(part, xsc);  // the same in the four lanes of a quad
            }
            cw0 = __shfl_sync(0xffffffffu, xsc.undo, (2 * t) * 4), cw1 = __shfl_sync(0xffffffffu, xsc.undo, (2 * t + 1) * 4);
#pragma unroll
            for (int jj = 0; jj < NGS; ++jj) {
                xs0[jj] = __shfl_sync(0xffffffffu, xs[jj], (2 * t) * 4);
                xs1[jj] = __shfl_sync(0xffffffffu, xs[jj], (2 * t + 1) * 4);
            }
        }
        if (lane == 0) mbar_arrive(xbar);  // this warp holds its x fragments: the producer may fill the rest of the ring

        // Offsets within a stage of the lane's words and scale/bias words (of a group that the warp does not have: the window's
        // last, unused). MMA rows g and g + 8 are rows rl and rl + 8 of the
        // stage (row rl of either bank of a pair): the same swizzle, 1024 bytes (a bank) apart. rl = 0, 2, 4, 6, 1, 3, 5, 7 for
        // g = 0 .. 7: the two 16-byte pieces that the quad of a row reads then fall on eight different ones over each half warp.
        const uint32_t rl = 2 * (g & 3u) + (g >> 2);
        uint32_t woff[NGS], soff[ONE ? NQ : NGS];
        auto pair_at = [&](uint32_t gi) { return off_sb + (gi >> 5) * kBox + rl * 128 + ((((gi & 31u) >> 2) ^ rl) << 4) + (gi & 3u) * 4; };
#pragma unroll
        for (int jj = 0; jj < NGS; ++jj) {
            const uint32_t gi = min(g_lo + jj, gw - 1), byte = gi * (G / 2), in = (byte & 127u) + t * (G / 8);
            woff[jj] = (byte >> 7) * kBox + rl * 128 + (((in >> 4) ^ rl) << 4) + (in & 15u);
            if constexpr (!ONE) soff[jj] = pair_at(gi);
        }
        if constexpr (ONE) {
#pragma unroll
            for (int q = 0; q < NQ; ++q) soff[q] = pair_at(min(g_lo + 4 * q + t, gw - 1));
        }
        const uint32_t whi = NB == 2 ? p.chunks * kBox : 1024u, shi = NB == 2 ? p.sb_boxes * kBox : 1024u;
        const uint32_t part_off = off_part + (ONE ? lw * 512 + rl * 4 : ((lw * 16 + rl) * 8 + 2 * t) * 4);
        uint32_t s = 0, ph = 0;
        for (uint32_t j = 0; j < n_local; ++j) {
            if (!mbar_wait(full(s), ph, abortp, 32)) {
                if (lane == 0) fail(2, j);
                break;
            }
            const uint32_t st = ring + s * stage_bytes;
            // rows rl, rl + 8 x columns 2 t, 2 t + 1: the groups' scale * dot + bias * group sum in units of cw, one
            // accumulator per group class jj % 4 (the order of q4_gemv_mma.cuh)
            float acc[4][4] = {};
            float vlo = 0.0f, vhi = 0.0f;  // one row of x: rows rl and rl + 8, the group class t
#pragma unroll
            for (int b0 = 0; b0 < NGS; b0 += 4) {  // four groups at a time: their MMA chains are interleaved
                uint32_t wl[4 * WPG], wh[4 * WPG], sl[4], sh[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    if (b0 + i >= NGS) continue;
                    const uint32_t lo = st + woff[b0 + i];
                    if constexpr (WPG == 1) {
                        wl[i] = lds32(lo), wh[i] = lds32(lo + whi);
                    } else if constexpr (WPG == 2) {
                        const uint2 a = lds64(lo), b = lds64(lo + whi);
                        wl[2 * i] = a.x, wl[2 * i + 1] = a.y, wh[2 * i] = b.x, wh[2 * i + 1] = b.y;
                    } else {
                        const uint4 a = q4k::lds128(lo), b = q4k::lds128(lo + whi);
                        wl[4 * i] = a.x, wl[4 * i + 1] = a.y, wl[4 * i + 2] = a.z, wl[4 * i + 3] = a.w;
                        wh[4 * i] = b.x, wh[4 * i + 1] = b.y, wh[4 * i + 2] = b.z, wh[4 * i + 3] = b.w;
                    }
                }
                if constexpr (ONE) {
                    sl[0] = lds32(st + soff[b0 / 4]), sh[0] = lds32(st + soff[b0 / 4] + shi);
                } else if constexpr (EVEN && NGS % 4 == 0) {
                    const uint4 a = q4k::lds128(st + soff[b0]), b = q4k::lds128(st + soff[b0] + shi);
                    sl[0] = a.x, sl[1] = a.y, sl[2] = a.z, sl[3] = a.w, sh[0] = b.x, sh[1] = b.y, sh[2] = b.z, sh[3] = b.w;
                } else if constexpr (EVEN && NGS == 2) {
                    const uint2 a = lds64(st + soff[0]), b = lds64(st + soff[0] + shi);
                    sl[0] = a.x, sl[1] = a.y, sh[0] = b.x, sh[1] = b.y;
                } else {
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        if (b0 + i < NGS) sl[i] = lds32(st + soff[b0 + i]), sh[i] = lds32(st + soff[b0 + i] + shi);
                }
                float d[4][4] = {};
#pragma unroll
                for (int u = 0; u < WPG; ++u) {
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        if (b0 + i >= NGS) continue;
                        const uint32_t a = wl[i * WPG + u], b = wh[i * WPG + u];
                        const uint32_t(&x)[4] = xb[(b0 + i) * WPG + u];
                        if (EVEN || b0 + i < NGS - 1 || whole)
                            mma_bf16(d[i], a & 0x000f000fu, b & 0x000f000fu, a & 0x00f000f0u, b & 0x00f000f0u, x[0], x[1]);
                    }
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        if (b0 + i >= NGS) continue;
                        const uint32_t a = wl[i * WPG + u] >> 8, b = wh[i * WPG + u] >> 8;
                        const uint32_t(&x)[4] = xb[(b0 + i) * WPG + u];
                        if (EVEN || b0 + i < NGS - 1 || whole)
                            mma_bf16(d[i], a & 0x000f000fu, b & 0x000f000fu, a & 0x00f000f0u, b & 0x00f000f0u, x[2], x[3]);
                    }
                }
                if constexpr (ONE) {
                    float dl = 0.0f, dh = 0.0f;
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        if (b0 + i < NGS && t == (uint32_t)i) dl = d[i][0], dh = d[i][2];
                    const uint32_t jj = b0 + t;
                    if (jj < (uint32_t)NGS - 1u || (jj == (uint32_t)NGS - 1u && whole)) {
                        const float xg = xs0[b0 / 4];
                        vlo = fmaf(dev::bf16_lo(sl[0]), dl, fmaf(dev::bf16_hi(sl[0]), xg, vlo));
                        vhi = fmaf(dev::bf16_lo(sh[0]), dh, fmaf(dev::bf16_hi(sh[0]), xg, vhi));
                    }
                } else {
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        if (b0 + i >= NGS) continue;
                        if (EVEN || b0 + i < NGS - 1 || whole) {
                            const float s0 = dev::bf16_lo(sl[i]), z0 = dev::bf16_hi(sl[i]), s1 = dev::bf16_lo(sh[i]), z1 = dev::bf16_hi(sh[i]);
                            acc[0][i] = fmaf(s0, d[i][0], fmaf(z0, xs0[b0 + i], acc[0][i]));
                            acc[1][i] = fmaf(s0, d[i][1], fmaf(z0, xs1[b0 + i], acc[1][i]));
                            acc[2][i] = fmaf(s1, d[i][2], fmaf(z1, xs0[b0 + i], acc[2][i]));
                            acc[3][i] = fmaf(s1, d[i][3], fmaf(z1, xs1[b0 + i], acc[3][i]));
                        }
                    }
                }
            }
            if constexpr (ONE) {
                vlo += __shfl_xor_sync(0xffffffffu, vlo, 1), vhi += __shfl_xor_sync(0xffffffffu, vhi, 1);
                vlo += __shfl_xor_sync(0xffffffffu, vlo, 2), vhi += __shfl_xor_sync(0xffffffffu, vhi, 2);
                vlo *= cw0, vhi *= cw0;
                if (t == 0) {
                    asm volatile("st.shared.f32 [%0], %1;" ::"r"(st + part_off), "f"(vlo) : "memory");
                    asm volatile("st.shared.f32 [%0], %1;" ::"r"(st + part_off + 32), "f"(vhi) : "memory");
                }
            } else {
                float o[4];
#pragma unroll
                for (int c = 0; c < 4; ++c) o[c] = ((acc[c][0] + acc[c][1]) + (acc[c][2] + acc[c][3])) * (c & 1 ? cw1 : cw0);
                asm volatile("st.shared.v2.f32 [%0], {%1,%2};" ::"r"(st + part_off), "f"(o[0]), "f"(o[1])
                             : "memory");
                asm volatile("st.shared.v2.f32 [%0], {%1,%2};" ::"r"(st + part_off + 256), "f"(o[2]), "f"(o[3])
                             : "memory");
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(done(s));  // release: the partial sums are visible to the reducer
            if (++s == S) s = 0, ph ^= 1u;
        }
    }
    // No CTA leaves while another one of its cluster may still reach into its shared memory. (After a timeout sums may be
    // on their way to the first CTA that nobody waits for: they get time to land.)
    if (nwin > 1) {
        __syncwarp();
        if (*abortp) {
            const long long t0 = clock64();
            while (clock64() - t0 < 200000) __nanosleep(1000);
        }
        if (warp <= kConsumers) asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
        asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
    }
}

}  // namespace q4b
}  // namespace tessl
