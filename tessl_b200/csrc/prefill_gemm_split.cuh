// MLX Q4 prefill GEMM for few rows of X: the weights are the MMA's M side and K is split over a cluster.
//
// The CTA-pair kernel (prefill_gemm_pair.cuh) puts X on the M side, 256 rows at a time, and one cluster walks all of K.
// With 77 rows of X most of its MMA is padding, and with few tiles the call is one serial chain of K blocks on part of the
// chip (77 x 4096 x 12288: 64 tiles of 204 K blocks at 0.25 us on 74 clusters). Here
//
//   * a tile is 128 weight rows x up to 160 rows of X, D^T[n, m] = W[n, :] . X[m, :]: X is the MMA's N, in steps of 16 rows;
//   * the S CTAs of a cluster take S parts of K of one tile and add their f32 accumulators up through distributed shared
//     memory, every CTA the sum of its share of the columns, in the order of the parts (shorter chains of f32 sums, too: the
//     relative error against 64 bits at 77 x 4096 x 12288 falls from 1.4e-5 to 3e-6);
//   * a dequant thread expands one weight row of a unit of two K blocks (128 weights) straight into TMEM, which the MMA takes its
//     A operand from: no shared-memory store and fetch of the expanded weights, and no proxy fence, which in the pair kernel
//     waits for the thread's outstanding global loads, so that scale words can be fetched two units ahead;
//   * a lane holds one weight row of D, so 32 lanes store 32 neighbours of a row of y: whole lines without a transposition,
//     for any N.
//
// What bounds it: per K block and SM 0.2 us, most of it the dequant warps' instructions (77 x 4096 x 12288 in clusters of four, over
// the whole launch: issue slots 41 % busy, ALU pipe 27 %, f16 FMA 19 %, tensor pipe 24 %), then ~4 us around them (pre-pass, start,
// first copies, last stores) and 2 - 3 us for the exchange of a cluster. On the way: one wait and one commit per unit instead of two rings
// and a commit per K block 0.25 -> 0.19 us per K block; row scales read once per CTA instead of by every epilogue warp from the
// same lines of L2 9 -> 2 us per tile; scale words in the dequant threads' registers instead of copied by one warp 22.5 ->
// 15.9 us at 100 x 1000 x 2080. Tried: two CTAs per SM with half the TMEM each (the scheduler packs them on half of the SMs:
// 56 us where one per SM took 38), three dequant groups instead of four (the same).
//
// Before (pair kernel) -> here, back to back in a graph: 77 x 4096 x 12288 53.5 -> 21.7 us, 25 x 4096 x 4096 19.1 -> 11.1,
// 128 x 2048 x 2048 12.8 -> 10.2, 300 x 4096 x 4096 26.7 -> 19.3, 509 x 2048 x 6144 31.1 -> 23.6, 64 x 12288 x 4096 28.9 -> 20.6.
// The pair kernel stays the faster one where its tiles fill the clusters and the rows (200 x 12288 x 4096 29.4 against 41).
//
// Same operands, exact products and f32 accumulation as the other prefill kernels (prefill_gemm.cu).
//
// Roles: warp 0 TMA producer of X, warp 1 TMEM allocation and MMA issue, warp 2 TMA producer of the packed weights, warp 3 row
// scales, warps 4-19 four groups of dequant warps on successive units, then the epilogue. A CTA's units are a range of the
// sequence (extra K blocks one by one, main ones in pairs). Every wait is bounded; on a timeout the status word is set and all
// roles fall through to the cluster barriers.
#pragma once
#include "prefill_common.cuh"

namespace tessl {
namespace pf {

struct SplitCfg {
    static constexpr int ROWS = 128;       // weight rows per tile = MMA M
    static constexpr int MAX_X = 160;      // rows of X per tile = MMA N, at most
    static constexpr int NG = 4;           // dequant groups of four warps; group g expands units g, g + NG, ...
    static constexpr int SQ = 8;           // packed stages, a unit (two K blocks) each
    static constexpr int MAX_SU = 6;       // stages of (X tiles, expanded weights), a unit each
    static constexpr uint32_t MAX_SPLIT = 6;  // CTAs per tile: clusters of eight find room for 16 at most
    static constexpr int FIRST_DW = 4;     // first dequant warp
    static constexpr int THREADS = (FIRST_DW + NG * 4) * 32;
    static constexpr uint32_t UNIT_COLS = 64;           // TMEM columns of an expanded unit
    static constexpr uint32_t Q_BYTES = ROWS * 64;      // packed rows of a unit, 64-byte swizzle
    static constexpr int NBARS = 2 * MAX_SU + 2 * SQ + 1;
    static constexpr uint32_t RS_BYTES = MAX_X * 4;     // row scales
    static constexpr uint32_t FIXED = SQ * Q_BYTES + RS_BYTES + NBARS * 8 + 1024;  // + slack to align the base to 1 KiB
    static constexpr uint32_t BUDGET = 226 * 1024;
};
// What a group waits for must not be a whole round of a ring ahead of what it has seen, or the parity is ambiguous. Packed ring:
// copies may land out of order, so a stage belongs to one group (with 6 stages a group could pass its wait on the round before,
// whose copy another group still waited for: a wait of a long run timed out). TMEM ring: commits are in order, and a group
// has waited for that of unit u - NG - su when it comes to unit u, which is as late as u - 2 su if su >= NG.
static_assert(SplitCfg::SQ % SplitCfg::NG == 0, "a packed stage would change hands");
static_assert(SplitCfg::FIXED + SplitCfg::NG * 2 * SplitCfg::MAX_X * BK * 2 <= SplitCfg::BUDGET &&
                  SplitCfg::NG * SplitCfg::UNIT_COLS + SplitCfg::MAX_X <= kTmemCols,
              "fewer stages than dequant groups");

struct SplitParams {
    const uint32_t *sb;
    const float *row_scale;
    void *y;
    uint32_t M, N, gshift, gpr;
    uint32_t nkb_main, nkb_extra;
    uint32_t tiles_m, x_rows;  // rows of X per tile, a multiple of 16
    uint32_t split;            // CTAs per tile
    uint32_t su;               // stages of the (X tiles, expanded weights) ring
    uint32_t sb_tiled;         // the extra units' words come by TMA
    uint32_t sb_words;         // scale words that one load may take: 1, 2 or 4
    int out_bf16;
    uint32_t *status;
};

__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32])
{
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,"
        "%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};" ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
        "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]),
        "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]),
        "r"(r[31])
        : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float (&v)[8])
{
    uint32_t r[8];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
        : "r"(taddr));
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = __uint_as_float(r[j]);
}
/// One K block: D[tmem] (+)= A[tmem] . B[smem]^T in four K = 16 slices. A converged warp runs this; one election for all four.
__device__ __forceinline__ void tcgen05_block_ts_elect(uint32_t tmem_d, uint32_t tmem_a, uint32_t bdesc_lo, uint32_t idesc,
                                                       uint32_t accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p, e;\n\t.reg .b64 b0, b1, b2, b3;\n\t.reg .b32 a1, a2, a3, l1, l2, l3;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "add.u32 a1, %1, 8;\n\tadd.u32 a2, %1, 16;\n\tadd.u32 a3, %1, 24;\n\t"
        "add.u32 l1, %2, 2;\n\tadd.u32 l2, %2, 4;\n\tadd.u32 l3, %2, 6;\n\t"
        "mov.b64 b0, {%2, %5};\n\tmov.b64 b1, {l1, %5};\n\tmov.b64 b2, {l2, %5};\n\tmov.b64 b3, {l3, %5};\n\t"
        "elect.sync _|e, 0xffffffff;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], b0, %3, p;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [a1], b1, %3, 1;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [a2], b2, %3, 1;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [a3], b3, %3, 1;\n\t}" ::"r"(tmem_d),
        "r"(tmem_a), "r"(bdesc_lo), "r"(idesc), "r"(accumulate), "r"(kUmmaDescHi)
        : "memory");
}
__device__ __forceinline__ void tcgen05_commit_elect(uint32_t bar)
{
    asm volatile(
        "{\n\t.reg .pred e;\n\telect.sync _|e, 0xffffffff;\n\t"
        "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(bar)
        : "memory");
}
__device__ __forceinline__ uint32_t lds32(uint32_t a)
{
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    return v;
}
/// Position in a ring whose depth is a launch parameter.
struct RunRing {
    uint32_t stage = 0, phase = 0;
    __device__ __forceinline__ void advance(uint32_t depth, uint32_t n = 1)  // n <= depth
    {
        stage += n;
        if (stage >= depth) stage -= depth, phase ^= 1u;
    }
};

__global__ void __launch_bounds__(SplitCfg::THREADS, 1)
    q4_prefill_gemm_split_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w,
                                 const __grid_constant__ CUtensorMap map_s, const SplitParams p)
{
    using C = SplitCfg;
    extern __shared__ uint8_t smem_raw[];
    __shared__ uint32_t tmem_base_slot;
    __shared__ int abort_flag;
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();
    const uint32_t x_block = p.x_rows * (BK * 2), x_bytes = 2 * x_block;  // X tiles of a K block, of a unit
    const uint32_t off_q = base + p.su * x_bytes, off_rs = off_q + C::SQ * C::Q_BYTES,
                   bar0 = off_rs + C::RS_BYTES;
    //   full / empty       ring of units: both X tiles have landed and the weights are in TMEM; the MMAs have read them
    //   q_full / q_empty   ring of packed units      acc_full   the accumulator is complete
    auto full = [&](uint32_t s) { return bar0 + 8 * s; };
    auto empty = [&](uint32_t s) { return bar0 + 8 * (C::MAX_SU + s); };
    auto q_full = [&](uint32_t s) { return bar0 + 8 * (2 * C::MAX_SU + s); };
    auto q_empty = [&](uint32_t s) { return bar0 + 8 * (2 * C::MAX_SU + C::SQ + s); };
    const uint32_t acc_full = bar0 + 8 * (C::NBARS - 1);

    // This CTA's tile and its part of the unit sequence: the extra K blocks, one unit each, then the main ones in pairs.
    const uint32_t tile = blockIdx.x / p.split;
    const uint32_t m0 = (tile % p.tiles_m) * p.x_rows, n0 = (tile / p.tiles_m) * C::ROWS;
    // Parts of about as many K blocks; a cut among the main ones falls between two units.
    const uint32_t total = p.nkb_extra + p.nkb_main;
    auto cut = [&](uint32_t r) {
        const uint32_t k = r * total / p.split;
        return k <= p.nkb_extra ? k : p.nkb_extra + (k - p.nkb_extra + 1) / 2;
    };
    const uint32_t u0 = cut(rank), u1 = cut(rank + 1);
    // First K block of unit u, and how many it has.
    auto main_block = [&](uint32_t u) { return 2 * (u - p.nkb_extra); };
    auto unit_blocks = [&](uint32_t u) { return u < p.nkb_extra || main_block(u) + 1 >= p.nkb_main ? 1u : 2u; };

    if (warp == 0) {
        if (lane < C::MAX_SU) mbar_init(full(lane), 1 + 4), mbar_init(empty(lane), 1);
        if (lane < C::SQ) mbar_init(q_full(lane), 1), mbar_init(q_empty(lane), 4);
        if (lane == 0) {
            abort_flag = 0;
            mbar_init(acc_full, 1);
            asm volatile("prefetch.tensormap [%0];" ::"l"(&map_x) : "memory");
            asm volatile("prefetch.tensormap [%0];" ::"l"(&map_w) : "memory");
            if (p.sb_tiled) asm volatile("prefetch.tensormap [%0];" ::"l"(&map_s) : "memory");
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_slot)),
                     "r"(kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem_base = tmem_base_slot, tmem_a = tmem_base + kTmemCols - p.su * C::UNIT_COLS;
    volatile int *abortp = &abort_flag;
    auto fail = [&](uint32_t role, uint32_t where) {
        *abortp = 1;
        *(volatile uint32_t *)p.status = (role << 24) | (where & 0xffffffu);
    };
    const uint32_t quarter = (uint32_t)warp & 3u;  // the TMEM lanes that a dequant / epilogue warp may reach
    const uint32_t lane_base = (quarter * 32u) << 16;

    if (warp == 0) {
        // ------------------------------------------------ TMA producer: X tiles ---
        if (lane == 0) {
            // as in the pair kernel: ordinary stores of the pre-pass, read here through the async proxy
            asm volatile("griddepcontrol.wait;\n\tfence.proxy.async.global;" ::: "memory");
            RunRing ring;
            uint32_t issued = 0;
            for (uint32_t u = u0; u < u1; ++u) {
                if (!mbar_wait(empty(ring.stage), ring.phase ^ 1u, abortp, 40)) {
                    fail(1, u);
                    break;
                }
                // both K blocks; the second of a unit that has only one is not used (past the last, zeros)
                const uint32_t kb = u < p.nkb_extra ? p.nkb_main + u : main_block(u);
                mbar_expect_tx(full(ring.stage), x_bytes);
                tma_load_3d(base + ring.stage * x_bytes, &map_x, 0, (int)m0, (int)kb, full(ring.stage));
                ++issued;
                ring.advance(p.su);
            }
            if (*abortp) {
                // The stages' barriers also count the dequant warps' arrivals, which may never come now: wait out the copies' time.
                const long long t0 = clock64();
                for (uint32_t i = issued > p.su ? issued - p.su : 0; i < issued; ++i)
                    while (!mbar_try(full(i % p.su), (i / p.su) & 1u))
                        if (clock64() - t0 > 20000000ll) break;
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------ MMA issuer ---
        const uint32_t idesc = (1u << 4) | ((p.x_rows >> 3) << 17) | ((uint32_t)(C::ROWS >> 4) << 24);
        // A wait and a commit cost this warp ~200 clocks each and the four MMAs of a K block ~80, so both come once per unit (with
        // a pair of rings and a commit per K block 77 x 4096 x 12288 took 0.25 us per K block, most of it here).
        const uint32_t x_lo0 = umma_desc_lo(base);
        RunRing ring;
        uint32_t acc = 0;  // the first MMA overwrites
        for (uint32_t u = u0; u < u1; ++u) {
            if (!mbar_wait(full(ring.stage), ring.phase, abortp)) {
                if (lane == 0) fail(2, u);
                break;
            }
            tcgen05_fence_after();
            const uint32_t a = tmem_a + ring.stage * C::UNIT_COLS, x_lo = x_lo0 + ring.stage * (x_bytes >> 4);
            tcgen05_block_ts_elect(tmem_base, a, x_lo, idesc, acc);
            if (unit_blocks(u) == 2) tcgen05_block_ts_elect(tmem_base, a + 32u, x_lo + (x_block >> 4), idesc, 1u);
            acc = 1;
            tcgen05_commit_elect(empty(ring.stage));
            ring.advance(p.su);
        }
        // Also after an abort: nothing may still read shared memory or write TMEM when the CTA winds down.
        tcgen05_commit_elect(acc_full);
        const long long t0 = clock64();
        while (!mbar_try(acc_full, 0u))
            if (clock64() - t0 > 4000000000ll) break;
        __syncwarp();
    } else if (warp == 2) {
        // ------------------------------------------------ TMA producer: packed weights ---
        if (lane == 0) {
            RunRing ring;
            uint32_t issued = 0;
            for (uint32_t u = u0; u < u1; ++u) {
                if (!mbar_wait(q_empty(ring.stage), ring.phase ^ 1u, abortp, 40)) {
                    fail(4, u);
                    break;
                }
                const uint32_t dst = off_q + ring.stage * C::Q_BYTES, bar = q_full(ring.stage);
                if (u >= p.nkb_extra) {
                    mbar_expect_tx(bar, C::Q_BYTES);
                    tma_load_2d(dst, &map_w, (int)(main_block(u) * 32), (int)n0, bar);
                } else if (p.sb_tiled) {  // 16 groups' words of every row
                    mbar_expect_tx(bar, C::Q_BYTES);
                    tma_load_2d(dst, &map_s, (int)(u * 64), (int)n0, bar);
                } else {
                    mbar_arrive(bar);
                }
                ++issued;
                ring.advance(C::SQ);
            }
            if (*abortp) {
                const long long t0 = clock64();
                for (uint32_t j = issued > (uint32_t)C::SQ ? issued - C::SQ : 0; j < issued; ++j)
                    while (!mbar_try(q_full(j % C::SQ), (j / C::SQ) & 1u))
                        if (clock64() - t0 > 20000000ll) break;
            }
        }
    } else if (warp == 3) {
        // Row scales once per CTA (every epilogue warp fetching them from the same few lines of L2 took 2 us per 16 rows).
        asm volatile("griddepcontrol.wait;" ::: "memory");
        for (uint32_t j = lane; j < p.x_rows; j += 32) {
            const float rs = m0 + j < p.M ? *(volatile const float *)(p.row_scale + m0 + j) : 0.0f;
            asm volatile("st.shared.f32 [%0], %1;" ::"r"(off_rs + j * 4), "f"(rs) : "memory");
        }
    } else {
        // ------------------------------------------------ dequant warps ---
        // A thread expands one weight row of its group's units.
        const uint32_t grp = (uint32_t)(warp - C::FIRST_DW) >> 2;
        const uint32_t row = quarter * 32 + lane;
        // 64-byte swizzle of the packed rows: 16-byte chunk c of row r lies at chunk c ^ ((r >> 1) & 3)
        const uint32_t q_row = off_q + row * 64, swz = (row >> 1) & 3u;
        // Scale words of unit u: of its four 32-column pieces. Fetched two units of this group ahead, into registers. (A warp that
        // copied them into the packed ring for all bounded the CTA: 32 rows are 32 lines, ~90 clocks a copy.)
        const uint32_t *sbrow = p.sb + (size_t)min(n0 + row, p.N - 1) * p.gpr;  // rows past N repeat the last
        auto scale_words = [&](uint32_t u) {
            uint4 s = make_uint4(0, 0, 0, 0);
            if (u >= u1 || u < p.nkb_extra) return s;
            const uint32_t k = main_block(u) * 64, g = k >> p.gshift;
            if (p.sb_words == 4) {
                s = __ldg(reinterpret_cast<const uint4 *>(sbrow + g));
            } else if (p.sb_words == 2) {
                const uint2 t = __ldg(reinterpret_cast<const uint2 *>(sbrow + g));
                s.x = s.y = t.x, s.z = s.w = t.y;
            } else {
                auto word = [&](uint32_t c) { return __ldg(sbrow + min((k + c) >> p.gshift, p.gpr - 1)); };
                s.x = word(0), s.y = p.gshift == 5 ? word(32) : s.x;
                s.z = p.gshift == 7 ? s.x : word(64), s.w = p.gshift == 5 ? word(96) : s.z;
            }
            return s;
        };
        uint4 s0 = scale_words(u0 + grp), s1 = scale_words(u0 + grp + C::NG);
        RunRing qr, ar;
        qr.advance(C::SQ, grp);
        for (uint32_t g = 0; g < grp; ++g) ar.advance(p.su);
        for (uint32_t u = u0 + grp; u < u1; u += C::NG) {
            if (!mbar_wait(q_full(qr.stage), qr.phase, abortp, 20)) {
                if (lane == 0) fail(6, u);
                break;
            }
            const uint4 s2 = scale_words(u + 2 * C::NG);
            const uint32_t q = q_row + qr.stage * C::Q_BYTES;
            const uint32_t d = tmem_a + lane_base + ar.stage * C::UNIT_COLS;
            uint4 w[4];
#pragma unroll
            for (uint32_t c = 0; c < 4; ++c) w[c] = lds128(q + ((c ^ swz) << 4));
            uint32_t o[32];
            if (u >= p.nkb_extra) {
                const uint32_t sc[4] = {scale_h2(s0.x), scale_h2(s0.y), scale_h2(s0.z), scale_h2(s0.w)};
                __syncwarp();
                if (lane == 0) mbar_arrive(q_empty(qr.stage));
#pragma unroll
                for (uint32_t h = 0; h < 2; ++h) {
                    const uint32_t a[8] = {w[2 * h].x, w[2 * h].y, w[2 * h].z, w[2 * h].w,
                                           w[2 * h + 1].x, w[2 * h + 1].y, w[2 * h + 1].z, w[2 * h + 1].w};
#pragma unroll
                    for (int v = 0; v < 8; ++v) expand_q4_word(a[v], sc[2 * h + (v >> 2)], o + 4 * v);
                    if (h == 0) {
                        if (!mbar_wait(empty(ar.stage), ar.phase ^ 1u, abortp, 20)) {
                            if (lane == 0) fail(7, u);
                            break;
                        }
                        __syncwarp();
                        tcgen05_fence_after();
                    }
                    tmem_st32(d + h * 32u, o);
                }
                if (*abortp) break;
            } else {
                if (p.sb_tiled) {
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        extra_pair(w[c].x, o[8 * c], o[8 * c + 1]), extra_pair(w[c].y, o[8 * c + 2], o[8 * c + 3]);
                        extra_pair(w[c].z, o[8 * c + 4], o[8 * c + 5]), extra_pair(w[c].w, o[8 * c + 6], o[8 * c + 7]);
                    }
                } else {
#pragma unroll
                    for (uint32_t t = 0; t < 16; ++t)
                        extra_pair(u * 16 + t < p.gpr ? __ldg(sbrow + u * 16 + t) : 0u, o[2 * t], o[2 * t + 1]);
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(q_empty(qr.stage));
                if (!mbar_wait(empty(ar.stage), ar.phase ^ 1u, abortp, 20)) {
                    if (lane == 0) fail(7, u);
                    break;
                }
                __syncwarp();
                tcgen05_fence_after();
                tmem_st32(d, o);
            }
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(full(ar.stage));
            s0 = s1, s1 = s2;
            qr.advance(C::SQ, C::NG);
#pragma unroll
            for (int g = 0; g < C::NG; ++g) ar.advance(p.su);
        }
        if (!mbar_wait(acc_full, 0u, abortp, 40) && lane == 0) fail(8, 0);
        __syncwarp();
        tcgen05_fence_after();
    }

    // ------------------------------------------------ epilogue ---
    // Columns of D (rows of X) in granules of 8; granule g is summed and stored by CTA g % split. Its other CTAs' parts arrive
    // in this CTA's shared memory, over the rings, once every CTA of the cluster is done with its own.
    const uint32_t grp = (uint32_t)(warp - C::FIRST_DW) >> 2;  // of the NG epilogue warps per lane quarter
    const uint32_t ngran = p.x_rows / 8, own = (ngran + p.split - 1) / p.split;
    const uint32_t mrow = quarter * 32 + lane;
    __syncthreads();
    if (p.split > 1) {
        cluster_sync_all();
        if (warp >= C::FIRST_DW) {
            for (uint32_t g = grp; g < ngran; g += C::NG) {
                const uint32_t owner = g % p.split;
                if (owner == rank) continue;
                float v[8];
                tmem_ld8(tmem_base + lane_base + g * 8u, v);
                const uint32_t src = rank < owner ? rank : rank - 1;
                const uint32_t dst = map_to_cta(base + (src * own + g / p.split) * (C::ROWS * 32) + mrow * 16, owner);
#pragma unroll
                for (uint32_t j = 0; j < 2; ++j)
                    asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(dst + j * (C::ROWS * 16)), "f"(v[4 * j]),
                                 "f"(v[4 * j + 1]), "f"(v[4 * j + 2]), "f"(v[4 * j + 3])
                                 : "memory");
            }
        }
        __syncwarp();
        cluster_sync_all();
    }
    if (warp >= C::FIRST_DW) {
        asm volatile("griddepcontrol.wait;" ::: "memory");  // y belongs to the stream's order
        const uint32_t n = n0 + mrow;
        for (uint32_t g = rank + grp * p.split; g < ngran; g += C::NG * p.split) {
            const uint32_t m = m0 + g * 8;
            float v[8], sum[8];
            tmem_ld8(tmem_base + lane_base + g * 8u, v);
            for (uint32_t s = 0; s < p.split; ++s) {
                float t[8];
                if (s == rank) {
#pragma unroll
                    for (uint32_t j = 0; j < 8; ++j) t[j] = v[j];
                } else {
                    const uint32_t part = base + ((s < rank ? s : s - 1) * own + g / p.split) * (C::ROWS * 32) + mrow * 16;
                    const uint4 lo = lds128(part), hi = lds128(part + C::ROWS * 16);
                    t[0] = __uint_as_float(lo.x), t[1] = __uint_as_float(lo.y), t[2] = __uint_as_float(lo.z), t[3] = __uint_as_float(lo.w);
                    t[4] = __uint_as_float(hi.x), t[5] = __uint_as_float(hi.y), t[6] = __uint_as_float(hi.z), t[7] = __uint_as_float(hi.w);
                }
#pragma unroll
                for (uint32_t j = 0; j < 8; ++j) sum[j] = s == 0 ? t[j] : sum[j] + t[j];
            }
            if (n < p.N) {
#pragma unroll
                for (uint32_t j = 0; j < 8; ++j) {
                    if (m + j >= p.M) break;
                    const size_t at = (size_t)(m + j) * p.N + n;
                    const float o = sum[j] * __uint_as_float(lds32(off_rs + (g * 8 + j) * 4));
                    if (p.out_bf16) {
                        static_cast<uint16_t *>(p.y)[at] = dev::f32_to_bf16_store(o);
                    } else {
                        static_cast<float *>(p.y)[at] = o;
                    }
                }
            }
        }
    }
    tcgen05_fence_before();
    __syncthreads();
    if (warp == 1) {
        tcgen05_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
    }
}

}  // namespace pf
}  // namespace tessl
