// 8-bit affine GEMV kernels for sm_100a.
//
//  * gemv_q8: the reference's Q8 convention (`nn::gemv_q8`, src/nn.rs:716-795;
//    kernels/gemv_q8.metal in the reference project): signed int8 codes,
//    f32 scale and zero per group, w = scale * (q - zero), f32 x, M = 1.
//  * gemm_q8_mlx: MLX's bank convention at eight bits: unsigned codes, one
//    bf16 (scale, bias) pair per group, w = scale * code + bias, bf16 x, M <= 8.
//
// Same shape as the Q4 kernels: a block owns R rows, its warps split K into
// 512-column chunks, a lane reads 16 codes per row and chunk with one 128-bit
// load and all R loads are issued before any is used. Codes become floats by a
// byte permute into the mantissa of 2^23 and one subtraction (exact).
#include <algorithm>

#include "q4_common.cuh"
#include "q4_gemv_tma.cuh"
#include "runtime.h"

namespace tessl {
namespace {

constexpr int kChunk8 = 512;  // 32 lanes x 16 codes

/// Byte B of `u` (an unsigned code 0..255) as the float 2^23 + code.
template <int B>
__device__ __forceinline__ float byte_to_f2p23(uint32_t u)
{
    return __uint_as_float(__byte_perm(u, 0x4b000000u, 0x7440u | B));
}

/// The 16 unsigned codes of `w` as exact floats.
__device__ __forceinline__ void codes16(const uint4 &w, float (&q)[16])
{
    const uint32_t words[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        q[4 * j + 0] = byte_to_f2p23<0>(words[j]) - 8388608.0f;
        q[4 * j + 1] = byte_to_f2p23<1>(words[j]) - 8388608.0f;
        q[4 * j + 2] = byte_to_f2p23<2>(words[j]) - 8388608.0f;
        q[4 * j + 3] = byte_to_f2p23<3>(words[j]) - 8388608.0f;
    }
}

struct Q8Params {
    const uint8_t *codes;
    const uint32_t *sb;     // mlx: bf16 (scale, bias) pairs
    const float *scales;    // i8: f32 tables
    const float *zeros;
    const void *x;
    void *y;
    uint32_t rows, cols, group_size;
    int out_bf16;
};

/// MLX-layout Q8, M activation rows, R output rows per block.
template <int M, int R>
__global__ void __launch_bounds__(128) q8_mlx_kernel(const Q8Params p)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
    const uint32_t rows = p.rows, cols = p.cols;
    const uint32_t row0 = blockIdx.x * R;
    const uint32_t gpr = cols / p.group_size;
    const uint16_t *x = static_cast<const uint16_t *>(p.x);
    float acc[R][M];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int m = 0; m < M; ++m) acc[r][m] = 0.0f;

    for (uint32_t k0 = warp * kChunk8 + lane * 16; k0 < cols; k0 += nwarps * kChunk8) {
        uint4 wq[R];
        uint32_t sbw[R];
        const uint32_t g = k0 / p.group_size;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const uint32_t row = min(row0 + r, rows - 1);
            wq[r] = dev::ldg_stream16(p.codes + (size_t)row * cols + k0);
            sbw[r] = dev::ldg_stream4(p.sb + (size_t)row * gpr + g);
        }
        float xs[M][16];
        float xsum[M];
#pragma unroll
        for (int m = 0; m < M; ++m) {
            const uint4 *xp = reinterpret_cast<const uint4 *>(x + (size_t)m * cols + k0);
            float t = 0.0f;
#pragma unroll
            for (int v = 0; v < 2; ++v) {
                const uint4 xv = __ldg(xp + v);
                const uint32_t xw[4] = {xv.x, xv.y, xv.z, xv.w};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    xs[m][8 * v + 2 * j] = dev::bf16_lo(xw[j]);
                    xs[m][8 * v + 2 * j + 1] = dev::bf16_hi(xw[j]);
                    t += xs[m][8 * v + 2 * j] + xs[m][8 * v + 2 * j + 1];
                }
            }
            xsum[m] = t;
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
            float q[16];
            codes16(wq[r], q);
            const float scale = dev::bf16_lo(sbw[r]), bias = dev::bf16_hi(sbw[r]);
#pragma unroll
            for (int m = 0; m < M; ++m) {
                float d0 = 0.0f, d1 = 0.0f;
#pragma unroll
                for (int i = 0; i < 16; i += 2) {
                    d0 = fmaf(xs[m][i], q[i], d0);
                    d1 = fmaf(xs[m][i + 1], q[i + 1], d1);
                }
                acc[r][m] = fmaf(scale, d0 + d1, fmaf(bias, xsum[m], acc[r][m]));
            }
        }
    }

    __shared__ float red[4][R * M];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int m = 0; m < M; ++m) {
            const float v = dev::warp_sum(acc[r][m]);
            if (lane == 0) red[warp][r * M + m] = v;
        }
    __syncthreads();
    const int t = threadIdx.x;
    if (t < R * M) {
        const int r = t / M, m = t % M;
        const uint32_t row = row0 + r;
        if (row < rows) {
            float v = red[0][t];
            for (int w = 1; w < nwarps; ++w) v += red[w][t];
            const size_t idx = (size_t)m * rows + row;
            if (p.out_bf16) {
                static_cast<uint16_t *>(p.y)[idx] = dev::f32_to_bf16_store(v);
            } else {
                static_cast<float *>(p.y)[idx] = v;
            }
        }
    }
}

// ------------------------------------------------------- reference convention ---

constexpr uint32_t kI8MaxCols = 8192;  // of the streamed kernel

/// Warps that share a row, 512 columns each or several times 512. The order of a row's sums is a function of cols alone, in both
/// kernels, so a slice of a bank has the bits of the whole, wherever its tables lie. Above 4096 columns the warps walk the row in even
/// rounds: with eight at nine chunks the second round would leave seven idle (1820 x 4608 6.3 us with eight, 5.6 with five; 7281 x 4608
/// 16.0 / 12.8; 1365 x 7168 5.4 with eight, 5.3 with seven).
uint32_t i8_warps_per_row(uint32_t cols)
{
    const uint32_t chunks = (cols + kChunk8 - 1) / kChunk8, rounds = (chunks + 7) / 8;
    return cols > kI8MaxCols ? 4 : (chunks + rounds - 1) / rounds;  // beyond the streamed kernel's rows
}

/// A lane's 16 signed codes of a row against its columns of x, added to `acc` with the group's scale and zero.
__device__ __forceinline__ void i8_dot16(const uint4 &q, const float (&xs)[16], float xsum, float scale, float zero, float &acc)
{
    // flipping the top bit of each byte gives code + 128 unsigned; it goes again with the 2^23 of the conversion
    const uint32_t u[4] = {q.x ^ 0x80808080u, q.y ^ 0x80808080u, q.z ^ 0x80808080u, q.w ^ 0x80808080u};
    float d0 = 0.0f, d1 = 0.0f;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        d0 = fmaf(xs[4 * j], byte_to_f2p23<0>(u[j]) - 8388736.0f, d0);
        d1 = fmaf(xs[4 * j + 1], byte_to_f2p23<1>(u[j]) - 8388736.0f, d1);
        d0 = fmaf(xs[4 * j + 2], byte_to_f2p23<2>(u[j]) - 8388736.0f, d0);
        d1 = fmaf(xs[4 * j + 3], byte_to_f2p23<3>(u[j]) - 8388736.0f, d1);
    }
    acc = fmaf(scale, fmaf(-zero, xsum, d0 + d1), acc);  // sum x * (q - zero)
}

/// Reference-convention Q8 (int8, f32 scale/zero, f32 x), vector path: needs
/// group_size and cols multiples of 16 so a lane's 16 codes share one group.
template <int R, int THREADS>
__global__ void __launch_bounds__(THREADS) q8_i8_kernel(const Q8Params p)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
    const uint32_t rows = p.rows, cols = p.cols;
    const uint32_t row0 = blockIdx.x * R;
    const uint32_t gpr = cols / p.group_size;
    const float *x = static_cast<const float *>(p.x);
    float acc[R];
#pragma unroll
    for (int r = 0; r < R; ++r) acc[r] = 0.0f;

    for (uint32_t k0 = warp * kChunk8 + lane * 16; k0 < cols; k0 += nwarps * kChunk8) {
        uint4 wq[R];
        float sc[R], zp[R];
        const uint32_t g = k0 / p.group_size;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const uint32_t row = min(row0 + r, rows - 1);
            wq[r] = dev::ldg_stream16(p.codes + (size_t)row * cols + k0);
            sc[r] = __ldg(p.scales + (size_t)row * gpr + g);
            zp[r] = __ldg(p.zeros + (size_t)row * gpr + g);
        }
        float xs[16];
        float xsum = 0.0f;
        const float4 *xp = reinterpret_cast<const float4 *>(x + k0);
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            const float4 xv = __ldg(xp + v);
            xs[4 * v] = xv.x, xs[4 * v + 1] = xv.y, xs[4 * v + 2] = xv.z, xs[4 * v + 3] = xv.w;
            xsum += (xv.x + xv.y) + (xv.z + xv.w);
        }
#pragma unroll
        for (int r = 0; r < R; ++r) i8_dot16(wq[r], xs, xsum, sc[r], zp[r], acc[r]);
    }
    __shared__ float red[THREADS / 32][R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const float v = dev::warp_sum(acc[r]);
        if (lane == 0) red[warp][r] = v;
    }
    __syncthreads();
    const int t = threadIdx.x;
    if (t < R && row0 + t < rows) {
        float v = red[0][t];
        for (int w = 1; w < nwarps; ++w) v += red[w][t];
        static_cast<float *>(p.y)[row0 + t] = v;
    }
}

// ------------------------------------------------ reference convention, streamed ---

constexpr uint32_t kI8Rows = 4;                  // rows of a stage per team
constexpr uint32_t kI8Consumers = 16, kI8Threads = (1 + kI8Consumers) * 32;
constexpr uint32_t kI8MaxStages = 32, kI8Ring = 200 * 1024, kI8StageMin = 8 * 1024, kI8StageBest = 16 * 1024, kI8StageMax = 24 * 1024;

struct I8Plan {
    uint32_t per_row;     // warps that share a row, 512 columns each (or several times 512)
    uint32_t share;       // groups of such warps (teams) that share a stage, kI8Rows rows for each
    uint32_t sets;        // sets of `share` teams, which take turns at the stages
    uint32_t stages;      // a multiple of sets
    uint32_t stage_bytes;
    uint32_t row_step;    // rows per block, a multiple of kI8Rows
    uint32_t *status;
};

/// Reference-convention Q8 (int8, f32 scale/zero, f32 x): groups and rows of a multiple of 16 columns, tables at 16-byte
/// boundaries, at most 8192 columns.
///
/// HBM-bound in intent (18.9 MB at 4096 x 4096): one block per SM owns a run of rows and a producer warp streams them, about 16 KB at a
/// time, with three bulk copies (codes, scales, zeros: each contiguous) into a ring of up to 200 KB; 44 KB in flight would cover
/// bandwidth times latency. Smaller stages pay the copy unit per copy (4 KB at 1024 columns: 14336 rows 11.2 us against 7.3), larger
/// ones start late (32 KB at 4096 x 4096: 7.9 us against 7.0). Consumer warps keep x in registers, each lane the 16 columns it has of
/// every row (rows of up to 4096 columns). q8_i8_kernel issues its loads per two or eight rows and waits for them, and reads x from
/// L1 again for each.
/// Before (q8_i8_kernel) -> here, back to back: 4096 x 4096 9.6 -> 7.0 us, 14336 x 4096 24.8 -> 17.0 (3.9 TB/s), 14336 x 1024 9.4 -> 6.7,
/// 2048 x 2560 4.5 -> 3.9, 4096 x 512 5.4 -> 2.6, 21845 x 1536 15.0 -> 11.9; relative error against 64 bits 1.9e-7 -> 1.1e-7 (signed codes
/// are summed, not codes + 128).
/// What bounds it now: the FMA and ALU pipes (a byte permute, a subtraction and an FMA per code) and ~2 us of start. Rows dealt out
/// one by one instead of four by four change nothing or lose (2048 x 4096 4.65 -> 4.9): a block's time goes by its stages.
/// A ring slot belongs to one set of teams, so a parity that a team waits for is never a round behind.
/// A row's sums are reduced over the lanes, then over the warps in order.
__global__ void __launch_bounds__(kI8Threads, 1) q8_i8_stream_kernel(const Q8Params p, const I8Plan plan)
{
    extern __shared__ __align__(128) uint8_t ring[];
    __shared__ __align__(8) uint64_t bars[2 * kI8MaxStages];
    __shared__ float red[2][kI8Consumers][kI8Rows];
    __shared__ int abort_flag;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t cols = p.cols, gpr = cols / p.group_size;
    const uint32_t first = blockIdx.x * plan.row_step, last = min(first + plan.row_step, p.rows);
    const uint32_t stage_rows = plan.share * kI8Rows, nst = (last - first + stage_rows - 1) / stage_rows;
    const uint32_t bar0 = q4k::smem_u32(bars), ring0 = q4k::smem_u32(ring);
    auto full = [&](uint32_t s) { return bar0 + 8 * s; };
    auto empty = [&](uint32_t s) { return bar0 + 8 * (kI8MaxStages + s); };
    if (threadIdx.x < plan.stages) {
        q4k::mbar_init(full(threadIdx.x), 1), q4k::mbar_init(empty(threadIdx.x), plan.share * plan.per_row);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (threadIdx.x == 0) abort_flag = 0;
    __syncthreads();
    volatile int *abortp = &abort_flag;
    auto fail = [&](uint32_t role, uint32_t where) {
        *abortp = 1;
        *(volatile uint32_t *)plan.status = (role << 24) | (where & 0xffffffu);
    };
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const uint32_t off_sc = stage_rows * cols, off_zp = off_sc + stage_rows * gpr * 4;

    if (warp == 0) {
        uint32_t slot = 0, phase = 0, issued = 0;
        for (uint32_t st = 0; st < nst; ++st) {
            if (!q4k::mbar_wait(empty(slot), phase ^ 1u, abortp, 20)) {
                if (lane == 0) fail(1, st);
                break;
            }
            __syncwarp();
            const uint32_t row = first + st * stage_rows, rows = min(stage_rows, last - row);
            const uint32_t dst = ring0 + slot * plan.stage_bytes, code_bytes = rows * cols, tab_bytes = rows * gpr * 4;
            const size_t g0 = (size_t)row * gpr;
            const bool whole = tab_bytes % 16 == 0;  // the last rows' tables may not be a whole number of 16 bytes
            if (!whole) {
                for (uint32_t i = lane; i < rows * gpr; i += 32) {
                    asm volatile("st.shared.f32 [%0], %1;" ::"r"(dst + off_sc + i * 4), "f"(p.scales[g0 + i]) : "memory");
                    asm volatile("st.shared.f32 [%0], %1;" ::"r"(dst + off_zp + i * 4), "f"(p.zeros[g0 + i]) : "memory");
                }
                __syncwarp();
            }
            if (lane == 0) {
                q4k::mbar_expect_tx(full(slot), code_bytes + (whole ? 2 * tab_bytes : 0));
                q4k::bulk_g2s(dst, p.codes + (size_t)row * cols, code_bytes, full(slot));
                if (whole) {
                    q4k::bulk_g2s(dst + off_sc, p.scales + g0, tab_bytes, full(slot));
                    q4k::bulk_g2s(dst + off_zp, p.zeros + g0, tab_bytes, full(slot));
                }
            }
            ++issued;
            if (++slot == plan.stages) slot = 0, phase ^= 1u;
        }
        if (lane == 0 && *abortp) {  // let what is in flight land before the block may exit
            const long long t0 = clock64();
            for (uint32_t i = issued > plan.stages ? issued - plan.stages : 0; i < issued; ++i)
                while (!q4k::mbar_try(full(i % plan.stages), (i / plan.stages) & 1u))
                    if (clock64() - t0 > 20000000ll) break;
        }
        return;
    }
    const uint32_t w = warp - 1, team = w / plan.per_row, part = w - team * plan.per_row;
    if (team >= plan.share * plan.sets) return;
    const uint32_t set = team / plan.share, seat = team - set * plan.share;
    const uint32_t k_first = part * kChunk8 + lane * 16, k_step = plan.per_row * kChunk8, nch = (cols + k_step - 1) / k_step;
    const float *x = static_cast<const float *>(p.x);
    float xs[16], xsum = 0.0f;
    auto load_x = [&](uint32_t k) {
        xsum = 0.0f;
#pragma unroll
        for (uint32_t v = 0; v < 4; ++v) {
            const uint4 u = k < cols ? dev::ld_after_wait16(x + k + 4 * v) : make_uint4(0, 0, 0, 0);
            xs[4 * v] = __uint_as_float(u.x), xs[4 * v + 1] = __uint_as_float(u.y);
            xs[4 * v + 2] = __uint_as_float(u.z), xs[4 * v + 3] = __uint_as_float(u.w);
            xsum += (xs[4 * v] + xs[4 * v + 1]) + (xs[4 * v + 2] + xs[4 * v + 3]);
        }
    };
    load_x(k_first);
    uint32_t g = min(k_first, cols - 1) / p.group_size;
    uint32_t slot = set, phase = 0, parity = 0;
    bool dead = false;
    for (uint32_t st = set; st < nst; st += plan.sets, parity ^= 1u) {
        // After a wait that ran out the team goes on to its barriers, without waiting for copies: no warp is left behind at one.
        if (!dead && !__all_sync(0xffffffffu, q4k::mbar_wait(full(slot), phase, abortp, 0))) {
            if (lane == 0) fail(2, st);
            dead = true;
        }
        const uint32_t row0 = first + st * stage_rows + seat * kI8Rows;
        if (row0 >= last) break;  // the last stage has no rows for this team
        const uint32_t src = ring0 + slot * plan.stage_bytes, rt0 = seat * kI8Rows;
        float acc[kI8Rows] = {0.0f, 0.0f, 0.0f, 0.0f};
        for (uint32_t c = 0; c < nch; ++c) {
            const uint32_t k = k_first + c * k_step;
            if (k >= cols) break;  // the bytes there are another row's
            if (nch > 1) load_x(k), g = k / p.group_size;
#pragma unroll
            for (uint32_t r = 0; r < kI8Rows; ++r) {
                const uint4 q = q4k::lds128(src + (rt0 + r) * cols + k);
                float sc, zp;
                asm volatile("ld.shared.f32 %0, [%1];" : "=f"(sc) : "r"(src + off_sc + ((rt0 + r) * gpr + g) * 4) : "memory");
                asm volatile("ld.shared.f32 %0, [%1];" : "=f"(zp) : "r"(src + off_zp + ((rt0 + r) * gpr + g) * 4) : "memory");
                i8_dot16(q, xs, xsum, sc, zp, acc[r]);
            }
        }
        __syncwarp();
        if (lane == 0) q4k::mbar_arrive(empty(slot));
        // Lanes: four rows halve to one per lane (lane bits 4 and 3 pick the row), then the other bits.
#pragma unroll
        for (int h = kI8Rows / 2; h > 0; h >>= 1) {
            const bool up = (lane & (8 * h)) != 0;
#pragma unroll
            for (int r = 0; r < h; ++r) {
                const float send = up ? acc[r] : acc[r + h], keep = up ? acc[r + h] : acc[r];
                acc[r] = keep + __shfl_xor_sync(0xffffffffu, send, 8 * h);
            }
        }
        float v = acc[0];
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (plan.per_row > 1) {
            if ((lane & 7) == 0) red[parity][w][lane >> 3] = v;
            // the team's warps; this buffer is written again after the next of these barriers only
            asm volatile("bar.sync %0, %1;" ::"r"(1 + team), "r"(plan.per_row * 32) : "memory");
            if (part == 0 && lane < kI8Rows) {
                v = red[parity][w][lane];
                for (uint32_t i = 1; i < plan.per_row; ++i) v += red[parity][w + i][lane];
            }
        } else {
            v = __shfl_sync(0xffffffffu, v, (lane & 3) * 8);
        }
        const uint32_t row = row0 + lane;
        if (part == 0 && lane < kI8Rows && row < last) static_cast<float *>(p.y)[row] = v;
        slot += plan.sets;
        if (slot >= plan.stages) slot -= plan.stages, phase ^= 1u;
    }
}

Result launch_i8_stream(TesslRuntime *rt, const Q8Params &p)
{
    I8Plan plan{};
    const uint32_t gpr = p.cols / p.group_size;
    plan.per_row = i8_warps_per_row(p.cols);
    const uint32_t teams = kI8Consumers / plan.per_row;
    // Stages of 8 to 24 KB of codes: as many teams busy as can be, then the stage nearest to 16 KB. (With shares that divide the teams
    // only, five teams over 1280 .. 1536 columns took stages of 5 KB: 21845 x 1536 16.3 us, 11.9 now, 15.0 with q8_i8_kernel.)
    plan.share = teams, plan.sets = 1;  // narrow rows: no stage is large
    uint32_t used = 0, off = 0;
    for (uint32_t d = 1; d <= teams; ++d) {
        const uint32_t codes = d * kI8Rows * p.cols, n = teams / d * d;
        if (codes > kI8StageMax && d > 1) break;
        const uint32_t o = codes < kI8StageBest ? kI8StageBest - codes : codes - kI8StageBest;
        if (codes >= kI8StageMin && (n > used || (n == used && o < off))) plan.share = d, plan.sets = teams / d, used = n, off = o;
    }
    plan.stage_bytes = plan.share * kI8Rows * (p.cols + 8 * gpr);  // a multiple of 16; at most 48 KB
    plan.stages = std::min<uint32_t>(kI8MaxStages, kI8Ring / plan.stage_bytes) / plan.sets * plan.sets;
    const uint32_t batches = (p.rows + kI8Rows - 1) / kI8Rows, blocks = std::min<uint32_t>(batches, (uint32_t)rt->sm_count);
    plan.row_step = (batches + blocks - 1) / blocks * kI8Rows;
    plan.status = rt->status_dev;
    const size_t smem = (size_t)plan.stages * plan.stage_bytes;
    TESSL_TRY(smem_opt_in(rt, reinterpret_cast<const void *>(q8_i8_stream_kernel), smem, "gemv_q8: shared memory opt-in", true));
    return launch_pdl(rt, "gemv_q8 launch", q8_i8_stream_kernel, dim3((p.rows + plan.row_step - 1) / plan.row_step), dim3(kI8Threads), smem,
                      p, plan);
}

/// Any group size and alignment: one warp per row, lanes stride the columns,
/// w = scale * (q - zero) per element as the reference's scalar path does
/// (kernels/gemv_q8.metal:101-113).
__global__ void __launch_bounds__(128) q8_i8_scalar_kernel(const Q8Params p)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t row = blockIdx.x * (blockDim.x >> 5) + warp;
    if (row >= p.rows) return;
    const uint32_t cols = p.cols, gpr = cols / p.group_size;
    const int8_t *q = reinterpret_cast<const int8_t *>(p.codes) + (size_t)row * cols;
    const float *x = static_cast<const float *>(p.x);
    float acc = 0.0f;
    for (uint32_t c = lane; c < cols; c += 32) {
        const size_t gi = (size_t)row * gpr + c / p.group_size;
        const float w = p.scales[gi] * ((float)q[c] - p.zeros[gi]);
        acc = fmaf(w, x[c], acc);
    }
    acc = dev::warp_sum(acc);
    if (lane == 0) static_cast<float *>(p.y)[row] = acc;
}

template <int M, int R>
Result launch_mlx(TesslRuntime *rt, const Q8Params &p, int warps)
{
    q8_mlx_kernel<M, R><<<(p.rows + R - 1) / R, warps * 32, 0, rt->stream>>>(p);
    rt->dispatch_count += 1;
    return cuda_check(rt, cudaGetLastError(), "q8_mlx launch");
}

}  // namespace

namespace nn {

Result gemv_q8(TesslRuntime *rt, const TesslBuf &packed, const TesslBuf &scales, const TesslBuf &zeros,
               const TesslBuf &x, const TesslBuf &y, uint32_t rows, uint32_t cols, uint32_t group_size)
{
    if (group_size == 0) return "gemv_q8: group_size must be non-zero";
    if (cols % group_size != 0) {
        return fmt("gemv_q8: cols %u is not a multiple of group_size %u; the kernel would silently drop the ragged "
                   "tail group",
                   cols, group_size);
    }
    const uint64_t weights = elems(rows, cols);
    const uint64_t groups = elems(rows, cols / group_size);
    TESSL_TRY(require(packed, weights, 1, "gemv_q8 packed"));
    TESSL_TRY(require(scales, groups, 4, "gemv_q8 scales"));
    TESSL_TRY(require(zeros, groups, 4, "gemv_q8 zeros"));
    TESSL_TRY(require(x, cols, 4, "gemv_q8 x"));
    TESSL_TRY(require(y, rows, 4, "gemv_q8 y"));
    if (rows == 0) return ok();
    const Named writes[] = {{"y", &y}};
    const Named reads[] = {{"packed", &packed}, {"scales", &scales}, {"zeros", &zeros}, {"x", &x}};
    TESSL_TRY(require_disjoint_writes("gemv_q8", writes, 1, reads, 4));
    Q8Params p{};
    p.codes = static_cast<const uint8_t *>(packed.ptr);
    p.scales = static_cast<const float *>(scales.ptr);
    p.zeros = static_cast<const float *>(zeros.ptr);
    p.x = x.ptr;
    p.y = y.ptr;
    p.rows = rows, p.cols = cols, p.group_size = group_size;
    const bool vec = group_size % 16 == 0 && cols % 16 == 0 && ((uintptr_t)packed.ptr & 15u) == 0 &&
                     ((uintptr_t)x.ptr & 15u) == 0 && cols > 0;
    if (vec) {
        // The tables of every fourth row start at 16-byte boundaries if the buffers do. For small calls the start of the ring costs more
        // than it gives: 512 x 1024 2.35 us without it, 2.55 with it, 513 x 4096 2.8 / 2.6; 192 x 8192 3.0 / 3.4, 384 x 8192 4.0 / 3.7.
        const uint32_t warps = i8_warps_per_row(cols);
        const uint64_t least = cols <= 4096 ? 1u << 20 : 2u << 20;
        if (cols <= kI8MaxCols && weights >= least && (((uintptr_t)scales.ptr | (uintptr_t)zeros.ptr) & 15u) == 0)
            return launch_i8_stream(rt, p);
        // Blocks of up to four warps have instantiations of their own: with a bound of 256 threads the compiler schedules the loop
        // differently, and 21 x 12288 took 4.4 us instead of 4.2.
        auto go = [&](auto kernel, uint32_t r) { kernel<<<(rows + r - 1) / r, warps * 32, 0, rt->stream>>>(p); };
        if ((uint64_t)rows >= (uint64_t)(8 * 3 * rt->sm_count)) {
            warps <= 4 ? go(q8_i8_kernel<8, 128>, 8) : go(q8_i8_kernel<8, 256>, 8);
        } else {
            warps <= 4 ? go(q8_i8_kernel<2, 128>, 2) : go(q8_i8_kernel<2, 256>, 2);
        }
    } else {
        q8_i8_scalar_kernel<<<(rows + 3) / 4, 128, 0, rt->stream>>>(p);
    }
    rt->dispatch_count += 1;
    return cuda_check(rt, cudaGetLastError(), "gemv_q8 launch");
}

Result gemm_q8_mlx(TesslRuntime *rt, const TesslBuf &codes, const TesslBuf &sb, const TesslBuf &x_bf16,
                   const TesslBuf &y, const TesslQuantShape &shape, uint32_t m, OutKind out)
{
    const char *entry = "gemm_q8_mlx";
    if (m == 0) return ok();
    if (m > TESSL_GEMM_Q4_MLX_MAX_M) return fmt("%s: M = %u exceeds the small-batch limit %u", entry, m, 8u);
    TESSL_TRY(quant_shape_validate(shape, entry));
    if (shape.group_size % 32 != 0 || 512 % shape.group_size != 0) {
        return fmt("%s: group_size %u is outside the MLX kernel domain {32, 64, 128, 256, 512}", entry,
                   shape.group_size);
    }
    TESSL_TRY(require(codes, elems(shape.rows, shape.cols), 1, What(entry) + " codes"));
    TESSL_TRY(require(sb, elems(shape.rows, shape.cols / shape.group_size), 4,
                      What(entry) + " scales_biases (bfloat2 per group)"));
    TESSL_TRY(require(x_bf16, elems(m, shape.cols), 2, What(entry) + " x_bf16"));
    TESSL_TRY(require(y, elems(m, shape.rows), out == OUT_BF16 ? 2 : 4, What(entry) + " y"));
    if (shape.rows == 0) return ok();
    const Named writes[] = {{"y", &y}};
    const Named reads[] = {{"codes", &codes}, {"scales_biases", &sb}, {"x_bf16", &x_bf16}};
    TESSL_TRY(require_disjoint_writes(entry, writes, 1, reads, 3));
    TESSL_TRY(require_aligned16(codes, What(entry) + " codes"));
    TESSL_TRY(require_aligned16(x_bf16, What(entry) + " x_bf16"));
    {
        // rows of 512 .. 4096 codes in groups of 32 or 64: the tensor-core GEMV kernel (q4_gemv_mma.cuh)
        bool handled = false;
        TESSL_TRY(q8_mlx_mma(rt, codes, sb, x_bf16, y, shape.rows, shape.cols, shape.group_size, m, out, &handled));
        if (handled) return ok();
    }
    Q8Params p{};
    p.codes = static_cast<const uint8_t *>(codes.ptr);
    p.sb = static_cast<const uint32_t *>(sb.ptr);
    p.x = x_bf16.ptr;
    p.y = y.ptr;
    p.rows = shape.rows, p.cols = shape.cols, p.group_size = shape.group_size;
    p.out_bf16 = out == OUT_BF16;
    const int warps = (int)std::max<uint32_t>(1u, std::min<uint32_t>(4u, (shape.cols + kChunk8 - 1) / kChunk8));
    const bool big = (uint64_t)shape.rows >= (uint64_t)(8 * 3 * rt->sm_count);
    switch (m) {
    case 1: return big ? launch_mlx<1, 8>(rt, p, warps) : launch_mlx<1, 2>(rt, p, warps);
    case 2: return big ? launch_mlx<2, 8>(rt, p, warps) : launch_mlx<2, 2>(rt, p, warps);
    case 3: return launch_mlx<3, 4>(rt, p, warps);
    case 4: return launch_mlx<4, 4>(rt, p, warps);
    case 5: return launch_mlx<5, 2>(rt, p, warps);
    case 6: return launch_mlx<6, 2>(rt, p, warps);
    case 7: return launch_mlx<7, 2>(rt, p, warps);
    default: return launch_mlx<8, 2>(rt, p, warps);
    }
}

}  // namespace nn
}  // namespace tessl
