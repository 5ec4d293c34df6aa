// MLX affine Q4 GEMV (M = 1) and small-batch GEMM (M <= 8) for sm_100a: the host-side wrappers that mirror
// the reference's `nn::gemv_q4_mlx_*`, `nn::gemm_q4_mlx` and `nn::embed_lookup_q4_mlx` (src/nn.rs:3592-4619 of
// the reference project): validation in the reference's order and wording, the choice of kernel and
// instantiation, the launch.
//
// Kernels: q4_gemv_mma.cuh (one row of x at the common widths: dot products on the tensor cores, bulk-copy ring; also
// the MLX Q8 mode and the column-sharded launches that exchange their outputs over NVLink), q4_batch_mma.cuh (2..8 rows,
// and one row at the other widths: the same arithmetic, any whole number of 256-column chunks), and the FMA-pipe
// fallbacks q4_gemv_tma.cuh, q4_gemv_warp.cuh, q4_gemv_main.cuh / q4_gemv_kernel.cuh for the shapes these do not take.
#include "q4_gemv_main.cuh"
#include "q4_gemv_warp.cuh"
#include "q4_gemv_tma.cuh"
#include "q4_gemv_mma.cuh"
#include "q4_batch_mma.cuh"

#include <cstdio>
#include <cstdlib>
#include "runtime.h"
#include "tensormap.h"

namespace tessl {
namespace {

using q4k::EPI_ADD_RESID;
using q4k::EPI_GATE_UP_GELU;
using q4k::EPI_GATE_UP_SILU;
using q4k::EPI_STORE;
using Q4Seg = q4k::Seg;
using Q4GemvParams = q4k::Params;

/// silu(gate) * up (or GELU), four neighbouring elements per thread where the buffers allow 16-byte accesses (VEC = 4).
/// Bound by its 10 (bf16) or 12 bytes per element; with one element per thread a prompt's 509 x 6144 was bound by its
/// load instructions.
template <int VEC>
__global__ void __launch_bounds__(256) swiglu_kernel(const float *gate, const float *up, void *out, uint32_t n, int out_bf16, int gelu)
{
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const uint64_t i = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) * VEC;
    if (i >= n) return;
    float g[VEC], u[VEC];
    if constexpr (VEC == 4) {
        const uint4 a = dev::ld_after_wait16(gate + i), b = dev::ld_after_wait16(up + i);
        g[0] = __uint_as_float(a.x), g[1] = __uint_as_float(a.y), g[2] = __uint_as_float(a.z), g[3] = __uint_as_float(a.w);
        u[0] = __uint_as_float(b.x), u[1] = __uint_as_float(b.y), u[2] = __uint_as_float(b.z), u[3] = __uint_as_float(b.w);
    } else {
        g[0] = *(volatile const float *)(gate + i), u[0] = *(volatile const float *)(up + i);
    }
    float v[VEC];
#pragma unroll
    for (int k = 0; k < VEC; ++k) v[k] = (gelu ? dev::gelu_pytorch_tanh(g[k]) : dev::silu(g[k])) * u[k];
    if (out_bf16) {
        uint16_t h[VEC];
#pragma unroll
        for (int k = 0; k < VEC; ++k) h[k] = dev::f32_to_bf16_store(v[k]);
        uint16_t *o = static_cast<uint16_t *>(out) + i;
        if constexpr (VEC == 4) {
            *reinterpret_cast<uint2 *>(o) = make_uint2((uint32_t)h[0] | ((uint32_t)h[1] << 16), (uint32_t)h[2] | ((uint32_t)h[3] << 16));
        } else {
            o[0] = h[0];
        }
    } else {
        float *o = static_cast<float *>(out) + i;
        if constexpr (VEC == 4) {
            *reinterpret_cast<float4 *>(o) = make_float4(v[0], v[1], v[2], v[3]);
        } else {
            o[0] = v[0];
        }
    }
}

Result launch_swiglu(TesslRuntime *rt, const char *what, const float *gate, const float *up, void *out, uint32_t n, int out_bf16, int gelu)
{
    const bool vec = n % 4 == 0 && (((uintptr_t)gate | (uintptr_t)up) & 15u) == 0 && ((uintptr_t)out & (out_bf16 ? 7u : 15u)) == 0;
    const uint32_t work = vec ? n / 4 : n;
    const dim3 grid(work / 256 + (work % 256 != 0));
    if (vec) return launch_pdl(rt, what, swiglu_kernel<4>, grid, dim3(256), 0, gate, up, out, n, out_bf16, gelu);
    return launch_pdl(rt, what, swiglu_kernel<1>, grid, dim3(256), 0, gate, up, out, n, out_bf16, gelu);
}

__global__ void q4_unpack_kernel(const uint8_t *packed, uint8_t *out, uint64_t n_bytes)
{
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_bytes) return;
    const uint8_t b = packed[i];
    out[2 * i] = b & 0x0f;
    out[2 * i + 1] = b >> 4;
}

/// Geometry of the staged layout for rows of `cols` columns and groups of `group` (see q4_gemv_mma.cuh).
struct StagedGeom {
    uint32_t row_bytes, pair_pitch, sb_row_bytes, unit_bytes;
};
__host__ __device__ inline StagedGeom staged_geom(uint32_t cols, uint32_t group)
{
    StagedGeom g;
    g.row_bytes = cols / 2;
    g.pair_pitch = 2 * g.row_bytes + q4m::kRowPad;
    g.sb_row_bytes = (cols / group) * 4;
    g.unit_bytes = 4 * g.pair_pitch + 8 * g.sb_row_bytes;
    return g;
}

/// One thread per 16 bytes of the staged image: a piece of a packed row, of a pad, or of a scale/bias row.
__global__ void q4_repack_staged_kernel(const uint4 *packed, const uint4 *sb, uint4 *out, uint32_t rows, uint32_t cols,
                                        uint32_t group, uint64_t n16)
{
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n16) return;
    const StagedGeom g = staged_geom(cols, group);
    const uint64_t byte = i * 16;
    const uint32_t unit = (uint32_t)(byte / g.unit_bytes), o = (uint32_t)(byte % g.unit_bytes);
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (o < 4 * g.pair_pitch) {
        const uint32_t pair = o / g.pair_pitch, within = o % g.pair_pitch;
        if (within < 2 * g.row_bytes) {
            const uint32_t row = 8 * unit + 2 * pair + within / g.row_bytes;
            if (row < rows) v = packed[((size_t)row * g.row_bytes + within % g.row_bytes) / 16];
        }
    } else {
        const uint32_t so = o - 4 * g.pair_pitch;
        const uint32_t row = 8 * unit + so / g.sb_row_bytes;
        if (row < rows) v = sb[((size_t)row * g.sb_row_bytes + so % g.sb_row_bytes) / 16];
    }
    out[i] = v;
}

__global__ void q4_dequant_kernel(const uint8_t *packed, const uint32_t *sb, float *out, uint32_t rows, uint32_t cols,
                                  uint32_t group_shift)
{
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;  // byte index
    if (i >= (uint64_t)rows * cols / 2) return;
    const uint64_t e = 2 * i;
    const uint32_t row = (uint32_t)(e / cols), col = (uint32_t)(e % cols);
    const uint32_t pair = sb[(size_t)row * (cols >> group_shift) + (col >> group_shift)];
    const float scale = dev::bf16_lo(pair), bias = dev::bf16_hi(pair);
    const uint8_t b = packed[i];
    // Separate multiply and add, as the reference's host dequant (scale * q is exact anyway).
    out[e] = __fadd_rn(__fmul_rn(scale, (float)(b & 0x0f)), bias);
    out[e + 1] = __fadd_rn(__fmul_rn(scale, (float)(b >> 4)), bias);
}

/// One thread per 32 consecutive columns of one token's row (16 packed bytes, never more than one
/// quantization group): a 128-bit load of the nibbles, one scale/bias pair, eight 128-bit stores.
/// A token id outside the table gives a row of zeros (kernels/embed_lookup.metal:24-27 of the
/// reference project).
__global__ void embed_lookup_q4_mlx_kernel(const uint8_t *packed, const uint32_t *sb, const uint32_t *token_ids, float *out,
                                           uint32_t hidden, uint32_t group_shift, uint32_t vocab, uint64_t total32)
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total32) return;
    const uint32_t per_row = hidden / 32;
    const uint32_t m = (uint32_t)(i / per_row), c = (uint32_t)(i % per_row);
    const uint32_t tid = *(volatile const uint32_t *)(token_ids + m);
    float4 *o = reinterpret_cast<float4 *>(out + (size_t)m * hidden + (size_t)c * 32);
    if (tid >= vocab) {
#pragma unroll
        for (int k = 0; k < 8; ++k) o[k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        return;
    }
    const uint4 w = dev::ldg_stream16(packed + (size_t)tid * (hidden / 2) + (size_t)c * 16);
    const uint32_t pair = sb[(size_t)tid * (hidden >> group_shift) + ((c * 32) >> group_shift)];
    const float scale = dev::bf16_lo(pair), bias = dev::bf16_hi(pair);
    const uint32_t words[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        float v[8];
#pragma unroll
        for (int n = 0; n < 8; ++n) v[n] = __fadd_rn(__fmul_rn(scale, (float)((words[k] >> (4 * n)) & 15u)), bias);
        o[2 * k] = make_float4(v[0], v[1], v[2], v[3]);
        o[2 * k + 1] = make_float4(v[4], v[5], v[6], v[7]);
    }
}

uint32_t log2_u32(uint32_t v)
{
    uint32_t s = 0;
    while ((1u << s) < v) ++s;
    return s;
}

template <int M, int NB, int R, int NCH>
Result launch_one(TesslRuntime *rt, Q4GemvParams &p, int warps)
{
    auto kernel = q4k::q4_gemv_kernel<M, NB, R, NCH>;
    uint32_t groups = 0;
    for (int s = 0; s < p.nseg; ++s) {
        p.seg[s].group_begin = groups;
        groups += (p.seg[s].rows + R - 1) / R;
    }
    p.ngroups = groups;
    if (groups == 0) return ok();
    // Persistent grid: as many blocks as stay resident, each walking its share of the groups.
    static int per_sm[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    if (per_sm[warps] == 0) {
        int n = 0;
        cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, warps * 32, 0);
        if (e != cudaSuccess || n < 1) n = 1;
        per_sm[warps] = n;
    }
    const uint32_t grid = std::min<uint32_t>(groups, (uint32_t)(rt->sm_count * per_sm[warps]));
    kernel<<<grid, warps * 32, 0, rt->stream>>>(p);
    rt->dispatch_count += 1;
    return cuda_check(rt, cudaGetLastError(), "q4_gemv launch");
}

template <int NB, int R, int NCH>
Result launch_warp(TesslRuntime *rt, const Q4GemvParams &p)
{
    auto kernel = q4k::q4_gemv_warp_kernel<NB, R, NCH>;
    static int per_sm = 0;
    if (per_sm == 0) {
        int n = 0;
        cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, 32, 0);
        per_sm = (e != cudaSuccess || n < 1) ? 1 : n;
    }
    q4k::WarpParams wp{};
    uint64_t total_rows = 0;
    for (int s = 0; s < p.nseg; ++s) total_rows += p.seg[s].rows;
    if (total_rows == 0) return ok();
    // One wave: every warp gets the same number of consecutive rows.
    const uint64_t capacity = (uint64_t)rt->sm_count * per_sm;
    uint64_t r = (total_rows + capacity - 1) / capacity;
    r = (r + R - 1) / R * R;
    uint32_t blocks = 0;
    for (int s = 0; s < p.nseg; ++s) {
        const Q4Seg &a = p.seg[s];
        wp.seg[s] = q4k::WarpSeg{a.packed0, a.sb0, a.packed1, a.sb1, a.out, a.resid, a.rows, blocks};
        blocks += (uint32_t)((a.rows + r - 1) / r);
    }
    wp.nseg = p.nseg;
    wp.rows_per_block = (uint32_t)r;
    wp.x = p.x, wp.cols = p.cols, wp.group_shift = p.group_shift, wp.epi = p.epi, wp.out_bf16 = p.out_bf16;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(blocks), cfg.blockDim = dim3(32), cfg.dynamicSmemBytes = 0, cfg.stream = rt->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr, cfg.numAttrs = 1;
    cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, wp);
    rt->dispatch_count += 1;
    return cuda_check(rt, e, "q4_gemv launch");
}

/// Experiment knobs for the staged kernel: "consumers,ring_kib,blocks_per_sm".
struct TmaCfg {
    int consumers = 16, ring_kib = 148, blocks_per_sm = 1, head_stages = 1, enabled = 1;
};
const TmaCfg &tma_cfg()
{
    static TmaCfg c = [] {
        TmaCfg t;
        if (const char *e = std::getenv("TESSL_B200_GEMV_TMA")) {
            int a = 0, b = 0, d = 0, h = 0;
            const int n = std::sscanf(e, "%d,%d,%d,%d", &a, &b, &d, &h);
            if (n >= 4 && h > 0) t.head_stages = h;
            if (n >= 1 && a == 0) t.enabled = 0;
            if (n >= 1 && a > 0) t.consumers = std::min(a, 16);
            if (n >= 2 && b > 0) t.ring_kib = b;
            if (n >= 3 && d > 0) t.blocks_per_sm = d;
        }
        return t;
    }();
    return c;
}

template <int NB, int RS, int NCH>
Result launch_tma(TesslRuntime *rt, const Q4GemvParams &p)
{
    auto kernel = q4k::q4_gemv_tma_kernel<NB, RS, NCH>;
    const TmaCfg &cfg = tma_cfg();
    q4k::TmaParams tp{};
    uint32_t rb = 0;
    for (int s = 0; s < p.nseg; ++s) {
        const Q4Seg &a = p.seg[s];
        tp.seg[s] = q4k::TmaSeg{a.packed0, a.sb0, a.packed1, a.sb1, a.out, a.resid, a.rows, rb};
        rb += (a.rows + RS - 1) / RS;
    }
    if (rb == 0) return ok();
    tp.nseg = p.nseg, tp.total_rb = rb;
    tp.x = p.x, tp.cols = p.cols, tp.group_shift = p.group_shift, tp.epi = p.epi, tp.out_bf16 = p.out_bf16;
    tp.status = rt->status_dev;
    const uint32_t stage_bytes = NB * RS * ((p.cols >> 1) + (p.cols >> p.group_shift) * 4);
    const uint32_t warps = (uint32_t)cfg.consumers;
    const uint32_t stages = std::max<uint32_t>(1u, (uint32_t)cfg.ring_kib * 1024u / (stage_bytes * warps));
    tp.stages = stages;
    tp.head_stages = (uint32_t)cfg.head_stages;
    const size_t smem = (size_t)warps * stages * (stage_bytes + 8);
    TESSL_TRY(smem_opt_in(rt, reinterpret_cast<const void *>(kernel), smem, "q4_gemv_tma: shared memory opt-in"));
    const uint32_t grid = std::min<uint32_t>(rb, (uint32_t)(rt->sm_count * cfg.blocks_per_sm));
    cudaLaunchConfig_t lc{};
    lc.gridDim = dim3(grid), lc.blockDim = dim3(cfg.consumers * 32), lc.dynamicSmemBytes = smem;
    lc.stream = rt->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    lc.attrs = attr, lc.numAttrs = 1;
    cudaError_t e = cudaLaunchKernelEx(&lc, kernel, tp);
    rt->dispatch_count += 1;
    return cuda_check(rt, e, "q4_gemv launch");
}

/// The tensor-core kernel (q4_gemv_mma.cuh): rows of 1024, 2048 or 4096 columns
/// whose sixteenth holds whole quantization groups, scale/bias rows that a bulk
/// copy can fetch. TESSL_B200_GEMV_MMA=0 turns it off (tuning runs).
bool mma_enabled()
{
    static int on = -1;
    if (on < 0) {
        const char *e = std::getenv("TESSL_B200_GEMV_MMA");
        on = (e && e[0] == '0') ? 0 : 1;
    }
    return on != 0;
}

bool mma_ok(const Q4GemvParams &p)
{
    if (!mma_enabled()) return false;
    if (p.cols != 1024 && p.cols != 2048 && p.cols != 4096) return false;
    if (p.group_shift < 5 || p.group_shift > 7) return false;
    if (((p.cols / 16) >> p.group_shift) == 0) return false;
    for (int s = 0; s < p.nseg && !p.staged; ++s) {
        const Q4Seg &a = p.seg[s];
        if (((uintptr_t)a.sb0 & 15u) || (a.sb1 && ((uintptr_t)a.sb1 & 15u))) return false;
    }
    return true;
}

/// Shared memory one block of the tensor-core GEMV may use: the per-block maximum of sm_100 less the kernel's few
/// static bytes.
constexpr uint32_t kMmaSmemBudget = 232448u - 512u;

template <int SW, int WPG, int NB, bool BATCH, bool Q8 = false, int NWIN = 1, int ROWS = 16, bool STAGED = false>
Result launch_mma_one(TesslRuntime *rt, const Q4GemvParams &p, int m)
{
    auto kernel = q4m::q4_gemv_mma_kernel<SW, WPG, NB, BATCH, Q8, NWIN, ROWS, STAGED>;
    constexpr uint32_t RPB = ROWS / NB;
    q4m::Params mp{};
    uint32_t rb = 0;
    for (int s = 0; s < p.nseg; ++s) {
        const Q4Seg &a = p.seg[s];
        mp.seg[s] = q4m::Seg{a.packed0, a.sb0, a.packed1, a.sb1, a.out, a.resid, a.rows, rb};
        rb += (a.rows + RPB - 1) / RPB;
    }
    if (rb == 0) return ok();
    mp.nseg = p.nseg, mp.total_rb = rb;
    mp.x = p.x, mp.m = (uint32_t)m, mp.cols = p.cols, mp.group_shift = p.group_shift;
    mp.epi = p.epi, mp.out_bf16 = p.out_bf16;
    mp.status = rt->status_dev;
    if ((p.staged != 0) != STAGED) return "q4_gemv: the staged layout runs on the one-row Q4 kernel only";
    if (p.peer) {
        const TesslPeerGather &g = *static_cast<const TesslPeerGather *>(p.peer);
        if (BATCH || Q8 || p.nseg != 1) return "q4_gemv: a sharded launch has one bank (or one gate/up pair) and one row of x";
        for (uint32_t r = 0; r < g.world; ++r) {
            mp.peer.out[r] = static_cast<uint8_t *>(g.buffers[r]) + (size_t)g.rank * g.bytes_per_rank;
            mp.peer.flags[r] = g.flags[r];
        }
        mp.peer.rank = g.rank, mp.peer.world = g.world, mp.peer_world = g.world;
        mp.peer.wait_clocks = rt->peer_wait_clocks ? (long long)rt->peer_wait_clocks : kPeerWaitClocks;
        mp.peer.defer = p.peer_defer ? 1u : 0u;
    }
    if (p.xwait) {
        const TesslPeerGather &g = *static_cast<const TesslPeerGather *>(p.xwait);
        if (BATCH || Q8) return "q4_gemv: a gathered x is one row";
        mp.xwait.flags = g.flags[g.rank];
        mp.xwait.rank = g.rank, mp.xwait.world = g.world, mp.xwait_world = g.world;
        mp.xwait.wait_clocks = rt->peer_wait_clocks ? (long long)rt->peer_wait_clocks : kPeerWaitClocks;
    }
    const uint32_t gpr = p.cols >> p.group_shift;
    const uint32_t part = BATCH ? q4m::kConsumers * 16 * 8 * 4 : q4m::kConsumers * 16 * 4;
    const uint32_t stage_bytes = ROWS * ((p.cols >> 1) + q4m::kRowPad) + ROWS * gpr * 4 + part;
    // the warps' staged slices of x: only the Q4 kernel for one row of x stages them
    const uint32_t x_stage = 32 + ((BATCH || Q8) ? 0u : q4m::kConsumers * q4m::kXStageBytes * NWIN);
    uint32_t stages = std::min<uint32_t>(8u, (kMmaSmemBudget - x_stage) / (stage_bytes + 24));
    if (stages < 2) return "q4_gemv_mma: the ring does not fit two stages";
    mp.stages = stages;
    const size_t smem = (size_t)stages * (stage_bytes + 24) + x_stage;
    TESSL_TRY(smem_opt_in(rt, reinterpret_cast<const void *>(kernel), smem, "q4_gemv_mma: shared memory opt-in", true));
    const uint32_t grid = std::min<uint32_t>(rb, (uint32_t)rt->sm_count);
    {
        const uint64_t step = (((uint64_t)rb << 32) + grid - 1) / grid;  // rb <= 2^32 - 1 and grid <= rb: step fits 64 bits
        mp.rb_step_lo = (uint32_t)step, mp.rb_step_hi = (uint32_t)(step >> 32);
    }
    // four rows per bulk copy wherever two row pairs are adjacent in memory (one bank, dense rows): 151936 x 4096
    // 58.8 -> 52.7 us, 6144 x 4096 5.30 -> 5.05 us, 12288 x 4096 8.00 -> 7.90 us on one box, back to back.
    // Not for Q8: its row pair is already 8 KB, and 16 KB copies ran 14336 x 4096 in 17.0 us against 14.5.
    mp.quads = (!BATCH && !Q8 && NWIN == 1 && !p.staged) ? 1u : 0u;
    cudaLaunchConfig_t lc{};
    lc.gridDim = dim3(grid), lc.blockDim = dim3(q4m::kThreads), lc.dynamicSmemBytes = smem;
    lc.stream = rt->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    lc.attrs = attr, lc.numAttrs = 1;
    cudaError_t e = cudaLaunchKernelEx(&lc, kernel, mp);
    rt->dispatch_count += 1;
    return cuda_check(rt, e, "q4_gemv launch");
}

template <int SW, int WPG>
Result launch_mma_sw(TesslRuntime *rt, const Q4GemvParams &p, int nb)
{
    if (p.staged) {
        if (nb == 2) return launch_mma_one<SW, WPG, 2, false, false, 1, 16, true>(rt, p, 1);
        return launch_mma_one<SW, WPG, 1, false, false, 1, 16, true>(rt, p, 1);
    }
    if (nb == 2) return launch_mma_one<SW, WPG, 2, false>(rt, p, 1);
    return launch_mma_one<SW, WPG, 1, false>(rt, p, 1);
}

/// One row of x.
Result launch_mma(TesslRuntime *rt, const Q4GemvParams &p, int nb)
{
    const int sw = (int)(p.cols / 512), wpg = 1 << (p.group_shift - 5);
    if (sw == 8) {
        if (wpg == 1) return launch_mma_sw<8, 1>(rt, p, nb);
        if (wpg == 2) return launch_mma_sw<8, 2>(rt, p, nb);
        return launch_mma_sw<8, 4>(rt, p, nb);
    }
    if (sw == 4) {
        if (wpg == 1) return launch_mma_sw<4, 1>(rt, p, nb);
        if (wpg == 2) return launch_mma_sw<4, 2>(rt, p, nb);
        return launch_mma_sw<4, 4>(rt, p, nb);
    }
    if (wpg == 1) return launch_mma_sw<2, 1>(rt, p, nb);
    return launch_mma_sw<2, 2>(rt, p, nb);
}

/// One row of x over rows of 8192 or 12288 columns (a 4096 x 12288 down projection): the tensor-core kernel
/// with every stage holding whole long rows, the warps walking the 4096-column windows inside it. Two
/// stages fit in shared memory (of 16 rows at 8192 columns, of 14 at 12288). Taken for every M = 1 form at
/// these widths, whatever the row count, so that a row's summation order still depends on K and G alone.
bool mma_long_ok(const Q4GemvParams &p, int m)
{
    if (!mma_enabled() || m != 1) return false;
    if (p.cols != 8192 && p.cols != 12288) return false;
    if (p.group_shift < 5 || p.group_shift > 7) return false;
    for (int s = 0; s < p.nseg; ++s) {
        const Q4Seg &a = p.seg[s];
        if (((uintptr_t)a.sb0 & 15u) || (a.sb1 && ((uintptr_t)a.sb1 & 15u))) return false;
    }
    return true;
}

Result launch_mma_long(TesslRuntime *rt, const Q4GemvParams &p)
{
    const int wpg = 1 << (p.group_shift - 5);
    if (p.cols == 8192) {
        if (wpg == 1) return launch_mma_one<8, 1, 1, false, false, 2, 16>(rt, p, 1);
        if (wpg == 2) return launch_mma_one<8, 2, 1, false, false, 2, 16>(rt, p, 1);
        return launch_mma_one<8, 4, 1, false, false, 2, 16>(rt, p, 1);
    }
    if (wpg == 1) return launch_mma_one<8, 1, 1, false, false, 3, 14>(rt, p, 1);
    if (wpg == 2) return launch_mma_one<8, 2, 1, false, false, 3, 14>(rt, p, 1);
    return launch_mma_one<8, 4, 1, false, false, 3, 14>(rt, p, 1);
}

/// How the batch kernel (q4_batch_mma.cuh) cuts a row: windows of whole units, each window's groups dealt out to the
/// 16 consumer warps. `ngs` is the busiest warp's share; 0 if the kernel does not take the shape.
struct BatchPlan {
    uint32_t unit_cols = 0, units = 0, nwin = 0, chunks = 0, sb_boxes = 0;
    int ngs = 0;
    bool even = false;  // every warp has ngs groups in every window, and ngs is a power of two
};
BatchPlan batch_plan(uint32_t cols, uint32_t group_shift)
{
    BatchPlan b;
    if (group_shift < 5 || group_shift > 7 || cols == 0) return b;
    // a window starts on a whole 256-column chunk of the packed rows and a whole quad of groups (16 bytes of pairs)
    b.unit_cols = std::max<uint32_t>(q4b::kChunkCols, 4u << group_shift);
    if (cols % b.unit_cols != 0) return b;
    b.units = cols / b.unit_cols;
    const uint32_t per = q4b::kWindowCols / b.unit_cols;
    b.nwin = (b.units + per - 1) / per;
    // Four windows instead of three: clusters of three leave 13 SMs without one and start late (4096 x 8192 at M = 8 cut in
    // 2 / 3 / 4: 7.4 / 11.3 / 7.2 us; 4096 x 12288 in 3 / 4: 10.4 / 8.9 us).
    if (b.nwin == 3) b.nwin = 4;
    if (b.nwin > q4b::kMaxWindows) return b;
    uint32_t widest = 0, narrowest = ~0u;
    for (uint32_t c = 0; c < b.nwin; ++c) {
        const uint32_t n = (c + 1) * b.units / b.nwin - c * b.units / b.nwin;
        widest = std::max(widest, n), narrowest = std::min(narrowest, n);
    }
    const uint32_t gpu = b.unit_cols >> group_shift;  // groups per unit
    b.chunks = widest * (b.unit_cols / q4b::kChunkCols);
    b.sb_boxes = (widest * gpu + 31) / 32;
    const int ngs = (int)((widest * gpu + q4b::kConsumers - 1) / q4b::kConsumers);
    if ((int)(narrowest * gpu / q4b::kConsumers) < ngs - 1) return b;  // warps hold ngs or ngs - 1 groups in every window
    b.ngs = ngs;
    b.even = narrowest == widest && widest * gpu == (uint32_t)ngs * q4b::kConsumers && (ngs & (ngs - 1)) == 0;
    return b;
}

bool batch_ok(const Q4GemvParams &p, int m, int nb)
{
    if (!mma_enabled() || m < 1 || m > 8 || (nb != 1 && m != 1) || p.staged || p.peer || p.xwait) return false;
    for (int s = 0; s < p.nseg; ++s) {
        const Q4Seg &a = p.seg[s];
        if (((uintptr_t)a.sb0 | (uintptr_t)a.packed0 | (uintptr_t)a.sb1 | (uintptr_t)a.packed1) & 15u) return false;
    }
    return batch_plan(p.cols, p.group_shift).ngs != 0;
}

template <int WPG, int NGS, bool EVEN, int NB, bool ONE>
Result launch_batch_one(TesslRuntime *rt, const Q4GemvParams &p, int m, const BatchPlan &b)
{
    auto kernel = q4b::q4_batch_mma_kernel<WPG, NGS, EVEN, NB, ONE>;
    constexpr uint32_t RPB = q4b::kRows / NB;
    const char *what = "q4_gemv";
    EncodeTiled enc = nullptr;
    TESSL_TRY(tensormap_encoder(rt, what, &enc));
    q4b::Maps maps;
    q4b::Params bp{};
    const uint32_t gpr = p.cols >> p.group_shift;
    auto encode = [&](int i, const uint8_t *packed, const uint32_t *sb, uint32_t rows) -> Result {
        const cuuint64_t dims[3] = {128, rows, p.cols / q4b::kChunkCols}, strides[2] = {p.cols / 2, 128};
        const cuuint32_t box[3] = {128, RPB, b.chunks};
        TESSL_TRY(make_map(enc, what, &maps.w[i], CU_TENSOR_MAP_DATA_TYPE_UINT8, packed, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B));
        const cuuint64_t sdims[2] = {gpr, rows}, sstrides[1] = {(cuuint64_t)gpr * 4};
        const cuuint32_t sbox[2] = {32, RPB};
        return make_map(enc, what, &maps.sb[i], CU_TENSOR_MAP_DATA_TYPE_UINT32, sb, sdims, sstrides, sbox, CU_TENSOR_MAP_SWIZZLE_128B);
    };
    for (int s = 0; s < p.nseg; ++s) {
        const Q4Seg &a = p.seg[s];
        if (a.rows == 0) return fmt("%s: a bank with no rows takes no part in a launch", what);
        TESSL_TRY(encode(s, a.packed0, a.sb0, a.rows));
        if (NB == 2) TESSL_TRY(encode(1, a.packed1, a.sb1, a.rows));
        bp.seg[s] = q4b::Seg{a.out, a.resid, a.rows, bp.total_rb};
        bp.total_rb += (uint32_t)(((uint64_t)a.rows + RPB - 1) / RPB);
    }
    bp.x = p.x, bp.status = rt->status_dev;
    bp.nseg = (uint32_t)p.nseg, bp.cols = p.cols, bp.m = (uint32_t)m, bp.group_shift = p.group_shift;
    bp.units = b.units, bp.unit_cols = b.unit_cols, bp.nwin = b.nwin, bp.chunks = b.chunks, bp.sb_boxes = b.sb_boxes;
    bp.epi = p.epi, bp.out_bf16 = p.out_bf16;
    const uint32_t stage_bytes = (b.chunks + b.sb_boxes) * q4b::kBoxBytes + q4b::kPartBytes;
    const uint32_t fixed = 1024 + q4b::kMailSlots * (b.nwin - 1) * q4b::kMailBytes + 8 * (1 + 2 * q4b::kMailSlots);
    bp.stages = std::min<uint32_t>(8u, (kMmaSmemBudget - fixed) / (stage_bytes + 24));
    if (bp.stages < (uint32_t)q4b::kReducers) return "q4_batch_mma: the ring does not fit two stages";
    const size_t smem = fixed + (size_t)bp.stages * (stage_bytes + 24);
    TESSL_TRY(smem_opt_in(rt, reinterpret_cast<const void *>(kernel), smem, "q4_batch_mma: shared memory opt-in", true));

    cudaLaunchConfig_t lc{};
    lc.blockDim = dim3(q4b::kThreads), lc.dynamicSmemBytes = smem;
    lc.stream = rt->stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = b.nwin, attr[1].val.clusterDim.y = 1, attr[1].val.clusterDim.z = 1;
    lc.attrs = attr, lc.numAttrs = b.nwin > 1 ? 2 : 1;
    uint32_t clusters = (uint32_t)rt->sm_count;
    if (b.nwin > 1) {
        // how many clusters of this size the device holds at once (one CTA per SM; a cluster lies in one GPC)
        int &n = rt->max_clusters[std::make_pair(reinterpret_cast<const void *>(kernel), b.nwin)];
        if (n == 0) {
            lc.gridDim = dim3(b.nwin * (rt->sm_count / b.nwin));
            const cudaError_t e = cudaOccupancyMaxActiveClusters(&n, kernel, &lc);
            if (e != cudaSuccess || n < 1) {
                cudaGetLastError();
                n = std::max(1, rt->sm_count / (int)b.nwin);
            }
        }
        clusters = (uint32_t)n;
    }
    clusters = std::min(clusters, bp.total_rb);
    const uint64_t step = (((uint64_t)bp.total_rb << 32) + clusters - 1) / clusters;
    bp.rb_step_lo = (uint32_t)step, bp.rb_step_hi = (uint32_t)(step >> 32);
    lc.gridDim = dim3(clusters * b.nwin);
    const cudaError_t e = cudaLaunchKernelEx(&lc, kernel, maps, bp);
    rt->dispatch_count += 1;
    return cuda_check(rt, e, "q4_gemv launch");
}

template <int WPG, int NGS>
Result launch_batch_ngs(TesslRuntime *rt, const Q4GemvParams &p, int m, int nb, const BatchPlan &b)
{
    if constexpr (NGS > 1) {
        if (b.ngs != NGS) return launch_batch_ngs<WPG, NGS - 1>(rt, p, m, nb, b);
    }
    if (nb == 2) return launch_batch_one<WPG, NGS, false, 2, true>(rt, p, m, b);
    if (m == 1) return launch_batch_one<WPG, NGS, false, 1, true>(rt, p, m, b);
    if constexpr ((NGS & (NGS - 1)) == 0) {
        if (b.even) return launch_batch_one<WPG, NGS, true, 1, false>(rt, p, m, b);
    }
    return launch_batch_one<WPG, NGS, false, 1, false>(rt, p, m, b);
}

Result launch_batch(TesslRuntime *rt, const Q4GemvParams &p, int m, int nb)
{
    const BatchPlan b = batch_plan(p.cols, p.group_shift);
    if (p.group_shift == 5) return launch_batch_ngs<1, 8>(rt, p, m, nb, b);
    if (p.group_shift == 6) return launch_batch_ngs<2, 4>(rt, p, m, nb, b);
    return launch_batch_ngs<4, 2>(rt, p, m, nb, b);
}

template <int SW, int WPG>
Result launch_mma_q8_sw(TesslRuntime *rt, const Q4GemvParams &p, int m)
{
    // 4096 codes per row: a 16-row stage with the batch's partial sums is 77 KB and only two fit; 10-row stages
    // (part of each MMA idle, which this format can afford: one MMA per 8 bytes of weights) give four. A stage's
    // compute does not depend on its height, so fewer and taller stages win as long as the ring stays deep enough:
    // 14336 x 4096 at M = 2 / 4 / 8: 8 rows (five stages) 16.5 / 17.0 / 17.5 us, 10 rows 14.6 / 15.0 / 15.6 us,
    // 12 rows (three stages) 16.8 / 17.1 / 17.7 us.
    if (SW == 16 && m > 1) return launch_mma_one<SW, WPG, 1, true, true, 1, 10>(rt, p, m);
    if (SW == 16 && m == 1) {
        // One row of x over 4096 codes per row is bound by the stream, not by the consumers (a stage's compute does
        // not depend on its height, its bytes do), so the stage height that leaves the shortest tail wins: the
        // busiest SM streams ceil(stages / SMs) x height rows. 14336 rows: 16 -> 14.4 us, 12 -> 14.05, 10 -> 13.7,
        // 8 -> 15.4 (half of every MMA idle begins to cost). Ties go to the taller stage.
        uint32_t rows = 0;
        for (int s = 0; s < p.nseg; ++s) rows += p.seg[s].rows;
        const uint32_t sms = (uint32_t)rt->sm_count;
        auto tail = [&](uint32_t h) { return (((rows + h - 1) / h + sms - 1) / sms) * h; };
        if (tail(10) < tail(16) && tail(10) < tail(12)) return launch_mma_one<SW, WPG, 1, false, true, 1, 10>(rt, p, m);
        if (tail(12) < tail(16)) return launch_mma_one<SW, WPG, 1, false, true, 1, 12>(rt, p, m);
    }
    if (m == 1) return launch_mma_one<SW, WPG, 1, false, true>(rt, p, m);
    return launch_mma_one<SW, WPG, 1, true, true>(rt, p, m);
}

/// The staged kernel needs every bulk copy 16-byte aligned and sized.
bool tma_ok(const Q4GemvParams &p)
{
    if (!tma_cfg().enabled) return false;
    if (p.cols == 0 || p.cols > 4096) return false;
    if ((((p.cols >> p.group_shift) * 4) & 15u) != 0) return false;
    for (int s = 0; s < p.nseg; ++s) {
        const Q4Seg &a = p.seg[s];
        if (((uintptr_t)a.sb0 & 15u) || (a.sb1 && ((uintptr_t)a.sb1 & 15u))) return false;
    }
    return true;
}

/// Picks the split of K over warps (a function of `cols` only, so a row's
/// summation order never depends on the launch) and the matching instantiation.
Result launch_q4_gemv(TesslRuntime *rt, Q4GemvParams p, int m, int nb)
{
    if (p.xwait && !(m == 1 && (mma_ok(p) || mma_long_ok(p, m)))) {
        // a width the tensor-core kernel does not take: the wait as a launch of its own, then whichever kernel serves it
        const TesslPeerGather *g = static_cast<const TesslPeerGather *>(p.xwait);
        p.xwait = nullptr;
        TESSL_TRY(nn::peer_wait(rt, *g));
        return launch_q4_gemv(rt, p, m, nb);
    }
    if (p.peer && !(m == 1 && (mma_ok(p) || (mma_long_ok(p, m) && nb == 1)))) {
        // shapes the tensor-core kernel does not take: the slice by whichever kernel serves it, then the
        // stand-alone exchange (same flag words, same result)
        const TesslPeerGather *g = static_cast<const TesslPeerGather *>(p.peer);
        p.peer = nullptr;
        TESSL_TRY(launch_q4_gemv(rt, p, m, nb));
        return nn::peer_gather(rt, *g);
    }
    const uint32_t nchunks = std::max<uint32_t>(1u, (p.cols + q4k::kChunk - 1) / q4k::kChunk);
    if (p.staged && !(m == 1 && mma_ok(p)))
        return "q4_gemv: the staged layout needs the tensor-core GEMV kernel (one row of x, rows of 1024, 2048 or 4096 columns)";
    if (m > 1 && batch_ok(p, m, nb)) return launch_batch(rt, p, m, nb);
    if (m == 1 && mma_ok(p)) return launch_mma(rt, p, nb);
    if (mma_long_ok(p, m)) {
        // The kernel takes one bank per launch at these widths. The bank-routed forms run as one launch per
        // bank, the gate/up forms as two launches into scratch and the activation kernel: what the fused
        // launches are defined to equal bit for bit.
        if (nb == 1) {
            for (int sidx = 0; sidx < p.nseg; ++sidx) {
                Q4GemvParams q = p;
                q.seg[0] = p.seg[sidx], q.nseg = 1;
                TESSL_TRY(launch_mma_long(rt, q));
            }
            return ok();
        }
        const uint32_t rows = p.seg[0].rows;
        void *tmp = nullptr;
        TESSL_TRY(scratch_reserve(rt, (size_t)rows * 8, &tmp));
        float *g = static_cast<float *>(tmp), *u = g + rows;
        Q4GemvParams q = p;
        q.epi = EPI_STORE, q.out_bf16 = 0, q.peer = nullptr;
        q.seg[0].packed1 = nullptr, q.seg[0].sb1 = nullptr, q.seg[0].out = g;
        TESSL_TRY(launch_mma_long(rt, q));
        q.seg[0].packed0 = p.seg[0].packed1, q.seg[0].sb0 = p.seg[0].sb1, q.seg[0].out = u;
        TESSL_TRY(launch_mma_long(rt, q));
        TESSL_TRY(launch_swiglu(rt, "gate/up activation launch", g, u, p.seg[0].out, rows, p.out_bf16, p.epi == EPI_GATE_UP_GELU ? 1 : 0));
        if (p.peer) return nn::peer_gather(rt, *static_cast<const TesslPeerGather *>(p.peer));
        return ok();
    }
    // One row of x over shorter rows leaves most of the 16 consumer warps without a group: 60000 x 512 8.8 us on the FMA
    // pipe against 12.0 here, 4096 x 512 2.32 / 2.34; from 1024 columns on 1024 x 1280 2.60 / 1.87, 6144 x 2560 5.55 / 3.72,
    // 2048 x 6144 4.81 / 4.38, 2560 x 9216 7.89 / 6.01, 4096 x 17408 24.6 / 10.4, 40000 x 6144 35.8 / 23.1, gate/up 13824 x 5120
    // 25.0 / 21.4, 2048 x 6144 6.41 / 6.46. Few rows over the windows of a cluster pay its fixed part: 257 x 7168 2.76 / 2.92,
    // 1024 x 9216 4.46 / 4.51 (groups of 128: 4.41 / 4.86), gate/up 512 x 9216 4.00 / 4.71. The line is one of K alone all the
    // same, so that a row's summation order is one of K and G (fused and separate launches, slices of a bank).
    if (m == 1 && p.cols >= 1024 && batch_ok(p, m, nb)) return launch_batch(rt, p, m, nb);
    if (m == 1 && nchunks <= 4 && tma_ok(p)) {
        if (nb == 1) {
            if (nchunks == 1) return launch_tma<1, 8, 1>(rt, p);
            if (nchunks == 2) return launch_tma<1, 4, 2>(rt, p);
            if (nchunks == 3) return launch_tma<1, 2, 3>(rt, p);
            return launch_tma<1, 2, 4>(rt, p);
        }
        if (nchunks == 1) return launch_tma<2, 4, 1>(rt, p);
        if (nchunks == 2) return launch_tma<2, 2, 2>(rt, p);
        if (nchunks == 3) return launch_tma<2, 1, 3>(rt, p);
        return launch_tma<2, 1, 4>(rt, p);
    }
    if (m == 1 && nchunks <= 4) {
        // Rows of at most 4096 columns: one warp keeps all of x resident.
        if (nb == 1) {
            if (nchunks == 1) return launch_warp<1, 8, 1>(rt, p);
            if (nchunks == 2) return launch_warp<1, 4, 2>(rt, p);
            if (nchunks == 3) return launch_warp<1, 2, 3>(rt, p);
            return launch_warp<1, 2, 4>(rt, p);
        }
        if (nchunks == 1) return launch_warp<2, 4, 1>(rt, p);
        if (nchunks == 2) return launch_warp<2, 2, 2>(rt, p);
        if (nchunks == 3) return launch_warp<2, 1, 3>(rt, p);
        return launch_warp<2, 1, 4>(rt, p);
    }
    if (m == 1) {
        int warps, nch;
        if (nchunks <= 4) {
            warps = (int)nchunks, nch = 1;
        } else if (nchunks <= 16) {
            warps = (int)(nchunks + 1) / 2, nch = 2;
        } else if (nchunks <= 32) {
            warps = (int)(nchunks + 3) / 4, nch = 4;
        } else {
            warps = 8, nch = 0;
        }
        if (nb == 1) {
            if (nch == 1) return launch_one<1, 1, 8, 1>(rt, p, warps);
            if (nch == 2) return launch_one<1, 1, 4, 2>(rt, p, warps);
            if (nch == 4) return launch_one<1, 1, 2, 4>(rt, p, warps);
            return launch_one<1, 1, 8, 0>(rt, p, warps);
        }
        if (nch == 1) return launch_one<1, 2, 4, 1>(rt, p, warps);
        if (nch == 2) return launch_one<1, 2, 2, 2>(rt, p, warps);
        if (nch == 4) return launch_one<1, 2, 1, 4>(rt, p, warps);
        return launch_one<1, 2, 4, 0>(rt, p, warps);
    }
    const int warps = (int)std::min<uint32_t>(4u, nchunks);
    switch (m) {
    case 2: return launch_one<2, 1, 4, 0>(rt, p, warps);
    case 3: return launch_one<3, 1, 2, 0>(rt, p, warps);
    case 4: return launch_one<4, 1, 2, 0>(rt, p, warps);
    case 5: return launch_one<5, 1, 2, 0>(rt, p, warps);
    case 6: return launch_one<6, 1, 2, 0>(rt, p, warps);
    case 7: return launch_one<7, 1, 2, 0>(rt, p, warps);
    case 8: return launch_one<8, 1, 2, 0>(rt, p, warps);
    default: return fmt("q4_gemv: no kernel for m=%d", m);
    }
}

Q4Seg make_seg(const TesslQ4MlxBank &b0, const TesslQ4MlxBank *b1, const TesslBuf &out, const TesslBuf *resid,
               uint32_t rows)
{
    Q4Seg s{};
    s.packed0 = static_cast<const uint8_t *>(b0.packed.ptr);
    s.sb0 = static_cast<const uint32_t *>(b0.scales_biases.ptr);
    s.packed1 = b1 ? static_cast<const uint8_t *>(b1->packed.ptr) : nullptr;
    s.sb1 = b1 ? static_cast<const uint32_t *>(b1->scales_biases.ptr) : nullptr;
    s.out = out.ptr;
    s.resid = resid ? static_cast<const float *>(resid->ptr) : nullptr;
    s.rows = rows;
    return s;
}

bool staged_domain(uint32_t cols, uint32_t group)
{
    if (cols != 1024 && cols != 2048 && cols != 4096) return false;
    if (group != 32 && group != 64 && group != 128) return false;
    return (cols / 16) / group >= 1;
}

Result check_alignment(const TesslQ4MlxBank &b, const What &what);

/// The bank checks of an entry that takes either layout: the reference's for a row-major bank, size,
/// domain and alignment of the image for a staged one.
Result bank_validate_layout(const TesslQ4MlxBank &bank, const TesslQuantShape &shape, uint32_t layout, const What &what)
{
    if (layout != TESSL_Q4_B200_STAGED) return q4_bank_validate(bank, shape, what);
    TESSL_TRY(quant_shape_validate(shape, what));
    if (!staged_domain(shape.cols, shape.group_size))
        return fmt("%s: the B200 staged layout exists for rows of 1024, 2048 or 4096 columns and groups of 32, 64 or 128 "
                   "(got %u columns, group %u)", what.str().c_str(), shape.cols, shape.group_size);
    TESSL_TRY(require(bank.packed, nn::q4_mlx_staged_bytes(shape.rows, shape.cols, shape.group_size), 1, what + " staged image"));
    return require_aligned16(bank.packed, what + " staged image");
}

Result check_alignment(const TesslQ4MlxBank &b, const What &what)
{
    TESSL_TRY(require_aligned16(b.packed, what + " packed"));
    if (((uintptr_t)b.scales_biases.ptr & 3u) != 0)
        return fmt("%s scales_biases: device pointer must be 4-byte aligned", what.str().c_str());
    return ok();
}

}  // namespace

namespace nn {

/// MLX Q8 (unsigned codes, bf16 pairs, bf16 x, M <= 8) on the tensor-core GEMV kernel: a row of `cols`
/// codes is laid out and staged like a row of 2 cols nibbles with groups of 2 group_size (the kernel's sizes
/// are in nibbles); the codes themselves go to the MMA as bf16 bit patterns, two per register. `*handled` is false when the shape is
/// not one the kernel is built for (the caller then uses its FMA-pipe kernel).
Result q8_mlx_mma(TesslRuntime *rt, const TesslBuf &codes, const TesslBuf &sb, const TesslBuf &x_bf16, const TesslBuf &y,
                  uint32_t rows, uint32_t cols, uint32_t group_size, uint32_t m, OutKind out, bool *handled)
{
    *handled = false;
    if (!mma_enabled()) return ok();
    if (m < 1) return ok();
    if (cols != 512 && cols != 1024 && cols != 2048 && cols != 4096) return ok();
    if (group_size != 32 && group_size != 64) return ok();
    if (((uintptr_t)sb.ptr & 15u) != 0 || ((uintptr_t)x_bf16.ptr & 7u) != 0) return ok();
    if (((2 * cols / 16) / (2 * group_size)) == 0) return ok();  // a warp's slice holds whole groups
    *handled = true;
    Q4GemvParams p{};
    p.nseg = 1;
    p.seg[0] = Q4Seg{};
    p.seg[0].packed0 = static_cast<const uint8_t *>(codes.ptr);
    p.seg[0].sb0 = static_cast<const uint32_t *>(sb.ptr);
    p.seg[0].out = y.ptr;
    p.seg[0].rows = rows;
    p.x = static_cast<const uint16_t *>(x_bf16.ptr);
    p.cols = 2 * cols;
    p.group_shift = log2_u32(2 * group_size);
    p.epi = EPI_STORE;
    p.out_bf16 = out == OUT_BF16;
    const int sw = (int)(p.cols / 512);
    const bool g64 = group_size == 64;  // 128 nibbles: 4 words per lane and group; 32 codes: 2
    switch (sw) {
    case 2: return g64 ? launch_mma_q8_sw<2, 2>(rt, p, (int)m) : launch_mma_q8_sw<2, 2>(rt, p, (int)m);
    case 4: return g64 ? launch_mma_q8_sw<4, 4>(rt, p, (int)m) : launch_mma_q8_sw<4, 2>(rt, p, (int)m);
    case 8: return g64 ? launch_mma_q8_sw<8, 4>(rt, p, (int)m) : launch_mma_q8_sw<8, 2>(rt, p, (int)m);
    default: return g64 ? launch_mma_q8_sw<16, 4>(rt, p, (int)m) : launch_mma_q8_sw<16, 2>(rt, p, (int)m);
    }
}


Result gemv_q4_mlx_simd(TesslRuntime *rt, const TesslQ4MlxBank &bank, const TesslBuf &x_bf16, const TesslBuf &y,
                        const TesslQuantShape &shape, uint32_t layout, const TesslBuf *resid, OutKind out)
{
    const char *entry = resid ? "gemv_q4_mlx_simd_add" : "gemv_q4_mlx_simd";
    const bool staged = layout == TESSL_Q4_B200_STAGED;
    TESSL_TRY(refuse_layout(layout, entry, true));
    TESSL_TRY(bank_validate_layout(bank, shape, layout, entry));
    TESSL_TRY(require(x_bf16, shape.cols, 2, What(entry) + " x_bf16"));
    TESSL_TRY(require(y, shape.rows, out == OUT_BF16 ? 2 : 4, What(entry) + " y"));
    if (resid) TESSL_TRY(require(*resid, shape.rows, 4, What(entry) + " resid"));
    if (shape.rows == 0) return ok();
    const Named writes[] = {{"y", &y}};
    const Named reads[] = {{"packed", &bank.packed}, {"scales_biases", &bank.scales_biases}, {"x_bf16", &x_bf16}};
    TESSL_TRY(require_disjoint_writes(entry, writes, 1, reads, 3));
    if (!staged) TESSL_TRY(check_alignment(bank, entry));
    TESSL_TRY(require_aligned16(x_bf16, What(entry) + " x_bf16"));
    if (shape.cols == 0) {
        // No columns: every sum is empty. The kernel's loop never runs and the
        // epilogue stores 0 (+ resid), as the reference's does.
    }
    Q4GemvParams p{};
    p.seg[0] = make_seg(bank, nullptr, y, resid, shape.rows);
    p.nseg = 1;
    p.x = static_cast<const uint16_t *>(x_bf16.ptr);
    p.cols = shape.cols;
    p.group_shift = log2_u32(shape.group_size);
    p.epi = resid ? EPI_ADD_RESID : EPI_STORE;
    p.out_bf16 = out == OUT_BF16;
    p.staged = staged;
    return launch_q4_gemv(rt, p, 1, 1);
}

Result gemv_q4_mlx_gate_up(TesslRuntime *rt, const char *entry, const char *what, bool silu,
                           const TesslQ4MlxBank &gate, const TesslQ4MlxBank &up, const TesslBuf &x,
                           const TesslBuf &mid, const TesslQuantShape &shape, uint32_t layout, bool mid_as_bf16)
{
    const bool staged = layout == TESSL_Q4_B200_STAGED;
    TESSL_TRY(refuse_layout(layout, entry, true));
    TESSL_TRY(bank_validate_layout(gate, shape, layout, What(entry) + " gate"));
    TESSL_TRY(bank_validate_layout(up, shape, layout, What(entry) + " up"));
    TESSL_TRY(require(x, shape.cols, 2, What(entry) + " x"));
    if (mid_as_bf16) {
        TESSL_TRY(require(mid, shape.rows, 2, What(entry) + " mid (bf16)"));
    } else {
        TESSL_TRY(require(mid, shape.rows, 4, What(entry) + " mid"));
    }
    if (shape.rows == 0) return ok();
    const Named writes[] = {{"mid", &mid}};
    const Named reads[] = {{"gate_packed", &gate.packed},
                           {"gate_scales_biases", &gate.scales_biases},
                           {"up_packed", &up.packed},
                           {"up_scales_biases", &up.scales_biases},
                           {"x", &x}};
    TESSL_TRY(require_disjoint_writes(what, writes, 1, reads, 5));
    if (!staged) {
        TESSL_TRY(check_alignment(gate, What(entry) + " gate"));
        TESSL_TRY(check_alignment(up, What(entry) + " up"));
    }
    TESSL_TRY(require_aligned16(x, What(entry) + " x"));
    Q4GemvParams p{};
    p.staged = staged;
    p.seg[0] = make_seg(gate, &up, mid, nullptr, shape.rows);
    p.nseg = 1;
    p.x = static_cast<const uint16_t *>(x.ptr);
    p.cols = shape.cols;
    p.group_shift = log2_u32(shape.group_size);
    p.epi = silu ? EPI_GATE_UP_SILU : EPI_GATE_UP_GELU;
    p.out_bf16 = mid_as_bf16;
    return launch_q4_gemv(rt, p, 1, 2);
}

/// This rank's slot of its own gather buffer, as the output buffer of a sharded launch.
static Result sharded_out(const TesslPeerGather &g, const char *entry, uint64_t need_bytes, TesslBuf *out)
{
    TESSL_TRY(peer_gather_validate(g, entry));
    if (need_bytes > g.bytes_per_rank)
        return fmt("%s: the slice needs %llu bytes, the gather holds %llu per rank", entry, (unsigned long long)need_bytes,
                   (unsigned long long)g.bytes_per_rank);
    out->ptr = static_cast<uint8_t *>(g.buffers[g.rank]) + (size_t)g.rank * g.bytes_per_rank;
    out->nbytes = g.bytes_per_rank;
    return ok();
}

Result gemv_q4_mlx_simd_sharded(TesslRuntime *rt, const TesslQ4MlxBank &bank, const TesslBuf &x_bf16,
                                const TesslPeerGather &gather, const TesslQuantShape &shape, bool y_as_bf16, bool defer)
{
    const char *entry = "gemv_q4_mlx_simd_sharded";
    TesslBuf y{};
    TESSL_TRY(sharded_out(gather, entry, (uint64_t)shape.rows * (y_as_bf16 ? 2 : 4), &y));
    if (shape.rows == 0) return fmt("%s: a rank with no rows takes part through tessl_peer_gather", entry);
    TESSL_TRY(q4_bank_validate(bank, shape, entry));
    TESSL_TRY(require(x_bf16, shape.cols, 2, What(entry) + " x_bf16"));
    const Named writes[] = {{"gather slot", &y}};
    const Named reads[] = {{"packed", &bank.packed}, {"scales_biases", &bank.scales_biases}, {"x_bf16", &x_bf16}};
    TESSL_TRY(require_disjoint_writes(entry, writes, 1, reads, 3));
    TESSL_TRY(check_alignment(bank, entry));
    TESSL_TRY(require_aligned16(x_bf16, What(entry) + " x_bf16"));
    Q4GemvParams p{};
    p.seg[0] = make_seg(bank, nullptr, y, nullptr, shape.rows);
    p.nseg = 1;
    p.x = static_cast<const uint16_t *>(x_bf16.ptr);
    p.cols = shape.cols;
    p.group_shift = log2_u32(shape.group_size);
    p.epi = EPI_STORE;
    p.out_bf16 = y_as_bf16;
    p.peer = gather.world > 1 ? &gather : nullptr;
    p.peer_defer = defer;
    return launch_q4_gemv(rt, p, 1, 1);
}

Result gemv_q4_mlx_simd_gathered(TesslRuntime *rt, const TesslQ4MlxBank &bank, const TesslPeerGather &gather,
                                 const TesslBuf &y, const TesslQuantShape &shape, const TesslBuf *resid, OutKind out)
{
    const char *entry = "gemv_q4_mlx_simd_gathered";
    TESSL_TRY(peer_gather_validate(gather, entry));
    TesslBuf x{};
    x.ptr = gather.buffers[gather.rank];
    x.nbytes = (uint64_t)gather.world * gather.bytes_per_rank;
    TESSL_TRY(q4_bank_validate(bank, shape, entry));
    TESSL_TRY(require(x, shape.cols, 2, What(entry) + " gathered x"));
    TESSL_TRY(require(y, shape.rows, out == OUT_BF16 ? 2 : 4, What(entry) + " y"));
    if (resid) TESSL_TRY(require(*resid, shape.rows, 4, What(entry) + " resid"));
    if (shape.rows == 0) return ok();
    const Named writes[] = {{"y", &y}};
    const Named reads[] = {{"packed", &bank.packed}, {"scales_biases", &bank.scales_biases}, {"gathered x", &x}};
    TESSL_TRY(require_disjoint_writes(entry, writes, 1, reads, 3));
    TESSL_TRY(check_alignment(bank, entry));
    Q4GemvParams p{};
    p.seg[0] = make_seg(bank, nullptr, y, resid, shape.rows);
    p.nseg = 1;
    p.x = static_cast<const uint16_t *>(x.ptr);
    p.cols = shape.cols;
    p.group_shift = log2_u32(shape.group_size);
    p.epi = resid ? EPI_ADD_RESID : EPI_STORE;
    p.out_bf16 = out == OUT_BF16;
    p.xwait = gather.world > 1 ? &gather : nullptr;
    return launch_q4_gemv(rt, p, 1, 1);
}

Result gemv_q4_mlx_gate_up_silu_sharded(TesslRuntime *rt, const TesslQ4MlxBank &gate, const TesslQ4MlxBank &up,
                                        const TesslBuf &x, const TesslPeerGather &gather, const TesslQuantShape &shape,
                                        bool mid_as_bf16, bool defer)
{
    const char *entry = "gemv_q4_mlx_gate_up_silu_sharded";
    TesslBuf mid{};
    TESSL_TRY(sharded_out(gather, entry, (uint64_t)shape.rows * (mid_as_bf16 ? 2 : 4), &mid));
    if (shape.rows == 0) return fmt("%s: a rank with no rows takes part through tessl_peer_gather", entry);
    TESSL_TRY(q4_bank_validate(gate, shape, What(entry) + " gate"));
    TESSL_TRY(q4_bank_validate(up, shape, What(entry) + " up"));
    TESSL_TRY(require(x, shape.cols, 2, What(entry) + " x"));
    const Named writes[] = {{"gather slot", &mid}};
    const Named reads[] = {{"gate_packed", &gate.packed},
                           {"gate_scales_biases", &gate.scales_biases},
                           {"up_packed", &up.packed},
                           {"up_scales_biases", &up.scales_biases},
                           {"x", &x}};
    TESSL_TRY(require_disjoint_writes(entry, writes, 1, reads, 5));
    TESSL_TRY(check_alignment(gate, What(entry) + " gate"));
    TESSL_TRY(check_alignment(up, What(entry) + " up"));
    TESSL_TRY(require_aligned16(x, What(entry) + " x"));
    Q4GemvParams p{};
    p.seg[0] = make_seg(gate, &up, mid, nullptr, shape.rows);
    p.nseg = 1;
    p.x = static_cast<const uint16_t *>(x.ptr);
    p.cols = shape.cols;
    p.group_shift = log2_u32(shape.group_size);
    p.epi = EPI_GATE_UP_SILU;
    p.out_bf16 = mid_as_bf16;
    p.peer = gather.world > 1 ? &gather : nullptr;
    p.peer_defer = defer;
    return launch_q4_gemv(rt, p, 1, 2);
}

Result gemv_q4_mlx_kv(TesslRuntime *rt, const TesslQ4MlxBank &k, const TesslQ4MlxBank &v, const TesslBuf &x_bf16,
                      const TesslBuf &k_out, const TesslBuf &v_out, const TesslQuantShape &shape, uint32_t layout)
{
    const char *entry = "gemv_q4_mlx_simd_kv";
    TESSL_TRY(refuse_layout(layout, entry));
    TESSL_TRY(q4_bank_validate(k, shape, What(entry) + " k"));
    TESSL_TRY(q4_bank_validate(v, shape, What(entry) + " v"));
    TESSL_TRY(require(x_bf16, shape.cols, 2, What(entry) + " x_bf16"));
    TESSL_TRY(require(k_out, shape.rows, 4, What(entry) + " k_out"));
    TESSL_TRY(require(v_out, shape.rows, 4, What(entry) + " v_out"));
    if (shape.rows == 0) return ok();
    const Named writes[] = {{"k_out", &k_out}, {"v_out", &v_out}};
    const Named reads[] = {{"k_packed", &k.packed},
                           {"k_scales_biases", &k.scales_biases},
                           {"v_packed", &v.packed},
                           {"v_scales_biases", &v.scales_biases},
                           {"x_bf16", &x_bf16}};
    TESSL_TRY(require_disjoint_writes("gemv_q4_mlx_kv", writes, 2, reads, 5));
    TESSL_TRY(check_alignment(k, What(entry) + " k"));
    TESSL_TRY(check_alignment(v, What(entry) + " v"));
    TESSL_TRY(require_aligned16(x_bf16, What(entry) + " x_bf16"));
    Q4GemvParams p{};
    p.seg[0] = make_seg(k, nullptr, k_out, nullptr, shape.rows);
    p.seg[1] = make_seg(v, nullptr, v_out, nullptr, shape.rows);
    p.nseg = 2;
    p.x = static_cast<const uint16_t *>(x_bf16.ptr);
    p.cols = shape.cols;
    p.group_shift = log2_u32(shape.group_size);
    p.epi = EPI_STORE;
    return launch_q4_gemv(rt, p, 1, 1);
}

Result gemv_q4_mlx_qkv(TesslRuntime *rt, const TesslQ4MlxBank &q, const TesslQ4MlxBank &k, const TesslQ4MlxBank &v,
                       const TesslBuf &x_bf16, const TesslQkvOutputs &out, uint32_t rows_q, uint32_t rows_kv,
                       uint32_t cols, uint32_t group_size, uint32_t layout)
{
    const char *entry = "gemv_q4_mlx_simd_qkv";
    TESSL_TRY(refuse_layout(layout, entry));
    const TesslQuantShape q_shape{rows_q, cols, group_size}, kv_shape{rows_kv, cols, group_size};
    TESSL_TRY(q4_bank_validate(q, q_shape, What(entry) + " q"));
    TESSL_TRY(q4_bank_validate(k, kv_shape, What(entry) + " k"));
    TESSL_TRY(q4_bank_validate(v, kv_shape, What(entry) + " v"));
    TESSL_TRY(require(x_bf16, cols, 2, What(entry) + " x_bf16"));
    TESSL_TRY(require(out.q_out, rows_q, 4, What(entry) + " q_out"));
    TESSL_TRY(require(out.k_out, rows_kv, 4, What(entry) + " k_out"));
    TESSL_TRY(require(out.v_out, rows_kv, 4, What(entry) + " v_out"));
    if (rows_q == 0 && rows_kv == 0) return ok();
    // Only the banks that produce output take part in the aliasing check.
    Named writes[3];
    Named reads[7];
    int nw = 0, nr = 0;
    if (rows_q != 0) {
        writes[nw++] = {"q_out", &out.q_out};
        reads[nr++] = {"q_packed", &q.packed};
        reads[nr++] = {"q_scales_biases", &q.scales_biases};
    }
    if (rows_kv != 0) {
        writes[nw++] = {"k_out", &out.k_out};
        writes[nw++] = {"v_out", &out.v_out};
        reads[nr++] = {"k_packed", &k.packed};
        reads[nr++] = {"k_scales_biases", &k.scales_biases};
        reads[nr++] = {"v_packed", &v.packed};
        reads[nr++] = {"v_scales_biases", &v.scales_biases};
    }
    reads[nr++] = {"x_bf16", &x_bf16};
    TESSL_TRY(require_disjoint_writes(entry, writes, nw, reads, nr));
    TESSL_TRY(require_aligned16(x_bf16, What(entry) + " x_bf16"));
    Q4GemvParams p{};
    p.nseg = 0;
    if (rows_q != 0) {
        TESSL_TRY(check_alignment(q, What(entry) + " q"));
        p.seg[p.nseg++] = make_seg(q, nullptr, out.q_out, nullptr, rows_q);
    }
    if (rows_kv != 0) {
        TESSL_TRY(check_alignment(k, What(entry) + " k"));
        TESSL_TRY(check_alignment(v, What(entry) + " v"));
        p.seg[p.nseg++] = make_seg(k, nullptr, out.k_out, nullptr, rows_kv);
        p.seg[p.nseg++] = make_seg(v, nullptr, out.v_out, nullptr, rows_kv);
    }
    p.x = static_cast<const uint16_t *>(x_bf16.ptr);
    p.cols = cols;
    p.group_shift = log2_u32(group_size);
    p.epi = EPI_STORE;
    return launch_q4_gemv(rt, p, 1, 1);
}

Result swiglu(TesslRuntime *rt, const TesslBuf &gate, const TesslBuf &up, const TesslBuf &out, uint32_t n,
              bool out_as_bf16)
{
    TESSL_TRY(require(gate, n, 4, "swiglu gate"));
    TESSL_TRY(require(up, n, 4, "swiglu up"));
    TESSL_TRY(require(out, n, out_as_bf16 ? 2 : 4, "swiglu out"));
    if (n == 0) return ok();
    return launch_swiglu(rt, "swiglu launch", static_cast<const float *>(gate.ptr), static_cast<const float *>(up.ptr), out.ptr, n,
                         out_as_bf16 ? 1 : 0, 0);
}

/// A validated prefill call with few rows, run as batches of up to 8 rows on the tensor-core GEMV kernel, at the widths where a
/// single row has the tensor-core kernel; `*handled` is false at the others. One or two batches are faster than the prefill GEMM's
/// 25 rows everywhere (16 rows / 25 rows, us: 12288 x 4096 15.9 / 18.9, 4096 x 4096 9.1 / 11.4, 2048 x 2048 5.2 / 8.2, 1024 x 1024 4.2 /
/// 8.1). Three batches were, too, against the GEMM of 256-row tiles that the line at 24 was drawn for; against the split
/// kernel they lose at the wide calls (24 rows: 23.3, 13.3, 7.7, 6.2 us).
Result prefill_as_small_batches(TesslRuntime *rt, const TesslQ4MlxBank &bank, const TesslBuf &x_bf16, const TesslBuf &y,
                                const TesslQuantShape &shape, uint32_t m, OutKind out, bool *handled)
{
    *handled = false;
    if (m == 0 || m > 24) return ok();
    Q4GemvParams probe{};
    probe.nseg = 1;
    probe.seg[0] = make_seg(bank, nullptr, y, nullptr, shape.rows);
    probe.cols = shape.cols;
    probe.group_shift = log2_u32(shape.group_size);
    if (!mma_ok(probe)) return ok();
    *handled = true;
    const size_t esz = out == OUT_BF16 ? 2 : 4;
    for (uint32_t b = 0; b < m; b += 8) {
        const uint32_t mb = std::min<uint32_t>(8u, m - b);
        Q4GemvParams p = probe;
        p.seg[0].out = static_cast<char *>(y.ptr) + (size_t)b * shape.rows * esz;
        p.x = static_cast<const uint16_t *>(x_bf16.ptr) + (size_t)b * shape.cols;
        p.epi = EPI_STORE;
        p.out_bf16 = out == OUT_BF16;
        TESSL_TRY(launch_q4_gemv(rt, p, (int)mb, 1));
    }
    return ok();
}

Result gemm_q4_mlx(TesslRuntime *rt, const TesslQ4MlxBank &bank, const TesslBuf &x_bf16, const TesslBuf &y,
                   const TesslQuantShape &shape, uint32_t m, uint32_t layout, const TesslBuf *resid, OutKind out)
{
    const char *entry = resid ? "gemm_q4_mlx_simd_add" : "gemm_q4_mlx_simd";
    TESSL_TRY(refuse_layout(layout, entry));
    if (m == 0) return ok();
    if (m > TESSL_GEMM_Q4_MLX_MAX_M) {
        return fmt("%s: M = %u exceeds GEMM_MAX_M = %u; the kernel clamps to that internally, so rows %u..%u would "
                   "be left unwritten rather than computed",
                   entry, m, TESSL_GEMM_Q4_MLX_MAX_M, TESSL_GEMM_Q4_MLX_MAX_M, m);
    }
    TESSL_TRY(q4_bank_validate(bank, shape, entry));
    const uint64_t out_elems = elems(m, shape.rows);
    TESSL_TRY(require(x_bf16, elems(m, shape.cols), 2, What(entry) + " x_bf16"));
    TESSL_TRY(require(y, out_elems, out == OUT_BF16 ? 2 : 4, What(entry) + " y"));
    if (resid) TESSL_TRY(require(*resid, out_elems, 4, What(entry) + " resid"));
    if (shape.rows == 0) return ok();
    const Named writes[] = {{"y", &y}};
    const Named reads[] = {{"packed", &bank.packed}, {"scales_biases", &bank.scales_biases}, {"x_bf16", &x_bf16}};
    TESSL_TRY(require_disjoint_writes("gemm_q4_mlx", writes, 1, reads, 3));
    TESSL_TRY(check_alignment(bank, entry));
    TESSL_TRY(require_aligned16(x_bf16, What(entry) + " x_bf16"));
    Q4GemvParams p{};
    p.seg[0] = make_seg(bank, nullptr, y, resid, shape.rows);
    p.nseg = 1;
    p.x = static_cast<const uint16_t *>(x_bf16.ptr);
    p.cols = shape.cols;
    p.group_shift = log2_u32(shape.group_size);
    p.epi = resid ? EPI_ADD_RESID : EPI_STORE;
    p.out_bf16 = out == OUT_BF16;
    return launch_q4_gemv(rt, p, (int)m, 1);
}

Result embed_lookup_q4_mlx(TesslRuntime *rt, const TesslQ4MlxBank &bank, const TesslBuf &token_ids, const TesslBuf &out,
                           uint32_t vocab, uint32_t hidden, uint32_t group_size, uint32_t n_tokens)
{
    const char *what = "embed_lookup_q4_mlx";
    const TesslQuantShape shape{vocab, hidden, group_size};
    TESSL_TRY(q4_bank_validate(bank, shape, what));
    const uint64_t total = elems(n_tokens, hidden);
    TESSL_TRY(require(token_ids, n_tokens, 4, What(what) + " token_ids"));
    TESSL_TRY(require(out, total, 4, What(what) + " out"));
    const Named writes[] = {{"out", &out}};
    const Named reads[] = {{"packed", &bank.packed}, {"scales_biases", &bank.scales_biases}, {"token_ids", &token_ids}};
    TESSL_TRY(require_disjoint_writes(what, writes, 1, reads, 3));
    if (total == 0) return ok();
    TESSL_TRY(check_alignment(bank, what));
    TESSL_TRY(require_aligned16(out, What(what) + " out"));
    if (((uintptr_t)token_ids.ptr & 3u) != 0) return fmt("%s token_ids: device pointer must be 4-byte aligned", what);
    const uint64_t total32 = total / 32;  // hidden is a multiple of the group size, itself a multiple of 32
    return launch_pdl(rt, "embed_lookup_q4_mlx launch", embed_lookup_q4_mlx_kernel, dim3((unsigned)((total32 + 127) / 128)), dim3(128), 0,
                      static_cast<const uint8_t *>(bank.packed.ptr), static_cast<const uint32_t *>(bank.scales_biases.ptr),
                      static_cast<const uint32_t *>(token_ids.ptr), static_cast<float *>(out.ptr), hidden, log2_u32(group_size), vocab,
                      total32);
}

uint64_t q4_mlx_staged_bytes(uint32_t rows, uint32_t cols, uint32_t group_size)
{
    if (!staged_domain(cols, group_size)) return 0;
    return (uint64_t)((rows + 7) / 8) * staged_geom(cols, group_size).unit_bytes;
}

Result q4_mlx_repack_staged(TesslRuntime *rt, const TesslQ4MlxBank &bank, const TesslQuantShape &shape, const TesslBuf &out)
{
    const char *entry = "q4_mlx_repack_staged";
    TESSL_TRY(q4_bank_validate(bank, shape, entry));
    if (!staged_domain(shape.cols, shape.group_size))
        return fmt("%s: the B200 staged layout exists for rows of 1024, 2048 or 4096 columns and groups of 32, 64 or 128 "
                   "(got %u columns, group %u)", entry, shape.cols, shape.group_size);
    const uint64_t nbytes = q4_mlx_staged_bytes(shape.rows, shape.cols, shape.group_size);
    TESSL_TRY(require(out, nbytes, 1, What(entry) + " out"));
    if (shape.rows == 0) return ok();
    const Named writes[] = {{"out", &out}};
    const Named reads[] = {{"packed", &bank.packed}, {"scales_biases", &bank.scales_biases}};
    TESSL_TRY(require_disjoint_writes(entry, writes, 1, reads, 2));
    TESSL_TRY(require_aligned16(bank.packed, What(entry) + " packed"));
    TESSL_TRY(require_aligned16(bank.scales_biases, What(entry) + " scales_biases"));
    TESSL_TRY(require_aligned16(out, What(entry) + " out"));
    const uint64_t n16 = nbytes / 16;
    q4_repack_staged_kernel<<<(unsigned)((n16 + 255) / 256), 256, 0, rt->stream>>>(
        static_cast<const uint4 *>(bank.packed.ptr), static_cast<const uint4 *>(bank.scales_biases.ptr),
        static_cast<uint4 *>(out.ptr), shape.rows, shape.cols, shape.group_size, n16);
    rt->dispatch_count += 1;
    return cuda_check(rt, cudaGetLastError(), "q4_mlx_repack_staged launch");
}

Result q4_mlx_unpack(TesslRuntime *rt, const TesslQ4MlxBank &bank, const TesslQuantShape &shape, const TesslBuf &out)
{
    TESSL_TRY(q4_bank_validate(bank, shape, "q4_mlx_unpack"));
    const uint64_t n = elems(shape.rows, shape.cols);
    TESSL_TRY(require(out, n, 1, "q4_mlx_unpack out"));
    if (n == 0) return ok();
    const uint64_t bytes = n / 2;
    q4_unpack_kernel<<<(unsigned)((bytes + 255) / 256), 256, 0, rt->stream>>>(
        static_cast<const uint8_t *>(bank.packed.ptr), static_cast<uint8_t *>(out.ptr), bytes);
    rt->dispatch_count += 1;
    return cuda_check(rt, cudaGetLastError(), "q4_mlx_unpack launch");
}

Result q4_mlx_dequant(TesslRuntime *rt, const TesslQ4MlxBank &bank, const TesslQuantShape &shape,
                      const TesslBuf &out)
{
    TESSL_TRY(q4_bank_validate(bank, shape, "q4_mlx_dequant"));
    const uint64_t n = elems(shape.rows, shape.cols);
    TESSL_TRY(require(out, n, 4, "q4_mlx_dequant out"));
    if (n == 0) return ok();
    const uint64_t bytes = n / 2;
    q4_dequant_kernel<<<(unsigned)((bytes + 255) / 256), 256, 0, rt->stream>>>(
        static_cast<const uint8_t *>(bank.packed.ptr), static_cast<const uint32_t *>(bank.scales_biases.ptr),
        static_cast<float *>(out.ptr), shape.rows, shape.cols, log2_u32(shape.group_size));
    rt->dispatch_count += 1;
    return cuda_check(rt, cudaGetLastError(), "q4_mlx_dequant launch");
}

}  // namespace nn
}  // namespace tessl
