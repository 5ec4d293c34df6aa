// The steps either side of a projection in Qwen3.5 decode: the zero-centred RMSNorm that produces
// the bf16 activations a Q4 projection reads, the residual add, and the two in one launch.
//
// Mirrors `qwen35::rms_norm`, `qwen35::residual_add` and `qwen35::add_rms_norm`
// (src/qwen35.rs:2586-2755 of the reference project) and their kernels
// (kernels/qwen35_mlp.metal:53-171): out[r, :] = x[r, :] * rsqrt(mean(x[r, :]^2) + eps) * (1 + w[:]),
// f32 in, f32 or bf16 out, `1 + w` formed in f32 here. The fused form adds y into resid first and is
// bit-identical to the two separate calls: the add is the same f32 add, every element is read back by
// the thread that wrote it, and the sum of squares is reduced in the same order by the same code.
//
// One block per row; a thread holds its part of the row in registers, so a row of up to 8192 columns costs one round
// trip to memory and one barrier. The rows are a few KB, so the kernels are latency-bound; they are launched with
// programmatic stream serialization so that a following GEMV can already stream its weights while they run. 512 threads
// of 32 registers (rows of up to 4096) fit an SM beside a block of the GEMV in front, so the block is resident when that
// one ends.
//
// The order of a row's sum is a function of dim alone: chain t takes the pieces t, t + n, t + 2n, ... in one run of FMAs,
// 32 chains meet in an xor butterfly, the sums of 32 in another (n chains: chain_count).
#include <type_traits>

#include "q4_common.cuh"
#include "runtime.h"

namespace tessl {
namespace {

constexpr uint32_t kMaxChains = 512;
constexpr uint32_t kHeld = 4;  // pieces of four columns that a chain has, at most, in rows that are held in registers

/// Sum over the block's chains, CPT per thread, the same value in every thread: lanes by xor butterfly, then the sums of 32
/// chains likewise.
template <int CPT>
__device__ __forceinline__ float block_sum(const float (&v)[CPT], float *scratch)
{
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
#pragma unroll
    for (uint32_t c = 0; c < CPT; ++c) {
        const float s = dev::warp_sum(v[c]);
        if (lane == 0) scratch[c * warps + warp] = s;
    }
    __syncthreads();
    return dev::warp_sum(lane < CPT * warps ? scratch[lane] : 0.0f);
}

__device__ __forceinline__ float4 load4(const float *p)
{
    const uint4 v = dev::ld_after_wait16(p);
    return make_float4(__uint_as_float(v.x), __uint_as_float(v.y), __uint_as_float(v.z), __uint_as_float(v.w));
}
__device__ __forceinline__ float load1(const float *p)
{
    float v;
    asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ float4 load4_words(const float *p) { return make_float4(load1(p), load1(p + 1), load1(p + 2), load1(p + 3)); }

template <bool OUT_BF16>
__device__ __forceinline__ void store4(void *out, size_t at, const float4 &o)
{
    if constexpr (OUT_BF16) {
        uint2 b;
        b.x = (uint32_t)dev::f32_to_bf16_store(o.x) | ((uint32_t)dev::f32_to_bf16_store(o.y) << 16);
        b.y = (uint32_t)dev::f32_to_bf16_store(o.z) | ((uint32_t)dev::f32_to_bf16_store(o.w) << 16);
        *reinterpret_cast<uint2 *>(static_cast<uint16_t *>(out) + at) = b;
    } else {
        *reinterpret_cast<float4 *>(static_cast<float *>(out) + at) = o;
    }
}

/// NV: float4 pieces of the row per chain, held in registers with their weights, CPT chains per thread. NV = 0: rows of more than
/// 8192 columns, in float4 steps, and rows whose length is no multiple of 4, word by word, both read twice. WIDE_W: weights at a
/// 16-byte boundary (else word by word: 1 x 8192 2.9 -> 3.1 us).
///
/// Times, back to back in a graph: with 256 threads that read the row twice and its weights word by word after the sum / here, us:
/// 1 x 4096 3.5 / 2.2, with the add 4.1 / 2.5; 1 x 8192 5.4 / 2.9; 1 x 12288 7.3 / 4.1, with the add 9.0 / 5.0; 2048 x 4096 15.7 / 10.8;
/// 1 x 4095 5.9 / 3.3, 16384 x 4095 97.9 / 114.9 (the one that lost). The loads of the add are issued with the others: with a store
/// behind each pair of them 1 x 4096 2.8, 1 x 8192 4.1. Bound by latency up to some hundred rows, by memory from there (16384 x 4096
/// 5.0 TB/s).
template <bool ADD, bool OUT_BF16, int NV, int CPT, bool WIDE_W>
__global__ void __launch_bounds__(kMaxChains / CPT, NV *CPT <= 2 ? 2048 / kMaxChains * CPT : 2)
    qwen35_rms_norm_kernel(const float *y, float *x_or_resid, const float *weight, void *out, uint32_t dim, float eps)
{
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    __shared__ float scratch[kMaxChains / 32];
    const size_t base = (size_t)blockIdx.x * dim;
    const uint32_t tid = threadIdx.x, nt = blockDim.x;
    float *xr = x_or_resid + base;
    const float *yr = ADD ? y + base : nullptr;
    float ss[CPT] = {};
    auto square = [&](int c, const float4 &v) {
        ss[c] = fmaf(v.x, v.x, ss[c]), ss[c] = fmaf(v.y, v.y, ss[c]), ss[c] = fmaf(v.z, v.z, ss[c]), ss[c] = fmaf(v.w, v.w, ss[c]);
    };
    auto scale = [&] { return __fdiv_rn(1.0f, __fsqrt_rn(__fdiv_rn(block_sum<CPT>(ss, scratch), (float)dim) + eps)); };
    auto one = [](float x, float inv, float w) { return __fmul_rn(__fmul_rn(x, inv), 1.0f + w); };
    auto four = [&](const float4 &v, float inv, const float4 &w) {
        return make_float4(one(v.x, inv, w.x), one(v.y, inv, w.y), one(v.z, inv, w.z), one(v.w, inv, w.w));
    };
    const float4 zero = make_float4(0, 0, 0, 0);
    if constexpr (NV > 0) {
        // Every load of the row is issued before any is waited for (a store between them would wait for its operands).
        constexpr int N = NV * CPT;  // piece i / CPT of chain i % CPT
        float4 v[N], a[ADD ? N : 1], w[N];
        auto column = [&](int i) { return (i * nt + tid) * 4; };
#pragma unroll
        for (int i = 0; i < N; ++i) v[i] = column(i) < dim ? load4(xr + column(i)) : zero;
        if constexpr (ADD) {
#pragma unroll
            for (int i = 0; i < N; ++i) a[i] = column(i) < dim ? load4(yr + column(i)) : zero;
        }
#pragma unroll
        for (int i = 0; i < N; ++i) w[i] = column(i) >= dim ? zero : WIDE_W ? load4(weight + column(i)) : load4_words(weight + column(i));
        if constexpr (ADD) {
#pragma unroll
            for (int i = 0; i < N; ++i) {
                v[i].x += a[i].x, v[i].y += a[i].y, v[i].z += a[i].z, v[i].w += a[i].w;
                if (column(i) < dim) *reinterpret_cast<float4 *>(xr + column(i)) = v[i];
            }
        }
#pragma unroll
        for (int i = 0; i < N; ++i) square(i % CPT, v[i]);
        const float inv = scale();
#pragma unroll
        for (int i = 0; i < N; ++i)
            if (column(i) < dim) store4<OUT_BF16>(out, base + column(i), four(v[i], inv, w[i]));
    } else if (dim % 4 == 0) {
        constexpr uint32_t B = ADD ? 2 : 4;  // pieces whose loads are issued together
        for (uint32_t d0 = tid * 4; d0 < dim; d0 += B * nt * 4) {
            float4 v[B], a[B];
#pragma unroll
            for (uint32_t i = 0; i < B; ++i) {
                const uint32_t d = d0 + i * nt * 4;
                v[i] = d < dim ? load4(xr + d) : zero;
                if (ADD) a[i] = d < dim ? load4(yr + d) : zero;
            }
#pragma unroll
            for (uint32_t i = 0; i < B; ++i) {
                const uint32_t d = d0 + i * nt * 4;
                if constexpr (ADD) {
                    v[i].x += a[i].x, v[i].y += a[i].y, v[i].z += a[i].z, v[i].w += a[i].w;
                    if (d < dim) *reinterpret_cast<float4 *>(xr + d) = v[i];
                }
                square(i % CPT, v[i]);
            }
        }
        const float inv = scale();
        for (uint32_t d0 = tid * 4; d0 < dim; d0 += 2 * nt * 4) {
            float4 v[2], w[2];
#pragma unroll
            for (uint32_t i = 0; i < 2; ++i) {
                const uint32_t d = d0 + i * nt * 4;
                v[i] = d < dim ? load4(xr + d) : zero;  // its own writes, if ADD
                w[i] = d >= dim ? zero : WIDE_W ? load4(weight + d) : load4_words(weight + d);
            }
#pragma unroll
            for (uint32_t i = 0; i < 2; ++i) {
                const uint32_t d = d0 + i * nt * 4;
                if (d < dim) store4<OUT_BF16>(out, base + d, four(v[i], inv, w[i]));
            }
        }
    } else {
        auto put = [&](uint32_t d, float o) {
            if constexpr (OUT_BF16) {
                static_cast<uint16_t *>(out)[base + d] = dev::f32_to_bf16_store(o);
            } else {
                static_cast<float *>(out)[base + d] = o;
            }
        };
        constexpr uint32_t B = 4;
        uint32_t d0 = tid;
        for (; d0 + (B - 1) * nt < dim; d0 += B * nt) {
            float v[B], a[B];
#pragma unroll
            for (uint32_t i = 0; i < B; ++i) {
                v[i] = load1(xr + d0 + i * nt);
                if (ADD) a[i] = load1(yr + d0 + i * nt);
            }
#pragma unroll
            for (uint32_t i = 0; i < B; ++i) {
                if constexpr (ADD) v[i] += a[i], xr[d0 + i * nt] = v[i];
                ss[i % CPT] = fmaf(v[i], v[i], ss[i % CPT]);
            }
        }
#pragma unroll
        for (uint32_t i = 0; i < B - 1; ++i) {
            const uint32_t d = d0 + i * nt;
            if (d >= dim) break;
            float v = xr[d];
            if constexpr (ADD) v += yr[d], xr[d] = v;
            ss[i % CPT] = fmaf(v, v, ss[i % CPT]);
        }
        const float inv = scale();
        for (d0 = tid; d0 + (B - 1) * nt < dim; d0 += B * nt) {
            float v[B], w[B];
#pragma unroll
            for (uint32_t i = 0; i < B; ++i) v[i] = load1(xr + d0 + i * nt), w[i] = load1(weight + d0 + i * nt);  // its own writes, if ADD
#pragma unroll
            for (uint32_t i = 0; i < B; ++i) put(d0 + i * nt, one(v[i], inv, w[i]));
        }
        for (; d0 < dim; d0 += nt) put(d0, one(xr[d0], inv, weight[d0]));
    }
}

template <bool ADD, bool OUT_BF16>
Result launch_norm(TesslRuntime *rt, const char *what, const float *y, float *x, const float *w, void *out, uint32_t rows, uint32_t dim,
                   float eps)
{
    // Rows start 16-byte aligned where dim is a multiple of 4 (the wrappers check the buffers).
    const uint32_t pieces = (dim + 3) / 4;
    uint32_t nv = (pieces + kMaxChains - 1) / kMaxChains;
    if (dim % 4 != 0 || nv > kHeld) nv = 0;
    const uint32_t chains = nv ? ((pieces + nv - 1) / nv + 31) & ~31u : kMaxChains;
    const bool wide_w = ((uintptr_t)w & 15u) == 0;
    // Many rows: half the threads with two chains each, so that twice the rows are in flight (same bits). 16384 x 2048 58.9 -> 47.0 us,
    // with the add 77.4 -> 69.9; 2048 x 4096 11.8 -> 10.8. A few hundred rows do not fill the SMs either way (509 x 2048 3.3 -> 3.7), and four
    // pieces a chain alone lose (2048 x 8192 23.9 -> 26.7; with the add 48.4 -> 39.7).
    const bool many = rows >= 1024 && chains % 64 == 0 && (ADD || nv < 4);
    auto go = [&](auto kernel, uint32_t threads) {
        return launch_pdl(rt, what, kernel, dim3(rows), dim3(threads), 0, y, x, w, out, dim, eps);
    };
    auto held = [&](auto n) {
        constexpr int NV = decltype(n)::value;
        if (many) return wide_w ? go(qwen35_rms_norm_kernel<ADD, OUT_BF16, NV, 2, true>, chains / 2)
                                : go(qwen35_rms_norm_kernel<ADD, OUT_BF16, NV, 2, false>, chains / 2);
        return wide_w ? go(qwen35_rms_norm_kernel<ADD, OUT_BF16, NV, 1, true>, chains)
                      : go(qwen35_rms_norm_kernel<ADD, OUT_BF16, NV, 1, false>, chains);
    };
    switch (nv) {
    case 1: return held(std::integral_constant<int, 1>{});
    case 2: return held(std::integral_constant<int, 2>{});
    case 3: return held(std::integral_constant<int, 3>{});
    case 4: return held(std::integral_constant<int, 4>{});
    default: return held(std::integral_constant<int, 0>{});
    }
}

__global__ void qwen35_residual_add_kernel(const float *y, float *resid, uint64_t n)
{
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) resid[i] = resid[i] + y[i];
}

/// `nn::validate_rms_scalars` (src/nn.rs:190-202 of the reference project).
Result validate_rms_scalars(uint32_t dim, float eps, const char *what)
{
    if (dim == 0) return fmt("%s: dim must be non-zero", what);
    if (!(eps > 0.0f) || !(eps < 3.0e38f)) return fmt("%s: eps must be finite and positive", what);
    return ok();
}

Result require_aligned4(const TesslBuf &b, const char *what)
{
    if (((uintptr_t)b.ptr & 15u) != 0) return fmt("%s: device pointer must be 16-byte aligned", what);
    return ok();
}

}  // namespace

namespace nn {

Result qwen35_rms_norm(TesslRuntime *rt, const TesslBuf &x, const TesslBuf &w, const TesslBuf &out, bool out_as_bf16,
                       uint32_t rows, uint32_t dim, float eps)
{
    const char *what = "qwen35::rms_norm";
    TESSL_TRY(validate_rms_scalars(dim, eps, what));
    const uint64_t n = elems(rows, dim);
    TESSL_TRY(require(x, n, 4, "rms_norm x"));
    TESSL_TRY(require(w, dim, 4, "rms_norm w"));
    TESSL_TRY(require(out, n, out_as_bf16 ? 2 : 4, "rms_norm out"));
    if (rows == 0) return ok();
    const Named writes[] = {{"out", &out}};
    if (out_as_bf16) {
        const Named reads[] = {{"x", &x}, {"w", &w}};
        TESSL_TRY(require_disjoint_writes(what, writes, 1, reads, 2));
    } else {
        // an f32 output may be x itself: every element is read and written by the same thread
        const Named reads[] = {{"w", &w}};
        TESSL_TRY(require_disjoint_writes(what, writes, 1, reads, 1));
        if (aliases(out, x) && out.ptr != x.ptr) return fmt("%s: out overlaps x without being x", what);
    }
    TESSL_TRY(require_aligned4(x, "rms_norm x"));
    TESSL_TRY(require_aligned4(out, "rms_norm out"));
    float *xp = static_cast<float *>(x.ptr);
    const float *wp = static_cast<const float *>(w.ptr);
    const char *launch = "qwen35_rms_norm launch";
    if (out_as_bf16) return launch_norm<false, true>(rt, launch, nullptr, xp, wp, out.ptr, rows, dim, eps);
    return launch_norm<false, false>(rt, launch, nullptr, xp, wp, out.ptr, rows, dim, eps);
}

Result qwen35_residual_add(TesslRuntime *rt, const TesslBuf &y, const TesslBuf &resid, uint32_t rows, uint32_t width)
{
    const char *what = "qwen35::residual_add";
    const uint64_t n = elems(rows, width);
    TESSL_TRY(require(y, n, 4, "residual_add y"));
    TESSL_TRY(require(resid, n, 4, "residual_add resid"));
    if (n == 0) return ok();
    const Named writes[] = {{"resid", &resid}};
    const Named reads[] = {{"y", &y}};
    TESSL_TRY(require_disjoint_writes(what, writes, 1, reads, 1));
    return launch_pdl(rt, "qwen35_residual_add launch", qwen35_residual_add_kernel, dim3((unsigned)((n + 255) / 256)), dim3(256), 0,
                      static_cast<const float *>(y.ptr), static_cast<float *>(resid.ptr), n);
}

Result qwen35_add_rms_norm(TesslRuntime *rt, const TesslBuf &y, const TesslBuf &resid, const TesslBuf &w, const TesslBuf &out,
                           bool out_as_bf16, uint32_t rows, uint32_t dim, float eps)
{
    const char *what = "qwen35::add_rms_norm";
    TESSL_TRY(validate_rms_scalars(dim, eps, what));
    const uint64_t n = elems(rows, dim);
    TESSL_TRY(require(y, n, 4, "add_rms_norm y"));
    TESSL_TRY(require(resid, n, 4, "add_rms_norm resid"));
    TESSL_TRY(require(w, dim, 4, "add_rms_norm w"));
    TESSL_TRY(require(out, n, out_as_bf16 ? 2 : 4, "add_rms_norm out"));
    if (rows == 0) return ok();
    const Named writes[] = {{"resid", &resid}, {"out", &out}};
    const Named reads[] = {{"y", &y}, {"w", &w}};
    TESSL_TRY(require_disjoint_writes(what, writes, 2, reads, 2));
    TESSL_TRY(require_aligned4(y, "add_rms_norm y"));
    TESSL_TRY(require_aligned4(resid, "add_rms_norm resid"));
    TESSL_TRY(require_aligned4(out, "add_rms_norm out"));
    const float *yp = static_cast<const float *>(y.ptr), *wp = static_cast<const float *>(w.ptr);
    float *rp = static_cast<float *>(resid.ptr);
    const char *launch = "qwen35_add_rms_norm launch";
    if (out_as_bf16) return launch_norm<true, true>(rt, launch, yp, rp, wp, out.ptr, rows, dim, eps);
    return launch_norm<true, false>(rt, launch, yp, rp, wp, out.ptr, rows, dim, eps);
}

}  // namespace nn
}  // namespace tessl
