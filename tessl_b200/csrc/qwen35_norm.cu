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
// One block per row, as wide as the row asks for; a thread holds its part of the row in registers, so
// a row costs one round trip to memory and one barrier. The rows are a few KB, so the kernels are
// latency-bound; they are launched with programmatic stream serialization so that a following GEMV can
// already stream its weights while they run. 512 threads of 32 registers (rows of up to 4096) fit an SM
// beside a block of the GEMV in front, so the block is resident when that one ends.
#include "q4_common.cuh"
#include "runtime.h"

namespace tessl {
namespace {

constexpr int kNormThreads = 512;  // at most

/// Sum over the block, the same value in every thread: lanes by xor butterfly, then the warps' sums likewise.
__device__ __forceinline__ float block_sum(float v, float *scratch)
{
    v = dev::warp_sum(v);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0) scratch[warp] = v;
    __syncthreads();
    return dev::warp_sum(lane < (int)(blockDim.x >> 5) ? scratch[lane] : 0.0f);
}

__device__ __forceinline__ float4 load4(const float *p)
{
    const uint4 v = dev::ld_after_wait16(p);
    return make_float4(__uint_as_float(v.x), __uint_as_float(v.y), __uint_as_float(v.z), __uint_as_float(v.w));
}

/// NV: float4 pieces of the row per thread, held in registers with their weights. NV = 0: any other row (its length no multiple of
/// 4, or too long to hold, or weights at an odd address), read twice. With 256 threads that read the row twice and its weights
/// word by word after the sum, a step of four layers of 4096 in a graph took 152.4 us; with this 130.6 (nine norms, 2.4 us each), five
/// streams over two layers of 2560 80.9 / 71.2.
template <bool ADD, bool OUT_BF16, int NV>
__global__ void __launch_bounds__(kNormThreads) qwen35_rms_norm_kernel(const float *y, float *x_or_resid, const float *weight,
                                                                      void *out, uint32_t dim, float eps)
{
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    __shared__ float scratch[kNormThreads / 32];
    const size_t base = (size_t)blockIdx.x * dim;
    const uint32_t tid = threadIdx.x, nt = blockDim.x;
    float *xr = x_or_resid + base;
    const float *yr = ADD ? y + base : nullptr;
    float ss = 0.0f;
    auto scale = [&] { return __fdiv_rn(1.0f, __fsqrt_rn(__fdiv_rn(block_sum(ss, scratch), (float)dim) + eps)); };
    if constexpr (NV > 0) {
        float4 v[NV], w[NV];
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const uint32_t d = (i * nt + tid) * 4;
            v[i] = w[i] = make_float4(0, 0, 0, 0);
            if (d < dim) {
                v[i] = load4(xr + d);
                if constexpr (ADD) {
                    const float4 a = load4(yr + d);
                    v[i].x += a.x, v[i].y += a.y, v[i].z += a.z, v[i].w += a.w;
                    *reinterpret_cast<float4 *>(xr + d) = v[i];
                }
                w[i] = load4(weight + d);
            }
        }
#pragma unroll
        for (int i = 0; i < NV; ++i)
            ss = fmaf(v[i].x, v[i].x, ss), ss = fmaf(v[i].y, v[i].y, ss), ss = fmaf(v[i].z, v[i].z, ss), ss = fmaf(v[i].w, v[i].w, ss);
        const float inv = scale();
        auto one = [&](float x, float wt) { return __fmul_rn(__fmul_rn(x, inv), 1.0f + wt); };
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const uint32_t d = (i * nt + tid) * 4;
            if (d >= dim) break;
            const float4 o = make_float4(one(v[i].x, w[i].x), one(v[i].y, w[i].y), one(v[i].z, w[i].z), one(v[i].w, w[i].w));
            if constexpr (OUT_BF16) {
                uint2 b;
                b.x = (uint32_t)dev::f32_to_bf16_store(o.x) | ((uint32_t)dev::f32_to_bf16_store(o.y) << 16);
                b.y = (uint32_t)dev::f32_to_bf16_store(o.z) | ((uint32_t)dev::f32_to_bf16_store(o.w) << 16);
                *reinterpret_cast<uint2 *>(static_cast<uint16_t *>(out) + base + d) = b;
            } else {
                *reinterpret_cast<float4 *>(static_cast<float *>(out) + base + d) = o;
            }
        }
    } else {
        for (uint32_t d = tid; d < dim; d += nt) {
            float v = xr[d];
            if constexpr (ADD) {
                v = v + yr[d];
                xr[d] = v;
            }
            ss = fmaf(v, v, ss);
        }
        const float inv = scale();
        for (uint32_t d = tid; d < dim; d += nt) {
            const float o = __fmul_rn(__fmul_rn(xr[d], inv), 1.0f + weight[d]);  // its own writes, if ADD
            if constexpr (OUT_BF16) {
                static_cast<uint16_t *>(out)[base + d] = dev::f32_to_bf16_store(o);
            } else {
                static_cast<float *>(out)[base + d] = o;
            }
        }
    }
}

template <bool ADD, bool OUT_BF16>
Result launch_norm(TesslRuntime *rt, const char *what, const float *y, float *x, const float *w, void *out, uint32_t rows, uint32_t dim,
                   float eps)
{
    // Rows start 16-byte aligned where dim is a multiple of 4 (the wrappers check the buffers; the weights' may be any).
    const uint32_t pieces = (dim + 3) / 4;
    uint32_t nv = (pieces + kNormThreads - 1) / kNormThreads;
    if (dim % 4 != 0 || nv > 4 || ((uintptr_t)w & 15u) != 0) nv = 0;
    const uint32_t nt = nv ? ((pieces + nv - 1) / nv + 31) & ~31u : kNormThreads;
    auto go = [&](auto kernel) { return launch_pdl(rt, what, kernel, dim3(rows), dim3(nt), 0, y, x, w, out, dim, eps); };
    switch (nv) {
    case 1: return go(qwen35_rms_norm_kernel<ADD, OUT_BF16, 1>);
    case 2: return go(qwen35_rms_norm_kernel<ADD, OUT_BF16, 2>);
    case 3: return go(qwen35_rms_norm_kernel<ADD, OUT_BF16, 3>);
    case 4: return go(qwen35_rms_norm_kernel<ADD, OUT_BF16, 4>);
    default: return go(qwen35_rms_norm_kernel<ADD, OUT_BF16, 0>);
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
    return launch_pdl(rt, "qwen35_residual_add launch", qwen35_residual_add_kernel, dim3((unsigned)((n + 255) / 256)), dim3(256), 0, static_cast<const float *>(y.ptr), static_cast<float *>(resid.ptr), n);
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
