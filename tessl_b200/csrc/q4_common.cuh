// Device helpers shared by the MLX Q4/Q8 kernels: streaming loads, bf16
// widening/narrowing with the reference's store rule, nibble-to-float tricks and
// the activations of kernels/act.h (reference project path).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace tessl {
namespace dev {

/// 16-byte read-only load that does not allocate in L1: weights are touched
/// exactly once per launch.
__device__ __forceinline__ uint4 ldg_stream16(const void *p)
{
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(p));
    return v;
}

__device__ __forceinline__ uint32_t ldg_stream4(const void *p)
{
    uint32_t v;
    asm volatile("ld.global.nc.L1::no_allocate.u32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}

/// Loads of data that the preceding kernel of the stream may have written, for kernels launched with programmatic
/// stream serialization: coherent, and volatile so that the compiler keeps them behind `griddepcontrol.wait`. A
/// read-only load (`__ldg`) is neither: the compiler may move it in front of the wait, and did (a GEMV over 2560
/// columns read its activations before the norm that wrote them had run).
__device__ __forceinline__ uint4 ld_after_wait16(const void *p)
{
    uint4 v;
    asm volatile("ld.global.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ uint2 ld_after_wait8(const void *p)
{
    uint2 v;
    asm volatile("ld.global.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p) : "memory");
    return v;
}

/// The two bf16 halves of a word, widened (a bf16 is the top half of an f32).
__device__ __forceinline__ float bf16_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }

/// Power-of-two scaling of a slice of bf16 activations that meets nibbles held as bf16 subnormals (q * 2^-133): `mul` =
/// (2^e, 2^e) and `mul16` = (2^(e-4), 2^(e-4)) as bf16 pairs, `undo` = 2^(133-e). e brings the slice's largest magnitude
/// to 2^126, as far as a bf16 factor (e <= 127) and an f32 undo (e >= 6) can. The affine fold of the slice then runs in
/// units of `undo` (`scaled_sum`: a group sum in those units), without a multiplication per dot product, and rounds as
/// the plain values do wherever nothing leaves the range:
///   * `undo` >= 2^6, so no sum overflows before the plain one would;
///   * it is the smallest unit that can be had (2^6, or 2^7 times the slice's largest power of two), so the fold reaches
///     the f32 subnormals only with scales below 2^-122 (the smallest normal bf16 is 2^-126), or results below 2^-120. With the
///     slice brought to 2^100 only, scales below 2^-93 lost their bits;
///   * products are multiples of 2^-149 as long as the slice's largest magnitude is below 2^10, subnormal activations
///     included, so the tensor cores lose none; above, those over 2^135 times smaller than the largest lose bits;
///   * from 2^122 on a scaled activation overflows: Inf or NaN results, as from f32 sums of a group of such activations.
struct XScale {
    uint32_t mul, mul16;
    float undo, sum1;
};
__device__ __forceinline__ XScale x_scale(uint32_t amax)
{
    const int e = min(127, max(6, 126 + 127 - (int)(amax >> 7)));
    return XScale{(uint32_t)(e + 127) * 0x00800080u, (uint32_t)(e + 123) * 0x00800080u, __uint_as_float((uint32_t)(127 + 133 - e) << 23),
                  __uint_as_float((uint32_t)(e + 57) << 23)};
}
/// sum * 2^(e - 133), in two factors that are normal for every e.
__device__ __forceinline__ float scaled_sum(float sum, const XScale &s) { return sum * s.sum1 * 0x1p-63f; }
__device__ __forceinline__ uint32_t bf2_mul(uint32_t a, uint32_t b)
{
    uint32_t r;
    asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
/// Eight activations -> the B registers of the two MMAs that take the eight nibbles of a packed word:
/// (x0, x4), (x1, x5) / 16, (x2, x6), (x3, x7) / 16, scaled. Only exponents change (within the bounds above).
__device__ __forceinline__ void x_fragment(const uint4 &v, const XScale &s, uint32_t (&f)[4])
{
    f[0] = bf2_mul(__byte_perm(v.x, v.z, 0x5410), s.mul), f[1] = bf2_mul(__byte_perm(v.x, v.z, 0x7632), s.mul16);
    f[2] = bf2_mul(__byte_perm(v.y, v.w, 0x5410), s.mul), f[3] = bf2_mul(__byte_perm(v.y, v.w, 0x7632), s.mul16);
}

/// f32 -> bf16 bits as the reference's device cast stores them
/// (`f32_to_bf16_bits_gpu`, src/tensor.rs:815-831 of the reference project):
/// any NaN becomes 0x7fc0, an f32 subnormal flushes to a zero of its sign,
/// everything else rounds to nearest even.
__device__ __forceinline__ uint16_t f32_to_bf16_store(float x)
{
    const uint32_t bits = __float_as_uint(x);
    const uint32_t mag = bits & 0x7fffffffu;
    if (mag > 0x7f800000u) return 0x7fc0u;
    if (mag < 0x00800000u) return (uint16_t)((bits >> 16) & 0x8000u);
    return (uint16_t)((bits + 0x7fffu + ((bits >> 16) & 1u)) >> 16);
}

/// Byte `B` of `bytes` (each byte one nibble value 0..15) as the float
/// 128 + q: the byte lands in mantissa bits 16..23 under exponent 2^7. One
/// PRMT, no integer-to-float conversion.
template <int B>
__device__ __forceinline__ float nib_byte_to_f128(uint32_t bytes)
{
    return __uint_as_float(__byte_perm(bytes, 0x00004300u, 0x5044u | (B << 8)));
}

/// kernels/act.h:36-46 (reference project): sigmoid through e = exp(-|x|) so
/// no intermediate overflows, then x * sigmoid(x).
__device__ __forceinline__ float silu(float x)
{
    const float e = expf(-fabsf(x));
    const float r = __fdiv_rn(1.0f, 1.0f + e);
    return x * (x >= 0.0f ? r : e * r);
}

/// kernels/act.h:24-30 (reference project): tanh-approximate GELU with the
/// cubic's input clamped to +-20 and the tanh argument to +-10; the outer
/// factor stays the original x.
__device__ __forceinline__ float gelu_pytorch_tanh(float x)
{
    const float xc = fminf(fmaxf(x, -20.0f), 20.0f);
    const float x3 = xc * xc * xc;
    const float inner = 0.7978845608028654f * (xc + 0.044715f * x3);
    const float t = tanhf(fminf(fmaxf(inner, -10.0f), 10.0f));
    return 0.5f * x * (1.0f + t);
}

__device__ __forceinline__ float warp_sum(float v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

}  // namespace dev
}  // namespace tessl
