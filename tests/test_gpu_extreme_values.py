"""Activations and scales at the ends of their ranges, in every tensor-core form of the small products (one row of x, one row
over windows, one row at another width, batches, 8-bit codes): what a form computes is the affine product in f32, whatever
power of two the activations of a slice are scaled by on their way to the tensor cores."""
import numpy as np
import pytest

from gpu_util import assert_gamma_bound, rt, seeded_f32, upload_bank  # noqa: F401
from oracle import api
from tessl_b200 import nn, synth

pytestmark = pytest.mark.gpu

ROWS = 24
# (m, columns, group): one kernel or window plan each
FORMS = [(1, 1024, 64), (1, 4096, 32), (1, 8192, 64), (1, 2560, 128), (1, 9216, 64), (8, 512, 64), (8, 2048, 32), (5, 4096, 128),
         (8, 12288, 64), (3, 9216, 64)]


def _bank(cols, group, scale):
    """Codes of any value, scales of one magnitude, biases about -8 scales."""
    packed, sb = synth.q4_bank(0x7E551400 + cols + group, ROWS, cols, group)
    f = synth.bf16_bits_to_f32(sb.reshape(-1)).reshape(-1, 2)
    s = (f[:, 0] / np.float32(0.01) * np.float32(scale)).astype(np.float32)
    sb = synth.f32_to_bf16_bits(np.stack((s, np.float32(-8.0) * s), axis=-1).reshape(-1))
    return packed.view(np.uint8).reshape(-1), sb


def _x(m, cols, seed):
    return synth.bf16_bits_to_f32(synth.normal_bf16(seed + cols, m * cols)).reshape(m, cols)


def _run(rt, packed, sb, x_bits, m, cols, group):
    bank, xb, y = upload_bank(rt, packed, sb), rt.buffer_from(x_bits), seeded_f32(rt, m * ROWS)
    shape = nn.QuantShape(ROWS, cols, group)
    if m == 1:
        nn.gemv_q4_mlx_simd(rt, bank, xb, y, shape)
    else:
        nn.gemm_q4_mlx(rt, bank, xb, y, shape, m)
    return y.read(np.float32, m * ROWS).reshape(m, ROWS)


@pytest.mark.parametrize("m,cols,group", FORMS)
@pytest.mark.parametrize("x_exp,s_exp", [(0, -124), (0, -118), (0, -90), (20, -120), (-20, 100), (-100, 120), (-60, 40), (104, -40),
                                         (-119, 6)])
def test_any_magnitude_of_activations_and_scales(rt, m, cols, group, x_exp, s_exp):
    """2^x_exp activations meet 2^s_exp scales; the intermediates of the plain f32 product are normal numbers."""
    packed, sb = _bank(cols, group, 2.0 ** s_exp)
    x = synth.f32_to_bf16_bits(_x(m, cols, 0x7E551410) * np.float32(2.0 ** x_exp)).reshape(-1)
    got = _run(rt, packed, sb, x, m, cols, group)
    assert_gamma_bound(got, packed, sb, x, m, ROWS, cols, group, what=f"x 2^{x_exp} scales 2^{s_exp}")


@pytest.mark.parametrize("m,cols,group", FORMS)
def test_subnormal_zero_and_mixed_activations(rt, m, cols, group):
    packed, sb = _bank(cols, group, 2.0 ** 10)
    base = _x(m, cols, 0x7E551420)
    k = np.arange(cols)
    tiny = base * np.float32(2.0 ** -128)                                       # mostly bf16 subnormals
    mixed = base * np.where((k // 16) % 3 == 0, 2.0 ** -120, np.where((k // 16) % 3 == 1, 1.0, 2.0 ** -30)).astype(np.float32)
    slices = base * np.where((k * 16 // cols) % 2 == 0, 0.0, 2.0 ** -122).astype(np.float32)  # whole slices of zeros
    for what, v in (("subnormal", tiny), ("mixed", mixed), ("zero slices", slices)):
        x = synth.f32_to_bf16_bits(v).reshape(-1)
        got = _run(rt, packed, sb, x, m, cols, group)
        assert_gamma_bound(got, packed, sb, x, m, ROWS, cols, group, what=what)
    assert np.all(_run(rt, packed, sb, np.zeros(m * cols, np.uint16), m, cols, group) == 0.0)


@pytest.mark.parametrize("m,cols,group", FORMS)
@pytest.mark.parametrize("bits", [0x7F80, 0xFF80, 0x7FC0])
def test_infinities_and_nans_stay_in_their_row(rt, m, cols, group, bits):
    """An Inf or a NaN meets codes of both signs of (code - 8): every output of its row of x is Inf or NaN, no other row
    of a batch changes a bit."""
    packed, sb = _bank(cols, group, 0.01)
    x = synth.f32_to_bf16_bits(_x(m, cols, 0x7E551430)).reshape(m, cols)
    clean = _run(rt, packed, sb, x.reshape(-1), m, cols, group)
    bad = m // 2
    x[bad, cols - 5] = bits
    got = _run(rt, packed, sb, x.reshape(-1), m, cols, group)
    assert not np.any(np.isfinite(got[bad]))
    keep = np.arange(m) != bad
    assert np.array_equal(got[keep].view(np.uint32), clean[keep].view(np.uint32))


@pytest.mark.parametrize("m", [1, 4])
@pytest.mark.parametrize("cols,group", [(512, 32), (2048, 64), (4096, 32)])
@pytest.mark.parametrize("x_exp,s_exp", [(0, -124), (0, -118), (-20, 100), (104, -40), (-119, 6)])
def test_any_magnitude_in_the_8_bit_form(rt, m, cols, group, x_exp, s_exp):
    codes, sb = synth.q8_bank(0x7E551440 + cols, ROWS, cols, group)
    f = synth.bf16_bits_to_f32(sb.reshape(-1)).reshape(-1, 2)
    s = (f[:, 0] / f[:, 0].max() * np.float32(2.0 ** s_exp)).astype(np.float32)
    sb = synth.f32_to_bf16_bits(np.stack((s, np.float32(-128.0) * s), axis=-1).reshape(-1))
    x = synth.f32_to_bf16_bits(_x(m, cols, 0x7E551450) * np.float32(2.0 ** x_exp)).reshape(-1)
    y = seeded_f32(rt, m * ROWS)
    nn.gemm_q8_mlx(rt, rt.buffer_from(codes), rt.buffer_from(sb), rt.buffer_from(x), y, nn.QuantShape(ROWS, cols, group), m)
    got = y.read(np.float32, m * ROWS).reshape(m, ROWS).astype(np.float64)
    w8 = codes.view(np.uint8).reshape(ROWS, cols).astype(np.float64)
    sf = synth.bf16_bits_to_f32(sb).astype(np.float64).reshape(ROWS, cols // group, 2).repeat(group, axis=1)
    xf = synth.bf16_bits_to_f32(x).astype(np.float64).reshape(m, cols)
    want = xf @ (w8 * sf[..., 0] + sf[..., 1]).T
    mag = np.abs(xf) @ (w8 * np.abs(sf[..., 0]) + np.abs(sf[..., 1])).T
    assert np.all(np.isfinite(got))
    assert np.all(np.abs(got - want) <= api.gamma(cols + 2 * (cols // group)) * mag)
