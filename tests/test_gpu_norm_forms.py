"""Every form of the norm kernel: one to four pieces of a row per thread with a last thread in use or not, rows that are read twice
(odd lengths, long ones, weights at an odd address), alone and with the residual add, against the product in 64 bits."""
import numpy as np
import pytest

from gpu_util import SENTINEL_F32, rt, seeded_f32  # noqa: F401
from oracle import api
from tessl_b200 import nn, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,w_offset", [(4, 0), (124, 0), (2048, 0), (2052, 0), (4096, 0), (5120, 0), (6148, 0), (8192, 0), (8196, 0),
                                          (2047, 0), (4096, 4)])
def test_norm_forms(rt, dim, w_offset):
    rows, eps = 3, 1e-6
    d = synth.splitmix_draws(0x7E553300 + dim, rows * dim * 2 + dim)
    x, y = synth.unit_from_draws(d[: rows * dim]) * np.float32(3.0), synth.unit_from_draws(d[rows * dim: 2 * rows * dim])
    w = synth.unit_from_draws(d[2 * rows * dim:]) * np.float32(0.5)
    wb = rt.alloc_buffer(w.nbytes + w_offset)
    wb.write(w, w_offset)
    wb = wb.view(w_offset, w.nbytes)
    of = seeded_f32(rt, rows * dim, 16)
    nn.qwen35_rms_norm(rt, rt.buffer_from(x), wb, of, False, rows, dim, eps)
    got = of.read(np.float32, rows * dim + 16)
    assert np.all(got[rows * dim:] == SENTINEL_F32)
    # f32 sums of at most 17 squares in a row (8196 columns over 512 chains in pieces of four) and ten levels: far inside 2e-6 of the root
    np.testing.assert_allclose(got[: rows * dim].reshape(rows, dim), api.qwen35_rms_norm_f64(x, w, rows, dim, eps), rtol=2e-6, atol=1e-6)
    r1, r2, yb = rt.buffer_from(x), rt.buffer_from(x), rt.buffer_from(y)
    o1, o2 = rt.alloc_buffer(rows * dim * 4), rt.alloc_buffer(rows * dim * 4)
    nn.qwen35_residual_add(rt, yb, r1, rows, dim)
    nn.qwen35_rms_norm(rt, r1, wb, o1, True, rows, dim, eps)
    nn.qwen35_add_rms_norm(rt, yb, r2, wb, o2, True, rows, dim, eps)
    assert np.array_equal(r1.read(np.uint32, rows * dim), r2.read(np.uint32, rows * dim))
    assert np.array_equal(o1.read(np.uint16, rows * dim), o2.read(np.uint16, rows * dim))


def _outputs(rt, x, y, wb, rows, dim, bf16):
    """The norm, the sum and its norm, as bits."""
    word = np.uint16 if bf16 else np.uint32
    r, o1, o2 = rt.buffer_from(x), rt.alloc_buffer(rows * dim * 4), rt.alloc_buffer(rows * dim * 4)
    nn.qwen35_rms_norm(rt, r, wb, o1, bf16, rows, dim, 1e-6)
    nn.qwen35_add_rms_norm(rt, rt.buffer_from(y), r, wb, o2, bf16, rows, dim, 1e-6)
    out = [o1.read(word, rows * dim), o2.read(word, rows * dim), r.read(np.uint32, rows * dim)]
    for b in (r, o1, o2):
        b.free()
    return out


@pytest.mark.parametrize("dim", [4, 60, 124, 1028, 2048, 2052, 3072, 4100, 6148, 8192, 8196, 12288, 16388, 2047, 9217])
def test_bits_depend_on_the_rows_alone(rt, dim):
    """The same rows with their weights at any address of a float, and among many rows (whose blocks hold two chains per thread)."""
    rows, many = 3, 1025
    d = synth.splitmix_draws(0x7E553500 + dim, rows * dim * 2 + dim)
    x, y = synth.unit_from_draws(d[: rows * dim]) * np.float32(3.0), synth.unit_from_draws(d[rows * dim: 2 * rows * dim])
    w = synth.unit_from_draws(d[2 * rows * dim:]) * np.float32(0.5)
    tile = lambda a: np.tile(a.reshape(rows, dim), (many // rows + 1, 1))[:many].reshape(-1)  # noqa: E731
    for bf16 in (False, True):
        want = _outputs(rt, x, y, rt.buffer_from(w), rows, dim, bf16)
        for offset in (4, 8, 12):
            big = rt.alloc_buffer(w.nbytes + offset)
            big.write(w, offset)
            got = _outputs(rt, x, y, big.view(offset, w.nbytes), rows, dim, bf16)
            assert all(np.array_equal(a, b) for a, b in zip(got, want)), offset
        got = _outputs(rt, tile(x), tile(y), rt.buffer_from(w), many, dim, bf16)
        assert all(np.array_equal(a, tile(b)) for a, b in zip(got, want))


@pytest.mark.parametrize("dim,w_offset", [(9217, 0), (12288, 4), (16384, 0), (32768, 0)])
def test_long_rows(rt, dim, w_offset):
    rows = 2
    d = synth.splitmix_draws(0x7E553600 + dim, rows * dim + dim)
    x, w = synth.unit_from_draws(d[: rows * dim]) * np.float32(3.0), synth.unit_from_draws(d[rows * dim:]) * np.float32(0.5)
    wb = rt.alloc_buffer(w.nbytes + w_offset)
    wb.write(w, w_offset)
    of = seeded_f32(rt, rows * dim, 16)
    nn.qwen35_rms_norm(rt, rt.buffer_from(x), wb.view(w_offset, w.nbytes), of, False, rows, dim, 1e-6)
    got = of.read(np.float32, rows * dim + 16)
    assert np.all(got[rows * dim:] == SENTINEL_F32)
    # a chain of at most 64 squares: gamma of 64 + 10 operations on a sum of squares is 4.5e-6 of it, half of that of its root
    np.testing.assert_allclose(got[: rows * dim].reshape(rows, dim), api.qwen35_rms_norm_f64(x, w, rows, dim, 1e-6), rtol=3e-6, atol=1e-6)
