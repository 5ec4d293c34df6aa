"""The prefill kernel for few rows of X, which divides K over a cluster: every cluster size, partial tiles of rows and of X, an odd
number of K blocks, scale words that come in pieces of one, two and four, with and without tiles of them, against the exact
product (gamma_t S of the whole K: the sums of the parts are shorter chains)."""
import numpy as np
import pytest

from gpu_util import SENTINEL_F32, assert_gamma_bound, assert_north_star, rt, seeded_f32, upload_bank  # noqa: F401
from oracle import api
from tessl_b200 import nn, synth

pytestmark = pytest.mark.gpu


def _run(rt, m, n, k, group, sb_offset=0):
    packed, sb = synth.q4_bank(0x7E553100 + n + m, n, k, group)
    packed, sb = packed.view(np.uint8).reshape(-1), sb.reshape(-1)
    x = synth.normal_bf16(0x7E553107 + m, m * k)
    bank, xb, shape = upload_bank(rt, packed, sb), rt.buffer_from(x), nn.QuantShape(n, k, group)
    if sb_offset:
        big = rt.alloc_buffer(sb.nbytes + sb_offset)
        big.write(sb, sb_offset)
        bank = nn.Q4MlxBank(bank.packed, big.view(sb_offset, sb.nbytes))
    y = seeded_f32(rt, m * n, 256)
    nn.gemm_q4_mlx_tensorops(rt, bank, xb, y, shape, m)
    assert rt.last_prefill_tile() == (64, 1)
    out = y.read(np.float32, m * n + 256)
    assert np.all(out[m * n:] == SENTINEL_F32), "wrote past y"
    yb = rt.buffer_from(np.full(m * n + 256, 0xA5A5, np.uint16))
    nn.gemm_q4_mlx_tensorops(rt, bank, xb, yb, shape, m, y_as_bf16=True)
    gb = yb.read(np.uint16, m * n + 256)
    assert np.all(gb[m * n:] == 0xA5A5) and np.array_equal(gb[: m * n], synth.f32_to_bf16_bits(out[: m * n]))
    return packed, sb, x, out[: m * n].reshape(m, n)


@pytest.mark.parametrize("m,n,k,group", [
    (25, 128, 1088, 64),      # 17 main K blocks: a last unit of one; 17 groups: no tiles of scale words, pieces of one
    (16, 1, 1152, 64),        # one weight row; pieces of two
    (33, 257, 2080, 32),      # pieces of one, two per K block; 65 groups
    (40, 300, 1024, 32),      # pieces of four
    (25, 129, 4224, 128),     # a group per unit
    (77, 4096, 12288, 64),    # clusters of four
    (128, 3072, 2048, 64), (100, 2048, 4096, 64),  # of five, of six
    (48, 6144, 4096, 128), (160, 5504, 2048, 64),  # of two, of three
    (64, 12288, 1024, 64), (161, 9216, 1024, 32),  # one CTA per tile
    (320, 1024, 4096, 64), (200, 2560, 9216, 64),  # two tiles of X
    (25, 20000, 2048, 64),    # more tiles than SMs
])
def test_split_matches_the_exact_product(rt, m, n, k, group):
    packed, sb, x, got = _run(rt, m, n, k, group)
    rows = np.array(sorted({r for r in (0, 7, 8, 31, 32, m // 2, 79, 80, 127, 128, 159, 160, m - 1) if r < m}))
    xs = np.ascontiguousarray(x.reshape(m, k)[rows]).reshape(-1)
    assert_north_star(got[rows], api.q4_dense_gemm(packed, sb, xs, len(rows), n, k, group), "rows")
    assert_gamma_bound(got[rows].reshape(-1), packed, sb, xs, len(rows), n, k, group, extra_terms=group, what="rows")
    w = api.q4_dequant(packed, sb, n, k, group).astype(np.float64)
    want = w @ synth.bf16_bits_to_f32(x).reshape(m, k).astype(np.float64).sum(axis=0)
    g64 = got.astype(np.float64)
    assert np.all(np.abs(g64.sum(axis=0) - want) <= 1e-5 * np.abs(g64).sum(axis=0) + 1e-3)  # every output takes part


def test_scale_words_at_a_four_byte_boundary_give_the_same_bits(rt):
    a, b = _run(rt, 40, 300, 2048, 64)[3], _run(rt, 40, 300, 2048, 64, sb_offset=4)[3]
    assert np.array_equal(a.view(np.uint32), b.view(np.uint32))


def test_long_rows_of_x(rt):
    """The pre-pass holds one or two chunks of a row per thread, or reads longer rows twice."""
    for k in (6144, 6208, 12288, 12352, 20480):
        packed, sb, x, got = _run(rt, 26, 130, k, 64)
        assert_gamma_bound(got.reshape(-1), packed, sb, x, 26, 130, k, 64, extra_terms=64, what=f"K={k}")
