"""The prefill kernel for few rows of X, which divides K over a cluster: every cluster size, partial tiles of rows and of X, an odd
number of K blocks, scale words that come in pieces of one, two and four, with and without tiles of them, against the exact
product (gamma_t S of the whole K: the sums of the parts are shorter chains)."""
import numpy as np
import pytest

from gpu_util import SENTINEL_F32, assert_gamma_bound, assert_north_star, rt, seeded_f32, upload_bank  # noqa: F401
from oracle import api
from tessl_b200 import nn, synth

pytestmark = pytest.mark.gpu


def _run(rt, m, n, k, group, split, sb_offset=0):
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
    assert rt.last_prefill_tile() == (64, 1) and rt.last_prefill_split() == split
    out = y.read(np.float32, m * n + 256)
    assert np.all(out[m * n:] == SENTINEL_F32), "wrote past y"
    yb = rt.buffer_from(np.full(m * n + 256, 0xA5A5, np.uint16))
    nn.gemm_q4_mlx_tensorops(rt, bank, xb, yb, shape, m, y_as_bf16=True)
    gb = yb.read(np.uint16, m * n + 256)
    assert np.all(gb[m * n:] == 0xA5A5) and np.array_equal(gb[: m * n], synth.f32_to_bf16_bits(out[: m * n]))
    return packed, sb, x, out[: m * n].reshape(m, n)


def _check(packed, sb, x, got, m, n, k, group):
    rows = np.array(sorted({r for r in (0, 7, 8, 31, 32, m // 2, 79, 80, 127, 128, 159, 160, m - 1) if r < m}))
    xs = np.ascontiguousarray(x.reshape(m, k)[rows]).reshape(-1)
    assert_north_star(got[rows], api.q4_dense_gemm(packed, sb, xs, len(rows), n, k, group), "rows")
    assert_gamma_bound(got[rows].reshape(-1), packed, sb, xs, len(rows), n, k, group, extra_terms=group, what="rows")
    w = api.q4_dequant(packed, sb, n, k, group).astype(np.float64)
    want = w @ synth.bf16_bits_to_f32(x).reshape(m, k).astype(np.float64).sum(axis=0)
    g64 = got.astype(np.float64)
    assert np.all(np.abs(g64.sum(axis=0) - want) <= 1e-5 * np.abs(g64).sum(axis=0) + 1e-3)  # every output takes part


@pytest.mark.parametrize("m,n,k,group,split", [
    (25, 128, 1088, 64, 4),      # 17 main K blocks: a last unit of one; 17 groups: no tiles of scale words, pieces of one
    (16, 1, 1152, 64, 5),        # one weight row; pieces of two
    (33, 257, 2080, 32, 5),      # pieces of one, two per K block; 65 groups
    (40, 300, 2048, 32, 6),      # pieces of four
    (100, 4096, 2048, 32, 4),
    (25, 129, 4224, 128, 6),     # a group per unit
    (77, 4096, 12288, 64, 4),
    (128, 3072, 2048, 64, 5), (100, 2048, 4096, 64, 6),
    (48, 6144, 4096, 128, 2), (160, 5504, 2048, 64, 3),
    (64, 12288, 1024, 64, 1), (161, 9216, 1024, 32, 1),
    (320, 1024, 4096, 64, 5), (200, 2560, 9216, 64, 3),  # two tiles of X
    (25, 20000, 2048, 64, 1),    # more tiles than SMs
])
def test_split_matches_the_exact_product(rt, m, n, k, group, split):
    """The clusters that the library picks."""
    _check(*_run(rt, m, n, k, group, split), m, n, k, group)


@pytest.mark.parametrize("split", [1, 2, 3, 4, 5, 6])
@pytest.mark.parametrize("m,n,k,group", [(33, 257, 2080, 32), (9, 130, 2048, 64), (161, 300, 2048, 32), (300, 129, 1600, 64), (40, 1, 1536, 32)])
def test_every_cluster_size(rt, split, m, n, k, group):
    """Scale words in pieces of one, two and four with every number of CTAs per tile, up to the fewest K blocks that one may have."""
    rt.set_prefill_split(split)
    try:
        _check(*_run(rt, m, n, k, group, split), m, n, k, group)
    finally:
        rt.set_prefill_split(-1)


def test_the_choice_can_be_forced_and_asked_for(rt):
    packed, sb = synth.q4_bank(0x7E553190, 64, 1024, 64)
    bank, shape = upload_bank(rt, packed.view(np.uint8).reshape(-1), sb.reshape(-1)), nn.QuantShape(64, 1024, 64)
    xb, y = rt.buffer_from(synth.normal_bf16(0x7E553191, 40 * 1024)), seeded_f32(rt, 40 * 64)
    try:
        for split, want in ((4, ((64, 1), 4)), (0, ((64, 1), 0))):
            rt.set_prefill_split(split)
            nn.gemm_q4_mlx_tensorops(rt, bank, xb, y, shape, 40)
            assert (rt.last_prefill_tile(), rt.last_prefill_split()) == want
        nn.gemm_q4_mlx_tensorops(rt, bank, xb, y, shape, 8)  # a few rows: no tile kernel
        assert (rt.last_prefill_tile(), rt.last_prefill_split()) == ((0, 0), 0)
        rt.set_prefill_split(5)  # 16 + 1 blocks of 64 columns
        rt.take_dispatch_count()
        with pytest.raises(nn.TesslError, match="17 blocks, a split over 5 CTAs takes 20"):
            nn.gemm_q4_mlx_tensorops(rt, bank, xb, y, shape, 40)
        assert rt.take_dispatch_count() == 0
        for bad in (-2, 7):
            with pytest.raises(nn.TesslError, match="outside -1 .. 6"):
                rt.set_prefill_split(bad)
    finally:
        rt.set_prefill_split(-1)


def test_scale_words_at_a_four_byte_boundary_give_the_same_bits(rt):
    a, b = _run(rt, 40, 300, 2048, 64, 5)[3], _run(rt, 40, 300, 2048, 64, 5, sb_offset=4)[3]
    assert np.array_equal(a.view(np.uint32), b.view(np.uint32))


def test_long_rows_of_x(rt):
    """The pre-pass holds one or two chunks of a row per thread, or reads longer rows twice."""
    for k in (6144, 6208, 12288, 12352, 20480):
        packed, sb, x, got = _run(rt, 26, 130, k, 64, 6)
        assert_gamma_bound(got.reshape(-1), packed, sb, x, 26, 130, k, 64, extra_terms=64, what=f"K={k}")
