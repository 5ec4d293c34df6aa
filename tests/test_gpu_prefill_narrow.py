"""The 64-wide tile of the CTA-pair prefill GEMM, which the library picks when wider tiles would leave clusters idle: ragged
edges in both directions, every group size, f32 and bf16, against the exact product. Some of these shapes are the split
kernel's by choice; they are kept from it here."""
import numpy as np
import pytest

from gpu_util import SENTINEL_F32, assert_gamma_bound, assert_north_star, rt, seeded_f32, upload_bank  # noqa: F401
from oracle import api
from tessl_b200 import nn, synth

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _pair_kernel(rt):
    rt.set_prefill_split(0)
    yield
    rt.set_prefill_split(-1)


@pytest.mark.parametrize("m,n,k,group", [(77, 4096, 1536, 64), (33, 65, 2080, 32), (25, 300, 4224, 128), (257, 1999, 1088, 64),
                                         (512, 2368, 512, 128), (509, 2048, 2048, 64)])
def test_narrow_tiles_match_the_exact_product(rt, m, n, k, group):
    packed, sb = synth.q4_bank(0x7E552100 + n + m, n, k, group)
    packed, sb = packed.view(np.uint8).reshape(-1), sb.reshape(-1)
    x = synth.normal_bf16(0x7E552107 + m, m * k)
    bank, xb, shape = upload_bank(rt, packed, sb), rt.buffer_from(x), nn.QuantShape(n, k, group)
    y = seeded_f32(rt, m * n, 256)
    nn.gemm_q4_mlx_tensorops(rt, bank, xb, y, shape, m)
    assert rt.last_prefill_tile() == (64, 1) and rt.last_prefill_split() == 0
    out = y.read(np.float32, m * n + 256)
    assert np.all(out[m * n:] == SENTINEL_F32), "wrote past y"
    got = out[: m * n].reshape(m, n)
    rows = np.array(sorted({0, 31, 32, m // 2, m - 1} | {r for r in (127, 128, 255, 256) if r < m}))
    rows = rows[rows < m]
    xs = np.ascontiguousarray(x.reshape(m, k)[rows]).reshape(-1)
    assert_north_star(got[rows], api.q4_dense_gemm(packed, sb, xs, len(rows), n, k, group), "rows")
    assert_gamma_bound(got[rows].reshape(-1), packed, sb, xs, len(rows), n, k, group, extra_terms=group, what="rows")
    w = api.q4_dequant(packed, sb, n, k, group).astype(np.float64)
    want = w @ synth.bf16_bits_to_f32(x).reshape(m, k).astype(np.float64).sum(axis=0)
    g64 = got.astype(np.float64)
    assert np.all(np.abs(g64.sum(axis=0) - want) <= 1e-5 * np.abs(g64).sum(axis=0) + 1e-3)  # every output takes part
    yb = rt.buffer_from(np.full(m * n + 256, 0xA5A5, np.uint16))
    nn.gemm_q4_mlx_tensorops(rt, bank, xb, yb, shape, m, y_as_bf16=True)
    gb = yb.read(np.uint16, m * n + 256)
    assert np.all(gb[m * n:] == 0xA5A5) and np.array_equal(gb[: m * n], synth.f32_to_bf16_bits(got.reshape(-1)))


@pytest.mark.parametrize("m,n,k,group,forced", [(19500, 60, 192, 64, False), (700, 20011, 128, 128, True), (300, 9000, 384, 32, True),
                                                (40, 72, 2048, 64, True)])
def test_several_narrow_tiles_per_cluster(rt, m, n, k, group, forced):
    """More tiles than clusters: both accumulator buffers, a ring position and dequant groups carried across tiles."""
    packed, sb = synth.q4_bank(0x7E552200 + n, n, k, group)
    packed, sb = packed.view(np.uint8).reshape(-1), sb.reshape(-1)
    x = synth.normal_bf16(0x7E552207 + m, m * k)
    bank, xb, shape = upload_bank(rt, packed, sb), rt.buffer_from(x), nn.QuantShape(n, k, group)
    y = seeded_f32(rt, m * n, 1024)
    if forced:
        rt.set_prefill_tile(64, 1)
    try:
        nn.gemm_q4_mlx_tensorops(rt, bank, xb, y, shape, m)
    finally:
        rt.set_prefill_tile(0, -1)
    assert rt.last_prefill_tile() == (64, 1) and rt.last_prefill_split() == 0
    out = y.read(np.float32, m * n + 1024)
    assert np.all(out[m * n:] == SENTINEL_F32), "wrote past y"
    got = out[: m * n].reshape(m, n)
    assert_north_star(got, api.q4_dense_gemm(packed, sb, x, m, n, k, group), "every output")
    rows = np.unique(np.linspace(0, m - 1, 24).astype(int))
    xs = np.ascontiguousarray(x.reshape(m, k)[rows]).reshape(-1)
    assert_gamma_bound(got[rows].reshape(-1), packed, sb, xs, len(rows), n, k, group, extra_terms=group, what="rows")


def test_the_narrow_tile_needs_the_pair(rt):
    for pair in (0, -1):
        with pytest.raises(nn.TesslError, match="two-CTA kernel only"):
            rt.set_prefill_tile(64, pair)
