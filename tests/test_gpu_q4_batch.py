"""The batch kernel (csrc/q4_batch_mma.cuh) where its cutting of a row can go wrong: one chunk, groups that do not divide
evenly among the warps, one to eight windows (even and uneven) in a cluster, ragged row counts, every batch size, and the
widths just outside its domain, against the exact product within the reference's own bound."""
import numpy as np
import pytest

import ref_cases as rc
from gpu_util import SENTINEL_F32, assert_gamma_bound, assert_north_star, rt, seeded_f32, upload_bank  # noqa: F401
from oracle import api
from tessl_b200 import nn, synth

pytestmark = pytest.mark.gpu

SHAPES = [(1, 256, 64), (15, 256, 32), (33, 512, 128), (17, 768, 64), (64, 1024, 128), (40, 2560, 64), (40, 2304, 32),
          (48, 2560, 128), (31, 3840, 32), (2400, 2560, 64),
          # more than one window: 9 + 8 chunks, 3 even, 14 + 13 + 14 + 13 + 14, groups of 32 and 128, the widest (8)
          (33, 4352, 64), (4111, 9216, 64), (16, 17408, 64), (33, 4608, 32), (40, 12800, 128), (20, 32768, 64),
          # outside the domain: not a whole chunk, not a whole quad of groups, too many windows
          (40, 1408, 64), (40, 2304, 128), (8, 33024, 64)]


@pytest.mark.parametrize("rows,cols,group", SHAPES)
def test_batches_over_any_width(rt, rows, cols, group):
    packed, sb = synth.q4_bank(0x7E551000 + rows + cols, rows, cols, group)
    packed, sb = packed.view(np.uint8).reshape(-1), sb.reshape(-1)
    bank, shape = upload_bank(rt, packed, sb), nn.QuantShape(rows, cols, group)
    first = None
    for m in (1, 2, 5, 8):
        x = synth.normal_bf16(0x7E551077 + cols, 8 * cols)[: m * cols]
        xb, y = rt.buffer_from(x), seeded_f32(rt, m * rows, 8)
        rt.take_dispatch_count()
        if m == 1:
            nn.gemv_q4_mlx_simd(rt, bank, xb, y, shape)
        else:
            nn.gemm_q4_mlx(rt, bank, xb, y, shape, m)
        assert rt.take_dispatch_count() == 1
        got = y.read(np.float32, m * rows + 8)
        assert np.all(got[m * rows:] == SENTINEL_F32), "wrote past y"
        got = got[: m * rows].reshape(m, rows)
        assert_north_star(got, api.q4_dense_gemm(packed, sb, x, m, rows, cols, group), f"m={m}")
        assert_gamma_bound(got, packed, sb, x, m, rows, cols, group, what=f"m={m}")
        if m >= 2:  # a row's result does not depend on what else is in the batch
            if first is not None:
                assert np.array_equal(got[:2].view(np.uint32), first)
            first = got[:2].view(np.uint32).copy()
        # the residual is one f32 add (in place too), a bf16 result the rounded f32 one
        resid = rc.rand_f32(m * rows, 0x5300 + rows * m)
        r, yb = rt.buffer_from(resid), rt.buffer_from(np.full(m * rows + 8, 0xA5A5, np.uint16))
        call = (lambda out, **kw: nn.gemv_q4_mlx_simd(rt, bank, xb, out, shape, **kw)) if m == 1 else (
            lambda out, **kw: nn.gemm_q4_mlx(rt, bank, xb, out, shape, m, **kw))
        call(r, resid=r)
        assert np.array_equal(r.read(np.float32, m * rows), got.reshape(-1) + resid)
        call(yb, y_as_bf16=True)
        gb = yb.read(np.uint16, m * rows + 8)
        assert np.all(gb[m * rows:] == 0xA5A5) and np.array_equal(gb[: m * rows], synth.f32_to_bf16_bits(got.reshape(-1)))


@pytest.mark.parametrize("rows,cols,group", [(40, 2560, 64), (7, 768, 64), (100, 5120, 128), (17, 9216, 64), (64, 3328, 32)])
def test_fused_single_row_forms_equal_separate_launches(rt, rows, cols, group):
    banks = [upload_bank(rt, *synth.q4_bank(0x7E551200 + i + rows, r, cols, group)) for i, r in enumerate((rows, rows, rows // 3 + 1))]
    xb = rt.buffer_from(synth.normal_bf16(0x7E551210 + cols, cols))
    kv = rows // 3 + 1
    outs = []
    for bank, r in zip(banks + [banks[2]], (rows, rows, kv, kv)):
        y = seeded_f32(rt, r)
        nn.gemv_q4_mlx_simd(rt, bank, xb, y, nn.QuantShape(r, cols, group))
        outs.append(y)
    got = [seeded_f32(rt, r, 8) for r in (rows, kv, kv)]
    rt.take_dispatch_count()
    nn.gemv_q4_mlx_qkv(rt, banks[0], banks[2], banks[2], xb, nn.QkvOutputs(*got), rows, kv, cols, group)
    mid = seeded_f32(rt, rows, 8)
    nn.gemv_q4_mlx_gate_up_silu(rt, banks[0], banks[1], xb, mid, nn.QuantShape(rows, cols, group), False)
    assert rt.take_dispatch_count() == 2
    for buf, r, want in zip(got, (rows, kv, kv), (outs[0], outs[2], outs[3])):
        v = buf.read(np.float32, r + 8)
        assert np.array_equal(v[:r].view(np.uint32), want.read(np.uint32, r)) and np.all(v[r:] == SENTINEL_F32)
    want = seeded_f32(rt, rows)
    nn.swiglu(rt, outs[0], outs[1], want, rows, False)
    v = mid.read(np.float32, rows + 8)
    assert np.array_equal(v[:rows].view(np.uint32), want.read(np.uint32, rows)) and np.all(v[rows:] == SENTINEL_F32)


@pytest.mark.parametrize("rows,cols,group", [(40, 1024, 64), (40, 2048, 32), (40, 4096, 128), (40, 2560, 64), (17, 3840, 32), (33, 9216, 64),
                                             (16, 17408, 64), (20, 12800, 128)])
def test_a_batch_row_equals_the_vector_alone(rt, rows, cols, group):
    """Bit for bit at 1024, 2048 and 4096 columns (the single-row kernel sums in the same order) and where one row runs on
    the batch kernel itself."""
    bank, shape = upload_bank(rt, *synth.q4_bank(0x7E551700 + cols, rows, cols, group)), nn.QuantShape(rows, cols, group)
    x = synth.normal_bf16(0x7E551710 + cols, 8 * cols)
    y8, y1 = seeded_f32(rt, 8 * rows), seeded_f32(rt, rows)
    nn.gemm_q4_mlx(rt, bank, rt.buffer_from(x), y8, shape, 8)
    got = y8.read(np.uint32, 8 * rows).reshape(8, rows)
    for i in (0, 5, 7):
        nn.gemv_q4_mlx_simd(rt, bank, rt.buffer_from(x[i * cols:(i + 1) * cols].copy()), y1, shape)
        assert np.array_equal(y1.read(np.uint32, rows), got[i])
