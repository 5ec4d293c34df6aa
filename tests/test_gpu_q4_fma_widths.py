"""The FMA-pipe forms of the single-row and batch products at the widths and alignments that the tensor-core kernels refuse:
rows over 4096 columns that are no whole number of chunks, groups of 256, more columns than windows, scale/bias pairs that
start on a 4-byte boundary only."""
import numpy as np
import pytest

import ref_cases as rc
from gpu_util import SENTINEL_F32, assert_gamma_bound, assert_north_star, rt, seeded_f32, upload_bank  # noqa: F401
from oracle import api
from tessl_b200 import nn, synth

pytestmark = pytest.mark.gpu

# (rows, columns, group, bytes by which the pairs are off a 16-byte boundary)
SHAPES = [(40, 5248, 64, 0), (33, 16512, 64, 0), (24, 6144, 256, 0), (21, 20480, 256, 0), (8, 33024, 64, 0), (40, 9216, 64, 4),
          (17, 17408, 64, 8), (40, 2560, 64, 4), (24, 4096, 64, 4)]


def _bank(rt, packed, sb, off):
    if not off:
        return upload_bank(rt, packed, sb)
    raw = np.zeros(sb.nbytes + 16, np.uint8)
    raw[off:off + sb.nbytes] = sb.reshape(-1).view(np.uint8)
    return nn.Q4MlxBank(rt.buffer_from(packed), rt.buffer_from(raw).view(off, sb.nbytes))


@pytest.mark.parametrize("rows,cols,group,off", SHAPES)
def test_widths_and_alignments_of_the_fma_pipe(rt, rows, cols, group, off):
    flat = []
    for i in range(2):
        packed, sb = synth.q4_bank(0x7E551600 + i + rows + cols, rows, cols, group)
        flat.append((packed.view(np.uint8).reshape(-1), sb.reshape(-1)))
    banks = [_bank(rt, p, s, off) for p, s in flat]
    (packed, sb), shape = flat[0], nn.QuantShape(rows, cols, group)
    for m in (1, 2, 5, 8):
        x = synth.normal_bf16(0x7E551610 + cols, 8 * cols)[: m * cols]
        xb, y = rt.buffer_from(x), seeded_f32(rt, m * rows, 8)

        def call(out, **kw):
            if m == 1:
                nn.gemv_q4_mlx_simd(rt, banks[0], xb, out, shape, **kw)
            else:
                nn.gemm_q4_mlx(rt, banks[0], xb, out, shape, m, **kw)

        call(y)
        got = y.read(np.float32, m * rows + 8)
        assert np.all(got[m * rows:] == SENTINEL_F32), "wrote past y"
        got = got[: m * rows].reshape(m, rows)
        assert_north_star(got, api.q4_dense_gemm(packed, sb, x, m, rows, cols, group), f"m={m}")
        assert_gamma_bound(got, packed, sb, x, m, rows, cols, group, what=f"m={m}")
        resid = rc.rand_f32(m * rows, 0x5400 + rows * m)
        r = rt.buffer_from(resid)
        call(r, resid=r)
        assert np.array_equal(r.read(np.float32, m * rows), got.reshape(-1) + resid)
    xb = rt.buffer_from(synth.normal_bf16(0x7E551611, cols))
    mid, want = seeded_f32(rt, rows, 8), seeded_f32(rt, rows)
    nn.gemv_q4_mlx_gate_up_silu(rt, banks[0], banks[1], xb, mid, shape, False)
    parts = []
    for bank in banks:
        y = seeded_f32(rt, rows)
        nn.gemv_q4_mlx_simd(rt, bank, xb, y, shape)
        parts.append(y)
    nn.swiglu(rt, parts[0], parts[1], want, rows, False)
    v = mid.read(np.float32, rows + 8)
    assert np.array_equal(v[:rows].view(np.uint32), want.read(np.uint32, rows)) and np.all(v[rows:] == SENTINEL_F32)
