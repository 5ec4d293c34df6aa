"""`gemv_q8` over the streamed kernel's plans: one to eight warps per row, one set of teams or several, rows of more than 4096 columns, a last
stage of one to three rows whose tables are no whole number of 16 bytes, the shapes either side of its domain, and the same bits of a row
on either side."""
import numpy as np
import pytest

from gpu_util import SENTINEL_F32, rt, seeded_f32  # noqa: F401
from oracle import api
from tessl_b200 import nn, synth

pytestmark = pytest.mark.gpu


def _inputs(rows, cols, group):
    d = synth.splitmix_draws(0x7E553400 + rows + cols, rows * cols + 2 * rows * (cols // group) + cols)
    n, g = rows * cols, rows * (cols // group)
    q = (d[:n] >> np.uint64(17)).astype(np.uint8).view(np.int8)
    scales = np.abs(synth.unit_from_draws(d[n:n + g])) * np.float32(0.005) + np.float32(1e-4)
    zeros = synth.unit_from_draws(d[n + g:n + 2 * g]) * np.float32(8.0)
    return q, scales.astype(np.float32), zeros.astype(np.float32), synth.unit_from_draws(d[n + 2 * g:])


def _check(rt, q, scales, zeros, x, rows, cols, group, sb, zb):
    y = seeded_f32(rt, rows, 8)
    nn.gemv_q8(rt, rt.buffer_from(q), sb, zb, rt.buffer_from(x), y, rows, cols, group)
    got = y.read(np.float32, rows + 8)
    assert np.all(got[rows:] == SENTINEL_F32)
    want = api.q8_gemv_f64(q, scales, zeros, x, rows, cols, group)
    # gamma of cols + 3 groups f32 operations on the sum of the terms' magnitudes
    w = np.abs(scales.reshape(rows, -1, 1) * (np.abs(q.astype(np.float64)).reshape(rows, -1, group) + np.abs(zeros.reshape(rows, -1, 1))))
    mag = (w.reshape(rows, cols) * np.abs(x.astype(np.float64))).sum(axis=1)
    n = (cols + 3 * (cols // group)) * 2.0 ** -24
    assert np.all(np.abs(got[:rows] - want) <= n / (1 - n) * mag)
    return got[:rows]


@pytest.mark.parametrize("rows,cols,group", [(2049, 512, 32), (2051, 512, 16), (1366, 768, 48), (1025, 1024, 1024), (701, 1536, 64),
                                             (4097, 1152, 32), (515, 2048, 2048), (411, 2560, 2560), (343, 3072, 64), (299, 3584, 64),
                                             (258, 4096, 64), (4096, 4096, 4096), (227, 4624, 16), (130, 8192, 16), (131, 8192, 8192),
                                             (130, 8208, 16), (255, 4096, 64), (20000, 512, 64)])
def test_streamed_plans(rt, rows, cols, group):
    q, scales, zeros, x = _inputs(rows, cols, group)
    _check(rt, q, scales, zeros, x, rows, cols, group, rt.buffer_from(scales), rt.buffer_from(zeros))


def _bits(rt, q, scales, zeros, x, rows, cols, group, offset=0):
    tables = []
    for t in (scales, zeros):
        b = rt.alloc_buffer(t.nbytes + offset)
        b.write(t, offset)
        tables.append(b.view(offset, t.nbytes))
    return _check(rt, q, scales, zeros, x, rows, cols, group, *tables).view(np.uint32)


@pytest.mark.parametrize("rows,cols,group", [(66000, 16, 16), (6000, 192, 64), (2731, 384, 128), (1400, 768, 32), (1200, 1280, 64),
                                             (1000, 1536, 64), (600, 2176, 64), (400, 3072, 64), (300, 4096, 64), (600, 4608, 64),
                                             (500, 5120, 64), (400, 6144, 64), (400, 6672, 16), (300, 8192, 64), (300, 8208, 16)])
def test_a_row_has_the_same_bits_in_every_bank(rt, rows, cols, group):
    """The whole bank through the ring, its tables at an address that is no multiple of 16, and slices below the ring's least size."""
    q, scales, zeros, x = _inputs(rows, cols, group)
    whole = _bits(rt, q, scales, zeros, x, rows, cols, group)
    assert np.array_equal(whole, _bits(rt, q, scales, zeros, x, rows, cols, group, offset=4))
    gpr = cols // group
    for first, n in ((0, 5), (rows - 7, 7), (rows // 2, 64)):
        part = _bits(rt, q[first * cols:(first + n) * cols], scales[first * gpr:(first + n) * gpr], zeros[first * gpr:(first + n) * gpr], x,
                     n, cols, group)
        assert np.array_equal(whole[first:first + n], part)
