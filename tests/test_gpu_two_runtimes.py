"""Two runtimes on one device: what one of them launches does not take away what the other may launch. A kernel's limit of
dynamic shared memory belongs to the device's context, so a runtime that asked for less than another would lower it."""
import numpy as np
import pytest

from gpu_util import rt, seeded_f32, upload_bank  # noqa: F401
from tessl_b200 import nn, synth

pytestmark = pytest.mark.gpu


def _project(r, bank, xb, rows, cols, group, m):
    y = seeded_f32(r, m * rows)
    if m == 1:
        nn.gemv_q4_mlx_simd(r, bank, xb, y, nn.QuantShape(rows, cols, group))
    else:
        nn.gemm_q4_mlx(r, bank, xb, y, nn.QuantShape(rows, cols, group), m)
    return y.read(np.uint32, m * rows)


# (m, group, the first runtime's columns, the second's): one kernel each, the second asking for less shared memory
@pytest.mark.parametrize("m,group,wide,narrow", [(8, 64, 8192, 4096), (2, 64, 2560, 2304), (1, 32, 896, 512), (1, 64, 2560, 2304)])
def test_widths_alternate_between_two_runtimes(rt, m, group, wide, narrow):
    rows = 40
    with nn.Runtime() as other:
        sides = []
        for r, cols in ((rt, wide), (other, narrow)):
            bank = upload_bank(r, *synth.q4_bank(0x7E551300 + cols, rows, cols, group))
            xb = r.buffer_from(synth.normal_bf16(0x7E551310 + cols, m * cols))
            sides.append((r, bank, xb, rows, cols, group, m))
        first = [_project(*s) for s in sides]
        for _ in range(2):
            for s, want in zip(sides, first):
                assert np.array_equal(_project(*s), want)
        assert not rt.is_poisoned() and not other.is_poisoned()
