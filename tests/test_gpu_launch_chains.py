"""Chains of launches over shared buffers, each of which may start before the one in front of it ends: the embedding gather, the
norm, projections of every kind, the activation. Several steps with tokens of their own rewrite the same intermediate buffers;
every step gives the bits that it gives when each call is waited for, captured in a CUDA graph and call by call."""
import numpy as np
import pytest

from gpu_util import rt, upload_bank  # noqa: F401
from tessl_b200 import nn, synth

pytestmark = pytest.mark.gpu

VOCAB, STEPS = 97, 5


# rows of tokens, hidden width, MLP width, group, the prefill entry without allocation
@pytest.mark.parametrize("m,hidden,inter,group,noalloc", [(1, 2560, 1024, 64, False), (1, 8192, 512, 64, False), (5, 768, 9216, 64, False),
                                                          (40, 512, 1408, 32, False), (40, 512, 1408, 32, True),
                                                          (300, 1024, 640, 128, False), (300, 1024, 640, 128, True)])
def test_every_step_of_a_chain_sees_its_own_inputs(rt, m, hidden, inter, group, noalloc):
    import torch

    table = upload_bank(rt, *synth.q4_bank(0x7E551500, VOCAB, hidden, group))
    gate, up = (upload_bank(rt, *synth.q4_bank(0x7E551501 + i, inter, hidden, group)) for i in range(2))
    down = upload_bank(rt, *synth.q4_bank(0x7E551505, hidden, inter, group))
    w = rt.buffer_from(synth.bf16_bits_to_f32(synth.normal_bf16(0x7E551506, hidden)))
    ids = [rt.buffer_from(((np.arange(m) * 13 + 29 * s) % VOCAB).astype(np.uint32)) for s in range(STEPS)]
    resid, x = rt.alloc_buffer(m * hidden * 4), rt.alloc_buffer(m * hidden * 2)
    g, u, mid = rt.alloc_buffer(m * inter * 4), rt.alloc_buffer(m * inter * 4), rt.alloc_buffer(m * inter * 2)
    ys = [rt.alloc_buffer(m * hidden * 4) for _ in range(STEPS)]
    s_up, s_down = nn.QuantShape(inter, hidden, group), nn.QuantShape(hidden, inter, group)

    def project(bank, a, y, shape):
        if m == 1:
            nn.gemv_q4_mlx_simd(rt, bank, a, y, shape)
        elif m <= nn.GEMM_Q4_MLX_MAX_M:
            nn.gemm_q4_mlx(rt, bank, a, y, shape, m)
        elif noalloc:
            nn.gemm_q4_mlx_tensorops_noalloc(rt, bank, a, y, shape, m)
        else:
            nn.gemm_q4_mlx_tensorops(rt, bank, a, y, shape, m)

    def chain():
        for s in range(STEPS):
            nn.embed_lookup_q4_mlx(rt, table, ids[s], resid, VOCAB, hidden, group, m)
            nn.qwen35_rms_norm(rt, resid, w, x, True, m, hidden, 1e-6)
            if m == 1 and s % 2:
                nn.gemv_q4_mlx_gate_up_silu(rt, gate, up, x, mid, s_up, True)
            else:
                project(gate, x, g, s_up)
                project(up, x, u, s_up)
                nn.swiglu(rt, g, u, mid, m * inter, True)
            project(down, mid, ys[s], s_down)

    chain()
    want = [y.read(np.uint32, m * hidden) for y in ys]
    assert len({v.tobytes() for v in want}) == STEPS, "the steps' inputs differ"

    def check(how):
        rt.synchronize()
        for s in range(STEPS):
            assert np.array_equal(ys[s].read(np.uint32, m * hidden), want[s]), f"{how}: step {s}"
            ys[s].write(np.zeros(m * hidden, np.uint32))

    st = torch.cuda.ExternalStream(rt.stream)
    rt.set_encode_only(True)
    try:
        for y in ys:
            y.write(np.zeros(m * hidden, np.uint32))
        chain()
        check("call by call")
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=st):
            chain()
        with torch.cuda.stream(st):
            for _ in range(3):
                graph.replay()
        check("graph")
    finally:
        rt.set_encode_only(False)
