"""CUDA graphs of matmul calls on a stream that goes on being used: a captured kernel holds the address of its stream's scratch, so whatever
eager calls make that scratch grow afterwards, a replay has to give the bits of the eager call."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import bits
from halo_b200 import backend as hb
from halo_b200 import capi, synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def be():
    return hb.CudaBackend(0)


class Op:
    """One projection with operands of its own."""

    def __init__(self, be, st, t, n, k, m, seed, allow_gemm=False):
        self.be, self.shape = be, (m, n)
        w, x = synth.quant_weights(t, n, k, seed, 1), synth.activations(m, k, seed, 2)
        wb, variant = be.import_host_readonly(np.ascontiguousarray(w).view(np.uint8).reshape(-1)), 0
        if t != synth.Q4_K:
            wb, variant = be.repack(st, t, hb.TensorRef.of(wb), n, k), be.repacked_variant(t, k)
        self.held = wb, be.import_host_readonly(x), be.allocate(m * n * 4)
        self.args = hb.GemvArgs(t, *(hb.TensorRef.of(b) for b in self.held), n, k, m, variant, allow_gemm=allow_gemm)

    def call(self, st):
        self.be.gemv(st, self.args)

    def clear(self, st):
        self.be.upload(st, self.args.y, np.full(self.shape, -77.0, np.float32))
        st.wait()

    def result(self, st):
        y = np.empty(self.shape, np.float32)
        self.be.download(st, self.args.y, y)
        st.wait()
        return y


def capture(ops, st):
    import torch
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=torch.cuda.ExternalStream(st.handle)):
        for op in ops:
            op.call(st)
    return graph


def test_replay_after_eager_calls_grew_the_scratch(be):
    import torch
    st = be.create_stream()
    # row blocks cut over CTAs (counters and partial sums), a batch (staged x), a short prompt (16-bit x, K splits)
    ops = [Op(be, st, synth.Q8_0, 2048, 5120, 1, 61), Op(be, st, synth.Q4_K, 640, 2560, 7, 62), Op(be, st, synth.Q4_K, 2560, 2048, 77, 63, allow_gemm=True)]
    larger = [Op(be, st, synth.Q8_0, 5120, 17408, 16, 64), Op(be, st, synth.Q6_K, 2560, 5632, 300, 65, allow_gemm=True)]
    want = []
    for op in ops:
        op.call(st)
        want.append(op.result(st))
    graph = capture(ops, st)
    for _ in range(2):
        before = be.scratch_bytes()
        for op in larger:
            op.call(st)
        st.wait()
        assert be.scratch_bytes() >= before
        for op in ops:
            op.clear(st)
        graph.replay()
        torch.cuda.synchronize()
        for op, y in zip(ops, want):
            assert np.array_equal(bits(op.result(st)), bits(y))
    del graph
