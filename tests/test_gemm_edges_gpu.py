"""The prefill GEMM at the edges of its tiles: W rows around a CTA's 128 and a pair's 256, tokens around the multiples of 32 a tile is
made of, K of one block and of block counts that splits divide unevenly; and, with the plan of every shape asserted, its states: pairs that
run several tiles, full accumulators, both accumulators in one tile, whole tiles beside split ones.

The reference is the fp64 product of the operands as rounded to the 16-bit type; the fp32 accumulation may differ from it by
(cols + 4) * 2^-24 * sum|h(W) h(x)| (the reference's bound for its own GEMM, tests/unit/vulkan/test_vk_head.cpp:1005-1013)."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

from halo_b200 import backend as hb
from halo_b200 import capi, synth

pytestmark = pytest.mark.gpu
GUARD = 12  # floats behind every y row that must stay as they were


@pytest.fixture(scope="module")
def be():
    return hb.CudaBackend(0)


def rounded(a: np.ndarray, bf16: bool) -> np.ndarray:
    if not bf16:
        return a.astype(np.float16).astype(np.float64)
    u = np.ascontiguousarray(a, np.float32).view(np.uint32).astype(np.uint64)
    u = (u + 0x7FFF + ((u >> 16) & 1)) >> 16 << 16
    return u.astype(np.uint32).view(np.float32).astype(np.float64)


@pytest.mark.parametrize("t", (synth.Q4_K, synth.Q6_K, synth.Q8_0, synth.Q4_0))
@pytest.mark.parametrize("bf16", (False, True))
@pytest.mark.parametrize("m,n,k", [(1, 1, 256), (33, 129, 512), (64, 128, 2816), (97, 257, 4352), (255, 40, 512), (257, 513, 768), (513, 384, 1024), (700, 2000, 512)])
def test_gemm_tile_edges(be, checker, t, bf16, m, n, k):
    st = be.create_stream()
    w, x = synth.quant_weights(t, n, k, 80 + m, 1), synth.activations(m, k, 80 + m, 2)
    wb = raw = be.import_host_readonly(np.ascontiguousarray(w).view(np.uint8).reshape(-1))
    variant = capi.GEMM_TCGEN05_BF16 if bf16 else capi.GEMM_TCGEN05_F16
    if t != synth.Q4_K:
        wb, variant = be.repack(st, t, hb.TensorRef.of(raw), n, k), capi.GEMM_TCGEN05_BF16_R if bf16 else capi.GEMM_TCGEN05_F16_R
    xb, yb, stride = be.import_host_readonly(x), be.allocate(m * (n + GUARD) * 4), (n + GUARD) * 4
    got = []
    for _ in range(2):  # a second call finds the counters and partial sums as the first one left them
        be.upload(st, hb.TensorRef.of(yb), np.full(m * (n + GUARD), -77.0, np.float32))
        be.gemv(st, hb.GemvArgs(t, hb.TensorRef.of(wb), hb.TensorRef.of(xb), hb.TensorRef(yb, 0, 0, stride), n, k, m, variant, allow_gemm=True))
        y = np.empty((m, n + GUARD), np.float32)
        be.download(st, hb.TensorRef.of(yb), y)
        st.wait()
        got.append(y)
    assert np.array_equal(got[0], got[1])
    assert np.all(got[0][:, n:] == -77.0)
    hw, hx = rounded(checker.dequantize(t, w, n * k).reshape(n, k), bf16), rounded(x, bf16)
    err = np.abs(got[0][:, :n].astype(np.float64) - hx @ hw.T)
    assert np.all(err <= (k + 4) * 2.0**-24 * (np.abs(hx) @ np.abs(hw).T))


def test_gemm_captured_on_a_stream_that_never_ran_splits(be, checker):
    # 2560 x 2048 at 77 tokens splits K; captured on a stream without scratch for the splits' sums it has the eager call's plan and bits
    import torch
    t, n, k, m = synth.Q4_K, 2560, 2048, 77
    assert plan_of(be, t, n, k, m).splits > 1
    w, x = synth.quant_weights(t, n, k, 85, 1), synth.activations(m, k, 85, 2)
    wb, xb = be.import_host_readonly(np.ascontiguousarray(w).view(np.uint8).reshape(-1)), be.import_host_readonly(x)
    yb = be.allocate(m * n * 4)

    def call(st, cols=k, no_scratch=False):
        a = hb.GemvArgs(t, hb.TensorRef.of(wb), hb.TensorRef.of(xb), hb.TensorRef.of(yb), n, cols, m, capi.GEMM_TCGEN05_F16, allow_gemm=True, no_scratch=no_scratch)
        before = be.scratch_bytes()
        be.gemv(st, a)
        return be.scratch_bytes() - before

    def result(st):
        y = np.empty((m, n), np.float32)
        be.download(st, hb.TensorRef.of(yb), y)
        st.wait()
        return y

    eager, captured = be.create_stream(), be.create_stream()
    call(eager)
    want = result(eager)
    # the captured stream has its 16-bit copy of x from a call of one block of K, which is never split
    call(captured, cols=256)
    captured.wait()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=torch.cuda.ExternalStream(captured.handle)):
        assert call(captured) > 0
    be.upload(captured, hb.TensorRef.of(yb), np.full(m * n, -77.0, np.float32))
    captured.wait()
    graph.replay()
    torch.cuda.synchronize()
    assert np.array_equal(result(captured), want)
    # and the plan without splits, which needs none of that scratch
    assert call(captured, no_scratch=True) == 0
    hw, hx = rounded(checker.dequantize(t, w, n * k).reshape(n, k), False), rounded(x, False)
    assert np.all(np.abs(result(captured) - want) <= 2 * (k + 4) * 2.0**-24 * (np.abs(hx) @ np.abs(hw).T))


def plan_of(be, t, n, k, m):
    import torch
    p = capi.GemmPlan()
    assert be.lib.halo_cuda_gemm_plan(t, n, k, m, torch.cuda.get_device_properties(0).multi_processor_count, 0, ctypes.byref(p)) == 0, capi.last_error()
    return p


def check_tiled_rows(be, checker, t, n, k, m, bf16=False):
    """W as copies of 640 rows one below the other: every row of the product against the rounded operands at the price of 640."""
    st = be.create_stream()
    block = synth.quant_weights(t, 640, k, 90 + m, 1)
    rows = np.ascontiguousarray(block).view(np.uint8).reshape(640, -1)
    w = np.ascontiguousarray(np.tile(rows, (-(-n // 640), 1))[:n])
    x = synth.activations(m, k, 90 + m, 2)
    wb, variant = be.import_host_readonly(w.reshape(-1)), capi.GEMM_TCGEN05_BF16 if bf16 else capi.GEMM_TCGEN05_F16
    if t != synth.Q4_K:
        wb, variant = be.repack(st, t, hb.TensorRef.of(wb), n, k), capi.GEMM_TCGEN05_BF16_R if bf16 else capi.GEMM_TCGEN05_F16_R
    xb, yb = be.import_host_readonly(x), be.allocate(m * n * 4)
    be.upload(st, hb.TensorRef.of(yb), np.full(m * n, np.nan, np.float32))
    be.gemv(st, hb.GemvArgs(t, hb.TensorRef.of(wb), hb.TensorRef.of(xb), hb.TensorRef.of(yb), n, k, m, variant, allow_gemm=True))
    y = np.empty((m, n), np.float32)
    be.download(st, hb.TensorRef.of(yb), y)
    st.wait()
    for b in (wb, xb, yb):
        b.free()
    hw, hx = rounded(checker.dequantize(t, block, 640 * k).reshape(640, k), bf16), rounded(x, bf16)
    ref, bound = hx @ hw.T, (k + 4) * 2.0**-24 * (np.abs(hx) @ np.abs(hw).T)
    for first in range(0, n, 640):
        r = min(640, n - first)
        assert np.all(np.abs(y[:, first:first + r] - ref[:, :r]) <= bound[:, :r]), f"rows from {first}"


# (rows, K, tokens) by state and format; rows and tokens ragged
STATES = {
    "several tiles a pair": {synth.Q4_K: (580, 256, 1713), synth.Q6_K: (551, 256, 1640), synth.Q8_0: (606, 256, 1629), synth.Q4_0: (572, 256, 1594)},
    "a full accumulator": {synth.Q4_K: (19693, 1024, 232), synth.Q6_K: (19837, 1024, 228), synth.Q8_0: (26130, 1024, 226), synth.Q4_0: (19258, 1280, 228)},
    "whole and split": {synth.Q4_K: (20027, 1024, 33), synth.Q6_K: (19170, 768, 33), synth.Q8_0: (20963, 1024, 33), synth.Q4_0: (20083, 1024, 44)},
    "both accumulators": {synth.Q4_K: (27312, 4352, 582), synth.Q6_K: (27448, 3328, 578), synth.Q8_0: (28303, 4096, 588), synth.Q4_0: (28131, 4864, 577)},
    "both accumulators, whole and split": {synth.Q4_K: (22057, 4096, 262), synth.Q6_K: (19345, 3584, 265), synth.Q8_0: (19779, 4608, 260), synth.Q4_0: (19109, 5888, 266)},
}


@pytest.mark.parametrize("bf16", (False, True))
@pytest.mark.parametrize("t", (synth.Q4_K, synth.Q6_K, synth.Q8_0, synth.Q4_0))
@pytest.mark.parametrize("state", STATES)
def test_gemm_states(be, checker, state, t, bf16):
    n, k, m = STATES[state][t]
    p = plan_of(be, t, n, k, m)
    assert p.units > p.pairs, "no pair runs a second unit"
    assert p.accumulators == (2 if "both" in state else 1)
    assert ((p.whole > 0 and p.splits > 1) if "split" in state else p.splits == 1)
    if state == "a full accumulator":
        assert p.tile_tokens == 256
    check_tiled_rows(be, checker, t, n, k, m, bf16)


# Shapes whose cheapest tile takes both accumulators (320 to 448 tokens), with and without K splits, and ragged in rows and tokens
@pytest.mark.parametrize("t,n,k,m", [(synth.Q4_K, 3200, 13824, 259), (synth.Q6_K, 17895, 3328, 280), (synth.Q4_K, 16034, 3584, 282), (synth.Q6_K, 14222, 3840, 346),
                                     (synth.Q4_0, 9461, 11008, 770)])
def test_gemm_wide_tiles(be, checker, t, n, k, m):
    assert plan_of(be, t, n, k, m).accumulators == 2
    check_tiled_rows(be, checker, t, n, k, m)


@pytest.mark.parametrize("t", (synth.Q4_K, synth.Q8_0))
def test_gemm_of_one_w_row_has_no_use_for_its_pitch(be, checker, t):
    # any multiple of 16 is a valid pitch of a matrix of one row, also one the copy engine could not step by
    k, m = 512, 65
    w, x = synth.quant_weights(t, 1, k, 97, 1), synth.activations(m, k, 97, 2)
    st = be.create_stream()
    wb, variant = be.import_host_readonly(np.ascontiguousarray(w).view(np.uint8).reshape(-1)), capi.GEMM_TCGEN05_F16
    if t != synth.Q4_K:
        wb, variant = be.repack(st, t, hb.TensorRef.of(wb), 1, k), capi.GEMM_TCGEN05_F16_R
    xb, yb = be.import_host_readonly(x), be.allocate(m * 4)
    got = []
    for pitch in (0, 16, 1 << 41):
        g = capi.Gemv(wtype=t, variant_id=variant, w=wb.ptr, w_stride=pitch, x=xb.ptr, y=yb.ptr, rows=1, cols=k, n_vec=m, flags=capi.FLAG_ALLOW_GEMM)
        assert be.lib.halo_cuda_gemv(be.ctx, ctypes.byref(g), st.handle) == 0, capi.last_error()
        y = np.empty(m, np.float32)
        be.download(st, hb.TensorRef.of(yb), y)
        st.wait()
        got.append(y)
    assert np.array_equal(got[0], got[1]) and np.array_equal(got[0], got[2]) and np.any(got[0] != 0)
