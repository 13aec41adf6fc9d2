"""gemv_warp_f32 over raw Q8_0 / Q4_0 / Q6_K rows at the edges of its shared-memory form: K around a lane's 64 weights and a slot's 2048,
rows around a warp's passes, every batch form, rows at any even address, the shortest K each format takes and the longest below it, and K on
both sides of every step of the launch: four x rows beside a large and a small ring, two, one, and what no longer fits (the form without
shared memory).

Bounds: against the fp64 product of the exact weights, each product, group sum, group term and tree level rounds once, at most
(K / 32 + 32 + 8) roundings of 2^-24 on sum |w x|."""
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


def run(be, st, t, wb, offset, stride, x, n, k):
    m = x.shape[0]
    xb, yb = be.import_host_readonly(x), be.allocate((m * n + 8) * 4)
    be.upload(st, hb.TensorRef.of(yb), np.full(m * n + 8, -77.0, np.float32))
    be.gemv(st, hb.GemvArgs(t, hb.TensorRef(wb, offset, 0, stride), hb.TensorRef.of(xb), hb.TensorRef(yb, 16, 0, 0), n, k, m, capi.GEMV_WARP_F32))
    y = np.empty(m * n + 8, np.float32)
    be.download(st, hb.TensorRef.of(yb), y)
    st.wait()
    assert np.all(y[:4] == -77.0) and np.all(y[-4:] == -77.0)
    return y[4:-4].reshape(m, n)


@pytest.mark.parametrize("t", (synth.Q8_0, synth.Q4_0, synth.Q6_K))
@pytest.mark.parametrize("n,k", [(1, 32), (7, 96), (37, 2048), (300, 2080), (95, 5120), (1185, 288), (70, 352), (70, 384), (41, 608), (41, 640), (50, 1024), (50, 1280), (33, 8192), (24, 17408), (9, 28672), (3, 65536)])
@pytest.mark.parametrize("pad,offset", ((0, 0), (6, 2), (2, 14)))
def test_raw_rows_edges(be, checker, t, n, k, pad, offset):
    k = -(-k // synth.BLOCK_ELEMS[t]) * synth.BLOCK_ELEMS[t]
    w, x = synth.quant_weights(t, n, k, 90 + n, 1), synth.activations(11, k, 90 + n, 2)
    rows = np.ascontiguousarray(w).view(np.uint8).reshape(n, -1)
    stride = rows.shape[1] + pad
    buf = np.full(offset + (n - 1) * stride + rows.shape[1], 0xFF, np.uint8)  # all-ones padding: a scale read from it is a NaN
    for r in range(n):
        buf[offset + r * stride:offset + r * stride + rows.shape[1]] = rows[r]
    st = be.create_stream()
    wb = be.import_host_readonly(buf)
    y = run(be, st, t, wb, offset, stride, x, n, k)
    wf = checker.dequantize(t, w, n * k).reshape(n, k).astype(np.float64)
    err = np.abs(y - x.astype(np.float64) @ wf.T)
    assert np.all(err <= (k / 32 + 40) * 2.0**-24 * (np.abs(x).astype(np.float64) @ np.abs(wf).T))
    for m in (1, 2, 3, 5):  # one, two and four x rows a block, whole and cut: the same bits
        assert np.array_equal(bits(run(be, st, t, wb, offset, stride, x[:m], n, k)), bits(y[:m]))


# the largest K of four x rows beside eight warps' rings of eight and of four slots, of two beside four, of one beside sixteen and eight warps'
LIMITS = {synth.Q8_0: (5632, 9728, 19968, 22528, 40448), synth.Q4_0: (9728, 11776, 24064, 38912, 48640), synth.Q6_K: (7680, 10752, 22016, 30720, 44032)}


@pytest.mark.parametrize("t", sorted(LIMITS))
@pytest.mark.parametrize("step", range(5))
@pytest.mark.parametrize("beyond", (False, True))
def test_raw_rows_on_both_sides_of_a_step(be, checker, t, step, beyond):
    n, k = 21, LIMITS[t][step] + (synth.BLOCK_ELEMS[t] if beyond else 0)
    w, x = synth.quant_weights(t, n, k, 95 + step, 1), synth.activations(5, k, 95 + step, 2)
    st = be.create_stream()
    wb = be.import_host_readonly(np.ascontiguousarray(w).view(np.uint8).reshape(-1))
    y = run(be, st, t, wb, 0, 0, x, n, k)
    wf = checker.dequantize(t, w, n * k).reshape(n, k).astype(np.float64)
    err = np.abs(y - x.astype(np.float64) @ wf.T)
    assert np.all(err <= (k / 32 + 40) * 2.0**-24 * (np.abs(x).astype(np.float64) @ np.abs(wf).T))
    for m in (1, 2, 3):
        assert np.array_equal(bits(run(be, st, t, wb, 0, 0, x[:m], n, k)), bits(y[:m]))
