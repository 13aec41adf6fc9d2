"""Row kernels at the sizes where they can go wrong: the dequantising gather and the repack at block edges, remainders of their tiles,
strided operands and odd addresses (where they fall back to a byte-wise form).  Both are exact: the outputs are compared bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import bits
from halo_b200 import backend as hb
from halo_b200 import capi, synth
from test_repacked_gpu import unrepack

pytestmark = pytest.mark.gpu
REPACKABLE = (synth.Q6_K, synth.Q8_0, synth.Q4_0)


@pytest.fixture(scope="module")
def be():
    return hb.CudaBackend(0)


def strided(w: np.ndarray, stride: int, offset: int) -> np.ndarray:
    buf = np.full(offset + w.shape[0] * stride, 0xA5, np.uint8)
    for r in range(w.shape[0]):
        buf[offset + r * stride:offset + r * stride + w.shape[1]] = w[r]
    return buf


# blocks per row: one, less than a warp's worth, a whole block of threads and one more
@pytest.mark.parametrize("blocks", (1, 3, 16, 129))
@pytest.mark.parametrize("pad,offset,out_pad", ((0, 0, 0), (32, 16, 4), (2, 2, 0), (1, 3, 1)))
@pytest.mark.parametrize("t", (synth.Q4_K, *REPACKABLE))
def test_get_rows_edges(be, checker, t, blocks, pad, offset, out_pad):
    cols, rows = blocks * synth.BLOCK_ELEMS[t], 7
    w = synth.random_blocks_finite(t, rows, cols, 41, t)
    ids = np.array([6, 0, 3, 3], np.int32)
    st = be.create_stream()
    tb, ib = be.import_host_readonly(strided(w, w.shape[1] + pad, offset)), be.import_host_readonly(ids)
    ostride = (cols + out_pad) * 4
    ob, sb = be.allocate(len(ids) * ostride), be.allocate(4)
    be.upload(st, hb.TensorRef.of(ob), np.full(len(ids) * ostride // 4, -77.0, np.float32))
    be.get_rows(st, hb.GetRowsArgs(t, hb.TensorRef(tb, offset, 0, w.shape[1] + pad), hb.TensorRef.of(ib), hb.TensorRef(ob, 0, 0, ostride), rows, cols, len(ids)), status=sb)
    got, status = np.empty((len(ids), cols + out_pad), np.float32), np.empty(1, np.uint32)
    be.download(st, hb.TensorRef.of(ob), got)
    be.download(st, hb.TensorRef.of(sb), status)
    st.wait()
    assert status[0] == 0
    for i, r in enumerate(ids):
        assert np.array_equal(bits(got[i, :cols]), bits(checker.dequantize(t, w[r], cols)))
    assert np.all(got[:, cols:] == -77.0)


# 256-weight groups per row: one, a tile's remainder, exactly a tile of one of the formats, more than one tile
@pytest.mark.parametrize("groups", (1, 5, 32, 67))
@pytest.mark.parametrize("pad,offset", ((0, 0), (0, 2), (6, 14), (3, 1)))
@pytest.mark.parametrize("t", REPACKABLE)
def test_repack_edges(be, t, groups, pad, offset):
    rows, cols = 5, 256 * groups
    w = synth.random_blocks_finite(t, rows, cols, 43, t)
    st = be.create_stream()
    src = be.import_host_readonly(strided(w, w.shape[1] + pad, offset))
    prb = be.repacked_row_bytes(t, cols)
    for dpad in (0, 48):
        dst = be.allocate(rows * (prb + dpad))
        be.upload(st, hb.TensorRef.of(dst), np.full(rows * (prb + dpad), 0x5A, np.uint8))
        rc = be.lib.halo_cuda_repack_rows(be.ctx, t, src.ptr + offset, w.shape[1] + pad, dst.ptr, prb + dpad, rows, cols, st.handle)
        assert rc == 0, capi.last_error()
        out = np.empty((rows, prb + dpad), np.uint8)
        be.download(st, hb.TensorRef.of(dst), out)
        st.wait()
        assert np.array_equal(unrepack(t, np.ascontiguousarray(out[:, :prb]), rows, cols), w)
        if t == synth.Q6_K:
            assert not np.any(out[:, :prb].reshape(rows, groups, 224)[..., 18:32])
        assert np.all(out[:, prb:] == 0x5A)


@pytest.mark.parametrize("cols", (4864, 5120))  # a last pair of items that is half there, and whole ones
@pytest.mark.parametrize("t", (synth.Q4_K, *REPACKABLE))
def test_get_rows_many_ids(be, checker, t, cols):
    rows, n = 5, 400  # enough items for the form with two a thread
    w = synth.random_blocks_finite(t, rows, cols, 45, t)
    ids = (np.arange(n, dtype=np.int32) * 3) % rows
    st = be.create_stream()
    tb, ib, ob, sb = be.import_host_readonly(w), be.import_host_readonly(ids), be.allocate(n * cols * 4), be.allocate(4)
    be.get_rows(st, hb.GetRowsArgs(t, hb.TensorRef.of(tb), hb.TensorRef.of(ib), hb.TensorRef.of(ob), rows, cols, n), status=sb)
    got, status = np.empty((n, cols), np.float32), np.empty(1, np.uint32)
    be.download(st, hb.TensorRef.of(ob), got)
    be.download(st, hb.TensorRef.of(sb), status)
    st.wait()
    assert status[0] == 0
    want = np.stack([checker.dequantize(t, w[r], cols) for r in range(rows)])
    assert np.array_equal(bits(got), bits(want[ids]))
