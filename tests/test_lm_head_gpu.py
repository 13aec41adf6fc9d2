"""GPU parity of the fused LM head against the reference's outputs (tests/unit/backend/test_cpu_backend.cpp:479-603)."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import bits, golden
from halo_b200 import backend as hb
from halo_b200 import capi, synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def hz():
    from gpu_util import Harness
    return Harness()


@pytest.mark.parametrize("name", ["q8_0", "q4_k"])
def test_lm_head_exact_variant_equals_reference_words(hz, name):
    g = golden("lm_head.npz")
    t, V, E, n, seed = (int(v) for v in g[f"{name}_meta"])
    w = synth.quant_weights(t, V, E, seed, 1)
    x = g[f"{name}_x"]
    res, logits, ids = hz.lm_head(t, w, x, V, E, variant=capi.GEMV_EXACT8)
    assert np.array_equal(res, g[f"{name}_result"])
    assert np.array_equal(bits(logits), bits(g[f"{name}_logits"]))
    assert np.array_equal(ids, g[f"{name}_ids"])
    # argmax only (no logits operand) gives the same words
    res2, _, _ = hz.lm_head(t, w, x, V, E, variant=capi.GEMV_EXACT8, want_logits=False, want_ids=False)
    assert np.array_equal(res2, res)
    res_v, _, ids_v = hz.lm_head(t, w, x, V, E, variant=capi.GEMV_EXACT8, valid_rows=5000, want_logits=False)
    assert np.array_equal(res_v, g[f"{name}_result_valid5000"])
    assert np.array_equal(ids_v, g[f"{name}_ids_valid5000"])
    x2 = x.copy()
    x2[1, 0] = np.nan
    res_n, _, ids_n = hz.lm_head(t, w, x2, V, E, variant=capi.GEMV_EXACT8, want_logits=False)
    assert np.array_equal(res_n, g[f"{name}_result_nanrow1"])
    assert np.array_equal(ids_n, g[f"{name}_ids_nanrow1"])
    dec = hb.decode_argmax(res_n)
    assert dec[1][0] == -1 and np.isnan(dec[1][1]) and dec[0][0] == int(res[0, 0])


def test_lm_head_fast_variant_index_matches_when_gap_exceeds_bound(hz, checker):
    # the argmax index must equal the CPU's whenever the CPU's top-2 gap exceeds twice the error bound
    # (tests/unit/backend/test_hip_backend.cpp:603-653)
    from gpu_util import summation_bound
    t, V, E, n = synth.Q4_0, 20000, 1024, 16
    w = synth.quant_weights(t, V, E, 77, 1)
    x = synth.activations(n, E, 77, 2)
    ref_res, ref_logits, _ = checker.lm_head(t, w, x, V, E)
    res, logits, ids = hz.lm_head(t, w, x, V, E)
    bound = summation_bound(checker.dequantize, t, w, x, V, E, depth=2 * (E // 8 + 8))
    assert np.all(np.abs(logits.astype(np.float64) - ref_logits) <= bound)
    checked = 0
    for i in range(n):
        top2 = np.sort(ref_logits[i])[-2:]
        # the winner is always the argmax of the values this backend itself produced
        assert int(res[i, 0]) == int(np.argmax(logits[i])) and ids[i] == int(res[i, 0])
        assert res[i, 1] == bits(logits[i])[int(res[i, 0])]
        if top2[1] - top2[0] > 2 * bound[i].max():
            assert int(res[i, 0]) == int(ref_res[i, 0])
            checked += 1
    assert checked >= n // 2


def test_lm_head_shard_offsets_merge_to_the_full_answer(hz, checker):
    # a vocabulary split over shards: per-shard winners carry their row offset; merging by (value desc, index asc)
    # gives the single-call answer because that order is total (backends/cpu/matmul.cpp:19-22)
    t, V, E, n = synth.Q8_0, 4096, 512, 4
    w = synth.quant_weights(t, V, E, 78, 1)
    x = synth.activations(n, E, 78, 2)
    full, _, _ = hz.lm_head(t, w, x, V, E, variant=capi.GEMV_EXACT8, want_logits=False)
    parts = [hz.lm_head(t, w[o:o + 1024], x, 1024, E, variant=capi.GEMV_EXACT8, want_logits=False, row_offset=o)[0] for o in range(0, V, 1024)]
    for i in range(n):
        cand = [(-(p[i, 1:2].view(np.float32)[0]), int(p[i, 0])) for p in parts]
        best = min(cand)
        assert best[1] == int(full[i, 0])


# Logits whose rows start on 16-byte boundaries (whole chunks of 8192 are read in 16-byte words) or do not (one by one), and a ragged last chunk
@pytest.mark.parametrize("pad", (0, 1, 2, 3))
@pytest.mark.parametrize("valid", (0, 3, 8192, 8192 + 7, 3 * 8192 + 2))
def test_argmax_over_ties_infinities_and_nan(hz, pad, valid):
    be, st = hz.be, hz.st
    V, E, stride = 3 * 8192 + 4, 32, 3 * 8192 + 4 + pad
    rng = np.random.default_rng(5)
    q = rng.integers(1, 100, V)                       # one code a row, scale 1: logit = code * x[0]
    q[[5000, 8191, 8192, 9001, V - 1]] = 120          # the largest in every chunk, at a chunk's edges, in the ragged one
    q[[2, 8195, 8198]] = 110
    w = np.zeros((V, 34), np.uint8)
    w[:, :2], w[:, 2] = np.frombuffer(np.float16(1.0).tobytes(), np.uint8), q.astype(np.uint8)
    head = np.array([1.0, -1.0, np.inf, -np.inf, np.nan, 0.0], np.float32)
    x = np.zeros((len(head), E), np.float32)
    x[:, 0] = head
    wb, xb = be.import_host_readonly(w.reshape(-1)), be.import_host_readonly(x)
    lb, rb, ib = be.allocate(len(head) * stride * 4), be.allocate(len(head) * 12), be.allocate(len(head) * 4)
    g = hb.GemvArgs(synth.Q8_0, hb.TensorRef.of(wb), hb.TensorRef.of(xb), hb.TensorRef(lb, 0, 0, stride * 4), V, E, len(head), capi.GEMV_EXACT8)
    be.lm_head(st, hb.LmHeadArgs(g, hb.TensorRef.of(rb), valid, hb.TensorRef.of(ib), 0))
    res, ids = np.zeros((len(head), 3), np.uint32), np.zeros(len(head), np.int32)
    be.download(st, hb.TensorRef.of(rb), res)
    be.download(st, hb.TensorRef.of(ib), ids)
    st.wait()
    limit = valid or V
    with np.errstate(invalid="ignore"):
        logits = (q.astype(np.float32) * head[:, None])[:, :limit]
    for i, h in enumerate(head):
        if np.isnan(h):
            assert res[i].tolist() == [0xFFFFFFFF, 0x7FC00000, 1] and ids[i] == 0
        else:
            best = int(np.argmax(logits[i]))  # the first of equals, as the sequential scan has it
            assert res[i].tolist() == [best, int(bits(logits[i, best:best + 1])[0]), 0] and ids[i] == best
