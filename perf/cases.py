"""The work that a host of this backend has it do, as cases to be timed and compared: single projections, the projections of one
transformer block from one decoded token to a prompt of thousands, the vocabulary head, the embedding rows of a prompt, and the repack
a loader does once per weight.

Everything goes through the C ABI (halo_cuda.h), the boundary a host binds, on one stream of one context, with device pointers.
Sizes: hidden 5120, FFN 17408 and the vocabulary of 151936 are this repository's benchmark configurations; `draw` spreads the same
operators over smaller and larger models, odd vocabularies and every batch size in between.
"""
from __future__ import annotations

import ctypes as C
import math

import torch

from halo_b200 import backend as hb
from halo_b200 import capi
from halo_b200.synth import BLOCK_BYTES, BLOCK_ELEMS, Q4_0, Q4_K, Q6_K, Q8_0, TYPE_IDS, row_bytes

MAX_FLOPS = 1.6e12     # of one pass: the largest listed case
MAX_WEIGHTS = 9.0e8    # of one pass: a vocabulary head of 151936 x 5120 and room for ragged ones


def listed() -> list[dict]:
    return [
        # the smallest call of a decoded token: the key and value projections, a launch's latency more than their 11 MB
        {"name": "kv_proj_m1", "op": "linear", "wtype": "q8_0", "rows": 2048, "cols": 5120, "m": 1, "raw": False},
        # one sequence decoding through a Gated-DeltaNet block: the norms in front fused in, the gate rows with their epilogue
        {"name": "gdn_layer_m1", "op": "layer", "kind": "gdn", "hidden": 5120, "inner": 6144, "kv": 2048, "ffn": 17408, "m": 1, "norm": True},
        # four parallel sequences through a grouped-query attention block in the Q4_K / Q6_K mix
        {"name": "gqa_layer_m4", "op": "layer", "kind": "gqa", "hidden": 5120, "inner": 5120, "kv": 1024, "ffn": 17408, "m": 4, "norm": False},
        # the down projection of a Q8_0 model for eight sequences
        {"name": "down_q8_0_m8", "op": "linear", "wtype": "q8_0", "rows": 5120, "cols": 17408, "m": 8, "raw": False},
        # speculative verify: four sequences of four draft tokens through the Q4_0 draft block
        {"name": "mtp_layer_m16", "op": "layer", "kind": "mtp", "hidden": 5120, "inner": 5120, "kv": 1024, "ffn": 17408, "m": 16, "norm": False},
        # the head behind it: logits and their argmax
        {"name": "head_q4_0_m16", "op": "head", "wtype": "q4_0", "vocab": 151936, "hidden": 5120, "m": 16},
        # a host without the repacking loader: rows as the file has them
        {"name": "raw_q8_0_m1", "op": "linear", "wtype": "q8_0", "rows": 5120, "cols": 17408, "m": 1, "raw": True},
        # a short prompt, a length no tile divides, on a small model
        {"name": "prompt_layer_m77", "op": "layer", "kind": "gqa", "hidden": 2048, "inner": 2048, "kv": 512, "ffn": 5632, "m": 77, "norm": False},
        # a prompt chunk through the up projection
        {"name": "prefill_q4_k_m512", "op": "linear", "wtype": "q4_k", "rows": 17408, "cols": 5120, "m": 512, "raw": False},
        # a long prompt through a whole block in the Q4_K / Q6_K mix: the largest pass
        {"name": "prefill_layer_m2048", "op": "layer", "kind": "gqa", "hidden": 5120, "inner": 5120, "kv": 1024, "ffn": 17408, "m": 2048, "norm": False},
        # the embedding rows of that prompt
        {"name": "embed_q4_k_2048", "op": "embed", "wtype": "q4_k", "vocab": 151936, "hidden": 5120, "ids": 2048},
        # what a loader does with a down projection once its bytes are on the device
        {"name": "repack_q6_k", "op": "repack", "wtype": "q6_k", "rows": 5120, "cols": 17408},
    ]


def _log_int(rng, lo: int, hi: int, step: int = 1) -> int:
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / step) * step))


def draw(rng) -> dict:
    while True:
        case = _draw(rng)
        w = work(case)
        weights = sum(p["rows"] * p["cols"] for p in _projections(case))
        if w["flops"] <= MAX_FLOPS and weights <= MAX_WEIGHTS:
            return case


def _draw(rng) -> dict:
    op = rng.choices(("linear", "layer", "head", "embed", "repack"), (30, 40, 10, 10, 10))[0]
    wtype = rng.choice(("q4_k", "q6_k", "q8_0", "q4_0"))
    if op == "linear":
        raw = wtype != "q4_k" and rng.random() < 0.3
        # raw rows of 32-weight blocks need not be whole groups of 256
        step = 32 if raw and wtype != "q6_k" else 256
        return {"op": op, "wtype": wtype, "rows": _log_int(rng, 256, 34816), "cols": _log_int(rng, 1024, 28672, step),
                "m": _log_int(rng, 1, 16 if raw else 1024), "raw": raw}
    hidden = _log_int(rng, 1024, 8192, 256)
    if op == "layer":
        m = _log_int(rng, 1, 2048)
        return {"op": op, "kind": rng.choice(("gdn", "gqa", "mtp")), "hidden": hidden, "inner": round(hidden * rng.uniform(0.8, 1.3) / 256) * 256,
                "kv": rng.choice((256, 512, 1024, 2048)), "ffn": round(hidden * rng.uniform(2.5, 3.7) / 256) * 256, "m": m,
                "norm": m == 1 and rng.random() < 0.5}
    vocab = _log_int(rng, 32000, 152064)
    if op == "head":
        return {"op": op, "wtype": wtype, "vocab": vocab, "hidden": hidden, "m": _log_int(rng, 1, 16)}
    if op == "embed":
        return {"op": op, "wtype": wtype, "vocab": vocab, "hidden": hidden, "ids": _log_int(rng, 1, 4096)}
    return {"op": op, "wtype": rng.choice(("q6_k", "q8_0", "q4_0")), "rows": _log_int(rng, 256, 34816), "cols": _log_int(rng, 1024, 17408, 256)}


# ---- what a case is made of ------------------------------------------------------------------------------------------------------

def _projections(case: dict) -> list[dict]:
    """The matrices of a case, in the order a forward pass reads them; projections of one x row are one operand, as a model holds them."""
    op = case["op"]
    if op in ("linear", "repack"):
        return [{"wtype": TYPE_IDS[case["wtype"]], "rows": case["rows"], "cols": case["cols"], "raw": case.get("raw", True) or case["wtype"] == "q4_k"}]
    if op in ("head", "embed"):
        return [{"wtype": TYPE_IDS[case["wtype"]], "rows": case["vocab"], "cols": case["hidden"], "raw": op == "embed"}]
    h, inner, kv, f, norm = case["hidden"], case["inner"], case["kv"], case["ffn"], case["norm"]

    def p(wtype, rows, cols, **more):
        return {"wtype": wtype, "rows": rows, "cols": cols, "raw": wtype == Q4_K, **more}

    if case["kind"] == "gdn":     # q|k|v|z, the beta|alpha gate rows (Q8_0, with their epilogue), out
        mix = [p(Q4_K, 2 * kv + 2 * inner, h, norm=norm), {"wtype": Q8_0, "rows": 2 * (inner // 128), "cols": h, "raw": True, "gates": inner // 128}, p(Q4_K, h, inner)]
    elif case["kind"] == "gqa":   # q|k, v (Q6_K), o
        mix = [p(Q4_K, inner + kv, h, norm=norm), p(Q6_K, kv, h, norm=norm), p(Q4_K, h, inner)]
    else:                         # the draft block: the projection of [embedding, hidden], q|k|v, o, all Q4_0
        return [p(Q4_0, h, 2 * h), p(Q4_0, inner + 2 * kv, h, norm=norm), p(Q4_0, h, inner), p(Q4_0, 2 * f, h, norm=norm), p(Q4_0, h, f)]
    return mix + [p(Q4_K, 2 * f, h, norm=norm), p(Q6_K, h, f)]


def work(case: dict) -> dict:
    op = case["op"]
    if op == "repack":  # the rows as the file has them in, the same codes and scales out
        p = _projections(case)[0]
        return {"bytes": 2 * p["rows"] * row_bytes(p["wtype"], p["cols"]), "flops": 0}
    if op == "embed":
        p = _projections(case)[0]
        return {"bytes": case["ids"] * (row_bytes(p["wtype"], p["cols"]) + 4 * p["cols"] + 4), "flops": 0}
    m = case["m"]
    nbytes = sum(p["rows"] * row_bytes(p["wtype"], p["cols"]) + 4 * m * (p["rows"] + p["cols"]) for p in _projections(case))
    return {"bytes": nbytes, "flops": sum(2 * m * p["rows"] * p["cols"] for p in _projections(case))}


def tolerance(case: dict):
    """Embedding rows and repacked bytes are exact.  A prompt of 64 rows and up rounds x and W to fp16 (3e-4 of the product's norm), a
    smaller batch rounds x to 16 bits per 256 elements (5e-5); raw rows of the 32-weight formats and Q6_K stay in fp32 (2e-7)."""
    if case["op"] in ("embed", "repack"):
        return "exact"
    if case["op"] == "linear" and case["raw"]:
        return {"rel": 1e-6}
    if case["m"] >= 64 and case["op"] != "head":
        return {"rel": 1.2e-3}
    return {"rel": 2e-4}


# ---- state -----------------------------------------------------------------------------------------------------------------------
_host = None


def _backend():
    """One context and one stream for the process, as a host keeps them."""
    global _host
    if _host is None:
        be = hb.CudaBackend(0)
        _host = (be, be.create_stream())
    return _host


def _check(rc: int) -> None:
    if rc != 0:
        raise hb.HaloError(rc, capi.last_error())


def _weights(gen: torch.Generator, wtype: int, rows: int, cols: int) -> torch.Tensor:
    """GGUF rows with uniform quant codes and fp16 scales uniform on [0.001, 0.02] (halo_b200.synth's distributions, made on the device)."""
    n, size = rows * (cols // BLOCK_ELEMS[wtype]), BLOCK_BYTES[wtype]
    raw = torch.randint(0, 256, (n, size), dtype=torch.uint8, device="cuda", generator=gen)
    if wtype == Q8_0:
        q = raw[:, 2:].view(torch.int8)
        q.clamp_(min=-127)
    if wtype == Q6_K:
        raw[:, 192:208] = ((raw[:, 192:208] & 127).to(torch.int16) - 64).to(torch.int8).view(torch.uint8)
    for at in {Q4_K: (0, 2), Q6_K: (208,), Q8_0: (0,), Q4_0: (0,)}[wtype]:
        d = torch.rand((n, 1), device="cuda", generator=gen) * 0.019 + 0.001
        raw[:, at:at + 2] = d.to(torch.float16).view(torch.uint8)
    return raw.view(rows, -1)


def _repacked(raw: torch.Tensor, wtype: int, rows: int, cols: int) -> torch.Tensor:
    be, st = _backend()
    out = torch.empty((rows, be.repacked_row_bytes(wtype, cols)), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    _check(be.lib.halo_cuda_repack_rows(be.ctx, wtype, raw.data_ptr(), 0, out.data_ptr(), 0, rows, cols, st.handle))
    st.wait()
    return out


def _operand(gen: torch.Generator, p: dict, m: int, prompt: bool):
    """A projection as a loader leaves it (Q4_K rows as the file has them, the other types repacked unless the host does not), its x rows
    and its y, and the call that goes with them."""
    be, _ = _backend()
    wtype, rows, cols = p["wtype"], p["rows"], p["cols"]
    w = _weights(gen, wtype, rows, cols)
    variant = 0
    if not p["raw"]:
        w, variant = _repacked(w, wtype, rows, cols), be.repacked_variant(wtype, cols)
    x = torch.randn((m, cols), device="cuda", generator=gen)
    y = torch.zeros((m, rows), device="cuda")
    g = capi.Gemv(wtype=wtype, variant_id=variant, w=w.data_ptr(), x=x.data_ptr(), y=y.data_ptr(), rows=rows, cols=cols, n_vec=m,
                  flags=capi.FLAG_ALLOW_GEMM if prompt else 0)
    return g, y, (w, x)


def prepare(case: dict, seed: int):
    be, st = _backend()
    lib, ctx, s = be.lib, be.ctx, st.handle
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    op, keep, calls, outputs = case["op"], [], [], []
    if op == "repack":
        p = _projections(case)[0]
        raw = _weights(gen, p["wtype"], p["rows"], p["cols"])
        out = torch.empty((p["rows"], be.repacked_row_bytes(p["wtype"], p["cols"])), dtype=torch.uint8, device="cuda")
        calls = [(lib.halo_cuda_repack_rows, (ctx, p["wtype"], raw.data_ptr(), 0, out.data_ptr(), 0, p["rows"], p["cols"], s))]
        keep, outputs = [raw], [out]
    elif op == "embed":
        p = _projections(case)[0]
        table = _weights(gen, p["wtype"], p["rows"], p["cols"])
        ids = torch.randint(0, p["rows"], (case["ids"],), dtype=torch.int32, device="cuda", generator=gen)
        out = torch.zeros((case["ids"], p["cols"]), device="cuda")
        status = torch.zeros(1, dtype=torch.int32, device="cuda")
        g = capi.GetRows(type=p["wtype"], table=table.data_ptr(), ids=ids.data_ptr(), out=out.data_ptr(), n_rows=p["rows"], cols=p["cols"],
                         n_ids=case["ids"], status=status.data_ptr())
        calls = [(lib.halo_cuda_get_rows, (ctx, C.byref(g), s))]
        keep, outputs = [table, ids, g], [out, status]
    elif op == "head":
        g, y, held = _operand(gen, _projections(case)[0], case["m"], False)
        result = torch.zeros((case["m"], 3), dtype=torch.int32, device="cuda")
        ids = torch.zeros(case["m"], dtype=torch.int32, device="cuda")
        h = capi.LmHead(gemv=g, result=result.data_ptr(), ids=ids.data_ptr())
        calls = [(lib.halo_cuda_lm_head, (ctx, C.byref(h), s))]
        keep, outputs = [held, h, result], [y, ids, result.view(torch.float32)[:, 1]]
    else:
        m = case["m"]
        prompt = m > 16 and not case.get("raw", False)  # a prompt's caller accepts the GEMM's numerics
        for p in _projections(case):
            g, y, held = _operand(gen, p, m, prompt)
            args = (ctx, C.byref(g), s)
            if p.get("gates"):
                dt_bias, a = torch.randn(p["gates"], device="cuda", generator=gen), -torch.rand(p["gates"], device="cuda", generator=gen)
                calls.append((lib.halo_cuda_gemv_gated, (ctx, C.byref(g), dt_bias.data_ptr(), a.data_ptr(), p["gates"], s)))
                keep += [dt_bias, a]
            elif p.get("norm"):
                norm_w = 1.0 + 0.1 * torch.randn(p["cols"], device="cuda", generator=gen)
                calls.append((lib.halo_cuda_gemv_normed, (ctx, C.byref(g), norm_w.data_ptr(), 1e-6, s)))
                keep.append(norm_w)
            else:
                calls.append((lib.halo_cuda_gemv, args))
            keep += [g, held]
            outputs.append(y)
    torch.cuda.synchronize()
    return {"calls": calls, "outputs": outputs, "keep": keep}


def run(state):
    for fn, args in state["calls"]:
        _check(fn(*args))
    return state["outputs"]
