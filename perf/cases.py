"""Workloads of the basecaller layer path, through the entry points a program calls.

Four kinds of pass, each at several sizes:

  lstm       the recurrent encoder: f16 features [T, B, H] are quantised per row, run through five
             factored-LSTM layers of alternating direction, and the last layer's int8 hidden output
             is dequantised and transposed to f16 [B, T, H] for the linear layer that follows
  lstm_step  one timestep of one layer in the two-kernel form, for a caller that drives the time
             loop itself (x and h down-projections, then the fused step on the carried state)
  tx         one transformer encoder layer on a quantised residual stream: QKV + rotary, per-row
             quantisation and output projection of the attention's result, norm, gated MLP, norm.
             The attention core and the MLP's second matrix are the caller's; their f16 results
             are inputs here. `dtype` says int8 or fp8 (e4m3)
  tx_f16     the row kernels of the same layer where the matrices stay f16 (a caller whose model
             has other dimensions): rotary on q and k in place, two norms, SiLU product

Inputs are normal, weights normal over the square root of the fan-in (0.02 for the transformer),
quantised as the model loader does it.
"""
import math

import torch

from fluke_b200 import lib, lstm, ops, prep

D, FF, HEADS, HEAD_DIM = 512, 2048, 8, 64   # the transformer dimensions the fused kernels have
RANK, LAYERS = 128, 5
ALPHA, EPS = 2.0, 1e-5


def listed():
    return [
        # The whole encoder over one full batch of chunks, and over the two batches that a server
        # with a queue of reads puts side by side.
        {"name": "lstm_1024x1000", "kind": "lstm", "B": 1024, "T": 1000, "H": 768},
        {"name": "lstm_2048x1000", "kind": "lstm", "B": 2048, "T": 1000, "H": 768},
        # The tail of a run: what is left of a batch, chunks of another length.
        {"name": "lstm_300x777", "kind": "lstm", "B": 300, "T": 777, "H": 768},
        # A few short chunks of a live read in the smaller model.
        {"name": "lstm_32x200_h384", "kind": "lstm", "B": 32, "T": 200, "H": 384},
        # A caller's own time loop: one step for few chunks, and for an ordinary batch of the
        # larger hidden size.
        {"name": "step_64", "kind": "lstm_step", "B": 64, "H": 768},
        {"name": "step_500_h1024", "kind": "lstm_step", "B": 500, "H": 1024},
        # int8 transformer layer: a batch of 32 chunks of 1000 positions, a ragged remainder, and
        # the single short chunk whose latency a live caller sees.
        {"name": "tx_i8_32x1000", "kind": "tx", "dtype": "i8", "chunks": 32, "seq": 1000},
        {"name": "tx_i8_7x1333", "kind": "tx", "dtype": "i8", "chunks": 7, "seq": 1333},
        {"name": "tx_i8_1x125", "kind": "tx", "dtype": "i8", "chunks": 1, "seq": 125},
        # fp8: the batch that fills the card's memory in a server, and a small odd one.
        {"name": "tx_fp8_128x1000", "kind": "tx", "dtype": "fp8", "chunks": 128, "seq": 1000},
        {"name": "tx_fp8_3x601", "kind": "tx", "dtype": "fp8", "chunks": 3, "seq": 601},
        # The f16 form of the layer.
        {"name": "tx_f16_32x1000", "kind": "tx_f16", "chunks": 32, "seq": 1000},
    ]


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["lstm", "lstm", "lstm_step", "tx", "tx", "tx", "tx_f16"])
    if kind == "lstm":
        h = rng.choice([384, 768, 768, 1024])
        return {"kind": kind, "B": _log(rng, 16, 1024 if h == 1024 else 2048), "T": _log(rng, 100, 1000), "H": h}
    if kind == "lstm_step":
        return {"kind": kind, "B": _log(rng, 16, 1024), "H": rng.choice([384, 768, 1024])}
    case = {"kind": kind, "chunks": _log(rng, 1, 128), "seq": rng.randint(100, 1500)}
    case["chunks"] = max(1, min(case["chunks"], 128000 // case["seq"]))
    if kind == "tx":
        case["dtype"] = rng.choice(["i8", "fp8"])
    return case


def _normal(gen, *shape, scale=1.0, mean=0.0, dtype=torch.float32):
    return (torch.randn(*shape, generator=gen, device="cuda", dtype=dtype) * scale + mean).to(dtype)


def _prepare_lstm(case, gen, cpu_gen):
    t, b, h = case["T"], case["B"], case["H"]
    layers = [lstm.FactoredLstmLayer.random(h, RANK, i % 2 == 1, cpu_gen, "cuda") for i in range(LAYERS)]
    need = lib.load().fluke_factored_lstm_layer_workspace(t, b, h, RANK)
    return {
        "layers": layers,
        "x": torch.randn(t, b, h, generator=gen, device="cuda", dtype=torch.float16),
        # what a program keeps from batch to batch
        "x_i8": torch.empty(t, b, h, dtype=torch.int8, device="cuda"),
        "x_scale": torch.empty(t * b, dtype=torch.float32, device="cuda"),
        "buffers": [torch.empty(t, b, h, dtype=torch.int8, device="cuda") for _ in range(2)],
        "workspace": torch.empty(need, dtype=torch.uint8, device="cuda"),
    }


def _run_lstm(s):
    x = s["x"]
    t, b, h = x.shape
    ops.quant_int8(x.view(t * b, h), out=s["x_i8"].view(t * b, h), scale=s["x_scale"])
    out, state = lstm.run_stack(s["layers"], s["x_i8"], s["x_scale"], workspace=s["workspace"], buffers=s["buffers"])
    y = ops.dequant_transpose(out, 1.0 / 127.0)
    return {"y": y, "c": [c for c, _ in state], "h": [h for _, h in state]}


def _prepare_step(case, gen, cpu_gen):
    b, h = case["B"], case["H"]
    x, xs = prep.quantize_int8_rows(_normal(gen, b, h))
    return {
        "layer": lstm.FactoredLstmLayer.random(h, RANK, False, cpu_gen, "cuda"),
        "x": x, "x_scale": xs,
        "c": _normal(gen, b, h, scale=0.3),
        "h": torch.randint(-90, 91, (b, h), generator=gen, device="cuda", dtype=torch.int8),
        "a": torch.empty(b, 2 * RANK, dtype=torch.float16, device="cuda"),
    }


def _run_step(s):
    layer, a = s["layer"], s["a"]
    ops.down_proj_i8(s["x"], layer.dn_ih, s["x_scale"], layer.dn_ih_scale, out=a[:, RANK:])
    ops.down_proj_i8(s["h"], layer.dn_hh, None, layer.dn_hh_scale, out=a[:, :RANK])
    ops.factored_lstm_step_i8(a, layer.w_up, layer.bias, s["c"], h_out=s["h"])
    return {"h": s["h"], "c": s["c"], "a": a}


def _prepare_tx(case, gen):
    m, seq, fp8 = case["chunks"] * case["seq"], case["seq"], case["dtype"] == "fp8"

    def quantise(t):
        q, scale = prep.quantize_fp8_rows(t) if fp8 else prep.quantize_int8_rows(t)
        return (q.view(torch.uint8) if fp8 else q).contiguous(), scale.contiguous()

    def weight(n, k):
        """Row-major int8, or the pre-shuffled fp8 layout whose copy is made when a model is loaded."""
        q, scale = quantise(_normal(gen, n, k, scale=0.02))
        if fp8:
            q = prep.preshuffle_fp8_weight(q)
            lib.load().fluke_fp8_release_weight(q.data_ptr())
            assert lib.load().fluke_fp8_prepare_weight(q.data_ptr(), n, k) == 0
        return q, scale

    a, sa = quantise(_normal(gen, m, D))
    sin, cos = prep.rotary_tables(seq, HEAD_DIM, device="cuda")
    return {
        "fp8": fp8, "seq": seq, "sin": sin, "cos": cos, "a": a, "sa": sa,
        "backend": ops.fp8_select(0, max_seq=2048) if fp8 else ops.int8_select(0, max_seq=2048),
        "wqkv": weight(3 * D, D), "gate": weight(FF, D), "up": weight(FF, D),
        "wo": quantise(_normal(gen, D, D, scale=0.02)),
        "norm1": _normal(gen, D, scale=0.1, mean=1.0, dtype=torch.float16),
        "norm2": _normal(gen, D, scale=0.1, mean=1.0, dtype=torch.float16),
        "attn": _normal(gen, m, D, dtype=torch.float16),   # the attention core's result
        "ff": _normal(gen, m, D, dtype=torch.float16),     # the MLP's second matrix's result
    }


def _run_tx(s):
    a, sa = s["a"], s["sa"]
    quant, gemm, norm, qkv_rotary, gated_mlp = (
        (ops.quant_fp8, ops.gemm_fp8, ops.rmsnorm_quant_fp8, ops.qkv_rotary_fp8, ops.gated_mlp_fp8) if s["fp8"] else
        (ops.quant_int8, ops.gemm_i8, ops.rmsnorm_quant_int8, ops.qkv_rotary_i8, ops.gated_mlp_i8))
    qkv = qkv_rotary(s["backend"], a, s["wqkv"][0], sa, s["wqkv"][1], s["sin"], s["cos"], s["seq"])
    attn_q, attn_s = quant(s["attn"])
    proj = gemm(attn_q, s["wo"][0], attn_s, s["wo"][1])
    norm(proj, s["norm1"], a, sa, ALPHA, EPS)
    act = gated_mlp(s["backend"], a, s["gate"][0], s["up"][0], sa, s["gate"][1], s["up"][1])
    norm(s["ff"], s["norm2"], a, sa, ALPHA, EPS)
    return {"qkv": qkv, "proj": proj, "act": act, "residual": a, "residual_scale": sa}


def _prepare_tx_f16(case, gen):
    n, seq = case["chunks"], case["seq"]
    m = n * seq
    sin, cos = prep.rotary_tables(seq, HEAD_DIM, device="cuda")

    def f16(*shape, **kw):
        return _normal(gen, *shape, dtype=torch.float16, **kw)

    return {
        "qkv": f16(n, seq, 3, HEADS, HEAD_DIM), "sin": sin, "cos": cos,
        "x": f16(m, D), "attn": f16(m, D), "ff": f16(m, D), "up_gate": f16(m, 2 * FF),
        "norm1": f16(D, scale=0.1, mean=1.0), "norm2": f16(D, scale=0.1, mean=1.0),
    }


def _run_tx_f16(s):
    ops.rotary_qkv_(s["qkv"], s["sin"], s["cos"], HEAD_DIM // 2)
    x1 = ops.rmsnorm(s["attn"], s["x"], s["norm1"], ALPHA, EPS)
    act = ops.silu_mul(s["up_gate"])
    x2 = ops.rmsnorm(s["ff"], x1, s["norm2"], ALPHA, EPS)
    return {"qkv": s["qkv"], "x1": x1, "act": act, "x2": x2}


_KINDS = {
    "lstm": (_prepare_lstm, _run_lstm),
    "lstm_step": (_prepare_step, _run_step),
    "tx": (lambda case, gen, cpu_gen: _prepare_tx(case, gen), _run_tx),
    "tx_f16": (lambda case, gen, cpu_gen: _prepare_tx_f16(case, gen), _run_tx_f16),
}


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    state = _KINDS[case["kind"]][0](case, gen, torch.Generator().manual_seed(seed))
    state["kind"] = case["kind"]
    return state


def run(state):
    return _KINDS[state["kind"]][1](state)


def work(case):
    """Inputs read once, outputs written once, multiply-adds as two operations."""
    kind = case["kind"]
    if kind in ("lstm", "lstm_step"):
        b, h = case["B"], case["H"]
        t, layers = (case["T"], LAYERS) if kind == "lstm" else (1, 1)
        weights = 2 * RANK * h + 8 * RANK + 4 * h * 2 * RANK * 2 + 4 * h * 4
        flops = 2 * t * b * layers * (4 * h * 2 * RANK + 2 * RANK * h)
        if kind == "lstm":   # f16 in and out; final c and h of every layer
            return {"bytes": 4 * t * b * h + layers * (weights + 5 * b * h), "flops": flops}
        return {"bytes": 3 * b * h + 4 * b + 8 * b * h + 2 * b * 2 * RANK + weights, "flops": flops}
    m, tables = case["chunks"] * case["seq"], 2 * 4 * case["seq"] * (HEAD_DIM // 2)
    if kind == "tx":
        n = 3 * D + D + 2 * FF
        residual = 2 * (m * D + 4 * m)
        return {"bytes": residual + 2 * 2 * m * D + 2 * m * (3 * D + D + FF) + n * D + 4 * n + tables + 2 * 2 * D,
                "flops": 2 * m * D * n}
    rows = 2 * 2 * m * 2 * D + 3 * 2 * m * D + 2 * 2 * m * D + 3 * 2 * m * FF
    return {"bytes": rows + tables + 2 * 2 * D, "flops": m * (2 * D * 3 + 2 * D * 8 + FF * 8)}


def tolerance(case):
    """f16 results round at 2^-11; the int8 and e4m3 codes of two correct implementations differ by
    one step where a value lies at a rounding boundary. In the recurrence such a step feeds back,
    so the dequantised output carries a share of one-code (1/127) differences."""
    if case["kind"] == "lstm":
        return {"rel": 5e-3, "max": 0.2, "differ": 0.01}
    if case["kind"] == "lstm_step":
        return {"rel": 1e-3, "max": 2e-2, "differ": 5e-3}
    if case["kind"] == "tx":
        return {"rel": 1e-3, "max": 2e-2, "differ": 2e-3}
    return {"rel": 1e-3, "max": 2e-2}
