"""The work that users of this library have it do, as cases that can be prepared, run and compared.

``listed()`` holds the fixed cases, ``draw(rng)`` gives one more of the same ranges, ``prepare(case, seed)`` makes what a
program holds before the call (weights in storage form, activations, runners), ``run(state)`` is one pass through the
public entry points. Kinds of case:

  linear     ``LinearRunner.forward`` of one layer: every weight format, native fp4 or the dequantizing arm, bias, AWQ
             pre-scale, GELU / SwiGLU in the epilogue
  ffn        an up / down pair through ``prepare`` + ``forward_prepared``, whole or in the row chunks the DiT uses
  block      ``Nvfp4Block.forward``: norms, projections, QK-norm and RoPE, self-attention, gated residuals, FFN
  attention  ``sfq_attention_forward`` by itself: a chunk of queries against all keys, grouped heads
  lora       ``LoraRunner.apply`` beside a projection
  f32        ``LinearRunner.forward_f32``, the few timestep rows behind the adaLN tables

Weights are N(0, 0.02) put into the storage form here with torch (not by the library's host packers, which are an offline
step), activations N(0, 1) with 0.1 % of them 20 times as large, as the benchmark configurations have them.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

import slopfab_b200 as sfq
from slopfab_b200.block import BlockWeights, Nvfp4Block, Nvfp4Linear
from slopfab_b200.lora import LoraRunner

HIDDEN, FFN = 5120, 13824  # the DiT of the benchmark configurations
HEAD_DIM = 128
FORMATS = {"nvfp4": sfq.NVFP4, "w4a8": sfq.W4A8, "w6a8": sfq.W6A8, "i8": sfq.I8, "f8": sfq.F8E4M3, "nf4": sfq.NF4, "f16": sfq.F16,
           "bf16": sfq.BF16, "f32": sfq.F32}
# stored bytes per weight, scales of the block formats included
STORED = {"nvfp4": 0.5 + 1 / 16, "w4a8": 0.5 + 1 / 16, "w6a8": 0.75 + 1 / 64, "i8": 1, "f8": 1, "nf4": 0.5 + 1 / 64, "f16": 2, "bf16": 2,
          "f32": 4}
ACTS = {"none": sfq.ACT_NONE, "gelu": sfq.ACT_GELU_TANH, "swiglu": sfq.ACT_SWIGLU}
MODULATION = ("scale_msa", "shift_msa", "gate_msa", "scale_mlp", "shift_mlp", "gate_mlp")


# ---------------------------------------------------------------- the cases

def _linear(fmt, rows, k, n, act="none", bias=False, native=True, awq=False):
    return {"kind": "linear", "fmt": fmt, "rows": rows, "k": k, "n": n, "act": act, "bias": bias, "native": native, "awq": awq}


def _ffn(fmt, rows, k, n, chunk, native):
    return {"kind": "ffn", "fmt": fmt, "rows": rows, "k": k, "n": n, "chunk": chunk, "native": native}


def _block(rows, heads, ffn, form, rope):
    return {"kind": "block", "rows": rows, "heads": heads, "ffn": ffn, "form": form, "rope": rope}


def listed():
    return [
        # Benchmark configuration 1: the smallest Linear that is quoted. Launches and host work are most of it.
        dict(_linear("nvfp4", 256, 1024, 1024, bias=True), name="nvfp4_256x1024x1024"),
        # The text rows of a prompt through the FFN up-projection: few rows, the whole weight has to be read.
        dict(_linear("nvfp4", 77, HIDDEN, FFN, act="gelu"), name="nvfp4_text_rows_up"),
        # A text encoder's INT8 weight-only layer with its ConvRot rotation, a prompt of some hundred tokens.
        dict(_linear("i8", 333, 4096, 4096), name="int8_encoder_layer"),
        # The timestep rows behind the adaLN tables of an unpruned checkpoint: six vectors per modality, fp32 throughout.
        {"kind": "f32", "fmt": "f32", "rows": 3, "k": HIDDEN, "n": 6 * HIDDEN, "bias": True, "name": "adaln_f32_timesteps"},
        # Benchmark configuration 2: the attention projection of an image-sized sequence.
        dict(_linear("w4a8", 4096, HIDDEN, HIDDEN, bias=True), name="w4a8_4096_projection"),
        # A style LoRA beside one projection of the same sequence.
        {"kind": "lora", "rows": 4096, "k": HIDDEN, "n": HIDDEN, "rank": 32, "name": "lora_rank32_4096"},
        # The library's default for NVFP4 (native off): dequantize once, then the DiT's 2048-row chunk loop in bf16.
        dict(_ffn("nvfp4", 6200, HIDDEN, FFN, chunk=2048, native=False), name="nvfp4_dense_ffn_chunks"),
        # One GPU's share of the video configuration's tokens on eight GPUs: NVFP4 up-projection.
        dict(_linear("nvfp4", 13950, HIDDEN, FFN), name="nvfp4_13950_up"),
        # ... and on four GPUs: the W4A8 down-projection with its wide activation.
        dict(_linear("w4a8", 27900, FFN, HIDDEN), name="w4a8_27900_down"),
        # Benchmark configuration 3: the W6A8 FFN pair with GELU between.
        dict(_ffn("w6a8", 32760, HIDDEN, FFN, chunk=0, native=True), name="w6a8_32760_ffn_pair"),
        # A block of a short clip in the H3 form: SwiGLU, QK-norm and RoPE, a row count that fits no tile.
        dict(_block(4747, 40, FFN, "swiglu", True), name="block_4747_h3"),
        # Benchmark configuration 4: one block at the full video latent. The largest case.
        dict(_block(75600, 40, FFN, "gelu", False), name="block_75600"),
    ]


def _spread(rng, lo, hi):
    """An integer of [lo, hi], spread over its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _multiple(rng, lo, hi, unit):
    return _spread(rng, lo // unit, hi // unit) * unit


def _rows_within(rng, lo, hi, cost_per_row, most):
    return _spread(rng, lo, max(lo, min(hi, int(most / cost_per_row))))


def draw(rng):
    kind = rng.choices(("linear", "ffn", "block", "attention", "lora", "f32"), (10, 3, 3, 3, 2, 2))[0]
    dit = rng.random() < 0.5  # the DiT's own layer sizes, or any
    if kind == "linear":
        fmt = rng.choice(("nvfp4", "nvfp4", "nvfp4", "w4a8", "w4a8", "w6a8", "i8", "f8", "nf4", "f16", "bf16"))
        k, n = rng.choice(((HIDDEN, HIDDEN), (HIDDEN, 3 * HIDDEN), (HIDDEN, FFN), (FFN, HIDDEN))) if dit else (
            _multiple(rng, 256, FFN, 256), _multiple(rng, 256, 15360, 128))
        if not dit and fmt in ("i8", "f8", "f16", "bf16"):
            n += rng.choice((0, 8, 40, 3))
        act = rng.choice(("none", "none", "none", "gelu", "swiglu"))
        if act == "swiglu" and n % 256:
            act = "gelu"
        rows = _rows_within(rng, 1, 111600, 2 * k * n, 8e12)
        native = fmt != "nvfp4" or rng.random() < 0.75
        return _linear(fmt, rows, k, n, act, rng.random() < 0.4, native, fmt in ("f16", "bf16", "nf4") and rng.random() < 0.25)
    if kind == "ffn":
        fmt = rng.choice(("nvfp4", "w4a8", "w6a8"))
        k, n = (HIDDEN, FFN) if dit else (_multiple(rng, 512, HIDDEN, 256), _multiple(rng, 1024, FFN, 256))
        return _ffn(fmt, _rows_within(rng, 64, 32760, 4 * k * n, 9e12), k, n, rng.choice((0, 0, 2048)), fmt != "nvfp4" or rng.random() < 0.5)
    if kind == "block":
        heads = rng.choice((8, 12, 24, 40))
        form = rng.choice(("gelu", "swiglu"))
        return _block(_spread(rng, 200, 24000), heads, _multiple(rng, 256 * heads, 384 * heads, 256), form, rng.random() < 0.5)
    if kind == "attention":
        kv_heads = rng.choice((4, 8, 10, 40))
        heads = kv_heads * (rng.choice((1, 2, 4)) if kv_heads < 40 else 1)
        seq_kv = _spread(rng, 60, 40000)
        seq_q = rng.choice((seq_kv, min(seq_kv, 2048), _spread(rng, 1, seq_kv)))
        return {"kind": "attention", "seq_q": seq_q, "seq_kv": seq_kv, "heads": heads, "kv_heads": kv_heads}
    if kind == "lora":
        return {"kind": "lora", "rows": _spread(rng, 1, 32760), "k": _multiple(rng, 512, FFN, 64), "n": _multiple(rng, 512, FFN, 64),
                "rank": rng.choice((4, 8, 16, 32, 64, 128))}
    return {"kind": "f32", "fmt": rng.choice(("f32", "bf16", "nvfp4")), "rows": _spread(rng, 1, 64), "k": _multiple(rng, 256, HIDDEN, 64),
            "n": _multiple(rng, 256, 6 * HIDDEN, 128), "bias": rng.random() < 0.5}


# ---------------------------------------------------------------- inputs

def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) & 0x7FFFFFFF)


def _activation(g, rows, k):
    x = torch.randn((rows, k), device="cuda", generator=g, dtype=torch.bfloat16)
    loud = torch.rand((rows, k), device="cuda", generator=g, dtype=torch.bfloat16) < 1e-3
    return torch.where(loud, x * 20, x)


def _pack_nibbles(codes, high_even):
    even, odd = codes[:, 0::2], codes[:, 1::2]
    return ((even << 4) | odd if high_even else even | (odd << 4)).contiguous()


def _tile_scales(s):
    """[n, k/16] scale bytes in the 128 x 4 tiling."""
    n, kb = s.shape
    return s.view(n // 128, 4, 32, kb // 4, 4).permute(0, 3, 2, 1, 4).contiguous().view(-1)


def _encode_nvfp4(w):
    n, k = w.shape
    top = float(w.abs().max()) / (6 * 448)
    blocks = (w / top).view(n, k // 16, 16)
    scale = (blocks.abs().amax(-1) / 6).clamp(max=448).to(torch.float8_e4m3fn)
    s = scale.float().unsqueeze(-1)
    v = torch.where(s > 0, blocks / s, torch.zeros_like(blocks))
    edges = torch.tensor([0.25, 0.75, 1.25, 1.75, 2.5, 3.5, 5.0], device=w.device)
    codes = torch.bucketize(v.abs(), edges, out_int32=True).to(torch.uint8) | ((v < 0).to(torch.uint8) << 3)
    return _pack_nibbles(codes.view(n, k), True), _tile_scales(scale.view(torch.uint8)), top


def _nvfp4_linear(g, n, k):
    data, scale, top = _encode_nvfp4(0.02 * torch.randn((n, k), device="cuda", generator=g))
    return Nvfp4Linear(data, scale, top, n, k)


def _encode_group_int(w, levels, group):
    """(codes 0 .. 2 levels - 1, e4m3 group scale bytes, fp32 channel scales) of W4A8 / W6A8: q = level * scale in int8 steps."""
    n, k = w.shape
    channel = w.abs().amax(1) / 127
    v = (w / channel.unsqueeze(1)).view(n, k // group, group)
    scale = (v.abs().amax(-1) / (levels - 1)).clamp(min=2 ** -6).to(torch.float8_e4m3fn)
    codes = (torch.round(v / scale.float().unsqueeze(-1)).clamp(-levels, levels - 1) + levels).to(torch.uint8)
    return codes.view(n, k), scale.view(torch.uint8).contiguous(), channel.float()


def _encode_nf4(w, block=64, nested=256):
    quantiles = torch.linspace(0.02, 0.98, 16, device=w.device)
    table = torch.special.ndtri(quantiles)
    table = (table / table.abs().max()).float()
    flat = w.reshape(-1, block)
    top = flat.abs().amax(1)
    offset = float(top.mean())
    rest = top - offset
    pad = (-rest.numel()) % nested
    outer = torch.nn.functional.pad(rest, (0, pad)).view(-1, nested).abs().amax(1).clamp(min=1e-12)
    inner_map = torch.linspace(-1, 1, 256, device=w.device)
    inner = rest / outer.repeat_interleave(nested)[: rest.numel()]
    absmax = torch.round((inner + 1) * 127.5).clamp(0, 255).to(torch.uint8)
    codes = torch.bucketize(flat / top.unsqueeze(1), (table[1:] + table[:-1]) / 2, out_int32=True).to(torch.uint8)
    return _pack_nibbles(codes.view(w.shape), True), absmax, table, inner_map.float(), outer.float(), offset


def _weight(g, fmt, n, k, bias, awq=False):
    """(QuantWeight, the tensors it points at)."""
    w = torch.randn((n, k), device="cuda", generator=g).mul_(0.02)
    f = {"format": FORMATS[fmt], "out_features": n, "in_features": k}
    keep = {}
    if fmt == "nvfp4":
        keep["data"], keep["block_scale"], f["global_scale"] = _encode_nvfp4(w)
    elif fmt in ("w4a8", "w6a8"):
        group = 16 if fmt == "w4a8" else 64
        codes, keep["block_scale"], keep["weight_scale"] = _encode_group_int(w, 8 if fmt == "w4a8" else 32, group)
        if fmt == "w4a8":
            keep["data"] = _pack_nibbles(codes, False)
            keep["w4_codebook"] = torch.arange(-8, 8, device="cuda", dtype=torch.float32)
        else:
            high = (codes >> 4).view(n, k // 4, 4)
            high = high[..., 0] | (high[..., 1] << 2) | (high[..., 2] << 4) | (high[..., 3] << 6)
            keep["data"] = torch.cat([_pack_nibbles(codes & 15, False), high], dim=1).contiguous()
        f.update(packed_group_size=group, convrot=1, convrot_group=256)
    elif fmt == "i8":
        keep["weight_scale"] = (w.abs().amax(1) / 127).contiguous()
        keep["data"] = torch.round(w / keep["weight_scale"].unsqueeze(1)).to(torch.int8)
        f.update(per_channel_scale=1, convrot=1, convrot_group=256)
    elif fmt == "f8":
        keep["weight_scale"] = (w.abs().max() / 448).view(1)
        keep["data"] = (w / keep["weight_scale"]).to(torch.float8_e4m3fn).view(torch.uint8)
    elif fmt == "nf4":
        (keep["data"], keep["nf4_absmax"], keep["nf4_quant_map"], keep["nf4_nested_quant_map"], keep["nf4_nested_absmax"],
         f["nf4_nested_offset"]) = _encode_nf4(w)
        f.update(nf4_block_size=64, nf4_nested_block_size=256)
    else:
        keep["data"] = w.to({"f16": torch.float16, "bf16": torch.bfloat16, "f32": torch.float32}[fmt])
    if bias:
        keep["bias"] = 0.01 * torch.randn(n, device="cuda", generator=g)
        f["bias_format"] = sfq.F32
    if awq:
        keep["pre_quant_scale"] = (0.5 + torch.rand(k, device="cuda", generator=g)).to(torch.bfloat16)
    return sfq.new_weight(**f, **{name: sfq.ptr(t) for name, t in keep.items()}), keep


def _runner(native=False, act="none"):
    r = sfq.LinearRunner()
    r.set_native(native)
    r.set_activation(ACTS[act])
    return r


def prepare(case, seed):
    g = _generator(seed)
    kind = case["kind"]
    s = {"case": case, "kind": kind}
    if kind == "linear":
        s["w"], s["keep"] = _weight(g, case["fmt"], case["n"], case["k"], case["bias"], case["awq"])
        s["x"] = _activation(g, case["rows"], case["k"])
        s["runner"] = _runner(case["native"], case["act"])
    elif kind == "ffn":
        k, n, rows = case["k"], case["n"], case["rows"]
        s["up"], s["up_keep"] = _weight(g, case["fmt"], n, k, False)
        s["down"], s["down_keep"] = _weight(g, case["fmt"], k, n, False)
        s["x"] = _activation(g, rows, k)
        s["r_up"], s["r_down"] = _runner(case["native"], "gelu"), _runner(case["native"])
        s["chunk"] = case["chunk"] or rows
        s["h"] = torch.empty((s["chunk"], n), dtype=torch.bfloat16, device="cuda")
        s["y"] = torch.empty((rows, k), dtype=torch.bfloat16, device="cuda")
    elif kind == "block":
        rows, heads, ffn = case["rows"], case["heads"], case["ffn"]
        hidden = heads * HEAD_DIM
        s["x"] = torch.randn((rows, hidden), device="cuda", generator=g).to(torch.bfloat16)
        ones = torch.ones(hidden, device="cuda", dtype=torch.bfloat16)
        head = (1 + 0.05 * torch.randn((2, HEAD_DIM), device="cuda", generator=g)).to(torch.bfloat16) if case["rope"] else None
        up = 2 * ffn if case["form"] == "swiglu" else ffn
        s["w"] = BlockWeights(_nvfp4_linear(g, 3 * hidden, hidden), _nvfp4_linear(g, hidden, hidden), _nvfp4_linear(g, up, hidden),
                              _nvfp4_linear(g, hidden, ffn), ones, ones, head[0] if case["rope"] else None, head[1] if case["rope"] else None)
        s["mod"] = {name: 0.1 * torch.randn((3, hidden), device="cuda", generator=g) for name in MODULATION}
        s["index"] = torch.zeros(rows, dtype=torch.int32, device="cuda")  # video rows, then a run of text, then audio
        s["index"][rows - rows // 8:] = 1
        s["index"][rows - rows // 32:] = 2
        s["rope"] = None
        if case["rope"]:
            angle = torch.arange(rows, device="cuda").unsqueeze(1) * torch.logspace(0, -4, 48, device="cuda").repeat(2)
            s["rope"] = (torch.cos(angle), torch.sin(angle))
        s["block"] = Nvfp4Block(rows, hidden, heads, ffn, ffn_form=case["form"])
    elif kind == "attention":
        sq, skv, hq, hk = case["seq_q"], case["seq_kv"], case["heads"], case["kv_heads"]
        s["q"] = torch.randn((sq, hq * HEAD_DIM), device="cuda", generator=g).to(torch.bfloat16)
        s["kv"] = torch.randn((skv, 2 * hk * HEAD_DIM), device="cuda", generator=g).to(torch.bfloat16)
        s["out"] = torch.empty_like(s["q"])
        size = ctypes.c_size_t()
        sfq.check(sfq.lib.sfq_attention_workspace_bytes(skv, hk, HEAD_DIM, ctypes.byref(size)))
        s["ws"] = torch.empty(size.value, dtype=torch.uint8, device="cuda")
    elif kind == "lora":
        rng = np.random.default_rng(seed)
        k, n, rank = case["k"], case["n"], case["rank"]
        s["lora"] = LoraRunner()
        s["lora"].attach(1, (rng.standard_normal((rank, k), np.float32) / math.sqrt(k)).astype(np.float32),
                         (0.1 * rng.standard_normal((n, rank), np.float32)).astype(np.float32))
        s["x"] = _activation(g, case["rows"], k)
        s["y"] = torch.randn((case["rows"], n), device="cuda", generator=g).to(torch.bfloat16)
    elif kind == "f32":
        s["w"], s["keep"] = _weight(g, case["fmt"], case["n"], case["k"], case["bias"])
        s["x"] = torch.randn((case["rows"], case["k"]), device="cuda", generator=g)
        s["runner"] = _runner()
    else:
        raise ValueError(f"unknown kind of case: {kind}")
    return s


# ---------------------------------------------------------------- one pass

def run(s):
    kind = s["kind"]
    if kind == "linear":
        return s["runner"].forward(s["w"], s["x"])
    if kind == "ffn":
        x, y, h, chunk = s["x"], s["y"], s["h"], s["chunk"]
        p_up, used_up = s["r_up"].prepare(s["up"], chunk)
        p_down, used_down = s["r_down"].prepare(s["down"], chunk)
        for r in range(0, x.shape[0], chunk):
            part = x[r:r + chunk]
            hidden = s["r_up"].forward_prepared(s["up"], p_up, used_up, part, h[:part.shape[0]])
            s["r_down"].forward_prepared(s["down"], p_down, used_down, hidden, y[r:r + chunk])
        return y
    if kind == "block":
        return s["block"].forward(s["x"], s["w"], s["mod"], s["index"], rope=s["rope"])
    if kind == "attention":
        c, q, kv, out, ws = s["case"], s["q"], s["kv"], s["out"], s["ws"]
        width = c["kv_heads"] * HEAD_DIM
        sfq.check(sfq.lib.sfq_attention_forward(q.data_ptr(), q.stride(0), kv.data_ptr(), kv.data_ptr() + 2 * width, kv.stride(0),
                                                out.data_ptr(), out.stride(0), c["seq_q"], c["seq_kv"], c["heads"], c["kv_heads"], HEAD_DIM,
                                                0.0, ws.data_ptr(), ws.numel(), sfq.stream_ptr()))
        return out
    if kind == "lora":
        return s["lora"].apply(1, s["x"], s["y"])
    return s["runner"].forward_f32(s["w"], s["x"])


# ---------------------------------------------------------------- what a pass cannot do without, and how close results come

def work(case):
    kind = case["kind"]
    if kind in ("linear", "f32"):
        rows, k, n = case["rows"], case["k"], case["n"]
        e = 4 if kind == "f32" else 2
        out = n // 2 if case.get("act") == "swiglu" else n
        return {"bytes": e * rows * (k + out) + STORED[case["fmt"]] * n * k, "flops": 2 * rows * n * k}
    if kind == "ffn":
        rows, k, n = case["rows"], case["k"], case["n"]
        return {"bytes": 4 * rows * k + 2 * STORED[case["fmt"]] * n * k, "flops": 4 * rows * n * k}
    if kind == "block":
        rows, hidden, ffn = case["rows"], case["heads"] * HEAD_DIM, case["ffn"]
        up = 2 * ffn if case["form"] == "swiglu" else ffn
        weights = 4 * hidden * hidden + (up + ffn) * hidden
        tables = rows * (4 + (8 * 96 if case["rope"] else 0))
        return {"bytes": 4 * rows * hidden + STORED["nvfp4"] * weights + tables, "flops": 2 * rows * weights + 4 * rows * rows * hidden}
    if kind == "attention":
        sq, skv, hq, hk = case["seq_q"], case["seq_kv"], case["heads"], case["kv_heads"]
        return {"bytes": 2 * HEAD_DIM * (2 * sq * hq + 2 * skv * hk), "flops": 4 * sq * skv * hq * HEAD_DIM}
    rows, k, n, rank = case["rows"], case["k"], case["n"], case["rank"]
    return {"bytes": 2 * (rows * (k + 2 * n) + rank * (k + n)), "flops": 2 * rows * rank * (k + n)}


def tolerance(case):
    """About four times what was measured between the path and the same sums in another order or in fp64 (figures beside each)."""
    kind = case["kind"]
    if kind == "f32":  # fp32 sums of 5120 products against fp64: 1.3e-6, 9.4e-6
        return {"rel": 5e-6, "max": 4e-5}
    if kind == "block":  # another attention kernel in the block: 1.0e-2, 0.26 (a last-bit difference moves an fp4 code of the next layer)
        return {"rel": 3e-2, "max": 0.99}
    if kind == "ffn" and (case["fmt"] != "nvfp4" or case["native"]):  # hidden rows that differ in the last bf16 bit: 5.1e-3, 6.2e-2
        return {"rel": 2e-2, "max": 0.25}
    if kind == "attention":  # against fp64: 2.3e-3, 1.0e-2
        return {"rel": 9e-3, "max": 4e-2}
    if kind == "lora":  # against fp64, the hidden rows rounded to bf16: 2.3e-3, 1.4e-2
        return {"rel": 9e-3, "max": 5e-2}
    if case.get("act", "none") != "none":  # bf16 sums through GELU / SwiGLU against fp64: 3.0e-3, 1.2e-2
        return {"rel": 1.2e-2, "max": 5e-2}
    return {"rel": 7e-3, "max": 1.6e-2}  # the bf16 rounding of a sum against fp64: 1.7e-3, 3.9e-3
