"""The work that is timed: what a program that uses this package has it do, in five kinds.

product  one fused dequantize-and-matmul, `qmm.quantized_matmul`, called as a layer calls it (no
         graph, a result of its own): 1 row (a decoded token) to 4096 rows (a prompt), int4 / int8
         affine and MXFP4 weights, bf16 / f16 / float32 activations and tables.
experts  the gathered SwiGLU expert block of a mixture-of-experts layer, `moe.moe_experts`, from a
         few decoded tokens to a prompt of 4096.
step     one decode step of a Llama-shaped model, `llama.DecodeStep`, replayed from its graph with
         new token ids, as a serving loop does.
program  a StableHLO program with quantized Dense layers, `engine.execute`: the drop-in path.
pack     a quantized layer's stored arrays made into the fused op's operands,
         `qmm.from_keras_int4`, as loading a model does for each of its layers.

Inputs are synthetic: codes uniform over their whole range, scales U(0.002, 0.02), biases at the
middle code, activations N(0, 1); the decode step's weights are N(0, 0.02) quantized per group of 64
(the projections into the residual stream smaller).
"""

from __future__ import annotations

import math

import torch

from metaljax_b200 import engine, llama, moe, qmm

DEV = "cuda"
DTYPES = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}
BYTES = {"bf16": 2, "f16": 2, "f32": 4}


def product(name, m, k, n, quant="int4", group=64, x="bf16", tables="bf16"):
    return {"name": name, "kind": "product", "m": m, "k": k, "n": n, "quant": quant, "group": group, "x": x, "tables": tables}


def listed():
    return [
        # the smallest call there is: one token through an attention output projection (launch latency)
        product("one_row_4096x4096", 1, 4096, 4096),
        # a few sequences decoded together, through a gate-and-up projection
        product("rows8_28672x4096", 8, 4096, 28672),
        # a few dozen rows, not a round number, in f16, through a down projection of 8-bit codes
        product("rows45_int8_4096x14336", 45, 14336, 4096, "int8", 128, "f16", "f16"),
        # a prompt of 2048 tokens through a gate projection
        product("prompt2048_14336x4096", 2048, 4096, 14336),
        # a prompt of 512 tokens, MXFP4, at a width that is not a multiple of 128
        product("prompt512_mxfp4_5760x2880", 512, 2880, 5760, "mxfp4", 32),
        # a model kept in float32 throughout (what keras does by default), a small batch
        product("rows33_float32_4096x4096", 33, 4096, 4096, "int4", 64, "f32", "f32"),
        # 8 sequences decoded through a layer of 8 experts, two of them per token
        {"name": "experts_8_tokens", "kind": "experts", "tokens": 8, "top": 2, "experts": 8, "d": 4096, "ffn": 14336, "quant": "int4", "group": 64},
        # a prompt of 4096 tokens through the same layer
        {"name": "experts_4096_tokens", "kind": "experts", "tokens": 4096, "top": 2, "experts": 8, "d": 4096, "ffn": 14336, "quant": "int4", "group": 64},
        # one sequence, and a full batch of them, decoded by an 8B-parameter model over 2048 positions of context
        {"name": "step_batch1", "kind": "step", "batch": 1, "layers": 32, "heads": 32, "kv_heads": 8, "ffn": 14336, "vocab": 128256, "ctx": 2048},
        {"name": "step_batch64", "kind": "step", "batch": 64, "layers": 32, "heads": 32, "kv_heads": 8, "ffn": 14336, "vocab": 128256, "ctx": 2048},
        # a compiled feed-forward block of int4 Dense layers, four rows a call
        {"name": "program_4_rows", "kind": "program", "m": 4, "d": 2048, "ffn": 5632, "group": 64},
        # one layer of a checkpoint on its way in
        {"name": "pack_4096x14336", "kind": "pack", "k": 4096, "n": 14336, "group": 64},
    ]


def spread(rng, lo, hi):
    """A whole number of [lo, hi], even over its logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["product"] * 10 + ["experts"] * 4 + ["step"] * 3 + ["program"] * 2 + ["pack"] * 2)
    if kind == "product":
        quant = rng.choice(["int4", "int4", "int4", "int8", "mxfp4"])
        group = 32 if quant == "mxfp4" else rng.choice([32, 64, 64, 128])
        x = rng.choice(["bf16", "bf16", "bf16", "bf16", "f16", "f32"])
        tables = "f32" if rng.random() < 0.2 else x
        m = spread(rng, 1, 16) if rng.random() < 0.4 else spread(rng, 1, 4096)
        k = 128 * spread(rng, 4, 112)
        if rng.random() < 0.3:
            k += group * rng.randrange(1, 4)              # not whole tiles of the contraction
        n = spread(rng, 256, 131072)
        if rng.random() < 0.6:
            n = max(256, n // 64 * 64)
        if x == "f32":
            m = min(m, 64)
        n = max(256, min(n, (64 * 4096 * 14336 if x == "f32" else 2048 * 4096 * 14336) // (m * k)))
        c = product("", m, k, n, quant, group, x, tables)
        del c["name"]
        return c
    if kind == "experts":
        d, ffn = 128 * rng.randrange(8, 33), 128 * rng.randrange(8, 113)
        tokens = spread(rng, 1, 32) if rng.random() < 0.5 else spread(rng, 1, 4096)
        quant = rng.choice(["int4", "int4", "mxfp4"])
        return {"kind": kind, "tokens": tokens, "top": rng.choice([1, 2, 2, 4]), "experts": rng.choice([8, 8, 16, 32]), "d": d, "ffn": ffn // 2 if d < 2048 else ffn,
                "quant": quant, "group": 32 if quant == "mxfp4" else 64}
    if kind == "step":
        return {"kind": kind, "batch": spread(rng, 1, 64), "layers": rng.randrange(2, 7), "heads": rng.choice([16, 32]), "kv_heads": 8, "ffn": 256 * rng.randrange(16, 57),
                "vocab": spread(rng, 16000, 128256), "ctx": rng.randrange(200, 2049)}
    if kind == "program":
        return {"kind": kind, "m": spread(rng, 1, 512), "d": 128 * rng.randrange(4, 33), "ffn": 128 * rng.randrange(8, 89), "group": rng.choice([32, 64, 128])}
    return {"kind": kind, "k": 128 * rng.randrange(4, 65), "n": spread(rng, 256, 16384) // 2 * 2, "group": rng.choice([32, 64, 128])}


# ---- inputs ------------------------------------------------------------------------------------


def weight(g, lead, n, k, quant, group, tables):
    """Packed codes and tables of `lead` weights: what a program keeps from when it loaded them."""
    bits = 8 if quant == "int8" else 4
    w = torch.randint(-(1 << 31), 1 << 31, (*lead, n, k * bits // 32), generator=g, device=DEV, dtype=torch.int64).to(torch.int32).view(torch.uint32)
    if quant == "mxfp4":
        return w, torch.randint(119, 128, (*lead, n, k // 32), generator=g, device=DEV).to(torch.uint8), None
    s = (torch.rand((*lead, n, k // group), generator=g, device=DEV) * 0.018 + 0.002).to(DTYPES[tables])
    return w, s, (-float(1 << (bits - 1)) * s.float()).to(DTYPES[tables])


def model_weights(g, shape, batch):
    """A model's weights and its sequences' caches. The projections that write into the residual stream
    start out smaller by the root of their number, as models are initialised, so that it does not
    grow with depth (and a rounding is not amplified from layer to layer)."""
    d, hd, narrow = shape.d_model, shape.head_dim, (2 * shape.layers) ** -0.5

    def linear(n, k, by=1.0):
        return llama.quantize_affine4(torch.randn((n, k), generator=g, device=DEV) * (0.02 * by), shape.group_size)

    def layer():
        return {"q": linear(shape.heads * hd, d), "k": linear(shape.kv_heads * hd, d), "v": linear(shape.kv_heads * hd, d), "o": linear(d, shape.heads * hd, narrow),
                "gate": linear(shape.ffn, d), "up": linear(shape.ffn, d), "down": linear(d, shape.ffn, narrow),
                "ln1": 1 + 0.1 * torch.randn(d, generator=g, device=DEV), "ln2": 1 + 0.1 * torch.randn(d, generator=g, device=DEV)}

    def cache():
        return torch.randn((shape.layers, batch, shape.kv_heads, shape.ctx, hd), generator=g, device=DEV, dtype=torch.bfloat16)

    return {"layers": [layer() for _ in range(shape.layers)], "final_norm": torch.ones(d, device=DEV), "lm_head": linear(shape.vocab, d),
            "embedding": torch.randn((shape.vocab, d), generator=g, device=DEV).to(torch.bfloat16), "k_cache": cache(), "v_cache": cache()}


def dense_program(m, d, ffn, group):
    """silu(x Wg) * (x Wu) Wd with the three weights as keras keeps them: int8 codes, a scale and a zero per group."""
    lines, args, count = [], [f"%arg0: tensor<{m}x{d}xbf16>"], [0]

    def op(text, *types):
        name = f"%{count[0]}"
        count[0] += 1
        lines.append(f"    {name} = stablehlo.{text.format(*types)}")
        return name

    def dense(x, rows, k, n):
        i = len(args)
        full, small, wide = f"tensor<{n}x{k}xbf16>", f"tensor<{n}x{k // group}xbf16>", f"tensor<{n}x{k // group}x{group}xbf16>"
        args.extend([f"%arg{i}: tensor<{n}x{k}xi8>", f"%arg{i + 1}: {small}", f"%arg{i + 2}: {small}"])

        def spread_out(arg):
            b = op(f"broadcast_in_dim %arg{arg}, dims = [0, 1] : ({small}) -> {wide}")
            return op(f"reshape {b} : ({wide}) -> {full}")

        c = op(f"convert %arg{i} : (tensor<{n}x{k}xi8>) -> {full}")
        c = op(f"subtract {c}, {spread_out(i + 2)} : {full}")
        c = op(f"multiply {c}, {spread_out(i + 1)} : {full}")
        return op(f"dot_general {x}, {c}, contracting_dims = [1] x [1] : (tensor<{rows}x{k}xbf16>, {full}) -> tensor<{rows}x{n}xbf16>")

    mid = f"tensor<{m}x{ffn}xbf16>"
    gate, up = dense("%arg0", m, d, ffn), dense("%arg0", m, d, ffn)
    act = op(f"multiply {gate}, {op(f'logistic {gate} : {mid}')} : {mid}")
    act = op(f"multiply {act}, {up} : {mid}")
    down = dense(act, m, ffn, d)
    out = f"tensor<{m}x{d}xbf16>"
    return "module @jit_feed_forward {\n  func.func public @main(" + ", ".join(args) + f") -> ({out}) {{\n" + "\n".join(lines) + f"\n    return {down} : {out}\n  }}\n}}\n"


def prepare(case, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    kind = case["kind"]
    if kind == "product":
        m, k, n = case["m"], case["k"], case["n"]
        x = torch.randn((m, k), generator=g, device=DEV).to(DTYPES[case["x"]])
        return {"kind": kind, "x": x, "w": weight(g, (), n, k, case["quant"], case["group"], case["tables"]),
                "how": {"group_size": case["group"], "bits": 8 if case["quant"] == "int8" else 4, "mode": "mxfp4" if case["quant"] == "mxfp4" else "affine"}}
    if kind == "experts":
        t, e, d, f = case["tokens"], case["experts"], case["d"], case["ffn"]
        up = [weight(g, (e,), f, d, case["quant"], case["group"], "bf16") for _ in range(2)]
        down = weight(g, (e,), d, f, case["quant"], case["group"], "bf16")
        x = (torch.randn((t, d), generator=g, device=DEV) * 0.5).to(torch.bfloat16)
        wts, idx = torch.topk(torch.softmax(torch.randn((t, e), generator=g, device=DEV), -1), case["top"], dim=-1)
        return {"kind": kind, "x": x, "idx": idx, "wts": wts / wts.sum(-1, keepdim=True), "w": (*up, down),
                "how": {"group_size": case["group"], "bits": 4, "mode": "mxfp4" if case["quant"] == "mxfp4" else "affine"}}
    if kind == "step":
        shape = llama.Shape(layers=case["layers"], d_model=case["heads"] * 128, heads=case["heads"], kv_heads=case["kv_heads"], head_dim=128, ffn=case["ffn"],
                            vocab=case["vocab"], ctx=case["ctx"])
        step = llama.DecodeStep(shape, case["batch"], DEV, full_weights=model_weights(g, shape, case["batch"]))
        step.capture()
        return {"kind": kind, "step": step, "ids": torch.randint(0, case["vocab"], (case["batch"],), generator=g, device=DEV)}
    if kind == "program":
        m, d, f, group = case["m"], case["d"], case["ffn"], case["group"]
        program = engine.compile_program(dense_program(m, d, f, group).encode())
        arrays = [((torch.randn((m, d), generator=g, device=DEV)).to(torch.bfloat16), 13)]
        for n, k in ((f, d), (f, d), (d, f)):
            arrays.append((torch.randint(-8, 8, (n, k), generator=g, device=DEV, dtype=torch.int8), 2))
            arrays.append(((torch.rand((n, k // group), generator=g, device=DEV) * 0.018 + 0.002).to(torch.bfloat16), 13))
            arrays.append((torch.randint(-3, 4, (n, k // group), generator=g, device=DEV).to(torch.bfloat16), 13))
        buffers = [engine.DeviceBuffer(a, enum) for a, enum in arrays]
        engine.execute(program, buffers)                    # (the weights are packed on a program's first call)
        return {"kind": kind, "program": program, "buffers": buffers}
    n, k, group = case["n"], case["k"], case["group"]
    packed = torch.randint(-128, 128, (k, n // 2), generator=g, device=DEV, dtype=torch.int8)
    scale = (torch.rand((k // group, n), generator=g, device=DEV) * 0.018 + 0.002).to(torch.bfloat16)
    zero = torch.randint(-8, 8, (k // group, n), generator=g, device=DEV, dtype=torch.int8)
    return {"kind": kind, "packed": packed, "scale": scale, "zero": zero}


def run(state):
    kind = state["kind"]
    if kind == "product":
        return qmm.quantized_matmul(state["x"], *state["w"], **state["how"])
    if kind == "experts":
        return moe.moe_experts(state["x"], state["idx"], state["wts"], *state["w"], **state["how"])
    if kind == "step":
        # What a step computes: the logits and the caches with the new position in them. (The next
        # ids are the arg max of the logits; where two of 128256 lie within a rounding of one
        # another either is right.)
        step = state["step"]
        step.tokens.copy_(state["ids"])
        step.replay()
        return {"logits": step.logits_l, "keys": step.k_cache, "values": step.v_cache}
    if kind == "program":
        return [b.data for b in engine.execute(state["program"], state["buffers"])]
    pack = qmm.from_keras_int4(state["packed"], state["scale"], state["zero"])
    return {"w": pack.w.view(torch.int32), "scales": pack.scales, "biases": pack.biases}


# ---- what a pass cannot do without ------------------------------------------------------------------


def weight_bytes(n, k, quant, group, tables="bf16"):
    codes = n * k * (8 if quant == "int8" else 4) // 8
    return codes + n * (k // group) * (1 if quant == "mxfp4" else 2 * BYTES[tables])


def work(case):
    kind = case["kind"]
    if kind == "product":
        m, k, n = case["m"], case["k"], case["n"]
        return {"bytes": weight_bytes(n, k, case["quant"], case["group"], case["tables"]) + m * (k + n) * BYTES[case["x"]], "flops": 2 * m * k * n}
    if kind == "experts":
        t, top, e, d, f = case["tokens"], case["top"], case["experts"], case["d"], case["ffn"]
        met = e * (1.0 - (1.0 - top / e) ** t)              # experts that some token meets, on average
        one = 2 * weight_bytes(f, d, case["quant"], case["group"]) + weight_bytes(d, f, case["quant"], case["group"])
        return {"bytes": met * one + 2 * t * d * 2 + t * top * 12, "flops": 2 * t * top * 3 * d * f}
    if kind == "step":
        b, d, f, hd = case["batch"], case["heads"] * 128, case["ffn"], 128
        layer = [((case["heads"] + 2 * case["kv_heads"]) * hd, d), (d, d), (2 * f, d), (d, f)]
        head = (case["vocab"], d)
        cache = 2 * case["layers"] * b * case["kv_heads"] * case["ctx"] * hd * 2
        weights = case["layers"] * sum(weight_bytes(n, k, "int4", 64) for n, k in layer) + weight_bytes(*head, "int4", 64)
        linear = case["layers"] * sum(n * k for n, k in layer) + head[0] * head[1]
        attention = 2 * case["layers"] * b * case["heads"] * case["ctx"] * hd
        return {"bytes": weights + cache + b * (case["vocab"] + d) * 2, "flops": 2 * b * linear + 2 * attention}
    if kind == "program":
        m, d, f = case["m"], case["d"], case["ffn"]
        return {"bytes": 3 * weight_bytes(f, d, "int4", case["group"]) + 2 * m * d * 2, "flops": 2 * m * 3 * d * f}
    n, k, group = case["n"], case["k"], case["group"]
    return {"bytes": n * k // 2 * 2 + n * (k // group) * (2 + 1 + 8), "flops": n * k}


def tolerance(case):
    """What rounding in the data types gives: the weights' and the results' 16-bit roundings, and in a
    decode step those of every layer's activations on top of one another (0.02 between kernels of this
    package that round at different places). Packing is exact."""
    kind = case["kind"]
    if kind == "product":
        return {"rel": {"bf16": 1e-2, "f16": 2e-3, "f32": 1e-5}[case["x"]]}
    if kind == "step":
        return {"rel": 3e-2}
    if kind == "pack":
        return "exact"
    return {"rel": 1e-2}
