"""The calls whose speed matters to a program that denoises images with this framework, over the sizes it meets.

A MOSS-Image denoising step is one forward of the 42-block quantized DiT (D = 3072, 24 heads; FFN width 8192 in the
published model, 12288 in the benchmark) for one to three rows (conditional, unconditional, skip-layer guidance), each
row `[video tokens | text tokens]`, and the guidance and update arithmetic on the latents after it. Video tokens are the latent grid:
256 for a 256 x 256 image, 1024 for 512 x 512, 4096 for 1024 x 1024, 16384 for 2048 x 2048. The kinds:

  forward    one step through ops.dit_forward (eager, or replayed from the step-graph cache), with the timestep's
             modulation computed the fp32 way (host MLP) or the bf16 way (device)
  prefill    ops.dit_prefill_references: the key / value cache of reference images, once per edit
  blocks     ops.dit_step: the block loop (or its first `depth` blocks) on tokens of the caller's
  attention  ops.attention_q8 on its own (ragged batch of sequences)
  update     ops.guided_velocity_step with an in-place latent update: what a step ends with
"""
import torch

from owoinfer_b200 import ops, synth

D, HEADS, BLOCKS, CHANNELS = 3072, 24, 42, 128
TIERS = {"int8": ops.TIER_INT8, "w4a4": ops.TIER_W4A4_VIA_INT8, "w4a8": ops.TIER_W4A8}


def _forward(height, width, texts, ffn=8192, tier="int8", launch="eager", time="fp32", refs=0):
    """texts: the rows' text lengths, "282,10" (two rows: conditional and unconditional; a third is the row that skips
    blocks for skip-layer guidance). refs: tokens of cached reference images (edits)."""
    return {"kind": "forward", "height": height, "width": width, "texts": texts, "ffn": ffn, "tier": tier, "launch": launch,
            "time": time, "refs": refs}


def listed():
    named = {
        # The end of every step, at the smallest image: one launch on a few hundred KB.
        "update 256x256": {"kind": "update", "height": 16, "width": 16, "skip": False, "order": 1},
        # A thumbnail or preview with guidance, the way a sampling loop should run it: launches replayed from a graph.
        "256x256 cfg graph": _forward(16, 16, "64,10", ffn=12288, launch="graph"),
        # The same size class at an odd aspect, guidance-distilled (one row), launched eagerly.
        "ragged 208x320 eager": _forward(13, 20, "37"),
        # Skip-layer guidance at 512 x 512: three rows, the third skips a few blocks, so blocks run on different row sets.
        "512x512 slg eager": _forward(32, 32, "141,10,141", time="bf16"),
        # The grouped 4-bit tier at 512 x 512.
        "512x512 cfg w4a8": _forward(32, 32, "282,10", ffn=12288, tier="w4a8"),
        # The published model's everyday step: 1024 x 1024, a prompt of 282 tokens, an empty negative prompt.
        "1024x1024 cfg": _forward(64, 64, "282,10"),
        # One block of the published files' 4-bit turbo tier at the same size, as a host that sequences blocks itself calls it.
        "w4a4 block 8484": {"kind": "blocks", "lengths": "4378,4106", "ffn": 8192, "tier": "w4a4", "depth": 1},
        # The benchmark's step: the block loop on two sequences of 4096 image + 4096 text tokens, FFN width 12288.
        "8192 tokens x 2": {"kind": "blocks", "lengths": "8192,8192", "ffn": 12288, "tier": "int8", "depth": BLOCKS},
        # An edit with one 1024 x 1024 reference image: its cache once per image, then every step attends to it.
        "prefill 1024x1024": {"kind": "prefill", "height": 64, "width": 64, "images": 1, "ffn": 8192, "tier": "int8"},
        "1024x1024 edit": _forward(64, 64, "282,10", refs=4096, time="bf16"),
        # Attention called on its own by a host that owns its QKV: ragged sequences, the high tier's default variant.
        "attention ragged": {"kind": "attention", "lengths": "1039,777,2500,64", "variant": "int8_fp8"},
        # The largest: a 2048 x 2048 image with 4096 text tokens in one guidance-distilled row.
        "2048x2048 one row": _forward(128, 128, "4096", ffn=12288),
    }
    return [dict(case, name=name) for name, case in named.items()]


def draw(rng):
    limit = max(_cost(c) for c in listed())
    while True:
        case = _draw_one(rng)
        if _cost(case) <= limit:
            return case


def _draw_one(rng):
    def log_int(lo, hi):
        return int(round(lo * (hi / lo) ** rng.random()))

    kind = rng.choices(["forward", "blocks", "prefill", "attention", "update"], [12, 2, 2, 2, 1])[0]
    height, width = log_int(10, 136), log_int(10, 136)
    ffn, tier = rng.choice([8192, 12288]), rng.choices(["int8", "w4a8"], [3, 1])[0]
    if kind == "forward":
        refs = rng.choice([0, 0, 0, log_int(200, 6000)])
        rows = rng.choice([1, 2, 2] if refs else [1, 2, 2, 3])
        texts = ",".join(str(log_int(5, 700)) for _ in range(rows))
        return _forward(height, width, texts, ffn, tier, rng.choice(["graph", "eager"]), rng.choice(["fp32", "bf16"]), refs)
    if kind == "blocks":
        lengths = ",".join(str(log_int(200, 12000)) for _ in range(rng.choice([1, 2, 3])))
        if rng.random() < 0.5:
            return {"kind": kind, "lengths": lengths, "ffn": ffn, "tier": "w4a4", "depth": 1}
        return {"kind": kind, "lengths": lengths, "ffn": ffn, "tier": tier, "depth": BLOCKS}
    if kind == "prefill":
        return {"kind": kind, "height": min(height, 80), "width": min(width, 80), "images": rng.choice([1, 1, 2]), "ffn": ffn, "tier": tier}
    if kind == "attention":
        lengths = ",".join(str(log_int(33, 9000)) for _ in range(rng.choice([1, 2, 3, 4])))
        return {"kind": kind, "lengths": lengths, "variant": rng.choice(["int8_fp8", "int8_fp8_f32acc"])}
    return {"kind": kind, "height": height, "width": width, "skip": rng.random() < 0.5, "order": rng.choice([1, 2])}


# ---------------------------------------------------------------------------------------------------- inputs

def _normal(shape, seed, std=1.0, dtype=torch.float32):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return (std * torch.randn(shape, generator=g, device="cuda", dtype=torch.float32)).to(dtype)


def _lens(text):
    return [int(n) for n in text.split(",")]


def _blocks(case, seed):
    blocks, keep = [], []
    for i in range(case.get("depth", BLOCKS)):
        w = synth.block_weights(D, case["ffn"], seed + 100 * i, tier=TIERS[case["tier"]])
        lin = {n: ops.make_w4(w[n][0], w[n][1], 64, w[n][2]) if case["tier"] == "w4a8" else w[n] for n in ("qkv", "o", "up_gate", "down")}
        blocks.append(ops.BlockWeights(w["norm1"], w["norm2"], w["q_norm"], w["k_norm"], lin["qkv"], lin["o"], lin["up_gate"], lin["down"]))
        keep.append(w)
    return blocks, keep


def _model(case, seed):
    """The whole model as a program holds it after loading: blocks, modulation, embedder, head, and the timestep MLP."""
    bf = torch.bfloat16
    blocks, keep = _blocks(case, seed)
    seed += 50000  # past the blocks' seeds
    # The residual stream of a trained model has a few channels far above the rest (1 % of them at 20 here, as in synth).
    video_bias = _normal(D, seed + 6, 0.1)
    video_bias[torch.randperm(D, generator=torch.Generator().manual_seed(seed))[:D // 100].cuda()] += 20.0
    shell = dict(block_mod_w=_normal((6 * D, D), seed + 1, 0.002, bf), block_mod_bias=_normal(6 * D, seed + 2, 0.1),
                 head_mod_w=_normal((2 * D, D), seed + 3, 0.002, bf), head_mod_bias=_normal(2 * D, seed + 4, 0.1),
                 video_w=_normal((D, CHANNELS), seed + 5, 0.09, bf), video_bias=video_bias.to(bf),
                 final_norm=synth.vector(D, seed + 7, 0.1, 1.0), final_w=_normal((CHANNELS, D), seed + 8, 0.02, bf),
                 final_bias=_normal(CHANNELS, seed + 9, 0.1, bf))
    s = {"model": ops.DitModel(blocks, case["ffn"], **shell), "keep": (keep, shell)}
    mlp = [_normal((D, 256), seed + 10, 0.06), _normal(D, seed + 11, 0.1), _normal((D, D), seed + 12, 0.02), _normal(D, seed + 13, 0.1)]
    if case.get("time", "fp32") == "fp32":
        s["mlp"] = [t.cpu().numpy() for t in mlp]
    else:
        s["mlp"] = [t.to(bf) for t in mlp] + [shell["block_mod_w"], shell["block_mod_bias"].to(bf), shell["head_mod_w"], shell["head_mod_bias"].to(bf)]
    return s


def prepare(case, seed):
    seed = (seed % (1 << 30)) * 100003 + 17
    return {"forward": _prepare_forward, "prefill": _prepare_prefill, "blocks": _prepare_blocks, "attention": _prepare_attention,
            "update": _prepare_update}[case["kind"]](case, seed)


def _skip_mask(row):
    return sum(1 << b for b in (6, 7, 8, 20)) if row == 2 else 0


def _prepare_forward(case, seed):
    s = _model(case, seed)
    seed += 60000
    texts = [synth.activations(n, D, seed + 1 + r) for r, n in enumerate(_lens(case["texts"]))]
    shape = (1, CHANNELS, case["height"], case["width"])
    s.update(case=case, t=0.05 + (seed % 9973) / 11000, latents=_normal(shape, seed + 4), outs=[torch.empty(shape[1:], device="cuda") for _ in texts],
             rows=[(x, _skip_mask(r), 0) for r, x in enumerate(texts)], workspace=None, kv=None)
    if case["refs"]:
        # k | v rows of every block, as a prefill leaves them: normalised keys, values of the same order.
        s["kv"] = _normal((BLOCKS, case["refs"], 2 * D), seed + 9, 1.0, torch.bfloat16)
    s["graphs"] = ops.DitGraphs() if case["launch"] == "graph" else None
    s["stream"] = torch.cuda.Stream() if case["launch"] == "graph" else None
    return s


def _prepare_prefill(case, seed):
    s = _model(case, seed)
    seed += 60000
    s.update(case=case, images=[_normal((CHANNELS, case["height"], case["width"]), seed + 4 + i) for i in range(case["images"])])
    return s


def _prepare_blocks(case, seed):
    lens = _lens(case["lengths"])
    total = sum(lens)
    blocks, keep = _blocks(case, seed)
    x0 = synth.activations(total, D, seed + 1)
    rope = torch.cat([ops.moss_rope_table(n // 64, 32, n - n // 64 * 32) for n in lens]).contiguous()
    run = ops.block_run(total, synth.cu_seqlens(lens), max(lens), D=D, F=case["ffn"], heads=HEADS, tier=TIERS[case["tier"]])
    workspace = torch.empty(ops.block_quant_workspace_bytes(run), dtype=torch.uint8, device="cuda")
    x = torch.empty_like(x0)
    return {"case": case, "blocks": blocks, "keep": keep, "x0": x0, "x": x, "run": run,
            "buffers": ops.block_buffers(x, synth.modulation(D, seed + 2), rope, workspace)}


def _prepare_attention(case, seed):
    lens = _lens(case["lengths"])
    total = sum(lens)
    qkv = synth.activations(total, 3 * D, seed + 1)
    rope = torch.cat([ops.moss_rope_table(n // 64, 32, n - n // 64 * 32) for n in lens]).contiguous()
    # The columns of a fused QKV projection with QK-norm and RoPE behind them.
    ops.qk_norm_rope_moss(qkv, HEADS, synth.vector(128, seed + 2, 0.1, 1.0), synth.vector(128, seed + 3, 0.1, 1.0), rope)
    q, k, v = (qkv[:, i * D:(i + 1) * D].unflatten(1, (HEADS, 128)) for i in range(3))
    options = ops.attention_options(variant=ops.ATTENTION_Q8_FP8 if case["variant"] == "int8_fp8" else ops.ATTENTION_Q8_FP8_F32ACC)
    need = ops.attention_q8_workspace_bytes(total, total, len(lens), max(lens), HEADS, options=options)
    return {"case": case, "q": q, "k": k, "v": v, "out": torch.empty((total, HEADS, 128), dtype=torch.bfloat16, device="cuda"),
            "cu": synth.cu_seqlens(lens), "longest": max(lens), "options": options, "workspace": torch.empty(need, dtype=torch.uint8, device="cuda")}


def _prepare_update(case, seed):
    shape = (CHANNELS, case["height"], case["width"])
    v = {n: _normal(shape, seed + i) for i, n in enumerate(("x", "v_cond", "v_uncond", "v_skip", "v_prev"))}
    if not case["skip"]:
        v["v_skip"] = None
    if case["order"] == 1:
        v["v_prev"] = None
    v["v_out"] = torch.empty(shape, device="cuda") if case["order"] == 2 else None  # the next step's v_prev
    return {"case": case, "vectors": v}


# ---------------------------------------------------------------------------------------------------- one pass

def run(s):
    kind = s["case"]["kind"]
    if kind == "forward":
        if s["stream"] is None:
            return _step(s)
        with torch.cuda.stream(s["stream"]):
            return _step(s)
    if kind == "prefill":
        return ops.dit_prefill_references(s["model"], s["images"], ops.time_vector_fp32(*s["mlp"], 0.0), tier=TIERS[s["case"]["tier"]])
    if kind == "blocks":
        s["x"].copy_(s["x0"])  # the loop works in place: every step starts from its own tokens
        ops.dit_step(s["blocks"], s["buffers"], s["run"])
        return s["x"]
    if kind == "attention":
        out, _ = ops.attention_q8(s["q"], s["k"], s["v"], s["out"], s["cu"], s["cu"], s["longest"], ops.SM_SCALE,
                                  workspace=s["workspace"], options=s["options"])
        return out
    v = s["vectors"]
    order = s["case"]["order"]
    x = ops.guided_velocity_step(v["v_cond"], x=v["x"], v_uncond=v["v_uncond"], v_skip=v["v_skip"], v_prev=v["v_prev"], v_out=v["v_out"],
                                 cfg_scale=4.0, slg_scale=2.5 if v["v_skip"] is not None else 0.0, h=-0.001, a=1.5, b=0.5, update=order)
    return [x, v["v_out"]]


def _step(s):
    time_vector = mod = head = None
    if s["case"]["time"] == "fp32":
        time_vector = ops.time_vector_fp32(*s["mlp"], s["t"])
    else:
        mod, head = ops.time_modulation_bf16(*s["mlp"], s["t"])
    outs, s["workspace"] = ops.dit_forward(s["model"], s["latents"], time_vector, s["rows"], tier=TIERS[s["case"]["tier"]],
                                           workspace=s["workspace"], ref_kv=s["kv"], graphs=s["graphs"], outs=s["outs"], mod=mod, head=head)
    return outs


# ---------------------------------------------------------------------------------------------------- work and tolerance

def _weight_bytes(case):
    per, rows = 4 * D * D + 3 * D * case["ffn"], 3 * D + D + 2 * case["ffn"] + D
    return per * {"int8": 1.0, "w4a4": 0.5, "w4a8": 0.5 + 1 / 64}[case["tier"]] + 4 * rows


def _block_flops(case, lens, keys):
    return 2 * sum(lens) * (4 * D * D + 3 * D * case["ffn"]) + sum(4 * q * k * D for q, k in zip(lens, keys))


def work(case):
    kind = case["kind"]
    if kind == "update":
        n = CHANNELS * case["height"] * case["width"]
        streams = 4 + case["skip"] + 2 * (case["order"] == 2)
        return {"bytes": 4 * n * streams, "flops": n * (5 + 3 * case["skip"] + 2 * (case["order"] == 2))}
    if kind == "attention":
        lens = _lens(case["lengths"])
        return {"bytes": 4 * 2 * D * sum(lens), "flops": sum(4 * n * n * D for n in lens)}
    if kind == "blocks":
        lens = _lens(case["lengths"])
        return {"bytes": case["depth"] * _weight_bytes(case) + 2 * 2 * D * sum(lens), "flops": case["depth"] * _block_flops(case, lens, lens)}
    hw = case["height"] * case["width"]
    shell = 2 * 8 * D * D + 2 * CHANNELS * D * 2  # modulation linears, embedder, head (bf16)
    if kind == "prefill":
        n = hw * case["images"]
        full = _block_flops(case, [n], [n])
        return {"bytes": BLOCKS * (_weight_bytes(case) + 2 * 2 * D * n) + shell + 4 * CHANNELS * n,
                "flops": (BLOCKS - 1) * full + 2 * n * 3 * D * D + 2 * n * CHANNELS * D}
    lens = [hw + n for n in _lens(case["texts"])]
    flops = 0
    for b in range(BLOCKS):
        on = [n for r, n in enumerate(lens) if not (_skip_mask(r) >> b) & 1]
        flops += _block_flops(case, on, [n + case["refs"] for n in on])
    latents = 4 * CHANNELS * hw * (1 + len(lens))
    return {"bytes": BLOCKS * (_weight_bytes(case) + 2 * 2 * D * case["refs"]) + shell + 2 * D * sum(_lens(case["texts"])) + latents,
            "flops": flops + 2 * hw * CHANNELS * D * (1 + len(lens))}


def _cost(case):
    """Rough seconds of a pass, for draw(): the larger of its operations and its bytes."""
    w = work(case)
    return max(w["flops"] / 2e15, w["bytes"] / 5e12)


def tolerance(case):
    if case["kind"] == "update":
        return {"rel": 1e-6}  # a handful of fp32 operations per element
    if case["kind"] == "attention":
        # P and V in e4m3 (three mantissa bits: 2.6 % rms per product): where P is rounded depends on the reference maximum.
        return {"rel": 0.03}
    # Activations are rounded to INT8 (INT4) four times per block: wherever P is rounded the other way, codes flip behind it,
    # and two equally exact forms are 1.4 to 1.7 % apart after 42 blocks (0.8 % after the one 4-bit block).
    return {"rel": 0.02}
