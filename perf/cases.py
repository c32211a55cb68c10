"""The work a user of this library has it do, as a list of measurable cases.

Every case goes through the public entry points a program would call: the torch custom classes (the FLUX blocks and the whole
transformer), the layer objects of lyradiff_b200.layers (one quantized linear each), and the functions of lyradiff_b200.ops
where a program strings the kernels together itself (the SDXL feed-forward block, the modulated LayerNorm in front of a linear,
the re-quantize of a LoRA swap).  Inputs are random with the distributions of the benchmark: activations N(0, 1), weights
N(0, 0.02), static activation scales of the size a calibration gives, QK norm weights around one, the rotary table of an image.

A case is a dict of plain values; "kind" picks the path, the rest are sizes and options:

  linear_fp8     Fp8Linear.forward                      m, n, k, gelu, residual, dtype
  linear_int8    SmoothQuantLinear.forward              m, n, k, dynamic, dtype
  linear_w4a4    W4A4Gemm.forward with its LoRA branch  m, n, k, gelu, dtype
  ff_int8        LayerNorm -> INT8 linear -> GEGLU -> INT8 linear + residual    rows, dim, dtype
  adaln          AdaLN modulation with quantized outputs                        batch, seq, dim, outputs, dtype
  lora_swap      merge of a low-rank update into a 16-bit weight, re-quantize   n, k, dtype
  single_block   FluxSingleTransformerBlockOp.forward   batch, tokens, level, dtype
  double_block   FluxTransformerBlockOp.forward         batch, text, height, width, level, dtype
  forward        FluxTransformer2DModelOp.transformer_forward     doubles, singles, text, height, width, level, dtype

height and width count the 16 x 16-pixel patches of the image, so 64 x 64 is a 1024 x 1024 image (4096 tokens).
"""

import torch

from lyradiff_b200 import layers, ops, rope, torch_classes

HIDDEN, HEADS, HEAD_DIM = 3072, 24, 128
IN_CHANNELS, JOINT, POOLED = 64, 4096, 768
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}
ACT_SCALE = 0.03          # static e4m3 input scale of the FLUX linears
MOD_STD = 0.0015          # weights of the modulation linears: gates of 0.05 to 0.1, so a block of a deep stack moves its stream a little
W4A4_LEVELS = (7, 8)


def listed():
    return [
        # The modulation linear of a block at quant_level 2: one conditioning vector, 28 MB of weights.  The smallest call there
        # is: launches, latency and the weight stream, nothing else.
        {"name": "linear_fp8_one_row", "kind": "linear_fp8", "m": 1, "n": 9216, "k": 3072, "gelu": False, "residual": False,
         "dtype": "bf16"},
        # The feed-forward output linear over an odd number of tokens (an image that is no multiple of a tile), deep K, residual.
        {"name": "linear_fp8_ragged", "kind": "linear_fp8", "m": 1317, "n": 3072, "k": 12288, "gelu": False, "residual": True,
         "dtype": "fp16"},
        # The GEGLU projection of the SDXL feed-forward with a dynamic per-token scale: two 1024 x 1024 latents at the 640 level.
        {"name": "linear_int8_sdxl", "kind": "linear_int8", "m": 8192, "n": 5120, "k": 640, "dynamic": True, "dtype": "fp16"},
        # The whole SDXL feed-forward block in INT8 at that level, static calibrated scales.
        {"name": "ff_int8_sdxl", "kind": "ff_int8", "rows": 8192, "dim": 640, "dtype": "fp16"},
        # The MLP projection of a FLUX block in W4A4 with its rank-32 LoRA branch, 1024 x 1024 image.
        {"name": "linear_w4a4_mlp", "kind": "linear_w4a4", "m": 4608, "n": 12288, "k": 3072, "gelu": True, "dtype": "bf16"},
        # AdaLN in front of an INT8 and an FP8 consumer: a pure memory pass over the tokens of a 1024 x 1024 image.
        {"name": "adaln_int8_e4m3", "kind": "adaln", "batch": 1, "seq": 4608, "dim": 3072, "outputs": "int8+e4m3", "dtype": "bf16"},
        # A LoRA swap on the largest square-ish weight of a block: merge in 16 bits, new scale, new e4m3 codes.
        {"name": "lora_swap_mlp", "kind": "lora_swap", "n": 12288, "k": 3072, "dtype": "bf16"},
        # The single-stream block in FP8 at 1024 x 1024: two thirds of a FLUX denoising step are this call.
        {"name": "single_fp8_1024px", "kind": "single_block", "batch": 1, "tokens": 4608, "level": 1, "dtype": "bf16"},
        # The double-stream block in FP8 at 1024 x 1024: the other third.
        {"name": "double_fp8_1024px", "kind": "double_block", "batch": 1, "text": 512, "height": 64, "width": 64, "level": 1,
         "dtype": "bf16"},
        # The double-stream block on a small image of odd proportions (560 x 528 pixels): few tiles per GEMM, ragged rows.
        {"name": "double_fp8_small", "kind": "double_block", "batch": 1, "text": 512, "height": 35, "width": 33, "level": 1,
         "dtype": "bf16"},
        # The single-stream block in W4A4 at 1024 x 1024.
        {"name": "single_int4_1024px", "kind": "single_block", "batch": 1, "tokens": 4608, "level": 7, "dtype": "bf16"},
        # A whole denoising step at 1024 x 1024 with two double-stream and four single-stream blocks (the model's one to two):
        # embedders, modulations issued ahead on a second stream, blocks, output layer.  The largest case.
        {"name": "forward_1024px", "kind": "forward", "doubles": 2, "singles": 4, "text": 512, "height": 64, "width": 64, "level": 1,
         "dtype": "bf16"},
    ]


FLUX_LINEARS = ((9216, 3072), (3072, 3072), (12288, 3072), (3072, 12288), (3072, 15360), (18432, 3072))
SDXL_LINEARS = ((640, 640), (5120, 640), (640, 2560), (1280, 1280), (10240, 1280), (1280, 5120), (640, 2048), (1280, 2048))


def _log(rng, lo, hi):
    return min(hi, max(lo, int(round(lo * (hi / lo) ** rng.random()))))


def _image(rng, most=4096):
    height = rng.randint(12, 80)
    return height, rng.randint(12, max(12, min(80, most // height)))


def draw(rng):
    kind = rng.choice(["linear_fp8", "linear_int8", "linear_w4a4", "ff_int8", "adaln", "lora_swap", "single_block", "double_block", "forward"])
    dtype = rng.choice(["bf16", "bf16", "fp16"])
    c = {"kind": kind}
    if kind == "linear_fp8":
        n, k = rng.choice(FLUX_LINEARS) if rng.random() < 0.6 else (64 * _log(rng, 4, 240), 64 * _log(rng, 4, 240))
        c.update(m=_log(rng, 1, 8192), n=n, k=k, gelu=rng.random() < 0.4, residual=rng.random() < 0.4)
    elif kind == "linear_int8":
        n, k = rng.choice(SDXL_LINEARS)
        c.update(m=_log(rng, 77, 16384), n=n, k=k, dynamic=rng.random() < 0.6)
        dtype = rng.choice(["fp16", "fp16", "bf16"])
    elif kind == "linear_w4a4":
        n, k = rng.choice(FLUX_LINEARS[:4] + ((21504, 3072),))
        c.update(m=_log(rng, 64, 8192), n=n, k=k, gelu=rng.random() < 0.4)
    elif kind == "ff_int8":
        c.update(rows=_log(rng, 128, 16384), dim=rng.choice([640, 1280]))
        dtype = rng.choice(["fp16", "fp16", "bf16"])
    elif kind == "adaln":
        c.update(batch=rng.randint(1, 4), seq=_log(rng, 64, 4608), dim=rng.choice([3072, 3072, 3072, 1536, 2432, 1152, 4096]),
                 outputs=rng.choice(["int8+e4m3", "int8", "e4m3", "16bit"]))
    elif kind == "lora_swap":
        n, k = rng.choice(FLUX_LINEARS) if rng.random() < 0.5 else (64 * _log(rng, 4, 240), 64 * _log(rng, 4, 240))
        c.update(n=n, k=k)
    elif kind == "single_block":
        batch = rng.choice([1, 1, 2, 3])
        c.update(batch=batch, tokens=_log(rng, 160, 4608 // batch), level=rng.choice([1, 1, 2, 7, 8]))
    elif kind == "double_block":
        batch = rng.choice([1, 1, 2])
        height, width = _image(rng, 4096 // batch)
        c.update(batch=batch, text=rng.choice([512, 512, 256, 77]), height=height, width=width, level=rng.choice([1, 1, 2, 7, 8]))
    else:
        height, width = _image(rng)
        c.update(doubles=rng.randint(1, 2), singles=rng.randint(1, 3), text=rng.choice([512, 256]), height=height, width=width,
                 level=rng.choice([1, 1, 2]))
    c["dtype"] = dtype
    return c


# ---------------------------------------------------------------------------------------------- inputs
class _Random:
    """Seeded tensors on the GPU."""

    def __init__(self, seed, dtype):
        self.gen = torch.Generator(device="cuda").manual_seed(seed)
        self.dtype = dtype

    def normal(self, *shape, std=1.0, mean=0.0, dtype=None):
        x = torch.randn(*shape, generator=self.gen, device="cuda")
        return (x * std + mean).to(dtype or self.dtype)

    def uniform(self, lo, hi, *shape, dtype=None):
        x = torch.rand(*shape, generator=self.gen, device="cuda")
        return (x * (hi - lo) + lo).to(dtype or self.dtype)


def _fp8_linear_dict(r, sd, name, n, k, quantized=True, std=0.02):
    sd[name + ".weight"] = r.normal(n, k, std=std)
    sd[name + ".bias"] = r.normal(n, std=0.02)
    if quantized:
        sd[name + "_input_scale"] = torch.tensor([ACT_SCALE])


def _w4a4_linear_dict(r, sd, name, n, k, bias=True):
    w = r.normal(n, k, std=0.02)
    sd[name + "packed_weight"] = torch.empty(n, k // 2, dtype=torch.uint8, device="cuda")
    sd[name + "weight_scale"] = torch.empty(n, k // 64, dtype=torch.float32, device="cuda")
    ops.weight_quant_int4_g64(sd[name + "packed_weight"], sd[name + "weight_scale"], w)
    sd[name + "smooth"] = r.uniform(0.5, 1.5, k, dtype=torch.float32)
    sd[name + "lora_down"] = r.normal(32, k, std=0.02)
    sd[name + "lora_up"] = r.normal(n, 32, std=0.02)
    if bias:
        sd[name + "bias"] = r.normal(n, std=0.02)


def _qk_norms(r, sd, names):
    for name in names:
        sd[name + ".weight"] = r.uniform(0.8, 1.6, HEAD_DIM)


def _single_dict(r, sd, prefix, level):
    D = HIDDEN
    _fp8_linear_dict(r, sd, prefix + "norm.linear", 3 * D, D, quantized=level in (2, 8), std=MOD_STD)
    _qk_norms(r, sd, (prefix + "attn.norm_q", prefix + "attn.norm_k"))
    if level in W4A4_LEVELS:
        _w4a4_linear_dict(r, sd, prefix + "attn.to_qkv.", 3 * D, D)
        _w4a4_linear_dict(r, sd, prefix + "proj_mlp.", 4 * D, D)
        _w4a4_linear_dict(r, sd, prefix + "proj_out.linears.0.", D, D)
        _w4a4_linear_dict(r, sd, prefix + "proj_out.linears.1.linear.", D, 4 * D, bias=False)
    else:
        _fp8_linear_dict(r, sd, prefix + "attn.to_qkv", 3 * D, D)
        _fp8_linear_dict(r, sd, prefix + "proj_mlp", 4 * D, D)
        _fp8_linear_dict(r, sd, prefix + "proj_out", D, 5 * D)


def _double_dict(r, sd, prefix, level):
    D = HIDDEN
    for norm, qkv, out, ff in (("norm1", "attn.to_qkv", "attn.to_out.0", "ff"),
                               ("norm1_context", "attn.to_added_qkv", "attn.to_add_out", "ff_context")):
        _fp8_linear_dict(r, sd, prefix + norm + ".linear", 6 * D, D, quantized=level in (2, 8), std=MOD_STD)
        if level in W4A4_LEVELS:
            _w4a4_linear_dict(r, sd, prefix + qkv + ".", 3 * D, D)
            _w4a4_linear_dict(r, sd, prefix + out + ".", D, D)
            _w4a4_linear_dict(r, sd, prefix + ff + ".net.0.proj.", 4 * D, D)
        else:
            _fp8_linear_dict(r, sd, prefix + qkv, 3 * D, D)
            _fp8_linear_dict(r, sd, prefix + out, D, D)
            _fp8_linear_dict(r, sd, prefix + ff + ".net.0.proj", 4 * D, D)
        _fp8_linear_dict(r, sd, prefix + ff + ".net.2", D, 4 * D)
    _qk_norms(r, sd, [prefix + "attn." + n for n in ("norm_q", "norm_k", "norm_added_q", "norm_added_k")])


def _rope(batch, text, height, width, dtype):
    ids = rope.flux_position_ids(text, height, width, batch=batch, device="cuda")
    return rope.flux_rope_table(ids)[:, 0].to(dtype).contiguous()


def _load_block(op_class, case, sd):
    ns = torch_classes.load()
    op = getattr(ns, op_class)(case["dtype"], HIDDEN, HEADS, HEAD_DIM, 4 if "Single" in op_class else 6, case["level"])
    op.initialize(ns.LyraDiffCommonContext())
    op.reload_model_from_state_dict("", sd, "cuda")
    return op


def _smoothing(r, k):
    """A SmoothQuant vector as calibration leaves it: most channels near one, the outlier channels divided by their size."""
    pre = r.uniform(0.5, 1.5, k, dtype=torch.float32)
    outliers = torch.randperm(k, generator=r.gen, device="cuda")[:max(1, k // 20)]
    pre[outliers] /= 20.0
    return pre, outliers


def prepare(case, seed):
    dtype = DTYPES[case["dtype"]]
    r = _Random(seed, dtype)
    kind, s = case["kind"], {"kind": case["kind"]}
    if kind == "linear_fp8":
        m, n, k = case["m"], case["n"], case["k"]
        scale = torch.full((1,), 4.5 / 448.0 if m > 1 else ACT_SCALE, device="cuda")
        s["layer"] = layers.Fp8Linear(r.normal(n, k, std=0.02), r.normal(n, std=0.02), scale, gelu=case["gelu"])
        s["x"] = r.normal(m, k)
        s["residual"] = r.normal(m, n) if case["residual"] else None
    elif kind == "linear_int8":
        m, n, k = case["m"], case["n"], case["k"]
        pre, outliers = _smoothing(r, k)
        scale = None if case["dynamic"] else torch.full((1,), 5.0 / 127.0, device="cuda")
        s["layer"] = layers.SmoothQuantLinear.from_float(r.normal(n, k, std=0.02), pre, r.normal(n, std=0.02), scale)
        s["x"] = r.normal(m, k)
        s["x"][:, outliers] *= 20.0
    elif kind == "linear_w4a4":
        m, n, k = case["m"], case["n"], case["k"]
        s["layer"] = layers.W4A4Gemm.from_float(r.normal(n, k, std=0.02), r.uniform(0.5, 1.5, k, dtype=torch.float32), r.normal(n, std=0.02),
                                                gelu=case["gelu"], lora_down=r.normal(32, k, std=0.02), lora_up=r.normal(n, 32, std=0.02))
        s["x"] = r.normal(m, k)
    elif kind == "ff_int8":
        rows, dim = case["rows"], case["dim"]
        hidden = 4 * dim
        s["x"] = r.normal(rows, dim)
        s["gamma"], s["beta"] = r.normal(dim, std=0.1, mean=1.0), r.normal(dim, std=0.1)
        s["pre1"], _ = _smoothing(r, dim)
        s["pre2"], _ = _smoothing(r, hidden)
        for name, n, k in (("1", 2 * hidden, dim), ("2", dim, hidden)):
            s["qw" + name] = torch.empty(n, k, dtype=torch.int8, device="cuda")
            s["sw" + name] = torch.empty(n, dtype=torch.float32, device="cuda")
            ops.invoke_get_int8_weight_scale(s["sw" + name], s["qw" + name], r.normal(n, k, std=0.02), s["pre" + name])
            s["b" + name] = r.normal(n, std=0.02)
        s["scale1"] = torch.full((1,), 6.0 / 127.0, device="cuda")
        s["scale2"] = torch.full((1,), 3.0 / 127.0, device="cuda")
    elif kind == "adaln":
        batch, seq, dim = case["batch"], case["seq"], case["dim"]
        s["x"] = r.normal(batch, seq, dim)
        s["scale"], s["shift"] = r.normal(batch, dim, std=0.1), r.normal(batch, dim, std=0.1)
        s["f8_scale"] = torch.full((1,), 6.0 / 448.0, device="cuda")
        s["outputs"] = case["outputs"]
    elif kind == "lora_swap":
        n, k = case["n"], case["k"]
        s["base"] = r.normal(n, k, std=0.02)
        s["update"] = r.normal(n, k, std=0.004)
    elif kind == "single_block":
        batch, tokens, level = case["batch"], case["tokens"], case["level"]
        sd = {}
        _single_dict(r, sd, "", level)
        s["op"] = _load_block("FluxSingleTransformerBlockOp", case, sd)
        s["x"] = r.normal(batch, tokens, HIDDEN)
        s["temb"] = torch.nn.functional.silu(r.normal(batch, HIDDEN))
        text = min(512, tokens // 2)
        s["rope"] = _rope(batch, text, 1, tokens - text, dtype)
    elif kind == "double_block":
        batch, text, height, width = case["batch"], case["text"], case["height"], case["width"]
        sd = {}
        _double_dict(r, sd, "", case["level"])
        s["op"] = _load_block("FluxTransformerBlockOp", case, sd)
        s["x"] = r.normal(batch, height * width, HIDDEN)
        s["context"] = r.normal(batch, text, HIDDEN)
        s["temb"] = torch.nn.functional.silu(r.normal(batch, HIDDEN))
        s["rope"] = _rope(batch, text, height, width, dtype)
    elif kind == "forward":
        D, sd = HIDDEN, {}
        for i in range(case["doubles"]):
            _double_dict(r, sd, "transformer_blocks.%d." % i, case["level"])
        for i in range(case["singles"]):
            _single_dict(r, sd, "single_transformer_blocks.%d." % i, case["level"])
        for name, n, k, std in (("x_embedder", D, IN_CHANNELS, 0.12), ("context_embedder", D, JOINT, 0.015), ("proj_out", IN_CHANNELS, D, 0.02),
                                ("norm_out.linear", 2 * D, D, MOD_STD)):   # both streams enter the blocks with values around one
            _fp8_linear_dict(r, sd, name, n, k, quantized=False, std=std)
        for name, k in (("timestep_embedder", 256), ("guidance_embedder", 256), ("text_embedder", POOLED)):
            _fp8_linear_dict(r, sd, "time_text_embed.%s.linear_1" % name, D, k, quantized=False, std=0.06)
            _fp8_linear_dict(r, sd, "time_text_embed.%s.linear_2" % name, D, D, quantized=False, std=0.03)
        ns = torch_classes.load()
        s["op"] = ns.FluxTransformer2DModelOp(case["dtype"], IN_CHANNELS, case["doubles"], case["singles"], HEAD_DIM, HEADS, POOLED,
                                              JOINT, True, case["level"])
        s["op"].initialize(ns.LyraDiffCommonContext())
        s["op"].reload_transformer_model_from_state_dict(sd, "cuda")
        s["latents"] = r.normal(1, case["height"] * case["width"], IN_CHANNELS)
        s["context"] = r.normal(1, case["text"], JOINT)
        s["pooled"] = r.normal(1, POOLED)
        s["rope"] = _rope(1, case["text"], case["height"], case["width"], dtype)
    else:
        raise ValueError(kind)
    return s


# ---------------------------------------------------------------------------------------------- one pass
def run(s):
    kind = s["kind"]
    if kind == "linear_fp8":
        return s["layer"].forward(s["x"], residual=s["residual"])
    if kind in ("linear_int8", "linear_w4a4"):
        return s["layer"].forward(s["x"])
    if kind == "ff_int8":
        x = s["x"]
        rows, dim = x.shape
        hidden, dev = s["qw2"].shape[1], x.device
        q1 = torch.empty(rows, dim, dtype=torch.int8, device=dev)
        ops.invoke_layer_norm_int8o(q1, x, s["gamma"], s["beta"], s["pre1"], s["scale1"])
        h = torch.empty(rows, 2 * hidden, dtype=x.dtype, device=dev)
        ops.run_gemm_int8(q1, s["qw1"], s["sw1"], s["scale1"], h)
        q2 = torch.empty(rows, hidden, dtype=torch.int8, device=dev)
        ops.invoke_fused_add_bias_geglu_int8o(q2, h, s["b1"], s["pre2"], s["scale2"])
        y = torch.empty_like(x)
        return ops.run_gemm_int8(q2, s["qw2"], s["sw2"], s["scale2"], y, bias=s["b2"], residual=x)
    if kind == "adaln":
        x, outs = s["x"], {}
        if "int8" in s["outputs"]:
            outs["q8"] = torch.empty(x.shape, dtype=torch.int8, device=x.device)
            outs["q8_scale"] = torch.empty(x.shape[:2], dtype=torch.float32, device=x.device)
        if "e4m3" in s["outputs"]:
            outs["qf8"] = torch.empty(x.shape, dtype=torch.uint8, device=x.device)
        y = torch.empty_like(x) if s["outputs"] == "16bit" else None
        ops.invoke_layer_norm_with_shift_and_scale(y, x, s["scale"], s["shift"], f8_scale=s["f8_scale"], **outs)
        if y is not None:
            outs["y"] = y
        return outs
    if kind == "lora_swap":
        w = s["base"].clone()
        ops.invoke_load_lora(w, s["update"], 0.8)
        q = torch.empty(w.shape, dtype=torch.uint8, device=w.device)
        scale = torch.empty(1, dtype=torch.float32, device=w.device)
        ops.weight_quant_fp8(q, scale, w)
        return {"q": q, "scale": scale}
    if kind == "single_block":
        return s["op"].forward(s["x"], s["rope"], s["temb"])
    if kind == "double_block":
        return s["op"].forward(s["x"], s["context"], s["rope"], s["temb"])
    return s["op"].transformer_forward(s["latents"], s["context"], s["rope"], s["pooled"], 500.0, 3500.0)


# ---------------------------------------------------------------------------------------------- what a pass cannot do without
def _linear_work(m, n, k, weight_bytes_per_element):
    """(bytes of the weight, flops) of one linear; activations between the linears of a block need not touch memory."""
    return n * k * weight_bytes_per_element, 2.0 * m * n * k


def _block_work(kind, batch, tokens, text, level):
    """Weights once, input and output activations once; every linear, and the two products of the attention."""
    D = HIDDEN
    wb = 0.5 + 4.0 / 64 if level in W4A4_LEVELS else 1.0
    mod = 1.0 if level in (2, 8) else 2.0
    if kind == "single_block":
        parts = [_linear_work(batch * tokens, n, k, wb) for n, k in ((3 * D, D), (4 * D, D), (D, 5 * D))] + [_linear_work(batch, 3 * D, D, mod)]
    else:
        parts = []
        for rows in (batch * (tokens - text), batch * text):
            parts += [_linear_work(rows, n, k, wb) for n, k in ((3 * D, D), (D, D), (4 * D, D))]
            parts += [_linear_work(rows, D, 4 * D, 1.0), _linear_work(batch, 6 * D, D, mod)]
    flops = sum(p[1] for p in parts) + 4.0 * batch * tokens * tokens * D
    return sum(p[0] for p in parts), flops


def work(case):
    kind = case["kind"]
    if kind in ("linear_fp8", "linear_int8", "linear_w4a4"):
        m, n, k = case["m"], case["n"], case["k"]
        wb = {"linear_fp8": 1.0, "linear_int8": 1.0, "linear_w4a4": 0.5 + 2.0 / 64}[kind]
        b, f = _linear_work(m, n, k, wb)
        b += 2.0 * m * k + 2.0 * m * n + (2.0 * m * n if case.get("residual") else 0.0)
        if kind == "linear_w4a4":
            b, f = b + 64.0 * (n + k), f + 2.0 * m * 32 * (n + k)
        return {"bytes": b, "flops": f}
    if kind == "ff_int8":
        rows, dim = case["rows"], case["dim"]
        return {"bytes": 4.0 * rows * dim + 12.0 * dim * dim, "flops": 2.0 * rows * 12.0 * dim * dim}
    if kind == "adaln":
        e = case["batch"] * case["seq"] * case["dim"]
        out = {"int8+e4m3": 2, "int8": 1, "e4m3": 1, "16bit": 2}[case["outputs"]]
        return {"bytes": float(e * (2 + out)), "flops": 10.0 * e}
    if kind == "lora_swap":
        return {"bytes": 5.0 * case["n"] * case["k"], "flops": 4.0 * case["n"] * case["k"]}
    D = HIDDEN
    if kind == "single_block":
        b, f = _block_work(kind, case["batch"], case["tokens"], 0, case["level"])
        return {"bytes": b + 4.0 * case["batch"] * case["tokens"] * D, "flops": f}
    image, text = case["height"] * case["width"], case["text"]
    if kind == "double_block":
        b, f = _block_work(kind, case["batch"], image + text, text, case["level"])
        return {"bytes": b + 4.0 * case["batch"] * (image + text) * D, "flops": f}
    bd, fd = _block_work("double_block", 1, image + text, text, case["level"])
    bs, fs = _block_work("single_block", 1, image + text, 0, case["level"])
    outer = 2.0 * D * (2 * image * IN_CHANNELS + text * JOINT)
    return {"bytes": case["doubles"] * bd + case["singles"] * bs + 4.0 * image * IN_CHANNELS + 2.0 * text * JOINT,
            "flops": case["doubles"] * fd + case["singles"] * fs + outer}


def tolerance(case):
    """About four times what the outputs move by when every sum is taken in another order: the contraction of a linear or the
    columns of a row permuted, the tokens of a block or a forward permuted (another order of the softmax sums).  A rounding that
    falls the other way moves a 16-bit value by one step and may move a quantized one, so it grows through the blocks behind it."""
    kind = case["kind"]
    if kind == "lora_swap":
        return "exact"                                                 # no sum: a maximum and element-wise roundings
    if kind in ("linear_fp8", "linear_w4a4", "linear_int8"):
        return {"rel": 1e-3, "max": 0.02}                              # seen 1.2e-4 and one 16-bit step, 0.0078
    if kind == "ff_int8":
        return {"rel": 1e-3, "max": 0.12}                              # seen 2.1e-4 and 0.031
    if kind == "adaln":
        return {"rel": 1e-3, "max": 0.03, "differ": 5e-4}              # seen 2.4e-5, 0.0078, 3.5e-7; a row maximum on a rounding edge moves its row
    if kind == "forward":
        return {"rel": 0.03, "max": 0.25}                              # seen 0.016 and 0.077
    if case["level"] in W4A4_LEVELS:
        return {"rel": 0.012, "max": 0.17}                             # seen 0.0030 and 0.043
    return {"rel": 0.0065, "max": 0.08}                                # seen 0.0016 and 0.020
