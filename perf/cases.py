"""What a user has this framework do, as cases that can be timed and compared.

The work is the SD3.5-medium denoiser (24 blocks, the first 13 with the extra
image-only attention, width 1536, 24 heads) through its public entry points:

  forward   Model.forward on tensors that are on the GPU
  dropin    the torch extension's DiT(...), called like the original project's scripts call it;
            float32 tensors there select the exact float32 arithmetic
  block     one dual block on float32 residual streams, in place: float32 weights through the
            extension's DiT_block_cuda(...), FP8 GEMMs through Model.block_forward.  (FP8 is a case of
            one block: over 24 blocks a rounding of an e4m3 operand that falls the other way, as a
            change of the order of a sum brings it, moves the result by 3 %.)
  sample    sd3_b200.sample: a flow-matching loop with classifier-free guidance
  pipeline  HostPipeline.submit: a batch in pinned host memory in, the result in host memory out

An image of h x w latent pixels (patch 2) is (h/2)(w/2) tokens; 333 context tokens are 77 CLIP
and 256 T5 positions, 154 and 77 what a prompt without T5 brings.  The range is one 256x256 image to
one 2048x2048 image or a batch of eight 1024x1024 ones.

`norm_spread` is the spread of the query/key RMSNorm weights (log-normal).  0.05 is a model near its
initialisation, whose scores have a small bound; at 0.6 single dimensions stand out as they do in
trained checkpoints and the bound is too large to be of use in most blocks.
"""
import importlib.util
import math
import os
import sys

import torch

E, HEADS, EXPAND, LAYERS, DUAL = 1536, 24, 4, 24, 13
POOLED, CAPTIONS, CHANNELS, PATCH, POS_MAX, BASE = 2048, 4096, 16, 2, 384, 128


def _load(name, file):
    if name not in sys.modules:
        spec = importlib.util.spec_from_file_location(name, os.path.join(os.getcwd(), "sd3.c_b200", file))
        mod = importlib.util.module_from_spec(spec)
        sys.modules[name] = mod
        spec.loader.exec_module(mod)
    return sys.modules[name]


def _sd3():
    return _load("sd3_b200", "sd3_b200.py")


def _custom_modules():
    return _load("custom_modules", "custom_modules.so")


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def _case(entry, dtype, batch, h, w, ctx, norm_spread=0.05, steps=1):
    return dict(entry=entry, dtype=dtype, batch=batch, h=h, w=w, ctx=ctx, norm_spread=norm_spread, steps=steps)


def listed():
    cases = [
        # the original project's own use: one block on float32 tensors, 256 image and 77 context tokens
        ("block_fp32_256tok", _case("block", "fp32", 1, 32, 32, 77)),
        # the same project's full model on float32 tensors: 512x512, one image
        ("dropin_fp32_512px_b1", _case("dropin", "fp32", 1, 64, 64, 333)),
        # a preview or thumbnail: the smallest call, all weights read for little work
        ("forward_256px_b1", _case("forward", "bf16", 1, 32, 32, 333)),
        # one 512x512 image
        ("forward_512px_b1", _case("forward", "bf16", 1, 64, 64, 333)),
        # one 1024x1024 image per GPU: a batch of eight over eight GPUs
        ("forward_1024px_b1", _case("forward", "bf16", 1, 128, 128, 333)),
        # the headline: a batch of eight 1024x1024 images
        ("forward_1024px_b8", _case("forward", "bf16", 8, 128, 128, 333)),
        # one 2048x2048 image: attention over 16717 tokens
        ("forward_2048px_b1", _case("forward", "bf16", 1, 256, 256, 333)),
        # an odd batch of portrait images (832x1216), prompt without T5, trained-like norm weights
        ("forward_832x1216_b3", _case("forward", "bf16", 3, 152, 104, 154, 0.6)),
        # one guided image (conditional and unconditional stacked) through the drop-in, trained-like
        ("dropin_1024px_b2", _case("dropin", "bf16", 2, 128, 128, 333, 0.6)),
        # FP8 GEMMs: a block of two guided 1024x1024 images
        ("block_fp8_1024px_b4", _case("block", "fp8", 4, 128, 128, 333)),
        # a whole image: 28 guided steps at 512x512
        ("sample_512px_28steps", _case("sample", "bf16", 1, 64, 64, 333, 0.05, 28)),
        # serving: batches of four 512x512 images from pinned host memory and back
        ("pipeline_512px_b4", _case("pipeline", "bf16", 4, 64, 64, 333)),
    ]
    return [dict(c, name=n) for n, c in cases]


def draw(rng):
    most = {"bf16": 9.0e13, "fp8": 4.5e12, "fp32": 2.44e12}  # operations, about those of the largest listed case
    while True:
        entry, dtype = rng.choice([("forward", "bf16")] * 4 + [("dropin", "bf16"), ("dropin", "fp32"), ("block", "fp32"),
                                                               ("block", "fp8"), ("sample", "bf16"), ("pipeline", "bf16")])
        tokens = math.exp(rng.uniform(math.log(256), math.log(16384)))
        aspect = math.exp(rng.uniform(-math.log(2), math.log(2)))
        rows = max(8, min(192, round(math.sqrt(tokens * aspect))))
        cols = max(8, min(192, round(tokens / rows)))
        batch = rng.choice([1, 1, 2, 3, 4, 5, 6, 8])
        ctx = rng.choice([77, 154, 333, rng.randint(20, 400)])
        steps = rng.choice([4, 8, 20, 28]) if entry == "sample" else 1
        c = _case(entry, dtype, batch, 2 * rows, 2 * cols, ctx, rng.choice([0.05, 0.05, 0.6]), steps)
        if 256 <= rows * cols and batch * rows * cols <= 32768 and work(c)["flops"] <= most[dtype]:
            return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _block_shapes(dual, last):
    s = {}

    def lin(name, i, o):
        s[name + ".weight"], s[name + ".bias"] = (i, o), (o,)

    for stream, prefix in (("context", "context"), ("latent", "latent")) + ((("latent", "latent_dual"),) if dual else ()):
        lin(prefix + "_to_qkv", E, 3 * E)
        s[prefix + "_rmsnorm_key.weight"] = s[prefix + "_rmsnorm_query.weight"] = (E // HEADS,)
        if not (last and stream == "context"):
            lin(prefix + "_attn_Wout", E, E)
    lin("context_ada_lnorm.linear", E, (2 if last else 6) * E)
    lin("latent_ada_lnorm.linear", E, (9 if dual else 6) * E)
    for stream in ("latent",) if last else ("context", "latent"):
        lin(stream + "_mlp.lin1", E, EXPAND * E)
        lin(stream + "_mlp.lin2", EXPAND * E, E)
    return s


def _model_shapes():
    s = {}

    def lin(name, i, o):
        s[name + ".weight"], s[name + ".bias"] = (i, o), (o,)

    lin("timestep_mlp.0", 256, E)
    lin("timestep_mlp.2", E, E)
    lin("pooled_mlp.0", POOLED, E)
    lin("pooled_mlp.2", E, E)
    lin("captions_linear", CAPTIONS, E)
    s["to_patch.conv.weight"], s["to_patch.conv.bias"] = (E, CHANNELS, PATCH, PATCH), (E,)
    for l in range(LAYERS):
        for k, v in _block_shapes(l < DUAL, l == LAYERS - 1).items():
            s["transformer.%d.%s" % (l, k)] = v
    lin("ada_ln_out.linear", E, 2 * E)
    lin("linear_out", E, PATCH * PATCH * CHANNELS)
    return s


def _params(shapes, dtype, gen, norm_spread):
    p = {}
    for name, shape in shapes.items():
        t = torch.empty(shape, device="cuda", dtype=dtype)
        if "rmsnorm" in name:
            p[name] = t.normal_(0.0, norm_spread, generator=gen).exp_()
        else:
            p[name] = t.normal_(0.0, 0.02, generator=gen)
    return p


def _model(params):
    s = _sd3()
    m = s.Model(LAYERS, range(DUAL), POOLED, CAPTIONS, CHANNELS, E, HEADS, EXPAND, PATCH, POS_MAX, BASE, True, s.PRECISION_BF16)
    return m.load(params)


def _fp8_block(params):
    s = _sd3()
    m = s.Model(1, [0], 0, 0, 0, E, HEADS, EXPAND, 0, 0, 0, True, s.PRECISION_FP8, last_discards_context=False, block_only=True)
    return m.load(params, prefix="transformer.0.")


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dtype = torch.float32 if case["dtype"] == "fp32" else torch.bfloat16
    entry, batch, h, w, ctx = case["entry"], case["batch"], case["h"], case["w"], case["ctx"]

    def randn(*shape, dtype=dtype):
        return torch.empty(shape, device="cuda", dtype=dtype).normal_(generator=gen)

    if entry == "block":
        params = _params(_block_shapes(True, False), dtype, gen, case["norm_spread"])
        tokens, f32 = (h // PATCH) * (w // PATCH), torch.float32
        state = dict(case=case, y=torch.nn.functional.silu(randn(batch, E, dtype=f32)), c=randn(batch, ctx, E, dtype=f32),
                     x=randn(batch, tokens, E, dtype=f32))
        return dict(state, model=_fp8_block(params)) if case["dtype"] == "fp8" else dict(state, params=params)
    params = _params(_model_shapes(), dtype, gen, case["norm_spread"])
    state = dict(case=case, latent=randn(batch, CHANNELS, h, w), captions=randn(batch, ctx, CAPTIONS),
                 pooled=randn(batch, POOLED), t=torch.rand(batch, generator=gen, device="cuda") * 1000.0)
    if entry == "dropin":
        state["params"] = params
        return state
    state["model"] = _model(params)
    if entry == "sample":
        state.update(no_captions=randn(batch, ctx, CAPTIONS), no_pooled=randn(batch, POOLED))
    if entry == "pipeline":
        for k in ("latent", "captions", "pooled", "t"):
            state[k] = state[k].cpu().pin_memory()
        state["out"] = torch.empty(batch, CHANNELS, h, w, dtype=dtype).pin_memory()
        state["pipe"] = _sd3().HostPipeline(state["model"], batch, ctx, CHANNELS, h, w, POOLED, CAPTIONS, dtype)
    return state


def run(state):
    case = state["case"]
    entry = case["entry"]
    if entry == "block":
        # the call works in place: the streams of every pass start from the same values
        c, x = state["c"].clone(), state["x"].clone()
        if case["dtype"] == "fp8":
            return state["model"].block_forward(0, state["y"], c, x)
        return _custom_modules().DiT_block_cuda(state["y"], c, x, state["params"], c.shape[0], c.shape[1], x.shape[1], E,
                                                HEADS, EXPAND, True, True, False)
    if entry == "dropin":
        return _custom_modules().DiT(state["pooled"], state["captions"], state["latent"], state["t"], state["params"],
                                     LAYERS, set(range(DUAL)), POOLED, CAPTIONS, CHANNELS, E, HEADS, EXPAND, PATCH,
                                     POS_MAX, BASE, True)
    if entry == "sample":
        return _sd3().sample(state["model"], state["latent"], state["captions"], state["pooled"], state["no_captions"],
                             state["no_pooled"], steps=case["steps"])
    if entry == "pipeline":
        state["pipe"].submit(state["pooled"], state["captions"], state["latent"], state["t"], state["out"])
        state["pipe"].flush()
        return state["out"]
    return state["model"].forward(state["pooled"], state["captions"], state["latent"], state["t"])


# ---------------------------------------------------------------------------
# what a pass cannot do without, and how exact its result is
# ---------------------------------------------------------------------------
def _block_flops(tx, tc, dual, last):
    """Multiply-adds as two operations, one sample; the last block needs no context output."""
    t, mlp = tx + tc, 4 * EXPAND * E * E
    f = 6 * t * E * E + 4 * (tx if last else t) * t * E + (tx if last else t) * (2 * E * E + mlp)
    if last:
        f -= 2 * tc * E * E  # its context queries
    if dual:
        f += 8 * tx * E * E + 4 * tx * tx * E
    return f + 2 * E * E * ((2 if last else 6) + (9 if dual else 6))


def work(case):
    tx, tc, b = (case["h"] // PATCH) * (case["w"] // PATCH), case["ctx"], case["batch"]
    size = {"fp32": 4, "bf16": 2, "fp8": 1}[case["dtype"]]
    if case["entry"] == "block":  # the streams are read and written in float32; AdaLN is not an FP8 GEMM
        weights = size * sum(math.prod(v) for v in _block_shapes(True, False).values())
        weights += 15 * E * E if case["dtype"] == "fp8" else 0
        return {"bytes": weights + 4 * b * E + 8 * b * (tx + tc) * E, "flops": b * _block_flops(tx, tc, True, False)}
    weights = size * sum(math.prod(v) for v in _model_shapes().values())
    flops = sum(_block_flops(tx, tc, l < DUAL, l == LAYERS - 1) for l in range(LAYERS))
    flops += 2 * tc * CAPTIONS * E + 4 * tx * CHANNELS * PATCH * PATCH * E
    flops += 2 * E * (256 + E + POOLED + E + 2 * E)
    latent, prompt = b * CHANNELS * case["h"] * case["w"], b * (tc * CAPTIONS + POOLED)
    if case["entry"] == "sample":  # each step runs both branches and has to read the weights again
        return {"bytes": case["steps"] * weights + size * 2 * prompt + (size + 4) * latent,
                "flops": case["steps"] * 2 * b * flops}
    return {"bytes": weights + size * (prompt + 2 * latent), "flops": b * flops}


def tolerance(case):
    """About four times what separates two correct results: measured against the same model in the
    next higher precision and, for what rounding does along 24 blocks, against a run whose pooled
    prompt is off by one unit in the last place in ten values."""
    if case["dtype"] == "fp32":  # 2e-6
        return {"rel": 1e-5, "max": 1e-4}
    if case["dtype"] == "fp8":  # one block: 2e-3, and e4m3 roundings of the largest hidden values
        return {"rel": 1.2e-2, "max": 0.45}
    return {"rel": 1e-2 if case["entry"] == "sample" else 1.6e-2, "max": 8e-2}  # 1.3e-3 (relative to the latents), 4e-3
