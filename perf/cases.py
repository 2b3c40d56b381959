"""The measured workloads of the framework: its layers through the public kernel ops (``llmq_b200.kernels_api``) and one whole
optimizer step through ``LLMQTrainer``.

A case is a dict of plain values; ``kind`` picks the path:

``linear``      one projection of a decoder block, forward (quantise + GEMM) or backward (input, weight and bias gradient)
``attention``   RoPE, causal GQA attention, its backward and RoPE's backward on a packed QKV tensor
``norm``        residual add + RMSNorm and RMSNorm backward
``swiglu``      SwiGLU and its backward, or SwiGLU straight to e4m3 (the recompute path of an fp8 model)
``head``        one chunk of the LM head: logits GEMM + fused cross-entropy with the gradient written in place
``optimizer``   global gradient norm, clipping and AdamW on one flat parameter tensor
``step``        forward, backward and update of a model
"""
import math

import torch
import torch.nn.functional as F

import llmq_b200.kernels_api as ops
from llmq_b200.api import LLMQTrainer
from llmq_b200.config import create_config_from_name
from llmq_b200.options import LLamaOptions

BF16, F8 = torch.bfloat16, torch.float8_e4m3fn
GRAD_TYPES = {"bf16": torch.bfloat16, "e4m3": torch.float8_e4m3fn, "e5m2": torch.float8_e5m2}
F8_MAX = {torch.float8_e4m3fn: 448.0, torch.float8_e5m2: 57344.0}

# (hidden, intermediate, query heads, key/value heads, head size, vocabulary) of the built-in configurations
MODELS = ((896, 4864, 14, 2, 64, 151936), (1536, 8960, 12, 2, 128, 151936), (2048, 11008, 16, 2, 128, 151936), (2048, 8192, 32, 8, 64, 128256),
          (3072, 8192, 24, 8, 128, 128256), (3584, 18944, 28, 4, 128, 152064), (4096, 14336, 32, 8, 128, 128256), (5120, 13824, 40, 8, 128, 152064))


# ---------------------------------------------------------------------------------------------------------------------------- cases
def listed():
    return [
        # the MLP up + gate projection of the headline configuration (7B, 8 x 2048 tokens): the largest GEMM of an fp8 step
        {"name": "up_projection_7b_e4m3", "kind": "linear", "pass": "forward", "dtype": "e4m3", "tokens": 16384, "in": 3584, "out": 37888, "bias": False},
        # the backward of the attention output projection of the same step: quantise, transposes, both gradient GEMMs
        {"name": "out_projection_backward_7b_e4m3", "kind": "linear", "pass": "backward", "dtype": "e4m3", "grad": "e4m3", "tokens": 16384, "in": 3584,
         "out": 3584, "bias": False, "accumulate": True},
        # bf16 training of the 1.5B configuration (16 x 1024 tokens): both gradient GEMMs of the up projection, operands as they lie in memory
        {"name": "up_projection_backward_1.5b_bf16", "kind": "linear", "pass": "backward", "dtype": "bf16", "grad": "bf16", "tokens": 16384, "in": 1536,
         "out": 17920, "bias": False, "accumulate": False},
        # fine-tuning of the 0.5B configuration on one batch of odd length: the three gradients of the QKV projection
        {"name": "qkv_backward_0.5b_bf16_short", "kind": "linear", "pass": "backward", "dtype": "bf16", "grad": "bf16", "tokens": 1001, "in": 896, "out": 1152,
         "bias": True, "accumulate": True},
        # the attention core of the headline configuration
        {"name": "attention_7b", "kind": "attention", "batch": 8, "seq": 2048, "q_heads": 28, "kv_heads": 4, "head": 128},
        # head size 64: the 0.5B configuration, 8 x 1024 tokens
        {"name": "attention_0.5b", "kind": "attention", "batch": 8, "seq": 1024, "q_heads": 14, "kv_heads": 2, "head": 64},
        # one short sequence of odd length through the 1.5B configuration: latency and launches
        {"name": "attention_1.5b_short", "kind": "attention", "batch": 1, "seq": 333, "q_heads": 12, "kv_heads": 2, "head": 128},
        # norms and activation of the headline configuration: the bandwidth-bound part of a block
        {"name": "norm_7b", "kind": "norm", "rows": 16384, "channels": 3584},
        {"name": "swiglu_7b", "kind": "swiglu", "mode": "bf16", "rows": 16384, "width": 18944},
        # one of the four LM-head chunks of the headline configuration
        {"name": "lm_head_chunk_7b", "kind": "head", "tokens": 4096, "channels": 3584, "vocab": 152064, "z_reg": 0.0},
        # gradient norm and AdamW with 16-bit moments on the down projection of the headline configuration
        {"name": "adamw_7b_down_projection", "kind": "optimizer", "numel": 3584 * 18944, "moments": "bf16"},
        # a bf16 step of a model with the 0.5B configuration's blocks, bf16 moments: many small kernels, the embedding and the optimizer among them
        {"name": "train_step_0.5b_6_layers", "kind": "step", "layers": 6, "batch": 4, "seq": 1024},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["linear", "linear", "linear", "attention", "attention", "norm", "swiglu", "head", "optimizer", "step"])
    C, D, Hq, Hkv, HS, V = rng.choice(MODELS)
    tokens = _log_int(rng, 256, 16384)
    if kind == "linear":
        n_in, n_out = rng.choice([(C, (Hq + 2 * Hkv) * HS), (C, C), (C, 2 * D), (D, C)])
        while tokens * n_in * n_out * 4 > 4.4e12:
            tokens //= 2
        which, dtype = rng.choice(["forward", "backward"]), rng.choice(["bf16", "e4m3"])
        case = {"kind": kind, "pass": which, "dtype": dtype, "tokens": tokens, "in": n_in, "out": n_out, "bias": rng.random() < 0.3}
        if which == "backward":
            case["grad"] = "bf16" if dtype == "bf16" else rng.choice(["e4m3", "e5m2"])
            case["accumulate"] = rng.random() < 0.5
            if dtype == "e4m3":
                case["tokens"] = tokens // 16 * 16       # fp8 rows of the transposed copies start at multiples of 16 bytes
        return case
    if kind == "attention":
        batch = _log_int(rng, 1, 8)
        return {"kind": kind, "batch": batch, "seq": max(65, min(8192, _log_int(rng, 100, 16384) // batch)), "q_heads": min(Hq, 32),
                "kv_heads": min(Hkv, 8) if Hq <= 32 else 8, "head": HS}
    if kind == "norm":
        return {"kind": kind, "rows": _log_int(rng, 100, 16384), "channels": C}
    if kind == "swiglu":
        return {"kind": kind, "mode": rng.choice(["bf16", "e4m3"]), "rows": tokens, "width": D}
    if kind == "head":
        return {"kind": kind, "tokens": min(tokens, 4096), "channels": min(C, 3584), "vocab": V, "z_reg": rng.choice([0.0, 1e-4])}
    if kind == "optimizer":
        return {"kind": kind, "numel": _log_int(rng, 1000, 1 << 20) * 128, "moments": rng.choice(["bf16", "e4m3", "fp32"])}
    seq = 8 * _log_int(rng, 32, 128)
    return {"kind": kind, "layers": rng.randint(2, 6), "batch": _log_int(rng, 1, 4), "seq": seq}


# --------------------------------------------------------------------------------------------------------------------------- inputs
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _randn(g, *shape, std=1.0, dtype=BF16):
    t = torch.randn(*shape, generator=g, device="cuda", dtype=dtype)
    return t if std == 1.0 else t.mul_(std)


def _zeros(*shape, dtype=BF16):
    return torch.zeros(*shape, device="cuda", dtype=dtype)


def _absmax(x):
    return x.abs().max().float().reshape(1)


def _to_f8(x, dtype=F8):
    """(values, dequantisation factor) of the per-tensor recipe: x * MAX / absmax, saturated."""
    am = _absmax(x)
    q = (x.float() * (F8_MAX[dtype] / am)).clamp(-F8_MAX[dtype], F8_MAX[dtype]).to(dtype)
    return q, am / F8_MAX[dtype]


def _linear_inputs(c, seed):
    g = _gen(seed)
    d = {"x": _randn(g, c["tokens"], c["in"]), "w": _randn(g, c["out"], c["in"], std=0.02),
         "b": _randn(g, c["out"], std=0.02) if c["bias"] else None}
    if c["pass"] == "backward":
        d["dout"] = _randn(g, c["tokens"], c["out"], std=1.0 / c["tokens"])
        if c["accumulate"]:
            d["dw"] = _randn(g, c["out"], c["in"], std=1.0 / math.sqrt(c["tokens"]))
            d["db"] = _randn(g, c["out"], std=1.0 / math.sqrt(c["tokens"])) if c["bias"] else None
        else:
            d["dw"], d["db"] = _zeros(c["out"], c["in"]), _zeros(c["out"]) if c["bias"] else None
    return d


def _attention_inputs(c, seed):
    g = _gen(seed)
    B, T, H = c["batch"], c["seq"], c["q_heads"] + 2 * c["kv_heads"]
    return {"qkv": _randn(g, B, T, H, c["head"]), "dout": _randn(g, B, T, c["q_heads"], c["head"], std=1.0 / T), "theta": 1e6}


def _rope_table(T, HS, theta):
    inv = theta ** (-torch.arange(HS // 2, dtype=torch.float64, device="cuda") * 2.0 / HS)
    ang = torch.arange(T, dtype=torch.float64, device="cuda")[:, None] * inv[None, :]
    return torch.stack([ang.cos(), ang.sin()], -1)


def _norm_inputs(c, seed):
    g = _gen(seed)
    R, C = c["rows"], c["channels"]
    return {"x": _randn(g, R, C, std=2.0), "y": _randn(g, R, C), "w": (1 + 0.1 * _randn(g, C, dtype=torch.float32)).to(BF16), "dout": _randn(g, R, C, std=1.0 / R),
            "dres": _randn(g, R, C, std=1.0 / R), "dw": _zeros(C)}


def _swiglu_inputs(c, seed):
    g = _gen(seed)
    return {"up": _randn(g, c["rows"], 2 * c["width"]), "dout": _randn(g, c["rows"], c["width"], std=1.0 / c["rows"]) if c["mode"] == "bf16" else None}


def _head_inputs(c, seed):
    g = _gen(seed)
    tg = torch.randint(0, c["vocab"], (c["tokens"],), generator=g, device="cuda", dtype=torch.int32)
    tg[::64] = -100                                      # masked positions
    return {"x": _randn(g, c["tokens"], c["channels"]), "w": _randn(g, c["vocab"], c["channels"], std=0.02), "targets": tg}


HYPER = {"lr": 3e-4, "beta1": 0.9, "beta2": 0.95, "step": 100, "eps": 1e-8, "weight_decay": 0.1}
CLIP = 1.0


def _optimizer_inputs(c, seed):
    g = _gen(seed)
    n, dt = c["numel"], {"bf16": BF16, "e4m3": BF16, "fp32": torch.float32}[c["moments"]]
    d = {"p": _randn(g, n, std=0.02), "g": _randn(g, n, std=1e-3), "v": _randn(g, n, dtype=torch.float32).square_().mul_(1e-6).to(dt)}
    m = _randn(g, n, std=1e-3, dtype=torch.float32)
    if c["moments"] == "e4m3":
        sc = m.view(-1, 128).abs().amax(-1) / 448.0
        d["m"], d["m_scales"] = (m.view(-1, 128) / sc[:, None]).clamp(-448, 448).to(F8).view(-1), sc
    else:
        d["m"], d["m_scales"] = m.to(dt), None
    return d


def _step_config(c):
    return create_config_from_name("Qwen2.5-0.5B").replace(num_hidden_layers=c["layers"])


def _step_weights(c, seed):
    """Name -> tensor, in the fused layout (q, k, v rows in one matrix, [up | gate] rows in one matrix)."""
    C, D, V, QC = 896, 4864, 151936, 1152
    g, out = _gen(seed), {}
    for l in range(c["layers"]):
        p = "layers.%d." % l
        out[p + "ln1_w"] = (1 + 0.1 * _randn(g, C, dtype=torch.float32)).to(BF16)
        out[p + "qkv_w"], out[p + "qkv_b"] = _randn(g, QC, C, std=0.02), _randn(g, QC, std=0.02)
        out[p + "o_w"] = _randn(g, C, C, std=0.02 / math.sqrt(2 * c["layers"]))
        out[p + "ln2_w"] = (1 + 0.1 * _randn(g, C, dtype=torch.float32)).to(BF16)
        out[p + "up_w"], out[p + "down_w"] = _randn(g, 2 * D, C, std=0.02), _randn(g, C, D, std=0.02 / math.sqrt(2 * c["layers"]))
    out["embed"], out["lnf_w"] = _randn(g, V, C, std=0.02), (1 + 0.1 * _randn(g, C, dtype=torch.float32)).to(BF16)
    return out


def _step_tokens(c, seed):
    g = torch.Generator().manual_seed(int(seed) + 1)
    t = torch.randint(0, 151936, (c["batch"], c["seq"] + 1), generator=g, dtype=torch.int32)
    return t[:, :-1].contiguous(), t[:, 1:].contiguous()


# -------------------------------------------------------------------------------------------------------------------------- prepare
def _prepare_linear(c, seed):
    s = _linear_inputs(c, seed)
    M, K, N = c["tokens"], c["in"], c["out"]
    if c["dtype"] == "e4m3":
        s["wq"], s["sw"] = _to_f8(s["w"])                # the work copy of the weight, made once per optimizer step
        s["amax_x"] = _absmax(s["x"])                    # written by the kernel that produced x
    if c["pass"] == "forward":
        s["y"] = _zeros(M, N)
        if c["dtype"] == "e4m3":
            s["xq"], s["sx"] = torch.empty(M, K, dtype=F8, device="cuda"), _zeros(1, dtype=torch.float32)
        return s
    s["dx"] = _zeros(M, K)
    s["bias_scratch"] = torch.empty(ops.get_bias_backward_scratch_size(BF16, N) // 4, device="cuda") if c["bias"] else None
    if c["dtype"] == "e4m3":
        gt = GRAD_TYPES[c["grad"]]
        s["xq"], s["sx"] = _to_f8(s["x"])                # kept from the forward pass
        s["amax_d"], s["sd"] = _absmax(s["dout"]), _zeros(1, dtype=torch.float32)
        s["dq"], s["dqT"] = torch.empty(M, N, dtype=gt, device="cuda"), torch.empty(N, M, dtype=gt, device="cuda")
        s["xqT"], s["wqT"] = torch.empty(K, M, dtype=F8, device="cuda"), torch.empty(K, N, dtype=F8, device="cuda")
    return s


def _prepare_attention(c, seed):
    s = _attention_inputs(c, seed)
    B, T, Hq, HS = c["batch"], c["seq"], c["q_heads"], c["head"]
    s["freqs"] = _rope_table(T, HS, s["theta"]).float()
    s["rotated"], s["out"], s["lse"] = torch.empty_like(s["qkv"]), _zeros(B, T, Hq, HS), _zeros(B, Hq, T, dtype=torch.float32)
    s["dqkv"], s["scratch"] = torch.empty_like(s["qkv"]), _zeros(B * Hq * T, dtype=torch.float32)
    s["dinp"], s["absmax"] = torch.empty_like(s["qkv"]), _zeros(1, dtype=torch.float32)
    return s


def _prepare_norm(c, seed):
    s = _norm_inputs(c, seed)
    R, C = c["rows"], c["channels"]
    s["residual"], s["normed"], s["rstd"] = _zeros(R, C), _zeros(R, C), _zeros(R, dtype=torch.float32)
    s["amax_f"], s["amax_b"] = _zeros(1, dtype=torch.float32), _zeros(1, dtype=torch.float32)
    s["scratch"] = torch.empty(ops.get_rmsnorm_backward_scratch_size(C) // 4, device="cuda")
    return s


def _prepare_swiglu(c, seed):
    s = _swiglu_inputs(c, seed)
    R, D = c["rows"], c["width"]
    if c["mode"] == "bf16":
        s["out"], s["dup"] = _zeros(R, D), _zeros(R, 2 * D)
        s["amax_f"], s["amax_b"] = _zeros(1, dtype=torch.float32), _zeros(1, dtype=torch.float32)
    else:
        s["q"], s["scale"] = torch.empty(R, D, dtype=F8, device="cuda"), _zeros(1, dtype=torch.float32)
        s["amax_f"] = torch.full((1,), 16.0, device="cuda")    # known from the forward pass
    return s


def _prepare_head(c, seed):
    s = _head_inputs(c, seed)
    s["logits"] = torch.empty(c["tokens"], c["vocab"], dtype=BF16, device="cuda")
    s["losses"], s["lse"] = _zeros(c["tokens"], dtype=torch.float32), _zeros(c["tokens"], dtype=torch.float32)
    return s


def _prepare_optimizer(c, seed):
    s = _optimizer_inputs(c, seed)
    s["partials"], s["io"], s["absmax"] = _zeros(512, dtype=torch.float32), _zeros(2, dtype=torch.float32), _zeros(1, dtype=torch.float32)
    s["seed"] = int(seed) % 1000003
    return s


def _prepare_step(c, seed):
    cfg = _step_config(c)
    opts = LLamaOptions(momentum_type=BF16, variance_type=BF16)
    tr = LLMQTrainer(ngpu=1, config=cfg, options=opts, batch_size=c["batch"], seq_len=c["seq"], grad_accum=1, device="cuda:0")
    w = _step_weights(c, seed)
    for name, master, _, _ in tr.model.weights.master_items():
        master.copy_(w[name].view(master.shape))
    tr.model.on_weights_changed()
    x, y = _step_tokens(c, seed)
    return {"trainer": tr, "x": x, "y": y}


def prepare(case, seed):
    s = {"linear": _prepare_linear, "attention": _prepare_attention, "norm": _prepare_norm, "swiglu": _prepare_swiglu, "head": _prepare_head,
         "optimizer": _prepare_optimizer, "step": _prepare_step}[case["kind"]](case, seed)
    s["case"] = dict(case)
    return s


# ------------------------------------------------------------------------------------------------------------------------------ run
def _run_linear(s, c):
    if c["pass"] == "forward":
        if c["dtype"] == "e4m3":
            ops.quantize_with_abs_max(s["xq"], s["sx"], s["x"], s["amax_x"])
            ops.matmul(s["y"], s["xq"], s["wq"], s["b"], s["sx"], s["sw"], None, "TN", False)
        else:
            ops.matmul(s["y"], s["x"], s["w"], s["b"], None, None, None, "TN", False)
        return {"y": s["y"]}
    if c["dtype"] == "e4m3":
        ops.quantize_with_abs_max(s["dq"], s["sd"], s["dout"], s["amax_d"])
        ops.quantize_and_transpose_with_abs_max(s["dqT"], s["sd"], s["dout"], s["amax_d"])
        ops.transpose(s["wqT"], s["wq"])
        ops.matmul(s["dx"], s["dq"], s["wqT"], None, s["sd"], s["sw"], None, "TN", False)
        ops.transpose(s["xqT"], s["xq"])
        ops.matmul(s["dw"], s["dqT"], s["xqT"], None, s["sd"], s["sx"], None, "TN", c["accumulate"])
        if c["bias"]:
            ops.backward_bias(s["db"], s["dq"], s["sd"], None, s["bias_scratch"], c["accumulate"])
    else:
        ops.matmul(s["dx"], s["dout"], s["w"], None, None, None, None, "TT", False)
        ops.matmul(s["dw"], s["dout"], s["x"], None, None, None, None, "NT", c["accumulate"])
        if c["bias"]:
            ops.backward_bias(s["db"], s["dout"], None, None, s["bias_scratch"], c["accumulate"])
    return {"dx": s["dx"], "dw": s["dw"], "db": s["db"]}


def _run_attention(s, c):
    Hq, Hkv = c["q_heads"], c["kv_heads"]
    ops.rope_forward(s["rotated"], s["qkv"], s["freqs"], None, Hq, Hkv)
    ops.attention_forward(s["out"], s["lse"], s["rotated"], Hq, Hkv)
    ops.attention_backward(s["dqkv"], s["scratch"], s["lse"], s["out"], s["dout"], s["rotated"], Hq, Hkv)
    ops.rope_backward(s["dinp"], s["dqkv"], s["freqs"], s["absmax"], Hq, Hkv)
    return {"out": s["out"], "lse": s["lse"], "dqkv": s["dinp"], "absmax": s["absmax"]}


def _run_norm(s, c):
    ops.fused_residual_rmsnorm_forward(s["residual"], s["normed"], s["rstd"], s["x"], s["y"], s["w"], s["amax_f"], 1e-6)
    ops.rmsnorm_backward(s["dres"], s["dw"], s["scratch"], s["dout"], s["residual"], s["w"], s["rstd"], s["amax_b"])
    return {"residual": s["residual"], "normed": s["normed"], "rstd": s["rstd"], "dres": s["dres"], "dw": s["dw"], "amax": s["amax_f"], "amax_b": s["amax_b"]}


def _run_swiglu(s, c):
    if c["mode"] == "e4m3":
        ops.swiglu_forward_quant(s["q"], s["scale"], s["up"], s["amax_f"])
        return {"q": s["q"], "scale": s["scale"]}
    ops.swiglu_forward(s["out"], s["up"], s["amax_f"])
    ops.swiglu_backward(s["dup"], s["dout"], s["up"], s["amax_b"])
    return {"out": s["out"], "dup": s["dup"], "amax_f": s["amax_f"], "amax_b": s["amax_b"]}


def _run_head(s, c):
    s["losses"].zero_()
    ops.matmul(s["logits"], s["x"], s["w"], None, None, None, None, "TN", False)
    ops.fused_classifier(s["logits"], s["losses"], s["lse"], 1.0 / c["tokens"], s["targets"], c["z_reg"] / c["tokens"], True)
    return {"dlogits": s["logits"], "losses": s["losses"], "lse": s["lse"]}


def _run_optimizer(s, c):
    s["partials"].zero_()
    ops.global_norm_squared(s["partials"], s["g"])
    ops.global_norm_finish(s["io"], s["partials"], CLIP)
    ops.adamw_update(s["p"], s["g"], s["m"], s["v"], grad_scale=s["io"][1:2], m_scales=s["m_scales"], abs_max=s["absmax"], seed=s["seed"], **HYPER)
    return {"p": s["p"], "m": s["m"], "v": s["v"], "m_scales": s["m_scales"], "norm": s["io"], "absmax": s["absmax"]}


def _run_step(s, c):
    tr = s["trainer"]
    tr.step(s["x"], s["y"])
    r = tr.update(lr=1e-5, beta1=0.9, beta2=0.95, step=1, weight_decay=0.1, grad_clip=1.0)
    return {"loss": r["loss"], "norm": r["norm"], "gradients": tr.get_gradients()}


def run(state):
    c = state["case"]
    return {"linear": _run_linear, "attention": _run_attention, "norm": _run_norm, "swiglu": _run_swiglu, "head": _run_head,
            "optimizer": _run_optimizer, "step": _run_step}[c["kind"]](state, c)


# ----------------------------------------------------------------------------------------------------------------------------- work
def work(case):
    c = case
    if c["kind"] == "linear":
        M, K, N = c["tokens"], c["in"], c["out"]
        wb = 1 if c["dtype"] == "e4m3" else 2
        if c["pass"] == "forward":
            return {"bytes": M * K * 2 + N * K * wb + M * N * 2, "flops": 2.0 * M * K * N}
        return {"bytes": M * N * 2 + M * K * wb + N * K * wb + M * K * 2 + N * K * (4 if c["accumulate"] else 2), "flops": 4.0 * M * K * N}
    if c["kind"] == "attention":
        B, T, Hq, Hkv, HS = c["batch"], c["seq"], c["q_heads"], c["kv_heads"], c["head"]
        pairs = B * Hq * T * (T + 1) / 2.0
        return {"bytes": 2.0 * B * T * HS * (2 * (Hq + 2 * Hkv) + 2 * Hq) + 4.0 * B * Hq * T, "flops": 14.0 * pairs * HS}
    if c["kind"] == "norm":
        n = c["rows"] * c["channels"]
        return {"bytes": 14.0 * n, "flops": 16.0 * n}     # x, y in; residual, normed out; dout, dres in; dres out
    if c["kind"] == "swiglu":
        n = c["rows"] * c["width"]
        return {"bytes": (5.0 if c["mode"] == "e4m3" else 12.0) * n, "flops": 16.0 * n}
    if c["kind"] == "head":
        M, C, V = c["tokens"], c["channels"], c["vocab"]
        return {"bytes": 2.0 * (M * C + V * C + M * V), "flops": 2.0 * M * C * V}
    if c["kind"] == "optimizer":
        n, mv = c["numel"], {"bf16": 4, "e4m3": 3, "fp32": 8}[c["moments"]]
        return {"bytes": n * (2.0 + 4.0 + 2.0 * mv), "flops": 16.0 * n}
    C, D, V, QC, L, T = 896, 4864, 151936, 1152, c["layers"], c["batch"] * c["seq"]
    block = C * QC + C * C + 3 * C * D
    n = L * block + V * C
    return {"bytes": n * 14.0, "flops": 6.0 * T * n + 14.0 * L * T * (c["seq"] + 1) / 2 * C}


def tolerance(case):
    """About four times what another correct implementation at the same precision shows: fp32 sums in another order, then the
    rounding of the output (bf16: 2^-9 of a value at most; a flipped tie is 2^-8), 16-bit probabilities inside attention."""
    k = case["kind"]
    if k == "linear":
        return {"rel": 4e-3, "max": 0.05}
    if k == "attention":
        return {"rel": 1.2e-2, "max": 0.2}
    if k == "norm":
        return {"rel": 4e-3, "max": 0.05}
    if k == "swiglu":
        return {"rel": 4e-3, "max": 0.15}
    if k == "head":
        return {"rel": 1e-3, "max": 0.05}                  # the target column of a row, near -1 / tokens, carries its norm
    if k == "optimizer":
        return {"rel": 4e-3, "max": 0.15}
    return {"rel": 3e-2, "max": 0.8}                      # a change of rounding in one layer travels through all that follow


# ---------------------------------------------------------------------------------------------------------------------------- exact
def _exact_linear(c, seed):
    d = _linear_inputs(c, seed)
    x, w = d["x"].double(), d["w"].double()
    if c["dtype"] == "e4m3":
        (xq, sx), (wq, sw) = _to_f8(d["x"]), _to_f8(d["w"])
        x, w = xq.double() * sx.double(), wq.double() * sw.double()
    if c["pass"] == "forward":
        y = x @ w.t()
        return {"y": y if d["b"] is None else y.add_(d["b"].double())}
    dout = d["dout"].double()
    if c["dtype"] == "e4m3":
        dq, sd = _to_f8(d["dout"], GRAD_TYPES[c["grad"]])
        dout = dq.double() * sd.double()
    return {"dx": dout @ w, "dw": d["dw"].double() + dout.t() @ x, "db": None if d["db"] is None else d["db"].double() + dout.sum(0)}


def _rotate(x, table, heads, sign=1.0):
    """RoPE (its transpose with sign = -1) on the first ``heads`` heads of x[B, T, H, HS]."""
    h = x.shape[-1] // 2
    cos, sin = table[:, None, :, 0], sign * table[:, None, :, 1]
    a, b = x[:, :, :heads, :h], x[:, :, :heads, h:]
    return torch.cat([torch.cat([a * cos - b * sin, b * cos + a * sin], -1), x[:, :, heads:]], 2)


def _exact_attention(c, seed):
    d = _attention_inputs(c, seed)
    B, T, Hq, Hkv, HS = c["batch"], c["seq"], c["q_heads"], c["kv_heads"], c["head"]
    table, G, scale = _rope_table(T, HS, d["theta"]), Hq // Hkv, 1.0 / math.sqrt(HS)
    qkv = _rotate(d["qkv"].double(), table, Hq + Hkv)
    dout = d["dout"].double()
    out, lse, dqkv = torch.empty_like(dout), torch.empty(B, Hq, T, dtype=torch.float64, device="cuda"), torch.zeros_like(qkv)
    hidden = torch.ones(T, T, dtype=torch.bool, device="cuda").triu(1)
    for b in range(B):
        for h in range(Hq):
            k_at, v_at = Hq + h // G, Hq + Hkv + h // G
            q, k, v, do = qkv[b, :, h], qkv[b, :, k_at], qkv[b, :, v_at], dout[b, :, h]
            s = (q @ k.t()).mul_(scale).masked_fill_(hidden, -math.inf)
            lse[b, h] = torch.logsumexp(s, -1)
            p = s.sub_(lse[b, h][:, None]).exp_()
            out[b, :, h] = p @ v
            dqkv[b, :, v_at] += p.t() @ do
            ds = (do @ v.t()).sub_((do * out[b, :, h]).sum(-1, keepdim=True)).mul_(p).mul_(scale)
            dqkv[b, :, h] = ds @ k
            dqkv[b, :, k_at] += ds.t() @ q
    dinp = _rotate(dqkv, table, Hq + Hkv, -1.0)
    return {"out": out, "lse": lse, "dqkv": dinp, "absmax": dinp.abs().max().reshape(1)}


def _exact_norm(c, seed):
    d = _norm_inputs(c, seed)
    r = (d["x"].float() + d["y"].float()).to(BF16).double()        # the residual stream is bf16
    w, dy = d["w"].double(), d["dout"].double()
    rstd = torch.rsqrt(r.square().mean(-1, keepdim=True) + 1e-6)
    xh = r * rstd
    normed = xh * w
    dres = d["dres"].double() + (w * dy - xh * (w * dy * xh).mean(-1, keepdim=True)) * rstd
    return {"residual": r, "normed": normed, "rstd": rstd[:, 0], "dres": dres, "dw": (dy * xh).sum(0), "amax": normed.abs().max().reshape(1),
            "amax_b": dres.abs().max().reshape(1)}


def _exact_swiglu(c, seed):
    d = _swiglu_inputs(c, seed)
    D = c["width"]
    up, gate = d["up"][:, :D].double(), d["up"][:, D:].double()
    s = torch.sigmoid(gate)
    out = up * gate * s
    if c["mode"] == "e4m3":
        return {"q": out * (448.0 / 16.0), "scale": torch.full((1,), 16.0 / 448.0, dtype=torch.float64, device="cuda")}
    do = d["dout"].double()
    dup = torch.cat([do * gate * s, do * up * s * (1 + gate * (1 - s))], -1)
    return {"out": out, "dup": dup, "amax_f": out.abs().max().reshape(1), "amax_b": dup.abs().max().reshape(1)}


def _exact_head(c, seed):
    d = _head_inputs(c, seed)
    lg = d["x"].double() @ d["w"].double().t()
    tg = d["targets"].long()
    ok, safe, rows = tg >= 0, tg.clamp_min(0), torch.arange(c["tokens"], device="cuda")
    lse = torch.logsumexp(lg, -1)
    losses = torch.where(ok, lse - lg[rows, safe], torch.zeros_like(lse))
    scale = (1.0 + c["z_reg"] * lse) / c["tokens"]
    g = lg.sub_(lse[:, None]).exp_().mul_((scale * ok)[:, None])
    g[rows, safe] -= ok.double() / c["tokens"]
    return {"dlogits": g, "losses": losses, "lse": torch.where(ok, lse, torch.zeros_like(lse))}


def _exact_optimizer(c, seed):
    d = _optimizer_inputs(c, seed)
    g, p, v, m = d["g"].double(), d["p"].double(), d["v"].double(), d["m"].double()
    if d["m_scales"] is not None:
        m = m * d["m_scales"].double().repeat_interleave(128)
    norm = g.square().sum().sqrt()
    clip = torch.clamp(CLIP / norm, max=1.0)
    h = HYPER
    g = g * clip
    m = h["beta1"] * m + (1 - h["beta1"]) * g
    v = h["beta2"] * v + (1 - h["beta2"]) * g * g
    p = p - h["lr"] * (m / (1 - h["beta1"] ** h["step"]) / ((v / (1 - h["beta2"] ** h["step"])).sqrt() + h["eps"]) + h["weight_decay"] * p)
    sc = m.view(-1, 128).abs().amax(-1) / 448.0 if d["m_scales"] is not None else None
    return {"p": p, "m": m if sc is None else (m.view(-1, 128) / sc[:, None]).view(-1), "v": v, "m_scales": sc, "norm": torch.stack([norm, clip]),
            "absmax": p.abs().max().reshape(1)}


def _exact_step(c, seed):
    C, D, Hq, Hkv, HS, L = 896, 4864, 14, 2, 64, c["layers"]
    w = {n: t.double().requires_grad_(True) for n, t in _step_weights(c, seed).items()}
    x, y = (t.cuda().long() for t in _step_tokens(c, seed))
    B, T = x.shape
    table = _rope_table(T, HS, 1e6)
    norm = lambda h, g: h * torch.rsqrt(h.square().mean(-1, keepdim=True) + 1e-6) * g  # noqa: E731
    h = w["embed"][x]
    for l in range(L):
        p = lambda n: w["layers.%d.%s" % (l, n)]  # noqa: E731
        qkv = _rotate((norm(h, p("ln1_w")) @ p("qkv_w").t() + p("qkv_b")).view(B, T, Hq + 2 * Hkv, HS), table, Hq + Hkv).transpose(1, 2)
        k, v = (t.repeat_interleave(Hq // Hkv, 1) for t in (qkv[:, Hq:Hq + Hkv], qkv[:, Hq + Hkv:]))
        s = (qkv[:, :Hq] @ k.transpose(-1, -2)) / math.sqrt(HS)
        s = s.masked_fill(torch.ones(T, T, dtype=torch.bool, device="cuda").triu(1), -math.inf)
        h = h + (torch.softmax(s, -1) @ v).transpose(1, 2).reshape(B, T, C) @ p("o_w").t()
        ug = norm(h, p("ln2_w")) @ p("up_w").t()
        h = h + (ug[..., :D] * F.silu(ug[..., D:])) @ p("down_w").t()
    loss = F.cross_entropy((norm(h, w["lnf_w"]) @ w["embed"].t()).view(B * T, -1), y.view(-1))
    loss.backward()
    return {"loss": float(loss), "norm": float(torch.stack([t.grad.square().sum() for t in w.values()]).sum().sqrt()),
            "gradients": {n: t.grad for n, t in w.items()}}


def exact(case, seed):
    return {"linear": _exact_linear, "attention": _exact_attention, "norm": _exact_norm, "swiglu": _exact_swiglu, "head": _exact_head,
            "optimizer": _exact_optimizer, "step": _exact_step}[case["kind"]](case, seed)
