"""The workloads the framework's speed is judged by: training steps and logits of the model, and its operators.

Sizes are those of the named configurations (160M, 410M, 840M, 1.4B), of the operator tests, or generic ones of the
same ranges.  Every case is one of these kinds:

* `train`      `Transformer(ids, labels)` under autocast and the backward pass of the scaled loss.  With `buckets` the
               gradients are written into flat buckets (`dp.GradBuckets`), as the benchmark and a data-parallel run do;
               without, they are the parameters' own `.grad`, as in a plain PyTorch loop.
* `logits`     `Transformer(ids, None)` without gradients: scoring a batch of prompts.
* `attention`  the causal attention Function, forward and backward; no bias, or ALiBi as slopes or as the table.
* `linear`     one of the four linear Functions, forward and backward.
* `layernorm`, `softmax`, `loss`  the row-wise Functions, forward and backward.
* `adamw`      the optimizer step on gradient buckets.
"""
import math

import torch

import tritonformer_b200 as tfb
from tritonformer_b200.dp import GradBuckets
from tritonformer_b200.optim import FusedAdamW, LossScaler
from tritonformer_b200.transformer import Transformer, TransformerConfig, generate_alibi_mask, get_slopes

DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16, "fp32": torch.float32}
LOSS_SCALE = {"fp16": 4096.0, "bf16": 1.0}


def _model(name, kind, d, layers, head_dim, vocab, batch, seq, dtype, bias=False, alibi=False, buckets=True):
    return {"name": name, "kind": kind, "d": d, "layers": layers, "head_dim": head_dim, "vocab": vocab, "batch": batch,
            "seq": seq, "dtype": dtype, "bias": bias, "alibi": alibi, "buckets": buckets}


def listed():
    return [
        # a small model as one trains while developing: a step is a few hundred short kernels, gradients in .grad
        _model("train_small", "train", 256, 3, 64, 1024, 2, 256, "fp16", buckets=False),
        # the 160M configuration at its own batch of 2 x 1024 tokens
        _model("train_160m", "train", 768, 12, 64, 50304, 2, 1024, "fp16"),
        # the 410M configuration, 4 x 2048 tokens: the headline step
        _model("train_410m", "train", 1024, 24, 64, 50304, 4, 2048, "fp16"),
        # the 840M configuration: head_dim 128 and the long context
        _model("train_840m", "train", 1536, 24, 128, 50304, 1, 4096, "fp16"),
        # two layers of the 1.4B configuration: bf16, linear biases, ALiBi table
        _model("train_1b4_layers", "train", 2048, 2, 128, 50304, 2, 2048, "bf16", bias=True, alibi=True),
        # the shortest prompt on the 160M model: what one call costs when there is hardly any work
        _model("logits_160m_short", "logits", 768, 12, 64, 50304, 1, 64, "fp16"),
        # prompts padded to a multiple of 64 on the 410M model with ALiBi, a vocabulary that is no multiple of anything
        _model("logits_410m_ragged", "logits", 1024, 24, 64, 50257, 3, 704, "bf16", alibi=True),
        # the attention operator of the 410M configuration with ALiBi slopes
        {"name": "attention_slopes", "kind": "attention", "batch": 4, "heads": 16, "seq": 2048, "head_dim": 64,
         "dtype": "fp16", "bias": "slopes"},
        # a sequence that is an odd multiple of 64, a batch and a head count of no special form
        {"name": "attention_ragged", "kind": "attention", "batch": 3, "heads": 11, "seq": 1472, "head_dim": 64,
         "dtype": "bf16", "bias": "none"},
        # a linear layer with bias and ReLU whose sizes are multiples of nothing
        {"name": "linear_ragged", "kind": "linear", "batch": 5, "rows": 1003, "in": 1477, "out": 2930, "bias": True,
         "relu": True, "dtype": "fp16"},
        # softmax over rows of ordinary length in fp32, the one operator that takes it
        {"name": "softmax_fp32", "kind": "softmax", "batch": 16, "rows": 640, "cols": 1000, "dtype": "fp32"},
        # the optimizer step on the parameters of the 160M model's size
        {"name": "adamw_160m", "kind": "adamw", "tensors": 64, "numel": 768 * 3072, "dtype": "fp16"},
    ]


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["train", "train", "train", "logits", "logits", "attention", "attention", "attention", "linear",
                       "linear", "layernorm", "softmax", "loss", "adamw"])
    half = rng.choice(["fp16", "bf16"])
    if kind in ("train", "logits"):
        head_dim = rng.choice([32, 64, 64, 64, 128])
        heads = rng.randint(max(2, 192 // head_dim), 1536 // head_dim)
        c = {"kind": kind, "d": heads * head_dim, "head_dim": head_dim, "layers": rng.randint(1, 8),
             "vocab": rng.choice([_log(rng, 500, 50304), 64 * rng.randint(8, 786)]), "seq": 64 * _log(rng, 1, 32),
             "dtype": half, "bias": rng.random() < 0.3, "alibi": rng.random() < 0.3, "buckets": rng.random() < 0.6}
        if kind == "train":
            c["buckets"] = c["buckets"] or half == "bf16"  # bf16 needs no loss scale and is what large runs use
            c["layers"] = min(c["layers"], 2 if half == "bf16" else 8 if c["buckets"] else 4)
        c["batch"] = _log(rng, 1, max(1, min(16, 8192 // c["seq"])))
        return c
    if kind == "attention":
        c = {"kind": kind, "heads": rng.randint(4, 31), "seq": 64 * _log(rng, 1, 64),
             "head_dim": rng.choice([32, 64, 64, 128]), "dtype": half, "bias": rng.choice(["none", "none", "slopes", "table"])}
        c["batch"] = _log(rng, 1, max(1, min(8, 8192 // c["seq"])))
        return c
    if kind == "linear":
        ragged = rng.random() < 0.5
        size = (lambda low, high: _log(rng, low, high)) if ragged else (lambda low, high: 64 * _log(rng, low // 64, high // 64))
        return {"kind": kind, "batch": rng.randint(1, 7), "rows": size(64, 2048), "in": size(64, 4096),
                "out": size(64, 4096), "bias": rng.random() < 0.5, "relu": rng.random() < 0.5, "dtype": half}
    if kind == "layernorm":
        return {"kind": kind, "batch": rng.randint(1, 31), "rows": _log(rng, 64, 1024), "cols": _log(rng, 64, 2048), "dtype": half}
    if kind == "softmax":
        return {"kind": kind, "batch": rng.randint(1, 31), "rows": _log(rng, 64, 1024), "cols": _log(rng, 64, 1024),
                "dtype": rng.choice(["fp32", half])}
    if kind == "loss":
        return {"kind": kind, "rows": _log(rng, 1, 4096), "cols": _log(rng, 256, 64000), "dtype": half}
    return {"kind": kind, "tensors": rng.randint(4, 64), "numel": _log(rng, 4096, 768 * 3072), "dtype": half}


class _Draws:
    """Seeded values on the GPU."""

    def __init__(self, seed):
        self.gen = torch.Generator(device="cuda").manual_seed(seed)

    def normal(self, *shape, dtype=torch.float32, scale=1.0):
        return (torch.randn(shape, generator=self.gen, device="cuda") * scale).to(dtype)

    def integers(self, high, shape):
        return torch.randint(0, high, shape, generator=self.gen, device="cuda")


def _build_model(case, seed):
    """The configured architecture with weights N(0, 0.02), the LM head and the linear biases too (the initial head
    is zero, and every gradient but its own with it), and embeddings N(0, 1), the usual default.  The residual stream
    is then of unit size, as in a model under way, and a hidden unit whose pre-activation rounds to the other side of
    zero under the ReLU moves the gradients below it little; with a stream of size 0.03 it moves them by a few percent
    from one correct 16-bit implementation to the next."""
    torch.manual_seed(seed)
    config = TransformerConfig(
        vocab_size=case["vocab"], hidden_size=case["d"], max_position_embeddings=case["seq"],
        num_attention_heads=case["d"] // case["head_dim"], head_dim=case["head_dim"], ffn_dim=4 * case["d"],
        num_hidden_layers=case["layers"], use_linear_bias=case["bias"], attn_bias=case["alibi"])
    model = Transformer(config, device="cuda")
    with torch.no_grad():
        model.logits_out.weight.normal_(0.0, 0.02)
        for layer in model.layer_list:  # as in a model of 24 layers, whatever part of it the case runs
            for linear in (layer.attention.out_proj, layer.mlp.dense_4h_to_h):
                linear.weight.normal_(0.0, 0.02 / math.sqrt(48))
        model.embed_tokens.weight.normal_(0.0, 1.0)
        if model.embed_positions is not None:
            model.embed_positions.weight.normal_(0.0, 1.0)
        for name, p in model.named_parameters():
            if name.endswith("bias") and "layernorm" not in name:
                p.normal_(0.0, 0.02)
    if case["dtype"] == "bf16":
        table = model.attn_bias
        model = model.to(torch.bfloat16)
        if table is not None:
            model.attn_bias = table  # the ALiBi table keeps its fp16 rounding
    return model.fuse_projection_weights()


def prepare(case, seed):
    kind, dtype, draws = case["kind"], DTYPES[case["dtype"]], _Draws(seed)
    state = {"case": case}
    if kind in ("train", "logits"):
        state["ids"] = draws.integers(case["vocab"], (case["batch"], case["seq"]))
        state["model"] = model = _build_model(case, seed)
        if kind == "train" and case["buckets"]:
            state["buckets"] = GradBuckets(model.parameters(), bucket_bytes=128 << 20,
                                           column_blocks=model.projection_weight_groups())
    elif kind == "attention":
        b, h, t, hd = case["batch"], case["heads"], case["seq"], case["head_dim"]
        # head-split views of (B, T, H * head_dim) buffers, as the projections give them
        state["qkv"] = [draws.normal(b, t, h * hd, dtype=dtype).view(b, t, h, hd).transpose(1, 2).requires_grad_(True)
                        for _ in range(3)]
        state["grad"] = draws.normal(b, t, h * hd, dtype=dtype).view(b, t, h, hd).transpose(1, 2)
        if case["bias"] == "slopes":
            state["bias"] = torch.tensor(get_slopes(h), device="cuda")
        elif case["bias"] == "table":
            state["bias"] = generate_alibi_mask(t, h)[0]
    elif kind == "linear":
        n, k = case["out"], case["in"]
        args = [draws.normal(case["batch"], case["rows"], k, dtype=dtype), draws.normal(k, n, dtype=dtype, scale=k ** -0.5)]
        if case["bias"]:
            args.append(draws.normal(n, dtype=dtype, scale=0.02))
        state["args"] = [a.requires_grad_(True) for a in args]
        state["grad"] = draws.normal(case["batch"], case["rows"], n, dtype=dtype)
    elif kind in ("layernorm", "softmax"):
        shape = (case["batch"], case["rows"], case["cols"])
        args = [draws.normal(*shape, dtype=dtype)]
        if kind == "layernorm":
            args += [1.0 + draws.normal(case["cols"], dtype=dtype, scale=0.1), draws.normal(case["cols"], dtype=dtype, scale=0.1)]
        state["args"] = [a.requires_grad_(True) for a in args]
        state["grad"] = draws.normal(*shape, dtype=dtype)
    elif kind == "loss":
        state["args"] = [draws.normal(case["rows"], case["cols"], dtype=dtype).requires_grad_(True)]
        state["labels"] = draws.integers(case["cols"], (case["rows"],))
        state["grad"] = torch.full((case["rows"],), LOSS_SCALE[case["dtype"]] / case["rows"], device="cuda", dtype=dtype)
    else:
        params = [torch.nn.Parameter(draws.normal(case["numel"], dtype=dtype, scale=0.02)) for _ in range(case["tensors"])]
        state["buckets"] = buckets = GradBuckets(params, bucket_bytes=32 << 20)
        scale = LOSS_SCALE[case["dtype"]]
        state["optimizer"] = FusedAdamW(buckets, lr=1e-4, betas=(0.9, 0.95), weight_decay=0.1,
                                        scaler=LossScaler(torch.device("cuda"), init_scale=scale))
        for p in params:
            p.grad.copy_(draws.normal(case["numel"], scale=1e-4 * scale))
    return state


def _run_train(state):
    case, model, ids = state["case"], state["model"], state["ids"]
    dtype, scale, buckets = DTYPES[case["dtype"]], LOSS_SCALE[case["dtype"]], state.get("buckets")
    if buckets is None:
        model.zero_grad(set_to_none=True)
        with torch.autocast("cuda", dtype=dtype):
            logits, loss = model(ids, ids)
        (loss * scale).backward()
        grads = [p.grad for p in model.parameters()]
    else:
        buckets.zero(skip_written=True)
        with buckets.accumulate(overwrite=True, defer_weight_grads=True):
            with torch.autocast("cuda", dtype=dtype):
                logits, loss = model(ids, ids)
            (loss * scale).backward()
        grads = buckets.buckets
    return {"loss": loss.detach(), "logits": logits.detach(), "grads": grads}


def run(state):
    kind = state["case"]["kind"]
    if kind == "train":
        return _run_train(state)
    if kind == "logits":
        with torch.no_grad(), torch.autocast("cuda", dtype=DTYPES[state["case"]["dtype"]]):
            return state["model"](state["ids"], None)
    if kind == "adamw":
        opt = state["optimizer"]
        opt.step()
        return {"params": opt.params16, "master": opt.master, "exp_avg": opt.exp_avg, "exp_avg_sq": opt.exp_avg_sq,
                "scaler": opt.scaler.state}
    if kind == "attention":
        args = state["qkv"]
        if "bias" in state:
            out = tfb.fast_causal_attention_with_bias.apply(*args, state["bias"])
        else:
            out = tfb.fast_causal_attention.apply(*args)
    elif kind == "linear":
        args, c = state["args"], state["case"]
        fn = {(False, False): tfb.linear_no_bias, (False, True): tfb.linear_fused_relu, (True, False): tfb.linear_bias,
              (True, True): tfb.linear_fused_bias_relu}[(c["bias"], c["relu"])]
        out = fn.apply(*args)
    elif kind == "layernorm":
        args = state["args"]
        out = tfb.layer_norm.apply(*args, 1e-5)
    elif kind == "softmax":
        args = state["args"]
        out = tfb.softmax.apply(*args)
    else:
        args = state["args"]
        out = tfb.cross_entropy_loss.apply(*args, state["labels"])
    return (out.detach(),) + torch.autograd.grad(out, args, state["grad"])


def work(case):
    kind, e = case["kind"], 4 if case["dtype"] == "fp32" else 2
    if kind in ("train", "logits"):
        d, layers, vocab, tokens, seq = case["d"], case["layers"], case["vocab"], case["batch"] * case["seq"], case["seq"]
        matrices = layers * 12 * d * d + d * vocab
        params = matrices + d * vocab + (0 if case["alibi"] else d * seq) + layers * ((9 if case["bias"] else 4) * d) + 2 * d
        gathered = d * min(vocab, tokens)  # of the token table, only these rows can be read
        used = params - d * vocab + gathered
        flops = 2.0 * tokens * matrices + 2.0 * layers * tokens * seq * d
        if kind == "logits":
            return {"bytes": 8.0 * tokens + e * (used + tokens * vocab), "flops": flops}
        return {"bytes": 16.0 * tokens + 4 + e * (used + params + tokens * vocab),
                "flops": 6.0 * tokens * matrices + 7.0 * layers * tokens * seq * d}
    if kind == "attention":
        n = case["batch"] * case["heads"] * case["seq"] * case["head_dim"]
        return {"bytes": 8.0 * e * n, "flops": 7.0 * n * case["seq"]}
    if kind == "linear":
        m, k, n = case["batch"] * case["rows"], case["in"], case["out"]
        return {"bytes": e * (2.0 * m * k + 2.0 * k * n + 2.0 * m * n), "flops": 6.0 * m * n * k}
    if kind == "loss":
        n = case["rows"] * case["cols"]
        return {"bytes": 2.0 * e * n, "flops": 8.0 * n}
    if kind == "adamw":
        n = case["tensors"] * case["numel"]
        return {"bytes": 28.0 * n, "flops": 15.0 * n}
    n = case["batch"] * case["rows"] * case["cols"]
    return {"bytes": 4.0 * e * n, "flops": 16.0 * n}


def tolerance(case):
    if case["kind"] == "train":
        # part of a gradient's norm follows from hidden units whose pre-activation rounds to the other side of zero;
        # a single value can be off by as much as the values are large
        return {"rel": 0.025 if case["dtype"] == "bf16" else 0.02, "max": 0.99}
    if case["dtype"] == "fp32":
        return {"rel": 1e-5}
    if case["kind"] == "adamw":
        # fp32 state; the 16-bit parameters may round the other way
        return {"rel": 1e-4, "max": 1e-2}
    if case["kind"] == "linear" and case["relu"]:
        # the same, for the one ReLU of the operator
        return {"rel": 1e-2, "max": 0.9}
    return {"rel": 1e-2 if case["dtype"] == "bf16" else 3e-3, "max": 0.2}
