"""Performance cases of the HSTU attention path: what a training job and a serving process ask of
this package through its public functions.

Kinds of cases:

``mha``     ``hstu_mha`` on jagged q, k, v; forward only (inference) or forward and gradients
``fp8``     inference on e4m3 operands: ``quantize_e4m3_block`` of q, k, v, then ``hstu_mha_fp8``
``infer``   forward of an ``STUStack`` under ``no_grad``
``train``   forward and gradients (input and every parameter) of an ``STUStack`` in training mode
``cached``  ``STUStack.cached_forward``: new rows of every user against a kept K / V cache
``norms``   the two normalisations of a layer in training: ``layer_norm`` and
            ``hstu_norm_mul_dropout``, forward and gradients
``embed``   the steps around a stack in training: contextual rows in front of the sequence
            (``concat_2D_jagged``), position and time embeddings (``HSTUPositionalEncoder``),
            candidates split off (``split_2D_jagged``), forward and gradients

The lengths of a batch are quantiles of the case's distribution, so that a case always has the same
amount of work; the seed orders the sequences and draws all values.
"""

import functools
import math

import numpy as np
import torch

import generative_recommenders_b200 as hstu

_DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}

# what a case says only where it differs from this
_DEFAULTS = {
    "dtype": "bf16",      # of activations and weights
    "grad": False,        # (mha) forward and gradients
    "batch": 1,           # sequences
    "heads": 4,
    "dim": 128,           # of a head, for q / k and for v
    "width": 512,         # embedding dimension of a layer
    "layers": 1,
    "max_len": 1024,      # max_seq_len of the call
    "low": 1,             # shortest sequence
    "lengths": "uniform",
    "targets": 0,         # num_targets: 1 .. targets per sequence
    "all_targets": False,  # every sequence has exactly `targets`
    "context": 0,         # contextual_seq_len
    "window": 0,          # max_attn_len
    "full_tail": 0,       # min_full_attn_seq_len
    "bias": False,        # (mha) relative position bias by distance, trained where there are gradients
    "dropout": 0.0,       # output dropout
    "recompute": True,    # (train) the layers' recompute switches
    "delta": 0,           # (cached) new rows per user
    "rows": 0,            # (norms)
    "act": "none",        # (norms) activation on u
}


def listed():
    return [
        # The smallest call in 32 bits: a numerics check or a small research model.
        {"name": "mha_fp32_small", "kind": "mha", "dtype": "fp32", "grad": True, "batch": 16, "heads": 2, "dim": 32,
         "max_len": 256},
        # The training step of a ranking model's attention, the headline benchmark's sizes.
        {"name": "mha_train", "kind": "mha", "grad": True, "batch": 64, "max_len": 1024, "low": 128, "targets": 32},
        # Long user histories in fp16 with 64-wide heads: window, contextual prefix, full tail and odd
        # sizes together.
        {"name": "mha_train_window_fp16", "kind": "mha", "dtype": "fp16", "grad": True, "batch": 23, "heads": 6,
         "dim": 64, "max_len": 3001, "low": 37, "targets": 50, "context": 5, "window": 517, "full_tail": 100},
        # A research model that trains a relative position bias; most sequences short, a few long.
        {"name": "mha_train_bias", "kind": "mha", "grad": True, "batch": 128, "max_len": 4096, "low": 16,
         "lengths": "power", "targets": 64, "context": 6, "bias": True},
        # Scoring of 256 candidates per user against long histories in a local window.
        {"name": "mha_infer_window", "kind": "mha", "batch": 256, "max_len": 8192, "low": 320, "lengths": "zipf",
         "targets": 256, "all_targets": True, "window": 1024},
        # The same traffic on quantised operands.
        {"name": "fp8_infer_window", "kind": "fp8", "batch": 256, "max_len": 8192, "low": 320, "lengths": "zipf",
         "targets": 256, "all_targets": True, "window": 1024},
        # One ranking request: a handful of users through a serving stack; latency.
        {"name": "infer_request", "kind": "infer", "layers": 4, "batch": 4, "max_len": 700, "low": 150, "targets": 64,
         "all_targets": True, "context": 6},
        # One GPU's share of bulk ranking with a wide model and long histories.
        {"name": "infer_bulk", "kind": "infer", "layers": 4, "batch": 256, "heads": 8, "width": 1024,
         "max_len": 16384, "low": 81, "lengths": "lognormal", "targets": 64, "all_targets": True, "context": 16},
        # Candidates scored against users' kept K / V.
        {"name": "cached_request", "kind": "cached", "layers": 4, "batch": 32, "max_len": 1024, "low": 64, "delta": 20,
         "context": 6},
        # A training step of a deep stack on a batch of mostly short sequences.
        {"name": "train_deep", "kind": "train", "layers": 8, "batch": 128, "max_len": 4096, "low": 16,
         "lengths": "power", "targets": 64, "context": 6, "dropout": 0.3},
        # A training step of the two normalisations on a large batch.
        {"name": "norms_train", "kind": "norms", "rows": 200003, "heads": 4, "dim": 128, "width": 512, "dropout": 0.3},
        # A training step of the embedding of the sequences, before the first layer.
        {"name": "embed_train", "kind": "embed", "batch": 250, "width": 512, "max_len": 2048, "low": 64,
         "targets": 20, "context": 4},
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    """One more case of the listed kinds, sizes spread over the range from the smallest request to
    the largest batch."""
    most = max(_cost(c) for c in listed())
    while True:
        c = _draw_one(rng)
        if _cost(c) <= most:
            return c


def _cost(case):
    w = work(case)
    return max(w["bytes"], w["flops"] / 50)


def _draw_one(rng):
    kind = rng.choice(["mha", "mha", "mha", "fp8", "infer", "infer", "cached", "train", "train", "norms", "embed"])
    c = {"kind": kind, "dtype": rng.choice(["bf16", "bf16", "bf16", "fp16"])}
    if kind == "norms":
        c["heads"], c["dim"] = rng.choice([(4, 64), (2, 128), (4, 128), (8, 64), (6, 128), (8, 128)])
        c["width"] = rng.choice([256, 512, 768, 1024])
        c["rows"] = _log_int(rng, 300, 300000)
        c["dropout"] = rng.choice([0.0, 0.1, 0.3])
        c["act"] = rng.choice(["none", "none", "silu"])
        return c
    # batches from one request to a training batch, sequences from short to long, most of them odd
    tokens = _log_int(rng, 1000, {"mha": 300000, "infer": 300000, "embed": 300000, "train": 60000}.get(kind, 200000))
    longest = _log_int(rng, 100, 8192 if kind != "train" else 4096)
    c["max_len"] = longest
    c["low"] = rng.randint(20, max(20, min(longest, 200)))
    c["lengths"] = rng.choice(["uniform", "uniform", "power", "zipf", "lognormal"])
    c["context"] = rng.choice([0, 0, 3, 6, 16])
    c["targets"] = rng.choice([0, 1, 20, 64, 200])
    c["all_targets"] = rng.random() < 0.3
    c["batch"] = 1
    mean = float(_quantiles(dict(_DEFAULTS, **dict(c, batch=64))).mean())
    c["batch"] = min(1024, max(1, int(tokens / mean)))
    if kind == "mha":
        c["grad"] = rng.random() < 0.5
        c["heads"], c["dim"] = rng.choice([(4, 128), (2, 128), (8, 128), (4, 64), (8, 64), (3, 64)])
        if rng.random() < 0.15:   # 32 bits are for checks and small models
            c.update(dtype="fp32", heads=2, dim=rng.choice([32, 64]), max_len=min(longest, 512))
            c["low"] = min(c["low"], c["max_len"])
            c["batch"] = min(c["batch"], 32)
        if rng.random() < 0.4:
            c["window"] = rng.choice([100, 256, 517, 1024])
            c["full_tail"] = rng.choice([0, 0, 100])
        c["bias"] = c["dtype"] != "fp32" and rng.random() < 0.2
    elif kind == "fp8":
        c.update(dtype="bf16", heads=rng.choice([2, 4, 8]), window=rng.choice([0, 256, 1024]))
    elif kind == "embed":
        c["width"] = rng.choice([256, 512, 1024])
        c["targets"] = max(1, c["targets"])
    else:
        c["width"], c["heads"], c["dim"] = rng.choice([(256, 4, 64), (512, 4, 128), (512, 8, 64), (768, 6, 128),
                                                       (1024, 8, 128)])
        c["layers"] = rng.randint(1, 4) if kind == "train" else rng.randint(2, 8)
        c["window"] = rng.choice([0, 0, 0, 256])
        if kind == "train":
            c["dropout"] = rng.choice([0.0, 0.1, 0.3])
            c["recompute"] = rng.random() < 0.5
        if kind == "cached":
            c["delta"] = rng.choice([1, 7, 20, 64, 128])
            c["batch"] = min(c["batch"], 256)
            c["targets"] = 0
            c["all_targets"] = False
    return c


# ------------------------------------------------------------------------------------------------
# sizes
# ------------------------------------------------------------------------------------------------
def _full(case):
    return dict(_DEFAULTS, **case)


def _quantiles(c):
    """Sequence lengths of the batch: evenly spaced quantiles of the distribution, [B] int64."""
    low, high = c["low"], c["max_len"]
    u = (np.arange(c["batch"]) + 0.5) / c["batch"]
    if c["lengths"] == "uniform":
        n = low + np.floor(u * (high - low + 1))
    elif c["lengths"] == "power":        # Pareto, exponent 1.2: many short sequences, few long ones
        n = np.floor(low * (1.0 - u) ** (-1.0 / 1.2))
    elif c["lengths"] == "zipf":         # exponent 1.1: a third shortest, half cut off at the longest
        n = np.floor((1.0 - u) ** (-1.0 / 0.1))
    elif c["lengths"] == "lognormal":    # median 1100, one e-fold either way
        n = np.round(np.exp(7.0 + np.array([math.sqrt(2) * _erfinv(2 * v - 1) for v in u])))
    else:
        raise ValueError(c["lengths"])
    least = c["context"] + 2
    return np.clip(n, max(low, least), max(high, least)).astype(np.int64)


def _erfinv(y):
    return float(torch.erfinv(torch.tensor(y, dtype=torch.float64)))


def _batch(c):
    """(lengths, targets) of the batch; targets leave at least one history row beside the prefix."""
    lengths = _quantiles(c)
    t = c["targets"]
    if t == 0:
        return lengths, np.zeros_like(lengths)
    # spread over 1 .. t, in an order that has nothing to do with the lengths
    targets = np.full_like(lengths, t) if c["all_targets"] else 1 + (np.arange(len(lengths)) * 7919) % t
    return lengths, np.minimum(targets, lengths - c["context"] - 1)


def _pairs(c):
    """Visible (query, key) pairs of the batch."""
    lengths, targets = _batch(c)
    return sum(_pairs_of(int(n), int(t), c["context"], c["window"], c["full_tail"]) for n, t in zip(lengths, targets))


@functools.lru_cache(maxsize=100000)
def _pairs_of(n, t, ctx, window, tail):
    u = n - t                                    # rows of prefix and history
    first = max(ctx - 1, 0)                      # prefix rows share one id with what comes before row ctx
    top = n - first - t                          # id of a target
    ids = np.minimum(np.maximum(np.arange(u, dtype=np.int64) - first, 0), top) if ctx else np.arange(u)
    rows = np.append(ids[ctx:], top)             # a history row each, and what every target row sees
    seen = rows if ctx == 0 else rows - 1        # history keys with a smaller id
    pre = np.full_like(rows, ctx)
    if window:
        near = (rows <= window) | ((rows >= top - tail) & (tail > 0))
        full = (rows >= top - tail) & (tail > 0)
        seen = np.where(full, seen, np.minimum(seen, window))
        pre = np.where(near, ctx, 0)
    per = np.maximum(seen, 0) + pre + 1
    return int(per[:-1].sum() + t * per[-1] + min(ctx, u) * u)


def work(case):
    c = _full(case)
    s = 4 if c["dtype"] == "fp32" else 2
    H, d, D = c["heads"], c["dim"], c["width"]
    hd = H * d
    if c["kind"] == "norms":
        # forward: x -> y; attn, u -> [u, attn, y].  backward: dy, x -> dx; d[u, attn, y], attn, u -> two
        n = c["rows"]
        return {"bytes": n * s * (2 * D + 3 * D + 5 * hd + 7 * hd), "flops": n * (30 * D + 60 * hd)}
    lengths, targets = _batch(c)
    B, L = len(lengths), int(lengths.sum())
    if c["kind"] == "embed":
        x = 2 * L * D * s                        # read and written once each way
        return {"bytes": 2 * x + 8 * L, "flops": 8.0 * L * D}
    pairs = _pairs(c)
    if c["kind"] == "mha":
        flops, bytes_ = 4.0 * hd * pairs, 4 * L * hd * s
        if c["grad"]:
            flops, bytes_ = 3.5 * flops, bytes_ + 7 * L * hd * s
        return {"bytes": bytes_, "flops": flops}
    if c["kind"] == "fp8":
        return {"bytes": 3 * L * hd * (2 + 1) + L * hd * (3 + 2), "flops": 4.0 * hd * pairs}
    weights = D * 4 * hd + 3 * hd * D
    if c["kind"] == "cached":
        n, seen = B * c["delta"], int((lengths + 1).sum()) * c["delta"]
        return {"bytes": c["layers"] * s * (2 * L * hd + weights) + 2 * n * D * s,
                "flops": c["layers"] * (2.0 * n * weights + 4.0 * hd * seen)}
    flops = c["layers"] * (2.0 * L * weights + 4.0 * hd * pairs)
    bytes_ = c["layers"] * s * weights + 2 * L * D * s
    if c["kind"] == "train":
        flops = c["layers"] * (6.0 * L * weights + 14.0 * hd * pairs)
        bytes_ = c["layers"] * s * (3 * weights) + 4 * L * D * s
    return {"bytes": bytes_, "flops": flops}


def tolerance(case):
    c = _full(case)
    if c["dtype"] == "fp32":
        return {"rel": 1e-5, "max": 1e-3}
    if c["kind"] in ("infer", "cached", "train"):
        # a chain of 16-bit stages, each of which rounds its results, through several layers
        return {"rel": 2e-2, "max": 0.8}
    return {"rel": 1e-2, "max": 0.4}


# ------------------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------------------
class _Draw:
    def __init__(self, c, seed):
        self.dtype = _DTYPES[c["dtype"]]
        self.gen = torch.Generator(device="cuda").manual_seed(seed)
        self.rng = np.random.RandomState(seed % (1 << 31))

    def normal(self, *shape, std=1.0, dtype=None):
        x = torch.randn(*shape, generator=self.gen, device="cuda", dtype=torch.float32)
        return x.mul_(std).to(dtype or self.dtype)

    def sequences(self, c):
        """(lengths, offsets, targets) on the GPU, int64, in the seed's order."""
        lengths, targets = _batch(c)
        order = self.rng.permutation(len(lengths))
        host = torch.from_numpy(np.stack([lengths[order], targets[order]])).cuda()
        lengths, targets = host[0].contiguous(), host[1].contiguous()
        return lengths, _offsets(lengths), targets if c["targets"] else None


def _offsets(lengths):
    return torch.cat([lengths.new_zeros(1), torch.cumsum(lengths, 0)])


def _stack(c, draw, seed):
    """An STUStack with weights as initialised; norms and biases moved off their initial ones and
    zeros, as training does."""
    torch.manual_seed(seed)
    config = hstu.STULayerConfig(
        embedding_dim=c["width"], num_heads=c["heads"], hidden_dim=c["dim"], attention_dim=c["dim"],
        output_dropout_ratio=c["dropout"], max_attn_len=c["window"] or None, contextual_seq_len=c["context"],
        recompute_normed_x=c["recompute"], recompute_uvqk=c["recompute"], recompute_y=c["recompute"])
    with torch.device("cuda"):
        stack = hstu.STUStack([hstu.STULayer(config) for _ in range(c["layers"])])
    with torch.no_grad():
        for p in stack.parameters():
            if p.dim() == 1:
                p.add_(draw.normal(*p.shape, std=0.05, dtype=torch.float32))
    return stack.to(draw.dtype).train(c["kind"] == "train")


def prepare(case, seed):
    c = _full(case)
    draw_ = _Draw(c, seed)
    return c, _PREPARE[c["kind"]](c, draw_, seed)


def _prepare_mha(c, draw, seed):
    lengths, offsets, targets = draw.sequences(c)
    L, H, d = int(_batch(c)[0].sum()), c["heads"], c["dim"]
    q, k, v = (draw.normal(L, H, d, std=0.5).requires_grad_(c["grad"]) for _ in range(3))
    bias = None
    if c["bias"]:
        bias = draw.normal(c["max_len"], std=0.1, dtype=torch.float32).requires_grad_(c["grad"])
    return {"qkv": (q, k, v), "bias": bias, "offsets": offsets, "targets": targets,
            "dout": draw.normal(L, H, d) if c["grad"] else None}


def _prepare_fp8(c, draw, seed):
    _, offsets, targets = draw.sequences(c)
    L = int(_batch(c)[0].sum())
    return {"qkv": tuple(draw.normal(L, c["heads"], c["dim"]) for _ in range(3)), "offsets": offsets,
            "targets": targets}


def _prepare_stack(c, draw, seed):
    lengths, offsets, targets = draw.sequences(c)
    L = int(_batch(c)[0].sum())
    train = c["kind"] == "train"
    stack = _stack(c, draw, seed)
    return {"stack": stack, "x": draw.normal(L, c["width"]).requires_grad_(train), "lengths": lengths,
            "offsets": offsets, "targets": targets, "dy": draw.normal(L, c["width"]) if train else None,
            "params": list(stack.parameters()), "seed": seed}


def _prepare_cached(c, draw, seed):
    lengths, offsets, _ = draw.sequences(c)
    L, B = int(_batch(c)[0].sum()), c["batch"]
    stack = _stack(c, draw, seed)
    longest = int(_batch(c)[0].max())
    with torch.no_grad():
        stack(draw.normal(L, c["width"]), lengths, offsets, longest, None, max_kv_caching_len=longest,
              kv_caching_lengths=lengths)
    return {"stack": stack, "x": draw.normal(B * c["delta"], c["width"]),
            "targets": torch.full((B,), c["delta"], dtype=torch.int64, device="cuda")}


def _prepare_norms(c, draw, seed):
    n, D, hd = c["rows"], c["width"], c["heads"] * c["dim"]

    def affine(width):
        return (draw.normal(width, std=0.05) + 1).requires_grad_(), draw.normal(width, std=0.05).requires_grad_()

    return {"x": draw.normal(n, D).requires_grad_(), "norm": affine(D), "dy": draw.normal(n, D),
            "attn": draw.normal(n, hd, std=0.2).requires_grad_(), "u": draw.normal(n, hd, std=0.5).requires_grad_(),
            "out_norm": affine(hd), "dcat": draw.normal(n, 3 * hd),
            "dropout_seed": torch.randint(0, 2 ** 62, (1,), generator=draw.gen, device="cuda")}


def _prepare_embed(c, draw, seed):
    lengths, targets = _batch(c)
    order = draw.rng.permutation(len(lengths))
    lengths, targets = (torch.from_numpy(t[order]).cuda() for t in (lengths, targets))
    L, T, B, D, ctx = int(lengths.sum()), int(targets.sum()), c["batch"], c["width"], c["context"]
    torch.manual_seed(seed)
    with torch.device("cuda"):
        encoder = hstu.HSTUPositionalEncoder(num_position_buckets=int(c["max_len"]), num_time_buckets=2048,
                                             embedding_dim=D, contextual_seq_len=ctx, is_inference=False)
    gaps = (torch.rand(L, generator=draw.gen, device="cuda") * 12).exp().long()
    return {"encoder": encoder.to(draw.dtype), "rows": (L, T, int((lengths - targets).max()), c["targets"]),
            "prefix": draw.normal(B * ctx, D).requires_grad_() if ctx else None,
            "x": draw.normal(L - B * ctx, D).requires_grad_(), "lengths": lengths, "targets": targets,
            "offsets": _offsets(lengths), "own": _offsets(lengths - ctx), "target_offsets": _offsets(targets),
            "history_offsets": _offsets(lengths - targets), "stamps": torch.cumsum(gaps, 0),
            "d_history": draw.normal(L - T, D), "d_targets": draw.normal(T, D)}


_PREPARE = {"mha": _prepare_mha, "fp8": _prepare_fp8, "infer": _prepare_stack, "train": _prepare_stack,
            "cached": _prepare_cached, "norms": _prepare_norms, "embed": _prepare_embed}


# ------------------------------------------------------------------------------------------------
# one pass
# ------------------------------------------------------------------------------------------------
def run(state):
    c, s = state
    return _RUN[c["kind"]](c, s)


def _run_mha(c, s):
    q, k, v = s["qkv"]
    out = hstu.hstu_mha(
        max_seq_len=c["max_len"], alpha=1.0 / c["dim"], q=q, k=k, v=v, seq_offsets=s["offsets"], causal=True,
        training=c["grad"], num_targets=s["targets"], max_attn_len=c["window"], contextual_seq_len=c["context"],
        min_full_attn_seq_len=c["full_tail"], bias_by_distance=s["bias"])
    if not c["grad"]:
        return out
    of = (q, k, v) if s["bias"] is None else (q, k, v, s["bias"])
    return out.detach(), torch.autograd.grad(out, of, s["dout"])


def _run_fp8(c, s):
    offsets = s["offsets"]
    q8, q_scale, blocks = hstu.quantize_e4m3_block(s["qkv"][0], offsets)
    k8, k_scale, _ = hstu.quantize_e4m3_block(s["qkv"][1], offsets, blocks)
    v8, v_scale, _ = hstu.quantize_e4m3_block(s["qkv"][2], offsets, blocks)
    return hstu.hstu_mha_fp8(c["max_len"], 1.0 / c["dim"], q8, k8, v8, q_scale, k_scale, v_scale, blocks, offsets,
                             num_targets=s["targets"], max_attn_len=c["window"], contextual_seq_len=c["context"])


def _run_infer(c, s):
    with torch.no_grad():
        return s["stack"](s["x"], s["lengths"], s["offsets"], c["max_len"], s["targets"])


def _run_train(c, s):
    if c["dropout"]:
        torch.cuda.manual_seed(s["seed"])        # the same masks on every pass over this state
    y = s["stack"](s["x"], s["lengths"], s["offsets"], c["max_len"], s["targets"])
    return y.detach(), torch.autograd.grad(y, [s["x"]] + s["params"], s["dy"])


def _run_cached(c, s):
    with torch.no_grad():
        return s["stack"].cached_forward(s["x"], s["targets"])


def _run_norms(c, s):
    y = hstu.layer_norm(s["x"], s["norm"][0], s["norm"][1], 1e-6)
    d_first = torch.autograd.grad(y, (s["x"],) + s["norm"], s["dy"])
    cat = hstu.hstu_norm_mul_dropout(
        s["attn"], s["u"], s["out_norm"][0], s["out_norm"][1], 1e-6, c["dropout"], True, concat_u=True, concat_x=True,
        mul_u_activation_type=c["act"], num_heads=c["heads"], linear_dim=c["dim"],
        dropout_seed=s["dropout_seed"] if c["dropout"] else None)
    d_second = torch.autograd.grad(cat, (s["attn"], s["u"]) + s["out_norm"], s["dcat"])
    return y.detach(), d_first, cat.detach(), d_second


def _run_embed(c, s):
    L, T, longest_history, most_targets = s["rows"]
    x = s["x"]
    if c["context"]:
        x = hstu.concat_2D_jagged(c["max_len"], s["prefix"], x, max_len_left=c["context"],
                                  max_len_right=c["max_len"] - c["context"], offsets_right=s["own"])
    x = s["encoder"](c["max_len"], s["lengths"], s["offsets"], s["stamps"], x, s["targets"])
    history, targets = hstu.split_2D_jagged(
        c["max_len"], x, total_len_left=L - T, total_len_right=T, max_len_left=longest_history,
        max_len_right=most_targets, offsets_left=s["history_offsets"], offsets_right=s["target_offsets"])
    of = [t for t in (s["prefix"], s["x"]) if t is not None] + list(s["encoder"].parameters())
    grads = torch.autograd.grad((history, targets), of, (s["d_history"], s["d_targets"]))
    return history.detach(), targets.detach(), grads


_RUN = {"mha": _run_mha, "fp8": _run_fp8, "infer": _run_infer, "train": _run_train, "cached": _run_cached,
        "norms": _run_norms, "embed": _run_embed}
