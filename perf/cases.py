"""The work a user of this framework has it do, as cases that can be timed and compared.

Each case is one call (or one short sequence of calls) through the public entry points: training steps of the decoder
and of the memory transformer through `nn.DecoderLm`, evaluation and generation through `generation`, and the two
groups of eager ops that a program with a model of its own builds on, causal attention and linear layers (`cuda`).
Sizes come from the repository's benchmark, its kernel sweep and its tests, or are generic.

A case is a plain dict; `kind` says which path it takes:

    train      one optimizer step: host tokens in, loss out (`DecoderLm.train_step`), or forward_backward and
               optimizer_step_policy for a memory transformer with one of its update policies
    eval       `generation.evaluate_token_loss` over a token stream
    generate   `generation.generate`: a prefix in, new tokens out
    attention  flash attention forward and backward on a fused q/k/v buffer
    linear     a linear layer forward and backward (bf16: with bias and GELU; f32: with bias)
"""
import math

import numpy as np
import torch

from heirloom_b200 import cuda, generation, nn

GPT_124M = dict(vocab=50304, d_model=768, n_layers=12, n_heads=12, d_ff=3072, context=1024)
MEMORY = dict(vocab=32000, d_model=512, n_layers=8, n_heads=8, d_ff=2048, context=512)
TABLES = dict(memory_layers="4,6", slots=262144, key_dim=512, value_dim=512, top_k=32)
SMALL = dict(vocab=512, d_model=128, n_layers=2, n_heads=2, d_ff=256, context=128)
TINY = dict(vocab=256, d_model=128, n_layers=4, n_heads=4, d_ff=512, context=64)
BATCHES = 4  # token batches a training program has at hand; each step takes the next one
NO_EOS = 1 << 40


def listed():
    return [
        # a small model in a unit test or a parameter sweep: every kernel is short, launches and host work count
        dict(name="train_small_bf16", kind="train", precision="bf16", batch=2, clip=0.0, **SMALL),
        # the byte-level model on the reference's own precision (f32 values, f64 sums)
        dict(name="train_tiny_f32", kind="train", precision="f32", batch=16, clip=0.0, **TINY),
        # nothing is a multiple of a tile, heads of 32 channels, gradient clipping
        dict(name="train_ragged_bf16", kind="train", precision="bf16", batch=7, clip=1.0, vocab=1000, d_model=192, n_layers=3,
             n_heads=6, d_ff=776, context=100),
        # an ordinary step: a middle-sized decoder at a small batch with clipping
        dict(name="train_dense_bf16", kind="train", precision="bf16", batch=8, clip=1.0, **MEMORY),
        # the benchmark's training step
        dict(name="train_gpt_124m", kind="train", precision="bf16", batch=16, clip=0.0, **GPT_124M),
        # the memory transformer, pre-training (every parameter) ...
        dict(name="train_memory_full", kind="train", precision="bf16", batch=32, clip=0.0, policy="full", **MEMORY, **TABLES),
        # ... and sparse fine-tuning of the rows that were looked up
        dict(name="train_memory_sparse_rows", kind="train", precision="bf16", batch=4, clip=1.0, policy="sparse_rows", **MEMORY,
             **TABLES),
        # held-out loss between training steps: a full batch of windows and a rest
        dict(name="eval_gpt_124m", kind="eval", precision="bf16", batch=16, windows=19, **GPT_124M),
        # greedy continuation of half a context
        dict(name="generate_gpt_124m", kind="generate", precision="bf16", batch=1, prefix=500, new=8, temperature=0.0, top_k=0,
             top_p=1.0, repetition=1.0, **GPT_124M),
        # sampled bytes with every control in use, past the end of the context
        dict(name="generate_tiny_f32", kind="generate", precision="f32", batch=1, prefix=40, new=32, temperature=0.8, top_k=40,
             top_p=0.95, repetition=1.1, **TINY),
        # a program with its own model: long sequences, wide heads
        dict(name="attention_t4096", kind="attention", batch=4, time=4096, heads=12, head_dim=128),
        # ... and the first layer of its feed-forward at a row count that is no multiple of anything
        dict(name="linear_ragged_bf16", kind="linear", precision="bf16", rows=4099, inputs=768, outputs=3072),
    ]


# ---- drawn cases ---------------------------------------------------------------------------------------------------
MOST_FLOPS = 1.3e13      # the benchmark's training step
MOST_F32_FLOPS = 1.0e10  # f32 products sum in f64: the same time takes far fewer of them


def _spread(rng, low, high, multiple=1):
    """A whole number between the two, evenly over its logarithm, a multiple of `multiple`."""
    x = math.exp(rng.uniform(math.log(low), math.log(high)))
    return min(high // multiple, max(-(-low // multiple), round(x / multiple))) * multiple


def _model(rng, precision):
    if precision == "f32":
        heads = _spread(rng, 1, 6)
        d = heads * rng.choice([16, 32, 64])
        time = _spread(rng, 8, 128)
        return dict(precision=precision, vocab=_spread(rng, 64, 1024, 8), d_model=d, n_layers=_spread(rng, 1, 6), n_heads=heads,
                    d_ff=_spread(rng, d, 4 * d, 4), context=time, batch=max(1, _spread(rng, 32, 2048) // time))
    head = rng.choice([64, 64, 64, 64, 128, 128, 32])
    heads = _spread(rng, 1, 256 // head if head == 32 else 768 // head)
    d = head * heads
    time = _spread(rng, 16, 200 if head == 32 else 1024)
    return dict(precision=precision, vocab=_spread(rng, 256, 50304, 8), d_model=d, n_layers=_spread(rng, 1, 12), n_heads=heads,
                d_ff=_spread(rng, 2 * d, 4 * d, 8), context=time, batch=max(1, _spread(rng, 64, 2048 if head == 32 else 16384) // time))


def _memory_model(rng, precision):
    small = precision == "f32"
    heads = _spread(rng, 1, 2 if small else 8)
    layers = _spread(rng, 2, 3 if small else 8)
    where = sorted({layers // 2, layers - 1} if rng.random() < 0.6 else {layers // 2})
    time = _spread(rng, 16, 64 if small else 512, 16)
    side = _spread(rng, 32, 64 if small else 512)
    return dict(precision=precision, vocab=_spread(rng, 256, 1024 if small else 32000, 8), d_model=64 * heads, n_layers=layers,
                n_heads=heads, d_ff=_spread(rng, 128 * heads, 256 * heads, 8), context=time,
                batch=4 * max(1, _spread(rng, 64, 1024 if small else 16384) // (4 * time)),
                memory_layers=",".join(map(str, where)), slots=side * side, key_dim=_spread(rng, 64, 64 if small else 512, 64),
                value_dim=_spread(rng, 64, 64 if small else 512, 64), top_k=rng.choice([4, 8, 16, 32]))


def draw(rng):
    kind = rng.choices(["train", "memory", "eval", "generate", "attention", "linear"], [6, 2, 1, 2, 1, 1])[0]
    precision = rng.choices(["bf16", "f32"], [3, 1])[0]
    while True:
        if kind == "train":
            case = dict(kind=kind, clip=rng.choice([0.0, 1.0]), **_model(rng, precision))
        elif kind == "memory":
            case = dict(kind="train", clip=rng.choice([0.0, 1.0]), **_memory_model(rng, precision),
                        policy=rng.choice(["full", "full", "sparse_rows", "dense_plus_sparse_values", "memory_only"]))
        elif kind == "eval":
            model = _model(rng, precision)
            case = dict(kind=kind, windows=rng.randint(1, 2 * model["batch"]), **model)
        elif kind == "generate":
            model = dict(_model(rng, precision), batch=1)
            if model["d_model"] < 64:  # too narrow to tell a vocabulary's tokens apart: every step would be a near-tie
                continue
            sampled = rng.random() < 0.5
            case = dict(kind=kind, prefix=_spread(rng, 1, model["context"]), new=_spread(rng, 4, 32),
                        temperature=0.8 if sampled else 0.0, top_k=40 if sampled else 0, top_p=0.95 if sampled else 1.0,
                        repetition=1.1 if sampled else 1.0, **model)
        elif kind == "attention":
            time = _spread(rng, 64, 4096)
            case = dict(kind=kind, batch=max(1, _spread(rng, 64, 16384) // time), time=time, heads=_spread(rng, 1, 16),
                        head_dim=rng.choice([64, 128]))
        else:
            most = (16384, 4096) if precision == "bf16" else (1024, 768)
            case = dict(kind=kind, precision=precision, rows=_spread(rng, 64, most[0]), inputs=_spread(rng, 64, most[1], 8),
                        outputs=_spread(rng, 64, most[1], 8))
        if work(case)["flops"] <= (MOST_F32_FLOPS if case.get("precision") == "f32" else MOST_FLOPS):
            return case


# ---- inputs --------------------------------------------------------------------------------------------------------
_contexts = []


def _context():
    """The one context that a program keeps."""
    if not _contexts:
        _contexts.append(cuda.Context(0))
    return _contexts[0]


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _zipf(gen, vocab, shape):
    """Token ids with the frequencies of text: Zipf, exponent 1.1."""
    cdf = torch.cumsum(torch.arange(1, vocab + 1, dtype=torch.float64, device="cuda") ** -1.1, 0)
    u = torch.rand(shape, generator=gen, device="cuda", dtype=torch.float64) * cdf[-1]
    return torch.searchsorted(cdf, u).clamp_(max=vocab - 1)


def _decoder(case, gen):
    """The model with fresh weights: N(0, 0.02), residual projections scaled down, half keys of unit length.

    A model that generates has learnt something: its head gives each token's successor (a fixed permutation) most of
    the probability, as a trained model does, instead of the near-ties of random weights."""
    precision = nn.PRECISION_F32 if case["precision"] == "f32" else nn.PRECISION_AMP_BF16
    cfg = nn.DecoderConfig(precision=precision, **{k: case[k] for k in ("vocab", "d_model", "n_layers", "n_heads", "d_ff", "context", "batch")})
    memory = None
    if "slots" in case:
        memory = nn.MemoryConfig(memory_layers=tuple(int(x) for x in case["memory_layers"].split(",")),
                                 **{k: case[k] for k in ("slots", "key_dim", "value_dim", "top_k")})
    model = nn.DecoderLm(_context(), cfg, memory)
    learnt = case["kind"] == "generate"
    state = {}
    for name, shape in model.parameter_shapes().items():
        if name.endswith(".bias"):
            w = torch.zeros(shape)
        elif ".ln" in name or name.startswith("ln_f"):
            w = torch.ones(shape)
        else:
            w = torch.randn(shape, generator=gen, device="cuda") * 0.02
            if "out_proj" in name or "fc2" in name:
                w *= (2.0 * case["n_layers"]) ** -0.5
            elif "product_key" in name:
                w *= 50.0 * shape[-1] ** -0.5
            elif name == "token_embedding.weight" and learnt:
                w *= 25.0
                embedding = w
            elif name == "lm_head.weight" and learnt:
                w[torch.randperm(case["vocab"], generator=gen, device="cuda")] = embedding * (40.0 / case["d_model"])
        state[name] = w.cpu().numpy()
    model.load_state_dict(state)
    return model


def prepare(case, seed):
    gen = _generator(seed)
    ctx = _context()
    kind = case["kind"]
    if kind == "train":
        model = _decoder(case, gen)
        model.set_optimizer(lr=3e-4, weight_decay=0.01, clip_norm=case["clip"] or None)
        tokens = _zipf(gen, case["vocab"], (BATCHES, case["batch"], case["context"] + 1))
        pairs = [(t[:, :-1].contiguous(), t[:, 1:].contiguous()) for t in tokens]
        if "policy" not in case:  # the loader hands out pinned host memory
            pairs = [(x.cpu().pin_memory(), y.cpu().pin_memory()) for x, y in pairs]
        return dict(kind=kind, model=model, pairs=pairs, step=0, policy=case.get("policy"))
    if kind == "eval":
        model = _decoder(case, gen)
        stream = _zipf(gen, case["vocab"], (case["windows"] * case["context"] + 1,)).cpu().numpy()
        return dict(kind=kind, model=model, stream=stream, batch=case["batch"])
    if kind == "generate":
        model = _decoder(case, gen)
        options = generation.GenerationOptions(case["new"], NO_EOS, temperature=case["temperature"], top_k=case["top_k"] or None,
                                               top_p=case["top_p"] if case["top_p"] < 1.0 else None, repetition_penalty=case["repetition"])
        options.validate()
        return dict(kind=kind, model=model, prefix=_zipf(gen, case["vocab"], (case["prefix"],)).tolist(), options=options, seed=seed)
    if kind == "attention":
        rows, channels = case["batch"] * case["time"], case["heads"] * case["head_dim"]
        qkv = torch.randn(rows, 3 * channels, generator=gen, device="cuda").to(torch.bfloat16)
        dout = torch.randn(rows, channels, generator=gen, device="cuda").to(torch.bfloat16)
        return dict(kind=kind, ctx=ctx, qkv=qkv.split(channels, dim=1), dout=dout, sizes=(case["batch"], case["time"], case["heads"]))
    dtype = torch.float32 if case["precision"] == "f32" else torch.bfloat16
    m, k, n = case["rows"], case["inputs"], case["outputs"]
    x = torch.randn(m, k, generator=gen, device="cuda").to(dtype)
    w = (torch.randn(n, k, generator=gen, device="cuda") * k ** -0.5).to(dtype)
    bias = torch.randn(n, generator=gen, device="cuda") * 0.1
    dy = torch.randn(m, n, generator=gen, device="cuda").to(dtype)
    return dict(kind=kind, ctx=ctx, x=x, w=w, bias=bias, dy=dy, f32=dtype == torch.float32)


# ---- one pass ------------------------------------------------------------------------------------------------------
class Trained(dict):
    """What a training step leaves: its loss, and the model's gradients and parameters.  Those stay on the device, where
    the next step needs them, and are read when they are asked for, as a program does when it writes a checkpoint."""

    def __init__(self, model, loss):
        super().__init__(loss=loss, gradients=None, parameters=None)
        self._model = model

    def __getitem__(self, key):
        if key == "loss":
            return super().__getitem__(key)
        read = self._model.grad if key == "gradients" else self._model.parameter
        return torch.cat([torch.from_numpy(read(name)).reshape(-1).cuda() for name in self._model.parameter_names()])


def run(state):
    kind = state["kind"]
    if kind == "train":
        model = state["model"]
        x, y = state["pairs"][state["step"] % BATCHES]
        state["step"] += 1
        if state["policy"] is None:
            return Trained(model, model.train_step(x, y))
        model.forward_backward(x, y)
        model.optimizer_step_policy(state["policy"])
        return Trained(model, model.loss())
    if kind == "eval":
        m = generation.evaluate_token_loss(state["model"], state["stream"], state["batch"])
        return dict(loss=m.loss, perplexity=m.perplexity, tokens=m.tokens)
    if kind == "generate":
        out = generation.generate(state["model"], state["prefix"], state["options"], generation.HeirloomRng(state["seed"]))
        return dict(tokens=np.array(out.tokens, np.int64), probabilities=np.array([s.probability for s in out.steps]))
    ctx = state["ctx"]
    if kind == "attention":
        (q, k, v), dout, sizes = state["qkv"], state["dout"], state["sizes"]
        out, lse = cuda.flash_attention_forward(ctx, q, k, v, *sizes)
        return dict(out=out, lse=lse, dqkv=cuda.flash_attention_backward(ctx, q, k, v, out, dout, lse, *sizes))
    x, w, bias, dy = state["x"], state["w"], state["bias"], state["dy"]
    if state["f32"]:
        y = cuda.bias_add_f32(ctx, cuda.matmul_f32_strided(ctx, x, w.t()), bias)
        return dict(y=y, dx=cuda.matmul_f32_strided(ctx, dy, w), dw=cuda.matmul_f32_strided(ctx, dy.t(), x), db=cuda.bias_grad(ctx, dy))
    (m, k), n = x.shape, w.shape[0]
    h, g = cuda.gemm_bf16(ctx, x, w, m, n, k, epilogue=cuda.EPI_BIAS_GELU, bias=bias, want_aux_out=True)
    dx = cuda.gemm_bf16(ctx, dy, w, m, k, n, cuda.K_MAJOR, cuda.MN_MAJOR)
    dw = cuda.gemm_bf16(ctx, dy, x, n, k, m, cuda.MN_MAJOR, cuda.MN_MAJOR, out_dtype=torch.float32)
    return dict(h=h, g=g, dx=dx, dw=dw, db=cuda.bias_grad(ctx, dy))


# ---- what a pass cannot do without -----------------------------------------------------------------------------------
def _model_work(case):
    """(matmul weights of the blocks, weights of the head, parameters, attention flops of one token's forward)."""
    d, f, v, layers = case["d_model"], case["d_ff"], case["vocab"], case["n_layers"]
    memory = len(case["memory_layers"].split(",")) if "slots" in case else 0
    blocks = layers * 4 * d * d + (layers - memory) * 2 * d * f
    tables = 0
    if memory:
        side = math.isqrt(case["slots"])
        blocks += memory * (d * case["key_dim"] + 2 * d * case["value_dim"] + side * case["key_dim"])
        tables = case["slots"] * case["value_dim"] + side * case["key_dim"]
    return blocks, d * v, blocks + 2 * d * v + d * case["context"] + tables, 2.0 * layers * case["context"] * d


def work(case):
    kind = case["kind"]
    if kind in ("train", "eval", "generate"):
        blocks, head, parameters, attention = _model_work(case)
        item = 4 if case["precision"] == "f32" else 2
    if kind == "train":
        tokens = case["batch"] * case["context"]
        moved = 28.0 * parameters  # read: parameter and both moments; written: those and the gradient
        if case.get("policy") == "sparse_rows":  # weights read, gradients written, the looked-up rows updated
            rows = min(case["slots"], tokens * case["top_k"])
            moved = (item + 4.0) * parameters + 20.0 * rows * case["value_dim"]
        elif case.get("policy") == "memory_only":
            moved = (item + 4.0) * parameters + 24.0 * case["slots"] * case["value_dim"]
        return dict(bytes=moved + 16.0 * tokens, flops=3.0 * tokens * (2.0 * (blocks + head) + attention))
    if kind == "eval":
        tokens = case["windows"] * case["context"]
        return dict(bytes=float(item * (blocks + head) + 16 * tokens), flops=tokens * (2.0 * (blocks + head) + attention))
    if kind == "generate":
        seen = min(case["context"], case["prefix"] + case["new"])
        return dict(bytes=float(case["new"] * item * (blocks + head)),
                    flops=(case["prefix"] + case["new"]) * 2.0 * blocks + case["new"] * 2.0 * head + seen * attention)
    if kind == "attention":
        elements = case["batch"] * case["time"] * case["heads"] * case["head_dim"]
        return dict(bytes=2.0 * 8 * elements + 4.0 * elements / case["head_dim"], flops=7.0 * elements * case["time"])
    m, k, n = case["rows"], case["inputs"], case["outputs"]
    if case["precision"] == "f32":
        return dict(bytes=4.0 * (2 * m * k + 2 * n * k + 2 * m * n + 2 * n), flops=6.0 * m * n * k)
    return dict(bytes=2.0 * (2 * m * k + n * k + 3 * m * n) + 4.0 * (n * k + 2 * n), flops=6.0 * m * n * k)


def tolerance(case):
    # bf16: operands carry 8 bits; single elements of a gradient or of a first Adam step (whose size is that of the sign
    # of the gradient) may differ by much of their own size where it nearly cancels.  f32: sums in f64 rounded to f32.
    if case.get("precision") == "f32":
        return {"rel": 1e-5, "max": 1e-2}
    return {"rel": 1e-2, "max": 0.5}
