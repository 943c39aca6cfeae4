"""Step-level parity of the decoder executor (amp-bf16 route) against the oracle's AMP restatement."""
import contextlib
import math

import numpy as np
import pytest
import torch

from oracle import heirloom_oracle as ho
from tests.gpu_util import ctx, full_device

pytestmark = pytest.mark.gpu

# parameters whose true gradient is identically zero (a constant added to every key leaves the
# softmax unchanged), so what reaches AdamW is rounding noise on both sides
NULL_GRADIENT = ("attention.k_proj.bias",)


def make(cfg_kwargs, batch, seed=0):
    from heirloom_b200 import nn
    c = ctx()
    cfg = nn.DecoderConfig(batch=batch, **cfg_kwargs)
    model = nn.DecoderLm(c, cfg)
    ocfg = ho.DecoderConfig(**cfg_kwargs)
    params = ho.init_parameters(ocfg, seed)
    model.load_state_dict(params)
    return c, model, ocfg, params


def test_parameter_names_follow_state_dict_order():
    kw = dict(vocab=512, d_model=128, n_layers=2, n_heads=2, d_ff=256, context=128)
    _, model, ocfg, _ = make(kw, 2)
    assert model.parameter_names() == ho.parameter_names(ocfg)
    assert model.parameter_shapes() == ho.parameter_shapes(ocfg)
    model.close()


@pytest.mark.parametrize("n_heads", [2, 4, 1])  # head_dim 64 (tcgen05 flash kernels), 32 and 128 (f32 attention kernels)
def test_one_step_loss_and_gradients_match_the_amp_oracle(n_heads):
    kw = dict(vocab=512, d_model=128, n_layers=2, n_heads=n_heads, d_ff=256, context=128)
    c, model, ocfg, params = make(kw, 2)
    rng = np.random.default_rng(3)
    tok = ho.zipf_tokens(rng, ocfg.vocab, (2, 129))
    x, y = tok[:, :-1].copy(), tok[:, 1:].copy()
    model.forward_backward(torch.tensor(x, device="cuda"), torch.tensor(y, device="cuda"))
    loss = model.loss()
    oloss, ograds = ho.decoder_loss_and_grads(ocfg, params, x, y, amp_bf16=True)
    assert abs(loss - oloss) <= 2e-3 * abs(oloss), (loss, oloss)
    for name in ho.parameter_names(ocfg):
        g, w = model.grad(name).astype(np.float64), ograds[name]
        scale = np.abs(w).max() + 1e-12
        if any(name.endswith(s) for s in NULL_GRADIENT):
            assert np.abs(g).max() <= 2e-2 * max(np.abs(ograds[name.replace("k_proj", "q_proj")]).max(), 1e-12)
            continue
        # bf16 operands: compare against the tensor's scale, elementwise and on average
        assert np.abs(g - w).max() <= 0.06 * scale, (name, np.abs(g - w).max(), scale)
        assert np.abs(g - w).mean() <= 0.01 * scale, (name, np.abs(g - w).mean(), scale)
    model.close()


def test_ten_steps_parameters_and_losses_track_the_amp_oracle():
    kw = dict(vocab=512, d_model=128, n_layers=2, n_heads=2, d_ff=256, context=128)
    c, model, ocfg, params = make(kw, 2, seed=1)
    model.set_optimizer(lr=1e-3, weight_decay=0.01)
    state = ho.AdamWState(lr=1e-3, weight_decay=0.01)
    rng = np.random.default_rng(4)
    losses, olosses = [], []
    for _ in range(10):
        tok = ho.zipf_tokens(rng, ocfg.vocab, (2, 129))
        x, y = tok[:, :-1].copy(), tok[:, 1:].copy()
        losses.append(model.train_step(torch.tensor(x).pin_memory(), torch.tensor(y).pin_memory()))
        olosses += ho.train_steps(ocfg, params, [(x, y)], state, amp_bf16=True)
    assert model.optimizer_steps == 10
    assert np.max(np.abs(np.array(losses) - np.array(olosses)) / np.array(olosses)) <= 0.01
    # parameters after 10 steps: |a-b| <= 2e-2 * max(|b|, floor); the floor covers elements whose
    # value is comparable to the 10*lr an Adam update can move them when the gradient sign is noise
    floor = 10 * 1e-3
    worst = 0.0
    for name in ho.parameter_names(ocfg):
        if any(name.endswith(s) for s in NULL_GRADIENT):
            continue
        got, want = model.parameter(name).astype(np.float64), params[name]
        viol = np.abs(got - want) / np.maximum(np.abs(want), floor)
        frac_bad = np.mean(viol > 2e-2)
        worst = max(worst, frac_bad)
        assert frac_bad <= 0.015, (name, frac_bad, viol.max())  # measured worst: 0.011 (a 1024-element bias)
    print("amp dense model, worst fraction of elements outside 2e-2 after 10 steps:", worst)
    model.close()


def test_launch_count_is_reported_and_nonzero():
    kw = dict(vocab=512, d_model=128, n_layers=1, n_heads=2, d_ff=256, context=128)
    c, model, ocfg, _ = make(kw, 1)
    model.set_optimizer()
    tok = torch.zeros(1, 128, dtype=torch.int64, device="cuda")
    model.train_step_device(tok, tok)
    c.sync()
    assert model.launches_last_step > 20
    assert c.counters().gemm_tcgen05_launches >= 13
    model.close()


def test_f32_route_one_step_matches_the_f64_oracle_tightly():
    from heirloom_b200 import nn
    kw = dict(vocab=96, d_model=64, n_layers=2, n_heads=2, d_ff=128, context=24)
    c = ctx()
    model = nn.DecoderLm(c, nn.DecoderConfig(batch=3, precision=nn.PRECISION_F32, **kw))
    ocfg = ho.DecoderConfig(**kw)
    params = ho.init_parameters(ocfg, 5)
    rng = np.random.default_rng(6)
    for n in params:  # larger weights: gradients well above rounding noise everywhere
        if params[n].ndim == 2:
            params[n] = ho.f32_round(rng.standard_normal(params[n].shape) * 0.2)
    model.load_state_dict(params)
    tok = rng.integers(0, ocfg.vocab, (3, 25))
    x, y = tok[:, :-1].copy(), tok[:, 1:].copy()
    model.forward_backward(torch.tensor(x, device="cuda"), torch.tensor(y, device="cuda"))
    oloss, ograds = ho.decoder_loss_and_grads(ocfg, params, x, y)
    assert abs(model.loss() - oloss) <= 1e-6 * abs(oloss)
    for name in ho.parameter_names(ocfg):
        g, w = model.grad(name).astype(np.float64), ograds[name]
        scale = np.abs(w).max()
        if name.endswith("attention.k_proj.bias"):
            assert np.abs(g).max() <= 1e-5 * np.abs(ograds[name.replace("k_proj", "q_proj")]).max()
            continue
        assert np.abs(g - w).max() <= 2e-6 * scale + 1e-9, (name, np.abs(g - w).max(), scale)
    model.close()


def test_f32_route_tracks_the_reference_loss_trace_for_200_steps():
    """north_star gate: f32 per-step loss within 1e-5 relative on the tiny byte-level decoder."""
    import json
    from pathlib import Path
    from heirloom_b200 import nn
    from tests.golden.make_tiny_trace import BATCH, CONFIG, STEPS, WEIGHT_SEED, batches
    trace = json.loads((Path(__file__).parent / "golden" / "tiny_decoder_trace.json").read_text())
    assert trace["config"] == CONFIG and trace["steps"] == STEPS
    c = ctx()
    model = nn.DecoderLm(c, nn.DecoderConfig(batch=BATCH, precision=nn.PRECISION_F32, **CONFIG))
    model.load_state_dict(ho.init_parameters(ho.DecoderConfig(**CONFIG), WEIGHT_SEED))
    model.set_optimizer(lr=1e-3, beta1=0.9, beta2=0.999, eps=1e-8, weight_decay=0.01, clip_norm=None)
    losses = [model.train_step(torch.tensor(x).pin_memory(), torch.tensor(y).pin_memory()) for x, y in batches(STEPS)]
    rel = np.abs(np.array(losses) - np.array(trace["losses"])) / np.array(trace["losses"])
    assert rel.max() <= 1e-5, (rel.max(), int(rel.argmax()))
    for name, (want_sum, want_sumsq) in trace["final_parameter_sum_and_sumsq"].items():
        p = model.parameter(name).astype(np.float64)
        assert abs((p * p).sum() - want_sumsq) <= 1e-4 * want_sumsq, name
    model.close()


def test_amp_route_tracks_the_oracle_loss_trace_for_200_steps():
    """north_star gate: bf16 loss within 1 % of the reference's AMP route at every one of 200 steps, on token streams
    whose loss actually falls (6.26 -> 4.39)."""
    import json
    from pathlib import Path
    from heirloom_b200 import nn
    from tests.golden import make_amp_trace as mt
    trace = json.loads((Path(__file__).parent / "golden" / "amp_decoder_trace.json").read_text())
    assert trace["config"] == mt.CONFIG and trace["steps"] == mt.STEPS
    c = ctx()
    model = nn.DecoderLm(c, nn.DecoderConfig(batch=mt.BATCH, **mt.CONFIG))
    model.load_state_dict(ho.init_parameters(ho.DecoderConfig(**mt.CONFIG), mt.WEIGHT_SEED))
    model.set_optimizer(lr=1e-3, beta1=0.9, beta2=0.999, eps=1e-8, weight_decay=0.01, clip_norm=None)
    losses = [model.train_step(torch.tensor(x).pin_memory(), torch.tensor(y).pin_memory()) for x, y in mt.batches(mt.STEPS)]
    model.close()
    rel = np.abs(np.array(losses) - np.array(trace["losses"])) / np.array(trace["losses"])
    print("amp 200-step trace: worst relative loss deviation", rel.max(), "at step", int(rel.argmax()))
    assert rel.max() <= 0.01, (rel.max(), int(rel.argmax()))
    assert losses[-1] < 4.6


def test_collected_weight_gradients_equal_those_of_two_half_batches():
    """18000 tokens: the weight gradients of several layers in one launch, ragged in every size (960/320/1000 by 320/1000 in tiles of
    256 by 256, 282 token blocks of 64).  9000 tokens: each product for itself.  The loss is a mean, so that the two halves'
    gradients are exactly twice as large in every bf16 rounding.  What differs is the order of f32 sums: 2^-24 relative per
    addition, at random over 18000 of them 8e-6, times ten for what cancels in a sum; and, below the last block, bf16 values of
    the residual stream's gradient that such a difference tips over (2^-8 of a value, for fewer than one in a hundred)."""
    from heirloom_b200 import nn
    c = ctx()
    rng = np.random.default_rng(5)
    x = torch.from_numpy(rng.integers(0, 1000, (18, 1000))).cuda()
    y = torch.from_numpy(rng.integers(0, 1000, (18, 1000))).cuda()
    state, grads = None, []
    for part in (slice(0, 18), slice(0, 9), slice(9, 18)):
        model = nn.DecoderLm(c, nn.DecoderConfig(vocab=1000, d_model=320, n_layers=3, n_heads=5, d_ff=1000, context=1000,
                                                 batch=len(range(18)[part])))
        if state is None:
            state = {n: (np.ones(s) if ".ln" in n or n.startswith("ln_f") else rng.standard_normal(s) * 0.05)
                     for n, s in model.parameter_shapes().items()}
        model.load_state_dict(state)
        model.forward_backward(x[part].contiguous(), y[part].contiguous())
        grads.append({n: model.grad(n).astype(np.float64) for n in state})
        model.close()
    for name, whole in grads[0].items():
        if name.endswith("k_proj.bias"):
            continue  # the exact gradient is zero
        halves = (grads[1][name] + grads[2][name]) / 2
        tipped = 0 if name.startswith(("lm_head", "ln_f", "block.2")) else 2 ** -8 * 0.1 * (4 if "embedding" in name else 2)
        assert np.linalg.norm(whole - halves) <= (2 ** -24 * np.sqrt(18000) * 10 + tipped) * np.linalg.norm(halves), name


def test_training_with_tiles_from_a_counter_equals_training_without(monkeypatch):
    """HEIRLOOM_GEMM_DYNAMIC=1 over five training steps, more than the plain, the captured and a replayed pass would take: every
    tile of the head's product (256 of 128 x 256, single CTAs) is computed in each of them.  Which CTA computes a
    tile changes no bits; the products that the small-product kernel takes without the setting round alike but sum in another
    order, which bf16 activations and AdamW's first steps turn into 1e-2 of a gradient at most."""
    from heirloom_b200 import cuda, nn
    c = ctx()
    rng = np.random.default_rng(0)
    tokens = torch.from_numpy(rng.integers(0, 4096, (5, 2, 16, 128))).cuda()
    monkeypatch.setenv("HEIRLOOM_GEMM_PAIRS", "0")
    state, runs = None, []
    for dynamic in "01":
        monkeypatch.setenv("HEIRLOOM_GEMM_DYNAMIC", dynamic)
        model = nn.DecoderLm(c, nn.DecoderConfig(vocab=4096, d_model=128, n_layers=1, n_heads=2, d_ff=256, context=128, batch=16))
        if state is None:
            state = {n: (np.ones(s) if ".ln" in n or n.startswith("ln_f") else rng.standard_normal(s) * 0.05)
                     for n, s in model.parameter_shapes().items()}
        model.load_state_dict(state)
        model.set_optimizer(lr=1e-2, weight_decay=0.0)
        steps = []
        for x, y in tokens:
            model.forward_backward(x, y)
            steps.append((model.loss(), model.grad("lm_head.weight")))
            model.optimizer_step()
        runs.append(steps)
        model.close()
    for step, ((want, want_grad), (got, got_grad)) in enumerate(zip(*runs)):
        assert got == pytest.approx(want, rel=1e-3), step
        assert np.linalg.norm(got_grad - want_grad) <= 2e-2 * np.linalg.norm(want_grad), step
    # the host still knows the counter: an eager product computes all of its tiles as well
    a = torch.randn(4096, 320, device="cuda").bfloat16()
    b = torch.randn(2048, 320, device="cuda").bfloat16()
    out = cuda.gemm_bf16(c, a, b, 4096, 2048, 320, out_dtype=torch.float32)
    c.sync()
    want = a.double() @ b.double().t()
    assert (out.double() - want).abs().max() <= 2e-6 * np.sqrt(320) * want.abs().max()


def test_a_caller_may_capture_the_step():
    """Forward, backward and AdamW inside a capture of the context's stream that the caller began, after one and three passes of its
    own: a step each, whose replay leaves the parameters of a step that was not captured (scatter-adds and dQ reductions have
    no fixed order: 1e-6 of a parameter's scale, and where a gradient is noise AdamW's step of at most lr)."""
    import ctypes
    from heirloom_b200 import nn
    c = ctx()
    rt = ctypes.CDLL("libcudart.so.12")
    c.lib.hl_ctx_stream.restype = ctypes.c_void_p
    stream = ctypes.c_void_p(c.lib.hl_ctx_stream(c.handle))
    rng = np.random.default_rng(0)
    x = torch.from_numpy(rng.integers(0, 256, (4, 64))).cuda()
    y = torch.from_numpy(rng.integers(0, 256, (4, 64))).cuda()
    torch.cuda.synchronize()
    for precision in (nn.PRECISION_AMP_BF16, nn.PRECISION_F32):
        state = None
        for passes in (1, 3):
            results = []
            for captured in (False, True):
                model = nn.DecoderLm(c, nn.DecoderConfig(vocab=256, d_model=128, n_layers=2, n_heads=2, d_ff=256, context=64, batch=4,
                                                         precision=precision))
                if state is None:
                    state = {n: (np.ones(s) if ".ln" in n or n.startswith("ln_f") else rng.standard_normal(s) * 0.05)
                             for n, s in model.parameter_shapes().items()}
                model.load_state_dict(state)
                model.set_optimizer(lr=1e-3)
                for _ in range(passes):
                    model.forward_backward(x, y)
                c.sync()
                error = None
                if captured:
                    graph, exe = ctypes.c_void_p(), ctypes.c_void_p()
                    assert rt.cudaStreamBeginCapture(stream, 2) == 0  # relaxed
                    try:
                        model.train_step_device(x, y)
                    except Exception as e:
                        error = e
                    ended = rt.cudaStreamEndCapture(stream, ctypes.byref(graph))
                    if error is None and ended == 0:
                        assert rt.cudaGraphInstantiate(ctypes.byref(exe), graph, ctypes.c_ulonglong(0)) == 0
                        assert rt.cudaGraphLaunch(exe, stream) == 0
                    c.sync()
                    if exe:
                        rt.cudaGraphExecDestroy(exe)
                    if graph:
                        rt.cudaGraphDestroy(graph)
                    error = error or (ended or None)
                else:
                    model.train_step_device(x, y)
                    c.sync()
                results.append({n: model.parameter(n) for n in state})
                model.close()
                assert error is None, (precision, passes, error)
            for n in state:
                if not n.endswith("k_proj.bias"):  # its exact gradient is zero
                    diff = np.abs(results[1][n] - results[0][n])
                    assert np.mean(diff > 1e-6 * max(1.0, np.abs(results[0][n]).max())) <= 0.01 and diff.max() <= 2.1e-3, (precision, passes, n)


def test_passes_run_on_a_device_without_memory_for_their_graphs():
    """Six models of twelve layers, no memory left on the device: more graphs than fit into what the driver still has.  A pass that
    cannot be captured runs plainly, every time, with the same losses as in a device with room."""
    from heirloom_b200 import nn
    c = ctx()
    rng = np.random.default_rng(0)
    x = torch.from_numpy(rng.integers(0, 256, (4, 64))).cuda()
    runs = []
    for full in (False, True):
        rng = np.random.default_rng(1)
        models = []
        for _ in range(6):
            model = nn.DecoderLm(c, nn.DecoderConfig(vocab=256, d_model=128, n_layers=12, n_heads=2, d_ff=256, context=64, batch=4))
            model.load_state_dict({n: rng.standard_normal(s) * 0.05 for n, s in model.parameter_shapes().items()})
            model.forward_backward(x, x)
            model.eval_loss_device(x, x)
            models.append(model)
        c.sync()
        losses = []
        with full_device() if full else contextlib.nullcontext():
            for model in models:
                for _ in range(3):
                    try:
                        model.forward_backward(x, x)
                        losses += [model.loss(), model.eval_loss_device(x, x)]
                    except Exception as e:
                        losses.append(str(e))
        for model in models:
            model.close()
        runs.append(losses)
    assert runs[0] == runs[1]


@pytest.mark.parametrize("batch,d_model,d_ff,layers,roundings", [(3, 64, 8, 1, 4), (16, 64, 8, 1, 4), (100, 128, 256, 1, 4),
                                                                (16, 128, 512, 12, 12), (5, 768, 3072, 5, 12)])
def test_bias_gradients_of_many_tokens_are_column_sums(batch, d_model, d_ff, layers, roundings):
    """The head's bias gradient beside its weight gradient, against the f64 sums of the same bf16 dlogits (3072 to 102400 tokens of one
    logit row each, made by the same loss kernel); a product of its own, and one of a group of layers' (the last two).  Four values
    at a time are added in f32, two roundings (in a group eight such sums one after the other, eight more), the rest in
    f64, rounded once as a part and once as the result: that many times 2^-24 of the terms' magnitudes."""
    from heirloom_b200 import cuda, nn
    c = ctx()
    vocab, time = 64, 1024
    rng = np.random.default_rng(batch)
    model = nn.DecoderLm(c, nn.DecoderConfig(vocab=vocab, d_model=d_model, n_layers=layers, n_heads=d_model // 64, d_ff=d_ff, context=time,
                                             batch=batch))
    state = {n: np.zeros(s, np.float32) for n, s in model.parameter_shapes().items()}  # every token's logits are the head's bias
    state["lm_head.bias"] = rng.standard_normal(vocab).astype(np.float32) * 3
    model.load_state_dict(state)
    x = torch.from_numpy(rng.integers(0, vocab, (batch, time))).cuda()
    y = torch.from_numpy(rng.integers(0, vocab, (batch, time))).cuda()
    model.forward_backward(x, y)
    got = model.grad("lm_head.bias").astype(np.float64)
    model.close()
    logits = torch.from_numpy(np.tile(state["lm_head.bias"], (batch * time, 1))).cuda()
    _, dlogits = cuda.cross_entropy(c, logits, y.reshape(-1), dlogits_dtype=torch.bfloat16)
    c.sync()
    want, magnitude = dlogits.double().sum(0).cpu().numpy(), dlogits.double().abs().sum(0).cpu().numpy()
    assert (np.abs(got - want) <= roundings * 2.0 ** -24 * magnitude).all(), (np.abs(got - want) / magnitude).max()


@pytest.mark.parametrize("batch,layers", [(8, 8), (2, 8)])
def test_a_model_without_room_for_operand_copies_is_created_without_them(batch, layers):
    """The weight gradients of several layers in one launch (batch 8), or on a second stream (batch 2), want copies of operands; with 20 MB
    less than those take the model is created all the same and trains alike (other kernels and sums for the weight gradients: 1e-2 of
    a gradient's norm at most, measured against bf16 operands)."""
    from heirloom_b200 import cuda, nn
    ctx()
    c = cuda.Context(0)
    kw = dict(vocab=64, d_model=512, n_layers=layers, n_heads=8, d_ff=2048, context=512, batch=batch)
    rng = np.random.default_rng(0)
    x = torch.from_numpy(rng.integers(0, 64, (batch, 512))).cuda()
    state, runs, sizes = None, [], []
    for full in (False, True):
        c.reset_counters()
        model, error = None, None
        with full_device(leave=sizes[0] - (20 << 20)) if full else contextlib.nullcontext():
            try:
                model = nn.DecoderLm(c, nn.DecoderConfig(**kw))
            except Exception as e:
                error = str(e)
        if model is not None:
            sizes.append(int(c.counters().allocated_bytes))
            if state is None:
                state = {n: (np.ones(s) if ".ln" in n or n.startswith("ln_f") else rng.standard_normal(s) * 0.05)
                         for n, s in model.parameter_shapes().items()}
            model.load_state_dict(state)
            model.forward_backward(x, x)
            runs.append((model.loss(), {n: model.grad(n) for n in state}))
            model.close()
    c.close()
    assert error is None, error
    assert sizes[1] < sizes[0] - (20 << 20) and runs[0][0] == pytest.approx(runs[1][0], rel=1e-6)
    for n in state:
        if not n.endswith("k_proj.bias"):
            assert np.linalg.norm(runs[1][1][n] - runs[0][1][n]) <= 1e-2 * np.linalg.norm(runs[0][1][n]), n


@pytest.mark.parametrize("precision", [0, 1])
def test_clipping_by_the_global_norm_of_a_dense_step(precision):
    """The factor is worked out on the device: parameters and moments of a step with a limit below the norm are those of the oracle's
    update with the f64 factor, a limit above it changes nothing, and a norm that is not finite is an error that leaves
    parameters, moments and the step count as they were; the next step is right again."""
    from heirloom_b200 import nn
    from heirloom_b200._lib import HeirloomError
    c = ctx()
    rng = np.random.default_rng(2)
    x = torch.from_numpy(rng.integers(0, 64, (4, 32))).cuda()
    y = torch.from_numpy(rng.integers(0, 64, (4, 32))).cuda()
    model = nn.DecoderLm(c, nn.DecoderConfig(vocab=64, d_model=64, n_layers=2, n_heads=1, d_ff=128, context=32, batch=4, precision=precision))
    state = {n: (np.ones(s) if ".ln" in n or n.startswith("ln_f") else rng.standard_normal(s) * 0.1)
             for n, s in model.parameter_shapes().items()}
    before = {n: v.astype(np.float32) for n, v in state.items()}

    def stepped(limit):
        model.load_state_dict(state)
        model.set_optimizer(lr=1e-3, beta1=0.9, beta2=0.999, eps=1e-8, weight_decay=0.01, clip_norm=limit)
        for n in state:
            model.set_moments(n, np.zeros_like(before[n]), np.zeros_like(before[n]))
        model.set_optimizer_steps(0)
        model.forward_backward(x, y)
        grads = {n: model.grad(n) for n in state}
        error = None
        try:
            model.optimizer_step()
            c.sync()
        except HeirloomError as e:
            error = str(e)
        return grads, {n: (model.parameter(n),) + model.moments(n) for n in state}, model.optimizer_steps, error

    grads, free, steps, error = stepped(None)
    norm = math.sqrt(sum(float((g.astype(np.float64) ** 2).sum()) for g in grads.values()))
    results = {limit: stepped(limit) for limit in (norm * 0.25, norm * 4.0)}
    broken = dict(state, **{"lm_head.bias": np.full_like(state["lm_head.bias"], np.nan)})
    model.load_state_dict(broken)
    model.set_optimizer(lr=1e-3, clip_norm=1.0)
    model.set_optimizer_steps(5)
    model.forward_backward(x, y)
    kept = {n: (model.parameter(n),) + model.moments(n) for n in state}
    with pytest.raises(HeirloomError, match="non-finite or negative global gradient"):
        model.optimizer_step()
    after, count = {n: (model.parameter(n),) + model.moments(n) for n in state}, model.optimizer_steps
    again = stepped(norm * 0.25)
    model.close()
    assert error is None and steps == 1 and count == 5
    assert all(np.array_equal(a, b, equal_nan=True) for n in state for a, b in zip(kept[n], after[n]))
    for limit, (g, got, _, error) in list(results.items()) + [(norm * 0.25, again)]:
        assert error is None
        own = math.sqrt(sum(float((v.astype(np.float64) ** 2).sum()) for v in g.values()))
        factor = min(1.0, limit / (own + 1e-12)) if own > limit else 1.0
        for n in state:
            # AdamW's first moment of a first step is (1 - beta1) x (factor x gradient + decay x parameter) with f32 constants: f32
            # roundings of a few terms
            want = float(np.float32(1) - np.float32(0.9)) * (factor * g[n].astype(np.float64) + float(np.float32(0.01)) * before[n])
            assert np.abs(got[n][1] - want).max() <= 4 * 2.0 ** -24 * (np.abs(0.1 * factor * g[n]).max() + np.abs(1e-3 * before[n]).max()) + 1e-12, n


@pytest.mark.parametrize("context,vocab,masked,d_model", [(103, 8200, False, 128), (128, 5000, False, 128), (128, 5000, True, 128), (103, 16384, True, 128),
                                                          (128, 4104, False, 320), (103, 12000, True, 1024)])
def test_head_of_many_rows_equals_the_head_that_stores_its_logits(context, vocab, masked, d_model):
    """From 1024 rows on the logits are formed twice instead of stored (1030 and 1280 rows, ragged last columns): loss and head
    gradients are the average of those of two halves below that, in whose scale the same bf16 values are a factor of two larger.
    A gradient of a row may round the other way (a few of a column's, each at most 2^-8 of 1 / rows); masked columns have none."""
    from heirloom_b200 import nn
    kw = dict(vocab=vocab, d_model=d_model, n_layers=1, n_heads=d_model // 64, d_ff=128, context=context)
    rng = np.random.default_rng(vocab)
    c = ctx()
    whole, half = nn.DecoderLm(c, nn.DecoderConfig(batch=10, **kw)), nn.DecoderLm(c, nn.DecoderConfig(batch=5, **kw))
    state = {n: rng.standard_normal(s) * 0.2 for n, s in whole.parameter_shapes().items()}
    off = np.arange(300, 700) if masked else np.arange(0)
    state["lm_head.bias"][off] = -np.inf
    x = torch.from_numpy(rng.integers(0, vocab, (10, context))).cuda()
    y = torch.from_numpy(rng.choice(np.setdiff1d(np.arange(vocab), off), (10, context))).cuda()
    y[0, :2] = torch.tensor([0, vocab - 1])
    for m in (whole, half):
        m.load_state_dict(state)
    names = ("lm_head.bias", "lm_head.weight")
    want, loss = {n: 0.0 for n in names}, 0.0
    for part in range(2):
        half.forward_backward(x[part * 5:part * 5 + 5].contiguous(), y[part * 5:part * 5 + 5].contiguous())
        loss += half.loss() / 2
        for n in names:
            want[n] = want[n] + half.grad(n).astype(np.float64) / 2
    for _ in range(3):  # plain, captured, replayed
        whole.forward_backward(x, y)
        assert whole.loss() == pytest.approx(loss, rel=2e-6)
        rounding = 2.0 ** -8 / (10 * context)
        bias, weight = (whole.grad(n).astype(np.float64) for n in names)
        assert np.abs(bias - want["lm_head.bias"]).max() <= 8 * rounding
        assert np.abs(weight - want["lm_head.weight"]).max() <= 8 * rounding * 4.0  # |z| of a layer norm of gamma 0.2: below 4
        assert not bias[off].any() and not weight[off].any()
    whole.close()
    half.close()


def _profile_of_a_pass(batch, context, vocab, d_model):
    """What the profile says that one forward and backward pass of a one-block model worked, by category."""
    import ctypes
    from heirloom_b200 import cuda, nn
    from heirloom_b200._lib import Profile
    c = ctx()
    model = nn.DecoderLm(c, nn.DecoderConfig(batch=batch, context=context, vocab=vocab, d_model=d_model, n_layers=1, n_heads=d_model // 64, d_ff=128))
    rng = np.random.default_rng(0)
    model.load_state_dict({n: rng.standard_normal(s) * 0.2 for n, s in model.parameter_shapes().items()})
    x = torch.from_numpy(rng.integers(0, vocab, (batch, context))).cuda()
    cuda.check(c.lib.hl_profile_enable(c.handle, 1))
    try:
        model.forward_backward(x, x)
        c.sync()
        p = Profile()
        cuda.check(c.lib.hl_profile_read(c.handle, ctypes.byref(p)))
    finally:
        cuda.check(c.lib.hl_profile_enable(c.handle, 0))
        model.close()
    return list(p.work)


def test_the_heads_second_product_counts_as_time_and_not_as_work():
    """Rates are made of what a step needs: with 1030 rows, whose logits are formed twice, the profile reports the products' flop of two
    passes of 515."""
    assert _profile_of_a_pass(10, 103, 8200, 128)[0] == 2 * _profile_of_a_pass(5, 103, 8200, 128)[0]


@pytest.mark.parametrize("batch,vocab,d_model,twice", [(8, 8000, 960, False), (8, 8000, 768, True), (8, 32000, 960, True), (16, 2000, 832, False),
                                                       (12, 8000, 832, True), (32, 2000, 832, True), (7, 32000, 512, False)])
def test_which_heads_form_their_logits_twice(batch, vocab, d_model, twice):
    """Contexts of 128: 1024 rows, or few columns and wide rows, or too few rows.  The loss reads eight bytes for every 128 columns of a row,
    or all of its logits."""
    loss = _profile_of_a_pass(batch, 128, vocab, d_model)[4]
    assert (loss < batch * 128 * vocab) == twice
