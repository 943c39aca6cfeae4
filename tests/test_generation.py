"""Sampling controls, the RNG stream, evaluation and generation (reference: src/nn.rs:1595-1751,
src/rng.rs:29-45, src/memory_transformer.rs:1730-1984, tests/transformer_runtime.rs:1530-1575)."""
import math

import numpy as np
import pytest
import torch

from heirloom_b200 import generation as gen
from oracle import heirloom_oracle as ho


def test_rng_stream_is_splitmix64_and_uniforms_have_24_bits():
    rng = gen.HeirloomRng(0)
    # SplitMix64 from state 0: published first outputs of the generator
    assert [rng.next_u64() for _ in range(3)] == [0xE220A8397B1DCDAF, 0x6E789E6AA1B965F4, 0x06C45D188009454F]
    a, b = gen.HeirloomRng(123), gen.HeirloomRng(123)
    ua = [a.uniform_f32() for _ in range(8)]
    assert ua == [b.uniform_f32() for _ in range(8)] and all(0.0 <= u < 1.0 for u in ua)
    assert all(u * (1 << 24) == int(u * (1 << 24)) for u in ua)
    assert a.state == b.state and a.state != 123


def test_greedy_and_filters_follow_the_reference_rules():
    o = gen.GenerationOptions.greedy(4, 2)
    logits = [0.1, 2.0, 2.0, -1.0]
    t, p, lp = gen.sample_token(logits, [], o, gen.HeirloomRng(0))
    assert t == 2  # max_by keeps the last of equal maxima
    assert p == pytest.approx(math.exp(2.0) / (2 * math.exp(2.0) + math.exp(0.1) + math.exp(-1.0))) and lp == pytest.approx(math.log(p))
    # top_k = 1 at temperature 1 is greedy whatever the draw (tests/transformer_runtime.rs:1546-1562)
    o1 = gen.GenerationOptions(4, 2, temperature=1.0, top_k=1, top_p=1.0)
    assert gen.sample_token([0.1, 2.5, 2.0, -1.0], [], o1, gen.HeirloomRng(123))[0] == 1
    # top_p keeps the smallest prefix of the ranked distribution that reaches the mass
    keep = gen.sampling_filter(np.log(np.array([0.5, 0.3, 0.15, 0.05])), gen.GenerationOptions(1, 0, temperature=1.0, top_p=0.75))
    assert keep.tolist() == [True, True, False, False]
    keep = gen.sampling_filter(np.array([1.0, 3.0, 2.0, 0.0]), gen.GenerationOptions(1, 0, temperature=1.0, top_k=2))
    assert keep.tolist() == [False, True, True, False]
    # repetition controls: positive logits divided, negative multiplied, then frequency and presence
    o2 = gen.GenerationOptions(1, 0, repetition_penalty=2.0, frequency_penalty=0.5, presence_penalty=0.25)
    adj = np.array([2.0, -2.0, 1.0])
    gen._apply_repetition_controls(adj, [0, 0, 1, 7], o2)
    assert adj.tolist() == [2.0 / 2 - 0.5 * 2 - 0.25, -2.0 * 2 - 0.5 - 0.25, 1.0]
    # all-filtered input falls back to one-hot on index 0
    assert gen.softmax_logits(np.array([-np.inf, -np.inf])).tolist() == [1.0, 0.0]
    # sampling walks the cumulative distribution with one 24-bit uniform draw
    rng = gen.HeirloomRng(5)
    draw = gen.HeirloomRng(5).uniform_f32()
    probs = np.array([0.2, 0.5, 0.3])
    want = int(np.searchsorted(np.cumsum(probs), draw, side="left"))
    assert gen.sample_token(np.log(probs), [], gen.GenerationOptions(1, 9, temperature=1.0), rng)[0] == want


def stated_sample(logits, context, o, rng):
    """The sampling rules written out over the module's own filters."""
    x = np.asarray(logits, np.float64).copy()
    gen._apply_repetition_controls(x, context, o)
    if o.temperature > 0.0:
        x /= o.temperature
    x[~gen.sampling_filter(x, o)] = -np.inf
    probs = gen.softmax_logits(x)
    t = gen.argmax_filtered(x)
    if o.temperature > 0.0:
        draw, cumulative = rng.uniform_f32(), 0.0
        for i, p in enumerate(probs):
            cumulative += p
            if draw <= cumulative:
                t = i
                break
    return t, float(probs[t])


@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 1000, 50304])
def test_native_sampling_follows_the_stated_rules(n):
    """Vocabularies around the lane width and the largest one, every control, ties and -inf entries.  Probabilities are
    f64 sums in another order: at most n * 2^-53 relative, 1e-11 here."""
    r = np.random.default_rng(n)
    context = r.integers(0, n + 3, 50).tolist()  # ids past the vocabulary are ignored
    for case in range(12 if n < 5000 else 5):
        logits = r.standard_normal(n) * r.choice([0.1, 3.0, 30.0])
        if case % 3 == 1:
            logits = np.round(logits)  # ties
        if case % 4 == 2:
            logits[r.random(n) < 0.3] = -np.inf
        logits[0] = max(logits[0], -50.0)  # at least one finite entry
        for kw in (dict(), dict(temperature=0.7), dict(temperature=1.3, top_k=5), dict(top_k=3), dict(temperature=1.0, top_p=0.9),
                   dict(temperature=0.9, top_k=40, top_p=0.5, repetition_penalty=1.2, frequency_penalty=0.1, presence_penalty=0.2),
                   dict(temperature=0.5, top_k=10 ** 6, top_p=1.0)):
            o = gen.GenerationOptions(1, 0, **kw)
            a, b = gen.HeirloomRng(case), gen.HeirloomRng(case)
            t, p, logp = gen.sample_token(logits, context, o, a)
            want_t, want_p = stated_sample(logits, context, o, b)
            assert t == want_t and p == pytest.approx(want_p, rel=1e-11), (case, kw)
            assert logp == pytest.approx(math.log(max(p, np.finfo(np.float64).tiny))) and a.state == b.state


def test_sampling_options_of_any_number_type():
    """NumPy integers and floats, and a top_k past 64 bits, are the options that Python's own numbers are."""
    logits = np.random.default_rng(0).standard_normal(50)
    for kind in (np.int64, np.int32, np.uint8):
        o = gen.GenerationOptions(1, 0, temperature=np.float32(0.5), top_k=kind(3), top_p=np.float64(0.75), repetition_penalty=np.float32(1.25))
        want = gen.GenerationOptions(1, 0, temperature=0.5, top_k=3, top_p=0.75, repetition_penalty=1.25)
        assert gen.sample_token(logits, [1], o, gen.HeirloomRng(4)) == gen.sample_token(logits, [1], want, gen.HeirloomRng(4))
    assert gen.sample_token(logits, [], gen.GenerationOptions(1, 0, temperature=1.0, top_k=2 ** 64 + 1), gen.HeirloomRng(9)) == \
        gen.sample_token(logits, [], gen.GenerationOptions(1, 0, temperature=1.0), gen.HeirloomRng(9))


class Counting:
    """A model whose next token is the count of tokens so far."""
    def generate_token(self, tokens, length, appended, options, draw):
        assert tokens[:length].tolist() == list(range(length)) and appended == (length > 3)
        return length, 1.0, 0.0


def test_generation_until_eos_has_no_bound_on_its_tokens():
    """The token array grows with what is generated: a max_new_tokens that no memory would hold, an end after 2500 tokens; and a prefix of
    one-element tensors."""
    out = gen.generate(Counting(), [torch.tensor(0), np.int32(1), 2], gen.GenerationOptions(2 ** 60, 2499), gen.HeirloomRng(0))
    assert out.finish_reason == "eos" and out.tokens == list(range(2500)) and out.new_token_count == 2497
    out = gen.generate(Counting(), range(3), gen.GenerationOptions(1500, -1), gen.HeirloomRng(0))
    assert out.finish_reason == "max_new_tokens" and out.tokens == list(range(1503))


class OwnLogits:
    """A model that is not the library's: the token after the last one, modulo 7, gets most of the probability."""
    class cfg:
        context = 4

    def next_token_logits_device(self, window):
        out = np.zeros(7, np.float32)
        out[(int(window[-1]) + 1) % 7] = 5.0
        return out


def test_generation_over_a_model_that_only_gives_logits(monkeypatch):
    monkeypatch.setattr(torch.Tensor, "cuda", lambda self: self)
    out = gen.generate(OwnLogits(), [2, 3], gen.GenerationOptions(9, 10 ** 9), gen.HeirloomRng(0))
    assert out.tokens == [2, 3, 4, 5, 6, 0, 1, 2, 3, 4, 5]
    out = gen.generate(OwnLogits(), [2], gen.GenerationOptions(3, 10 ** 9, temperature=1.0, top_k=1), gen.HeirloomRng(7))
    rng = gen.HeirloomRng(7)
    [rng.uniform_f32() for _ in range(3)]
    assert out.tokens == [2, 3, 4, 5] and out.rng_state == rng.state


@pytest.mark.gpu
def test_generation_asks_an_overridden_method_for_the_logits():
    """A subclass, and an instance, that bans a token in next_token_logits_device: generate follows it."""
    from heirloom_b200 import nn
    from tests.gpu_util import ctx

    class Banning(nn.DecoderLm):
        def next_token_logits_device(self, window):
            out = super().next_token_logits_device(window)
            out[banned] = -100.0
            return out

    models = []
    for kind in (nn.DecoderLm, Banning, nn.DecoderLm):
        model = kind(ctx(), nn.DecoderConfig(vocab=64, d_model=64, n_layers=1, n_heads=1, d_ff=64, context=8, batch=1))
        rng = np.random.default_rng(1)
        model.load_state_dict({n: rng.standard_normal(s) * 0.3 for n, s in model.parameter_shapes().items()})
        models.append(model)
    banned = gen.generate_greedy(models[0], [1, 2], 1, -1)[-1]
    plain = models[2].next_token_logits_device
    models[2].next_token_logits_device = lambda window: np.where(np.arange(64) == banned, np.float32(-100.0), plain(window))
    chains = [gen.generate_greedy(m, [1, 2], 6, -1) for m in models]
    for m in models:
        m.close()
    assert banned in chains[0] and banned not in chains[1][2:] and chains[1] == chains[2]


HUGE_ROW = """
import ctypes
from heirloom_b200 import _lib, generation as gen
lib = _lib.load()
o = gen._sampling_options(gen.GenerationOptions(1, 0))
row, t, p, lp = (ctypes.c_double * 8)(), ctypes.c_int64(), ctypes.c_double(), ctypes.c_double()
for vocab in (1 << 60, 1 << 50):
    rc = lib.hl_sample_token(row, 2, ctypes.c_longlong(vocab), None, ctypes.c_longlong(0), ctypes.byref(o), ctypes.c_double(0.0),
                             ctypes.byref(t), ctypes.byref(p), ctypes.byref(lp))
    assert rc != 0
print(lib.hl_last_error().decode())
"""


def test_a_row_that_no_memory_holds_is_an_error_and_no_abort():
    import subprocess
    import sys
    from pathlib import Path
    res = subprocess.run([sys.executable, "-c", HUGE_ROW], cwd=str(Path(__file__).resolve().parents[1]), capture_output=True, text=True,
                         timeout=120)
    assert res.returncode == 0 and "hl_sample_token" in res.stdout, (res.returncode, res.stdout, res.stderr)


def test_option_validation_messages():
    for kwargs, text in ((dict(temperature=-1.0), "temperature must be non-negative"), (dict(top_k=0), "top_k must be greater than zero"),
                         (dict(top_p=0.0), "top_p must be in"), (dict(repetition_penalty=0.5), "at least 1.0"),
                         (dict(presence_penalty=-0.1), "must be non-negative")):
        with pytest.raises(Exception, match=text):
            gen.GenerationOptions(1, 0, **kwargs).validate()


@pytest.mark.gpu
def test_logits_eval_and_generation_on_the_device_match_the_oracle():
    import torch

    from heirloom_b200 import nn
    from tests.gpu_util import ctx
    c = ctx()
    kw = dict(vocab=64, d_model=64, n_layers=2, n_heads=1, d_ff=128, context=16)
    ocfg = ho.DecoderConfig(**kw)
    params = ho.init_parameters(ocfg, 4)
    rng = np.random.default_rng(2)
    for n in params:  # larger weights so that the argmax chain is not a string of near ties
        if n.endswith(".weight") and params[n].ndim == 2:
            params[n] = ho.f32_round(params[n] * 8.0)
    stream = rng.integers(0, 64, 16 * 5 + 3)
    for precision, tol in ((nn.PRECISION_F32, 2e-5), (nn.PRECISION_AMP_BF16, 3e-2)):
        amp = precision == nn.PRECISION_AMP_BF16
        model = nn.DecoderLm(c, nn.DecoderConfig(batch=3, precision=precision, **kw))
        model.load_state_dict(params)
        # windows shorter than, equal to and longer than the context
        for length in (1, 5, 16, 23):
            toks = stream[:length]
            got = gen.next_token_logits(model, toks)
            want = ho.decoder_logits(ocfg, params, toks[-16:][None, :], amp_bf16=amp)[0, -1]
            assert np.abs(got - want).max() <= tol * max(1.0, np.abs(want).max()), (precision, length)
        # evaluation: two full batches of 3 windows would need 6 windows; the stream holds 5, so the second batch has 2 rows
        m = gen.evaluate_token_loss(model, stream, 3)
        assert (m.batches, m.examples, m.tokens) == (2, 5, 80)
        rows = np.stack([stream[i * 16:(i + 1) * 16] for i in range(5)])
        tgts = np.stack([stream[i * 16 + 1:(i + 1) * 16 + 1] for i in range(5)])
        logits = ho.decoder_logits(ocfg, params, rows, amp_bf16=amp).reshape(80, 64)
        want_loss = float(ho.cross_entropy(logits, tgts.reshape(80)))
        assert m.loss == pytest.approx(want_loss, rel=1e-5 if not amp else 5e-3) and m.perplexity == pytest.approx(math.exp(m.loss))
        assert gen.evaluate_token_loss(model, stream, 2, max_batches=1).examples == 2
        with pytest.raises(Exception, match="more than block_size tokens"):
            gen.evaluate_token_loss(model, stream[:16], 2)
        if not amp:
            # greedy generation follows the oracle's argmax chain
            want_tokens = list(stream[:4])
            for _ in range(6):
                lg = ho.decoder_logits(ocfg, params, np.asarray(want_tokens[-16:])[None, :])[0, -1]
                want_tokens.append(gen.argmax_filtered(lg))
            got_tokens = gen.generate_greedy(model, stream[:4], 6, eos_id=10**9)
            assert got_tokens == [int(t) for t in want_tokens]
            out = gen.generate(model, stream[:4], gen.GenerationOptions(6, 10**9, temperature=1.0, top_k=1, top_p=1.0), gen.HeirloomRng(123))
            assert out.tokens == got_tokens and out.new_token_count == 6 and out.finish_reason == "max_new_tokens"
            assert all(s.probability > 0.0 for s in out.steps) and out.rng_state != 123
            eos = got_tokens[5]
            assert gen.generate(model, stream[:4], gen.GenerationOptions.greedy(6, eos), gen.HeirloomRng(0)).finish_reason == "eos"
        model.close()


@pytest.mark.gpu
@pytest.mark.parametrize("heads,memory", [(1, False), (2, False), (4, False), (1, True)])
def test_one_token_steps_equal_the_full_window(heads, memory):
    """prefill + decode_next against a full-window pass for every length from 1 to the context, head sizes 128, 64 and 32, with
    and without a memory block: f32 within the rounding of its sums, bf16 within a few steps of bf16 of the logits' scale
    (each of the two layers rounds its row to bf16 at about ten points, 2^-9 relative each)."""
    from heirloom_b200 import nn
    from tests.gpu_util import ctx
    c = ctx()
    kw = dict(vocab=72, d_model=128, n_layers=2, n_heads=heads, d_ff=200, context=19)
    mem = dict(memory_layers=(1,), slots=64, key_dim=32, value_dim=32, top_k=4)
    stream = np.random.default_rng(3).integers(0, 72, 19)
    for precision, tol in ((nn.PRECISION_F32, 2e-6), (nn.PRECISION_AMP_BF16, 3e-2)):
        batch = 64 if memory else 1
        model = nn.DecoderLm(c, nn.DecoderConfig(batch=batch, precision=precision, **kw), nn.MemoryConfig(**mem) if memory else None)
        rng = np.random.default_rng(heads)
        model.load_state_dict({n: (np.ones(s) if ".ln" in n or n.startswith("ln_f") else rng.standard_normal(s) * 0.1)
                               for n, s in ((n, s) for n, s in model.parameter_shapes().items())})
        got = [model.prefill(stream[:1])] + [model.decode_next(int(t)) for t in stream[1:]]
        assert model.cached_positions == 19
        with pytest.raises(Exception, match="context is full"):
            model.decode_next(0)
        for n in range(1, 20):
            want = gen.next_token_logits(model, stream[:n])
            assert np.abs(got[n - 1] - want).max() <= tol * max(1.0, np.abs(want).max()), (precision, n)
        assert model.cached_positions == 0
        with pytest.raises(Exception, match="no window is cached"):
            model.decode_next(0)
        model.close()


@pytest.mark.gpu
@pytest.mark.parametrize("d_model,heads,d_ff,context,prefix", [
    (16, 1, 8, 9, 1),          # the smallest: half a step of the contraction, one CTA with hidden units
    (48, 3, 200, 40, 30),      # heads of 16 channels, a slice of hidden units that is cut short
    (1024, 16, 4096, 24, 17),  # the widest row (f32: too much shared memory, kernels of their own)
    (256, 2, 776, 1024, 1000), # a thread's second key
    (128, 1, 64, 1030, 1021),  # contexts beyond that: kernels of their own
    (64, 8, 64, 19, 10),       # heads of 8 channels: kernels of their own
    (16, 1, 65536, 9, 1),      # a hidden unit a thread
    (16, 1, 65544, 9, 1),      # more of them: kernels of their own
])
def test_one_token_steps_of_all_sizes_equal_the_full_window(d_model, heads, d_ff, context, prefix):
    """prefill + decode_next against a full-window pass, on both sides of every limit of the kernels that take a block in two
    launches; the tolerances of the test above (the sums are as long or shorter, or grow with the row as the logits do)."""
    from heirloom_b200 import nn
    from tests.gpu_util import ctx
    c = ctx()
    stream = np.random.default_rng(d_model).integers(0, 72, context)
    for precision, tol in ((nn.PRECISION_F32, 2e-6), (nn.PRECISION_AMP_BF16, 3e-2)):
        model = nn.DecoderLm(c, nn.DecoderConfig(vocab=72, d_model=d_model, n_layers=2, n_heads=heads, d_ff=d_ff, context=context, batch=1,
                                                 precision=precision))
        rng = np.random.default_rng(heads)
        model.load_state_dict({n: (np.ones(s) if ".ln" in n or n.startswith("ln_f") else rng.standard_normal(s) * (0.1 if len(s) == 1 else s[-1] ** -0.5))
                               for n, s in ((n, s) for n, s in model.parameter_shapes().items())})
        lengths = range(prefix, min(context, prefix + 8) + 1)
        got = [model.prefill(stream[:prefix])] + [model.decode_next(int(stream[n - 1])) for n in lengths[1:]]
        for n, logits in zip(lengths, got):
            want = gen.next_token_logits(model, stream[:n])
            assert np.abs(logits - want).max() <= tol * max(1.0, np.abs(want).max()), (precision, n)
        model.close()


@pytest.mark.gpu
@pytest.mark.parametrize("vocab", [8, 2048, 2056, 50304])
def test_the_device_picks_the_greedy_token_that_sampling_picks(vocab):
    """The last maximum and its probability, the row cut into blocks of 2048 logits: the same token as the host's sampling of
    the same logits, the probability to the rounding of two f64 sums of `vocab` terms; ties go to the last index."""
    from heirloom_b200 import nn
    from tests.gpu_util import ctx
    c = ctx()
    model = nn.DecoderLm(c, nn.DecoderConfig(vocab=vocab, d_model=64, n_layers=1, n_heads=1, d_ff=64, context=4, batch=1))
    rng = np.random.default_rng(vocab)
    for tied in (False, True):
        state = {n: rng.standard_normal(s) * 0.3 for n, s in model.parameter_shapes().items()}
        if tied:
            state = {n: v * (0.0 if n.startswith("lm_head") else 1.0) for n, v in state.items()}
        model.load_state_dict(state)
        tokens = rng.integers(0, vocab, 4)
        options = gen.GenerationOptions.greedy(1, -1)
        for n in (1, 2, 4):
            got = model.generate_token(tokens, n, n == 2, gen._sampling_options(options), 0.0)
            want = gen.sample_token(gen.next_token_logits(model, tokens[:n]), tokens[:n], options, gen.HeirloomRng(0))
            assert got[0] == want[0] and (not tied or got[0] == vocab - 1)
            assert got[1] == pytest.approx(want[1], rel=vocab * 2e-16 + 1e-14)
    model.close()


@pytest.mark.gpu
@pytest.mark.parametrize("batch,vocab", [(13, 5000), (12, 8200), (20, 3208)])
def test_evaluation_loss_equals_the_training_pass_loss(batch, vocab):
    """The head's product that leaves maxima and sums per 128 columns, against the logits and the loss kernel of a training
    pass on the same tokens: last rows and columns ragged (1300 x 5000, 1200 x 8200, 2000 x 3208), one sequence of it, targets in
    the first and last column.  Both add f32 exponentials of the same f32 logits: a few ulps of the loss."""
    from heirloom_b200 import nn
    from tests.gpu_util import ctx
    c = ctx()
    model = nn.DecoderLm(c, nn.DecoderConfig(vocab=vocab, d_model=128, n_layers=1, n_heads=2, d_ff=128, context=100, batch=batch))
    rng = np.random.default_rng(vocab)
    model.load_state_dict({n: rng.standard_normal(s) * 0.2 for n, s in model.parameter_shapes().items()})
    x = torch.from_numpy(rng.integers(0, vocab, (batch, 100))).cuda()
    y = torch.from_numpy(rng.integers(0, vocab, (batch, 100))).cuda()
    y[0, :2] = torch.tensor([0, vocab - 1])
    model.forward_backward(x, y)
    want = model.loss()
    for _ in range(3):  # plain, captured, replayed
        assert model.eval_loss_device(x, y) == pytest.approx(want, rel=2e-6)
    whole = [model.eval_loss_device(x[i:i + 1], y[i:i + 1]) for i in range(batch)]
    assert np.mean(whole) == pytest.approx(want, rel=2e-6)
    model.close()


@pytest.mark.gpu
@pytest.mark.parametrize("masked", [-np.inf, -3.4e38])
@pytest.mark.parametrize("vocab,columns", [(5000, np.arange(384, 416)), (5000, np.arange(2048)), (16384, np.arange(16384).reshape(-1, 8, 128)[:8, 1])])
def test_evaluation_loss_with_masked_words(vocab, columns, masked):
    """Words switched off by their head bias: the first 32 columns of a block of 128, sixteen whole blocks, and the 2nd, 10th, ... 58th
    block of 128, which are what one warp of the loss kernel reads first.  They carry no probability; the loss is the training pass's."""
    from heirloom_b200 import nn
    from tests.gpu_util import ctx
    c = ctx()
    model = nn.DecoderLm(c, nn.DecoderConfig(vocab=vocab, d_model=128, n_layers=1, n_heads=2, d_ff=128, context=128, batch=32))
    rng = np.random.default_rng(vocab)
    state = {n: rng.standard_normal(s) * 0.2 for n, s in model.parameter_shapes().items()}
    columns = columns.reshape(-1)
    state["lm_head.bias"][columns] = masked
    model.load_state_dict(state)
    x = torch.from_numpy(rng.integers(0, vocab, (32, 128))).cuda()
    y = torch.from_numpy(rng.choice(np.setdiff1d(np.arange(vocab), columns), (32, 128))).cuda()
    model.forward_backward(x, y)
    want, got = model.loss(), model.eval_loss_device(x, y)
    model.close()
    assert math.isfinite(want) and got == pytest.approx(want, rel=2e-6)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [0, 1])
def test_evaluation_and_generation_report_the_device_status(precision):
    """Ids past the vocabulary, and products whose pipeline wait runs out (the bound shortened, one block left out, which the
    GEMM returns from with its status): an error from the call itself, a fourth and a fifth time too (plain, captured and replayed
    passes), nothing left for the next call, and the next passes are right."""
    from heirloom_b200 import nn
    from heirloom_b200._lib import HeirloomError
    from tests.gpu_util import ctx
    c = ctx()
    model = nn.DecoderLm(c, nn.DecoderConfig(vocab=64, d_model=64, n_layers=2, n_heads=1, d_ff=128, context=16, batch=2, precision=precision))
    rng = np.random.default_rng(3)
    model.load_state_dict({n: rng.standard_normal(s) * 0.2 for n, s in model.parameter_shapes().items()})
    good = torch.from_numpy(rng.integers(0, 64, (2, 16))).cuda()
    bad = good.clone()
    bad[1, 7] = 64
    calls = [(lambda ids: model.eval_loss_device(ids, good), good, bad), (lambda ids: model.eval_loss_device(good, ids), good, bad),
             (lambda ids: gen.next_token_logits(model, ids), [3, 63], [3, 64]),
             (lambda ids: gen.generate_greedy(model, ids, 3, 10 ** 9), [3, 63], [3, 64]),
             (lambda ids: model.prefill(np.array(ids, np.int64)), [3, 63], [3, 64])]
    outcomes = []

    def attempt(call, ids):
        try:
            return np.asarray(call(ids))
        except HeirloomError as e:
            return str(e)

    for call, right, wrong in calls:
        want = attempt(call, right)
        errors = [attempt(call, wrong) for _ in range(5)]
        outcomes.append((want, errors, attempt(call, right)))
    if precision == nn.PRECISION_AMP_BF16:  # the f32 route's products have no waits
        for call, right, _ in calls[:4]:
            want = attempt(call, right)
            c.set_test_hooks(wait_limit_ns=200_000, gemm_skip_kblock=0)
            try:
                error = attempt(call, right)
            finally:
                c.set_test_hooks(0, -1)
            outcomes.append((want, [error], attempt(call, right)))
    model.close()
    for want, errors, after in outcomes:
        assert all(isinstance(e, str) and ("out-of-range index" in e or "wait expired" in e) for e in errors), errors
        assert not isinstance(want, str) and np.array_equal(after, want)


@pytest.mark.gpu
@pytest.mark.parametrize("d_model,heads", [(128, 1), (128, 8), (256, 4)])
def test_one_token_steps_whose_peers_do_not_answer_end_in_an_error(d_model, heads):
    """The hook makes every CTA of a cluster wait for bytes that no peer sends: the step ends with an error after the limit, leaves nothing
    cached, and the same calls work afterwards.  f32, whose other kernels take no hook; the window's last block has the same exchange."""
    from heirloom_b200 import nn
    from heirloom_b200._lib import HeirloomError
    from tests.gpu_util import ctx
    c = ctx()
    model = nn.DecoderLm(c, nn.DecoderConfig(vocab=64, d_model=d_model, n_layers=2, n_heads=heads, d_ff=256, context=32, batch=1,
                                             precision=nn.PRECISION_F32))
    rng = np.random.default_rng(3)
    model.load_state_dict({n: rng.standard_normal(s) * 0.2 for n, s in model.parameter_shapes().items()})
    prompt = rng.integers(0, 64, 20)
    steps = lambda: [model.prefill(prompt)] + [model.decode_next(t) for t in (5, 6)]
    want = steps()
    for call in (lambda: model.decode_next(7), lambda: model.prefill(prompt)):
        model.prefill(prompt)
        c.set_test_hooks(wait_limit_ns=200_000, gemm_skip_kblock=0)
        try:
            with pytest.raises(HeirloomError, match="wait expired"):
                call()
        finally:
            c.set_test_hooks(0, -1)
        assert model.cached_positions == 0
        for got, right in zip(steps(), want):
            np.testing.assert_array_equal(got, right)
    model.close()


@pytest.mark.gpu
def test_a_pass_that_ends_in_an_error_leaves_no_cache():
    """A training pass that runs out of memory in its first block (its fc2 product, 20 x 4 tiles over a contraction of 12288, deals out
    k blocks and wants 19 MB of scratch), after it has overwritten the block's q/k/v rows of a cached window."""
    from heirloom_b200 import cuda, nn
    from tests.gpu_util import ctx, full_device
    ctx()
    rng = np.random.default_rng(0)
    x = torch.from_numpy(rng.integers(0, 64, (20, 128))).cuda()
    for warm in (True, False):  # a kernel whose first launch finds no memory stays unusable in its process: all of them run once before
        c = cuda.Context(0)  # no scratch yet
        model = nn.DecoderLm(c, nn.DecoderConfig(vocab=64, d_model=1024, n_layers=1, n_heads=16, d_ff=12288, context=128, batch=20))
        model.load_state_dict({n: rng.standard_normal(s) * 0.02 for n, s in model.parameter_shapes().items()})
        if warm:
            model.forward_backward(x, x)
            c.sync()
            model.close()
            c.close()
    model.prefill(rng.integers(0, 64, 8))
    raised = False
    with full_device():
        try:
            model.forward_backward(x, x)
        except Exception as e:
            raised = "memory" in str(e)
    cached = model.cached_positions
    model.close()
    c.close()
    assert raised and cached == 0


@pytest.mark.gpu
@pytest.mark.parametrize("memory_layers", [(0, 1), (0,)])
def test_routing_after_one_token_steps_is_the_window_s(memory_layers):
    """selected_indices and memory_access_counts after a window of five tokens and seven one-token steps, and after generate, are what
    the last full-window pass over the same tokens leaves (f32 queries to the rounding of f64 sums: no near-ties here)."""
    from heirloom_b200 import nn
    from tests.gpu_util import ctx
    c = ctx()
    mem = dict(memory_layers=memory_layers, slots=64, key_dim=32, value_dim=32, top_k=4)
    model = nn.DecoderLm(c, nn.DecoderConfig(vocab=72, d_model=128, n_layers=2, n_heads=2, d_ff=200, context=16, batch=1,
                                             precision=nn.PRECISION_F32), nn.MemoryConfig(**mem))
    rng = np.random.default_rng(5)
    model.load_state_dict({n: (np.ones(s) if ".ln" in n or n.startswith("ln_f") else rng.standard_normal(s) * 0.3)
                           for n, s in model.parameter_shapes().items()})
    read = lambda: ([model.selected_indices(l).copy() for l in memory_layers], model.memory_access_counts().row_counts)
    stream = rng.integers(0, 72, 12)
    gen.next_token_logits(model, stream)
    want = read()
    gen.next_token_logits(model, rng.integers(0, 72, 16))
    model.prefill(stream[:5])
    for t in stream[5:]:
        model.decode_next(int(t))
    got = [a[:12] for a in read()[0]]
    out = gen.generate_greedy(model, stream[:3], 9, -1)
    after = [a[:11] for a in read()[0]]
    gen.next_token_logits(model, out[:11])
    window = [a[:11] for a in read()[0]]
    gen.next_token_logits(model, stream)
    model.prefill(stream[:5])
    for t in stream[5:]:
        model.decode_next(int(t))
    counts = read()[1]
    gen.next_token_logits(model, stream)
    want_counts = read()[1]
    model.close()
    assert all(np.array_equal(g, w[:12]) for g, w in zip(got, want[0]))
    assert all(np.array_equal(g, w) for g, w in zip(after, window))
    assert np.array_equal(counts, want_counts)
