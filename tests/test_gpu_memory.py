"""Parity of the product-key memory kernels: the reference's known answers, exact index equality
against the oracle on identical f32 scores, and random forward/backward checks."""
import numpy as np
import pytest
import torch

from oracle import heirloom_oracle as ho
from tests.gpu_util import assert_close, ctx, dev, full_device, host

pytestmark = pytest.mark.gpu
I64 = torch.int64


def test_topk_ties_known_answer_and_random(golden):
    from heirloom_b200 import cuda
    c = ctx()
    ka = golden["known_answers"]["topk_ties"]
    got = host(cuda.topk_rows(c, dev(ka["scores"]), ka["k"]))
    assert got.tolist() == ka["indices"]
    rng = np.random.default_rng(0)
    for rows, cols, k in ((7, 5, 5), (64, 512, 32), (33, 1000, 17)):
        s = rng.integers(-20, 20, (rows, cols)).astype(np.float32) / 4  # many exact ties
        assert np.array_equal(host(cuda.topk_rows(c, dev(s), k)), ho.topk_indices_dim1(s, k))


def test_product_key_primitives_known_answers(golden):
    from heirloom_b200 import cuda
    c = ctx()
    ka = golden["known_answers"]["product_key_primitives"]
    idx = cuda.product_key_topk_from_side_scores(c, dev(ka["left_scores"]), dev(ka["right_scores"]), ka["top_k"], ka["beam"])
    assert host(idx).tolist() == [[5, 3], [6, 0]]
    left, right = cuda.product_key_split_rows(c, dev(ka["split_rows"]["rows"], I64), ka["side"])
    assert host(left).tolist() == ka["split_rows"]["left"] and host(right).tolist() == ka["split_rows"]["right"]
    q, kl, kr = dev(ka["query"]), dev(ka["left_keys"]), dev(ka["right_keys"])
    indices = dev(ka["indices"], I64)
    s = cuda.memory_selected_scores_forward(c, indices, q, kl, kr)
    assert_close("scores", host(s), ka["scores"], atol=1e-6)
    dq, dl, dr = cuda.memory_selected_scores_backward(c, indices, q, kl, kr, dev(ka["grad_scores"]))
    assert_close("dq", host(dq), ka["grad_query"], atol=1e-6)
    assert_close("dleft", host(dl), ka["grad_left"], atol=1e-6)
    assert_close("dright", host(dr), ka["grad_right"], atol=1e-6)


def test_exact_lookup_and_weighted_value_known_answers(golden):
    from heirloom_b200 import cuda
    c = ctx()
    ka = golden["known_answers"]["selected_scores"]
    indices = dev(ka["indices"], I64)
    s = cuda.memory_selected_scores_forward(c, indices, dev(ka["query"]), dev(ka["keys"]))
    assert_close("scores", host(s), ka["scores"], atol=1e-6)
    dq, dk, _ = cuda.memory_selected_scores_backward(c, indices, dev(ka["query"]), dev(ka["keys"]), None, dev(ka["grad_scores"]))
    assert_close("dq", host(dq), ka["grad_query"], atol=1e-6)
    assert_close("dkeys", host(dk), ka["grad_keys"], atol=1e-6)
    ka = golden["known_answers"]["weighted_value"]
    indices = dev(ka["indices"], I64)
    # value rows of 2 are padded to 4 columns (row_dim must be a multiple of 4)
    vals = np.zeros((3, 4), np.float32); vals[:, :2] = ka["values"]
    out = cuda.memory_weighted_value_forward(c, indices, dev(ka["weights"]), dev(vals))
    assert_close("out", host(out)[:, :2], ka["output"], atol=1e-6)
    go = np.zeros((2, 4), np.float32); go[:, :2] = 1.0
    dw, dv = cuda.memory_weighted_value_backward(c, indices, dev(ka["weights"]), dev(vals), dev(go))
    assert_close("dw", host(dw), ka["grad_weights"], atol=1e-6)
    assert_close("dv", host(dv)[:, :2], ka["grad_values"], atol=1e-6)


@pytest.mark.parametrize("tokens,side,key_dim,top_k", [(5, 8, 16, 4), (300, 64, 64, 8), (1000, 512, 512, 32)])
def test_side_scores_are_bit_exact_and_indices_equal_the_oracle(tokens, side, key_dim, top_k):
    from heirloom_b200 import cuda
    c = ctx()
    rng = np.random.default_rng(tokens + side)
    half = key_dim // 2
    q = rng.standard_normal((tokens, key_dim)).astype(np.float32)
    kl = (rng.standard_normal((side, half)) / np.sqrt(half)).astype(np.float32)
    kr = (rng.standard_normal((side, half)) / np.sqrt(half)).astype(np.float32)
    ls, rs = cuda.product_key_side_scores(c, dev(q), dev(kl), dev(kr))
    want_l, want_r = ho.side_scores_f32(q[:, :half], kl), ho.side_scores_f32(q[:, half:], kr)
    assert np.array_equal(host(ls).astype(np.float32).view(np.uint32), want_l.view(np.uint32))
    assert np.array_equal(host(rs).astype(np.float32).view(np.uint32), want_r.view(np.uint32))
    beam = ho.product_key_beam(side, top_k)
    idx = cuda.product_key_topk_from_side_scores(c, ls, rs, top_k, beam)
    assert np.array_equal(host(idx), ho.product_key_indices_from_side_scores(want_l, want_r, top_k, beam))
    # quantised scores: many exact ties on both sides and in the sums
    ql = np.round(want_l * 4) / 4
    qr = np.round(want_r * 4) / 4
    idx = cuda.product_key_topk_from_side_scores(c, dev(ql), dev(qr), top_k, beam)
    assert np.array_equal(host(idx), ho.product_key_indices_from_side_scores(ql, qr, top_k, beam))


@pytest.mark.parametrize("tokens,side,top_k", [(64, 2048, 32), (33, 24, 16), (40, 512, 1), (17, 100, 9)])
def test_product_key_selection_on_degenerate_scores(tokens, side, top_k):
    """All-equal scores, signed zeros, a handful of distinct values, -inf entries: the selection must still
    follow (descending score, ascending index) and (descending sum, ascending slot)."""
    from heirloom_b200 import cuda
    c = ctx()
    rng = np.random.default_rng(side * 7 + top_k)
    beam = ho.product_key_beam(side, top_k)
    cases = []
    zeros = np.zeros((tokens, side), np.float32)
    cases.append((zeros, zeros))
    signed = np.where(rng.random((tokens, side)) < 0.5, np.float32(0.0), np.float32(-0.0)).astype(np.float32)
    cases.append((signed, signed[::-1].copy()))
    few_l = rng.integers(-2, 3, (tokens, side)).astype(np.float32)
    few_r = rng.integers(-2, 3, (tokens, side)).astype(np.float32)
    cases.append((few_l, few_r))
    holes = rng.standard_normal((tokens, side)).astype(np.float32)
    holes[rng.random((tokens, side)) < 0.3] = -np.inf
    cases.append((holes, rng.standard_normal((tokens, side)).astype(np.float32) * 1e-3))
    wide = (rng.standard_normal((tokens, side)) * 10.0 ** rng.integers(-30, 30, (tokens, side))).astype(np.float32)
    cases.append((wide, -wide))
    for left, right in cases:
        idx = cuda.product_key_topk_from_side_scores(c, dev(left), dev(right), top_k, beam)
        assert np.array_equal(host(idx), ho.product_key_indices_from_side_scores(left, right, top_k, beam))


def test_memory_layer_forward_backward_random():
    from heirloom_b200 import cuda
    c = ctx()
    rng = np.random.default_rng(3)
    tokens, side, key_dim, top_k, dim = 200, 32, 64, 8, 64
    q = rng.standard_normal((tokens, key_dim)).astype(np.float32)
    kl = rng.standard_normal((side, key_dim // 2)).astype(np.float32) * 0.2
    kr = rng.standard_normal((side, key_dim // 2)).astype(np.float32) * 0.2
    vals = rng.standard_normal((side * side, dim)).astype(np.float32)
    idx = rng.integers(0, side * side, (tokens, top_k))
    idx[:, 1] = idx[:, 0]  # repeated rows inside one token
    di = dev(idx, I64)
    s = cuda.memory_selected_scores_forward(c, di, dev(q), dev(kl), dev(kr))
    so = ho.product_key_selected_scores(idx, q, kl, kr)
    assert_close("scores", host(s), so, atol=1e-6, rtol=1e-6)
    w = cuda.softmax_rows(c, s)
    wo = ho.softmax(so, 1)
    assert_close("weights", host(w), wo, atol=1e-7, rtol=1e-5)
    out = cuda.memory_weighted_value_forward(c, di, w, dev(vals))
    assert_close("weighted", host(out), ho.memory_weighted_value(idx, wo, vals), atol=1e-5, rtol=1e-5)
    go = rng.standard_normal((tokens, dim)).astype(np.float32)
    dw, dv = cuda.memory_weighted_value_backward(c, di, w, dev(vals), dev(go))
    dwo, dvo = ho.memory_weighted_value_backward(idx, wo, vals, go)
    assert_close("dw", host(dw), dwo, atol=1e-5, rtol=1e-5)
    assert_close("dv", host(dv), dvo, atol=1e-4, rtol=1e-4)
    ds = cuda.softmax_rows_backward(c, w, dw)
    dso = ho.softmax_backward(wo, dwo, 1)
    assert_close("dscores", host(ds), dso, atol=1e-5, rtol=1e-4)
    dq, dl, dr = cuda.memory_selected_scores_backward(c, di, dev(q), dev(kl), dev(kr), ds)
    dqo, dlo, dro = ho.product_key_selected_scores_backward(idx, q, kl, kr, dso)
    assert_close("dq", host(dq), dqo, atol=1e-5, rtol=1e-4)
    assert_close("dleft", host(dl), dlo, atol=1e-4, rtol=1e-4)
    assert_close("dright", host(dr), dro, atol=1e-4, rtol=1e-4)


@pytest.mark.parametrize("tokens,top_k,side,key_dim", [(2048, 32, 130, 128), (2049, 5, 100, 320), (3000, 32, 512, 512), (2500, 1, 7, 16), (2048, 33, 64, 64),
                                                       (4200, 8, 2048, 64), (9000, 4, 2048, 512)])
def test_half_key_gradients_of_many_tokens(tokens, top_k, side, key_dim):
    """Ragged rows (130 = 128 + 2), columns (160 = 2.5 chunks, 8) and last stages; one case has too many slots for the tensor-core form, and
    with 2048 rows a CTA walks 33 and 71 stages, past the 32 after which the small products' accumulator is emptied, once and twice.
    Slots repeat within a token, some are out of range.  f32 sums of exact products: 2^-20 of the terms' magnitudes covers both forms
    (3e-7 measured).  The same bits every time."""
    from heirloom_b200 import cuda
    c = ctx()
    gen = torch.Generator(device="cuda").manual_seed(tokens + side)
    idx = torch.randint(0, side * side, (tokens, top_k), generator=gen, device="cuda")
    idx[::3, -1] = idx[::3, 0]
    idx[5, 0], idx[6, 0] = -1, side * side
    q, kl, kr = (torch.randn(s, generator=gen, device="cuda") for s in ((tokens, key_dim), (side, key_dim // 2), (side, key_dim // 2)))
    g = torch.randn(tokens, top_k, generator=gen, device="cuda") * 10.0 ** torch.randint(-6, 3, (tokens, 1), generator=gen, device="cuda")
    torch.cuda.synchronize()
    _, dl, dr = cuda.memory_selected_scores_backward(c, idx, q, kl, kr, g)
    c.sync()
    good = (idx >= 0) & (idx < side * side)
    for rows, got, part in ((idx // side, dl, q[:, :key_dim // 2]), (idx % side, dr, q[:, key_dim // 2:])):
        w = torch.zeros(tokens, side, dtype=torch.float64, device="cuda").scatter_add_(1, rows.where(good, 0), g.double() * good)
        want, size = w.t() @ part.double(), w.abs().t() @ part.double().abs()
        assert ((got.double() - want).abs() <= size * 2.0 ** -20).all()
    again = cuda.memory_selected_scores_backward(c, idx, q, kl, kr, g)
    c.sync()
    assert torch.equal(again[1], dl) and torch.equal(again[2], dr)


@pytest.mark.parametrize("top_k", [4, 33])
@pytest.mark.parametrize("what,value", [("score", np.inf), ("score", -np.inf), ("score", np.nan), ("score", 3.4e38), ("score", 1e37), ("query", np.inf),
                                        ("query", np.nan), ("query", 3.4e38), ("query", -1e30), ("both", 1e38)])
def test_half_key_gradients_of_values_that_pieces_cannot_hold(top_k, what, value):
    """Infinities, NaN and values whose products overflow reach the same places as in a dense product of W and the queries, zeros of W
    included, in either form (33 slots a token: the f32 one).  f32 sums: 2^-20 of the terms' magnitudes where those stay finite."""
    from heirloom_b200 import cuda
    c = ctx()
    tokens, side, key_dim = 2050, 130, 48
    gen = torch.Generator(device="cuda").manual_seed(top_k)
    idx = torch.randint(0, side * side, (tokens, top_k), generator=gen, device="cuda")
    q, kl, kr, g = (torch.randn(s, generator=gen, device="cuda") for s in ((tokens, key_dim), (side, key_dim // 2), (side, key_dim // 2), (tokens, top_k)))
    q[70, 5] = 0.0
    if what in ("score", "both"):
        g[70, 2] = value
    if what == "query":
        q[2049, 7] = q[3, key_dim - 2] = value
    if what == "both":
        q[70, 4], q[70, key_dim - 1] = value, -value
    torch.cuda.synchronize()
    _, dl, dr = cuda.memory_selected_scores_backward(c, idx, q, kl, kr, g)
    c.sync()
    for rows, got, part in ((idx // side, dl, q[:, :key_dim // 2]), (idx % side, dr, q[:, key_dim // 2:])):
        w = torch.zeros(tokens, side, dtype=torch.float64, device="cuda").scatter_add_(1, rows, g.double())
        terms = w.t()[:, :, None] * part.double()[None]  # [side, tokens, half]
        want, size = terms.sum(1), terms.abs().sum(1)
        overflow = want.abs() > torch.finfo(torch.float32).max
        want = torch.where(overflow, want.sign() * float("inf"), want)
        assert torch.equal(got.isnan(), want.isnan())
        assert torch.equal(got.double()[want.isinf()], want[want.isinf()])
        fine = want.isfinite()
        assert ((got.double() - want)[fine].abs() <= size[fine] * 2.0 ** -20).all()


def test_half_key_gradients_without_room_for_the_tensor_cores_scratch():
    """Where the device has no room for the larger scratch, the f32 form runs in the arena that there is: nothing is given back or
    allocated again, call after call."""
    from heirloom_b200 import cuda
    tokens, top_k, side, key_dim = 4096, 8, 256, 512
    gen = torch.Generator(device="cuda").manual_seed(1)
    idx = torch.randint(0, side * side, (tokens, top_k), generator=gen, device="cuda")
    q, kl, kr, g = (torch.randn(s, generator=gen, device="cuda") for s in ((tokens, key_dim), (side, key_dim // 2), (side, key_dim // 2), (tokens, top_k)))
    wide = torch.cat((idx, torch.full((tokens, 33 - top_k), -1, dtype=torch.int64, device="cuda")), 1)  # too many slots for the tensor-core form
    g_wide = torch.cat((g, torch.zeros(tokens, 33 - top_k, device="cuda")), 1)
    torch.cuda.synchronize()
    cuda.memory_selected_scores_backward(ctx(), idx, q, kl, kr, g)  # the kernels are on the device
    ctx().sync()
    c = cuda.Context(0)
    try:
        want = cuda.memory_selected_scores_backward(c, wide, q, kl, kr, g_wide)
        c.sync()
        before = c.counters().allocations
        outs = [[torch.zeros_like(t) for t in want] for _ in range(2)]  # from here on nothing is allocated in this process
        torch.cuda.synchronize()
        with full_device():
            for out in outs:
                cuda.check(c.lib.hl_memory_selected_scores_backward(
                    c.handle, cuda._p(idx), cuda._p(q), cuda.c_longlong(key_dim), cuda._p(kl), cuda._p(kr), cuda._p(g), cuda._p(out[0]),
                    cuda.c_longlong(key_dim), cuda._p(out[1]), cuda._p(out[2]), cuda.c_int(tokens), cuda.c_int(top_k), cuda.c_int(side),
                    cuda.c_int(key_dim), cuda.c_int(side * side)))
            c.sync()
        assert c.counters().allocations == before
        assert all(torch.equal(a, b) for out in outs for a, b in zip(out[1:], want[1:]))
    finally:
        c.close()


@pytest.mark.parametrize("stage", [0, 4])
def test_a_half_key_gradient_whose_wait_runs_out_reports_it_and_the_next_call_is_right(stage):
    """A stage of tokens that the test hook keeps from arriving: every role leaves, and the next synchronisation reports the status."""
    from heirloom_b200 import cuda
    from heirloom_b200._lib import HeirloomError
    c = ctx()
    gen = torch.Generator(device="cuda").manual_seed(stage)
    idx = torch.randint(0, 900 * 900, (4096, 8), generator=gen, device="cuda")  # eight to fifteen stages a CTA
    q, kl, kr, g = (torch.randn(s, generator=gen, device="cuda") for s in ((4096, 128), (900, 64), (900, 64), (4096, 8)))
    torch.cuda.synchronize()
    want = cuda.memory_selected_scores_backward(c, idx, q, kl, kr, g)
    c.sync()
    c.set_test_hooks(wait_limit_ns=200_000, gemm_skip_kblock=stage)
    try:
        cuda.memory_selected_scores_backward(c, idx, q, kl, kr, g)
        with pytest.raises(HeirloomError, match="bounded pipeline wait expired"):
            c.sync()
    finally:
        c.set_test_hooks(0, -1)
    again = cuda.memory_selected_scores_backward(c, idx, q, kl, kr, g)
    c.sync()
    assert all(torch.equal(a, w) for a, w in zip(again, want))


@pytest.mark.parametrize("rows,cols", [(1, 8), (37, 64), (4096, 520)])
def test_the_fused_gate_rounds_as_the_single_ops(rows, cols):
    """gelu, products and pieces of a memory block's gate in one pass, forward and backward: the bits of an op after the other."""
    import ctypes
    from heirloom_b200 import cuda
    c = ctx()

    class Dest(ctypes.Structure):
        _fields_ = [("out", ctypes.c_void_p), ("ld", ctypes.c_longlong), ("piece", ctypes.c_longlong), ("n", ctypes.c_int), ("id", ctypes.c_int * 3)]

    forward = c.lib["_ZN2hl19memory_gate_forwardEP6hl_ctxPKfS3_PfS4_xiRKNS_9PieceDestE"]  # no entry point of the C header
    backward = c.lib["_ZN2hl20memory_gate_backwardEP6hl_ctxPKfS3_S3_S3_PfS4_xiRKNS_9PieceDestES7_"]
    gen = torch.Generator(device="cuda").manual_seed(rows)
    gpre, weighted, dmv = (torch.randn(rows, cols, generator=gen, device="cuda") * 3 for _ in range(3))
    new = lambda *shape, dtype=torch.float32: torch.full(shape, 7.0, dtype=dtype, device="cuda")
    gate, mv, dweighted, dgpre = (new(rows, cols) for _ in range(4))
    beside, stacked = new(rows, 2 * cols + 8, dtype=torch.bfloat16), new(3 * rows, cols, dtype=torch.bfloat16)
    side = Dest(beside.data_ptr(), 2 * cols + 8, cols, 2, (ctypes.c_int * 3)(0, 1, 0))
    rest = Dest(stacked.data_ptr(), cols, rows * cols, 3, (ctypes.c_int * 3)(0, 1, 2))

    def pieces(x):
        hi = x.to(torch.bfloat16)
        mid = (x - hi.float()).to(torch.bfloat16)
        return hi, mid, (x - hi.float() - mid.float()).to(torch.bfloat16)

    torch.cuda.synchronize()
    cuda.check(forward(c.handle, cuda._p(gpre), cuda._p(weighted), cuda._p(gate), cuda._p(mv), cuda.c_longlong(rows), cuda.c_int(cols), ctypes.byref(side)))
    want_gate = cuda.gelu(c, gpre)
    want_mv = cuda.binary_f32(c, 2, weighted, want_gate)
    c.sync()
    assert torch.equal(gate, want_gate) and torch.equal(mv, want_mv)
    assert torch.equal(beside[:, :2 * cols], torch.cat(pieces(mv)[:2], 1)) and (beside[:, 2 * cols:] == 7).all()
    cuda.check(backward(c.handle, cuda._p(dmv), cuda._p(gate), cuda._p(weighted), cuda._p(gpre), cuda._p(dweighted), cuda._p(dgpre),
                        cuda.c_longlong(rows), cuda.c_int(cols), ctypes.byref(rest), ctypes.byref(side)))
    want_dweighted = cuda.binary_f32(c, 2, dmv, gate)
    want_dgpre = cuda.gelu_backward(c, gpre, cuda.binary_f32(c, 2, dmv, weighted))
    c.sync()
    assert torch.equal(dweighted, want_dweighted) and torch.equal(dgpre, want_dgpre)
    assert torch.equal(stacked, torch.cat(pieces(dgpre), 0))
    assert torch.equal(beside[:, :2 * cols], torch.cat(pieces(dgpre)[:2], 1)) and (beside[:, 2 * cols:] == 7).all()


@pytest.mark.parametrize("key", ["sparse_adamw_unique_rows", "sparse_adamw_row_mask"])
def test_sparse_adamw_known_answers(golden, key):
    from heirloom_b200 import cuda
    c = ctx()
    ka = golden["known_answers"][key]
    # rows of 2 padded to 4 columns so the same data also exercises vector-friendly shapes
    p = dev(ka["param"]); g = dev(ka["grad"])
    m, v = torch.zeros_like(p), torch.zeros_like(p)
    mask = dev(np.asarray(ka["row_mask"], np.uint8), torch.uint8) if "row_mask" in ka else None
    hp = cuda.adamw_params(ka["lr"], 0.9, 0.999, 1e-8, ka["weight_decay"], 1.0, 1)
    cuda.sparse_adamw_rows(c, p, g, m, v, dev(ka["selected_rows"], I64), hp, row_mask=mask)
    assert_close(key, host(p), ka["expected"], atol=ka["tolerance"])


def test_sparse_adamw_updates_each_selected_row_once_and_only_those():
    from heirloom_b200 import cuda
    c = ctx()
    rng = np.random.default_rng(9)
    rows, dim = 1000, 48
    p0 = rng.standard_normal((rows, dim)).astype(np.float32)
    g0 = rng.standard_normal((rows, dim)).astype(np.float32)
    sel = rng.integers(0, rows, 3000)
    sel[:50] = 7
    p, g = dev(p0), dev(g0)
    m, v = torch.zeros_like(p), torch.zeros_like(p)
    hp = cuda.adamw_params(1e-2, 0.9, 0.999, 1e-8, 0.01, 1.0, 1)
    cuda.sparse_adamw_rows(c, p, g, m, v, dev(sel, I64), hp, zero_grad_rows=True)
    want, wm, wv = ho.adamw_step_f32_kernel_order(p0, g0, np.zeros_like(p0), np.zeros_like(p0), 1e-2, 0.9, 0.999, 1e-8,
                                                  0.01, 1.0, np.float32(1 - 0.9), np.float32(1 - 0.999))
    touched = np.zeros(rows, bool); touched[sel] = True
    got = host(p)
    assert np.array_equal(got[touched], want[touched].astype(np.float64))
    assert np.array_equal(got[~touched], p0[~touched].astype(np.float64))
    assert np.all(host(g)[touched] == 0) and np.array_equal(host(g)[~touched], g0[~touched].astype(np.float64))
    assert np.all(host(m)[~touched] == 0)


def test_bad_memory_index_sets_status():
    from heirloom_b200 import cuda
    from heirloom_b200._lib import HeirloomError
    c = ctx()
    vals = dev(np.zeros((4, 8), np.float32))
    cuda.memory_weighted_value_forward(c, dev([[0, 9]], I64), dev([[0.5, 0.5]]), vals)
    with pytest.raises(HeirloomError, match="out-of-range"):
        c.sync()


def test_row_masks_compaction_and_packed_rows():
    from heirloom_b200 import cuda
    c = ctx()
    rng = np.random.default_rng(31)
    rows, dim = 5000, 24
    selected = rng.integers(0, rows, 700)
    selected[:50] = selected[50:100]  # duplicates
    mask_in = (rng.random(rows) < 0.7).astype(np.uint8)
    sel = torch.tensor(selected, device="cuda")
    flags = cuda.mark_rows(c, sel, rows)
    want = np.zeros(rows, np.uint8); want[selected] = 1
    assert np.array_equal(host(flags), want)
    flags_m = cuda.mark_rows(c, sel, rows, row_mask=torch.tensor(mask_in, device="cuda"))
    assert np.array_equal(host(flags_m), want & mask_in)
    idx = cuda.mask_to_indices(c, flags)
    assert np.array_equal(host(idx), np.flatnonzero(want))  # ascending, each row once
    assert cuda.mask_to_indices(c, torch.zeros(rows, dtype=torch.uint8, device="cuda")).numel() == 0
    table = rng.standard_normal((rows, dim)).astype(np.float32)
    t = torch.tensor(table, device="cuda")
    packed = cuda.gather_rows(c, t, idx)
    assert np.array_equal(host(packed), table[np.flatnonzero(want)])
    dst = torch.zeros(rows, dim, device="cuda")
    cuda.scatter_rows(c, packed * 2.0, idx, dst)
    c.sync()
    expect = np.zeros_like(table); expect[np.flatnonzero(want)] = 2.0 * table[np.flatnonzero(want)]
    assert np.array_equal(host(dst), expect)
    # clip norm over the active rows only: a set, filtered by the mask
    got = cuda.sparse_rows_sum_squares(c, t, sel, row_mask=torch.tensor(mask_in, device="cuda"))
    active = np.flatnonzero(want & mask_in)
    assert got == pytest.approx(float((table[active].astype(np.float64) ** 2).sum()), rel=1e-12)


@pytest.mark.parametrize("tokens,top_k,rows,dim", [(4096, 16, 1024, 256), (2048, 32, 300, 512), (4100, 8, 70000, 64),
                                                   (1030, 32, 4096, 640)])
def test_weighted_value_backward_in_row_order_matches_a_host_sum(tokens, top_k, rows, dim):
    """Event counts from 32768 up take the row-ordered path (sort by row, one set of atomics per run): many events per
    row, rows nobody selected, chunk boundaries inside a run, a row count that is not a power of two."""
    from heirloom_b200 import cuda
    c = ctx()
    rng = np.random.default_rng(tokens + rows)
    idx = (rng.zipf(1.3, (tokens, top_k)) % rows).astype(np.int64)
    idx[0, :] = rows - 1                      # the last row, a whole token's worth
    w = rng.standard_normal((tokens, top_k)).astype(np.float32)
    vals = rng.standard_normal((rows, dim)).astype(np.float32)
    go = rng.standard_normal((tokens, dim)).astype(np.float32)
    dw, dv = cuda.memory_weighted_value_backward(c, dev(idx, I64), dev(w), dev(vals), dev(go))
    want_dw = np.einsum("td,tkd->tk", go.astype(np.float64), vals[idx].astype(np.float64))
    want_dv = np.zeros((rows, dim), np.float64)
    np.add.at(want_dv, idx.reshape(-1), (w[..., None].astype(np.float64) * go[:, None, :]).reshape(-1, dim))
    assert_close("dw", host(dw), want_dw, atol=1e-5, rtol=1e-6)
    scale = np.abs(want_dv).max()
    assert np.abs(host(dv) - want_dv).max() <= 2e-6 * scale * np.sqrt(tokens * top_k / max(np.unique(idx).size, 1)) + 1e-5
    untouched = np.ones(rows, bool); untouched[np.unique(idx)] = False
    assert not np.any(host(dv)[untouched])


def test_row_ordered_value_backward_reports_a_bad_index_and_zeroes_its_weight_gradient():
    """An index past the table in the row-ordered path: the event is left out of the row sums, its weight gradient is
    written as zero (not left as stale scratch), and the next sync reports the status word; nothing faults."""
    from heirloom_b200 import cuda
    from heirloom_b200._lib import HeirloomError
    c = ctx()
    rng = np.random.default_rng(77)
    tokens, top_k, rows, dim = 2048, 32, 500, 64
    idx = rng.integers(0, rows, (tokens, top_k)).astype(np.int64)
    idx[5, 3], idx[100, 0] = rows, -1
    w = rng.standard_normal((tokens, top_k)).astype(np.float32)
    vals = rng.standard_normal((rows, dim)).astype(np.float32)
    go = rng.standard_normal((tokens, dim)).astype(np.float32)
    c.sync()
    dw, dv = cuda.memory_weighted_value_backward(c, dev(idx, I64), dev(w), dev(vals), dev(go))
    with pytest.raises(HeirloomError, match="out-of-range index"):
        c.sync()
    c.sync()
    got = dw.cpu().numpy()
    assert got[5, 3] == 0.0 and got[100, 0] == 0.0
    good = np.ones_like(idx, bool); good[5, 3] = good[100, 0] = False
    want_dw = np.einsum("td,tkd->tk", go.astype(np.float64), vals[np.clip(idx, 0, rows - 1)].astype(np.float64))
    assert np.allclose(got[good], want_dw[good], rtol=1e-5, atol=1e-5)


@pytest.mark.parametrize("tokens,top_k,side,key_dim,dim", [(37, 5, 9, 16, 4), (65, 33, 20, 136, 132), (41, 40, 16, 512, 512), (20, 32, 16, 1024, 1024),
                                                           (9, 7, 12, 1032, 1028), (30, 9, 10, 12, 8), (6400, 16, 40, 256, 260), (3200, 33, 30, 264, 640)])
def test_gathers_at_the_edges_of_their_forms(tokens, top_k, side, key_dim, dim):
    """Rows of one piece to more than a warp's, slots that fill no group of eight, forms for any size, few and many events of the value
    backward.  Bounds: f32 sums of at most 64 products (or top_k of them, or an event's run), so 2^-24 sqrt of that many of the terms'
    magnitudes, times a few."""
    from heirloom_b200 import cuda
    c = ctx()
    rng = np.random.default_rng(tokens + key_dim)
    q = rng.standard_normal((tokens, key_dim)).astype(np.float32)
    kl, kr = (rng.standard_normal((side, key_dim // 2)).astype(np.float32) for _ in range(2))
    vals = rng.standard_normal((side * side, dim)).astype(np.float32)
    idx = rng.integers(0, side * side, (tokens, top_k))
    idx[:, 1] = idx[:, 0]
    idx[-1, -1] = side * side - 1
    w = rng.random((tokens, top_k)).astype(np.float32)
    g = rng.standard_normal((tokens, top_k)).astype(np.float32)
    go = rng.standard_normal((tokens, dim)).astype(np.float32)
    di = dev(idx, I64)
    keys = np.concatenate([kl[idx // side], kr[idx % side]], axis=2).astype(np.float64)
    assert_close("scores", host(cuda.memory_selected_scores_forward(c, di, dev(q), dev(kl), dev(kr))), np.einsum("td,tkd->tk", q.astype(np.float64), keys),
                 atol=4e-6 * np.sqrt(key_dim), rtol=1e-6)
    dq, _, _ = cuda.memory_selected_scores_backward(c, di, dev(q), dev(kl), dev(kr), dev(g))
    assert_close("dq", host(dq), np.einsum("tk,tkd->td", g.astype(np.float64), keys), atol=4e-6 * np.sqrt(top_k), rtol=1e-6)
    picked = vals[idx].astype(np.float64)
    assert_close("value", host(cuda.memory_weighted_value_forward(c, di, dev(w), dev(vals))), np.einsum("tk,tkd->td", w.astype(np.float64), picked),
                 atol=4e-6 * np.sqrt(top_k), rtol=1e-6)
    dw, dv = cuda.memory_weighted_value_backward(c, di, dev(w), dev(vals), dev(go))
    assert_close("dw", host(dw), np.einsum("td,tkd->tk", go.astype(np.float64), picked), atol=4e-6 * np.sqrt(dim), rtol=1e-6)
    want = np.zeros((side * side, dim))
    np.add.at(want, idx.reshape(-1), (w[..., None].astype(np.float64) * go[:, None, :]).reshape(-1, dim))
    run = np.bincount(idx.reshape(-1)).max()
    assert_close("dv", host(dv), want, atol=1e-6 * np.sqrt(run) * 4 + 2e-7 * run, rtol=1e-6)


@pytest.mark.parametrize("tokens,side,key_dim,top_k", [(1, 8, 64, 5), (259, 40, 64, 32), (300, 512, 512, 32), (1001, 256, 192, 16), (257, 504, 1024, 1)])
@pytest.mark.parametrize("kind", ["random", "ties", "near", "huge", "tiny", "odd"])
def test_lookup_of_the_step_selects_what_exact_scores_do(tokens, side, key_dim, top_k, kind):
    """Scores that decide are formed in the order of hl_product_key_side_scores_f32, so the rows are the same, in order; also where many
    keys tie, lie closer than the approximation tells apart, or are out of its range."""
    from ctypes import c_int

    from heirloom_b200 import cuda
    c = ctx()
    rng = np.random.default_rng(side + key_dim)
    half = key_dim // 2
    q = rng.standard_normal((max(tokens, 10), key_dim)).astype(np.float32)
    keys = [rng.standard_normal((side, half)).astype(np.float32) for _ in range(2)]
    if kind == "ties":  # 16 distinct keys; whole numbers, whose sums are exact, in the right table
        keys[0] = keys[0][rng.integers(0, min(side, 16), side)]
        keys[1], q[:, half:] = rng.integers(-2, 3, keys[1].shape), rng.integers(-2, 3, (len(q), half))
    elif kind == "near":  # all of the left table within a few units in the last place
        keys[0] = (keys[0][:1] * (1 + 2e-7 * rng.standard_normal((side, half)))).astype(np.float32)
    elif kind == "huge":
        q[::2] *= 1e20
        q[1::4] *= 1e30
        keys[1] *= 1e7
    elif kind == "tiny":
        q[::2] *= 1e-25
        q[1::4, :half] = 0
        keys[1] *= 1e-20
    elif kind == "odd":
        q[3, 1], q[5, half], q[8], q[9, 0] = np.inf, -np.inf, 3e38, np.nan
        keys[0][side - 1, 0] = np.inf
    beam = min(side, max(top_k, int(np.ceil(np.sqrt(top_k)))))
    query, left, right = dev(q[:tokens]), dev(keys[0].astype(np.float32)), dev(keys[1].astype(np.float32))
    want = cuda.product_key_topk_from_side_scores(c, *cuda.product_key_side_scores(c, query, left, right), top_k, beam)
    got = torch.full_like(want, -1)
    pieces = torch.empty(6 * side * key_dim + 256, dtype=torch.uint8, device="cuda")
    query_pieces = torch.empty(tokens, 2 * key_dim, dtype=torch.bfloat16, device="cuda")
    approx = torch.empty(2, tokens, side, device="cuda")
    cuda.check(c.lib.hl_product_key_lookup(c.handle, cuda._p(query), cuda._p(left), cuda._p(right), cuda._p(pieces), cuda._p(query_pieces),
                                           cuda._p(approx[0]), cuda._p(approx[1]), cuda._p(got), c_int(tokens), c_int(side), c_int(key_dim),
                                           c_int(top_k), c_int(beam)))
    np.testing.assert_array_equal(host(got), host(want))


@pytest.mark.parametrize("tokens,side,key_dim,top_k", [(64, 64, 64, 8), (130, 512, 128, 32), (257, 256, 1024, 16)])
def test_lookup_of_values_whose_pieces_are_at_their_worst(tokens, side, key_dim, top_k):
    """1 + 2^-8 - 2^-17 - 2^-23 and 1 + 2^-8 - 2^-16 and their like, of either sign: a bf16 piece leaves 2^-8 of them, two leave 2^-17.  The
    approximate scores are off by what was derived, 2^-15 S from the pieces and 17 terms cut off at 2^-23 in each of the 3 half / 16
    steps.  More than 3 * 2^-18 S is seen.  Selected rows as by exact scores."""
    from ctypes import c_int

    from heirloom_b200 import cuda
    c = ctx()
    rng = np.random.default_rng(side + key_dim)
    half = key_dim // 2
    worst = np.array([1 + 2 ** -8 - 2 ** -17 - 2 ** -23, 1 + 2 ** -8 - 2 ** -16, 1 + 2 ** -8 - 2 ** -17], np.float32)
    draw = lambda *shape: (rng.choice(worst, shape, p=[0.8, 0.1, 0.1]) * rng.choice([1, 1, 1, -1], shape)).astype(np.float32)
    q, keys = draw(tokens, key_dim), [draw(side, half) for _ in range(2)]
    q[0], keys[0][0], keys[1][-1] = np.abs(q[0]), np.abs(keys[0][0]), np.abs(keys[1][-1])
    query, left, right = dev(q), dev(keys[0]), dev(keys[1])
    beam = min(side, max(top_k, int(np.ceil(np.sqrt(top_k)))))
    want = cuda.product_key_topk_from_side_scores(c, *cuda.product_key_side_scores(c, query, left, right), top_k, beam)
    got = torch.full_like(want, -1)
    pieces = torch.empty(6 * side * key_dim + 256, dtype=torch.uint8, device="cuda")
    query_pieces = torch.empty(tokens, 2 * key_dim, dtype=torch.bfloat16, device="cuda")
    approx = torch.empty(2, tokens, side, device="cuda")
    cuda.check(c.lib.hl_product_key_lookup(c.handle, cuda._p(query), cuda._p(left), cuda._p(right), cuda._p(pieces), cuda._p(query_pieces),
                                           cuda._p(approx[0]), cuda._p(approx[1]), cuda._p(got), c_int(tokens), c_int(side), c_int(key_dim),
                                           c_int(top_k), c_int(beam)))
    np.testing.assert_array_equal(host(got), host(want))
    seen = 0.0
    for sd in range(2):
        x, k = q[:, sd * half:][:, :half].astype(np.float64), keys[sd].astype(np.float64)
        s = np.linalg.norm(x, axis=1)[:, None] * np.linalg.norm(k, axis=1).max()
        off = np.abs(host(approx[sd]).astype(np.float64) - x @ k.T) / s
        assert off.max() <= 2 ** -15 + 3 * half / 16 * 17 * 2 ** -23
        seen = max(seen, off.max())
    assert seen > 3 * 2 ** -18


def test_lookup_refuses_what_its_kernels_cannot_take():
    """On the host, before anything is launched: sizes of the general form, more slots than the beams have pairs, no pointer, and one that
    sixteen-byte loads cannot read."""
    from ctypes import c_int, c_void_p

    from heirloom_b200 import cuda
    c = ctx()
    room = torch.zeros(1 << 20, dtype=torch.uint8, device="cuda")
    at = lambda i: c_void_p(room.data_ptr() + 65536 * i)

    def refused(match, tokens=4, side=16, key_dim=64, top_k=4, beam=4, **pointers):
        p = [pointers.get(n, at(i)) for i, n in enumerate(("query", "left", "right", "pieces", "query_pieces", "left_approx", "right_approx", "out"))]
        with pytest.raises(cuda.HeirloomError, match=match):
            cuda.check(c.lib.hl_product_key_lookup(c.handle, *p, c_int(tokens), c_int(side), c_int(key_dim), c_int(top_k), c_int(beam)))
    before = c.counters().launches
    for sizes in (dict(side=12), dict(side=520), dict(key_dim=96), dict(key_dim=1088)):
        refused("must be a multiple", **sizes)
    refused("top_k", top_k=17)
    refused("top_k", top_k=0)
    refused("beam", beam=17)
    refused("beam", side=64, beam=33)
    refused("non-zero", tokens=0)
    for i, name in enumerate(("query", "left", "right", "pieces", "query_pieces", "left_approx", "right_approx", "out")):
        refused("null", **{name: c_void_p(0)})
        refused("aligned", **{name: c_void_p(room.data_ptr() + 65536 * i + 4)})
    assert c.counters().launches == before
    c.sync()


@pytest.mark.parametrize("tokens", [65, 2048])
def test_half_key_gradients_without_the_querys(tokens):
    """A call for the tables' gradients alone gives the bits of one for all three, with no launch more; also behind a call whose
    values are too wide for bf16 pieces, which sets a word that every call of that form clears."""
    from ctypes import c_int, c_longlong, c_void_p

    from heirloom_b200 import cuda
    c = ctx()
    rng = np.random.default_rng(tokens)
    side, key_dim, top_k = 24, 64, 8
    q, g = dev(rng.standard_normal((tokens, key_dim)).astype(np.float32)), dev(rng.standard_normal((tokens, top_k)).astype(np.float32))
    kl, kr = (dev(rng.standard_normal((side, key_dim // 2)).astype(np.float32)) for _ in range(2))
    idx = dev(rng.integers(0, side * side, (tokens, top_k)), I64)

    def tables(query):
        dl, dr = torch.zeros_like(kl), torch.zeros_like(kr)
        cuda.check(c.lib.hl_memory_selected_scores_backward(
            c.handle, cuda._p(idx), cuda._p(query), c_longlong(key_dim), cuda._p(kl), cuda._p(kr), cuda._p(g), c_void_p(0), c_longlong(key_dim),
            cuda._p(dl), cuda._p(dr), c_int(tokens), c_int(top_k), c_int(side), c_int(key_dim), c_int(side * side)))
        return dl, dr
    before = c.counters().launches
    _, dl, dr = cuda.memory_selected_scores_backward(c, idx, q, kl, kr, g)
    whole = c.counters().launches - before
    wide = q.clone()
    wide[3, 5] = 2.0 ** 50
    for query in (q, wide, q):
        before = c.counters().launches
        got = tables(query)
        assert c.counters().launches - before <= whole
    assert torch.equal(got[0], dl) and torch.equal(got[1], dr)


@pytest.mark.parametrize("tokens,top_k,key_dim,dim", [(1, 1, 8, 4), (37, 1, 512, 1024), (1100, 2, 264, 516), (300, 3, 1024, 640), (65, 8, 256, 260),
                                                      (66, 9, 512, 256), (67, 16, 128, 128), (69, 17, 384, 132), (4097, 3, 64, 388)])
def test_gathers_of_few_slots(tokens, top_k, key_dim, dim):
    """One, two and four warps or pieces of a row for a token, at the slots and columns where one gives way to the other, with a slot that
    does not exist.  Bounds as in the test of the forms' edges above."""
    from heirloom_b200 import cuda
    c = ctx()
    rng = np.random.default_rng(tokens + key_dim)
    side = 16
    q = rng.standard_normal((tokens, key_dim)).astype(np.float32)
    kl, kr = (rng.standard_normal((side, key_dim // 2)).astype(np.float32) for _ in range(2))
    vals = rng.standard_normal((side * side, dim)).astype(np.float32)
    idx = rng.integers(0, side * side, (tokens, top_k))
    w, g = (rng.standard_normal((tokens, top_k)).astype(np.float32) for _ in range(2))
    go = rng.standard_normal((tokens, dim)).astype(np.float32)
    for bad in (None, side * side, -1):
        if bad is not None:
            idx[tokens // 2, top_k - 1] = bad
        there = (idx >= 0) & (idx < side * side)
        at = np.where(there, idx, 0)
        di = dev(idx, I64)
        keys = np.concatenate([kl[at // side], kr[at % side]], axis=2).astype(np.float64) * there[..., None]
        picked = vals[at].astype(np.float64) * there[..., None]
        scores = cuda.memory_selected_scores_forward(c, di, dev(q), dev(kl), dev(kr))
        dq, _, _ = cuda.memory_selected_scores_backward(c, di, dev(q), dev(kl), dev(kr), dev(g))
        value = cuda.memory_weighted_value_forward(c, di, dev(w), dev(vals))
        dw, dv = cuda.memory_weighted_value_backward(c, di, dev(w), dev(vals), dev(go))
        if bad is None:
            c.sync()
        else:
            with pytest.raises(cuda.HeirloomError, match="out-of-range index"):
                c.sync()
        assert_close("scores", host(scores), np.einsum("td,tkd->tk", q.astype(np.float64), keys), atol=4e-6 * np.sqrt(key_dim), rtol=1e-6)
        assert_close("dq", host(dq), np.einsum("tk,tkd->td", g.astype(np.float64), keys), atol=4e-6 * np.sqrt(top_k), rtol=1e-6)
        assert_close("value", host(value), np.einsum("tk,tkd->td", w.astype(np.float64), picked), atol=4e-6 * np.sqrt(top_k), rtol=1e-6)
        assert_close("dw", host(dw)[there], np.einsum("td,tkd->tk", go.astype(np.float64), picked)[there], atol=4e-6 * np.sqrt(dim), rtol=1e-6)
        want = np.zeros((side * side, dim))
        np.add.at(want, at[there], w[there][:, None].astype(np.float64) * np.repeat(go[:, None], top_k, 1)[there])
        run = np.bincount(at[there], minlength=1).max()
        assert_close("dv", host(dv), want, atol=1e-6 * np.sqrt(run) * 4 + 2e-7 * run, rtol=1e-6)
