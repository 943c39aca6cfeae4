"""Parity of the tcgen05 flash attention against the oracle's attention on bf16-valued inputs."""
import numpy as np
import pytest
import torch

from oracle import heirloom_oracle as ho
from tests.gpu_util import assert_close, ctx, dev, host

pytestmark = pytest.mark.gpu


def reference_lse(q, k, n_heads):
    B, T, C = q.shape
    hd = C // n_heads
    qh = q.reshape(B, T, n_heads, hd).transpose(0, 2, 1, 3)
    kh = k.reshape(B, T, n_heads, hd).transpose(0, 2, 1, 3)
    s = np.matmul(qh, kh.transpose(0, 1, 3, 2)) / np.sqrt(hd)
    s = np.where(np.tril(np.ones((T, T), bool)), s, -np.inf)
    m = s.max(-1)
    return m + np.log(np.exp(s - m[..., None]).sum(-1))


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("B,T,H", [(1, 128, 1), (2, 256, 3), (1, 200, 2), (2, 1024, 2), (1, 72, 4), (1, 4096, 1), (1, 2100, 2)])
def test_flash_forward_matches_oracle(B, T, H, hd):
    from heirloom_b200 import cuda
    c = ctx()
    C = hd * H
    rng = np.random.default_rng(B * 1000 + T + H)
    qkv = ho.bf16_round(rng.standard_normal((B * T, 3 * C)) * 1.2)
    fused = dev(qkv, torch.bfloat16)
    q, k, v = fused[:, :C], fused[:, C:2 * C], fused[:, 2 * C:]
    out, lse = cuda.flash_attention_forward(c, q, k, v, B, T, H)
    assert out.shape == (B * T, C)
    qn, kn, vn = (qkv[:, i * C:(i + 1) * C].reshape(B, T, C) for i in range(3))
    want = ho.causal_attention(qn, kn, vn, H, round_probs_bf16=True)
    # P is rounded to bf16 before the PV product (as the reference's tensor-core route does) and
    # the row maximum it is rounded against may differ by tile order: allow 2 bf16 ulps + 1e-2.
    assert_close("flash out", host(out).reshape(B, T, C), want, atol=1e-2, rtol=2 ** -6)
    assert_close("lse", host(lse), reference_lse(qn, kn, H), atol=1e-4, rtol=1e-5)


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("B,T,H", [(1, 1, 1), (2, 33, 1), (1, 65, 3), (3, 97, 2), (1, 129, 2), (90, 64, 5), (40, 200, 6)])
def test_flash_forward_of_streams_with_several_items_and_rising_scores(B, T, H, hd):
    """Items fewer and more than the streams of the chip, tiles of which a warp's rows see none, one or both halves, and scores that grow
    along the keys, so that rows raise the maximum that P is formed against (by far more than 2^8) in most tiles.  Bounds as above: P has
    one bf16 rounding, whatever it is formed against."""
    from heirloom_b200 import cuda
    c = ctx()
    C = hd * H
    rng = np.random.default_rng(T + H)
    qkv = rng.standard_normal((B, T, 3 * C)) * 1.2
    qkv[..., C:2 * C] = 0.1 * qkv[..., C:2 * C] + np.linspace(0, 4, T)[None, :, None]
    qkv[..., :C] = np.abs(qkv[..., :C])
    qkv = ho.bf16_round(qkv.reshape(B * T, 3 * C))
    fused = dev(qkv, torch.bfloat16)
    out, lse = cuda.flash_attention_forward(c, fused[:, :C], fused[:, C:2 * C], fused[:, 2 * C:], B, T, H)
    qn, kn, vn = (qkv[:, i * C:(i + 1) * C].reshape(B, T, C) for i in range(3))
    want = ho.causal_attention(qn, kn, vn, H, round_probs_bf16=True)
    assert_close("flash out", host(out).reshape(B, T, C), want, atol=1e-2, rtol=2 ** -6)
    assert_close("lse", host(lse), reference_lse(qn, kn, H), atol=1e-4, rtol=1e-5)


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("B,T,H", [(4, 4096, 12), (64, 300, 8)])
def test_flash_forward_gives_the_same_bits_every_time(B, T, H, hd):
    """Nothing in it depends on the order of events: P that is replaced, or O that is rescaled, before a product has read or written it
    shows as rows that differ from call to call."""
    from heirloom_b200 import cuda
    c = ctx()
    C = hd * H
    qkv = torch.randn(B * T, 3 * C, device="cuda", generator=torch.Generator(device="cuda").manual_seed(T)).to(torch.bfloat16)
    q, k, v = qkv.split(C, dim=1)
    torch.cuda.synchronize()
    first = cuda.flash_attention_forward(c, q, k, v, B, T, H)
    for _ in range(8):
        again = cuda.flash_attention_forward(c, q, k, v, B, T, H)
        c.sync()
        assert torch.equal(again[0], first[0]) and torch.equal(again[1], first[1])


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("B,T,H", [(4, 2048, 10), (1, 4096, 20), (64, 300, 8)])
def test_flash_backward_gives_the_same_dk_and_dv_every_time(B, T, H, hd):
    """dK and dV are sums in a fixed order (dQ's parts are not): P that is replaced before dV has read it, or dS before dK has, shows as rows
    that differ from call to call."""
    from heirloom_b200 import cuda
    c = ctx()
    C = hd * H
    gen = torch.Generator(device="cuda").manual_seed(T)
    qkv = torch.randn(B * T, 3 * C, device="cuda", generator=gen).to(torch.bfloat16)
    dout = torch.randn(B * T, C, device="cuda", generator=gen).to(torch.bfloat16)
    q, k, v = qkv.split(C, dim=1)
    torch.cuda.synchronize()
    out, lse = cuda.flash_attention_forward(c, q, k, v, B, T, H)
    first = cuda.flash_attention_backward(c, q, k, v, out, dout, lse, B, T, H)
    for _ in range(8):
        again = cuda.flash_attention_backward(c, q, k, v, out, dout, lse, B, T, H)
        c.sync()
        assert torch.equal(again[:, C:], first[:, C:])


@pytest.mark.parametrize("T,H", [(128, 12), (300, 8), (1000, 5), (2048, 4)])
def test_flash_forward_of_a_batch_equals_its_entries(T, H):
    """Heads of 64 take three streams an SM where there are many items and two where there are few: the same sums in the same order."""
    from heirloom_b200 import cuda
    c = ctx()
    C, B = 64 * H, 40
    qkv = torch.randn(B * T, 3 * C, device="cuda", generator=torch.Generator(device="cuda").manual_seed(T)).to(torch.bfloat16)
    q, k, v = qkv.split(C, dim=1)
    out, lse = cuda.flash_attention_forward(c, q, k, v, B, T, H)
    for b in (0, 17, 39):
        rows = slice(b * T, (b + 1) * T)
        alone = cuda.flash_attention_forward(c, q[rows], k[rows], v[rows], 1, T, H)
        c.sync()
        assert torch.equal(alone[0], out[rows]) and torch.equal(alone[1].reshape(-1), lse[b].reshape(-1))


def test_flash_forward_rejects_unsupported_shapes():
    from heirloom_b200 import cuda
    from heirloom_b200._lib import HeirloomError
    c = ctx()
    x = c.zeros((128, 96), torch.bfloat16)
    with pytest.raises(HeirloomError, match="head_dim must be 64 or 128"):
        cuda.flash_attention_forward(c, x, x, x, 1, 128, 3)


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("B,T,H", [(1, 128, 1), (2, 256, 2), (1, 200, 2), (1, 1024, 2), (2, 72, 3), (1, 4096, 1), (1, 2100, 2)])
def test_flash_backward_matches_oracle(B, T, H, hd):
    from heirloom_b200 import cuda
    c = ctx()
    C = hd * H
    rng = np.random.default_rng(B * 77 + T + H)
    qkv = ho.bf16_round(rng.standard_normal((B * T, 3 * C)))
    go = ho.bf16_round(rng.standard_normal((B * T, C)))
    fused = dev(qkv, torch.bfloat16)
    q, k, v = fused[:, :C], fused[:, C:2 * C], fused[:, 2 * C:]
    out, lse = cuda.flash_attention_forward(c, q, k, v, B, T, H)
    dqkv = cuda.flash_attention_backward(c, q, k, v, out, dev(go, torch.bfloat16), lse, B, T, H)
    got = host(dqkv)
    qn, kn, vn = (qkv[:, i * C:(i + 1) * C].reshape(B, T, C) for i in range(3))
    want = ho.causal_attention_backward(qn, kn, vn, H, go.reshape(B, T, C), bf16_operands=True)
    for i, name in enumerate(("dq", "dk", "dv")):
        w = want[i].reshape(B * T, C)
        g = got[:, i * C:(i + 1) * C]
        scale = np.abs(w).max()
        # bf16 operands on both sides; rounding of P/dS happens against slightly different f32
        # values, so compare at a few bf16 ulps of the tensor's scale
        assert_close("flash " + name, g, w, atol=scale * 2 ** -6, rtol=2 ** -5)
        assert np.abs(g - w).mean() <= scale * 2 ** -9


@pytest.mark.parametrize("B,T,H", [(1, 2, 1), (2, 63, 1), (1, 64, 2), (3, 65, 1), (1, 129, 3), (40, 192, 5)])
def test_flash_backward_at_the_edges_of_its_key_tiles(B, T, H):
    """Heads of 128 channels walk tiles of 64 keys against query tiles of 128: the last key tile absent, full or one row deep,
    and enough items that a CTA takes several.  (A single position's dQ and dK are exactly zero: nothing to scale a bound by.)"""
    test_flash_backward_matches_oracle(B, T, H, 128)


@pytest.mark.parametrize("B,T,H", [(90, 2, 1), (45, 64, 2), (30, 129, 2), (60, 200, 1), (24, 600, 2)])
def test_flash_backward_with_keys_as_rows(B, T, H):
    """Heads of 128 channels with enough walks for every SM take tiles of 128 keys: a tile almost empty, half full, a second one of one
    row, ragged, and several items a CTA with a ragged last tile."""
    test_flash_backward_matches_oracle(B, T, H, 128)


@pytest.mark.parametrize("B,T,H,hd", [(60, 192, 1, 128), (2, 192, 2, 128), (4, 72, 1, 128), (4, 192, 2, 64), (60, 100, 1, 64), (4, 40, 1, 64)])
def test_rows_of_the_next_batch_entry_stay_out_of_a_tile(B, T, H, hd):
    """Positions that are no multiple of a tile leave rows of the last tile empty: what the next entry holds there, infinities and NaN
    here, reaches none of this one's gradients (the first case takes keys as rows, the next two queries as rows)."""
    from heirloom_b200 import cuda
    c = ctx()
    C = H * hd
    gen = torch.Generator(device="cuda").manual_seed(9)
    qkv, go = (torch.randn(B * T, n * C, generator=gen, device="cuda").to(torch.bfloat16) for n in (3, 1))
    q, k, v = qkv.split(C, dim=1)
    torch.cuda.synchronize()
    out, lse = cuda.flash_attention_forward(c, q, k, v, B, T, H)
    c.sync()
    def run():
        torch.cuda.synchronize()
        return host(cuda.flash_attention_backward(c, q, k, v, out, go, lse, B, T, H)).reshape(B, T, -1)
    want = run()
    qkv.view(B, T, -1)[1::2, :T // 3] = float("nan")
    go.view(B, T, -1)[1::2, :T // 3] = float("inf")
    got = run()
    # the clean entries: the same products; dQ is summed by reductions in any order, in f32, and rounded to bf16
    assert np.isfinite(got[::2]).all()
    assert_close("clean entries", got[::2], want[::2], atol=np.abs(want).max() * 2 ** -8)


@pytest.mark.parametrize("B,T,H,hd", [(60, 192, 1, 128), (4, 72, 1, 128), (4, 192, 2, 64), (60, 100, 1, 64), (4, 40, 1, 64)])
def test_rows_of_the_next_batch_entry_stay_out_of_a_forward_tile(B, T, H, hd):
    """The same of the output and the rows' statistics, which are the same bits."""
    from heirloom_b200 import cuda
    c = ctx()
    C = H * hd
    qkv = torch.randn(B * T, 3 * C, generator=torch.Generator(device="cuda").manual_seed(9), device="cuda").to(torch.bfloat16)
    q, k, v = qkv.split(C, dim=1)
    def run():
        torch.cuda.synchronize()
        out, lse = cuda.flash_attention_forward(c, q, k, v, B, T, H)
        return host(out).reshape(B, T, -1), host(lse)
    want = run()
    qkv.view(B, T, -1)[1::2, :T // 3] = float("nan")
    got = run()
    assert all(np.array_equal(g[::2], w[::2]) for g, w in zip(got, want))
