"""The prompt's helpers (csrc/sal_decode_ops.cu) against torch: rotary step of many rows with the cache write, causal softmax in place
(rows of a multiple of eight scores and others, shorter and longer than a warp's stride, first rows that see one position, NaN and
infinities as torch.softmax treats them), and a prompt that takes several passes against one token at a time."""
import math

import pytest
import torch

from shiftaddllm_b200 import decode_ops
from shiftaddllm_b200.decoder import SHAPES, BcqLlamaDecoder, LlamaShape

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,kv_heads,hd,m,pos0", [(4, 4, 32, 1, 0), (4, 2, 64, 7, 3), (3, 1, 16, 70, 5), (8, 8, 128, 33, 30)])
def test_rope_rows(heads, kv_heads, hd, m, pos0):
    gen = torch.Generator(device="cuda").manual_seed(hd)
    q, k, v = (torch.randn(m, n * hd, device="cuda", generator=gen).half() for n in (heads, kv_heads, kv_heads))
    kc, vc = torch.zeros(pos0 + m + 2, kv_heads, hd, device="cuda").half(), torch.zeros(pos0 + m + 2, kv_heads, hd, device="cuda").half()
    ang = torch.arange(pos0 + m + 2, device="cuda").float()[:, None] / 10000 ** (torch.arange(0, hd, 2, device="cuda").float() / hd)
    cos, sin = ang.cos(), ang.sin()

    def rope(t, n):
        a, b = t.view(m, n, 2, hd // 2).float().unbind(2)
        c, s = cos[pos0:pos0 + m, None], sin[pos0:pos0 + m, None]
        return torch.cat((a * c - b * s, b * c + a * s), -1)

    want_q, want_k = rope(q, heads), rope(k, kv_heads)
    assert decode_ops.rope_rows(q, k, v, cos, sin, pos0, kc, vc, heads, kv_heads, hd)
    # one fp16 rounding of a value formed in fp32 from two products: 2**-11 of it, and 2**-22 of the products
    for got, want in ((q.view(m, heads, hd), want_q), (kc[pos0:pos0 + m], want_k)):
        assert ((got.float() - want).abs() <= 2.0 ** -11 * want.abs() + 2.0 ** -19).all()
    assert torch.equal(vc[pos0:pos0 + m], v.view(m, kv_heads, hd))
    assert not kc[:pos0].any() and not kc[pos0 + m:].any() and not vc[pos0 + m:].any()
    assert not decode_ops.rope_rows(q, k, v, cos, sin, 3, kc, vc, heads, kv_heads, hd + 8)      # not a multiple of 16: refused, nothing done


@pytest.mark.parametrize("m,total", [(1, 1), (5, 5), (8, 40), (33, 261), (64, 1024), (3, 7)])
def test_causal_softmax(m, total):
    gen = torch.Generator(device="cuda").manual_seed(m)
    scores, first, scale = (6 * torch.randn(3, m, total, device="cuda", generator=gen)).half(), total - m, 1 / math.sqrt(8)
    scores[0, 0, 0] = 65504
    scores[2, m - 1, :] = float("-inf")
    if total > 4:
        scores[1, m - 1, 2] = float("nan")
        if first > 0:   # a row of nothing but -inf is NaN; torch then fills the hidden places with it as well
            scores[1, 0, 0] = float("-inf")
    hidden = torch.arange(total, device="cuda")[None] > first + torch.arange(m, device="cuda")[:, None]
    want = torch.softmax((scores.float() * scale).masked_fill(hidden, float("-inf")), -1)
    decode_ops.causal_softmax(scores, first, scale)
    # fp16 rounding of a probability, and of exponentials whose arguments carry a relative 2**-22 of up to 46
    assert torch.allclose(scores.float(), want, rtol=2.0 ** -10, atol=2.0 ** -24, equal_nan=True)


@pytest.mark.parametrize("chunk", [64, 16])
def test_prompt_of_several_passes(chunk, monkeypatch):
    monkeypatch.setattr(BcqLlamaDecoder, "PREFILL_ROWS", 70)   # 150 tokens: passes of 70, 70 and 10
    model = BcqLlamaDecoder(SHAPES["tiny"], 3, 128, max_len=160)
    ids = torch.randint(0, 1000, (150,), generator=torch.Generator().manual_seed(1)).tolist()
    model.reset()
    model.feed(ids, chunk=1)
    want = [t.float().clone() for t in (model.logits, model.k_cache, model.v_cache)]
    model.reset()
    model.prefill(ids, chunk)
    assert int(model.pos) == 150
    # a token and a prompt round activations to fp16 at the same places but sum in another order: 2**-11 per layer and product, over the
    # two layers' chain of eight roundings with headroom for the logits' sum over the hidden size
    for got, ref in zip((model.logits, model.k_cache, model.v_cache), want):
        assert (got.float() - ref).norm() <= 8 * 2.0 ** -9 * ref.norm()


@pytest.mark.parametrize("chunk,passes", [(64, [64, 64, 22]), (63, [63, 63, 24]), (100, [100, 50]), (None, [70, 70, 10]), (1000, [150])])
def test_chunk_is_the_bound_on_the_rows_of_a_pass(chunk, passes, monkeypatch):
    from shiftaddllm_b200 import decoder

    rows, group = [], decoder._group
    monkeypatch.setattr(BcqLlamaDecoder, "PREFILL_ROWS", 70)
    monkeypatch.setattr(decoder, "_group", lambda lins, x, *a, **k: (rows.append(x.shape[0]), group(lins, x, *a, **k))[1])
    model = BcqLlamaDecoder(SHAPES["tiny"], 3, 128, max_len=160)
    model.feed(list(range(150)), **({} if chunk is None else {"chunk": chunk}))
    assert rows[::4 * SHAPES["tiny"].layers] == passes and len(rows) == 4 * SHAPES["tiny"].layers * len(passes)


def test_prompt_through_a_model_without_blocks():
    """Embedding, final norm and head alone: nothing is added that no block has written."""
    shape = LlamaShape(256, 0, 2, 2, 512, vocab=1000)
    model = BcqLlamaDecoder(shape, 3, 128, max_len=16)
    torch.full((1 << 20,), float("nan"), dtype=torch.float16, device="cuda")   # what freed memory then holds
    model.feed([1, 2, 3])
    want = torch.nn.functional.rms_norm(model.embed[3], (256,), model.final_norm, shape.eps) @ model.lm_head.t()
    assert (model.logits - want.float()).norm() <= 2.0 ** -9 * want.float().norm()
