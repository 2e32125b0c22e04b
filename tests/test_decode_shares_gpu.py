"""The persistent decode kernel's shares and pieces at their edges: ops with fewer units than warps, shares that touch several
tiles, CTAs with more tiles than warps, cache rows around a piece and a split, head widths that fill 4, 8 or 16 lanes."""
import numpy as np
import pytest

import vkllama_b200 as vk
from oracle import oracle as O
from util import LOGITS_MAX_ABS, load_from_oracle

pytestmark = pytest.mark.gpu


# weights; width, heads, feed-forward, vocabulary, cached rows before the calls
@pytest.mark.parametrize("f16", [False, True])
@pytest.mark.parametrize("dim,heads,ffn,vocab,pos", [
    (32, 2, 32, 20000, 3),     # one block per row: one unit per tile, empty shares
    (64, 8, 96, 61000, 20),    # heads of 8; 13 tiles of the output layer per CTA, two units each
    (96, 4, 416, 997, 33),     # heads of 24
    (128, 4, 256, 3001, 175),  # heads of 32, 16 rows per warp
    (320, 5, 864, 997, 180),   # heads of 64, a row more than a piece per warp
    (640, 5, 1696, 500, 383),  # heads of 128, the last row of one split, then two
    (160, 2, 416, 997, 30),    # heads of 80: half-filled lanes
    (480, 5, 1280, 997, 30),   # heads of 96
])
def test_one_token_calls_match_the_oracle(dev, f16, dim, heads, ffn, vocab, pos):
    cfg = dict(dim=dim, heads=heads, ffn=ffn, vocab=vocab, layers=2, maxlen=512)
    om = O.Model(seed=91, fp16=f16, **cfg)
    dm = vk.Model(dev, dim, heads, ffn, vocab, 2, 512, weight_dtype=vk.FP16 if f16 else vk.Q8_0)
    load_from_oracle(dm, om)
    text = O.synth_tokens(91, 1000, pos + 3, vocab)
    om.forward(text[:pos], 0)
    dm(text[:pos], 0)
    for i in range(pos, pos + 3):
        want, before = om.forward(text[i:i + 1], i), vk.kernel_launches()
        got = dm(text[i:i + 1], i)
        assert np.abs(got - want).max() <= LOGITS_MAX_ABS, i
        assert i == pos or vk.kernel_launches() - before == 1  # the persistent kernel (before its first launch the weights are packed)
    dm.close()


def test_fp16_decode_without_the_persistent_kernel(dev, monkeypatch):
    """The plan that a model falls back to where the device has no room for the decode kernel's copy of its weights."""
    cfg = dict(dim=256, heads=4, ffn=512, vocab=997, layers=2, maxlen=64)
    om = O.Model(seed=92, fp16=True, **cfg)
    text = O.synth_tokens(92, 1000, 12, 997)
    monkeypatch.setenv("VKLLAMA_DECODE", "graph")
    dm = vk.Model(dev, 256, 4, 512, 997, 2, 64, weight_dtype=vk.FP16)
    load_from_oracle(dm, om)
    om.forward(text[:9], 0)
    dm(text[:9], 0)
    for i in range(9, 12):
        before = vk.kernel_launches()
        assert np.abs(dm(text[i:i + 1], i) - om.forward(text[i:i + 1], i)).max() <= LOGITS_MAX_ABS, i
        assert vk.kernel_launches() - before > 5 * 2
    dm.close()
