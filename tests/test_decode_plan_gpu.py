"""Which plan a one-token call takes, and what it does where the persistent decode kernel's tables cannot be built or
the device has little memory left for the second copy of the weights."""
import numpy as np
import pytest
import torch

import vkllama_b200 as vk
from oracle import oracle as O
from test_model_gpu import fill
from util import LOGITS_MAX_ABS, load_from_oracle

pytestmark = pytest.mark.gpu


def launches(call):
    before = vk.kernel_launches()
    out = call()
    return out, vk.kernel_launches() - before


def model(dev, dims, f16, seed):
    dm = vk.Model(dev, *dims, weight_dtype=vk.FP16 if f16 else vk.Q8_0)
    dm.synth_weights(seed)
    return dm


def test_tables_that_could_not_be_built_are_not_taken_for_built(dev):
    """The decode kernel's copy of the weights gets its 128 MiB, the small buffer after it gets nothing: the call fails. Once there
    is room, a call of more rows has the tables built again, and the copy must be filled then."""
    dims = (4096, 32, 4096, 500, 1, 64)
    prompt, tok = O.synth_tokens(51, 1000, 20, 500), np.array([7], np.uint32)
    room = vk.Tensor(1, 4, 1 << 23, dev, vk.FP32)
    roomy = model(dev, dims, False, 51)
    roomy(prompt, 0)
    want = roomy(tok, 20)
    roomy.close()
    dm = model(dev, dims, False, 51)
    dm(prompt[:8], 0)
    filler = fill(dev, 8)
    try:
        with pytest.raises(vk.VklError):
            while True:
                filler.append(vk.Tensor(1, 1, 24 << 10, dev, vk.FP32))  # as large as the small buffer
        del room  # the pool keeps it, for a request of its size
        with pytest.raises(vk.VklError) as e:
            dm(tok, 8)
        assert e.value.code == 8
    finally:
        del filler
    dm(prompt, 0)
    got, n = launches(lambda: dm(tok, 20))
    assert (got == want).all() and n == 6  # five streams packed, one launch for the token
    dm.close()


@pytest.mark.parametrize("f16", [False, True])
def test_separate_merge_leaves_out_splits_of_a_longer_sequence(dev, monkeypatch, f16):
    """Four splits per head, then a shorter sequence with two: the merge must not add what the first sequence left in the others."""
    monkeypatch.setenv("VKLLAMA_DECODE_COMBINE", "separate")
    monkeypatch.setenv("VKLLAMA_SPLIT_ROWS", "32")
    cfg = dict(dim=256, heads=4, ffn=512, vocab=997, layers=2, maxlen=256)
    om = O.Model(seed=52, fp16=f16, **cfg)
    dm = vk.Model(dev, 256, 4, 512, 997, 2, 256, weight_dtype=vk.FP16 if f16 else vk.Q8_0)
    load_from_oracle(dm, om)
    for seed, n in ((52, 120), (53, 50)):
        text = O.synth_tokens(seed, 1000, n + 2, 997)
        om.forward(text[:n], 0)
        dm(text[:n], 0)
        for i in (n, n + 1):
            assert np.abs(dm(text[i:i + 1], i) - om.forward(text[i:i + 1], i)).max() <= LOGITS_MAX_ABS, (n, i)
    dm.close()


@pytest.mark.parametrize("f16", [False, True])
def test_output_layers_beyond_a_grid_dimension(dev, monkeypatch, f16):
    """A vocabulary of more than 65535 tiles of 32 rows."""
    dims = (64, 2, 64, 2097300, 1, 64)
    tok = np.array([2097299], np.uint32)
    monkeypatch.setenv("VKLLAMA_DECODE", "graph")
    graph = model(dev, dims, f16, 54)
    want = graph(tok, 0)
    graph.close()
    monkeypatch.delenv("VKLLAMA_DECODE")
    dm = model(dev, dims, f16, 54)
    dm(tok, 0)
    got, n = launches(lambda: dm(tok, 0))
    assert n == 1 and np.abs(got - want).max() <= LOGITS_MAX_ABS
    dm.close()


F16_DIMS = (4096, 32, 4096, 500, 1, 4096)  # the decode kernel's copy of these weights takes 256 MiB


def test_fp16_copy_where_memory_is_short_and_where_the_pool_has_it(dev):
    """No copy where less than twice its size is free (the graph then reads the weights as they are); blocks that the library's own
    pool holds count as free."""
    tok = np.array([7], np.uint32)
    dm = model(dev, F16_DIMS, True, 55)
    one = dm(tok, 0)
    want, n = launches(lambda: dm(tok, 1))
    assert n == 1
    dm.close()
    dm = model(dev, F16_DIMS, True, 55)
    filler = fill(dev, 300)
    try:
        assert np.abs(dm(tok, 0) - one).max() <= LOGITS_MAX_ABS
        got, n = launches(lambda: dm(tok, 1))
    finally:
        del filler
    assert n > 5 and np.abs(got - want).max() <= LOGITS_MAX_ABS
    dm.close()
    dm = model(dev, F16_DIMS, True, 55)
    pooled = vk.Tensor(1, 16, 1 << 23, dev, vk.FP32)
    filler = fill(dev, 60)
    try:
        del pooled
        dm(tok, 0)
        got, n = launches(lambda: dm(tok, 1))
    finally:
        del filler
    assert n == 1 and (got == want).all()
    dm.close()


def test_fp16_copy_makes_way_for_the_rows_of_a_call(dev):
    prompt, tok = O.synth_tokens(56, 1000, 4000, 500), np.array([7], np.uint32)
    dm = model(dev, F16_DIMS, True, 56)
    want = dm(prompt, 0)
    one = dm(tok, 4000)
    dm.close()
    dm = model(dev, F16_DIMS, True, 56)
    dm(prompt[:20], 0)
    dm(tok, 20)
    assert launches(lambda: dm(tok, 21))[1] == 1
    filler = fill(dev, 64)  # the rows need 230 MiB
    try:
        assert (dm(prompt, 0) == want).all()
        got, n = launches(lambda: dm(tok, 4000))
    finally:
        del filler
    assert n > 5 and np.abs(got - one).max() <= LOGITS_MAX_ABS
    dm.close()


def test_a_single_generated_id_has_no_use_for_the_copy(dev):
    dm = model(dev, F16_DIMS, True, 57)
    prompt = O.synth_tokens(57, 1000, 20, 500)
    dm(prompt, 0)
    fill(dev, 1 << 20)  # (empties the pool, fills nothing)
    free = [torch.cuda.mem_get_info()[0]]
    for n in (1, 2):
        dm.generate(prompt, n)
        free.append(torch.cuda.mem_get_info()[0])
    assert free[0] - free[1] < 64 << 20 < 200 << 20 < free[1] - free[2]
    dm.close()
