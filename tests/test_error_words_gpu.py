"""What the host does with the word that a kernel raises when one of its bounded waits has run out. The word is set from the
host (tests/cpp/error_word.cu reaches it), or the decode kernel's bound made so short that healthy waits run out."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

import vkllama_b200 as vk
from oracle import oracle as O
from util import LOGITS_MAX_ABS, load_from_oracle
from vkllama_b200 import build as B

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def words(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("words") / "error_word.so")
    subprocess.check_call([B.NVCC] + B.FLAGS + ["-shared", "-I", B.CSRC, os.path.join(ROOT, "tests", "cpp", "error_word.cu"), "-o", so])
    L = C.CDLL(so)
    for f in (L.raise_model_word, L.command_is_watched, L.raise_command_word, L.decode_word):
        f.argtypes = [C.c_void_p]
    L.decode_word.restype = C.c_uint32
    L.set_polls.argtypes = L.shift_v_cache.argtypes = [C.c_void_p, C.c_uint32]
    return L


def test_model_calls_report_their_own_waits(dev, words):
    """Rows of a block whose projections gave up are not handed out as a success, and the next call is not blamed; calls whose
    kernels have no waits do not ask."""
    dm = vk.Model(dev, 512, 8, 1600, 100, 2, 64)
    dm.synth_weights(71)
    x = O.synth_f16(71, 5, 40 * 512).reshape(40, 512)  # gate and up of 33 rows and more, 1.6 million weights: a kernel with bounded waits
    want = dm.block_forward(0, x, 0)
    assert words.raise_model_word(dm.h) == 0
    with pytest.raises(vk.VklError) as e:
        dm.block_forward(0, x, 0)
    assert e.value.code == 13
    assert (dm.block_forward(0, x, 0) == want).all()
    words.raise_model_word(dm.h)
    for T in (1, 8, 12, 32):  # no such kernel runs: the word is not asked for
        dm(np.arange(T, dtype=np.uint32), 0)
    with pytest.raises(vk.VklError) as e:
        dm(np.arange(33, dtype=np.uint32), 0)
    assert e.value.code == 13
    dm(np.arange(33, dtype=np.uint32), 0)
    dm.close()


def test_a_decode_wait_that_ran_out_on_any_sm_is_reported(dev, words):
    """CTA 0 has the only tile of the output layer (148 tiles lie before it), so the others wait for it at the end, and it for nobody.
    With a bound of a few dozen polls some of them give up there while it ends the launch. A call that succeeds leaves no word
    behind for a later call."""
    dm = vk.Model(dev, 256, 4, 544, 32, 2, 64)
    dm.synth_weights(73)
    tok = np.array([7], np.uint32)
    dm(tok, 0)
    want = dm(tok, 1)
    failed = 0
    for polls in list(range(20, 84)) * 3:
        words.set_polls(dm.h, polls)
        try:
            assert (dm(tok, 1) == want).all(), polls
        except vk.VklError as e:
            assert e.code == 13 and "bounded wait ran out" in e.message
            failed += 1
        assert words.decode_word(dm.h) == 0, polls
    assert failed
    dm.set_wait_limit(0)
    assert (dm(tok, 1) == want).all()
    dm.close()


def test_caches_that_the_decode_kernel_cannot_address_are_left_to_the_graph(dev, words):
    """It names the V cache by its distance from the K cache, in 256 bytes."""
    cfg = dict(dim=256, heads=4, ffn=512, vocab=1000, layers=2, maxlen=64)
    om = O.Model(seed=74, **cfg)
    dm = vk.Model(dev, 256, 4, 512, 1000, 2, 64)
    load_from_oracle(dm, om)
    assert words.shift_v_cache(dm.h, 1) == 0
    text = O.synth_tokens(74, 1000, 4, 1000)
    for i in range(4):
        before = vk.kernel_launches()
        assert np.abs(dm(text[i:i + 1], i) - om.forward(text[i:i + 1], i)).max() <= LOGITS_MAX_ABS, i
        assert vk.kernel_launches() - before > 10
    dm.close()


# Kernels with bounded waits: the few-row kernel (more than 8 rows, whole 32-column blocks, 5 million weights, 1.6 million from 33
# rows on; for 9 to 16 rows of Q8_0 at most 370 row tiles of 16 on 148 SMs), and the tensor-core GEMM.
@pytest.mark.parametrize("wt,M,N,K,watched", [("q8_0", 1, 1300, 3936, False), ("q8_0", 8, 1300, 3936, False), ("q8_0", 20, 1300, 3928, False), ("q8_0", 12, 6000, 864, False),
                                              ("q8_0", 20, 1300, 3808, False), ("q8_0", 9, 1300, 3936, True), ("q8_0", 17, 1300, 3936, True), ("q8_0", 33, 417, 3936, True),
                                              ("q8_0", 77, 417, 3936, True), ("f16", 12, 12000, 480, True), ("q8_0", 64, 64, 64, True)])
def test_a_command_asks_for_the_word_only_where_a_kernel_has_waits(dev, words, wt, M, N, K, watched):
    dt = vk.Q8_0 if wt == "q8_0" else vk.FP16
    w = O.synth_q8_0(72, 1, N, K, 0.0, 0.05) if wt == "q8_0" else O.synth_f16(72, 1, N * K, 0.0, 0.05)
    cmd = vk.Command(dev)
    cmd.begin()
    tw, tx = vk.Tensor(1, N, K, dev, dt), vk.Tensor(1, M, K, dev, vk.FP16)
    cmd.upload(w, tw)
    cmd.upload(O.synth_f16(72, 2, M * K), tx)
    op = vk.MatMul(dev, cmd, tw, 1.0, 0.0, 0, 0, True, vk.FP16, dt).init()
    want = cmd.download(op(tx))
    assert bool(words.command_is_watched(cmd.h)) == watched
    cmd.end()
    cmd.submit_and_wait()
    assert not words.command_is_watched(cmd.h)
    if not watched:
        return
    cmd.begin()
    op(tx)
    cmd.end()
    assert words.raise_command_word(cmd.h) == 0
    with pytest.raises(vk.VklError) as e:
        cmd.submit_and_wait()
    assert e.value.code == 13 and "code 1" in e.value.message
    cmd.begin()
    got = cmd.download(op(tx))
    cmd.end()
    cmd.submit_and_wait()
    assert (got == want).all()
