"""Block- and model-level parity of the CUDA token loop against the CPU oracle:
one Llama-2-7B-shaped block at position 511, a small model end to end (logits
and greedy ids through prefill + decode), and the full 7B greedy ids against
the committed oracle fixture (tests/golden/make_golden_7b.py)."""
import os

import numpy as np
import pytest
import torch

from oracle import decoder as D
from oracle import oracle as O
import kupuzen_util as U
import vkllama_b200 as vk
from util import LOGITS_MAX_ABS, assert_close, decided_prompt, load_from_oracle

pytestmark = pytest.mark.gpu

SMALL = dict(dim=256, heads=4, ffn=512, vocab=1000, layers=3, maxlen=128)


def small_pair(dev, seed=5, **over):
    cfg = dict(SMALL, **over)
    om = O.Model(seed=seed, **cfg)
    dm = vk.Model(dev, cfg["dim"], cfg["heads"], cfg["ffn"], cfg["vocab"], cfg["layers"], cfg["maxlen"])
    load_from_oracle(dm, om)
    return om, dm, cfg


def fp16_pair(dev, seed, **over):
    cfg = dict(SMALL, **over)
    om = O.Model(seed=seed, fp16=True, **cfg)
    dm = vk.Model(dev, cfg["dim"], cfg["heads"], cfg["ffn"], cfg["vocab"], cfg["layers"], cfg["maxlen"], weight_dtype=vk.FP16)
    load_from_oracle(dm, om)
    return om, dm, cfg


@pytest.mark.parametrize("P", [7, 48, 100, 128])
def test_fp16_weights_model_prefill_then_decode(dev, P):
    """FP16-weights model: prompts of 32 tokens and more prefill through the tcgen05 tensor-core
    GEMM, shorter ones and the decode steps through the weight-streaming kernels."""
    om, dm, cfg = fp16_pair(dev, seed=11)
    prompt = O.synth_tokens(11, 1000 + P, P, cfg["vocab"])
    want = om.forward(prompt, 0)
    got = dm(prompt, 0)
    assert np.abs(got - want).max() <= LOGITS_MAX_ABS
    tok = np.array([int(np.argmax(want))], np.uint32)
    for i in range(3):
        want = om.forward(tok, P + i)
        got = dm(tok, P + i)
        assert np.abs(got - want).max() <= LOGITS_MAX_ABS, "decode step %d" % i
        tok = np.array([int(np.argmax(want))], np.uint32)
    for l in range(cfg["layers"]):
        gk, gv = dm.read_kv(l)
        n = min(P + 3, cfg["maxlen"])
        assert_close(gk[:, :n], om.kcache(l)[:, :n], tol=5e-3, what="kcache layer %d" % l)
        assert_close(gv[:, :n], om.vcache(l)[:, :n], tol=5e-3, what="vcache layer %d" % l)


def test_fp16_weights_greedy_generate(dev):
    om, dm, cfg = fp16_pair(dev, seed=12)
    prompt, want = decided_prompt(lambda: O.Model(seed=12, fp16=True, **cfg), 12, 40, 16, cfg["vocab"])
    got = dm.generate(prompt, 16)[0]
    assert got.tolist() == want.tolist()


def test_block_7b_shape_decode_at_position_511(dev):
    """One decoder block with Llama-2-7B shapes, one decode step at position 511,
    fp16 KV cache prefilled with N(0,1) for 511 positions."""
    cfg = dict(dim=4096, heads=32, ffn=11008, vocab=64, layers=1, maxlen=512)
    om = O.Model(seed=20240602, **cfg)
    dm = vk.Model(dev, cfg["dim"], cfg["heads"], cfg["ffn"], cfg["vocab"], cfg["layers"], cfg["maxlen"])
    load_from_oracle(dm, om)
    k0 = O.synth_f16(20240602, 900, 32 * 512 * 128).reshape(32, 512, 128)
    v0 = O.synth_f16(20240602, 901, 32 * 512 * 128).reshape(32, 512, 128)
    om.kcache(0)[:] = k0
    om.vcache(0)[:] = v0
    dm.write_kv(0, k0, v0)
    x = O.synth_f16(20240602, 902, 4096).reshape(1, 4096)
    want = om.block(0, x, 1, 511)
    got = dm.block_forward(0, x, 511)
    assert_close(got, want, what="7B block @511")
    gk, gv = dm.read_kv(0)
    assert_close(gk[:, 511], om.kcache(0)[:, 511], tol=2e-3, what="appended k")
    assert_close(gv[:, 511], om.vcache(0)[:, 511], tol=2e-3, what="appended v")
    assert np.array_equal(gk[:, :511], k0[:, :511])


@pytest.mark.parametrize("T,offset", [(1, 0), (9, 0), (64, 0), (70, 0)])
def test_block_multi_token(dev, T, offset):
    om, dm, cfg = small_pair(dev, seed=6)
    x = O.synth_f16(6, 700 + T, T * cfg["dim"]).reshape(T, cfg["dim"])
    want = om.block(1, x, T, offset)
    got = dm.block_forward(1, x, offset)
    assert_close(got, want, what="block T=%d" % T)


def test_small_model_logits_prefill_then_decode(dev):
    om, dm, cfg = small_pair(dev, seed=7)
    prompt = O.synth_tokens(7, 1000, 12, cfg["vocab"])
    want = om.forward(prompt, 0)
    got = dm(prompt, 0)
    assert np.abs(got - want).max() <= LOGITS_MAX_ABS
    tok = np.array([int(np.argmax(want))], np.uint32)
    for i in range(5):
        want = om.forward(tok, 12 + i)
        got = dm(tok, 12 + i)
        assert np.abs(got - want).max() <= LOGITS_MAX_ABS, "decode step %d" % i
        tok = np.array([int(np.argmax(want))], np.uint32)
    for l in range(cfg["layers"]):
        gk, gv = dm.read_kv(l)
        assert_close(gk[:, :17], om.kcache(l)[:, :17], tol=5e-3, what="kcache layer %d" % l)
        assert_close(gv[:, :17], om.vcache(l)[:, :17], tol=5e-3, what="vcache layer %d" % l)


@pytest.mark.parametrize("weights", ["q8_0", "fp16"])
@pytest.mark.parametrize("P", [24, 47, 57])
def test_few_row_projections_in_a_block(dev, weights, P):
    """9 to 64 rows through a whole model that is wide enough for the few-row kernel (1.6 million weights in the smallest
    projection, 5 below 33 rows): three matrices, gate and up, and both projections that add to the stream. FP16: widths that the
    tensor-core GEMM does not take."""
    dims = dict(dim=2336, heads=73) if weights == "fp16" else dict(dim=2304, heads=18)
    om, dm, cfg = (fp16_pair if weights == "fp16" else small_pair)(dev, seed=24, ffn=2400, vocab=100, layers=2, maxlen=64, **dims)
    prompt = O.synth_tokens(24, 1000 + P, P, cfg["vocab"])
    assert np.abs(dm(prompt, 0) - om.forward(prompt, 0)).max() <= LOGITS_MAX_ABS
    for l in range(2):  # the second block's keys and values hold what the first one's projections added
        gk, gv = dm.read_kv(l)
        assert_close(gk[:, :P], om.kcache(l)[:, :P], tol=5e-3, what="kcache layer %d" % l)
        assert_close(gv[:, :P], om.vcache(l)[:, :P], tol=5e-3, what="vcache layer %d" % l)


@pytest.mark.parametrize("P", [128, 129, 300])
def test_q8_0_prompts_around_the_widened_weights_limit(dev, P):
    """129 tokens and more: the GEMMs' weights are turned into fp16 first. Row tiles of a matrix that end inside a 128-row half
    tile, blocks that end inside a group of four."""
    cfg = dict(dim=192, heads=3, ffn=320, vocab=500, layers=2, maxlen=320)
    om = O.Model(seed=21, **cfg)
    dm = vk.Model(dev, cfg["dim"], cfg["heads"], cfg["ffn"], cfg["vocab"], cfg["layers"], cfg["maxlen"])
    dm.synth_weights(21)
    prompt = O.synth_tokens(21, 1000 + P, P, cfg["vocab"])
    assert np.abs(dm(prompt, 0) - om.forward(prompt, 0)).max() <= LOGITS_MAX_ABS
    for l in range(cfg["layers"]):
        gk, gv = dm.read_kv(l)
        assert_close(gk[:, :P], om.kcache(l)[:, :P], tol=5e-3, what="kcache layer %d" % l)
        assert_close(gv[:, :P], om.vcache(l)[:, :P], tol=5e-3, what="vcache layer %d" % l)


def fill(dev, mib_left):
    """Tensors that leave less than mib_left + 4 MiB of the device's memory free, outside the pool too."""
    with pytest.raises(vk.VklError):
        vk.Tensor(1, 1 << 20, 1 << 18, dev, vk.FP32)  # 1 TiB: refused, after the pool's free blocks went back to the driver
    filler = []
    for mib in (4096, 512, 64, 16, 4):
        while torch.cuda.mem_get_info()[0] - (mib << 20) > mib_left << 20:
            filler.append(vk.Tensor(1, mib, 1 << 18, dev, vk.FP32))
    return filler


def test_q8_0_prompts_without_room_for_the_widened_weights(dev):
    """The fp16 copy of the weights (256 MiB here) is for speed: on a device that is full up to 160 MiB the prompt runs in the
    dequantising tiles, which write the same fp16 values. fp32 sums in another order: the logits differ by fp16 rounding."""
    dims = (4096, 32, 16384, 500, 1, 256)
    prompt = O.synth_tokens(22, 1000, 140, 500)
    roomy = vk.Model(dev, *dims)
    roomy.synth_weights(22)
    want = roomy(prompt, 0)
    roomy.close()
    dm = vk.Model(dev, *dims)
    dm.synth_weights(22)
    dm(prompt[:70], 0)  # everything that a prompt launches is loaded
    filler = fill(dev, 160)
    try:
        got = dm(prompt, 0)
    finally:
        del filler
    assert np.abs(got - want).max() <= LOGITS_MAX_ABS
    dm.close()


@pytest.mark.parametrize("design", ["llama", "layer list"])
def test_a_call_without_memory_for_its_rows_leaves_the_model_usable(dev, design):
    """Growing the activations fails half way; shorter calls after it must not meet the buffers that are missing."""
    if design == "llama":
        dm = vk.Model(dev, 4096, 32, 16384, 500, 1, 4096)
        dm.synth_weights(23)
    else:
        case = U.config([(U.attn(2, 1, 32, 32, 400, 8), 4096)], width=1088, vocab=500)
        W = U.weights(case, 23)
        dm = vk.Model.from_config(dev, case[0], 4096, vk.BF16, shapes=U.shapes(W))
        for k, v in W.items():
            dm.set_weight(k, vk.BF16, D.f32_to_bf16(v.reshape(-1)))
    prompt = O.synth_tokens(23, 1000, 4000, 500)
    want, one = dm(prompt[:20], 0), dm(prompt[20:21], 20)
    filler = fill(dev, 8)
    try:
        with pytest.raises(vk.VklError) as e:
            dm(prompt, 0)
        assert e.value.code == 8
    finally:
        del filler
    assert (dm(prompt[:20], 0) == want).all()
    assert (dm(prompt[20:21], 20) == one).all()
    dm.close()


@pytest.mark.parametrize("seed,P,n_gen", [(8, 9, 40), (9, 1, 20), (10, 33, 64)])
def test_small_model_greedy_ids_match_oracle(dev, seed, P, n_gen):
    om, dm, cfg = small_pair(dev, seed=seed)
    prompt = O.synth_tokens(seed, 1000, P, cfg["vocab"])
    want, gap = om.generate(prompt, n_gen)
    got, pre_ms, dec_ms = dm.generate(prompt, n_gen)
    bad = np.nonzero(got != want)[0]
    assert bad.size == 0, "first mismatch at step %d (oracle top-2 gap there %.4f)" % (bad[0], gap[bad[0]])
    # the generate loop and the host-driven loop (Model::operator() per token) agree
    logits = dm(prompt, 0)
    assert int(np.argmax(logits)) == int(got[0])


def test_generate_matches_host_driven_loop(dev):
    om, dm, cfg = small_pair(dev, seed=11)
    prompt = O.synth_tokens(11, 1000, 7, cfg["vocab"])
    ids, _, _ = dm.generate(prompt, 12)
    logits = dm(prompt, 0)
    tok = int(np.argmax(logits))
    host = [tok]
    for i in range(1, 12):
        logits = dm(np.array([tok], np.uint32), 7 + i - 1)
        tok = int(np.argmax(logits))
        host.append(tok)
    assert host == ids.tolist()


def test_device_synth_weights_equal_uploaded_oracle_weights(dev):
    om, dm, cfg = small_pair(dev, seed=12)
    dm2 = vk.Model(dev, cfg["dim"], cfg["heads"], cfg["ffn"], cfg["vocab"], cfg["layers"], cfg["maxlen"])
    dm2.synth_weights(12)
    prompt = O.synth_tokens(12, 1000, 10, cfg["vocab"])
    a = dm(prompt, 0)
    b = dm2(prompt, 0)
    assert np.array_equal(a, b)


def test_model_errors(dev):
    dm = vk.Model(dev, 256, 4, 512, 1000, 1, 32)
    with pytest.raises(vk.VklError) as e:  # weights not set
        dm(np.array([1], np.uint32), 0)
    assert e.value.code == 9
    with pytest.raises(vk.VklError) as e:
        dm.set_weight("blk.7.attn_q.weight", vk.Q8_0, np.zeros(34, np.uint8))
    assert e.value.code == 3
    with pytest.raises(vk.VklError) as e:  # wrong byte count
        dm.set_weight("blk.0.attn_q.weight", vk.Q8_0, np.zeros(34, np.uint8))
    assert e.value.code == 3
    dm.synth_weights(1)
    with pytest.raises(vk.VklError) as e:  # beyond the context length
        dm(np.zeros(33, np.uint32), 0)
    assert e.value.code == 11


UNDECIDED_ULPS = 4.0
GOLD7B = os.path.join(os.path.dirname(__file__), "golden", "llama2_7b_q8_0_greedy.npz")


@pytest.fixture(scope="module", params=["persistent", "graph"])
def model7b(dev, request):
    """The full 7B shape under both decode plans: the persistent kernel (default) and the CUDA graph
    of five kernels per layer."""
    if not os.path.exists(GOLD7B):
        pytest.skip("7B oracle fixture not generated")
    g = np.load(GOLD7B)
    old = os.environ.get("VKLLAMA_DECODE")
    if request.param == "graph":
        os.environ["VKLLAMA_DECODE"] = "graph"
    try:
        dm = vk.Model(dev, 4096, 32, 11008, 32000, 32, 4096)
        dm.synth_weights(int(g["seed"]))
        dm(np.array([1], np.uint32), 0)  # the decode plan is chosen at the first one-token step
    finally:
        if old is None:
            os.environ.pop("VKLLAMA_DECODE", None)
        else:
            os.environ["VKLLAMA_DECODE"] = old
    yield g, dm
    dm.close()


def test_llama2_7b_q8_0_greedy_ids_match_oracle_fixture(model7b):
    """Full Llama-2-7B shape, Q8_0, 32-token prompt, 64 free-running greedy tokens: every id equals
    the CPU oracle's, under both decode plans. The prompt was screened on the device
    (tests/golden/screen_prompts_gpu.py) and confirmed by the oracle (tests/golden/make_golden_7b.py):
    the oracle decides each of its 64 steps by at least 4 fp16 ulps, more than the 1-2 ulps by which
    implementations with different fp32 summation orders differ in the final logits."""
    g, dm = model7b
    assert float(g["sel_gap_ulps"].min()) >= UNDECIDED_ULPS
    prompt = g["sel_prompt"]
    logits = dm(prompt, 0)
    assert np.abs(logits - g["sel_prefill_logits"]).max() <= LOGITS_MAX_ABS
    n = len(g["sel_ids"])
    assert n >= 64
    got, pre_ms, dec_ms = dm.generate(prompt, n)
    bad = np.nonzero(got != g["sel_ids"])[0]
    assert bad.size == 0, "first mismatch at step %d where the oracle top-2 gap is %.1f ulps" % (bad[0], g["sel_gap_ulps"][bad[0]])
    # the host-driven loop (Model::operator() per token, host arg-max) gives the same ids
    tok, host = int(np.argmax(logits)), []
    for i in range(16):
        host.append(tok)
        tok = int(np.argmax(dm(np.array([tok], np.uint32), len(prompt) + i)))
    assert host == g["sel_ids"][:16].tolist()


def test_llama2_7b_q8_0_teacher_forced_steps(model7b):
    """Unselected base prompt, teacher-forced with the oracle's ids: every step whose
    oracle top-2 gap is at least 4 fp16 ulps must pick the oracle's id."""
    g, dm = model7b
    prompt, ids = g["base_prompt"], g["base_ids"]
    logits = dm(prompt, 0)
    assert np.abs(logits - g["base_prefill_logits"]).max() <= LOGITS_MAX_ABS
    picks = [int(np.argmax(logits))]
    for i in range(1, len(ids)):
        logits = dm(np.array([ids[i - 1]], np.uint32), len(prompt) + i - 1)
        picks.append(int(np.argmax(logits)))
    picks = np.array(picks)
    decided = g["base_gap_ulps"] >= UNDECIDED_ULPS
    assert np.array_equal(picks[decided], ids[decided])
    assert decided.sum() >= 50 and (picks == ids).mean() >= 0.9


@pytest.mark.parametrize("switch", [("VKLLAMA_DECODE", "graph"), ("VKLLAMA_DECODE_COMBINE", "separate"), ("VKLLAMA_SPLIT_ROWS", "0"),
                                    ("VKLLAMA_SPLIT_ROWS", "16"), ("VKLLAMA_PREFILL", "sequential")])
def test_decode_plan_switches_keep_parity(dev, monkeypatch, switch):
    """The alternative decode plans (multi-kernel CUDA graph, combine op after a grid barrier, all
    attention splits at every length or one split per 16 cached rows, token-by-token prefill through
    the decode kernel) give the same logits and greedy ids as the default plan, against the oracle."""
    monkeypatch.setenv(*switch)
    om, dm, cfg = small_pair(dev, seed=13)
    prompt, want = decided_prompt(lambda: O.Model(seed=13, **cfg), 13, 9, 24, cfg["vocab"])
    got = dm.generate(prompt, 24)[0]
    assert got.tolist() == want.tolist(), switch
    om2, dm2, _ = small_pair(dev, seed=13)
    tok = np.array([int(prompt[0])], np.uint32)
    for i in range(4):  # one-token calls: the decode plan under test
        w = om2.forward(tok, i)
        g = dm2(tok, i)
        assert np.abs(g - w).max() <= LOGITS_MAX_ABS, (switch, i)
        tok = np.array([int(np.argmax(w))], np.uint32)


# ---- callers either side of the token loop: checkpoint loading, samplers, chat-style sessions ----
@pytest.mark.parametrize("f16", [False, True])
def test_model_from_gguf_equals_model_from_set_weight(dev, tmp_path, f16):
    """Model::init from a GGUF file (models/llama2.h:348-681): the same logits, bit for bit, as
    the model whose tensors were handed over one by one."""
    from test_gguf_samplers_cpu import write_gguf
    cfg = dict(dim=256, heads=4, ffn=512, vocab=1000, layers=2, maxlen=128)
    om = O.Model(seed=31, fp16=f16, **cfg)
    path = str(tmp_path / "m.gguf")
    write_gguf(path, om, cfg, f16=f16)
    g = vk.Gguf(path)
    dm = vk.Model.from_gguf(dev, g)
    g.close()  # the weights are on the device: the mapping may go
    ref = vk.Model(dev, cfg["dim"], cfg["heads"], cfg["ffn"], cfg["vocab"], cfg["layers"], cfg["maxlen"], weight_dtype=vk.FP16 if f16 else vk.Q8_0)
    load_from_oracle(ref, om)
    prompt = O.synth_tokens(31, 1000, 11, cfg["vocab"])
    a, b = dm(prompt, 0), ref(prompt, 0)
    assert np.array_equal(a, b)
    assert np.abs(a - om.forward(prompt, 0)).max() <= LOGITS_MAX_ABS
    assert dm.generate(prompt, 12)[0].tolist() == ref.generate(prompt, 12)[0].tolist()
    # a shorter context than the file's llama.context_length
    g = vk.Gguf(path)
    short = vk.Model.from_gguf(dev, g, maxlen=32)
    assert short.cfg.maxlen == 32 and np.array_equal(short(prompt, 0), b)


def test_device_topk_and_topk_sampler(dev):
    om, dm, cfg = small_pair(dev, seed=14)
    prompt = O.synth_tokens(14, 1000, 9, cfg["vocab"])
    logits = dm(prompt, 0)
    for k in (1, 5, 40, 64):
        vals, ids = dm.topk(k)
        order = np.lexsort((np.arange(logits.size), -logits))[:k]
        assert ids.tolist() == order.tolist() and np.array_equal(vals, logits[order])
    assert dm.topk(1)[1][0] == dm.last_token()
    s = vk.TopkSampler(1, seed=3)
    assert s.sample_candidates(*dm.topk(8)) == int(np.argmax(logits))
    with pytest.raises(vk.VklError) as e:
        dm.topk(65)
    assert e.value.code == 3


def test_chat_session_multi_token_turns_on_top_of_history(dev):
    """app/chat.cpp:286-304 calls model(tokens, offset) with several new tokens on top of the cached
    history, then samples token by token, turn after turn: multi-token calls at offset > 0 and
    one-token calls must interleave on one cache."""
    om, dm, cfg = small_pair(dev, seed=15)
    pos = 0
    for turn, T in enumerate((7, 40, 3, 33)):  # 8 rows and fewer, and more
        toks = O.synth_tokens(15, 1100 + turn, T, cfg["vocab"])
        want, got = om.forward(toks, pos), dm(toks, pos)
        assert np.abs(got - want).max() <= LOGITS_MAX_ABS, "turn %d" % turn
        pos += T
        tok = np.array([int(np.argmax(want))], np.uint32)
        for i in range(3):
            want, got = om.forward(tok, pos), dm(tok, pos)
            assert np.abs(got - want).max() <= LOGITS_MAX_ABS, "turn %d step %d" % (turn, i)
            pos += 1
            tok = np.array([int(np.argmax(want))], np.uint32)
    for l in range(cfg["layers"]):
        gk, gv = dm.read_kv(l)
        assert_close(gk[:, :pos], om.kcache(l)[:, :pos], tol=5e-3, what="kcache layer %d" % l)
        assert_close(gv[:, :pos], om.vcache(l)[:, :pos], tol=5e-3, what="vcache layer %d" % l)


def test_multi_token_call_wraps_the_ring_cache(dev):
    """Positions beyond maxlen overwrite the oldest cache rows ((offset+row) % maxlen,
    update_kvcache_fp16.comp:35), also inside a multi-token call."""
    om, dm, cfg = small_pair(dev, seed=16, maxlen=32)
    a = O.synth_tokens(16, 1000, 28, cfg["vocab"])
    b = O.synth_tokens(16, 1001, 9, cfg["vocab"])
    om.forward(a, 0)
    dm(a, 0)
    want, got = om.forward(b, 28), dm(b, 28)  # rows 28..36: wraps at 32
    assert np.abs(got - want).max() <= LOGITS_MAX_ABS
    for l in range(cfg["layers"]):
        gk, gv = dm.read_kv(l)
        assert_close(gk, om.kcache(l), tol=5e-3, what="kcache layer %d" % l)
        assert_close(gv, om.vcache(l), tol=5e-3, what="vcache layer %d" % l)


# ---- failure detection: a bounded wait inside the decode kernel runs out ------------------------
def test_wait_that_runs_out_returns_an_error_and_leaves_the_device_usable(dev):
    """The counterpart of the reference's 60 s fence time-out (src/core/command.h:389-395). A
    two-rank tensor-parallel shard is created on ONE GPU and "connected" to itself, so the words of
    rank 1 never arrive: the all-reduce's wait gives up after the (shortened) bound, the kernel
    leaves through its normal path, the call reports which wait ran out, the shard refuses further
    steps until it is reconnected, and other models on the device keep working. Nothing faults and
    nothing waits for ever."""
    cfg = dict(dim=256, heads=4, ffn=512, vocab=1000, layers=2, maxlen=128)
    lone = vk.Model(dev, cfg["dim"], cfg["heads"], cfg["ffn"], cfg["vocab"], cfg["layers"], cfg["maxlen"], tp_rank=0, tp_size=2)
    lone.synth_weights(41)
    ptr, nbytes = lone.tp_buffer()
    lone.tp_connect_pointers([ptr, ptr])  # "rank 1" is this rank's own buffer: nobody fills rank 1's slots
    lone.set_wait_limit(4096)
    tok = np.array([5], np.uint32)
    with pytest.raises(vk.VklError) as e:
        lone(tok, 0)
    assert e.value.code == 13 and "code 4" in e.value.message, e.value.message
    with pytest.raises(vk.VklError) as e:  # out of step with its (imaginary) peer: refused on the host
        lone(tok, 0)
    assert e.value.code == 9
    lone.tp_connect_pointers([ptr, ptr])  # reconnecting clears the exchange buffer and the counters
    with pytest.raises(vk.VklError) as e:
        lone.generate(np.array([1, 2, 3], np.uint32), 4)
    assert e.value.code == 13 and "code 4" in e.value.message
    # the many-token prefill of a sharded model waits for the other ranks' partial sums in its row all-reduce:
    # the same bound, its own message, the same refusal afterwards
    lone.tp_connect_pointers([ptr, ptr])
    with pytest.raises(vk.VklError) as e:
        lone.generate(O.synth_tokens(41, 1000, 70, cfg["vocab"]), 2)
    assert e.value.code == 13 and "another tensor-parallel rank" in e.value.message, e.value.message
    with pytest.raises(vk.VklError) as e:
        lone(tok, 0)
    assert e.value.code == 9
    # the device and other models are unaffected
    om, dm, cfg2 = small_pair(dev, seed=42)
    prompt = O.synth_tokens(42, 1000, 6, cfg2["vocab"])
    want, _ = om.generate(prompt, 8)
    assert dm.generate(prompt, 8)[0].tolist() == want.tolist()
    with pytest.raises(vk.VklError) as e:
        dm.set_wait_limit(10)
    assert e.value.code == 3


def test_short_wait_bound_on_a_healthy_model_is_reported_not_hung(dev):
    """With a bound far below what a step needs, the first wait that cannot be met reports its code
    (weights or cache rows, the grid barrier or a tagged input); restoring the default bound makes the same
    model work again and give the oracle's ids."""
    om, dm, cfg = small_pair(dev, seed=43)
    prompt = O.synth_tokens(43, 1000, 5, cfg["vocab"])
    want, _ = om.generate(prompt, 6)
    assert dm.generate(prompt, 6)[0].tolist() == want.tolist()
    dm.set_wait_limit(1024)
    codes = set()
    for _ in range(3):
        try:
            dm(np.array([7], np.uint32), 5)
        except vk.VklError as e:
            assert e.code == 13 and "bounded wait ran out" in e.message
            codes.add(e.message)
    dm.set_wait_limit(0)
    assert dm.generate(prompt, 6)[0].tolist() == want.tolist()  # the sequence base was reset: stale tags do not match


def test_tagged_words_survive_the_16_bit_tag_wrap(dev, monkeypatch):
    """The activation words carry the low 16 bits of a sequence number that advances by the op count
    per token (8 ops for a one-block model): after 8192 tokens the tags come round again. A prompt of
    8300 tokens is fed token by token through the persistent kernel (66400 op numbers), then the
    logits and the following greedy steps are compared with the oracle: a word misread as current
    anywhere on the way would derail the residual stream for good."""
    monkeypatch.setenv("VKLLAMA_PREFILL", "sequential")
    cfg = dict(dim=128, heads=2, ffn=256, vocab=500, layers=1, maxlen=8448)
    om = O.Model(seed=17, **cfg)
    dm = vk.Model(dev, cfg["dim"], cfg["heads"], cfg["ffn"], cfg["vocab"], cfg["layers"], cfg["maxlen"])
    load_from_oracle(dm, om)
    P = 8300
    prompt = O.synth_tokens(17, 1000, P, cfg["vocab"])
    ids, _, _ = dm.generate(prompt, 6)
    ids2, _, _ = dm.generate(prompt, 6)  # a second job continues the sequence numbers where the first ended
    assert ids.tolist() == ids2.tolist()
    # The oracle takes the prompt in one call. (Its logits for that call are not comparable: in a multi-token
    # call the reference rotates the clipped query of the last block at the call's first position,
    # multiheadattention_v2.cpp:223-253, which a token-by-token prefill never does. The caches are.)
    om.forward(prompt, 0)
    gk, gv = dm.read_kv(0)
    assert_close(gk[:, :P], om.kcache(0)[:, :P], tol=5e-3, what="kcache after the wrap")
    assert_close(gv[:, :P], om.vcache(0)[:, :P], tol=5e-3, what="vcache after the wrap")
    tok = np.array([int(ids[0])], np.uint32)
    for i in range(3):
        w, g = om.forward(tok, P + i), dm(tok, P + i)
        assert np.abs(g - w).max() <= LOGITS_MAX_ABS, "step %d after the wrap" % i
        tok = np.array([int(np.argmax(w))], np.uint32)
