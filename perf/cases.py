"""Workloads of the library, as the programs that use it run them: what they hold (`prepare`), what they do (`run`), the least
memory traffic and arithmetic that takes (`work`), and the same results in 64 bits from plain torch (`exact`).

A case names a model by family and sizes and one of four uses:
  generate  a prompt from position 0 and `new` greedy tokens in one call, then the logits that follow the last of them
  chat      `pos` tokens are in the caches; a turn of `prompt` tokens and `new` more, one call each, logits on the host every time
  prompt    `prompt` tokens behind `pos` cached ones in one call, the last one's logits on the host
  block     one Llama-2 block put together from the operator classes, `prompt` rows behind `pos` cached ones
Families: `llama` with Q8_0 or FP16 weights; `rumalorn` and `kupuzen` with bfloat16 weights and bf16 or f32 arithmetic.
"""
import math

import numpy as np
import torch

import vkllama_b200 as vk

MAXLEN = 4096   # context length of every model
RANK = 128      # of the two-step projections of a delta-rule layer
WINDOW = 1024   # of a windowed attention layer


def _case(family, use, weights, width, heads, ffn, layers, vocab, pos, prompt, new, kv_heads=0, mix="", name=None):
    c = {"name": name} if name else {}
    c.update(family=family, use=use, weights=weights, width=width, heads=heads, kv_heads=kv_heads or heads, ffn=ffn, layers=layers,
             vocab=vocab, pos=pos, prompt=prompt, new=new, mix=mix)
    return c


def listed():
    return [
        # a chat with a toy model: nothing but launches and synchronisations
        _case("llama", "chat", "q8_0", 256, 4, 512, 2, 1000, 0, 8, 16, name="chat-tiny"),
        # the operator classes, one row: a program with a token loop of its own
        _case("llama", "block", "q8_0", 4096, 32, 11008, 1, 0, 200, 1, 0, name="block-1-row"),
        # the same with a ragged batch of prompt rows
        _case("llama", "block", "f16", 4096, 32, 11008, 1, 0, 0, 77, 0, name="block-77-rows"),
        # the headline: Llama-2-7B, a 32-token prompt, greedy tokens
        _case("llama", "generate", "q8_0", 4096, 32, 11008, 32, 32000, 0, 32, 64, name="generate-7b"),
        # a conversation near the end of its context, a sampler on the host (4 blocks of the 7B shape)
        _case("llama", "chat", "q8_0", 4096, 32, 11008, 4, 32000, 3500, 1, 12, name="chat-long"),
        # a user's turn of a few dozen tokens and the start of the answer (4 blocks of the 13B shape)
        _case("llama", "chat", "q8_0", 5120, 40, 13824, 4, 32000, 700, 45, 6, name="turn-13b"),
        # a page of text read in one call
        _case("llama", "prompt", "q8_0", 4096, 32, 11008, 4, 32000, 0, 509, 0, name="prompt-q8"),
        # a long document, 16-bit weights
        _case("llama", "prompt", "f16", 4096, 32, 11008, 4, 32000, 0, 2048, 0, name="prompt-f16"),
        # short question, short answer, 16-bit weights
        _case("llama", "generate", "f16", 4096, 32, 11008, 4, 32000, 0, 17, 32, name="generate-f16"),
        # routed experts and a loop over layers, a prompt of odd length
        _case("rumalorn", "prompt", "bf16", 2048, 16, 5632, 6, 32000, 0, 777, 0, kv_heads=4, mix="moe", name="rumalorn-moe-prompt"),
        # both kinds of mixer: a long prompt through the delta rule, then tokens
        _case("kupuzen", "generate", "bf16", 2048, 16, 5632, 8, 32000, 0, 2048, 32, mix="ddas", name="kupuzen-generate"),
        # 32-bit arithmetic throughout
        _case("kupuzen", "generate", "f32", 2048, 16, 5632, 4, 32000, 0, 300, 4, mix="ddas", name="kupuzen-32-bit"),
    ]


def draw(rng):
    spread = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))  # noqa: E731
    family = rng.choice(["llama", "llama", "rumalorn", "kupuzen"])
    heads = spread(2, 40)
    hd = rng.choice([64, 128])
    width = heads * hd
    ffn = max(2, spread(width * 2, width * 3) // 32) * 32
    vocab = rng.choice([997, 8000, 32000])
    layers = rng.randint(1, 4)
    if family == "llama":
        use = rng.choice(["generate", "chat", "prompt", "block"])
        weights = rng.choice(["q8_0", "q8_0", "f16"])
        kv, mix = heads, ""
    else:
        use = rng.choice(["generate", "prompt"] + (["chat"] if family == "rumalorn" else []))
        weights = rng.choice(["bf16", "bf16", "f32"])
        kv = rng.choice([heads] + [k for k in (1, heads // 2, heads // 4) if k and heads % k == 0])
        mix = rng.choice(["", "moe"] if family == "rumalorn" else ["d", "a", "ddas", "as"])
    most = 300 if weights == "f32" else 2048
    prompt = spread(2, most) if use in ("generate", "prompt") else spread(1, 300)
    pos = spread(1, 3000) if use in ("chat", "block") else spread(1, 1500) if use == "prompt" and family == "llama" else 0
    new = spread(1, 40) if use == "generate" else spread(1, 16) if use == "chat" else 0
    if use == "block":
        layers, vocab = 1, 0
    return _case(family, use, weights, width, heads, ffn, layers, vocab, pos, prompt, new, kv, mix)


# ---- what a model consists of ---------------------------------------------------------------
def _config(c):
    """config.json of a layer-list model."""
    d, h, g, f = c["width"], c["heads"], c["kv_heads"], c["ffn"]
    hd, n = d // h, c["layers"]
    mix = {"heads": h, "kv_heads": g, "dim": hd, "vdim": hd}
    if c["family"] == "rumalorn":
        moe = c["mix"] == "moe"
        mix.update(scale=hd ** -0.5, bias_max=1024, q_temp={"coef": 0.1, "every": 512})
        dense = {"kind": "dense", "ff": f, "limit": 7.0}
        routed = {"kind": "moe", "expert": {"ff": f // 4}, "router": {"experts": 16, "top": 2}}
        return {"architecture": "Rumalorn", "vocab": c["vocab"], "width": d, "logit_scale": 1.0, "norm": {"eps": 1e-6},
                "loop": {"start": 0, "stop": max(1, n // 2), "times": 2} if moe else None,
                "layers": [{"type": "attention", "mixer": mix, "mlp": routed if moe and i % 2 else dense} for i in range(n)]}
    attn = dict(mix, scale=hd ** -0.5, mask={"size": WINDOW},
                rot={"base": 500000.0, "dims": hd, "scaling": {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 8192}})
    layers = []
    for i in range(n):
        k = c["mix"][i % len(c["mix"])]
        m = dict(mix, conv=4) if k == "d" else dict(attn, kv_from=i - 1) if k == "s" else attn
        layers.append({"type": "channel_delta" if k == "d" else "attention", "mixer": m, "mlp": {"kind": "dense", "ff": f}})
    return {"architecture": "Kupuzen", "vocab": c["vocab"], "width": d, "embedding": {"scale": 1.0}, "residual_mult": 1.0,
            "logit_softcap": 30.0, "norm": {"eps": 1e-6}, "layers": layers}


def _tensors(c):
    """name -> (shape, mean, deviation). Deviations keep scores at a few units and every part of a layer in play."""
    d, h, f, v, n = c["width"], c["heads"], c["ffn"], c["vocab"], c["layers"]
    t = {}
    if c["family"] == "llama":
        if c["use"] != "block":
            t["token_embd.weight"] = ((v, d), 0.0, 1.0)
            t["output.weight"] = ((v, d), 0.0, 0.02)
            t["output_norm.weight"] = ((d,), 1.0, 0.1)
        for i in range(n):
            p = "blk.%d." % i
            for k in ("attn_norm", "ffn_norm"):
                t[p + k + ".weight"] = ((d,), 1.0, 0.1)
            std = 0.02 * (4096 / d) ** 0.5
            for k in ("attn_q", "attn_k", "attn_v"):
                t[p + k + ".weight"] = ((d, d), 0.0, std)
            for k in ("ffn_gate", "ffn_up"):
                t[p + k + ".weight"] = ((f, d), 0.0, std)
            # what adds to the stream is smaller the deeper the model, as training starts it
            t[p + "attn_output.weight"], t[p + "ffn_down.weight"] = ((d, d), 0.0, std * n ** -0.5), ((d, f), 0.0, std * n ** -0.5)
        return t
    cfg = _config(c)
    kupuzen = c["family"] == "kupuzen"
    t["embed"], t["head"] = ((v, d), 0.0, 1.0), ((v, d), 0.0, d ** -0.5)

    def norm(name):
        if kupuzen:
            t[name] = ((d,), 0.0, 0.1)
        else:
            t[name], t[name + ".b"], t[name + ".alpha"] = ((d,), 1.0, 0.2), ((d,), 0.0, 0.1), ((1,), 0.6, 0.0)

    norm("final.norm")
    if cfg.get("loop"):
        t["loop.step"] = ((cfg["loop"]["times"], d), 0.0, 0.3)
    for i, layer in enumerate(cfg["layers"]):
        a, ml, p = layer["mixer"], layer["mlp"], "l%d.mix." % i
        g, hd = a["kv_heads"], a["dim"]
        norm("l%d.norm1" % i)
        if layer["type"] == "channel_delta":
            for k, w in (("q", g * hd), ("k", g * hd), ("v", h * hd)):
                t[p + k], t[p + k + ".conv"] = ((w, d), 0.0, 2 * d ** -0.5), ((w, a["conv"]), 0.0, 0.6)
            t[p + "b"] = ((h, d), 0.0, 2 * d ** -0.5)
            t[p + "A_log"], t[p + "dt_bias"], t[p + "norm"] = ((h,), -2.0, 1.0), ((h * hd,), -1.5, 0.8), ((hd,), 1.0, 0.2)
            for k in ("a", "g"):
                t[p + k + "1"], t[p + k + "2"] = ((RANK, d), 0.0, d ** -0.5), ((h * hd, RANK), 0.0, 1.5 * RANK ** -0.5)
        elif kupuzen:
            t[p + "q"], t[p + "q.norm"] = ((h * hd, d), 0.0, d ** -0.5), ((h * hd,), 1.0, 0.2)
            if a.get("kv_from") is None:
                t[p + "k"], t[p + "k.norm"] = ((g * hd, d), 0.0, d ** -0.5), ((g * hd,), 1.0, 0.2)
                t[p + "v"] = ((g * hd, d), 0.0, d ** -0.5)
            t[p + "sink"] = ((h,), 0.0, 1.0)
        else:
            t[p + "q"], t[p + "q.b"] = ((h * hd, d), 0.0, 1.6 * d ** -0.5), ((h * hd,), 0.0, 0.3)
            t[p + "k"], t[p + "k.b"] = ((g * hd, d), 0.0, 1.6 * d ** -0.5), ((g * hd,), 0.0, 0.3)
            t[p + "rel"], t[p + "g"] = ((32, h), 0.0, 0.8), ((h, d), 0.0, 2 * d ** -0.5)
            t[p + "o.b"] = ((d,), 0.0, 0.1)
        t[p + "o"] = ((d, h * hd), 0.0, d ** -0.5)
        p = "l%d.mlp." % i
        if kupuzen:
            norm("l%d.norm2" % i)
        for e in range(ml["router"]["experts"]) if ml["kind"] == "moe" else (None,):
            q, ff = (p, ml["ff"]) if e is None else ("%se%d." % (p, e), ml["expert"]["ff"])
            for k, s in (("gate", (ff, d)), ("up", (ff, d)), ("down", (d, ff))):
                t[q + k] = (s, 0.0, 0.8 * s[1] ** -0.5 if k == "down" else 1.4 * s[1] ** -0.5)
        if ml["kind"] == "moe":
            t[p + "table"] = ((v, ml["router"]["top"]), 0.0, float(ml["router"]["experts"]))
    return t


def _q8_0(w):
    """34-byte blocks of 32 values (a half scale, 32 signed bytes), and the values they stand for."""
    b = w.reshape(w.shape[0], -1, 32)
    d = b.abs().amax(2, keepdim=True) / 127
    q = torch.where(d > 0, b / d, 0.0).round().clamp(-127, 127)
    d = d.half()
    blocks = torch.cat([d.view(torch.uint8), q.to(torch.int8).view(torch.uint8)], 2)
    return blocks, (q * d.float()).reshape(w.shape)


class _Weights:
    """A model's tensors, one at a time, from the seed: as stored (for the library) and as values (for `exact`)."""

    def __init__(self, c, seed):
        self.c, self.seed, self.t = c, seed, _tensors(c)
        self.at = {k: i for i, k in enumerate(self.t)}

    def _normal(self, name):
        shape, mean, std = self.t[name]
        g = torch.Generator("cuda").manual_seed(self.seed * 100003 + self.at[name])
        return torch.randn(shape, generator=g, device="cuda") * std + mean

    def get(self, name):
        """(dtype, stored tensor, values)."""
        llama = self.c["family"] == "llama"
        if name.endswith(".table"):
            (v, top), _, experts = self.t[name]
            g = torch.Generator("cuda").manual_seed(self.seed * 100003 + self.at[name])
            w = torch.rand((v, int(experts)), generator=g, device="cuda").argsort(1)[:, :top].to(torch.int32).contiguous()
            return vk.UINT32, w, w.long()
        w = self._normal(name)
        if name in ("output.weight", "head"):
            # as in a trained model, one continuation stands out: every id is mostly followed by the next one
            w += (3.0 if llama else 1.0) * w.shape[1] ** -0.5 * self._normal("token_embd.weight" if llama else "embed").roll(1, 0)
        if not llama:
            w = w.bfloat16()
            return vk.BF16, w, w.float()
        if w.dim() == 1:
            return vk.FP32, w, w
        if self.c["weights"] == "f16":
            w = w.half()
            return vk.FP16, w, w.float()
        return (vk.Q8_0,) + _q8_0(w)

    def value(self, name):
        v = self.get(name)[2]
        return v if v.dtype == torch.int64 else v.double()


_pinned = None


def _host(t):
    """The bytes of a GPU tensor in a page-locked buffer that the next call overwrites."""
    global _pinned
    b = t.contiguous().reshape(-1).view(torch.uint8)
    if _pinned is None or _pinned.numel() < b.numel():
        _pinned = torch.empty(max(b.numel(), 1 << 24), dtype=torch.uint8, pin_memory=True)
    _pinned[:b.numel()].copy_(b)
    return _pinned[:b.numel()].numpy()


_dev = None


def _device():
    global _dev
    if _dev is None:
        _dev = vk.Device(0)
    return _dev


def _text(c, seed):
    """Token ids of everything that the case reads, in order."""
    g = np.random.default_rng(seed * 7 + 1)
    return g.integers(0, max(2, c["vocab"]), c["pos"] + c["prompt"] + c["new"]).astype(np.uint32)


def _rows(c, seed):
    """Inputs of a block: the rows that fill its caches and the rows of the call, with a stream's magnitudes."""
    g = np.random.default_rng(seed * 7 + 1)
    x = g.normal(0, 1, (c["pos"] + c["prompt"], c["width"])).astype(np.float16)
    return x[:c["pos"]], x[c["pos"]:]


# ---- the library's side ---------------------------------------------------------------------
class _Block:
    """One Llama-2 block from the operator classes: attention and feed-forward, each behind a norm and added to the stream."""

    def __init__(self, dev, c, w):
        self.cmd = cmd = vk.Command(dev)
        self.keep = []
        fp16 = vk.FP16

        def tensor(name):
            dt, stored, values = w.get("blk.0.%s.weight" % name)
            shape = (1,) + tuple(values.shape) if values.dim() == 2 else (1, 1, values.numel())
            t = vk.Tensor(*shape, dev, dt)
            cmd.begin()
            cmd.upload(_host(stored), t)
            cmd.end()
            cmd.submit_and_wait()
            self.keep.append(t)
            return t

        n1, n2 = tensor("attn_norm"), tensor("ffn_norm")
        q, k, v, o = (tensor("attn_" + s) for s in ("q", "k", "v", "output"))
        gate, up, down = (tensor("ffn_" + s) for s in ("gate", "up", "down"))
        cmd.begin()
        self.norm1, self.norm2 = vk.RMSNorm(dev, cmd, n1, 1e-5, fp16).init(), vk.RMSNorm(dev, cmd, n2, 1e-5, fp16).init()
        self.attn = vk.MultiHeadAttentionV2(dev, cmd, k, q, v, o, MAXLEN, c["width"] // c["heads"], True, fp16, True, False).init()
        self.ff = vk.FeedForward(dev, cmd, gate, down, up, True, fp16 if c["weights"] == "f16" else vk.Q8_0).init()
        self.add1, self.add2 = vk.ElementWise(dev, cmd, 0, fp16).init(), vk.ElementWise(dev, cmd, 0, fp16).init()
        cmd.end()
        cmd.submit_and_wait()
        self.dev = dev

    def __call__(self, x, offset):
        cmd = self.cmd
        t = vk.Tensor(1, x.shape[0], x.shape[1], self.dev, vk.FP16)
        cmd.begin()
        cmd.upload(x, t)
        y = self.add1(self.attn(self.norm1(t), offset), t)
        z = self.add2(self.ff(self.norm2(y)), y)
        out = cmd.download(z)
        cmd.end()
        cmd.submit_and_wait()
        return out.view(np.float16)


def prepare(case, seed):
    c, w, dev = case, _Weights(case, seed), _device()
    if c["use"] == "block":
        before, x = _rows(c, seed)
        block = _Block(dev, c, w)
        if len(before):
            block(before, 0)
        return {"case": c, "block": block, "x": x}
    if c["family"] == "llama":
        dt = vk.FP16 if c["weights"] == "f16" else vk.Q8_0
        m = vk.Model(dev, c["width"], c["heads"], c["ffn"], c["vocab"], c["layers"], MAXLEN, weight_dtype=dt)
    else:
        shapes = {k: v[0] for k, v in w.t.items()}
        m = vk.Model.from_config(dev, _config(c), MAXLEN, vk.FP32 if c["weights"] == "f32" else vk.BF16, shapes=shapes)
    for name in w.t:
        dt, stored, _ = w.get(name)
        m.set_weight(name, dt, _host(stored))
    text = _text(c, seed)
    if c["pos"]:
        m(text[:c["pos"]], 0)
    return {"case": c, "model": m, "text": text, "logits": np.empty((c["new"] + 1, c["vocab"]), np.float32)}


def run(state):
    c = state["case"]
    if c["use"] == "block":
        return state["block"](state["x"], c["pos"])
    m, text, pos, n, new, logits = state["model"], state["text"], c["pos"], c["prompt"], c["new"], state["logits"]
    if c["use"] == "prompt":
        return m(text[pos:pos + n], pos, logits[0])
    if c["use"] == "generate":
        ids = m.generate(text[:n], new)[0]
        return {"ids": ids, "logits": m(ids[-1:], n + new - 1, logits[0])}
    m(text[pos:pos + n], pos, logits[0])
    for i in range(new):  # the ids that a sampler on the host picked
        at = pos + n + i
        m(text[at:at + 1], at, logits[i + 1])
    return logits


# ---- what it takes --------------------------------------------------------------------------
def work(case):
    c = case
    size = {"q8_0": 34 / 32, "f16": 2, "bf16": 2, "f32": 2}[c["weights"]]  # 32-bit models keep their weights as bfloat16
    act = 4 if c["weights"] == "f32" else 2
    d, h, g, v = c["width"], c["heads"], c["kv_heads"], c["vocab"]
    hd = d // h
    cfg = _config(c) if c["family"] != "llama" else None
    runs = list(range(c["layers"]))
    if cfg and cfg.get("loop"):
        lp = cfg["loop"]
        runs = runs[:lp["stop"]] * lp["times"] + runs[lp["stop"]:]
    elements = {k: float(np.prod(s[0])) for k, s in _tensors(c).items() if len(s[0]) == 2 and not k.endswith((".table", ".rel", ".conv", "step"))}
    layer = lambda i: ("blk.%d." if c["family"] == "llama" else "l%d.") % i  # noqa: E731

    def call(pos, n):
        """Bytes and operations of n tokens behind pos cached ones in one call."""
        b = f = 0.0
        for i in runs:
            here = {k: e for k, e in elements.items() if k.startswith(layer(i))}
            routed = sum(e for k, e in here.items() if ".mlp.e" in k)
            dense = sum(here.values()) - routed
            mix = cfg["layers"][i]["mixer"] if cfg else {}
            b += size * (dense + routed * (1 - (1 - 2 / 16) ** n))  # the experts that n tokens name
            f += 2 * n * (dense + routed * 2 / 16)
            if cfg and cfg["layers"][i]["type"] == "channel_delta":
                b += 2 * 4 * h * hd * hd
                f += 7 * n * h * hd * hd
            else:
                win = mix.get("mask", {}).get("size", 1 << 30)
                caches = 1 if c["family"] == "rumalorn" else 2
                pairs = sum(min(pos + j + 1, win) for j in range(n))
                b += act * caches * g * hd * (min(pos, win) + n)
                f += 4 * h * hd * pairs
        if v:
            b += size * v * d + 4 * v + size * n * d
            f += 2 * v * d
        else:
            b += 2 * 2 * n * d
        return b, f

    calls = [(c["pos"], c["prompt"])]
    if c["use"] in ("generate", "chat"):
        calls += [(c["pos"] + c["prompt"] + i, 1) for i in range(c["new"])]
    b, f = (sum(x) for x in zip(*(call(p, n) for p, n in calls)))
    return {"bytes": b, "flops": f}


def tolerance(case):
    # four times the distance from `exact` that was measured: fp16 and bf16 activations, 32-bit sums
    return {"rel": {"q8_0": 8e-3, "f16": 8e-3, "bf16": 2.5e-2, "f32": 1e-5}[case["weights"]], "differ": 0.0}


# ---- the same in 64 bits ---------------------------------------------------------------------
def _rotate(x, pos, freq):
    """x [T, heads, width]: neighbours turn by pos * freq."""
    a = pos.double()[:, None, None] * freq
    u, v = x[..., 0::2], x[..., 1::2]
    return torch.stack([u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin()], -1).flatten(2)


def _attend(q, k, v, scale, window=None, bias=None, sink=None):
    """q [T, H, d], k and v [T, G, d]; bias [H, distance]; sink [H]: one more term of the denominator."""
    T, H, _ = q.shape
    per = H // k.shape[1]
    back = torch.arange(T, device=q.device)[:, None] - torch.arange(T, device=q.device)[None, :]
    hidden = (back < 0) | (back >= (window or T + 1))
    out = torch.empty(T, H, v.shape[2], dtype=q.dtype, device=q.device)
    for h in range(H):
        s = (q[:, h] @ k[:, h // per].T) * scale
        if bias is not None:
            s += bias[h][back.clamp_min(0)]
        s.masked_fill_(hidden, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[h].expand(T, 1)], 1)
        out[:, h] = s.softmax(1)[:, :T] @ v[:, h // per]
    return out


def _rms(x, eps):
    return x / (x.square().mean(-1, keepdim=True) + eps).sqrt()


def _silu(x):
    return x * x.sigmoid()


def _llama_block(x, W, i, c, qpos):
    """qpos: the position that each row's query is turned by."""
    T, d, h = x.shape[0], c["width"], c["heads"]
    hd = d // h
    w = lambda k: W.value("blk.%d.%s.weight" % (i, k))  # noqa: E731
    freq = 10000.0 ** (-torch.arange(0, hd, 2, device=x.device, dtype=x.dtype) / hd)
    n = _rms(x, 1e-5) * w("attn_norm")
    q = _rotate((n @ w("attn_q").T).view(T, h, hd), qpos, freq)
    k = _rotate((n @ w("attn_k").T).view(T, h, hd), torch.arange(T, device=x.device), freq)
    v = (n @ w("attn_v").T).view(T, h, hd)
    x = x + _attend(q, k, v, hd ** -0.5).reshape(T, d) @ w("attn_output").T
    n = _rms(x, 1e-5) * w("ffn_norm")
    return x + (_silu(n @ w("ffn_gate").T) * (n @ w("ffn_up").T)) @ w("ffn_down").T


def _llama(W, c, text, calls):
    """Logits after each call of (position, tokens). Behind a call's last block the reference keeps one row only and turns
    its query as the call's first one."""
    T = len(text)
    pos = torch.arange(T, device="cuda")
    last = pos.clone()
    for p, n in calls:
        if n > 1:
            last[p + n - 1] = p
    x = W.value("token_embd.weight")[torch.from_numpy(text.astype(np.int64)).cuda()]
    for i in range(c["layers"]):
        x = _llama_block(x, W, i, c, last if i == c["layers"] - 1 else pos)
    rows = torch.tensor([p + n - 1 for p, n in calls], device="cuda")
    return (_rms(x[rows], 1e-6) * W.value("output_norm.weight")) @ W.value("output.weight").T


def _rumalorn(W, c, text, calls):
    cfg, d, h = _config(c), c["width"], c["heads"]
    T, hd, g = len(text), d // h, c["kv_heads"]
    ids = torch.from_numpy(text.astype(np.int64)).cuda()
    emb = W.value("embed")[ids]
    x, lp = emb, cfg["loop"]
    norm = lambda k, z: torch.tanh(W.value(k + ".alpha") * z) * W.value(k) + W.value(k + ".b")  # noqa: E731
    runs = [(i, None) for i in range(c["layers"])]
    if lp:
        runs = [(i, t) for t in range(lp["times"]) for i in range(lp["stop"])] + runs[lp["stop"]:]
    # rows of the distance table: the first half one by one, the others on a logarithmic scale that ends at 1024
    n, rows = np.arange(T), 32
    half = rows // 2
    bucket = np.array([j if j < half else min(rows - 1, half + next(k for k in range(half, -1, -1) if j ** half * half ** k >= 1024 ** k * half ** half)) for j in map(int, n)])
    temp = 1 + 0.1 * torch.log(torch.floor((torch.arange(T, device="cuda").double() + 1) / 512) + 1)
    for i, t in runs:
        if t is not None and i == 0:
            x = (x + emb if t else x) + W.value("loop.step")[t]
        z, p = norm("l%d.norm1" % i, x), "l%d.mix." % i
        q = (z @ W.value(p + "q").T + W.value(p + "q.b")).view(T, h, hd) * temp[:, None, None]
        k = (z @ W.value(p + "k").T + W.value(p + "k.b")).view(T, g, hd)
        o = _attend(q, k, k, hd ** -0.5, bias=W.value(p + "rel")[torch.from_numpy(bucket).cuda()].T)
        o = o * torch.sigmoid(z @ W.value(p + "g").T)[:, :, None]
        y = o.reshape(T, d) @ W.value(p + "o").T + W.value(p + "o.b")
        p = "l%d.mlp." % i
        if cfg["layers"][i]["mlp"]["kind"] == "dense":
            a = (z @ W.value(p + "gate").T).clamp_max(7.0)
            u = (z @ W.value(p + "up").T).clamp(-7.0, 7.0)
            y = y + (a * torch.sigmoid(1.702 * a) * (u + 1)) @ W.value(p + "down").T
        else:
            table = W.value(p + "table")[ids]
            for e in range(16):
                at = (table == e).any(1).nonzero()[:, 0]
                zz, q = z[at], "%se%d." % (p, e)
                y.index_add_(0, at, (_silu(zz @ W.value(q + "gate").T) * (zz @ W.value(q + "up").T)) @ W.value(q + "down").T / 2)
        x = x + y
    at = torch.tensor([p + n - 1 for p, n in calls], device="cuda")
    return norm("final.norm", x[at]) @ W.value("head").T


def _delta(z, W, p, mix, eps):
    T, h, g, hd = z.shape[0], mix["heads"], mix["kv_heads"], mix["dim"]

    def side(k):
        x, taps = z @ W.value(p + k).T, W.value(p + k + ".conv")
        n = taps.shape[1]
        padded = torch.cat([x.new_zeros(n - 1, x.shape[1]), x])
        return _silu(sum(padded[j:j + T] * taps[:, j] for j in range(n)))

    unit = lambda x: x / (x.square().sum(-1, keepdim=True) + 1e-6).sqrt()  # noqa: E731
    q = unit(side("q").view(T, g, hd)).repeat_interleave(h // g, 1) * hd ** -0.5
    k = unit(side("k").view(T, g, hd)).repeat_interleave(h // g, 1)
    v = side("v").view(T, h, hd)
    beta = torch.sigmoid(z @ W.value(p + "b").T)[:, :, None]
    step = torch.nn.functional.softplus(z @ W.value(p + "a1").T @ W.value(p + "a2").T + W.value(p + "dt_bias"), threshold=1e9).view(T, h, hd)
    keep = torch.exp(-torch.exp(W.value(p + "A_log"))[:, None] * step)[..., None]
    S, out = z.new_zeros(h, hd, hd), torch.empty_like(v)
    for t in range(T):
        S = S * keep[t]
        u = beta[t] * (v[t] - torch.matmul(k[t][:, None], S)[:, 0])
        S = torch.baddbmm(S, k[t][:, :, None], u[:, None])
        out[t] = torch.matmul(q[t][:, None], S)[:, 0]
    o = (_rms(out, eps) * W.value(p + "norm")).reshape(T, h * hd)
    return (o * torch.sigmoid(z @ W.value(p + "g1").T @ W.value(p + "g2").T)) @ W.value(p + "o").T


def _kupuzen(W, c, text, calls):
    cfg, d, h = _config(c), c["width"], c["heads"]
    T, hd, g, eps = len(text), d // h, c["kv_heads"], 1e-6
    x = W.value("embed")[torch.from_numpy(text.astype(np.int64)).cuda()]
    pos, kv = torch.arange(T, device="cuda"), None
    norm = lambda k, z: _rms(z, eps) * (1 + W.value(k))  # noqa: E731
    # long wavelengths are stretched by 8, short ones not at all, with a linear passage between
    freq = 500000.0 ** (-np.arange(0, hd, 2) / hd)
    s = np.clip((8192 * freq / (2 * math.pi) - 1.0) / 3.0, 0, 1)
    freq = torch.from_numpy((1 - s) * freq / 8.0 + s * freq).cuda()
    for i, layer in enumerate(cfg["layers"]):
        z, p = norm("l%d.norm1" % i, x), "l%d.mix." % i
        if layer["type"] == "channel_delta":
            y = _delta(z, W, p, layer["mixer"], eps)
        else:
            turned = lambda k, n: _rotate((_rms(z @ W.value(p + k).T, eps) * W.value(p + k + ".norm")).view(T, n, hd), pos, freq)  # noqa: E731
            if layer["mixer"].get("kv_from") is None:
                kv = turned("k", g), (z @ W.value(p + "v").T).view(T, g, hd)
            o = _attend(turned("q", h), *kv, hd ** -0.5, window=WINDOW, sink=W.value(p + "sink"))
            y = o.reshape(T, d) @ W.value(p + "o").T
        z, p = norm("l%d.norm2" % i, x), "l%d.mlp." % i
        x = x + y + (_silu(z @ W.value(p + "gate").T) * (z @ W.value(p + "up").T)) @ W.value(p + "down").T
    at = torch.tensor([p + n - 1 for p, n in calls], device="cuda")
    y = norm("final.norm", x[at]) @ W.value("head").T
    return 30.0 * torch.tanh(y / 30.0)


def exact(case, seed):
    if not torch.cuda.is_available():
        return None
    c, W = case, _Weights(case, seed)
    n, new, pos = c["prompt"], c["new"], c["pos"]
    if c["use"] == "block":
        x = torch.from_numpy(np.concatenate(_rows(c, seed))).cuda().double()
        return _llama_block(x, W, 0, c, torch.arange(len(x), device="cuda"))[pos:].cpu().numpy()[None]
    model = {"llama": _llama, "rumalorn": _rumalorn, "kupuzen": _kupuzen}[c["family"]]
    text = _text(c, seed)
    calls = [(pos, n)] + [(pos + n + i, 1) for i in range(new)]
    if c["use"] != "generate":
        y = model(W, c, text, calls).cpu().numpy()
        return y[0] if c["use"] == "prompt" else y
    # greedy ids: guess them all, take those that the logits confirm, guess the rest anew
    for i in range(new):
        text[n + i] = (text[n + i - 1] + 1) % c["vocab"]
    for _ in range(8):
        y = model(W, c, text, calls)
        best = y[:new].argmax(1).cpu().numpy().astype(np.uint32)
        wrong = np.nonzero(best != text[n:])[0]
        if not len(wrong):
            return {"ids": best.astype(np.float64), "logits": y[new].cpu().numpy()}
        text[n + wrong[0]:] = best[wrong[0]:]
    return None
