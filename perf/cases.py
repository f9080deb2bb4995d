"""What the framework's speed is measured on: requests as a user's program makes them, through the two public engines.

Two engines carry all work.  `capi.Model` is the quantized Llama-style decoder (INT4 / INT8 weights, fp32 activations and cache); its
users generate greedily for one request, read long prompts, and generate for a batch.  `seq.SeqModel` is the layered engine (bf16 weights);
its users bring prompts -- one long one, or several of different lengths in one step -- and decode live sequences token by token.
Widths, head counts, inner sizes and vocabularies are those of the repository's shape table (tinyllama, llama7b, bench-small) and of its
architecture benchmark (w1024, w2048, w4096); depth is cut, because every layer of a stack costs the same and a whole stack only makes a
pass longer.  The vocabulary stays whole, so the head has its real share of a short stack's time or more.

A case is one request pattern:
  kind "llama"            bits 4 / 8; call "generate" (prompt, new), "prefill" (prompt), "batch" (batch, prompt, new)
  kind "Binusun"          layers "w" (wkv recurrence) and "a" (windowed rotary attention + gated feed-forward); loop: the layers but the
                          last run twice.  Call "prompt" (lens: the portions of one step), "answer" (seqs, prompt, new)
  kind "Nubipel"          layers "l" (latent attention), "d" (delta rule), "a" (chunked attention), each with a dense feed-forward; the same calls

Weights come from the engines' own synthetic generator (splitmix64 of seed and element index), so that a state is made on the device in
well under a second and exact() can make the same numbers again.  "answer" feeds given tokens instead of picking them: the work of a
step is the same, and the logits of all steps can be compared."""
import math

import numpy as np
import torch

_M = (1 << 64) - 1


# ---- the cases ----------------------------------------------------------------------------------------------------------------
def _llama(call, hidden, layers, heads, inter, bits, vocab=32000, **kw):
    return dict(kind="llama", call=call, hidden=hidden, layers=layers, heads=heads, inter=inter, bits=bits, vocab=vocab, **kw)


def _seq(kind, call, layers, width, heads, kv_heads, dim, ff, window, vocab=32000, loop=False, **kw):
    return dict(kind=kind, call=call, layers=layers, width=width, heads=heads, kv_heads=kv_heads, dim=dim, ff=ff, window=window, vocab=vocab, loop=loop, **kw)


W1024 = dict(width=1024, heads=8, kv_heads=2, dim=128, ff=2816, window=512)
W2048 = dict(width=2048, heads=16, kv_heads=4, dim=128, ff=5632, window=1024)
W4096 = dict(width=4096, heads=32, kv_heads=8, dim=128, ff=11008, window=1024)


def listed():
    return [
        # the smallest model of the shape table answering one short request: launches, hand-overs and the call itself
        dict(_llama("generate", 256, 4, 4, 1024, 8, vocab=1000, prompt=4, new=32), name="llama_small_generate"),
        # one chat turn on a 1B-class decoder, INT4: the weights of a step are a few megabytes, latency decides
        dict(_llama("generate", 2048, 4, 32, 5632, 4, prompt=16, new=64), name="llama_1b_generate"),
        # one request on 7B-class layers, INT8: the weight stream decides
        dict(_llama("generate", 4096, 4, 32, 11008, 8, prompt=8, new=48), name="llama_7b_generate"),
        # a prompt that is no multiple of anything on the 1B class (heads of 64)
        dict(_llama("prefill", 2048, 4, 32, 5632, 8, prompt=333), name="llama_1b_prefill_333"),
        # the long prompt of the 7B class, INT4: the largest case
        dict(_llama("prefill", 4096, 4, 32, 11008, 4, prompt=2048), name="llama_7b_prefill_2048"),
        # batched generation in lockstep: a full batch on 7B-class layers, and a small one on the 1B class
        dict(_llama("batch", 4096, 4, 32, 11008, 4, batch=32, prompt=6, new=16), name="llama_7b_batch_32"),
        dict(_llama("batch", 2048, 4, 32, 5632, 4, batch=7, prompt=5, new=24), name="llama_1b_batch_7"),
        # the whole Binusun benchmark model (looped, seven layer runs) reading a long prompt
        dict(_seq("Binusun", "prompt", "waaw", loop=True, lens="2048", **W2048), name="binusun_prompt_2048"),
        # several requests' prompts of ragged lengths in one step: attention layers alone
        dict(_seq("Binusun", "prompt", "aa", lens="77,512,900,41", **W2048), name="attention_prompts_ragged"),
        # one attention and one recurrent layer answering four live requests
        dict(_seq("Binusun", "answer", "aw", seqs=4, prompt=200, new=24, **W1024), name="binusun_answer_4"),
        # wide Nubipel layers (latent attention, delta rule, chunked attention) reading a prompt of odd length
        dict(_seq("Nubipel", "prompt", "lda", lens="1999", **W4096), name="nubipel_prompt_1999"),
        # one request decoded behind a long context
        dict(_seq("Nubipel", "answer", "lda", seqs=1, prompt=1200, new=40, **W2048), name="nubipel_answer_1"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.choice(["generate", "prefill", "batch", "Binusun prompt", "Nubipel prompt", "Binusun answer", "Nubipel answer"])
    if what in ("generate", "prefill", "batch"):
        d = rng.choice([64, 64, 128])
        heads = rng.choice([4, 8, 12, 16, 20, 24, 32]) if d == 64 else rng.choice([4, 8, 12, 16, 24, 32])
        H = heads * d
        c = _llama(what, H, rng.randint(1, 4), heads, 32 * max(4, int(H * rng.uniform(2.3, 3.6) / 32)), rng.choice([4, 8]), vocab=rng.choice([1000, 8192, 32000]))
        if what == "generate":
            return dict(c, prompt=rng.randint(1, 30), new=_log(rng, 4, 64))
        if what == "prefill":
            return dict(c, prompt=_log(rng, 34, 2048))
        return dict(c, batch=rng.randint(2, 32), prompt=rng.randint(1, 12), new=rng.randint(4, 16))
    kind, call = what.split()
    z = dict(rng.choice([W1024, W2048, W2048, W4096]))
    z["window"] = rng.choice([z["window"], 256, 300, 700])
    layers = "".join(rng.choice("wa" if kind == "Binusun" else "lda") for _ in range(rng.randint(1, 3)))
    c = _seq(kind, call, layers, vocab=rng.choice([8192, 32000]), **z)
    if call == "prompt":
        n = rng.choice([1, 1, 2, 3, 5])
        return dict(c, lens=",".join(str(_log(rng, 9, 2048 // n)) for _ in range(n)))
    return dict(c, seqs=rng.choice([1, 1, 2, 4, 7]), prompt=_log(rng, 16, 1500), new=rng.randint(8, 40))


# ---- inputs: weights of the synthetic generator, tokens -------------------------------------------------------------------------
def _seed(seed, name):
    h = 1469598103934665603
    for b in name.encode():
        h = ((h ^ b) * 1099511628211) & _M
    return (h ^ (int(seed) * 0x9E3779B97F4A7C15)) & ((1 << 62) - 1)


def _tokens(seed, what, n, vocab):
    return [int(t) for t in np.random.default_rng([_seed(seed, what) & 0x7FFFFFFF, int(seed)]).integers(0, vocab, n)]


def _uniform(seed, shape, amp, offset=0.0):
    """The generator of both engines: uniform(-amp, amp) + offset from splitmix64(seed * odd constant + element index), in fp32."""
    def signed(v):
        v &= _M
        return v - (1 << 64) if v >> 63 else v

    def right(z, k):
        return (z >> k) & ((1 << (64 - k)) - 1)

    n = int(np.prod(shape))
    out = torch.empty(n, dtype=torch.float32, device="cuda")
    for a in range(0, n, 1 << 25):
        z = torch.arange(a, min(n, a + (1 << 25)), dtype=torch.int64, device="cuda") + signed(int(seed) * 0xD1342543DE82EF95 + 0x9E3779B97F4A7C15)
        z = (z ^ right(z, 30)) * signed(0xBF58476D1CE4E5B9)
        z = (z ^ right(z, 27)) * signed(0x94D049BB133111EB)
        z = z ^ right(z, 31)
        out[a:a + z.numel()] = (right(z, 40).to(torch.float32) * (2.0 / 16777216.0) - 1.0) * float(np.float32(amp))
    return (out + float(np.float32(offset))).reshape(shape)


def _llama_tensors(c):
    """name -> (shape, amplitude) of the projections ([in, out]) and the embedding table; the norms' gains are made apart"""
    H, I = c["hidden"], c["inter"]
    t = {"token_embeddings.weight": ((c["vocab"], H), 0.1), "lm_head.weight": ((H, c["vocab"]), H ** -0.5)}
    for i in range(c["layers"]):
        for s in "qkvo":
            t["layers.%d.attention.%s_proj.weight" % (i, s)] = ((H, H), H ** -0.5)
        t["layers.%d.mlp.up_proj.weight" % i] = ((H, I), H ** -0.5)
        t["layers.%d.mlp.gate_proj.weight" % i] = ((H, I), H ** -0.5)
        t["layers.%d.mlp.down_proj.weight" % i] = ((I, H), I ** -0.5)
    return t


def _llama_gains(c, seed):
    names = ["norm.weight"] + ["layers.%d.%s.weight" % (i, s) for i in range(c["layers"]) for s in ("attention_norm", "ffn_norm")]
    return {n: _uniform(_seed(seed, n), (c["hidden"],), 0.25, 1.0) for n in names}


def _seq_config(c):
    d, D = c["dim"], c["width"]
    rot = {"base": 10000.0, "dims": d // 2, "scaling": {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 8192}}
    heads = {"heads": c["heads"], "kv_heads": c["kv_heads"], "dim": d, "vdim": d, "mask": {"size": c["window"]}, "scale": d ** -0.5}
    mlp = {"kind": "dense", "ff": c["ff"]}
    if c["kind"] == "Binusun":
        part = {"a": {"type": "attention", "mixer": dict(heads, rot=rot), "mlp": mlp}, "w": {"type": "wkv", "mixer": {"heads": D // 64, "dim": 64}, "mlp": None}}
        cfg = {"architecture": "Binusun", "layers": [part[x] for x in c["layers"]], "norm": {"eps": 1e-5}, "logit_scale": 1.0}
        if c["loop"]:
            cfg["loop"] = {"start": 0, "stop": len(c["layers"]) - 1, "times": 2}
    else:
        part = {"a": {"type": "attention", "mixer": heads, "mlp": mlp},
                "l": {"type": "latent_attention", "mlp": mlp,
                      "mixer": {"heads": c["heads"], "dim": d, "vdim": d, "kv_rank": 256, "q_rank": 3 * D // 8, "scale": d ** -0.5}},
                "d": {"type": "delta", "mixer": {"heads": c["heads"], "kv_heads": max(1, c["heads"] // 2), "dim": d, "vdim": d, "conv": 4}, "mlp": mlp}}
        cfg = {"architecture": "Nubipel", "embedding": {"scale": math.sqrt(D)}, "layers": [part[x] for x in c["layers"]], "norm": {"eps": 1e-6},
               "logit_scale": 0.5, "logit_softcap": 30.0}
    return dict(cfg, vocab=c["vocab"], width=D)


def _seq_tensors(c):
    """name -> (shape, amplitude, offset, kept in bf16)"""
    cfg, D = _seq_config(c), c["width"]
    t = {}

    def mat(name, rows, cols):
        t[name] = ((rows, cols), math.sqrt(3.0 / cols), 0.0, True)

    def vec(name, shape, amp, offset):
        t[name] = (shape, amp, offset, False)

    binusun = c["kind"] == "Binusun"
    t["embed"] = ((c["vocab"], D), 1.0 if binusun else math.sqrt(3.0 / D), 0.0, True)
    if cfg.get("loop"):
        mat("loop.in", D, 2 * D)
    gain = () if binusun else (D,)
    for i, L in enumerate(cfg["layers"]):
        p, m = "l%d." % i, L["mixer"]
        H = m["heads"]
        vec(p + "norm1", gain, 0.25, 1.0)
        if binusun:
            vec(p + "norm1b", gain, 0.25, 1.0)
        p += "mix."
        if L["type"] == "wkv":
            C, R = H * m["dim"], 64
            for s in "rkvgw":
                vec(p + "mu." + s, (D,), 0.5, 0.5)
            for s in "rkvg":
                mat(p + s, C, D)
            mat(p + "w1", R, D)
            mat(p + "w2", C, R)
            vec(p + "w0", (C,), 1.0, -1.0)
            vec(p + "u", (H, m["dim"]), 1.0, 0.0)
            vec(p + "norm", (C,), 0.5, 1.0)
            mat(p + "o", D, C)
        elif L["type"] == "latent_attention":
            mat(p + "dq", m["q_rank"], D)
            vec(p + "dq.norm", (m["q_rank"],), 0.25, 1.0)
            mat(p + "uq", H * m["dim"], m["q_rank"])
            mat(p + "g", H * m["vdim"], D)
            mat(p + "dkv", m["kv_rank"], D)
            vec(p + "dkv.norm", (m["kv_rank"],), 0.25, 1.0)
            mat(p + "uk", H * m["dim"], m["kv_rank"])
            mat(p + "uv", H * m["vdim"], m["kv_rank"])
            mat(p + "o", D, H * m["vdim"])
        elif L["type"] == "delta":
            G = m["kv_heads"]
            for s, n in (("q", G * m["dim"]), ("k", G * m["dim"]), ("v", H * m["vdim"])):
                mat(p + s, n, D)
                vec(p + s + ".conv", (n, m["conv"]), 0.8, 0.0)
            for s in "ba":
                mat(p + s, H, D)
            vec(p + "A_log", (H,), 0.5, 0.0)
            vec(p + "dt_bias", (H,), 0.5, -3.0)
            vec(p + "norm", (m["vdim"],), 0.25, 1.0)
            mat(p + "g", H * m["vdim"], D)
            mat(p + "o", D, H * m["vdim"])
        else:
            mat(p + "q", H * m["dim"], D)
            mat(p + "k", m["kv_heads"] * m["dim"], D)
            mat(p + "v", m["kv_heads"] * m["vdim"], D)
            mat(p + "o", D, H * m["vdim"])
            if binusun:
                mat(p + "g", H, D)
            else:
                vec(p + "q.norm", (m["dim"],), 0.25, 1.0)
                vec(p + "k.norm", (m["dim"],), 0.25, 1.0)
                vec(p + "sink", (H,), 1.0, 0.0)
        p = "l%d." % i
        if L["mlp"]:
            if binusun:
                vec(p + "norm2", gain, 0.25, 1.0)
                vec(p + "norm2b", gain, 0.25, 1.0)
                mat(p + "mlp.gate", c["ff"], D)
            mat(p + "mlp.up", c["ff"], D)
            mat(p + "mlp.down", D, c["ff"])
    vec("final.norm", gain, 0.25, 1.0)
    if binusun:
        mat("head", c["vocab"], D)
    return t


# ---- one pass -------------------------------------------------------------------------------------------------------------------
class _State:
    """A loaded model and the tokens of the request; the model's memory goes back with the state."""

    def __init__(self, case, model):
        self.case, self.model = case, model

    def __del__(self):
        self.model.free()


def prepare(case, seed):
    c = case
    if c["kind"] == "llama":
        from turboinfer_b200 import capi
        capi.init(0)
        rows = c["prompt"] + c.get("new", 0)
        m = capi.Model(dict(vocab=c["vocab"], hidden=c["hidden"], layers=c["layers"], heads=c["heads"], inter=c["inter"]), capi.Q_INT4 if c["bits"] == 4 else capi.Q_INT8,
                       attn_mode=1, rope_mode=1, max_seq=rows + 8)
        s = _State(c, m)
        for name, (shape, amp) in _llama_tensors(c).items():
            m.set_tensor_synthetic(name, shape[0], shape[1], _seed(seed, name), amp)
        for name, g in _llama_gains(c, seed).items():
            m.set_tensor(name, g.cpu().numpy())
        m.finalize()
        n = c.get("batch", 1)
        s.prompt = _tokens(seed, "prompt", n * c["prompt"], c["vocab"])
        if c["call"] == "batch":
            s.prompt = [s.prompt[i * c["prompt"]:(i + 1) * c["prompt"]] for i in range(n)]
        return s
    from turboinfer_b200 import models, seq
    lens = [int(x) for x in c["lens"].split(",")] if c["call"] == "prompt" else [c["prompt"]] * c["seqs"]
    extra = c.get("new", 0)
    cfg, plan = _seq_config(c), _seq_tensors(c)
    room = sum((n + extra + 127) // 64 * 64 for n in lens)
    if c["kind"] == "Binusun":
        desc, layers = models.binusun_descs(cfg, seq.BF16, room, len(lens), {k: v[0] for k, v in plan.items()})
    else:
        desc, layers = models.nubipel_descs(cfg, seq.BF16, room, len(lens))
    m = seq.SeqModel(desc, layers)
    s = _State(c, m)
    for name, (shape, amp, offset, _) in plan.items():
        m.set_tensor_synthetic(name, shape, _seed(seed, name), amp, offset)
    m.finalize()
    s.prompts = [_tokens(seed, "prompt %d" % i, n, c["vocab"]) for i, n in enumerate(lens)]
    s.answers = [_tokens(seed, "answer %d" % i, extra, c["vocab"]) for i in range(len(lens))]
    return s


def run(state):
    c, m = state.case, state.model
    if c["call"] == "generate":
        m.reset()
        tokens, logits, _ = m.generate_greedy(state.prompt, c["new"], want_logits=True)
        return {"tokens": tokens, "logits": logits}
    if c["call"] == "prefill":
        return {"logits": m.prefill(state.prompt)}
    if c["call"] == "batch":
        tokens, logits, _ = m.generate_batch_greedy(state.prompt, c["new"], want_logits=True)
        return {"tokens": tokens, "logits": logits}
    ids = [m.open() for _ in state.prompts]
    out = [m.step(list(zip(ids, state.prompts)), [[len(p) - 1] for p in state.prompts])]
    for k in range(c.get("new", 0)):
        out.append(m.step([(i, [a[k]]) for i, a in zip(ids, state.answers)], [[0]] * len(ids)))
    for i in ids:
        m.close(i)
    return {"logits": np.stack(out)}


# ---- what a pass cannot do without ------------------------------------------------------------------------------------------------
def _positions(c):
    """(first position, rows) of every forward step of a pass, for every sequence"""
    if c["kind"] == "llama":
        n, new = c["prompt"], c.get("new", 0)
        return [[(0, n)] * c.get("batch", 1)] + [[(n + k, 1)] * c.get("batch", 1) for k in range(new - 1)]
    if c["call"] == "prompt":
        return [[(0, int(x)) for x in c["lens"].split(",")]]
    return [[(0, c["prompt"])] * c["seqs"]] + [[(c["prompt"] + k, 1)] * c["seqs"] for k in range(c["new"])]


def work(case):
    """Every step reads each weight once, the embedding rows it needs, the cache or state behind it, writes what it adds and the wanted
    rows' logits; two operations a weight and row (the head: wanted rows only), and the mixers' own products over visible keys or states."""
    c = case
    nbytes = flops = 0.0
    if c["kind"] == "llama":
        H, per, V = c["hidden"], 4 * c["hidden"] ** 2 + 3 * c["hidden"] * c["inter"], c["vocab"]
        for step in _positions(c):
            rows = sum(n for _, n in step)
            nbytes += (c["layers"] * per + H * V) * c["bits"] / 8 + rows * H * 4 + len(step) * V * 4
            flops += 2.0 * c["layers"] * per * rows + 2.0 * H * V * len(step)
            for p, n in step:
                nbytes += c["layers"] * 2 * H * 4 * (p + n)
                flops += c["layers"] * 4.0 * H * (n * p + n * (n + 1) / 2)
        return {"bytes": nbytes, "flops": flops}
    cfg, D, V = _seq_config(c), c["width"], c["vocab"]
    n = len(cfg["layers"])
    runs = list(range(n - 1)) * 2 + [n - 1] if cfg.get("loop") else list(range(n))
    sizes = {}
    for name, (shape, _, _, bf) in _seq_tensors(c).items():
        if bf and name[0] == "l" and name[1].isdigit():
            i = int(name[1:name.index(".")])
            sizes[i] = sizes.get(i, 0) + shape[0] * shape[1]
    once = sum(sizes.values()) + V * D + (2 * D * D if cfg.get("loop") else 0)
    for step in _positions(c):
        rows = sum(k for _, k in step)
        nbytes += once * 2 + rows * D * 2 + len(step) * V * 4
        flops += 2.0 * V * D * len(step) + (2 * 2.0 * 2 * D * D * rows if cfg.get("loop") else 0)
        for i in runs:
            L, m = cfg["layers"][i], cfg["layers"][i]["mixer"]
            H, d, dv = m["heads"], m["dim"], m.get("vdim", m["dim"])
            flops += 2.0 * sizes[i] * rows
            for p, k in step:
                if L["type"] in ("wkv", "delta"):
                    nbytes += 8.0 * H * d * dv
                    flops += (6.0 if L["type"] == "wkv" else 8.0) * H * d * dv * k
                    continue
                pos = np.arange(p, p + k)
                size = m["mask"]["size"] if m.get("mask") else 0
                seen = pos + 1 if not size else np.minimum(pos + 1, size) if c["kind"] == "Binusun" else pos % size + 1
                flops += 2.0 * H * (d + dv) * float(seen.sum())
                reach = p + k - max(0, p + 1 - size) if size and c["kind"] == "Binusun" else p + k - (p // size * size if size else 0)
                nbytes += 4.0 * (m["kv_rank"] if L["type"] == "latent_attention" else m["kv_heads"] * (d + dv)) * reach
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """llama: integer products of 24-bit activations are exact, fp32 sums around them (norm, softmax, attention) move the logits by
    about 1e-6 (measured against 64 bits: 4e-7 to 1.2e-6); a token differs only where two logits tie within that.  Layered engine:
    products of bf16-rounded rows with fp32 sums; a changed order of sums flips single roundings of the next product's rows.  Against 64
    bits: 0.012 after the seven layer runs of the looped model, 0.003 to 0.006 after one to three layers."""
    if case["kind"] == "llama":
        return {"rel": 1e-5, "max": 1e-4, "differ": 0.0}
    return {"rel": 0.03 if case["loop"] else 0.02, "max": 0.3}


# ---- the same in 64 bits ------------------------------------------------------------------------------------------------------------
def _norm(x, w, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _turn(x, angles):
    """coordinates (2i, 2i + 1) of the leading ones turned by angles [rows, i]; x [..., rows, heads, d]"""
    n = angles.shape[-1]
    c, s = torch.cos(angles)[:, None, :], torch.sin(angles)[:, None, :]
    y = x.clone()
    a, b = x[..., 0:2 * n:2], x[..., 1:2 * n:2]
    y[..., 0:2 * n:2], y[..., 1:2 * n:2] = a * c - b * s, a * s + b * c
    return y


def _angles(freq, first, rows):
    """position times frequency: both are fp32 numbers of the model, and so is their product"""
    return (torch.arange(first, first + rows, device="cuda", dtype=torch.float32)[:, None] * torch.as_tensor(freq, device="cuda", dtype=torch.float32)[None, :]).double()


def _llama_exact(c, seed):
    top = np.float32(127.0 if c["bits"] == 8 else 7.0)
    W = {}
    for name, (shape, amp) in _llama_tensors(c).items():
        w = _uniform(_seed(seed, name), shape, amp)
        if not name.startswith("token"):
            scale = w.abs().max() / torch.tensor(float(top), device="cuda")   # symmetric, one scale a tensor, fp32 as stored
            q = w / scale                                            # (tensor by tensor: a Python divisor would become a rounded reciprocal)
            q = torch.sign(q) * torch.floor(q.abs().double() + 0.5)  # halves away from zero
            w = q.clamp(-128.0 if c["bits"] == 8 else -7.0, float(top)) * scale.double()
        W[name] = w.double()
        del w
    W.update({k: v.double() for k, v in _llama_gains(c, seed).items()})
    H, heads = c["hidden"], c["heads"]
    d = H // heads
    freq = (np.float32(1.0) / np.power(np.float64(10000.0), np.float64(np.arange(0, d, 2, dtype=np.float32) / np.float32(d))).astype(np.float32)).astype(np.float32)
    cache = [[] for _ in range(c["layers"])]

    def forward(tokens, first):   # tokens [B, n] -> logits of the last position [B, V]
        B, n = tokens.shape
        x = W["token_embeddings.weight"][tokens]
        ang = _angles(freq, first, n)
        for i in range(c["layers"]):
            p = "layers.%d." % i
            h = _norm(x, W[p + "attention_norm.weight"], 1e-5)
            q, k, v = (((h @ W[p + "attention.%s_proj.weight" % s]).reshape(B, n, heads, d)) for s in "qkv")
            q, k = _turn(q, ang), _turn(k, ang)
            cache[i] = [k, v] if not first else [torch.cat([cache[i][0], k], 1), torch.cat([cache[i][1], v], 1)]
            K, Vv = cache[i]
            o = torch.empty_like(q)
            future = torch.arange(K.shape[1], device="cuda")[None, :] > torch.arange(first, first + n, device="cuda")[:, None]
            for j in range(heads):
                s = (q[:, :, j] @ K[:, :, j].transpose(1, 2)) / math.sqrt(d)
                o[:, :, j] = torch.softmax(s.masked_fill(future, -math.inf), -1) @ Vv[:, :, j]
            x = x + o.reshape(B, n, H) @ W[p + "attention.o_proj.weight"]
            h = _norm(x, W[p + "ffn_norm.weight"], 1e-5)
            x = x + ((h @ W[p + "mlp.up_proj.weight"]) * torch.nn.functional.silu(h @ W[p + "mlp.gate_proj.weight"])) @ W[p + "mlp.down_proj.weight"]
        return _norm(x[:, -1], W["norm.weight"], 1e-5) @ W["lm_head.weight"]

    n = c.get("batch", 1)
    t = torch.tensor(_tokens(seed, "prompt", n * c["prompt"], c["vocab"]), device="cuda").reshape(n, c["prompt"])
    logits = [forward(t, 0)]
    tokens = []
    for k in range(c.get("new", 0)):
        tokens.append(logits[-1].argmax(-1))
        if k + 1 < c["new"]:
            logits.append(forward(tokens[-1][:, None], c["prompt"] + k))
    if c["call"] == "prefill":
        return {"logits": logits[0][0]}
    if c["call"] == "generate":
        return {"tokens": torch.stack(tokens, 1)[0].int(), "logits": torch.stack(logits)[:, 0]}
    return {"tokens": torch.stack(tokens, 1).int(), "logits": logits[-1]}


def _rotary(rot):
    f = np.array([rot["base"] ** (-2.0 * i / rot["dims"]) for i in range(rot["dims"] // 2)])
    z = rot["scaling"]
    wl = 2.0 * math.pi / f
    s = (z["original"] / wl - z["low"]) / (z["high"] - z["low"])
    mid = (1.0 - s) * f / z["factor"] + s * f
    return np.where(wl > z["original"] / z["low"], f / z["factor"], np.where(wl < z["original"] / z["high"], f, mid)).astype(np.float32)


def _attend(q, k, v, scale, seen, sink=None):
    """q [n, H, d], k / v [n, G, .]: softmax over the seen keys, head by head; sink: one more term of the denominator"""
    H, G = q.shape[1], k.shape[1]
    out = torch.empty(q.shape[0], H, v.shape[2], dtype=torch.float64, device="cuda")
    for h in range(H):
        s = (q[:, h] @ k[:, h * G // H].T * scale).masked_fill(~seen, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[h].expand(len(s), 1)], 1)
        out[:, h] = torch.softmax(s, -1)[:, :len(k)] @ v[:, h * G // H]
    return out


def _mixer_exact(kind, L, W, h, eps):
    """h [n, width] -> the mixer's result; W: name without its prefix -> tensor"""
    m, n = L["mixer"], len(h)
    H, d = m["heads"], m["dim"]
    i = torch.arange(n, device="cuda")
    causal = i[None, :] <= i[:, None]

    def heads(x, k=H):
        return x.reshape(n, k, -1)

    if L["type"] == "attention":
        G = m["kv_heads"]
        q, k, v = heads(h @ W["q"].T), heads(h @ W["k"].T, G), heads(h @ W["v"].T, G)
        if kind == "Binusun":
            ang = _angles(_rotary(m["rot"]), 0, n)
            q, k = _norm(_turn(q, ang), 1.0, eps), _norm(_turn(k, ang), 1.0, eps)
            o = _attend(q, k, v, m["scale"], causal & (i[:, None] - i[None, :] < m["mask"]["size"])) * torch.sigmoid(h @ W["g"].T)[:, :, None]
        else:
            chunk = i // m["mask"]["size"]
            o = _attend(_norm(q, W["q.norm"], eps), _norm(k, W["k.norm"], eps), v, m["scale"], causal & (chunk[:, None] == chunk[None, :]), W["sink"])
    elif L["type"] == "latent_attention":
        z = _norm(h @ W["dkv"].T, W["dkv.norm"], eps)
        o = _attend(heads(_norm(h @ W["dq"].T, W["dq.norm"], eps) @ W["uq"].T), heads(z @ W["uk"].T), heads(z @ W["uv"].T), m["scale"], causal)
        o = o * torch.sigmoid(heads(h @ W["g"].T))
    elif L["type"] == "wkv":
        before = torch.cat([torch.zeros_like(h[:1]), h[:-1]])
        mix = {s: h + (before - h) * W["mu." + s] for s in "rkvgw"}
        r, k, v = (heads(mix[s] @ W[s].T) for s in "rkv")
        decay = heads(torch.exp(-torch.exp(torch.tanh(mix["w"] @ W["w1"].T) @ W["w2"].T + W["w0"])))
        S = torch.zeros(H, d, d, dtype=torch.float64, device="cuda")
        o = torch.empty_like(v)
        for t in range(n):
            kv = k[t][:, :, None] * v[t][:, None, :]
            o[t] = ((S + W["u"][:, :, None] * kv) * r[t][:, :, None]).sum(1)
            S = decay[t][:, :, None] * S + kv
        return (_norm(o, 1.0, eps).reshape(n, -1) * W["norm"] * torch.nn.functional.silu(mix["g"] @ W["g"].T)) @ W["o"].T
    else:
        G = m["kv_heads"]

        def branch(s, count):
            x, w = h @ W[s].T, W[s + ".conv"]
            y = sum(w[:, w.shape[1] - 1 - j] * torch.cat([torch.zeros_like(x[:j]), x[:n - j]]) for j in range(min(n, w.shape[1])))
            return torch.nn.functional.silu(y).reshape(n, count, -1)

        def unit(x):
            return x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6)

        q, k, v = branch("q", G), branch("k", G), branch("v", H)
        q, k = unit(q).repeat_interleave(H // G, 1) * d ** -0.5, unit(k).repeat_interleave(H // G, 1)
        decay = torch.exp(-torch.exp(W["A_log"]) * torch.nn.functional.softplus(h @ W["a"].T + W["dt_bias"]))
        beta = torch.sigmoid(h @ W["b"].T)
        S = torch.zeros(H, d, v.shape[2], dtype=torch.float64, device="cuda")
        o = torch.empty_like(v)
        for t in range(n):
            S = decay[t][:, None, None] * S
            u = beta[t][:, None] * (v[t] - (S * k[t][:, :, None]).sum(1))
            S = S + k[t][:, :, None] * u[:, None, :]
            o[t] = (S * q[t][:, :, None]).sum(1)
        o = _norm(o, W["norm"], eps) * torch.nn.functional.silu(heads(h @ W["g"].T))
    return o.reshape(n, -1) @ W["o"].T


def _seq_exact(c, seed):
    cfg = _seq_config(c)
    eps, binusun = cfg["norm"]["eps"], c["kind"] == "Binusun"
    W = {}
    for name, (shape, amp, offset, bf) in _seq_tensors(c).items():
        w = _uniform(_seed(seed, name), shape, amp, offset)
        W[name] = (w.bfloat16() if bf else w).double()
    n = len(cfg["layers"])
    runs = [(i, False) for i in range(n)]
    if cfg.get("loop"):
        runs = [(i, i == 0) for i in range(n - 1)] * 2 + [(n - 1, False)]
    lens = [int(x) for x in c["lens"].split(",")] if c["call"] == "prompt" else [c["prompt"]] * c["seqs"]
    new = c.get("new", 0)
    out = []
    for j, rows in enumerate(lens):
        t = torch.tensor(_tokens(seed, "prompt %d" % j, rows, c["vocab"]) + _tokens(seed, "answer %d" % j, new, c["vocab"]), device="cuda")
        x0 = W["embed"][t]
        x = x0 if binusun else x0 * float(np.float32(cfg["embedding"]["scale"]))
        for i, enters in runs:
            L, p = cfg["layers"][i], "l%d." % i
            mw = {k[len(p) + 4:]: v for k, v in W.items() if k.startswith(p + "mix.")}
            if enters:
                x = torch.cat([x, x0], -1) @ W["loop.in"].T
            h = _norm(x, W[p + "norm1"], eps)
            y = _mixer_exact(c["kind"], L, mw, h, eps)
            if binusun:
                x = x + _norm(y, W[p + "norm1b"], eps)
                if L["mlp"]:
                    h = _norm(x, W[p + "norm2"], eps)
                    x = x + _norm((torch.relu(h @ W[p + "mlp.gate"].T) * (h @ W[p + "mlp.up"].T)) @ W[p + "mlp.down"].T, W[p + "norm2b"], eps)
            else:
                x = x + y + torch.nn.functional.gelu(h @ W[p + "mlp.up"].T) @ W[p + "mlp.down"].T
        z = _norm(x[rows - 1:], W["final.norm"], eps)
        out.append(z @ W["head"].T if binusun else 30.0 * torch.tanh(z @ W["embed"].T * 0.5 / 30.0))
    return {"logits": torch.stack(out, 1)}


def exact(case, seed):
    return _llama_exact(case, seed) if case["kind"] == "llama" else _seq_exact(case, seed)
