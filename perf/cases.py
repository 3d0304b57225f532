"""The work that is measured: single products, attention calls and whole decoders, through the public entry points.

A case is a dict of sizes. `listed()` names the fixed ones, `draw(rng)` gives more of the same ranges, `prepare` builds what a
program holds before the call, `run` is one pass, `exact` the same outputs in 64 bits from plain torch. Sizes are those of a
Llama-3-8B-shaped decoder, of the repository's dense token-mixer decoders, or generic ones around them. Weights and inputs
are random, with the spreads of trained layers; the output head of a decoder repeats its embedding rows one place on, so that
the next token is as clear as a trained model's mostly is and the same for every correct implementation.
"""
import math
import zlib

import numpy as np
import torch

import kalosm_b200 as kb
from kalosm_b200 import koludra, sofudra, synth

BLOCK = {kb.Q4_0: (32, 18), kb.Q8_0: (32, 34), kb.Q4_K: (256, 144), kb.Q6_K: (256, 210)}
TYPES = {"q4_0": kb.Q4_0, "q8_0": kb.Q8_0, "q4_k": kb.Q4_K, "q6_k": kb.Q6_K}
EPILOGUES = {"none": kb.EPI_NONE, "residual": kb.EPI_RESIDUAL, "swiglu": kb.EPI_SWIGLU}
EPS = 1e-5
THETA = 500000.0
LLAMA_8B = dict(kind="llama", layers=32, width=4096, ffn=14336, heads=32, kv_heads=8, dim=128, vocab=128256, weights="q4_k_m")
KOLUDRA = dict(kind="koludra", width=2048, ffn=8192, layers=10, window=1024, vocab=32768, compute="bfloat16")
SOFUDRA = dict(kind="sofudra", width=2048, ffn=8192, layers=10, window=1024, vocab=32768, compute="bfloat16")


def listed():
    return [
        # one projection of one activation row: the smallest call, where latency counts
        dict(name="row_4096x4096_q4_0", kind="product", rows=1, n=4096, k=4096, type="q4_0", epilogue="none"),
        # the down projection of a few sequences (speculation, small batches), residual added
        dict(name="rows8_4096x14336_q6_k", kind="product", rows=8, n=4096, k=14336, type="q6_k", epilogue="residual"),
        # the gate / up projection of a long prompt
        dict(name="rows2048_28672x4096_q4_k", kind="product", rows=2048, n=28672, k=4096, type="q4_k", epilogue="swiglu"),
        # one new position of a few sequences against their caches, at an odd length
        dict(name="attention_decode_b5_3333", kind="attention", batch=5, heads=32, kv_heads=8, dim=128, queries=1, keys=3333),
        # causal attention of a prompt
        dict(name="attention_prompt_2048", kind="attention", batch=1, heads=32, kv_heads=8, dim=128, queries=2048, keys=2048),
        # the headline model: prompt, one sequence, sixteen sequences
        dict(LLAMA_8B, name="llama_8b_prompt_512", phase="prompt", batch=1, prompt=512, steps=0, sampled=False),
        dict(LLAMA_8B, name="llama_8b_decode_b1", phase="decode", batch=1, prompt=512, steps=16, sampled=False),
        dict(LLAMA_8B, name="llama_8b_decode_b16", phase="decode", batch=16, prompt=300, steps=8, sampled=False),
        # a long prompt and a short request of the delta-rule / latent-attention decoder
        dict(KOLUDRA, name="koludra_prompt_8192", phase="prompt", batch=1, prompt=8192, steps=0),
        dict(KOLUDRA, name="koludra_request_40_32", phase="decode", batch=1, prompt=40, steps=32),
        # an odd prompt and a short request of the looped attention / linear-attention decoder
        dict(SOFUDRA, name="sofudra_prompt_1111", phase="prompt", batch=1, prompt=1111, steps=0),
        dict(SOFUDRA, name="sofudra_request_100_32", phase="decode", batch=1, prompt=100, steps=32),
    ]


def _log(rng, lo, hi, step=1):
    """A size between lo and hi, evenly spread over its logarithm, a multiple of `step`."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(lo, min(hi, int(round(v / step)) * step))


def draw(rng):
    kind = rng.choice(["product", "product", "product", "attention", "attention", "llama", "llama", "koludra", "sofudra"])
    if kind == "product":
        t, e = rng.choice(sorted(TYPES)), rng.choice(sorted(EPILOGUES))
        n = _log(rng, 256, 28672, 32 if e == "swiglu" else 1)
        return dict(kind=kind, rows=rng.choice([1, _log(rng, 2, 32), _log(rng, 33, 2048)]), n=n, k=_log(rng, 512, 14336, 256), type=t, epilogue=e)
    if kind == "attention":
        heads, kv = rng.choice([(32, 8), (16, 4), (16, 16), (24, 8), (40, 8)])
        dim = rng.choice([64, 128])
        if rng.random() < 0.5:
            return dict(kind=kind, batch=_log(rng, 1, 32), heads=heads, kv_heads=kv, dim=dim, queries=1, keys=_log(rng, 64, 8192))
        q = _log(rng, 33, 3000)
        return dict(kind=kind, batch=1, heads=heads, kv_heads=kv, dim=dim, queries=q, keys=q + rng.choice([0, 0, _log(rng, 1, 2000)]))
    if kind == "llama":
        dim = rng.choice([64, 128])
        kv = rng.choice([2, 4, 8])
        heads = kv * rng.choice([1, 2, 4])
        c = dict(kind=kind, layers=rng.randint(2, 6), width=_log(rng, 1024, 4096, 256), ffn=_log(rng, 2048, 14336, 256), heads=heads, kv_heads=kv,
                 dim=dim, vocab=_log(rng, 16000, 64000), weights=rng.choice(["q4_k_m", "q4_k_m", "q8_0", "q4_0"]))
        if rng.random() < 0.4:
            return dict(c, phase="prompt", batch=rng.choice([1, 1, 2]), prompt=_log(rng, 9, 2048), steps=0, sampled=False)
        return dict(c, phase="decode", batch=rng.choice([1, _log(rng, 2, 32)]), prompt=_log(rng, 4, 1024), steps=rng.randint(4, 16), sampled=rng.random() < 0.3)
    c = dict(kind=kind, width=rng.choice([1024, 2048, 4096]), ffn=_log(rng, 2048, 12288, 64), layers=rng.randint(4, 8), window=_log(rng, 128, 2048),
             vocab=_log(rng, 8000, 40000), compute="bfloat16")
    if rng.random() < 0.5:
        return dict(c, phase="prompt", batch=1, prompt=_log(rng, 17, 4096), steps=0)
    return dict(c, phase="decode", batch=rng.choice([1, 1, 4]), prompt=_log(rng, 5, 200), steps=rng.randint(8, 32))


# ---- inputs -------------------------------------------------------------------------------------------------------------

def _gen(seed, name):
    return torch.Generator(device="cuda").manual_seed((int(seed) * 1000003 + zlib.crc32(name.encode())) % (1 << 62))


def _normal(seed, name, shape, sigma=1.0):
    return torch.randn(shape, generator=_gen(seed, name), device="cuda", dtype=torch.float32) * sigma


_held = {}


def _device():
    """The program's one handle."""
    if "device" not in _held:
        _held["device"] = kb.Device(0)
    return _held["device"]


def _host(t):
    """The bytes of a device tensor in a pinned buffer that every load reuses."""
    t = t.contiguous().view(torch.uint8).reshape(-1)
    if "pinned" not in _held or _held["pinned"].numel() < t.numel():
        _held["pinned"] = torch.empty(max(t.numel(), 1 << 26), dtype=torch.uint8, pin_memory=True)
    b = _held["pinned"][: t.numel()]
    b.copy_(t)
    return b.numpy()


def _tensor(t):
    """A framework tensor over a torch tensor's memory."""
    return kb.Tensor(_device(), t.shape, str(t.dtype).split(".")[1], ptr=t.data_ptr())


def _blocks(seed, name, n, k, sigma, ggml_type):
    """Raw blocks of an [n, k] matrix, on the GPU; long ones in portions of rows."""
    g = _gen(seed, name)
    parts = [synth.quantize(torch.randn((min(16384, n - r), k), generator=g, device="cuda") * sigma, ggml_type) for r in range(0, n, 16384)]
    return parts[0] if len(parts) == 1 else torch.cat(parts)


# the spread of the residual projections shrinks with depth, as initialisations of deep decoders have it
def _llama_plan(c):
    e, q, kv, f = c["width"], c["heads"] * c["dim"], c["kv_heads"] * c["dim"], c["ffn"]
    body, high = {"q4_k_m": (kb.Q4_K, kb.Q6_K), "q8_0": (kb.Q8_0, kb.Q8_0), "q4_0": (kb.Q4_0, kb.Q8_0)}[c["weights"]]
    s = 1.28 * e ** -0.5
    out = s * (2 * c["layers"]) ** -0.5
    plan = []
    for i in range(c["layers"]):
        plan += [("attn_q", i, body, q, e, s), ("attn_k", i, body, kv, e, s), ("attn_v", i, high, kv, e, s), ("attn_output", i, body, e, q, out),
                 ("ffn_gate", i, body, f, e, s), ("ffn_up", i, body, f, e, s), ("ffn_down", i, high, e, f, out)]
    return plan, body, high


def _llama_ends(c, seed, which):
    """Raw blocks of the embedding, or of the head: row j of the head is like row j - 1 of the embedding."""
    _, body, high = _llama_plan(c)
    g = _gen(seed, "embd")
    w = torch.randn((c["vocab"], c["width"]), generator=g, device="cuda")
    if which == "output":
        w = torch.roll(w, 1, 0).mul_(1.28 * c["width"] ** -0.5)
    t = body if which == "token_embd" else high
    return t, torch.cat([synth.quantize(p, t) for p in w.split(16384)])


def _llama_norm(seed, name, i, e):
    return 1.0 + _normal(seed, f"{name}{i}", (e,), 0.02)


def _llama_model(c, seed):
    m = kb.Llama(_device(), n_layer=c["layers"], hidden=c["width"], ffn=c["ffn"], n_head=c["heads"], n_kv_head=c["kv_heads"], head_dim=c["dim"],
                 vocab=c["vocab"], max_seq_len=_context(c), max_batch=c["batch"], rms_eps=EPS, rope_theta=THETA)
    for which in ("token_embd", "output"):
        t, raw = _llama_ends(c, seed, which)
        m.set_tensor(which, -1, t, (c["vocab"], c["width"]), _host(raw))
    for name, i, t, n, k, s in _llama_plan(c)[0]:
        m.set_tensor(name, i, t, (n, k), _host(_blocks(seed, f"{name}{i}", n, k, s, t)))
    for i in range(c["layers"]):
        for name in ("attn_norm", "ffn_norm"):
            m.set_tensor(name, i, kb.F32, (c["width"],), _host(_llama_norm(seed, name, i, c["width"])))
    m.set_tensor("output_norm", -1, kb.F32, (c["width"],), _host(_llama_norm(seed, "output_norm", 0, c["width"])))
    return m


def _context(c):
    return max(256, (c["prompt"] + c["steps"] + 127) // 128 * 128)


def _koludra_config(c):
    """128-wide heads, 512-wide latents, three delta rules to two attentions, every second attention reads the first one's rows."""
    h, mlp = c["width"] // 128, {"kind": "dense", "ff": c["ffn"]}
    d = {"type": "delta", "mixer": dict(heads=h, kv_heads=h // 2, dim=128, vdim=128, conv=4), "mlp": mlp}
    d2 = {"type": "delta_2", "mixer": dict(heads=h, kv_heads=h, dim=128, vdim=128, conv=4), "mlp": mlp}
    a = {"type": "latent_attention", "mlp": mlp, "mixer": dict(heads=h, dim=128, rot_dim=64, vdim=128, kv_rank=512, mask={"size": c["window"]},
                                                               rot={"base": THETA, "dims": 64}, scale=192 ** -0.5)}
    shared = dict(a, mixer=dict(a["mixer"], kv_from=1))
    return {"architecture": "Koludra", "layers": [(d, a, d2, d, shared)[i % 5] for i in range(c["layers"])], "norm": {"eps": EPS},
            "vocab": c["vocab"], "width": c["width"]}


def _sofudra_config(c):
    """128-wide heads, four query heads to a key head; two of the layers run twice."""
    h, mlp = c["width"] // 128, {"kind": "dense", "ff": c["ffn"]}
    att = dict(heads=h, kv_heads=h // 4, dim=128, vdim=128, scale=128 ** -0.5)
    a = {"type": "attention", "mlp": mlp, "mixer": dict(att, mask={"size": c["window"]}, rot={
        "base": THETA, "dims": 128, "scaling": {"factor": 8.0, "original": 4096, "fast": 32.0, "slow": 1.0}})}
    p = {"type": "parallel", "mlp": mlp, "mixer": dict(left_scale=0.7, right_scale=0.8, left=dict(att, softcap=50.0), right=dict(
        heads=h, dim=128, vdim=128, decay=[1.0 - 2.0 ** -(1 + 7.0 * i / h) for i in range(h)]))}
    return {"architecture": "Sofudra", "embedding": {"scale": c["width"] ** 0.5}, "layers": [(p, a)[i % 2] for i in range(c["layers"] - 2)],
            "logit_softcap": 30.0, "loop": dict(times=2, **({"start": 2, "stop": 4} if c["layers"] >= 6 else {"start": 0, "stop": 2})), "norm": {"eps": EPS}, "residual_mult": 0.5, "vocab": c["vocab"],
            "width": c["width"]}


def _mixer_rows(mx, linear):
    h, d, v = mx["heads"], mx["dim"], mx["vdim"]
    g = mx.get("kv_heads", h)
    return {"q": h * d, "k": g * d, "v": g * v, "g": h * v if linear else h}


def _dense_shape(cfg, name):
    width, vocab = cfg["width"], cfg["vocab"]
    if name in ("embed", "head", "final.norm", "loop.in"):
        return {"embed": (vocab, width), "head": (vocab, width), "final.norm": (width,), "loop.in": (width, 2 * width)}[name]
    layer, part = name.split(".", 1)
    L = cfg["layers"][int(layer[1:])]
    mx = L["mixer"]
    if part.startswith("norm"):
        return (width,)
    if part.startswith("mlp."):
        return (width, L["mlp"]["ff"]) if part == "mlp.down" else (L["mlp"]["ff"], width)
    part = part[4:]
    if L["type"].startswith("delta"):
        h, hv, qk = mx["heads"], mx["heads"] * mx["vdim"], mx["kv_heads"] * mx["dim"]
        rows = {"q": qk, "k": qk, "v": hv, "g": hv, "b": h, "a": h}
        if part.endswith(".conv"):
            return (rows[part[0]], mx["conv"])
        return {"o": (width, hv), "A_log": (h,), "dt_bias": (h,), "norm": (mx["vdim"],)}.get(part) or (rows[part], width)
    if L["type"] == "latent_attention":
        h, r = mx["heads"], mx["kv_rank"]
        return {"q": (h * (mx["dim"] + mx["rot_dim"]), width), "g": (h, width), "o": (width, h * mx["vdim"]), "uk": (h * mx["dim"], r),
                "uv": (h * mx["vdim"], r), "dkv": (r + mx["rot_dim"], width), "dkv.norm": (r,)}[part]
    linear = part.startswith("right.")
    if L["type"] == "parallel":
        side, part = part.split(".", 1)
        mx = mx[side]
    rows = _mixer_rows(mx, linear)
    if part.endswith(".b"):
        return (rows[part[0]],)
    if part.endswith(".norm"):
        return (mx["dim"],)
    return {"o": (width, mx["heads"] * mx["vdim"]), "norm": (mx["heads"] * mx["vdim"],), "sink": (mx["heads"],)}.get(part) or (rows[part], width)


def _dense_weight(cfg, seed, name):
    """One tensor of a dense decoder, as bf16."""
    shape = _dense_shape(cfg, name)
    if name == "head":
        w = torch.roll(_normal(seed, "embed", shape), 1, 0) * shape[1] ** -0.5
    elif name == "embed":
        w = _normal(seed, "embed", shape) / (cfg.get("embedding", {}).get("scale", 1.0))
    elif name == "loop.in":  # close to an average of its two inputs
        eye = torch.eye(shape[0], device="cuda")
        w = _normal(seed, name, shape, 0.3 * shape[1] ** -0.5) + 0.6 * torch.cat([eye, eye], 1)
    else:
        w = _normal(seed, name, shape)
        if len(shape) == 1:
            w = 1.0 + 0.1 * w if "norm" in name else 0.5 * w - 1.0 if name.endswith(("A_log", "dt_bias")) else 0.2 * w
        else:
            w *= 0.3 if name.endswith(".conv") else shape[1] ** -0.5
    return w.to(torch.bfloat16)


def _dense_model(c, seed):
    arch, cfg = (koludra, _koludra_config(c)) if c["kind"] == "koludra" else (sofudra, _sofudra_config(c))

    def tensor(name):
        return kb.BF16, _dense_shape(cfg, name), _host(_dense_weight(cfg, seed, name))
    return arch.build(_device(), cfg, tensor, _context(c), c["batch"], c["compute"])


def _prompt(c, seed):
    return np.random.default_rng(seed).integers(0, c["vocab"], size=(c["batch"], c["prompt"] + (c["phase"] == "decode")), dtype=np.uint32)


def prepare(case, seed):
    c = case
    if c["kind"] == "product":
        t, e = TYPES[c["type"]], c["epilogue"]
        n_out = c["n"] // 2 if e == "swiglu" else c["n"]
        w = kb.QMatrix.from_raw_bytes(_device(), (c["n"], c["k"]), _host(_blocks(seed, "w", c["n"], c["k"], 0.02, t)), t)
        x = _normal(seed, "x", (c["rows"], c["k"]))
        r = [_normal(seed, f"r{i}", (c["rows"], n_out)) for i in range(2)] if e == "residual" else []
        y = torch.empty((c["rows"], n_out), device="cuda")
        return dict(case=c, w=w, kept=(x, r), x=_tensor(x), r=[_tensor(v) for v in r], out=y, y=_tensor(y))
    if c["kind"] == "attention":
        q = _normal(seed, "q", (c["batch"], c["heads"], c["queries"], c["dim"]))
        k, v = (_normal(seed, n, (c["batch"], c["kv_heads"], c["keys"], c["dim"])).half() for n in ("k", "v"))
        y = torch.empty_like(q)
        return dict(case=c, kept=(q, k, v), q=_tensor(q), k=_tensor(k), v=_tensor(v), out=y, y=_tensor(y))
    m = _llama_model(c, seed) if c["kind"] == "llama" else _dense_model(c, seed)
    tokens = _prompt(c, seed)
    if c["kind"] == "llama" and c["phase"] == "decode":
        m.forward(tokens[:, :-1], want_logits=False)
    sampler = kb.SamplerConfig(temperature=0.8, top_k=64, top_p=0.95, seed=seed) if c.get("sampled") else None
    return dict(case=c, model=m, tokens=tokens, sampler=sampler)


def run(state):
    c = state["case"]
    if c["kind"] == "product":
        r = state["r"]
        state["x"].q_mat_mul(state["w"], EPILOGUES[c["epilogue"]], *r, out=state["y"])
        return state["out"]
    if c["kind"] == "attention":
        _device().flash_attention(state["q"], state["k"], state["v"], c["dim"] ** -0.5,
                                  mask_kind=kb.MASK_CAUSAL if c["queries"] > 1 else kb.MASK_NONE, out=state["y"])
        return state["out"]
    m, tokens = state["model"], state["tokens"]
    if c["phase"] == "prompt":  # a new session: the prompt's logits and the next token
        m.reset()
        logits, ids = m.forward(tokens)
        return {"logits": logits, "ids": ids}
    # tokens generated on the device, then the logits of one step more; a Llama session is taken back to the end of its
    # prompt, the sessions of the others (recurrent states cannot be rewound) start with theirs
    if c["kind"] == "llama":
        m.truncate(c["prompt"])
    else:
        m.reset()
        m.forward(tokens[:, :-1], want_logits=False)
    if state["sampler"] is not None:
        ids = m.generate_sampled(tokens[:, -1], c["steps"] - 1, state["sampler"])
    else:
        ids = m.generate_greedy(tokens[:, -1], c["steps"] - 1)
    logits, last = m.forward(ids[:, -1:])
    return {"logits": logits, "ids": ids, "last": last}


# ---- what a pass cannot do without ---------------------------------------------------------------------------------------

def _size(n, k, t):
    be, bb = BLOCK[t]
    return n * (k // be) * bb


def work(case):
    c = case
    if c["kind"] == "product":
        n_out = c["n"] // 2 if c["epilogue"] == "swiglu" else c["n"]
        return {"bytes": _size(c["n"], c["k"], TYPES[c["type"]]) + 4 * c["rows"] * (c["k"] + n_out * (3 if c["epilogue"] == "residual" else 1)),
                "flops": 2.0 * c["rows"] * c["n"] * c["k"]}
    if c["kind"] == "attention":
        q, k = c["queries"], c["keys"]
        pairs = q * k - q * (q - 1) / 2 if q > 1 else k
        return {"bytes": c["batch"] * c["dim"] * (8 * c["heads"] * q + 4 * c["kv_heads"] * k), "flops": 4.0 * c["batch"] * c["heads"] * c["dim"] * pairs}
    passes = [c["prompt"]] if c["phase"] == "prompt" else ([c["prompt"]] if c["kind"] != "llama" else []) + [1] * c["steps"]
    b, total = c["batch"], {"bytes": 0.0, "flops": 0.0}
    at = c["prompt"] if c["kind"] == "llama" and c["phase"] == "decode" else 0
    for n in passes:
        w, p, extra_bytes, extra_flops = (_llama_work if c["kind"] == "llama" else _dense_work)(c, n, at)
        total["bytes"] += w + extra_bytes
        total["flops"] += 2.0 * p * b * n + extra_flops
        at += n
    return total


def _pairs(n, at, window=0):
    """(query, visible key) pairs of n new positions behind `at` cached ones."""
    if window:
        return float(sum(min(window, at + i + 1) for i in range(n)))
    return n * at + n * (n + 1) / 2.0


def _llama_work(c, n, at):
    """(bytes of the weights, parameters met by every row, bytes of caches and rows, flops of attention and head)."""
    plan, _, high = _llama_plan(c)
    b, kv = c["batch"], 4 * c["kv_heads"] * c["dim"] * c["layers"]
    w = sum(_size(r, k, t) for _, _, t, r, k, _ in plan) + _size(c["vocab"], c["width"], high)
    return (w, sum(r * k for _, _, _, r, k, _ in plan), b * (kv * (at + 2 * n) + 4 * c["vocab"]),
            b * (4.0 * c["heads"] * c["dim"] * c["layers"] * _pairs(n, at) + 2.0 * c["vocab"] * c["width"]))


def _runs(cfg):
    loop = cfg.get("loop")
    order = list(range(len(cfg["layers"])))
    return order if not loop else order[: loop["start"]] + order[loop["start"]: loop["stop"]] * loop["times"] + order[loop["stop"]:]


def _matrices(L):
    if L["type"].startswith("delta"):
        names = ["mix." + n for n in ("q", "k", "v", "g", "b", "a", "o")]
    elif L["type"] == "latent_attention":
        names = ["mix." + n for n in ("q", "g", "o", "uk", "uv") + (() if "kv_from" in L["mixer"] else ("dkv",))]
    elif L["type"] == "attention":
        names = ["mix." + n for n in "qkvo"]
    else:
        names = ["mix.left." + n for n in "qkvog"] + ["mix.right." + n for n in "qkvog"]
    return names + (["mlp.up", "mlp.down"] if L["type"] in ("attention", "parallel") else ["mlp.gate", "mlp.up", "mlp.down"])


def _dense_work(c, n, at):
    cfg = _koludra_config(c) if c["kind"] == "koludra" else _sofudra_config(c)
    params = flops = extra = 0.0
    for i in _runs(cfg):
        L = cfg["layers"][i]
        mx = L["mixer"]
        params += sum(math.prod(_dense_shape(cfg, f"l{i}.{name}")) for name in _matrices(L))
        if L["type"].startswith("delta"):
            flops += 8.0 * mx["heads"] * mx["dim"] * mx["vdim"] * n
            extra += 8 * mx["heads"] * mx["dim"] * mx["vdim"]
        elif L["type"] == "latent_attention":
            flops += 2.0 * mx["heads"] * (mx["dim"] + mx["rot_dim"] + mx["vdim"]) * _pairs(n, at, c["window"])
            extra += 2 * (mx["kv_rank"] + mx["rot_dim"]) * (min(at, c["window"]) + n)
        else:
            full = L["type"] == "parallel"
            a = mx["left"] if full else mx
            flops += 2.0 * a["heads"] * (a["dim"] + a["vdim"]) * _pairs(n, at, 0 if full else c["window"])
            extra += 2 * a["kv_heads"] * (a["dim"] + a["vdim"]) * ((at if full else min(at, c["window"])) + n)
            if full:
                r = mx["right"]
                flops += 4.0 * r["heads"] * r["dim"] * r["vdim"] * n
                extra += 8 * r["heads"] * r["dim"] * r["vdim"]
    if cfg.get("loop"):
        params += cfg["loop"]["times"] * 2 * c["width"] ** 2
    b, head, size = c["batch"], c["vocab"] * c["width"], 2 if c["compute"] == "bfloat16" else 4
    return size * (params + head), params, b * (extra + 4.0 * c["vocab"]), b * (flops + 2.0 * head)


def tolerance(case):
    c = case
    if c["kind"] == "product":  # one row is summed in 32 bits; several rows have 11-bit operands
        return {"rel": 1e-5 if c["rows"] == 1 else 2e-3, "max": 0.02}
    if c["kind"] == "attention":
        return {"rel": 1e-3, "max": 0.05}
    if c["kind"] == "llama":  # 11-bit operands through every layer
        return {"rel": 8e-3, "max": 0.2, "differ": 0.0}
    return {"rel": 2.5e-2, "max": 0.5, "differ": 0.0}  # bf16 operands


# ---- the same in 64 bits -------------------------------------------------------------------------------------------------

def _half(raw, at):
    return raw[:, at: at + 2].contiguous().view(torch.float16).double()


def _decode(raw, n, k, t):
    """Values of raw blocks, [n, k] in 64 bits."""
    raw = raw.reshape(-1, BLOCK[t][1])
    nb = raw.shape[0]
    if t == kb.Q8_0:
        return (_half(raw, 0) * raw[:, 2:].contiguous().view(torch.int8).double()).reshape(n, k)
    if t == kb.Q4_0:
        q = torch.cat([raw[:, 2:] & 15, raw[:, 2:] >> 4], 1)
        return (_half(raw, 0) * (q.double() - 8)).reshape(n, k)
    if t == kb.Q4_K:
        p = raw[:, 4:16].to(torch.int32)
        sc = torch.cat([p[:, :4] & 63, (p[:, 8:] & 15) | ((p[:, :4] >> 6) << 4)], 1)
        mn = torch.cat([p[:, 4:8] & 63, (p[:, 8:] >> 4) | ((p[:, 4:8] >> 6) << 4)], 1)
        qs = raw[:, 16:].reshape(nb, 4, 32)
        q = torch.stack([qs & 15, qs >> 4], 2).reshape(nb, 8, 32).double()
        return ((_half(raw, 0) * sc)[:, :, None] * q - (_half(raw, 2) * mn)[:, :, None]).reshape(n, k)
    ql, qh = raw[:, :128].reshape(nb, 2, 2, 32), raw[:, 128:192].reshape(nb, 2, 1, 32)
    lo = torch.cat([ql & 15, ql >> 4], 2)
    hi = torch.cat([(qh >> s) & 3 for s in (0, 2, 4, 6)], 2)
    q = (lo | (hi << 4)).reshape(nb, 16, 16).double() - 32
    sc = raw[:, 192:208].contiguous().view(torch.int8).double()
    return (_half(raw, 208)[:, :, None] * sc[:, :, None] * q).reshape(n, k)


def _rms(x, w):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + EPS) * w


def _softmax_attend(q, k, v, scale, window=0, cap=0.0, sink=None):
    """q [S, d], k, v [T, ...] of one head, the queries are the last S positions."""
    s = (q @ k.T) * scale
    if cap:
        s = cap * torch.tanh(s / cap)
    S, T = s.shape
    i, j = torch.arange(T - S, T, device=q.device)[:, None], torch.arange(T, device=q.device)[None]
    s.masked_fill_((j > i) | (i - j >= window) if window else j > i, -math.inf)
    if sink is not None:
        s = torch.cat([s, sink.expand(S, 1)], 1)
    return torch.softmax(s, 1)[:, :T] @ v


def exact(case, seed):
    c = case
    if c["kind"] == "product":
        t, e = TYPES[c["type"]], c["epilogue"]
        w = _decode(_blocks(seed, "w", c["n"], c["k"], 0.02, t), c["n"], c["k"], t)
        y = _normal(seed, "x", (c["rows"], c["k"])).double() @ w.T
        if e == "residual":
            y += sum(_normal(seed, f"r{i}", y.shape).double() for i in range(2))
        if e == "swiglu":
            g, u = y.chunk(2, 1)
            y = torch.nn.functional.silu(g) * u
        return y
    if c["kind"] == "attention":
        q = _normal(seed, "q", (c["batch"], c["heads"], c["queries"], c["dim"])).double()
        k, v = (_normal(seed, n, (c["batch"], c["kv_heads"], c["keys"], c["dim"])).half().double() for n in ("k", "v"))
        rep = c["heads"] // c["kv_heads"]
        return torch.stack([torch.stack([_softmax_attend(q[b, h], k[b, h // rep], v[b, h // rep], c["dim"] ** -0.5)
                                         for h in range(c["heads"])]) for b in range(c["batch"])])
    # the next token of token t is t + 1 by the head's make; the ids that come back are those of the 64-bit logits
    tokens = torch.from_numpy(_prompt(c, seed).astype(np.int64)).cuda()
    if c["phase"] == "decode":
        more = (tokens[:, -1:] + 1 + torch.arange(c["steps"] - 1, device="cuda")) % c["vocab"]
        tokens = torch.cat([tokens, more], 1)
    tail = max(1, c["steps"])
    logits = _exact_llama(c, seed, tokens, tail) if c["kind"] == "llama" else _exact_dense(c, seed, tokens, tail)
    ids = logits.argmax(-1).to(torch.int64).cpu().numpy().astype(np.uint32)
    out = {"logits": logits[:, -1].cpu().numpy()}
    return dict(out, ids=ids[:, -1]) if c["phase"] == "prompt" else dict(out, ids=ids[:, :-1], last=ids[:, -1])


def _exact_llama(c, seed, tokens, tail):
    """64-bit logits of the last `tail` positions."""
    B, T = tokens.shape
    E, H, G, D = c["width"], c["heads"], c["kv_heads"], c["dim"]
    plan = {(name, i): (t, n, k, s) for name, i, t, n, k, s in _llama_plan(c)[0]}

    def get(name, i):
        t, n, k, s = plan[name, i]
        return _decode(_blocks(seed, f"{name}{i}", n, k, s, t), n, k, t)
    t, raw = _llama_ends(c, seed, "token_embd")
    be, bb = BLOCK[t]
    used, where = torch.unique(tokens, return_inverse=True)
    x = _decode(raw.reshape(c["vocab"], -1)[used].reshape(-1), used.numel(), E, t)[where]
    del raw
    angle = torch.arange(T, device="cuda", dtype=torch.float64)[:, None] * THETA ** (-2.0 * torch.arange(D // 2, device="cuda", dtype=torch.float64) / D)
    cos, sin = angle.cos()[:, None], angle.sin()[:, None]

    def turn(y):
        a, b = y[..., 0::2], y[..., 1::2]
        return torch.stack([a * cos - b * sin, a * sin + b * cos], -1).flatten(-2)
    for i in range(c["layers"]):
        h = _rms(x, _llama_norm(seed, "attn_norm", i, E).double())
        q, k, v = ((h @ get(n, i).T).reshape(B, T, heads, D) for n, heads in (("attn_q", H), ("attn_k", G), ("attn_v", G)))
        q, k = turn(q), turn(k)
        att = torch.empty_like(q)
        for b in range(B):
            for n in range(H):
                att[b, :, n] = _softmax_attend(q[b, :, n], k[b, :, n * G // H], v[b, :, n * G // H], D ** -0.5)
        y = att.reshape(B, T, H * D) @ get("attn_output", i).T + x
        h = _rms(y, _llama_norm(seed, "ffn_norm", i, E).double())
        h = torch.nn.functional.silu(h @ get("ffn_gate", i).T) * (h @ get("ffn_up", i).T)
        x = y + h @ get("ffn_down", i).T
    x = _rms(x[:, -tail:], _llama_norm(seed, "output_norm", 0, E).double())
    t, raw = _llama_ends(c, seed, "output")
    return x @ _decode(raw, c["vocab"], E, t).T


def _exact_dense(c, seed, tokens, tail):
    cfg = _koludra_config(c) if c["kind"] == "koludra" else _sofudra_config(c)

    def get(name):
        return _dense_weight(cfg, seed, name).double()
    x0 = get("embed")[tokens] * cfg.get("embedding", {}).get("scale", 1.0)
    out = []
    for b in range(tokens.shape[0]):
        x, rows, first = x0[b], {}, (cfg.get("loop") or {}).get("start")
        for i in _runs(cfg):
            L = cfg["layers"][i]
            W = lambda n, i=i: get(f"l{i}.{n}")  # noqa: E731
            if i == first:
                x = torch.cat([x, x0[b]], 1) @ get("loop.in").T
            h = _rms(x, W("norm1"))
            if c["kind"] == "koludra":
                M = lambda n: W("mix." + n)  # noqa: E731
                y = _exact_delta(h, L["mixer"], M) if L["type"].startswith("delta") else _exact_latent(h, L["mixer"], M, rows, i)
                x = x + y + (torch.nn.functional.silu(h @ W("mlp.gate").T) * (h @ W("mlp.up").T)) @ W("mlp.down").T
            else:
                f = torch.nn.functional.gelu(_rms(x, W("norm2")) @ W("mlp.up").T, approximate="tanh") @ W("mlp.down").T
                x = x + cfg["residual_mult"] * (_exact_sofudra_mixer(h, L, W) + f)
        out.append(_rms(x[-tail:], get("final.norm")) @ get("head").T)
    logits, cap = torch.stack(out), cfg.get("logit_softcap", 0.0)
    return cap * torch.tanh(logits / cap) if cap else logits


def _exact_delta(h, mx, W):
    T, H, G, D, V = h.shape[0], mx["heads"], mx["kv_heads"], mx["dim"], mx["vdim"]

    def conv(n):
        z, w = h @ W(n).T, W(n + ".conv")
        z = torch.nn.functional.pad(z.T[None], (w.shape[1] - 1, 0))
        return torch.nn.functional.silu(torch.nn.functional.conv1d(z, w[:, None], groups=w.shape[0])[0].T)

    def unit(z):
        return z * torch.rsqrt((z * z).sum(-1, keepdim=True) + 1e-6)
    q, k = (unit(conv(n).reshape(T, G, D)).repeat_interleave(H // G, 1) for n in "qk")
    q = q * D ** -0.5
    v = conv("v").reshape(T, H, V)
    beta = torch.sigmoid(h @ W("b").T)
    g = torch.exp(-torch.exp(W("A_log")) * torch.nn.functional.softplus(h @ W("a").T + W("dt_bias")))
    S, out = torch.zeros((H, D, V), dtype=h.dtype, device=h.device), []
    for t in range(T):
        S = S * g[t][:, None, None]
        u = beta[t][:, None] * (v[t] - torch.bmm(k[t][:, None], S)[:, 0])
        S = torch.baddbmm(S, k[t][:, :, None], u[:, None])
        out.append(torch.bmm(q[t][:, None], S)[:, 0])
    o = _rms(torch.stack(out), W("norm")) * torch.nn.functional.silu((h @ W("g").T).reshape(T, H, V))
    return o.reshape(T, H * V) @ W("o").T


def _turn_halves(x, freq, mul=1.0):
    """Entries i and i + n of the last axis turn by position x freq_i; x [T, heads, >= 2 n]."""
    a = (torch.arange(x.shape[0], device=x.device, dtype=x.dtype)[:, None] * freq)[:, None]
    cos, sin, n = a.cos() * mul, a.sin() * mul, freq.numel()
    u, v = x[..., :n], x[..., n: 2 * n]
    return torch.cat([u * cos - v * sin, v * cos + u * sin, x[..., 2 * n:]], -1)


def _frequencies(rot):
    i = np.arange(rot["dims"] // 2, dtype=np.float64)
    f, sc, dims, base = rot["base"] ** (-2.0 * i / rot["dims"]), rot.get("scaling"), rot["dims"], rot["base"]
    if not sc:
        return torch.from_numpy(f).cuda(), 1.0
    lo, hi = (dims * math.log(sc["original"] / (2.0 * math.pi * t)) / (2.0 * math.log(base)) for t in (sc["fast"], sc["slow"]))
    lo, hi = max(math.floor(lo), 0), min(math.ceil(hi), dims - 1)
    ramp = np.clip((i - lo) / max(hi - lo, 0.001), 0.0, 1.0)
    return torch.from_numpy(f / sc["factor"] * ramp + f * (1.0 - ramp)).cuda(), 0.1 * math.log(sc["factor"]) + 1.0


def _exact_latent(h, mx, W, rows, i):
    T, H, D, R, V = h.shape[0], mx["heads"], mx["dim"], mx["rot_dim"], mx["vdim"]
    freq = _frequencies(mx["rot"])[0]
    if "kv_from" in mx:
        latent, kr = rows[mx["kv_from"]]
    else:
        y = h @ W("dkv").T
        latent, kr = _rms(y[:, : mx["kv_rank"]], W("dkv.norm")), _turn_halves(y[:, None, mx["kv_rank"]:], freq)[:, 0]
        rows[i] = latent, kr
    q = (h @ W("q").T).reshape(T, H, D + R)
    q = torch.cat([q[..., :D], _turn_halves(q[..., D:], freq)], -1)
    k, v = (latent @ W("uk").T).reshape(T, H, D), (latent @ W("uv").T).reshape(T, H, V)
    o = torch.stack([_softmax_attend(q[:, n], torch.cat([k[:, n], kr], 1), v[:, n], mx["scale"], mx["mask"]["size"]) for n in range(H)], 1)
    return (o * torch.sigmoid(h @ W("g").T)[:, :, None]).reshape(T, H * V) @ W("o").T


def _exact_sofudra_mixer(h, L, W):
    T = h.shape[0]

    def attention(mx, P, beside):
        H, G, D, V = mx["heads"], mx["kv_heads"], mx["dim"], mx["vdim"]
        q, k, v = ((h @ P(n).T + (P(n + ".b") if beside else 0.0)).reshape(T, heads, size) for n, heads, size in (("q", H, D), ("k", G, D), ("v", G, V)))
        q, k = _rms(q, P("q.norm")), _rms(k, P("k.norm"))
        if mx.get("rot"):
            q, k = (_turn_halves(z, *_frequencies(mx["rot"])) for z in (q, k))
        sink = None if beside else P("sink")
        o = torch.stack([_softmax_attend(q[:, n], k[:, n * G // H], v[:, n * G // H], mx["scale"], (mx.get("mask") or {}).get("size", 0),
                                         mx.get("softcap", 0.0), None if sink is None else sink[n]) for n in range(H)], 1)
        if beside:
            o = o * torch.sigmoid(h @ P("g").T)[:, :, None]
        return o.reshape(T, H * V) @ P("o").T
    if L["type"] == "attention":
        return attention(L["mixer"], lambda n: W("mix." + n), False)
    mx = L["mixer"]
    r, R = mx["right"], lambda n: W("mix.right." + n)
    H, D, V = r["heads"], r["dim"], r["vdim"]
    q, k = (torch.nn.functional.silu(h @ R(n).T).reshape(T, H, D) for n in "qk")
    v = torch.nn.functional.silu(h @ R("v").T).reshape(T, H, V)
    i = torch.arange(T, device=h.device, dtype=h.dtype)
    gap = i[:, None] - i[None]
    o = torch.empty_like(v)
    for n in range(H):
        fade = torch.exp(gap.clamp(min=0) * math.log(r["decay"][n])).masked_fill_(gap < 0, 0.0)
        o[:, n] = ((q[:, n] @ k[:, n].T) * fade) @ v[:, n]
    o = _rms(o.reshape(T, H * V), R("norm")) * torch.sigmoid(h @ R("g").T)
    return mx["left_scale"] * attention(mx["left"], lambda n: W("mix.left." + n), True) + mx["right_scale"] * (o @ R("o").T)
