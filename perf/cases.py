"""The work a user of this framework has it do, as cases that can be timed and compared: decoding and prompt passes of a quantised llama through
its runner, one quantised product, the blocks of the other decoder families (attention over a ring cache, latent attention, the feed-forward's two
outer products, routed experts, the gated delta rule) through the ops a program builds them from, and a whole Vadodra model through its step function.

A case is a dict of plain values; prepare() makes what a program holds before the call, run() is one pass, exact() the same in 64 bits with plain
torch.  A program has one device per mode, so the devices live as long as the module."""
import math

import numpy as np
import torch

from crabml_b200 import CudaTensor, CudaTensorDevice, capi, seqops, vadodra
from crabml_b200 import runner as llama

EPS = 1e-5
WTYPES = {"q8_0": (capi.Q8_0, 34, 32), "q4_0": (capi.Q4_0, 18, 32), "q4_k": (capi.Q4_K, 144, 256), "q6_k": (capi.Q6_K, 210, 256)}
# offsets of a block's f16 factors, and the spread of a dequantised weight in units of its factor (what a row of length 1 needs)
F16_AT = {"q8_0": (0,), "q4_0": (0,), "q4_k": (0, 2), "q6_k": (208,)}
SPREAD = {"q8_0": 73.9, "q4_0": 4.6, "q4_k": 4.6 * 31.5, "q6_k": 18.5 * 73.9}

LLAMA_15M = {"dim": 288, "hidden": 768, "heads": 6, "kv_heads": 6, "vocab": 32000}
LLAMA_7B = {"dim": 4096, "hidden": 11008, "heads": 32, "kv_heads": 32, "vocab": 32000}
MISTRAL_7B = {"dim": 4096, "hidden": 14336, "heads": 32, "kv_heads": 8, "vocab": 32000}


# ---- the cases ------------------------------------------------------------------------------------------------------------------------
def listed():
    return [
        # a story model answering token by token, the caller sampling on the host: what a call costs at the least
        dict(LLAMA_15M, name="llama 15m q8_0 tokens", kind="llama", layers=6, weights="q8_0", classifier="q8_0", way="tokens", tokens=16, synth=False),
        # the headline: a 7B model decoding one sequence, every logit row read by the caller
        dict(LLAMA_7B, name="llama 7b q8_0 tokens", kind="llama", layers=32, weights="q8_0", classifier="q8_0", way="tokens", tokens=16, synth=True),
        # the same layers in a K-quant file (Q4_K with a Q6_K classifier, as such files have), some of the layers
        dict(LLAMA_7B, name="llama 7b-layers q4_k tokens", kind="llama", layers=4, weights="q4_k", classifier="q6_k", way="tokens", tokens=16, synth=False),
        # a prompt fed in one call: two layers of the Mistral-7B shape, grouped heads
        dict(MISTRAL_7B, name="mistral 2 layers q8_0 prompt", kind="llama", layers=2, weights="q8_0", classifier="q8_0", way="prompt", tokens=512, synth=False),
        # several sequences' next tokens against one matrix of a 7B layer
        {"name": "product q4_k 8 rows", "kind": "product", "weights": "q4_k", "m": 11008, "k": 4096, "rows": 8},
        # grouped-query attention of a late portion of a prompt over a full window
        {"name": "attention prompt", "kind": "attention", "tokens": 512, "pos": 1531, "heads": 16, "kv_heads": 4, "dk": 128, "dv": 128, "window": 1024, "latent": False},
        # one decoded token over a long cache of latent rows that are keys and values
        {"name": "latent attention token", "kind": "attention", "tokens": 1, "pos": 4000, "heads": 16, "kv_heads": 1, "dk": 576, "dv": 512, "window": 0, "latent": True},
        # norm and input product, gated units and joined output product with the residual sum: the products of one layer, a ragged portion
        {"name": "feed-forward block", "kind": "block", "tokens": 509, "width": 2048, "ff": 6144},
        # routed experts of a portion of a prompt
        {"name": "experts", "kind": "experts", "tokens": 512, "width": 1024, "experts": 16, "top": 4, "ff": 512},
        # the recurrence of a linear-attention layer over a portion of a prompt
        {"name": "delta rule", "kind": "delta", "tokens": 1000, "heads": 16, "kv_heads": 4, "dim": 128},
        # a whole model: a prompt, and a request of a short prompt and sixteen tokens
        {"name": "vadodra prompt", "kind": "vadodra", "way": "prompt", "width": 1024, "tokens": 2048, "prompt": 2048, "vocab": 32000, "dtype": "bfloat16"},
        {"name": "vadodra tokens", "kind": "vadodra", "way": "tokens", "width": 1024, "tokens": 16, "prompt": 100, "vocab": 32000, "dtype": "bfloat16"},
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["llama", "llama", "product", "product", "attention", "attention", "block", "experts", "delta", "vadodra"])
    if kind == "llama":
        way = rng.choice(["tokens", "prompt"])
        heads = rng.choice([4, 8, 16, 32])
        wt = rng.choice(sorted(WTYPES))
        return {"kind": kind, "dim": heads * 128, "hidden": 256 * rng.randint(heads, 3 * heads), "heads": heads, "kv_heads": rng.choice([heads, heads // 4]),
                "vocab": 256 * rng.randint(4, 125), "layers": rng.randint(1, 3), "weights": wt, "classifier": rng.choice([wt, "q6_k"]), "way": way,
                "tokens": rng.randint(3, 24) if way == "tokens" else _log(rng, 2, 1024), "synth": False}
    if kind == "product":
        return {"kind": kind, "weights": rng.choice(sorted(WTYPES)), "m": _log(rng, 200, 14336), "k": 256 * _log(rng, 2, 56), "rows": _log(rng, 1, 600)}
    if kind == "attention":
        latent = rng.random() < 0.4
        T, R = _log(rng, 1, 600), rng.choice([1, 2, 4, 8])
        G = 1 if latent else rng.choice([1, 2, 4])
        d = rng.choice([64, 80, 128])
        return {"kind": kind, "tokens": T, "pos": rng.randint(0, 2500), "heads": R * G, "kv_heads": G, "dk": 576 if latent else d, "dv": 512 if latent else d,
                "window": rng.choice([0, _log(rng, 16, 2048)]), "latent": latent}
    if kind == "block":
        w = 128 * rng.randint(3, 24)
        return {"kind": kind, "tokens": _log(rng, 1, 700), "width": w, "ff": 64 * rng.randint(w // 64, 3 * w // 64)}
    if kind == "experts":
        e = rng.choice([8, 16, 32])
        return {"kind": kind, "tokens": _log(rng, 1, 600), "width": 128 * rng.randint(4, 16), "experts": e, "top": rng.randint(1, 4), "ff": 64 * rng.randint(4, 16)}
    if kind == "delta":
        R = rng.choice([1, 2, 4])
        G = rng.choice([1, 2, 4])
        return {"kind": kind, "tokens": _log(rng, 1, 1500), "heads": R * G, "kv_heads": G, "dim": rng.choice([64, 128])}
    way = rng.choice(["prompt", "tokens"])
    p = _log(rng, 20, 1500)
    return {"kind": kind, "way": way, "width": 128 * rng.choice([4, 8, 12]), "tokens": p if way == "prompt" else rng.randint(2, 16), "prompt": p, "vocab": 1000 * rng.randint(2, 32),
            "dtype": rng.choice(["bfloat16", "bfloat16", "float32"])}


# ---- inputs ---------------------------------------------------------------------------------------------------------------------------
_devices = {}


def device(lazy):
    """lazy = 2: a fused token runs as one persistent kernel, the llama runner's serving mode; 0: the mode the other families' ops need"""
    if lazy not in _devices:
        _devices[lazy] = CudaTensorDevice(0, lazy=lazy)
    return _devices[lazy]


class Inputs:
    """torch values made on the GPU from the seed alone, in a fixed order"""

    def __init__(self, seed):
        self.g = torch.Generator(device="cuda")
        self.g.manual_seed(int(seed))

    def normal(self, *shape, scale=1.0):
        return torch.randn(shape, generator=self.g, device="cuda") * scale

    def uniform(self, *shape, lo=0.0, hi=1.0):
        return torch.rand(shape, generator=self.g, device="cuda") * (hi - lo) + lo

    def ids(self, n, vocab):
        return torch.randint(0, vocab, (n,), generator=self.g, device="cuda").tolist()

    def blocks(self, wt, rows, cols):
        """[rows, blocks, bytes] of GGUF blocks whose rows have about unit length"""
        _, nbytes, per = WTYPES[wt]
        raw = torch.randint(0, 256, (rows, cols // per, nbytes), generator=self.g, device="cuda", dtype=torch.uint8)
        for at in F16_AT[wt]:
            d = ((0.5 + self.uniform(rows, cols // per)) / (SPREAD[wt] * math.sqrt(cols))).to(torch.float16)
            if at == 2:                                      # the offset of a Q4_K block: half the range of its 4-bit numbers below zero
                d = (raw[..., 0:2].contiguous().view(torch.float16).squeeze(-1).float() * 7.5).to(torch.float16)
            raw[..., at:at + 2] = d.unsqueeze(-1).contiguous().view(torch.uint8)
        return raw


def _upload(t, dev):
    return CudaTensor.new(t.cpu().numpy(), list(t.shape), dev)


def _upload_blocks(raw, wt, shape, dev):
    return CudaTensor.from_cpu(raw.cpu().numpy().reshape(-1), list(shape), WTYPES[wt][0], dev)


def _bf16(t):
    return t.to(torch.bfloat16)


def _bits(t):
    return t.contiguous().view(torch.int16).cpu().numpy().view(np.uint16)


def _upload_bf16(t, dev):
    return CudaTensor.from_cpu(_bits(t), list(t.shape), capi.BF16, dev)


LLAMA_PARTS = (("wq", "dim", "dim"), ("wk", "kv", "dim"), ("wv", "kv", "dim"), ("wo", "dim", "dim"), ("ffn_gate", "hidden", "dim"), ("ffn_up", "hidden", "dim"), ("ffn_down", "dim", "hidden"))


def _llama_inputs(c, seed):
    """-> (token ids, iterator of (name, weight type or None, tensor): the order in which a file would give them)"""
    r = Inputs(seed)
    ids = r.ids(c["tokens"], c["vocab"])
    size = dict(c, kv=c["dim"] // c["heads"] * c["kv_heads"])

    def parts():
        for _ in range(c["layers"]):
            for name, m, k in LLAMA_PARTS:
                yield name, c["weights"], r.blocks(c["weights"], size[m], size[k])
            for name in ("rms_att", "rms_ffn"):
                yield name, None, 1.0 + 0.05 * r.normal(c["dim"])
        yield "token_embed", c["weights"], r.blocks(c["weights"], c["vocab"], c["dim"])
        yield "output_weight", c["classifier"], r.blocks(c["classifier"], c["vocab"], c["dim"])
        yield "rms_final", None, 1.0 + 0.05 * r.normal(c["dim"])
    return ids, parts()


def _attention_inputs(c, seed):
    r = Inputs(seed)
    seen = c["pos"] + c["tokens"]
    ring = min(seen, c["window"] - 1 + c["tokens"]) if c["window"] else seen
    q = r.normal(c["tokens"], c["heads"] * c["dk"])
    k = r.normal(ring, c["kv_heads"] * c["dk"])
    v = None if c["latent"] else r.normal(ring, c["kv_heads"] * c["dv"])
    return q, k, v


def _block_inputs(c, seed):
    r, D, ff = Inputs(seed), c["width"], c["ff"]
    return {"x": r.normal(c["tokens"], D), "a": r.normal(c["tokens"], D), "norm": 1.0 + 0.2 * r.normal(D), "w_in": _bf16(r.normal(2 * ff, D, scale=D ** -0.5)),
            "w_out": _bf16(r.normal(D, D + ff, scale=(D + ff) ** -0.5))}


def _experts_inputs(c, seed):
    r, D, E, ff = Inputs(seed), c["width"], c["experts"], c["ff"]
    return {"x": r.normal(c["tokens"], D), "router": r.normal(E, D, scale=D ** -0.5), "gate": _bf16(r.normal(E * ff, D, scale=D ** -0.5)),
            "up": _bf16(r.normal(E * ff, D, scale=D ** -0.5)), "down": _bf16(r.normal(E * D, ff, scale=ff ** -0.5))}


def _delta_inputs(c, seed):
    r, T, H, G, d = Inputs(seed), c["tokens"], c["heads"], c["kv_heads"], c["dim"]

    def unit(scale):
        t = r.normal(T, G, d)
        return (t / t.norm(dim=-1, keepdim=True) * scale).reshape(T, G * d)
    return {"q": unit(d ** -0.5), "k": unit(1.0), "v": r.normal(T, H * d), "a": r.normal(T, H), "b": r.normal(T, H), "a_log": r.uniform(H, lo=0.5, hi=4.0).log(),
            "dt_bias": r.uniform(H, lo=-3.0, hi=0.0)}


def vadodra_config(c):
    """window attention and latent attention alternating, the second latent layer over the first one's cache, a dense feed-forward of 3 x width each"""
    H = c["width"] // 128
    win = {"heads": H, "kv_heads": max(1, H // 4), "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "mask": {"size": 1024}, "rot": {"dims": 64, "base": 200000.0}}
    lat = {"heads": H, "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": 512, "scale": 192 ** -0.5, "rot": {"dims": 64, "base": 10000.0}}
    mlp = {"kind": "dense", "ff": 3 * c["width"], "limit": 7.0}
    layers = [{"type": "attention", "mixer": win, "mlp": mlp}, {"type": "latent_attention", "mixer": lat, "mlp": mlp}, {"type": "attention", "mixer": win, "mlp": mlp},
              {"type": "latent_attention", "mixer": dict(lat, kv_from=1), "mlp": mlp}]
    return {"architecture": "Vadodra", "vocab": c["vocab"], "width": c["width"], "embedding": {"scale": 1.0}, "norm": {"eps": EPS}, "layers": layers}


def _vadodra_inputs(c, seed):
    r = Inputs(seed)
    n = c["prompt"] + (c["tokens"] if c["way"] == "tokens" else 0)
    ids = r.ids(n, c["vocab"])
    w = {}
    for name, shape in vadodra.expected_tensors(vadodra.parse_config(vadodra_config(c))).items():
        w[name] = _bf16(1.0 + 0.2 * r.normal(*shape) if name.endswith(("norm1", ".norm")) else r.normal(*shape, scale=shape[-1] ** -0.5))
    return ids, w


class State(dict):
    """what a program holds; a model's runner goes when the program drops it"""

    def __del__(self):
        if "model" in self:
            self["model"].close()


def prepare(case, seed):
    c, kind = case, case["kind"]
    s = State(case=c)
    if kind == "llama":
        dev = device(2)
        s["conf"] = conf = llama.LlamaConfig(c["heads"], c["kv_heads"], c["layers"], c["dim"], c["hidden"], 4096, c["vocab"], EPS, c["dim"] // c["heads"])
        s["ids"], parts = _llama_inputs(c, seed)
        if c["synth"]:                                       # blocks made on the device: gigabytes of them need not cross the host
            s["weights"] = llama.synthetic_weights(dev, conf, WTYPES[c["weights"]][0], WTYPES[c["classifier"]][0], seed=int(seed))
        else:
            s["weights"] = w = {}
            for name, wt, t in parts:
                up = _upload_blocks(t, wt, [t.shape[0], t.shape[1] * WTYPES[wt][2]], dev) if wt else CudaTensor.from_cpu(t.cpu().numpy(), [t.numel()], capi.F32, dev)
                if name in ("token_embed", "output_weight", "rms_final"):
                    w[name] = up
                else:
                    w.setdefault(name, []).append(up)
        return s
    dev = device(0)
    if kind == "product":
        r = Inputs(seed)
        s["w"] = _upload_blocks(r.blocks(c["weights"], c["m"], c["k"]), c["weights"], [c["m"], c["k"]], dev)
        s["x"] = _upload(r.normal(c["rows"], c["k"]), dev)
        out = [c["rows"], c["m"]]
    elif kind == "attention":
        q, k, v = _attention_inputs(c, seed)
        s["q"], s["k"], s["v"] = _upload(q, dev), _upload(k, dev), None if v is None else _upload(v, dev)
        out = [c["tokens"], c["heads"] * c["dv"]]
    elif kind == "block":
        for name, t in _block_inputs(c, seed).items():
            s[name] = _upload_bf16(t, dev) if t.dtype == torch.bfloat16 else _upload(t, dev)
        out = [c["tokens"], c["width"]]
    elif kind == "experts":
        for name, t in _experts_inputs(c, seed).items():
            s[name] = _upload_bf16(t, dev) if t.dtype == torch.bfloat16 else _upload(t, dev)
        out = [c["tokens"], c["width"]]
    elif kind == "delta":
        for name, t in _delta_inputs(c, seed).items():
            s[name] = _upload(t, dev)
        n = c["heads"] * c["dim"]
        s["state"] = CudaTensor.alloc([n * c["dim"]], capi.F32, dev)
        s["state_host"] = torch.empty(n * c["dim"], pin_memory=True)
        out = [c["tokens"], n]
    else:
        ids, w = _vadodra_inputs(c, seed)
        s["ids"] = ids
        weights = {n: (t.float().cpu().numpy() if t.dim() == 1 else _bits(t)) for n, t in w.items()}
        s["model"] = vadodra.VadodraModel(dev, vadodra_config(c), (weights, {n for n, t in w.items() if t.dim() > 1}), c["dtype"], chunk=512, max_seq=len(ids) + 8)
        return s
    s["out"] = torch.empty(out, pin_memory=True)
    return s


# ---- one pass -------------------------------------------------------------------------------------------------------------------------
def _export(t, host):
    """a device tensor into pinned memory, in the device's order of work, without waiting"""
    t.device.check(t.device.lib.cc_tensor_export_f32_async(t.device.handle, t._view(), host.data_ptr(), host.numel()))
    return host


def run(s):
    c, kind = s["case"], s["case"]["kind"]
    if kind == "llama":
        n = c["tokens"]
        r = llama.LlamaRunner(device(2), s["conf"], s["weights"], (n + 63) // 64 * 64)
        try:
            if c["way"] == "prompt":
                return r.forward(s["ids"], 0).copy()
            return np.stack([r.forward([t], i).copy() for i, t in enumerate(s["ids"])])
        finally:
            r.close()
    if kind == "product":
        return _export(s["w"].matmul_vec(s["x"]), s["out"])
    if kind == "attention":
        y = seqops.masked_attention(s["q"], s["k"], s["v"], c["pos"], c["heads"], c["kv_heads"], c["dk"], c["dv"], c["dk"] ** -0.5, window=c["window"])
        return _export(y, s["out"])
    if kind == "block":
        ff = c["ff"]
        x = s["x"].dup()
        h = seqops.layer_norm_product(x, s["norm"], None, EPS, s["w_in"])
        seqops.joined_product_accumulate(x, s["w_out"], s["a"], h, 0, ff, ff, act=capi.ACT_SWISH, alpha=1.702, limit=7.0, up_shift=1.0)
        return _export(x, s["out"])
    if kind == "experts":
        ids, wts = seqops.moe_route(s["x"], s["router"], None, c["top"])
        return _export(seqops.moe_experts(s["x"], ids, wts, s["gate"], s["up"], s["down"], c["experts"], c["ff"]), s["out"])
    if kind == "delta":
        seqops.tensor_zero(s["state"])
        y = seqops.gated_delta_rule(s["q"], s["k"], s["v"], s["a"], s["b"], s["a_log"], s["dt_bias"], s["state"], c["heads"], c["kv_heads"], c["dim"], c["dim"])
        return [_export(y, s["out"]), _export(s["state"], s["state_host"])]
    m, ids, p = s["model"], s["ids"], c["prompt"]
    slot = m.open()
    try:
        if c["way"] == "prompt":
            return m.step(slot, ids, [p - 1])
        m.step(slot, ids[:p])
        return np.concatenate([m.step(slot, [t], [0]) for t in ids[p:]])
    finally:
        m.close_seq(slot)


# ---- what a pass cannot do without ----------------------------------------------------------------------------------------------------------
def _llama_weight_bytes(c):
    size = dict(c, kv=c["dim"] // c["heads"] * c["kv_heads"])
    per = {w: WTYPES[w][1] / WTYPES[w][2] for w in WTYPES}
    elements = sum(size[m] * size[k] for _, m, k in LLAMA_PARTS) * c["layers"]
    head = c["vocab"] * c["dim"]
    return elements * per[c["weights"]] + head * per[c["classifier"]], elements, head


def _visible(c):
    """the keys all queries of an attention case see together, and the rows of the ring any of them sees"""
    lo = [max(0, p - c["window"] + 1) if c["window"] else 0 for p in range(c["pos"], c["pos"] + c["tokens"])]
    return sum(p - a + 1 for p, a in zip(range(c["pos"], c["pos"] + c["tokens"]), lo)), c["pos"] + c["tokens"] - lo[0]


def work(case):
    c, kind, n = case, case["kind"], case["tokens"] if "tokens" in case else 0
    if kind == "llama":
        nbytes, elements, head = _llama_weight_bytes(c)
        kv = 2 * c["layers"] * (c["dim"] // c["heads"]) * c["kv_heads"] * 4
        if c["way"] == "tokens":                             # every token is asked for by itself: the weights once for each, and the cache so far
            return {"bytes": n * (nbytes + 4 * c["vocab"]) + kv * n * (n + 1) // 2, "flops": 2 * n * (elements + head) + 2 * n * (n + 1) * c["dim"] * c["layers"]}
        return {"bytes": nbytes + kv * n + 4 * c["vocab"], "flops": 2 * (n * elements + head) + 4 * n * n * c["dim"] * c["layers"]}
    if kind == "product":
        per = WTYPES[c["weights"]][1] / WTYPES[c["weights"]][2]
        return {"bytes": c["m"] * c["k"] * per + 4 * c["rows"] * (c["m"] + c["k"]), "flops": 2 * c["rows"] * c["m"] * c["k"]}
    if kind == "attention":
        pairs, rows = _visible(c)
        row = c["kv_heads"] * (c["dk"] + (0 if c["latent"] else c["dv"]))
        return {"bytes": 4 * (rows * row + n * c["heads"] * (c["dk"] + c["dv"])), "flops": 2 * pairs * c["heads"] * (c["dk"] + c["dv"])}
    if kind == "block":
        D, ff = c["width"], c["ff"]
        return {"bytes": 2 * (2 * ff * D + D * (D + ff)) + 4 * 3 * n * D, "flops": 2 * n * (2 * ff * D + D * (D + ff))}
    if kind == "experts":
        D, ff, used = c["width"], c["ff"], min(c["experts"], n * c["top"])
        return {"bytes": 2 * 3 * used * ff * D + 4 * (2 * n * D + c["experts"] * D), "flops": 2 * n * (c["top"] * 3 * ff * D + c["experts"] * D)}
    if kind == "delta":
        H, G, d = c["heads"], c["kv_heads"], c["dim"]
        return {"bytes": 4 * (n * (2 * G * d + 2 * H * d + 2 * H) + H * d * d), "flops": 7 * n * H * d * d}
    D, V, p = c["width"], c["vocab"], c["prompt"]
    H = D // 128
    G, ff, wb = max(1, H // 4), 3 * D, 2 if c["dtype"] == "bfloat16" else 4
    win, lat = D * (128 * (H + G) + 2 * ff) + D * (128 * H + ff), D * (H * 193 + 2 * ff) + D * (128 * H + ff) + H * 256 * 512
    elements = 2 * win + 2 * lat + D * 576
    passes, rows = (1, p) if c["way"] == "prompt" else (1 + n, p + n)
    cached = min(1024, rows) * 2 * 2 * G * 128 + rows * 576 * 2
    near = sum(min(1024, i + 1) for i in range(rows))
    return {"bytes": passes * elements * wb + (1 if c["way"] == "prompt" else n) * V * (D * wb + 4) + 4 * cached * (1 if c["way"] == "prompt" else n),
            "flops": 2 * rows * elements + 2 * H * (2 * near * 256 + 2 * rows * (rows + 1) // 2 * 320)}


def tolerance(case):
    kind = case["kind"]
    if kind == "llama":
        # the activation quantisers truncate, so a last-bit difference becomes a step of an 8-bit number, and layers carry it on: the two orders of
        # summation of the CPU code this framework follows differ by 1.6 to 4 % of the largest logit after six layers
        return {"rel": 0.03, "max": 0.3}
    if kind == "product":
        # up to 31 rows: exact integer products, 32-bit sums of them; more: the operands rounded to 16 bits once
        return {"rel": 1e-5} if case["rows"] < 32 else {"rel": 2e-3}
    if kind in ("attention", "delta"):
        return {"rel": 1e-5, "max": 2e-4}
    if kind in ("block", "experts"):
        return {"rel": 1e-2}
    return {"rel": 2e-2} if case["dtype"] == "bfloat16" else {"rel": 1e-4}


# ---- the same in 64 bits ------------------------------------------------------------------------------------------------------------------
F = torch.float64


def _f16_at(raw, at):
    return raw[..., at:at + 2].contiguous().view(torch.float16).to(F)                   # [rows, blocks, 1]


def _dequantise(wt, raw):
    rows, nb = raw.shape[:2]
    if wt == "q8_0":
        w = raw[..., 2:].contiguous().view(torch.int8).to(F) * _f16_at(raw, 0)
    elif wt == "q4_0":
        b = raw[..., 2:]
        w = (torch.cat([b & 15, b >> 4], -1).to(F) - 8.0) * _f16_at(raw, 0)
    elif wt == "q4_k":
        s = raw[..., 4:16].to(torch.int32)
        sc = torch.cat([s[..., 0:4] & 63, (s[..., 8:12] & 15) | ((s[..., 0:4] >> 6) << 4)], -1)
        mn = torch.cat([s[..., 4:8] & 63, (s[..., 8:12] >> 4) | ((s[..., 4:8] >> 6) << 4)], -1)
        b = raw[..., 16:].reshape(rows, nb, 4, 32)
        q = torch.stack([b & 15, b >> 4], -2).reshape(rows, nb, 8, 32).to(F)
        w = q * (_f16_at(raw, 0) * sc.to(F)).unsqueeze(-1) - (_f16_at(raw, 2) * mn.to(F)).unsqueeze(-1)
    else:
        ql, qh = raw[..., 0:128].reshape(rows, nb, 2, 2, 32).to(torch.int32), raw[..., 128:192].reshape(rows, nb, 2, 32).to(torch.int32)
        low = torch.stack([ql[..., 0, :] & 15, ql[..., 1, :] & 15, ql[..., 0, :] >> 4, ql[..., 1, :] >> 4], -2)
        high = torch.stack([(qh >> (2 * i)) & 3 for i in range(4)], -2)
        q = ((low | (high << 4)) - 32).to(F).reshape(rows, nb, 16, 16)
        w = q * (raw[..., 192:208].contiguous().view(torch.int8).to(F) * _f16_at(raw, 208)).unsqueeze(-1)
    return w.reshape(rows, -1)


def _quantise(wt, x):
    """the activation as the format's product takes it: 8-bit numbers of 32 (truncated) or 256 (rounded) beside one factor"""
    per = 256 if wt.endswith("_k") else 32
    b = x.reshape(*x.shape[:-1], -1, per)
    if per == 32:
        d = b.abs().amax(-1, keepdim=True) / 127.0
        q = torch.where(d > 0, torch.trunc(b / d.clamp_min(1e-300)), torch.zeros_like(b)) * d.to(torch.float16).to(F)
    else:
        top = torch.gather(b, -1, b.abs().argmax(-1, keepdim=True))
        d = -top / 128.0
        q = torch.where(top != 0, torch.clamp_max(torch.round(b / torch.where(top != 0, d, torch.ones_like(d))), 127.0), torch.zeros_like(b)) * d
    return q.reshape(x.shape)


def _product(wt, raw, x):
    return _quantise(wt, x) @ _dequantise(wt, raw).T


def _rms(x, w):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS) * w


def _turned(x, base, dims, halves):
    """x [T, heads, d], row t at position t: the first `dims` coordinates turned in pairs"""
    T, n = x.shape[0], dims // 2
    a = torch.arange(T, device="cuda", dtype=F)[:, None] * float(base) ** (-torch.arange(n, device="cuda", dtype=F) / n)
    cos, sin = a.cos()[:, None], a.sin()[:, None]
    lo, hi = (slice(0, n), slice(n, 2 * n)) if halves else (slice(0, dims, 2), slice(1, dims, 2))
    out = x.clone()
    out[..., lo] = x[..., lo] * cos - x[..., hi] * sin
    out[..., hi] = x[..., lo] * sin + x[..., hi] * cos
    return out


def _attend(q, k, v, scale, visible):
    """q [T, H, d], k [n, G, d], v [n, G, dv] with H / G query heads in a row on each key head; visible [T, n]"""
    R = q.shape[1] // k.shape[1]
    out = []
    for h in range(q.shape[1]):
        s = (q[:, h] @ k[:, h // R].T * scale).masked_fill(~visible, -math.inf)
        out.append(torch.softmax(s, -1) @ v[:, h // R])
    return torch.stack(out, 1)


def _exact_llama(c, seed):
    ids, parts = _llama_inputs(c, seed)
    tokens, wt, H, G = torch.tensor(ids, device="cuda"), c["weights"], c["heads"], c["kv_heads"]
    n, hd = len(ids), c["dim"] // c["heads"]
    got = {}
    for name, _, t in parts:
        got.setdefault(name, []).append(t)
    x = _dequantise(wt, got["token_embed"][0][tokens])
    # a token at a time each sees itself and those before it; a call's tokens all see each other
    visible = torch.ones(n, n, dtype=torch.bool, device="cuda")
    if c["way"] == "tokens":
        visible = visible.tril()
    order = [h % G for h in range(H)]                                                     # the query head h reads key head h mod G
    for i in range(c["layers"]):
        w = {p[0]: got[p[0]][i] for p in LLAMA_PARTS}
        h = _rms(x, got["rms_att"][i].to(F))
        q, k, v = (_product(wt, w[p], h).reshape(n, -1, hd) for p in ("wq", "wk", "wv"))
        q, k = _turned(q, 10000.0, hd, False), _turned(k, 10000.0, hd, False)
        x = x + _product(wt, w["wo"], _attend(q, k[:, order], v[:, order], hd ** -0.5, visible).reshape(n, -1))
        h = _rms(x, got["rms_ffn"][i].to(F))
        x = x + _product(wt, w["ffn_down"], torch.nn.functional.silu(_product(wt, w["ffn_gate"], h)) * _product(wt, w["ffn_up"], h))
    h = _rms(x if c["way"] == "tokens" else x[-1:], got["rms_final"][0].to(F))
    y = _product(c["classifier"], got["output_weight"][0], h)
    return y if c["way"] == "tokens" else y[0]


def _exact_attention(c, seed):
    q, k, v = (None if t is None else t.to(F) for t in _attention_inputs(c, seed))
    T, G, dk, dv = c["tokens"], c["kv_heads"], c["dk"], c["dv"]
    pos, ring = torch.arange(c["pos"], c["pos"] + T, device="cuda"), k.shape[0]
    keys = torch.arange(c["pos"] + T - ring, c["pos"] + T, device="cuda")                # the positions the ring holds
    k = k[keys % ring].reshape(ring, G, dk)
    v = k[..., :dv] if v is None else v[keys % ring].reshape(ring, G, dv)
    visible = keys[None] <= pos[:, None]
    if c["window"]:
        visible &= pos[:, None] - keys[None] < c["window"]
    return _attend(q.reshape(T, -1, dk), k, v, dk ** -0.5, visible).reshape(T, -1)


def _clamped_unit(g, u):
    g, u = g.clamp_max(7.0), u.clamp(-7.0, 7.0)
    return g * torch.sigmoid(1.702 * g) * (u + 1.0)


def _layer_norm(x, w):
    d = x - x.mean(-1, keepdim=True)
    return d / torch.sqrt((d * d).mean(-1, keepdim=True) + EPS) * w


def _exact_block(c, seed):
    t = {k: v.to(F) for k, v in _block_inputs(c, seed).items()}
    h = _layer_norm(t["x"], t["norm"]) @ t["w_in"].T
    return t["x"] + torch.cat([t["a"], _clamped_unit(h[:, :c["ff"]], h[:, c["ff"]:])], -1) @ t["w_out"].T


def _exact_experts(c, seed):
    t = {k: v.to(F) for k, v in _experts_inputs(c, seed).items()}
    x, D, E, ff = t["x"], c["width"], c["experts"], c["ff"]
    wts, ids = torch.softmax(x @ t["router"].T, -1).topk(c["top"], -1)
    gate, up, down = t["gate"].reshape(E, ff, D), t["up"].reshape(E, ff, D), t["down"].reshape(E, D, ff)
    out = torch.zeros_like(x)
    for e in range(E):
        y = (torch.nn.functional.silu(x @ gate[e].T) * (x @ up[e].T)) @ down[e].T
        out += y * (wts * (ids == e)).sum(-1, keepdim=True)
    return out


def _exact_delta(c, seed):
    t = {k: v.to(F) for k, v in _delta_inputs(c, seed).items()}
    T, H, G, d = c["tokens"], c["heads"], c["kv_heads"], c["dim"]
    q, k = (t[n].reshape(T, G, d).repeat_interleave(H // G, 1) for n in ("q", "k"))
    v, beta = t["v"].reshape(T, H, d), torch.sigmoid(t["b"])
    decay = torch.exp(-t["a_log"].exp() * torch.nn.functional.softplus(t["a"] + t["dt_bias"]))
    S, out = torch.zeros(H, d, d, dtype=F, device="cuda"), []
    for i in range(T):
        S = S * decay[i, :, None, None]
        u = beta[i, :, None] * (v[i] - torch.einsum("hkv,hk->hv", S, k[i]))
        S = S + k[i, :, :, None] * u[:, None, :]
        out.append(torch.einsum("hkv,hk->hv", S, q[i]))
    return [torch.stack(out).reshape(T, -1), S.reshape(-1)]


def _exact_vadodra(c, seed):
    ids, w = _vadodra_inputs(c, seed)
    w = {n: t.to(F) for n, t in w.items()}
    T, H = len(ids), c["width"] // 128
    x, cache = w["embed"][torch.tensor(ids, device="cuda")], {}
    causal = torch.ones(T, T, dtype=torch.bool, device="cuda").tril()
    near = causal & ~causal.tril(-1024)
    for i, L in enumerate(vadodra_config(c)["layers"]):
        p, q_, m = f"l{i}.", f"l{i}.mix.", L["mixer"]
        h = _layer_norm(x, w[p + "norm1"])
        if L["type"] == "attention":
            q, raw = (h @ w[q_ + n].T for n in ("q", "k"))
            q, raw = q.reshape(T, H, 128), raw.reshape(T, -1, 128)
            turned = [_turned(_rms(t, w[q_ + n]), m["rot"]["base"], 64, False) for t, n in ((q, "q.norm"), (raw, "k.norm"))]
            y = _attend(turned[0], turned[1], raw, m["scale"], near)
        else:
            if "kv_from" not in m:
                a = h @ w[q_ + "dkv"].T
                cache = {"c": _rms(a[:, :512], w[q_ + "dkv.norm"]), "r": _turned(a[:, None, 512:], 10000.0, 64, True)}
            q = (h @ w[q_ + "q"].T).reshape(T, H, 192)
            q = torch.cat([q[..., :128], _turned(q[..., 128:], 10000.0, 64, True)], -1)
            k = torch.cat([(cache["c"] @ w[q_ + "uk"].T).reshape(T, H, 128), cache["r"].expand(T, H, 64)], -1)
            y = _attend(q, k, (cache["c"] @ w[q_ + "uv"].T).reshape(T, H, 128), m["scale"], causal) * torch.sigmoid(h @ w[q_ + "g"].T).unsqueeze(-1)
        x = x + y.reshape(T, -1) @ w[q_ + "o"].T + _clamped_unit(h @ w[p + "mlp.gate"].T, h @ w[p + "mlp.up"].T) @ w[p + "mlp.down"].T
    return _layer_norm(x[-c["tokens"]:] if c["way"] == "tokens" else x[-1:], w["final.norm"]) @ w["embed"].T


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "llama":
        return None if c["synth"] else _exact_llama(c, seed)
    if kind == "product":
        r = Inputs(seed)
        raw = r.blocks(c["weights"], c["m"], c["k"])
        return _product(c["weights"], raw, r.normal(c["rows"], c["k"]).to(F))
    return {"attention": _exact_attention, "block": _exact_block, "experts": _exact_experts, "delta": _exact_delta, "vadodra": _exact_vadodra}[kind](c, seed)
