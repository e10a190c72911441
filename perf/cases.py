"""The workloads that this framework's speed is measured on: what its users have it do, through the public entry points.

Two layers of the interface are used in earnest. Programs that serve a model take prompts and generate through the runner
(`ops.Model`: the W8A8 Llama, and the floating-point families Pibidra and Sabisun); programs that bring a graph of their own call
the operators (`ops.pref_Linear_Layer_i8xi8`, `ops.dec_MLP_block`, `ops.MHA_i8xi8_Prefilling`, `ops.MHA_i8xi8_Decoding`).
`listed` names twelve workloads of these seven kinds, `draw` gives others of the same ranges, odd sizes among them.

Weights and activations are random, scaled as in a trained model: attention scores of order one, so that the softmax spreads over
many keys, and residual streams whose parts are of like size.
"""
import math
import random

import torch

from flexllm_b200 import models
from flexllm_b200 import ops as F

DEV = "cuda"
D64 = torch.float64

# layer sizes, as bench.py uses them; `llama` is the W8A8 model's own
SIZES = {
    "llama": dict(layers=16, width=2048, heads=32, kv_heads=8, dim=64, ff=8192, vocab=128256, window=1024),
    "wide": dict(layers=8, width=4096, heads=32, kv_heads=8, dim=128, ff=14336, vocab=128256, window=1024),
    "small": dict(layers=12, width=1024, heads=8, kv_heads=2, dim=128, ff=4096, vocab=32000, window=512),
}


def listed():
    return [
        # one projection of a short prompt: a user's own graph, where a call's fixed costs count
        dict(name="linear_128", kind="linear", M=128, N=2048, K=2048),
        # the feed-forward block of one decode step: a single conversation, and a full batch
        dict(name="mlp_1", kind="mlp", M=1),
        dict(name="mlp_64", kind="mlp", M=64),
        # attention of four prompts
        dict(name="mha_prefill_4x1024", kind="mha_prefill", B=4, S=1024, heads=32, kv_heads=8),
        # attention of one decode step over a paged cache, a full batch of long and short conversations
        dict(name="mha_decode_64", kind="mha_decode", B=64, lo=512, hi=8192, heads=32, kv_heads=8),
        # the W8A8 Llama: a batch of long prompts up to the first token
        dict(name="llama_prompt_32x1024", kind="llama_prompt", B=32, S=1024),
        # ... whole requests: a batch with longer answers, and one conversation alone
        dict(name="llama_request_32", kind="llama_request", B=32, S=256, new=96, top_k=0),
        dict(name="llama_request_1", kind="llama_request", B=1, S=1024, new=48, top_k=0),
        # the floating-point families: prompts of an odd length up to their logits, and whole requests
        dict(name="pibidra_prompt_4x1000", kind="family_prompt", family="Pibidra", size="llama", B=4, S=1000, dtype="bfloat16"),
        dict(name="pibidra_request_4", kind="family_request", family="Pibidra", size="llama", B=4, S=200, new=48, dtype="bfloat16"),
        dict(name="sabisun_prompt_4x1000", kind="family_prompt", family="Sabisun", size="llama", B=4, S=1000, dtype="bfloat16"),
        dict(name="sabisun_request_4", kind="family_request", family="Sabisun", size="llama", B=4, S=200, new=48, dtype="bfloat16"),
    ]


def draw(rng):
    def log(lo, hi, step=1):
        return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / step)) * step))

    kind = rng.choice(["linear", "mlp", "mha_prefill", "mha_decode", "llama_prompt", "llama_request", "family_prompt", "family_request"])
    if kind == "linear":
        return dict(kind=kind, M=log(9, 8192), N=log(512, 16384, 8), K=log(512, 8192, 16))
    if kind == "mlp":
        return dict(kind=kind, M=log(1, 64))
    if kind == "mha_prefill":
        kv = rng.choice([2, 4, 8])
        return dict(kind=kind, B=log(1, 8), S=log(64, 2048, 16), heads=kv * rng.choice([1, 2, 4]), kv_heads=kv)
    if kind == "mha_decode":
        lo = log(16, 4096)
        return dict(kind=kind, B=log(1, 64), lo=lo, hi=log(lo, 8192), heads=32, kv_heads=8)
    if kind == "llama_prompt":
        S = log(64, 2048, 16)
        return dict(kind=kind, B=log(1, min(32, 32768 // S)), S=S)
    if kind == "llama_request":
        return dict(kind=kind, B=log(1, 32), S=log(32, 1024, 16), new=log(8, 96), top_k=rng.choice([0, 0, 5]))
    family, size = rng.choice(["Pibidra", "Sabisun"]), rng.choice(["llama", "wide", "small"])
    dtype = "float32" if size == "small" and rng.random() < 0.3 else "bfloat16"
    most = 512 if dtype == "float32" else 8192
    if kind == "family_prompt":
        S = log(48, min(most, 2048))
        return dict(kind=kind, family=family, size=size, B=log(1, max(1, min(16, most // S))), S=S, dtype=dtype)
    return dict(kind=kind, family=family, size=size, B=log(1, 16 if dtype == "bfloat16" else 4), S=log(16, 512 if dtype == "bfloat16" else 100),
                new=log(8, 48), dtype=dtype)


# ------------------------------------------------------------------------------------------------- inputs
class Source:
    """Random tensors on the GPU, from a seed alone."""

    def __init__(self, seed):
        self.g = torch.Generator(device=DEV)
        self.g.manual_seed(1000003 * int(seed) + 17)

    def s8(self, *shape):
        return torch.randint(-127, 128, shape, dtype=torch.int8, device=DEV, generator=self.g)

    def uniform(self, lo, hi, *shape):
        return torch.rand(shape, device=DEV, generator=self.g) * (hi - lo) + lo

    def normal(self, *shape):
        return torch.randn(shape, device=DEV, generator=self.g)

    def bf16(self, *shape, s=1.0, add=0.0):
        return (torch.randn(shape, device=DEV, generator=self.g) * s + add).to(torch.bfloat16)

    def ids(self, vocab, *shape):
        return torch.randint(0, vocab, shape, dtype=torch.int32, device=DEV, generator=self.g)

    def host(self):
        """A generator for small plans made on the host (page tables, lengths)."""
        return random.Random(int(torch.randint(0, 1 << 30, (1,), device=DEV, generator=self.g).item()))


_rope = {}


def rope_tables(n):
    """llama3 cos/sin tables [n, 32] (theta 500000, factor 32, low 1, high 4, original context 8192)."""
    if n not in _rope:
        inv = torch.pow(torch.tensor(500000.0, dtype=D64), torch.arange(32, dtype=D64) * 2 / 64)
        f, wl = 1 / inv, 2 * math.pi * inv
        a = (8192.0 / wl - 1) / 3
        f = torch.where(wl < 2048, f, torch.where(wl > 8192, f / 32, (1 - a) * (f / 32) + a * f))
        th = torch.arange(n, dtype=D64)[:, None] * f[None]
        _rope[n] = (th.cos().float().to(DEV), th.sin().float().to(DEV))
    return _rope[n]


def linear_inputs(c, r):
    return dict(a=r.s8(c["M"], c["K"]), s=r.uniform(0.005, 0.05, c["M"]), w=r.s8(c["N"], c["K"]), sc=r.uniform(0.001, 0.01, c["N"]))


def mlp_inputs(c, r, D=2048, ff=8192):
    return dict(x=r.normal(c["M"], D), gamma=1 + 0.02 * r.normal(D), w_gu=r.s8(2 * ff, D), s_gu=r.uniform(0.5, 1.5, 2 * ff) / (73 * D ** 0.5),
                w_d=r.s8(D, ff), s_d=r.uniform(0.5, 1.5, D) / (73 * ff ** 0.5))


def mha_prefill_inputs(c, r):
    B, S, H, G = c["B"], c["S"], c["heads"], c["kv_heads"]
    cos, sin = rope_tables(S)
    return dict(q=r.s8(B, S, H, 64), qs=r.uniform(0.005, 0.05, B, S, H), k=r.s8(B, S, G, 64), ks=r.uniform(0.005, 0.05, B, S, G), v=r.s8(B, S, G, 64),
                vs=r.uniform(0.005, 0.05, B, S, G), cos=cos, sin=sin, a_s=torch.full((H,), 0.05 / 255, device=DEV))


def mha_decode_inputs(c, r):
    B, H, G = c["B"], c["heads"], c["kv_heads"]
    rng = r.host()
    ctx = [rng.randint(c["lo"], c["hi"]) for _ in range(B)]
    pages = [n // 64 + 1 for n in ctx]
    order = list(range(sum(pages) + 3))
    rng.shuffle(order)
    width = max(pages)
    table, at = [], 0
    for p in pages:
        table.append(order[at:at + p] + [0] * (width - p))
        at += p
    P = len(order)
    cos, sin = rope_tables(max(ctx) + 2)
    return dict(ctx=torch.tensor(ctx, dtype=torch.int32, device=DEV), table=torch.tensor(table, dtype=torch.int32, device=DEV), pages=P, max_ctx=max(ctx) + 1,
                q=r.s8(B, H, 64), qs=r.uniform(0.005, 0.05, B, H), k=r.s8(B, G, 64), ks=r.uniform(0.005, 0.05, B, G), v=r.s8(B, G, 64),
                vs=r.uniform(0.005, 0.05, B, G), cos=cos, sin=sin, a_s=torch.full((H,), 0.05 / 255, device=DEV),
                pool_k=r.s8(P, G, 64, 64), pool_ks=r.uniform(0.005, 0.05, P, G, 64), pool_v=r.s8(P, G, 64, 64), pool_vs=r.uniform(0.005, 0.05, P, G, 64))


def llama_weights(r, z):
    """One layer's tensors after another, then the head's. Scales as of weights of variance 1 / inputs (queries and keys a little less)."""
    D, ff, Q, KV = z["width"], z["ff"], z["heads"] * 64, z["kv_heads"] * 64
    scale = lambda n, k, gain=1.0: r.uniform(0.5, 1.5, n) * (gain / (73 * k ** 0.5))
    for i in range(z["layers"]):
        yield i, dict(wq=r.s8(Q, D), wk=r.s8(KV, D), wv=r.s8(KV, D), wo=r.s8(D, Q), wg=r.s8(ff, D), wu=r.s8(ff, D), wd=r.s8(D, ff),
                      sq=scale(Q, D, 0.9), sk=scale(KV, D, 0.9), sv=scale(KV, D), so=scale(D, Q), sg=scale(ff, D), su=scale(ff, D), sd=scale(D, ff),
                      gamma0=1 + 0.02 * r.normal(D), gamma1=1 + 0.02 * r.normal(D), a_s=torch.full((z["heads"],), 0.05 / 255, device=DEV))
    yield None, dict(lm_w=r.s8(z["vocab"], D), lm_s=r.uniform(0.5, 1.5, z["vocab"]) / 73, gamma_final=1 + 0.02 * r.normal(D))


def llama_model(r, max_batch, max_prefill, max_ctx):
    z = SIZES["llama"]
    m = F.Model(z["layers"], z["width"], z["heads"], z["kv_heads"], z["ff"], z["vocab"], max_batch, max_prefill, max_ctx)
    cos, sin = rope_tables(max_ctx + 1)
    for i, w in llama_weights(r, z):
        if i is None:
            m.load_head(w["lm_w"], w["lm_s"], w["gamma_final"], cos, sin)
        else:
            m.load_layer(i, **w)
    return m


def family_config(family, z):
    """config.json of a model of sizes z: Pibidra with windowed attention in every layer; Sabisun with state-space mixers in three
    of four layers and attention in the rest, every second one of these with the keys and values of the one before."""
    layers, last = [], None
    for i in range(z["layers"]):
        mlp = {"kind": "dense", "ff": z["ff"]}
        m = dict(heads=z["heads"], kv_heads=z["kv_heads"], dim=z["dim"], vdim=z["dim"], mask={"size": z["window"]}, scale=z["dim"] ** -0.5)
        if family == "Pibidra":
            m.update(bias_max=z["window"], softcap=30.0)
        elif i % 4 != 3:
            layers.append({"type": "mamba2", "mlp": mlp, "mixer": dict(heads=2 * z["width"] // 64, vdim=64, state=128, groups=8, conv=4, norm_groups=8)})
            continue
        else:
            m["mask"]["keep_first"] = 4
            if last is not None:
                m["kv_from"], last = last, None
            else:
                last = i
        layers.append({"type": "attention", "mixer": m, "mlp": mlp})
    c = {"architecture": family, "layers": layers, "norm": {"eps": 1e-5}, "vocab": z["vocab"], "width": z["width"]}
    if family == "Pibidra":
        c["embedding"] = {"scale": 4.0}
    else:
        c.update(logit_scale=z["width"] ** -0.5, residual_mult=0.3, streams=2)
    return c


def family_tensors(r, cfg, z):
    """(name, tensor) of every weight. The next token is clear, as it is after training: the output rows of Pibidra are the
    embeddings of a permutation of the ids, and Sabisun, whose embeddings are tied, repeats."""
    D, V = z["width"], z["vocab"]
    embed = r.bf16(V, D)
    yield "embed", embed
    if cfg["architecture"] == "Pibidra":
        head = torch.empty_like(embed)
        head[permutation(V)] = embed
        yield "head", (head.float() * D ** -0.5).to(torch.bfloat16)
        yield "final.norm", r.bf16(D, s=0.1)
    else:
        yield "final.norm", r.bf16(D, s=0.1, add=1.0)
    for i, l in enumerate(cfg["layers"]):
        p, m, ff = "l%d." % i, l["mixer"], l["mlp"]["ff"]
        if cfg["architecture"] == "Pibidra":
            for n in ("norm1", "norm1b", "norm2", "norm2b"):
                yield p + n, r.bf16(D, s=0.1)
        else:
            n = cfg["streams"]
            for q in "12":
                yield p + "norm" + q, r.bf16(D, s=0.1, add=1.0)
                yield p + "hc" + q + ".in", r.bf16(n, s=0.1, add=0.5)
                yield p + "hc" + q + ".out", r.bf16(n, s=0.1, add=1.0)
                yield p + "hc" + q + ".mix", (torch.eye(n, device=DEV) + 0.02 * r.normal(n, n)).to(torch.bfloat16)
        if l["type"] == "mamba2":
            H, inner = m["heads"], m["heads"] * m["vdim"]
            ch = inner + 2 * m["groups"] * m["state"]
            yield p + "mix.in", r.bf16(inner + ch + H, D, s=D ** -0.5)
            yield p + "mix.conv", r.bf16(ch, m["conv"], s=0.5)
            yield p + "mix.conv.b", r.bf16(ch, s=0.1)
            yield p + "mix.dt_bias", r.bf16(H, add=-3.0)
            yield p + "mix.A_log", r.bf16(H)
            yield p + "mix.D", r.bf16(H, s=0.1, add=1.0)
            yield p + "mix.norm", r.bf16(inner, s=0.1, add=1.0)
            yield p + "mix.o", r.bf16(D, inner, s=inner ** -0.5)
        else:
            H, G, d = m["heads"], m["kv_heads"], m["dim"]
            yield p + "mix.q", r.bf16(H * d, D, s=D ** -0.5)
            if "kv_from" not in m:
                yield p + "mix.k", r.bf16(G * d, D, s=D ** -0.5)
                yield p + "mix.v", r.bf16(G * d, D, s=D ** -0.5)
            yield p + "mix.o", r.bf16(D, H * d, s=(H * d) ** -0.5)
            if cfg["architecture"] == "Pibidra":
                for n, w in (("q", H), ("k", G), ("v", G)):
                    yield p + "mix." + n + ".b", r.bf16(w * d, s=0.1)
                yield p + "mix.q.norm", r.bf16(H * d, s=0.1, add=1.0)
                yield p + "mix.k.norm", r.bf16(G * d, s=0.1, add=1.0)
                yield p + "mix.rel", r.bf16(32, H, s=0.5)
                yield p + "mix.g", r.bf16(H * d, D, s=D ** -0.5)
            else:
                yield p + "mix.sink", r.bf16(H)
        if cfg["architecture"] == "Pibidra":
            yield p + "mlp.gate", r.bf16(ff, D, s=D ** -0.5)
        yield p + "mlp.up", r.bf16(ff, D, s=D ** -0.5)
        yield p + "mlp.down", r.bf16(D, ff, s=ff ** -0.5)


def permutation(V):
    """id -> the id that follows it: an affine map without a common factor."""
    a = 7919
    while math.gcd(a, V) != 1:
        a += 2
    return (torch.arange(V, device=DEV) * a + 4242) % V


def family_model(c, r, max_prefill, max_ctx):
    z = SIZES[c["size"]]
    cfg = family_config(c["family"], z)
    m = F.Model.adopt(models.create(cfg, c["B"], max_prefill, max_ctx, c["dtype"]))
    for name, t in family_tensors(r, cfg, z):
        m.load_tensor(name, t)
    return m


# ------------------------------------------------------------------------------------------------- the passes
def prepare(case, seed):
    c, r = case, Source(seed)
    kind = c["kind"]
    if kind == "linear":
        s = linear_inputs(c, r)
    elif kind == "mlp":
        s = mlp_inputs(c, r)
    elif kind == "mha_prefill":
        s = mha_prefill_inputs(c, r)
    elif kind == "mha_decode":
        s = mha_decode_inputs(c, r)
        cache = F.KVCache(1, s["pages"], c["kv_heads"])
        for pool, name in zip(cache.pools(0), ("pool_k", "pool_ks", "pool_v", "pool_vs")):
            pool.copy_(s.pop(name))
        s["cache"] = cache
    elif kind == "llama_prompt":
        ids = r.ids(SIZES["llama"]["vocab"], c["B"], c["S"])
        s = dict(ids=ids, model=llama_model(r, c["B"], c["S"], c["S"] + 64))
    elif kind == "llama_request":
        ids = r.ids(SIZES["llama"]["vocab"], c["B"], c["S"])
        rnd = r.uniform(0.0, 1.0, c["new"], c["B"])
        s = dict(ids=ids.cpu().pin_memory(), model=llama_model(r, c["B"], c["S"], c["S"] + c["new"]), new=c["new"])
        if c["top_k"]:
            s["model"].set_sampling(32, c["top_k"], rnd)
    else:
        ids = r.ids(SIZES[c["size"]]["vocab"], c["B"], c["S"])
        new = c.get("new", 0)
        s = dict(ids=ids if not new else ids.cpu().pin_memory(), model=family_model(c, r, c["S"], c["S"] + new + 1), new=new)
    s["case"] = c
    return s


def run(s):
    c = s["case"]
    kind = c["kind"]
    if kind == "linear":
        return F.pref_Linear_Layer_i8xi8(s["a"], s["s"], s["w"], s["sc"])[1]
    if kind == "mlp":
        return F.dec_MLP_block(s["x"], s["gamma"], s["w_gu"], s["s_gu"], s["w_d"], s["s_d"])
    if kind == "mha_prefill":
        return F.MHA_i8xi8_Prefilling(s["q"], s["qs"], s["k"], s["ks"], s["v"], s["vs"], s["cos"], s["sin"], s["a_s"])[0]
    if kind == "mha_decode":
        return F.MHA_i8xi8_Decoding(s["cache"], 0, s["q"], s["qs"], s["k"], s["ks"], s["v"], s["vs"], s["cos"], s["sin"], s["a_s"], s["table"], s["ctx"],
                                    s["max_ctx"])[0]
    m, B = s["model"], c["B"]
    if kind in ("llama_prompt", "family_prompt"):
        m.reset()
        logits, first = m.extend(s["ids"], want=[b * c["S"] + c["S"] - 1 for b in range(B)], next_token=True)
        return dict(first=first, logits=logits)
    tokens = m.generate_host(s["ids"], s["new"])
    V = SIZES[c.get("size", "llama")]["vocab"]
    # the last step's logits beside all tokens, in a tensor that outlives the model's own buffer
    return dict(tokens=tokens, logits=m.buffer(1, (B, V), torch.float32).clone())


# ------------------------------------------------------------------------------------------------- what a pass cannot do without
def layer_work(c):
    """(multiply-adds per token in the layers' products, weight bytes of the layers, bytes of one cached token, multiply-adds per
    key and query, of all layers, attention layers, head size of the vocabulary product in bytes)."""
    z = SIZES[c.get("size", "llama")]
    D, H, G, d, ff, V, L = (z[k] for k in ("width", "heads", "kv_heads", "dim", "ff", "vocab", "layers"))
    if c["kind"].startswith("llama"):
        w = D * (H + 2 * G) * d + H * d * D + 3 * D * ff
        return dict(w=L * w, wbytes=L * w, kv=L * G * 136, pair=L * H * 2 * d, head=V * D, width=1)
    es = 2
    if c["family"] == "Pibidra":
        w = D * (2 * H + 2 * G) * d + H * d * D + 3 * D * ff
        return dict(w=L * w, wbytes=es * L * w, kv=es * L * G * 2 * d, pair=L * H * 2 * d, head=V * D, width=es)
    inner = 2 * D
    n_att = sum(1 for i in range(L) if i % 4 == 3)
    own = (n_att + 1) // 2
    ssm = D * (2 * inner + 2 * 8 * 128 + inner // 64) + inner * D + 2 * inner * 128
    w = (L - n_att) * ssm + n_att * (2 * D * H * d) + own * 2 * D * G * d + L * 2 * D * ff
    return dict(w=w, wbytes=es * (w - (L - n_att) * 2 * inner * 128), kv=es * own * G * 2 * d, pair=n_att * H * 2 * d, head=V * D, width=es,
                state=(L - n_att) * inner * 128 * 8)


def work(case):
    c, kind = case, case["kind"]
    if kind == "linear":
        M, N, K = c["M"], c["N"], c["K"]
        return dict(bytes=M * K + N * K + 4 * (M + N + M * N), flops=2 * M * N * K)
    if kind == "mlp":
        M, D, ff = c["M"], 2048, 8192
        return dict(bytes=3 * D * ff + 4 * (2 * ff + 2 * D) + 8 * M * D, flops=2 * M * 3 * D * ff)
    if kind == "mha_prefill":
        B, S, H, G = c["B"], c["S"], c["heads"], c["kv_heads"]
        return dict(bytes=B * S * (H + 2 * G) * 68 + 4 * B * S * H * 64, flops=4 * B * H * 64 * S * (S + 1) // 2)
    if kind == "mha_decode":
        rows = c["B"] * ((c["lo"] + c["hi"]) / 2 + 1)              # the expected number of cached tokens
        return dict(bytes=rows * c["kv_heads"] * 136 + c["B"] * c["heads"] * 64 * 5, flops=4 * rows * c["heads"] * 64)
    w, B, S, new = layer_work(c), c["B"], c["S"], c.get("new", 0)
    win = SIZES[c.get("size", "llama")]["window"] if kind.startswith("family") else S + new
    seen = lambda n: sum(min(i + 1, win) for i in range(n))        # keys of the first n positions
    steps = max(0, new - 1)
    flops = 2 * B * (w["w"] * (S + steps) + w["pair"] * seen(S + steps) + w["head"] * (1 + steps))
    kv = w["kv"] * sum(min(S + i + 1, win) for i in range(steps)) + w.get("state", 0) * steps
    out = 4 * SIZES[c.get("size", "llama")]["vocab"]
    return dict(bytes=(w["wbytes"] + w["head"] * w["width"]) * (1 + steps) + B * (kv + out + w["kv"] * min(S, win)), flops=flops)


def tolerance(case):
    """Whole-number operators differ by the roundings of their scales alone; behind a quantiser a value may fall on the other side
    of a step where a sum is formed in another order. The families keep activations in 16 bits."""
    kind = case["kind"]
    if kind == "linear":
        return {"rel": 1e-6}
    if kind == "mlp":
        return {"rel": 5e-3}
    if kind.startswith("mha"):
        return {"rel": 5e-3}
    if kind.startswith("llama"):
        return {"rel": 3e-2, "differ": 1e-2}
    return {"rel": 2e-2 if case["dtype"] == "bfloat16" else 2e-4, "differ": 1e-2}


# ------------------------------------------------------------------------------------------------- the same in 64 bits
def round_away(x):
    return torch.sign(x) * torch.floor(x.abs() + 0.5)


def quantise(x):
    """Per-row symmetric int8: (values, scale)."""
    s = x.abs().amax(-1, keepdim=True) / 127
    s = torch.where(s == 0, torch.ones_like(s), s)
    return round_away(x / s), s


def hadamard(x):
    n, shape = x.shape[-1], x.shape
    h = 1
    while h < n:
        x = x.reshape(*shape[:-1], n // (2 * h), 2, h)
        x = torch.stack((x[..., 0, :] + x[..., 1, :], x[..., 0, :] - x[..., 1, :]), -2)
        h *= 2
    return x.reshape(shape)


def rms(x, eps=1e-5):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def product(x, w, scale):
    """Quantised rows x times the int8 rows w, in 64 bits."""
    q, s = quantise(x)
    return (q @ w.to(D64).T) * s * scale.to(D64)


def mlp64(x, gamma, wg, wu, sg, su, wd, sd):
    h = rms(x) * gamma.to(D64)
    g, u = product(h, wg, sg), product(h, wu, su)
    act = g / (1 + torch.exp(-g)) * u
    return x + product(hadamard(act) / math.sqrt(act.shape[-1]), wd, sd)


def rotate(x, pos, cos, sin):
    """x [.., T, heads, 64] at positions pos [.., T]: rotation, then the 64-point Hadamard transform over 8, then int8 per head."""
    c, s = cos.to(D64)[pos][..., None, :], sin.to(D64)[pos][..., None, :]
    a, b = x[..., :32], x[..., 32:]
    return quantise(hadamard(torch.cat((a * c - b * s, a * s + b * c), -1)) / 8)


def attend(q, qs, k, ks, v, vs, a_s, visible):
    """q [H,T,64], k, v [H,S,64] whole numbers with scales; visible [T,S]. Probabilities go to 8 bits against a_s [H]."""
    x = (q @ k.transpose(1, 2)) * qs * ks.transpose(1, 2) * 0.125
    p = torch.softmax(x.masked_fill(~visible, float("-inf")), -1)
    a = a_s.to(D64)[:, None, None]
    u = torch.clamp(torch.floor(p * vs.transpose(1, 2) / a + 0.5), max=255)
    return (u @ v) * a


def mha_prefill64(q, k, v, v_scale, cos, sin, a_s, pos):
    """One sequence: q [S,H,64], k [S,G,64] before the rotation, v whole numbers with scale [S,G,1] -> [S,H*64]."""
    S, H, G = q.shape[0], q.shape[1], k.shape[1]
    qi, qs = rotate(q, pos, cos, sin)
    ki, ks = rotate(k, pos, cos, sin)
    vis = torch.ones(S, S, dtype=torch.bool, device=DEV).tril()
    out, n = torch.empty(S, H, 64, dtype=D64, device=DEV), H // G
    t = lambda x: x.transpose(0, 1)
    for g in range(G):
        h = slice(g * n, (g + 1) * n)
        e = lambda x: t(x[:, g:g + 1]).expand(n, -1, -1)
        out[:, h] = t(attend(t(qi[:, h]), t(qs[:, h]), e(ki), e(ks), e(v), e(v_scale), a_s[h], vis))
    return out.reshape(S, H * 64)


def llama64(ids, r):
    """Logits of the last position."""
    z, (B, S) = SIZES["llama"], ids.shape
    H, G, D = z["heads"], z["kv_heads"], z["width"]
    cos, sin = rope_tables(S)
    layers = list(llama_weights(r, z))
    head = layers[-1][1]
    lm = lambda rows: head["lm_w"][rows].to(D64) * head["lm_s"][rows].to(D64)[:, None]
    x = [lm(ids[b].long()) for b in range(B)]
    pos = torch.arange(S, device=DEV)
    for _, w in layers[:-1]:
        w = {k: v.to(D64) if k[0] == "w" else v for k, v in w.items()}
        for b in range(B):
            h = rms(x[b]) * w["gamma0"].to(D64)
            q, k, v = product(h, w["wq"], w["sq"]), product(h, w["wk"], w["sk"]), product(h, w["wv"], w["sv"])
            vi, vs = quantise(v.reshape(S, G, 64))
            att = mha_prefill64(q.reshape(S, H, 64), k.reshape(S, G, 64), vi, vs, cos, sin, w["a_s"], pos)
            x[b] = mlp64(x[b] + product(att, w["wo"], w["so"]), w["gamma1"], w["wg"], w["wu"], w["sg"], w["su"], w["wd"], w["sd"])
    return torch.cat([product(rms(t[-1:]) * head["gamma_final"].to(D64), head["lm_w"], head["lm_s"]) for t in x])


def window_attention64(q, k, v, scale, window, keep, softcap, bias, sink):
    """One sequence: q [S,H,d], k, v [S,G,d]; bias [distance,H] or None; sink [H] (scores) or None -> [S,H*d]."""
    S, H, G = q.shape[0], q.shape[1], k.shape[1]
    dist = torch.arange(S, device=DEV)[:, None] - torch.arange(S, device=DEV)[None]
    vis = (dist >= 0) & ((dist < window) | (torch.arange(S, device=DEV)[None] < keep))
    out = torch.empty(S, H, v.shape[2], dtype=D64, device=DEV)
    for h in range(H):
        g = h // (H // G)
        x = q[:, h] @ k[:, g].T * scale
        if softcap:
            x = softcap * torch.tanh(x / softcap)
        if bias is not None:
            x = x + bias[dist.clamp(0, bias.shape[0] - 1), h]
        x = x.masked_fill(~vis, float("-inf"))
        x = torch.cat((x, sink[h].expand(S, 1)), 1)
        out[:, h] = torch.softmax(x, -1)[:, :S] @ v[:, g]
    return out.reshape(S, -1)


def distance_rows(table, bias_max, n):
    """table [rows,H] by bucketed distance -> [n,H]: exact up to half the rows, logarithmic up to bias_max after it."""
    rows, half = table.shape[0], table.shape[0] // 2
    at = [i if i < half else min(rows - 1, half + math.floor(math.log(i / half) / math.log(bias_max / half) * (rows - half) + 1e-9)) for i in range(n)]
    return table[torch.tensor(at, device=DEV)]


def state_space64(p, m, w, pre, eps):
    """One sequence through a Mamba-2 form mixer between its projections: p [S, z|x|B|C|dt] -> [S, inner]."""
    S, H, P, N, G = p.shape[0], m["heads"], m["vdim"], m["state"], m["groups"]
    inner, taps = H * P, m["conv"]
    z, u, dt = p[:, :inner], p[:, inner:2 * inner + 2 * G * N], p[:, 2 * inner + 2 * G * N:]
    back = torch.cat((torch.zeros(taps - 1, u.shape[1], dtype=D64, device=DEV), u))
    y = w(pre + "conv.b") + sum(w(pre + "conv")[:, i] * back[i:i + S] for i in range(taps))
    y = y * torch.sigmoid(y)
    x, Bm, Cm = y[:, :inner].reshape(S, H, P), y[:, inner:inner + G * N].reshape(S, G, N), y[:, inner + G * N:].reshape(S, G, N)
    dt = torch.nn.functional.softplus(dt + w(pre + "dt_bias"), threshold=1e9)
    run = torch.cumsum(-torch.exp(w(pre + "A_log")) * dt, 0)       # log of the decay up to each token
    out, low = torch.empty(S, H, P, dtype=D64, device=DEV), torch.ones(S, S, dtype=torch.bool, device=DEV).tril()
    for h in range(H):
        g = h // (H // G)
        decay = torch.exp((run[:, None, h] - run[None, :, h]).masked_fill(~low, float("-inf")))
        out[:, h] = (Cm[:, g] @ Bm[:, g].T * decay * dt[None, :, h]) @ x[:, h] + w(pre + "D")[h] * x[:, h]
    y = out.reshape(S, inner) * (z * torch.sigmoid(z))
    return rms(y.reshape(S, m["norm_groups"], -1), eps).reshape(S, inner) * w(pre + "norm")


def family64(c, r, ids):
    """Logits [B,V] of the last position of the sequences ids [B,S]."""
    z = SIZES[c["size"]]
    cfg = family_config(c["family"], z)
    t = dict(family_tensors(r, cfg, z))
    w = lambda n: t[n].to(D64)
    B, S = ids.shape
    eps, pib = cfg["norm"]["eps"], c["family"] == "Pibidra"
    gain = lambda n: w(n) + (1 if pib else 0)
    flat = ids.reshape(-1).long()
    x = t["embed"][flat].to(D64)
    xs = x * cfg["embedding"]["scale"] if pib else torch.stack([x] * cfg["streams"])
    rows = lambda y, f: torch.cat([f(y[b * S:(b + 1) * S], b) for b in range(B)])
    kv = {}
    for i, l in enumerate(cfg["layers"]):
        p, m = "l%d." % i, l["mixer"]
        pre = p + "mix."

        def mixer(h):
            if l["type"] == "mamba2":
                return rows(h @ w(pre + "in").T, lambda y, b: state_space64(y, m, w, pre, eps)) @ w(pre + "o").T
            H, G, d = m["heads"], m["kv_heads"], m["dim"]
            q = h @ w(pre + "q").T
            if "kv_from" in m:
                k, v = kv[m["kv_from"]]
            else:
                k, v = h @ w(pre + "k").T, h @ w(pre + "v").T
                if pib:
                    k, v = rms(k + w(pre + "k.b"), eps) * w(pre + "k.norm"), v + w(pre + "v.b")
                kv[i] = k, v
            bias, sink = None, None
            if pib:
                q = rms(q + w(pre + "q.b"), eps) * w(pre + "q.norm")
                bias, sink = distance_rows(w(pre + "rel"), m["bias_max"], min(S, m["mask"]["size"])), torch.zeros(H, dtype=D64, device=DEV)
            else:
                sink = w(pre + "sink")
            o = rows(q, lambda y, b: window_attention64(y.reshape(S, H, d), k[b * S:(b + 1) * S].reshape(S, G, d), v[b * S:(b + 1) * S].reshape(S, G, d), m["scale"],
                                                        m["mask"]["size"], m["mask"].get("keep_first", 0), m.get("softcap"), bias, sink))
            if pib:
                o = o * torch.sigmoid(h @ w(pre + "g").T)
            return o @ w(pre + "o").T

        def feed_forward(h):
            u = h @ w(p + "mlp.up").T
            if pib:
                u = torch.nn.functional.gelu(h @ w(p + "mlp.gate").T, approximate="tanh") * u
            else:
                u = torch.clamp(u, min=0) ** 2
            return u @ w(p + "mlp.down").T

        for q, sub in (("1", mixer), ("2", feed_forward)):
            if pib:
                xs = xs + rms(sub(rms(xs, eps) * gain(p + "norm" + q)), eps) * gain(p + "norm" + q + "b")
            else:
                a, o, mix = w(p + "hc" + q + ".in"), w(p + "hc" + q + ".out"), w(p + "hc" + q + ".mix")
                y = sub(rms((a[:, None, None] * xs).sum(0), eps) * gain(p + "norm" + q))
                xs = torch.einsum("st,srd->trd", mix, xs) + cfg["residual_mult"] * o[:, None, None] * y
    last = (xs if pib else xs.sum(0))[S - 1::S]
    out = rms(last, eps) * gain("final.norm") @ w("head" if pib else "embed").T
    return out if pib else out * cfg["logit_scale"]


def exact(case, seed):
    c, r = case, Source(seed)
    kind = c["kind"]
    if kind == "linear":
        s = linear_inputs(c, r)
        return (s["a"].to(D64) @ s["w"].to(D64).T) * s["s"].to(D64)[:, None] * s["sc"].to(D64)
    if kind == "mlp":
        s = mlp_inputs(c, r)
        (wg, wu), (sg, su) = s["w_gu"].chunk(2), s["s_gu"].chunk(2)
        return mlp64(s["x"].to(D64), s["gamma"], wg, wu, sg, su, s["w_d"], s["s_d"])
    if kind == "mha_prefill":
        s = mha_prefill_inputs(c, r)
        pos = torch.arange(c["S"], device=DEV)
        f = lambda t, sc: t.to(D64) * sc.to(D64)[..., None]
        return torch.stack([mha_prefill64(f(s["q"][b], s["qs"][b]), f(s["k"][b], s["ks"][b]), s["v"][b].to(D64), s["vs"][b].to(D64)[..., None], s["cos"], s["sin"],
                                          s["a_s"], pos) for b in range(c["B"])])
    if kind == "mha_decode":
        s = mha_decode_inputs(c, r)
        H, G, n = c["heads"], c["kv_heads"], c["heads"] // c["kv_heads"]
        out = []
        for b, ctx in enumerate(s["ctx"].tolist()):
            at = s["table"][b, :ctx // 64 + 1].long()
            pos = torch.tensor([ctx], device=DEV)
            new = lambda t, sc: rotate((t[b].to(D64) * sc[b].to(D64)[:, None])[None], pos, s["cos"], s["sin"])
            (qi, qs), (ki, ks) = new(s["q"], s["qs"]), new(s["k"], s["ks"])
            rows = lambda pool: pool[at].transpose(1, 2).reshape(len(at) * 64, G, -1)[:ctx].to(D64)
            k = torch.cat((rows(s["pool_k"]), ki)).transpose(0, 1)
            v = torch.cat((rows(s["pool_v"].transpose(2, 3)), s["v"][b].to(D64)[None])).transpose(0, 1)
            kss = torch.cat((rows(s["pool_ks"][..., None]), ks)).transpose(0, 1)
            vss = torch.cat((rows(s["pool_vs"][..., None]), s["vs"][b].to(D64)[None, :, None])).transpose(0, 1)
            e = lambda t: t.repeat_interleave(n, 0)
            vis = torch.ones(1, ctx + 1, dtype=torch.bool, device=DEV)
            out.append(attend(qi[0][:, None], qs[0][:, None], e(k), e(kss), e(v), e(vss), s["a_s"], vis).reshape(H * 64))
        return torch.stack(out)
    if kind == "llama_prompt":
        ids = r.ids(SIZES["llama"]["vocab"], c["B"], c["S"])
        return dict(first=None, logits=llama64(ids, r))
    if kind == "llama_request":
        return None                        # a chain of choices between near-equal logits of random weights, each step after the one before
    V = SIZES[c["size"]]["vocab"]
    ids = r.ids(V, c["B"], c["S"])
    if kind == "family_prompt":
        return dict(first=None, logits=family64(c, r, ids))
    follows = permutation(V) if c["family"] == "Pibidra" else torch.arange(V, device=DEV)
    tokens = [follows[ids[:, -1].long()]]
    while len(tokens) < c["new"]:
        tokens.append(follows[tokens[-1]])
    tokens = torch.stack(tokens, 1).to(torch.int32)
    return dict(tokens=None, logits=family64(c, r, torch.cat((ids, tokens[:, :-1]), 1)))
