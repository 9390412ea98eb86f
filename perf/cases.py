"""Workloads this library is timed on, each through the entry points a program calls, with the same results in 64 bits.

    moe        one mixture-of-experts layer (monoserve_b200/moe.py): decode batches of one token and more, prompts; bf16 and
               e4m3 weights; every expert in HBM, or most of them read in place from pinned host memory
    attention  paged grouped-query attention (monoserve_b200/attention.py): decode rows over long contexts, prompts, portions
               of prompts behind a past
    decoder    a mixture-of-experts decoder as lane programs on the fabric (monoserve_b200/model.py)
    layers     the layer-list decoders, also as lane programs (monoserve_b200/layer_list.py): Sinotar (selective scan, matrix
               memory, latent attention) and Teganex (gated linear attention, attention beside a gated delta rule)

Sizes are those of the benchmarks and tests (bench.py, monoserve_b200/benchmarks/), or odd ones of the same ranges.
A lane's programs are kept, as the serving loop keeps a decode batch's, and run once a pass: publish, start, wait, stop.
"""
import math
import struct
import types

import numpy as np
import torch

SHAPES = {   # of one mixture-of-experts layer
    "30b": dict(H=2048, I=768, E=128, K=8, scoring="softmax", fp8=False),     # the layer of bench.py
    "air": dict(H=4096, I=1408, E=128, K=8, scoring="sigmoid", fp8=True),     # benchmarks/glm_layer.py
}
DECODER = dict(H=2048, I=768, E=128, K=8, hq=32, hkv=4, vocab=32768, eps=1e-6, theta=1e6)
WIDTH, VOCAB, EPS, PAGE = 2048, 32768, 1e-5, 16
BF16 = torch.bfloat16


def listed():
    return [
        # one sequence being decoded: nothing but latency and the eight experts it picks
        dict(name="moe_token", kind="moe", shape="30b", tokens=1, hosted=0, skew=0.0),
        # a full decode batch of a server, routing as skewed as in bench.py
        dict(name="moe_decode", kind="moe", shape="30b", tokens=256, hosted=0, skew=1.1),
        # four prompts of 2048 tokens in one pass
        dict(name="moe_prompts", kind="moe", shape="30b", tokens=8192, hosted=0, skew=0.0),
        # the 8-bit layer under a decode batch
        dict(name="moe_decode_8bit", kind="moe", shape="air", tokens=64, hosted=0, skew=0.0),
        # three quarters of the experts in host memory: the link bounds it
        dict(name="moe_hosted", kind="moe", shape="30b", tokens=64, hosted=96, skew=1.1),
        # decode attention of 128 sequences with mixed contexts
        dict(name="attention_decode", kind="attention", requests=128, rows=1, past_lo=512, past_hi=8192, hq=32, hkv=4, page=16),
        # prompt attention, four prompts
        dict(name="attention_prompts", kind="attention", requests=4, rows=2048, past_lo=0, past_hi=0, hq=32, hkv=4, page=16),
        # the decoder's two directions: ragged prompts, and one step of a decode batch
        dict(name="decoder_prompts", kind="decoder", layers=4, requests=4, rows=1024, past_lo=0, past_hi=0),
        dict(name="decoder_step", kind="decoder", layers=4, requests=32, rows=1, past_lo=512, past_hi=4096),
        # the layer-list decoders: prompts of both designs, one step of a decode batch
        dict(name="sinotar_prompts", kind="layers", design="Sinotar", requests=4, rows=1024, past=0),
        dict(name="teganex_prompts", kind="layers", design="Teganex", requests=4, rows=1024, past=0),
        dict(name="teganex_step", kind="layers", design="Teganex", requests=32, rows=1, past=300),
    ]


def _spread(rng, lo, hi):
    """A whole number of [lo, hi], spread over its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))))


def draw(rng):
    kind = rng.choice(["moe", "moe", "attention", "attention", "decoder", "layers", "layers"])
    if kind == "moe":
        hosted = rng.choice([0, 0, 0, 64, 96])
        shape = "30b" if hosted else rng.choice(["30b", "30b", "air"])
        most = 64 if hosted else 8192 if shape == "30b" else 2048
        return dict(kind=kind, shape=shape, tokens=_spread(rng, 1, most), hosted=hosted, skew=rng.choice([0.0, 0.6, 1.1]))
    if kind == "attention":
        hq, hkv = rng.choice([(32, 4), (32, 4), (96, 8), (16, 2)])
        case = dict(kind=kind, hq=hq, hkv=hkv, page=rng.choice([8, 16, 16, 64]))
        if rng.random() < 0.5:
            requests, hi = _spread(rng, 1, 96 if hkv == 8 else 128), _spread(rng, 64, 8192 if hkv < 8 else 4096)
            return dict(case, requests=requests, rows=1, past_lo=max(1, hi // 8), past_hi=hi)
        requests = rng.randint(1, 4)
        rows = _spread(rng, 20, 2048 // (2 if hq == 96 else 1) // (2 if requests > 2 else 1))
        return dict(case, requests=requests, rows=rows, past_lo=0, past_hi=rng.choice([0, 0, 700, 1000]))
    if kind == "decoder":
        if rng.random() < 0.5:
            return dict(kind=kind, layers=4, requests=_spread(rng, 1, 64), rows=1, past_lo=100, past_hi=_spread(rng, 200, 4096))
        return dict(kind=kind, layers=4, requests=rng.randint(1, 4), rows=_spread(rng, 40, 1000), past_lo=0, past_hi=0)
    design = rng.choice(["Sinotar", "Teganex"])
    if rng.random() < 0.4:
        return dict(kind=kind, design=design, requests=_spread(rng, 1, 32), rows=1, past=_spread(rng, 40, 300))
    return dict(kind=kind, design=design, requests=rng.randint(1, 4), rows=_spread(rng, 40, 1000), past=0)


# ------------------------------------------------------------------------------------------ what a case's sizes are
def lengths(case):
    """New tokens of each request: one each, or ragged prompts of up to `rows` tokens."""
    n = case["requests"]
    return [1] * n if case["rows"] == 1 else [max(1, case["rows"] - i * case["rows"] // (4 * n) - i) for i in range(n)]


def pasts(case):
    """Tokens of each request that are cached before the pass."""
    if "past" in case:
        return [case["past"] + i % 7 for i in range(case["requests"])] if case["past"] else [0] * case["requests"]
    lo, hi, n = case["past_lo"], case["past_hi"], case["requests"]
    return [lo + (i * 2654435761 % 4096) * (hi - lo) // 4096 for i in range(n)]


def generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def normal(g, *shape, scale=1.0, at=0.0):
    t = torch.empty(*shape, dtype=BF16, device="cuda").normal_(0.0, scale, generator=g)
    return t + at if at else t


def quantised(g, *shape):
    """e4m3 rows N(0, 0.02) and one fp32 scale per row."""
    w = torch.empty(*shape, device="cuda").normal_(0.0, 0.02, generator=g)
    s = w.abs().amax(-1) / 448
    w.div_(s[..., None])
    return w.to(torch.float8_e4m3fn).view(torch.uint8), s


def page_table(case, page, seed, more=1):
    """Block table [requests, stride] over shuffled pages (page 0 is the sink), and the number of pages."""
    need = [-(-(p + n + more) // page) for p, n in zip(pasts(case), lengths(case))]
    perm = np.random.default_rng(seed).permutation(sum(need)) + 1
    table, at = np.zeros((len(need), max(need)), dtype=np.int32), 0
    for i, n in enumerate(need):
        table[i, :n] = perm[at:at + n]
        at += n
    return table, sum(need) + 1


# ------------------------------------------------------------------------------------------ mixture-of-experts layer
def moe_data(case, seed):
    c, g, T = SHAPES[case["shape"]], generator(seed), case["tokens"]
    H, I, E = c["H"], c["I"], c["E"]
    d = types.SimpleNamespace(**c, bias=None, s13=None, s2=None)
    # column 0 of every activation row is one, its router weights a log prior: a Zipf-skewed choice of experts
    d.wr = normal(g, E, H, scale=H ** -0.5)
    rank = torch.empty(E, device="cuda")
    rank[torch.randperm(E, generator=g, device="cuda")] = torch.arange(1, E + 1, device="cuda", dtype=torch.float32)
    d.prior = -case["skew"] * torch.log(rank)
    d.wr[:, 0] = d.prior.to(BF16)
    d.x, d.x2 = normal(g, T, H), normal(g, T, H)
    d.x[:, 0] = 1.0
    if c["fp8"]:
        d.w13, d.s13 = torch.empty(E, 2 * I, H, dtype=torch.uint8, device="cuda"), torch.empty(E, 2 * I, device="cuda")
        d.w2, d.s2 = torch.empty(E, H, I, dtype=torch.uint8, device="cuda"), torch.empty(E, H, device="cuda")
        for e in range(0, E, 16):
            d.w13[e:e + 16], d.s13[e:e + 16] = quantised(g, 16, 2 * I, H)
            d.w2[e:e + 16], d.s2[e:e + 16] = quantised(g, 16, H, I)
        d.bias = torch.empty(E, device="cuda").normal_(0.0, 0.01, generator=g)
    else:
        d.w13, d.w2 = normal(g, E, 2 * I, H, scale=0.02), normal(g, E, H, I, scale=0.02)
    return d


def moe_prepare(case, seed):
    from monoserve_b200.moe import REGION_HOT, REGION_HOST, MoELayer
    d = moe_data(case, seed)
    E = d.E
    layer = MoELayer(d.H, d.I, E, d.K, case["tokens"], scoring=d.scoring, fp8=d.fp8)
    layer.set_router(d.wr, d.bias)
    if d.fp8:
        layer.set_scales(d.s13, d.s2)
    hot = torch.argsort(d.prior, descending=True, stable=True)[:E - case["hosted"]].sort().values
    table = torch.zeros(E, 2, dtype=torch.int32)
    table[:, 1] = torch.arange(E)
    if case["hosted"]:
        host = [torch.empty(w.shape, dtype=w.dtype, pin_memory=True) for w in (d.w13, d.w2)]
        for to, w in zip(host, (d.w13, d.w2)):
            to.copy_(w)
        layer.set_region(REGION_HOST, *host)
        d.w13, d.w2 = d.w13[hot], d.w2[hot]
    layer.set_region(REGION_HOT, layer.pack_w13(d.w13), d.w2, packed=True)
    hot = hot.cpu()
    table[hot, 0] = REGION_HOT
    table[hot, 1] = torch.arange(len(hot), dtype=torch.int32)
    layer.set_table(table)
    layer.set_plan(ctas=0, credits=8, form=64)
    return dict(kind="moe", layer=layer, x=d.x, x2=d.x2)


def routed(x, wr, bias, K, scoring):
    """(ids, weights) of the router in 64 bits."""
    logits = x @ wr.double().T
    score = logits.softmax(-1) if scoring == "softmax" else logits.sigmoid()
    ids = (score if bias is None else score + bias.double()).topk(K, -1).indices
    w = score.gather(1, ids)
    return ids, w / w.sum(-1, keepdim=True)


def experts_exact(x, ids, w, w13, w2, s13=None, s2=None):
    I, out = w2.shape[-1], torch.zeros_like(x)
    for e in range(w13.shape[0]):
        t, k = (ids == e).nonzero(as_tuple=True)
        if not len(t):
            continue
        a, b = w13[e], w2[e]
        if s13 is not None:
            a = a.view(torch.float8_e4m3fn).double() * s13[e].double()[:, None]
            b = b.view(torch.float8_e4m3fn).double() * s2[e].double()[:, None]
        y = x[t] @ a.double().T
        y = (torch.nn.functional.silu(y[:, :I]) * y[:, I:]) @ b.double().T
        out.index_add_(0, t, y * w[t, k][:, None])
    return out


def moe_exact(case, seed):
    d = moe_data(case, seed)
    x = d.x.double()
    ids, w = routed(x, d.wr, d.bias, d.K, d.scoring)
    return d.x2.double() + experts_exact(x, ids, w, d.w13, d.w2, d.s13, d.s2)


def moe_work(case):
    c, T = SHAPES[case["shape"]], case["tokens"]
    active = c["E"] * (1 - (1 - c["K"] / c["E"]) ** T)
    expert = 3 * c["H"] * c["I"]
    return dict(bytes=active * expert * (1 if c["fp8"] else 2) + 6.0 * T * c["H"] + 2.0 * c["E"] * c["H"],
                flops=2.0 * T * c["K"] * expert + 2.0 * T * c["H"] * c["E"])


# ------------------------------------------------------------------------------------------ paged attention
def attention_data(case, seed):
    g = generator(seed)
    table, pages = page_table(case, case["page"], seed, more=0)
    T = sum(lengths(case))
    q = normal(g, T, case["hq"], 128)
    k, v = (normal(g, pages, case["page"], case["hkv"], 128) for _ in range(2))
    info, row = [], 0
    for n, p in zip(lengths(case), pasts(case)):
        info.append((row, p, n, p + n))
        row += n
    return q, k, v, torch.from_numpy(table).cuda(), info


def attention_prepare(case, seed):
    from monoserve_b200.attention import AttentionPlan
    q, k, v, table, info = attention_data(case, seed)
    return dict(kind="attention", plan=AttentionPlan(info, case["hq"], case["hkv"]), args=(q, k, v, table))


def causal_exact(q, k, v, past, scale):
    """q [n, H, d], k [past + n, G, d], v [past + n, G, e], all in 64 bits."""
    n, H, _ = q.shape
    per, out = H // k.shape[1], []
    later = torch.arange(past + n, device=q.device)[None] > past + torch.arange(n, device=q.device)[:, None]
    for h in range(k.shape[1]):
        s = torch.einsum("nhd,md->hnm", q[:, h * per:(h + 1) * per], k[:, h]) * scale
        out.append(torch.einsum("hnm,me->nhe", s.masked_fill_(later, -math.inf).softmax(-1), v[:, h]))
    return torch.cat(out, 1)


def attention_exact(case, seed):
    q, k, v, table, info = attention_data(case, seed)
    out = []
    for i, (row, past, n, keys) in enumerate(info):
        pages = table[i, :-(-keys // case["page"])].long()
        kk, vv = (c[pages].flatten(0, 1)[:keys].double() for c in (k, v))
        out.append(causal_exact(q[row:row + n].double(), kk, vv, past, 128 ** -0.5))
    return torch.cat(out)


def pairs(case):
    return sum(n * p + n * (n + 1) / 2 for n, p in zip(lengths(case), pasts(case)))


def attention_work(case):
    T, keys = sum(lengths(case)), sum(n + p for n, p in zip(lengths(case), pasts(case)))
    return dict(bytes=keys * case["hkv"] * 512.0 + T * case["hq"] * 512.0, flops=4.0 * 128 * case["hq"] * pairs(case))


# ------------------------------------------------------------------------------------------ lane programs
class Lane:
    """A fabric and a lane on it, with the two copies of a program that take turns (a lane starts a program that is not the
    one it ran last)."""

    def __init__(self, make, case, seed, page=PAGE):
        from monoserve_b200.fabric import Fabric
        self.table, pages = page_table(case, page, seed)
        self.fab = Fabric(pool_bytes=160 << 20)
        lens, past = lengths(case), pasts(case)
        self.requests, self.past = len(lens), past
        rows = max(sum(lens), sum(past) if "past" in case and past[0] else 0)
        self.lane = make(self.fab, pages, page, rows, self.requests, self.table.shape[1])
        torch.cuda.synchronize()   # the lane's buffers are there before the fabric's own stream writes to them
        for i, row in enumerate(self.table):
            self.lane.set_pages(i, row.tolist())
        self.workers = self.fab.num_workers
        self.programs = []

    def once(self, handle):
        done = self.fab.iterations(0)
        self.fab.publish(map=[0] * self.workers, caps=[4], order=[0], programs=[handle])
        self.fab.start()
        self.fab.iteration_times(0, done, 1)
        self.fab.stop()

    def prompts(self, tokens):
        self.programs = [self.lane.build_prefill([(i, t, 0) for i, t in enumerate(tokens)]) for _ in range(2)]
        self.step = None

    def steps(self, tokens):
        """One decode step behind the cached tokens, of the given last tokens."""
        self.programs = [self.lane.build_decode(list(range(self.requests))) for _ in range(2)]
        self.step = [(self.lane.seq_len.data_ptr(), struct.pack(f"<{self.requests}i", *self.past)),
                     (self.lane.last_token.data_ptr(), struct.pack(f"<{self.requests}i", *tokens))]

    def run(self):
        for at, data in self.step or ():
            self.fab.write(at, data)
        self.programs.reverse()
        self.once(self.programs[0])
        return self.lane.logits


def token_ids(case, seed, vocab):
    """[past + new tokens of each request]."""
    rng = np.random.default_rng(seed + 1)
    return [rng.integers(0, vocab, size=p + n).tolist() for p, n in zip(pasts(case), lengths(case))]


# ------------------------------------------------------------------------------------------ mixture-of-experts decoder
def decoder_data(case, seed):
    c, g, L = types.SimpleNamespace(**DECODER), generator(seed), case["layers"]
    w = types.SimpleNamespace(embed=normal(g, c.vocab, c.H), lm_head=normal(g, c.vocab, c.H, scale=c.H ** -0.5),
                              final_norm=normal(g, c.H, scale=0.1, at=1.0))
    for name, n in (("in_norm", c.H), ("post_norm", c.H), ("q_norm", 128), ("k_norm", 128)):
        setattr(w, name, [normal(g, n, scale=0.1, at=1.0) for _ in range(L)])
    w.qkv = [normal(g, (c.hq + 2 * c.hkv) * 128, c.H, scale=c.H ** -0.5) for _ in range(L)]
    w.o = [normal(g, c.H, c.hq * 128, scale=(c.hq * 128) ** -0.5) for _ in range(L)]
    w.router = [normal(g, c.E, c.H, scale=c.H ** -0.5) for _ in range(L)]
    # one stack of experts in every layer: a stack is 1.2 GB, far more than the L2 holds from one layer to the next
    w.w13, w.w2 = normal(g, c.E, 2 * c.I, c.H, scale=0.02), normal(g, c.E, c.H, c.I, scale=0.02)
    _, pages = page_table(case, PAGE, seed)
    cached = [tuple(normal(g, pages, PAGE, c.hkv, 128) for _ in range(2)) for _ in range(L)] if case["rows"] == 1 else None
    return c, w, cached, token_ids(case, seed, c.vocab)


def decoder_prepare(case, seed):
    from monoserve_b200.model import KVCache, ModelLane, ModelWeights
    c, w, cached, tokens = decoder_data(case, seed)
    cfg = types.SimpleNamespace(hidden=c.H, intermediate=c.I, num_experts=c.E, top_k=c.K, num_layers=case["layers"],
                                num_heads=c.hq, num_kv_heads=c.hkv, head_dim=128, vocab=c.vocab, rope_theta=c.theta,
                                rms_eps=c.eps, rotary_dim=128)
    host = [torch.empty(t.shape, dtype=t.dtype, pin_memory=True) for t in (w.w13, w.w2)]
    for to, t in zip(host, (w.w13, w.w2)):
        to.copy_(t)
    del w.w13, w.w2
    w.host_w13, w.host_w2 = ([t] * case["layers"] for t in host)
    weights = ModelWeights(cfg, w)
    s = dict(kind="decoder")

    def make(fab, pages, page, rows, slots, stride):
        s["kv"] = KVCache(cfg, pages, page)
        return ModelLane(fab, 0, cfg, weights, s["kv"], max_tokens=max(rows, slots), max_slots=slots, bt_stride=stride, logit_rows=slots)
    s["lane"] = Lane(make, case, seed)
    if cached:
        for l, (k, v) in enumerate(cached):
            s["kv"].k[l].copy_(k), s["kv"].v[l].copy_(v)
        torch.cuda.synchronize()
        s["lane"].steps([t[-1] for t in tokens])
    else:
        s["lane"].prompts(tokens)
    return s


def over_rms(x, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)


def rotated(x, pos, theta):
    """x [n, heads, 128], halves of a head as pairs."""
    f = theta ** (-torch.arange(64, device=x.device, dtype=torch.float64) / 64)
    a = (pos.double()[:, None] * f)[:, None]
    u, v = x[..., :64], x[..., 64:]
    return torch.cat([u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin()], -1)


def decoder_exact(case, seed):
    c, w, cached, tokens = decoder_data(case, seed)
    table, pages = page_table(case, PAGE, seed)
    table = torch.from_numpy(table).long().cuda()
    lens, past = lengths(case), pasts(case)
    x = w.embed[torch.tensor([t for p, ts in zip(past, tokens) for t in ts[p:]], device="cuda")].double()
    at = [torch.arange(p, p + n, device="cuda") for p, n in zip(past, lens)]
    pos = torch.cat(at)
    slot = torch.cat([table[i][a // PAGE] * PAGE + a % PAGE for i, a in enumerate(at)])
    starts, caches = np.cumsum([0] + lens).tolist(), {"k": [], "v": []}
    for l in range(case["layers"]):
        h = (over_rms(x, c.eps) * w.in_norm[l].double()) @ w.qkv[l].double().T
        q, k, v = h.view(len(x), -1, 128).split([c.hq, c.hkv, c.hkv], 1)
        q = rotated(over_rms(q, c.eps) * w.q_norm[l].double(), pos, c.theta)
        k = rotated(over_rms(k, c.eps) * w.k_norm[l].double(), pos, c.theta)
        o = []
        for i, n in enumerate(lens):
            a = slice(starts[i], starts[i] + n)
            kk, vv = k[a], v[a]
            if cached:
                old = [t[table[i]].flatten(0, 1)[:past[i]].double() for t in cached[l]]
                kk, vv = torch.cat([old[0], kk]), torch.cat([old[1], vv])
            o.append(causal_exact(q[a], kk, vv, past[i], 128 ** -0.5))
        for name, new in (("k", k), ("v", v)):   # the written caches of a prompt (a decode step's are hundreds of megabytes)
            caches[name].append(None if cached else torch.zeros(pages * PAGE, c.hkv, 128, dtype=torch.float64, device="cuda")
                                .index_copy_(0, slot, new).view(pages, PAGE, c.hkv, 128))
        x = x + torch.cat(o).flatten(1) @ w.o[l].double().T
        h = over_rms(x, c.eps) * w.post_norm[l].double()
        x = x + experts_exact(h, *routed(h, w.router[l], None, c.K, "softmax"), w.w13, w.w2)
    last = torch.tensor([a + n - 1 for a, n in zip(starts, lens)], device="cuda")
    return dict(logits=(over_rms(x[last], c.eps) * w.final_norm.double()) @ w.lm_head.double().T, **caches)


def decoder_work(case):
    c, T, R = types.SimpleNamespace(**DECODER), sum(lengths(case)), case["requests"]
    active, expert = c.E * (1 - (1 - c.K / c.E) ** T), 3 * c.H * c.I
    dense = (c.hq + 2 * c.hkv) * 128 * c.H + c.H * c.hq * 128 + c.E * c.H
    keys = sum(n + p for n, p in zip(lengths(case), pasts(case)))
    return dict(bytes=case["layers"] * (2.0 * dense + 2.0 * active * expert + keys * c.hkv * 512.0)
                + 2.0 * c.vocab * c.H + 4.0 * R * c.vocab + 2.0 * T * c.H,
                flops=case["layers"] * (2.0 * T * (dense + c.K * expert) + 4.0 * 128 * c.hq * pairs(case)) + 2.0 * R * c.vocab * c.H)


# ------------------------------------------------------------------------------------------ layer-list decoders
def layers_config(design):
    W = WIDTH
    if design == "Sinotar":
        mixers = [("mlstm", dict(heads=W // 512, dim=256, vdim=512, gate_cap=15.0)),
                  ("mamba1", dict(inner=2 * W, state=16, dt_rank=W // 16, conv=4)),
                  ("latent_attention", dict(heads=W // 128, dim=128, rot_dim=64, vdim=128, kv_rank=512, scale=192 ** -0.5,
                                            rot=dict(base=1e4, dims=64)))]
        more = dict(streams=4)
    else:
        mixers = [("gla", dict(heads=W // 128, dim=64, vdim=128, tau=16.0)),
                  ("parallel", dict(left=dict(heads=W // 128, kv_heads=8, dim=128, vdim=128, scale=128 ** -0.5),
                                    right=dict(heads=W // 128, kv_heads=W // 256, dim=128, vdim=128, conv=4))),
                  ("gla", dict(heads=W // 512, dim=256, vdim=512, tau=16.0))]
        more = dict(embedding=dict(scale=1.0), logit_scale=1.0, max_positions=4096)
    return dict(architecture=design, layers=[dict(type=k, mixer=m, mlp=dict(kind="dense", ff=3 * W)) for k, m in mixers],
                width=W, vocab=VOCAB, norm=dict(eps=EPS), **more)


def layers_tensors(c, seed):
    g, W, t = generator(seed), c["width"], {}

    def put(name, *shape, scale=1.0, at=0.0):
        t[name] = normal(g, *shape, scale=scale, at=at)

    def lin(name, out, inp):
        put(name, out, inp, scale=inp ** -0.5)

    put("embed", c["vocab"], W), lin("head", c["vocab"], W)
    sinotar = c["architecture"] == "Sinotar"
    one = dict(scale=0.1, at=0.0 if sinotar else 1.0)   # what a norm's weight is counted from
    put("final.norm", W, **one)
    if not sinotar:
        put("pos", c["max_positions"], W, scale=0.1)
    for i, layer in enumerate(c["layers"]):
        m, p, x, kind = layer["mixer"], f"l{i}.", f"l{i}.mix.", layer["type"]
        for q in (1, 2):
            put(f"{p}norm{q}", W, **one)
            if sinotar:
                s = c["streams"]
                t[f"{p}hc{q}.in"] = torch.full((s,), 1.0 / s, device="cuda")
                t[f"{p}hc{q}.out"] = torch.linspace(0.4, 0.6, s, device="cuda")
                t[f"{p}hc{q}.mix"] = 0.8 * torch.eye(s, device="cuda") + 0.2 / s
            else:
                put(f"{p}norm{q}b", W, **one)
        if kind == "mamba1":
            C, n, r = m["inner"], m["state"], m["dt_rank"]
            lin(x + "in", 2 * C, W), put(x + "conv", C, m["conv"], scale=0.5), put(x + "conv.b", C, scale=0.1)
            lin(x + "x", r + 2 * n, C), lin(x + "dt", C, r), put(x + "dt.b", C, at=-3.0)
            put(x + "A_log", C, n, scale=0.5), put(x + "D", C), lin(x + "o", W, C)
        elif kind == "mlstm":
            H, d, e = m["heads"], m["dim"], m["vdim"]
            for name, o in (("q", H * d), ("k", H * d), ("v", H * e), ("g", H * e), ("i", H), ("f", H)):
                lin(x + name, o, W)
            put(x + "i.b", H), put(x + "f.b", H, at=3.0), put(x + "norm", H * e, scale=0.1, at=1.0), lin(x + "o", W, H * e)
        elif kind == "latent_attention":
            H, d, r, e, k = m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"]
            lin(x + "q", H * (d + r), W), lin(x + "dkv", k + r, W), put(x + "dkv.norm", k, scale=0.1, at=1.0)
            lin(x + "uk", H * d, k), lin(x + "uv", H * e, k), lin(x + "o", W, H * e)
        elif kind == "gla":
            H, d, e = m["heads"], m["dim"], m["vdim"]
            for name, o in (("q", H * d), ("k", H * d), ("v", H * e), ("g", H * e), ("a1", 16)):
                lin(x + name, o, W)
            lin(x + "a2", H * d, 16), put(x + "a2.b", H * d, at=2.0), put(x + "norm", e, scale=0.1, at=1.0), lin(x + "o", W, H * e)
        else:
            a, b = m["left"], m["right"]
            for name, o in (("q", a["heads"] * a["dim"]), ("k", a["kv_heads"] * a["dim"]), ("v", a["kv_heads"] * a["vdim"]), ("g", a["heads"])):
                lin(f"{x}left.{name}", o, W)
            put(x + "left.q.norm", a["dim"], scale=0.1, at=1.0), put(x + "left.k.norm", a["dim"], scale=0.1, at=1.0)
            lin(x + "left.o", W, a["heads"] * a["vdim"])
            for name, o in (("q", b["kv_heads"] * b["dim"]), ("k", b["kv_heads"] * b["dim"]), ("v", b["heads"] * b["vdim"])):
                lin(f"{x}right.{name}", o, W), put(f"{x}right.{name}.conv", o, b["conv"], scale=0.5)
            for name, o in (("b", b["heads"]), ("a1", b["dim"]), ("g1", b["vdim"])):
                lin(f"{x}right.{name}", o, W)
            lin(x + "right.a2", b["heads"] * b["dim"], b["dim"]), lin(x + "right.g2", b["heads"] * b["vdim"], b["vdim"])
            put(x + "right.A_log", b["heads"]), put(x + "right.dt_bias", b["heads"] * b["dim"], at=-3.0)
            put(x + "right.norm", b["vdim"], scale=0.1, at=1.0), lin(x + "right.o", W, b["heads"] * b["vdim"])
            put(x + "left.out", W, scale=0.1, at=1.0), put(x + "right.out", W, scale=0.1, at=1.0)
        lin(p + "mlp.gate", layer["mlp"]["ff"], W), lin(p + "mlp.up", layer["mlp"]["ff"], W), lin(p + "mlp.down", W, layer["mlp"]["ff"])
    return t


def layers_prepare(case, seed):
    from monoserve_b200.layer_list import LayerListCache, LayerListLane, Weights, read_config
    c = layers_config(case["design"])
    cfg = read_config(c)
    weights = Weights(cfg, layers_tensors(c, seed))
    s = dict(kind="layers")

    def make(fab, pages, page, rows, slots, stride):
        s["kv"] = LayerListCache(cfg, pages, page, slots)
        return LayerListLane(fab, 0, cfg, weights, s["kv"], max_tokens=max(rows, slots), max_slots=slots, bt_stride=stride, logit_rows=slots)
    s["lane"] = lane = Lane(make, case, seed)
    tokens = token_ids(case, seed, c["vocab"])
    if case["past"]:
        torch.cuda.synchronize()
        lane.once(lane.lane.build_prefill([(i, t[:-1], 0) for i, t in enumerate(tokens)]))
        lane.steps([t[-1] for t in tokens])
    else:
        lane.prompts(tokens)
    return s


def log_sigmoid(x):
    return torch.nn.functional.logsigmoid(x)


def conv_exact(x, w, b=0.0):
    """x [R, T, C], w [C, taps] (the last tap meets the current token)."""
    taps = w.shape[1]
    padded = torch.nn.functional.pad(x, (0, 0, taps - 1, 0))
    return torch.nn.functional.silu(sum(padded[:, j:j + x.shape[1]] * w[:, j] for j in range(taps)) + b)


def kept(lens, t, new, old):
    """The recurrent state after token t, of the requests that have one."""
    return torch.where((lens > t).view(-1, *[1] * (new.dim() - 1)), new, old)


def mamba_exact(h, lens, p, m):
    C, n, r = m["inner"], m["state"], m["dt_rank"]
    x, z = (h @ p["in"].T).split([C, C], -1)
    x = conv_exact(x, p["conv"], p["conv.b"])
    dt, B, Cm = (x @ p["x"].T).split([r, n, n], -1)
    dt = torch.nn.functional.softplus(dt @ p["dt"].T + p["dt.b"])
    A, S, y = -p["A_log"].exp(), h.new_zeros(h.shape[0], C, n), []
    for t in range(h.shape[1]):
        S = kept(lens, t, (dt[:, t, :, None] * A).exp() * S + (dt[:, t] * x[:, t])[..., None] * B[:, t, None], S)
        y.append(torch.einsum("rcn,rn->rc", S, Cm[:, t]))
    y = torch.stack(y, 1) + p["D"] * x
    return (y * torch.nn.functional.silu(z)) @ p["o"].T, dict(state=S)


def mlstm_exact(h, lens, p, m):
    R, T, H, d, e, cap = *h.shape[:2], m["heads"], m["dim"], m["vdim"], m["gate_cap"]
    q, k, v = ((h @ p[a].T).view(R, T, H, -1) for a in "qkv")
    i, f = (cap * torch.tanh((h @ p[a].T + p[a + ".b"]) / cap) for a in "if")
    f, v = log_sigmoid(f), torch.cat([v, v.new_ones(R, T, H, 1)], -1)   # the last column sums the keys
    S, top, out = h.new_zeros(R, H, e + 1, d), h.new_zeros(R, H), []
    for t in range(T):
        new = torch.maximum(f[:, t] + top, i[:, t])
        keep, add = (f[:, t] + top - new).exp(), (i[:, t] - new).exp()
        S = kept(lens, t, keep[..., None, None] * S + (add[..., None] * v[:, t])[..., None] * k[:, t, :, None], S)
        top = kept(lens, t, new, top)
        o = torch.einsum("rhed,rhd->rhe", S, q[:, t] * d ** -0.5)
        out.append(o[..., :e] / (torch.maximum(o[..., e].abs(), (-top).exp()) + 1e-6)[..., None])
    o = over_rms(torch.stack(out, 1), EPS).flatten(2)
    return (o * p["norm"] * (h @ p["g"].T).sigmoid()) @ p["o"].T, dict(S=S)


def latent_exact(h, lens, p, m):
    R, T, H, d, r, e, c = *h.shape[:2], m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"]
    f = m["rot"]["base"] ** (-2.0 * torch.arange(r // 2, device="cuda", dtype=torch.float64) / r)
    a = torch.arange(T, device="cuda", dtype=torch.float64)[:, None] * f

    def turned(x):   # [..., T, r], neighbours as pairs
        u, v = x[..., 0::2], x[..., 1::2]
        return torch.stack([u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin()], -1).flatten(-2)

    q = (h @ p["q"].T).view(R, T, H, d + r)
    lat = h @ p["dkv"].T
    kr, lat = turned(lat[..., c:]), over_rms(lat[..., :c], EPS) * p["dkv.norm"]
    k, v = (lat @ p["uk"].T).view(R, T, H, d), (lat @ p["uv"].T).view(R, T, H, e)
    k = torch.cat([k, kr[:, :, None].expand(R, T, H, r)], -1)
    q = torch.cat([q[..., :d], turned(q[..., d:].transpose(1, 2)).transpose(1, 2)], -1)
    o = torch.stack([causal_exact(q[i], k[i], v[i], 0, m["scale"]) for i in range(R)])
    return o.flatten(2) @ p["o"].T, {}


def memory_exact(q, k, v, decay, beta, lens):
    """S <- diag(decay) S, then S + k (v or beta (v - S^T k))^T, read by q; S as [values, keys]."""
    R, T, H, d = q.shape
    S, out = q.new_zeros(R, H, v.shape[-1], d), []
    for t in range(T):
        new, u = decay[:, t, :, None] * S, v[:, t]
        if beta is not None:
            u = beta[:, t, :, None] * (u - torch.einsum("rhed,rhd->rhe", new, k[:, t]))
        S = kept(lens, t, new + u[..., None] * k[:, t, :, None], S)
        out.append(torch.einsum("rhed,rhd->rhe", S, q[:, t]))
    return torch.stack(out, 1), S


def gla_exact(h, lens, p, m):
    R, T, H, d = *h.shape[:2], m["heads"], m["dim"]
    q, k, v = ((h @ p[a].T).view(R, T, H, -1) for a in "qkv")
    decay = (log_sigmoid(h @ p["a1"].T @ p["a2"].T + p["a2.b"]) / m["tau"]).exp().view(R, T, H, d)
    o, S = memory_exact(q * d ** -0.5, k, v, decay, None, lens)
    o = (over_rms(o, EPS) * p["norm"]).flatten(2) * torch.nn.functional.silu(h @ p["g"].T)
    return o @ p["o"].T, dict(S=S)


def below(w, prefix):
    return {k[len(prefix):]: v for k, v in w.items() if k.startswith(prefix)}


def parallel_exact(h, lens, p, m):
    R, T = h.shape[:2]
    a, w = m["left"], below(p, "left.")
    q, k, v = ((h @ w[n].T).view(R, T, -1, 128) for n in "qkv")
    q, k = over_rms(q, EPS) * w["q.norm"], over_rms(k, EPS) * w["k.norm"]
    o = torch.stack([causal_exact(q[i], k[i], v[i], 0, a["scale"]) for i in range(R)])
    left = (o * (h @ w["g"].T).sigmoid()[..., None]).flatten(2) @ w["o"].T
    b, w = m["right"], below(p, "right.")
    H, G, d = b["heads"], b["kv_heads"], b["dim"]
    q, k, v = (conv_exact(h @ w[n].T, w[n + ".conv"]) for n in "qkv")

    def unit(x):
        x = x.view(R, T, G, d)
        return (x * torch.rsqrt((x * x).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // G, 2)

    z = torch.nn.functional.softplus(h @ w["a1"].T @ w["a2"].T + w["dt_bias"]).view(R, T, H, d)
    o, S = memory_exact(unit(q) * d ** -0.5, unit(k), v.view(R, T, H, -1), (-w["A_log"].exp()[:, None] * z).exp(),
                        (h @ w["b"].T).sigmoid(), lens)
    o = over_rms(o, EPS) * w["norm"] * (h @ w["g1"].T @ w["g2"].T).sigmoid().view(R, T, H, -1)
    right = o.flatten(2) @ w["o"].T
    return 0.5 * (over_rms(left, EPS) * p["left.out"] + over_rms(right, EPS) * p["right.out"]), dict(S=S)


EXACT_MIXERS = dict(mamba1=mamba_exact, mlstm=mlstm_exact, latent_attention=latent_exact, gla=gla_exact, parallel=parallel_exact)


def layers_exact(case, seed):
    c = layers_config(case["design"])
    w = {k: v.double() for k, v in layers_tensors(c, seed).items()}
    sinotar = c["architecture"] == "Sinotar"
    tokens = token_ids(case, seed, c["vocab"])
    lens = torch.tensor([len(t) for t in tokens], device="cuda")
    T = int(lens.max())
    x = w["embed"][torch.tensor([t + [0] * (T - len(t)) for t in tokens], device="cuda")]
    x = torch.stack([x] * c["streams"]) if sinotar else x + w["pos"][:T]
    states = []

    def norm(x, name):
        return over_rms(x, EPS) * (w[name] + (1 if sinotar else 0))

    for l, spec in enumerate(c["layers"]):
        p = f"l{l}."
        mlp = below(w, p + "mlp.")

        def feed(h):
            gate = h @ mlp["gate"].T
            gate = torch.nn.functional.gelu(gate, approximate="tanh") if sinotar else torch.nn.functional.silu(gate)
            return (gate * (h @ mlp["up"].T)) @ mlp["down"].T

        def mix(h):
            y, state = EXACT_MIXERS[spec["type"]](h, lens, below(w, p + "mix."), spec["mixer"])
            states.append(state)
            return y

        for q, f in ((1, mix), (2, feed)):
            if sinotar:
                hc = below(w, f"{p}hc{q}.")
                y = f(norm(torch.einsum("s,srtw->rtw", hc["in"], x), f"{p}norm{q}"))
                x = torch.einsum("su,srtw->urtw", hc["mix"], x) + hc["out"].view(-1, 1, 1, 1) * y
            else:
                x = x + norm(f(norm(x, f"{p}norm{q}")), f"{p}norm{q}b")
    x = x.sum(0) if sinotar else x
    rows = x[torch.arange(len(tokens), device="cuda"), lens - 1]
    return dict(logits=norm(rows, "final.norm") @ w["head"].T, states=states)


def layers_work(case):
    c, T, R = layers_config(case["design"]), sum(lengths(case)), case["requests"]
    W, keys = c["width"], sum(n + p for n, p in zip(lengths(case), pasts(case)))
    nbytes, flops = 2.0 * W * c["vocab"] + 4.0 * R * c["vocab"] + 2.0 * T * W, 2.0 * R * W * c["vocab"]
    for layer in c["layers"]:
        m, n, state = layer["mixer"], 3.0 * W * layer["mlp"]["ff"], 0
        if layer["type"] == "mamba1":
            n += m["inner"] * (3.0 * W + 2 * m["dt_rank"] + 2 * m["state"])
            state = m["inner"] * m["state"]
        elif layer["type"] == "latent_attention":
            n += W * (m["heads"] * (m["dim"] + m["rot_dim"]) + m["kv_rank"] + m["rot_dim"]) + m["heads"] * ((m["dim"] + m["vdim"]) * m["kv_rank"] + m["vdim"] * W)
            nbytes += 2.0 * keys * (m["kv_rank"] + m["rot_dim"])
            flops += 2.0 * m["heads"] * (m["dim"] + m["rot_dim"] + m["vdim"]) * pairs(dict(case, past_lo=0, past_hi=0))
        elif layer["type"] in ("mlstm", "gla"):
            n += W * m["heads"] * (2.0 * m["dim"] + 3 * m["vdim"])
            state = m["heads"] * m["dim"] * m["vdim"]
        else:
            a, b = m["left"], m["right"]
            n += W * (a["heads"] * (a["dim"] + a["vdim"]) + a["kv_heads"] * (a["dim"] + a["vdim"]))
            n += W * (2.0 * b["kv_heads"] * b["dim"] + 2 * b["heads"] * b["vdim"]) + b["heads"] * (b["dim"] ** 2 + b["vdim"] ** 2)
            state = b["heads"] * b["dim"] * b["vdim"]
            nbytes += 2.0 * keys * a["kv_heads"] * (a["dim"] + a["vdim"])
            flops += 2.0 * a["heads"] * (a["dim"] + a["vdim"]) * pairs(dict(case, past_lo=0, past_hi=0))
        nbytes += 2.0 * n + (8.0 if case["past"] else 4.0) * R * state
        flops += 2.0 * T * n + 6.0 * T * state
    return dict(bytes=nbytes, flops=flops)


# ------------------------------------------------------------------------------------------ what the measurement calls
def prepare(case, seed):
    return {"moe": moe_prepare, "attention": attention_prepare, "decoder": decoder_prepare, "layers": layers_prepare}[case["kind"]](case, seed)


def run(state):
    kind = state["kind"]
    if kind == "moe":
        return state["layer"].forward(state["x"], state["x2"])
    if kind == "attention":
        return state["plan"].run(*state["args"], check=False)
    logits = state["lane"].run()
    if kind == "decoder":
        return dict(logits=logits, k=state["kv"].k, v=state["kv"].v)
    return dict(logits=logits, states=[{n: t for n, t in run.items() if n in ("S", "state")} for run in state["kv"].runs])


def exact(case, seed):
    return {"moe": moe_exact, "attention": attention_exact, "decoder": decoder_exact, "layers": layers_exact}[case["kind"]](case, seed)


def work(case):
    return {"moe": moe_work, "attention": attention_work, "decoder": decoder_work, "layers": layers_work}[case["kind"]](case)


def tolerance(case):
    """About four times the distance of a pass from the same in 64 bits; a router's near tie moves single rows by more."""
    return {"moe": dict(rel=7e-3, max=0.2), "attention": dict(rel=1e-2, max=0.1), "decoder": dict(rel=3e-2, max=0.8),
            "layers": dict(rel=3e-2, max=0.5)}[case["kind"]]
