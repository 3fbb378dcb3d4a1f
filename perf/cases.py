"""Performance cases: the calls that a serving program makes, over the sizes it makes them with.

A case is a dict of plain values.  ``listed()`` names the standing ones, ``draw(rng)`` makes another one of the same ranges,
``prepare`` builds what the caller has in hand (weights, caches, inputs), ``run`` makes one pass through the public entry
points, ``work`` says what the pass cannot do without, ``tolerance`` how far two correct implementations may differ, and
``exact`` computes the same outputs in 64 bits with plain torch.

Kinds:
  linear    one W4A16 projection through ``LlamaLinear.forward``: what an embedding host calls per projection
  decode    one step of a whole W4A16 LLaMA (``LlamaModel.decode``, captured step, input tokens given), behind cached tokens
  prefill   new prompt tokens of a ragged batch through a W4A16 LLaMA (``LlamaModel.prefill``), on top of cached ones
  dense     the bf16 product of the config-driven decoders (``tm_gemm_dense``)
  window    decode step of window attention with pooled blocks (``tm_window_attention``)
  delta     prefill of the generalised delta rule (``tm_delta_rule``)
  chunk     prefill of attention within chunks (``tm_chunk_attention``)
  experts   mixture of experts behind a gate (``tm_moe``)
"""
import ctypes as C
import functools
import math
import weakref

import numpy as np
import torch

from lmdeploy_b200 import lib as tl
from lmdeploy_b200 import llama, turbomind

D = 128        # head size of every attention here
GROUP = 128    # rows that share a scale and a zero point
VOCAB = 32000
KV_SCALE = 4.0 / 127
SIZES = {"7b": llama.LLAMA2_7B, "70b": llama.LLAMA2_70B}
# (output features, input features, whether the gate / up epilogue belongs to it): the projections of both sizes, and those of
# the larger one on one of eight tensor-parallel ranks
PROJECTIONS = [(12288, 4096, False), (4096, 4096, False), (22016, 4096, True), (4096, 11008, False), (11008, 4096, False),
               (10240, 8192, False), (8192, 8192, False), (57344, 8192, True), (8192, 28672, False),
               (1280, 8192, False), (8192, 1024, False), (7168, 8192, True), (8192, 3584, False)]


def listed():
    return [
        # one token through the attention's output projection: the smallest product of a step for a single user
        dict(name="linear_o_1", kind="linear", n=4096, k=4096, tokens=1, silu=False),
        # sixteen tokens through a feed-forward projection: a small batch
        dict(name="linear_up_16", kind="linear", n=11008, k=4096, tokens=16, silu=False),
        # a single user's next token
        dict(name="decode_7b_1", kind="decode", size="7b", layers=32, batch=1, shortest=700, longest=700, int8=True),
        # a full batch of 64 sessions, prompts of 128 to 1024 tokens and some of their answers: the benchmark's step
        dict(name="decode_7b_64", kind="decode", size="7b", layers=32, batch=64, shortest=180, longest=1180, int8=True),
        # grouped heads, fp16 cache, longer sessions, a batch that fills no tile: some layers of the larger model
        dict(name="decode_70b_21", kind="decode", size="70b", layers=8, batch=21, shortest=512, longest=3000, int8=False),
        # three sessions go on: a few hundred new tokens each behind cached ones
        dict(name="prefill_7b_3", kind="prefill", size="7b", layers=4, batch=3, shortest=77, longest=413, history=801, int8=True),
        # eight long prompts at once
        dict(name="prefill_7b_8", kind="prefill", size="7b", layers=8, batch=8, shortest=2048, longest=2048, history=0, int8=False),
        # the input projections and gated feed-forward of a config-driven decoder's layer, one pass of prefill
        dict(name="dense_4096", kind="dense", n=22016, k=4096, tokens=4096),
        # window attention of sixteen sessions that have grown past the window
        dict(name="window_16", kind="window", batch=16, history=4096, window=2048, pool=16, softcap=30.0),
        # the recurrence over a long prompt
        dict(name="delta_4096", kind="delta", batch=1, tokens=4096),
        # chunk attention over a prompt of two chunks
        dict(name="chunk_4096", kind="chunk", batch=1, tokens=4096, chunk=2048),
        # the experts of a full batch's step
        dict(name="experts_64", kind="experts", tokens=64),
    ]


def _log(rng, lo, hi):
    return min(hi, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))


def draw(rng):
    kind = rng.choice(["linear"] * 3 + ["decode"] * 3 + ["prefill"] * 2 + ["dense", "window", "delta", "chunk", "experts"])
    if kind == "linear":
        n, k, gated = rng.choice(PROJECTIONS)
        return dict(kind=kind, n=n, k=k, tokens=_log(rng, 1, 2048), silu=gated and rng.random() < 0.8)
    if kind == "decode":
        size = rng.choice(["7b", "7b", "70b"])
        batch, int8 = _log(rng, 1, 64), rng.random() < 0.6
        # the slots that a batch of 64 has with 1288 slots each in int8
        longest = _log(rng, 64, min(4000, 1288 * 64 // batch // (1 if int8 else 2)))
        return dict(kind=kind, size=size, layers=rng.choice([8, 32] if size == "7b" else [4, 8]), batch=batch, shortest=_log(rng, 16, longest),
                    longest=longest, int8=int8)
    if kind == "prefill":
        batch = _log(rng, 1, 8)
        longest = _log(rng, 16, 2048)
        int8 = rng.random() < 0.5
        return dict(kind=kind, size="7b", layers=4 if int8 else rng.choice([4, 8]), batch=batch, shortest=_log(rng, 1, longest), longest=longest,
                    history=rng.choice([0, 0, _log(rng, 1, 1024)]), int8=int8)
    if kind == "dense":
        n, k = rng.choice([(22016, 4096), (4096, 11008), (4096, 4096), (10240, 4096)])
        return dict(kind=kind, n=n, k=k, tokens=_log(rng, 1, 4096))
    if kind == "window":
        window = rng.choice([1024, 2048])
        return dict(kind=kind, batch=_log(rng, 1, 64), history=_log(rng, 64, 8192), window=window, pool=rng.choice([0, 16]),
                    softcap=rng.choice([0.0, 30.0]))
    if kind == "delta":
        batch = _log(rng, 1, 8)
        return dict(kind=kind, batch=batch, tokens=_log(rng, 16, 4096))
    if kind == "chunk":
        batch = _log(rng, 1, 4)
        return dict(kind=kind, batch=batch, tokens=_log(rng, 16, 4096), chunk=rng.choice([512, 2048]))
    return dict(kind="experts", tokens=_log(rng, 1, 512))


# ---------------------------------------------------------------------------------------------------------------- values
def _device():
    return torch.device("cuda", torch.cuda.current_device())


def _gen(seed, *key):
    n = seed
    for k in key:
        n = (n * 1000003 + k + 1) % (1 << 62)
    return torch.Generator(device=_device()).manual_seed(n)


def _randn(gen, *shape):
    return torch.randn(*shape, device=gen.device, generator=gen)


def _weight(gen, n, k):
    """A quantised weight as groups of N(0, 0.02) rows give it -> values 0..15 [k, n], zero points, scales [k / 128, n]"""
    q = _randn(gen, k, n).mul_(2.7).add_(7.5).round_().clamp_(0, 15).to(torch.uint8)
    z = torch.randint(6, 10, (k // GROUP, n), device=gen.device, generator=gen, dtype=torch.int32)
    s = (0.0074 * (0.85 + 0.3 * torch.rand(k // GROUP, n, device=gen.device, generator=gen))).half()
    return q, z, s


def _pack(v):
    """values [rows, columns] -> words of eight columns in the order AWQ packs them"""
    v = v.view(v.shape[0], -1, 8)
    out = torch.zeros(v.shape[:2], dtype=torch.int32, device=v.device)
    for i, column in enumerate((0, 2, 4, 6, 1, 3, 5, 7)):
        out |= v[:, :, column].to(torch.int32) << (4 * i)
    return out


def _linear(gen, n, k):
    """-> the weight in the layout that the library runs from"""
    q, z, s = _weight(gen, n, k)
    qweight, qzeros = _pack(q), _pack(z)
    kernel = torch.empty_like(qweight)
    sz = torch.empty(k // GROUP, n, 2, dtype=torch.float16, device=s.device)
    ws = torch.empty(k // GROUP * n, dtype=torch.float16, device=s.device)
    turbomind.convert_s4_k_m8(kernel, sz, ws, qweight, s, qzeros, n, k, GROUP)
    return turbomind.LlamaDenseWeight(k, n, kernel, turbomind.WeightType.kINT4, None, sz, GROUP)


def _exact_weight(gen, n, k):
    """the same weight as numbers: fp16((value - zero) * scale), in 64 bits [k, n]"""
    q, z, s = _weight(gen, n, k)
    w = (q.view(-1, GROUP, n).half() - z[:, None].half()) * s[:, None]
    return w.view(k, n).double()


def _silu_pairs(y):
    return torch.nn.functional.silu(y[:, 0::2]) * y[:, 1::2]


def _spread(case, lo, hi):
    """one length per sequence, evenly spread over [lo, hi]"""
    b = case["batch"]
    return [lo + round((hi - lo) * (i + 0.5) / b) for i in range(b)]


# ----------------------------------------------------------------------------------------------------------------- LLaMA
class _Llama:
    """A model and the state of its sequences, closed when the caller lets go of it."""

    def __init__(self, case, seed):
        cfg, layers = SIZES[case["size"]], case["layers"]
        self.case = case
        self.cfg = llama.LlamaConfig(cfg.head_num, cfg.kv_head_num, cfg.inter_size, layers, VOCAB, quant_policy=4 if case["int8"] else 0,
                                     name=cfg.name)
        self.cached, self.new = _lengths(case)
        slots = (max(c + n for c, n in zip(self.cached, self.new)) + 7) // 8 * 8
        self.model = llama.LlamaModel(self.cfg, case["batch"], slots, _device().index)
        weakref.finalize(self, self.model.close)
        hid, kv = cfg.hidden, (KV_SCALE, 0.0, KV_SCALE, 0.0)
        for i in range(layers):
            g = _gen(seed, i)
            norms = _norms(g, hid)
            self.model.set_layer(i, *norms, *(_linear(g, n, k) for n, k in _layer_shapes(cfg)), kv_scale=kv)
        self.globals = _globals(seed, hid)
        self.model.set_globals(*self.globals)
        self.tokens = _tokens(case, seed)
        forced = [[t[0] for t in self.tokens]] if case["kind"] == "decode" else None
        self.state = self.model.new_state(case["batch"], 1, forced_ids=forced, keep_logits=case["kind"] == "decode")
        for b in range(case["batch"]):
            self.state.k_cache[b], self.state.v_cache[b] = _cached_rows(case, seed, b, slots)
        self.lengths = torch.tensor(self.cached, dtype=torch.int32, device=_device())
        self.stream = _serving_stream()
        self.stream.wait_stream(torch.cuda.current_stream())


@functools.lru_cache(maxsize=None)
def _serving_stream():
    """The one stream that steps run on: a step cannot be captured on the default stream, and a handle serves one stream."""
    return torch.cuda.Stream()


def _layer_shapes(cfg):
    hid = cfg.hidden
    return [((cfg.head_num + 2 * cfg.kv_head_num) * D, hid), (hid, hid), (2 * cfg.inter_size, hid), (hid, cfg.inter_size)]


def _norms(gen, hid):
    return tuple((1 + 0.1 * _randn(gen, hid)).half() for _ in range(2))


def _globals(seed, hid):
    g = _gen(seed, 1 << 20)
    return (_randn(g, VOCAB, hid) * 0.02).half(), (1 + 0.1 * _randn(g, hid)).half(), (_randn(g, VOCAB, hid) * 0.02).half()


def _lengths(case):
    """tokens cached before the call, and new tokens, per sequence"""
    if case["kind"] == "decode":
        return _spread(case, case["shortest"], case["longest"]), [1] * case["batch"]
    new = _spread(case, case["shortest"], case["longest"])
    return _spread(case, 0, case["history"]) if case["history"] else [0] * case["batch"], new


def _tokens(case, seed):
    r = np.random.default_rng(seed)
    return [[int(t) for t in r.integers(0, VOCAB, n)] for n in _lengths(case)[1]]


def _cached_rows(case, seed, b, slots):
    """keys and values of a sequence, [layers, kv heads, slots, 128] each: N(0, 1), rows without a token zero"""
    g, cached = _gen(seed, 1 << 21, b), _lengths(case)[0][b]
    out = []
    for _ in range(2):
        x = _randn(g, case["layers"], SIZES[case["size"]].kv_head_num, slots, D)
        x[:, :, cached:] = 0
        out.append(x.div_(KV_SCALE).round_().clamp_(-128, 127).to(torch.int8) if case["int8"] else x.half())
    return out


def _exact_llama(case, seed):
    cfg, batch, decode = SIZES[case["size"]], case["batch"], case["kind"] == "decode"
    H, G, hid, dev, f64 = cfg.head_num, cfg.kv_head_num, cfg.hidden, _device(), torch.float64
    cached, new = _lengths(case)
    slots = (max(c + n for c, n in zip(cached, new)) + 7) // 8 * 8
    emb, last_norm, head = _globals(seed, hid)
    rows = [_cached_rows(case, seed, b, slots) for b in range(batch)]
    kept = not case["int8"]
    stored = [[r[i].double() for r in rows] for i in range(2)] if kept and not decode else None
    added = [[[] for _ in range(batch)] for _ in range(2)]  # decode: the new keys and values, [sequence][layer][kv head, 128]
    x = emb[torch.tensor([t for s in _tokens(case, seed) for t in s], device=dev)].double()
    at = torch.cat([torch.arange(c, c + n, device=dev) for c, n in zip(cached, new)]).to(f64)
    angle = at[:, None] / (cfg.rope_theta ** (torch.arange(0, D, 2, device=dev, dtype=f64) / D))
    cos, sin = angle.cos()[:, None], angle.sin()[:, None]

    def rms(v, w):
        return v / torch.sqrt((v * v).mean(-1, keepdim=True) + cfg.norm_eps) * w.double()

    def turn(v):
        a, b = v[..., 0::2], v[..., 1::2]
        return torch.stack([a * cos - b * sin, a * sin + b * cos], -1).flatten(-2)

    for i in range(case["layers"]):
        g = _gen(seed, i)
        n1, n2 = _norms(g, hid)
        shapes = _layer_shapes(cfg)
        y = rms(x, n1) @ _exact_weight(g, *shapes[0])
        q, k, v = turn(y[:, :H * D].view(-1, H, D)), turn(y[:, H * D:(H + G) * D].view(-1, G, D)), y[:, (H + G) * D:].view(-1, G, D)
        out, t0 = torch.empty(len(x), H, D, dtype=f64, device=dev), 0
        for b in range(batch):
            c, n = cached[b], new[b]
            past = [(r[i, :, :c].double() * KV_SCALE if case["int8"] else r[i, :, :c].double()) for r in rows[b]]
            fresh = [u[t0:t0 + n].transpose(0, 1) for u in (k, v)]
            if case["int8"] and not decode:  # prefill reads its own rows from the cache too
                fresh = [(u / KV_SCALE).round().clamp(-128, 127) * KV_SCALE for u in fresh]
            if stored:
                for s, u in zip(stored, fresh):
                    s[b][i, :, c:c + n] = u
            if decode and kept:
                for a, u in zip(added, fresh):
                    a[b].append(u[:, 0])
            keys, values = (torch.cat(p, 1) for p in zip(past, fresh))
            mask = torch.arange(c + n, device=dev)[None, :] > torch.arange(c, c + n, device=dev)[:, None]
            for h0 in range(0, G, max(1, G // 8)):  # some kv heads at a time: the scores of all would take much memory
                h1 = min(G, h0 + max(1, G // 8))
                qs = q[t0:t0 + n].view(n, G, H // G, D)[:, h0:h1].permute(1, 2, 0, 3)
                s = (qs @ keys[h0:h1, None].transpose(-1, -2) / math.sqrt(D)).masked_fill_(mask, -math.inf)
                o = torch.softmax(s, -1) @ values[h0:h1, None]
                out[t0:t0 + n].view(n, G, H // G, D)[:, h0:h1] = o.permute(2, 0, 1, 3)
            t0 += n
        x = x + out.view(-1, H * D) @ _exact_weight(g, *shapes[1])
        x = x + _silu_pairs(rms(x, n2) @ _exact_weight(g, *shapes[2])) @ _exact_weight(g, *shapes[3])
    hidden = rms(x, last_norm)
    if decode:
        out = {"logits": hidden @ head.double().T}
        if kept:
            out["rows"] = [torch.stack(a[b]) for b in range(_returned(case)) for a in added]
        return out
    out = {"hidden": hidden}
    if kept:
        out["keys"], out["values"] = (torch.stack(s) for s in stored)
    return out


def _returned(case):
    """sequences whose new cache rows a decode pass returns"""
    return min(case["batch"], 28)


# ------------------------------------------------------------------------------------- operators of the other decoders
HEADS, KV_HEADS = 32, 8           # window and chunk attention
DELTA_HEADS, DELTA_DIM, DELTA_RANK = 64, 64, 96
EXPERTS, IDENTITY, TOP, EXPERT_FF, WIDTH = 30, 2, 4, 2752, 4096
EXPERT_GROUPS, EXPERT_KEEP, LIMIT, SLOPE, MULT, NORM_EPS = 4, 2, 7.0, 1.702, 0.5, 1e-6


def _call(proj, out, history, n, slabs, decode):
    c = tl.TmMixerCall()
    c.proj, c.proj_ld, c.out, c.out_ld, c.batch = proj.data_ptr(), proj.shape[1], out.data_ptr(), out.shape[1], len(n)
    c.history, c.n = (C.c_int * len(n))(*history), (C.c_int * len(n))(*n)
    c.slabs = (C.c_void_p * len(n))(*[s.data_ptr() for s in slabs])
    c.dtype, c.decode = tl.TM_DTYPE_BF16, int(decode)
    return c


def _stream():
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


def _bf16(gen, *shape):
    return _randn(gen, *shape).to(torch.bfloat16)


def _window_parts(case, seed):
    """ring and pooled rows, [batch, kv heads, rows, 128] each, and the step's projections"""
    ring = -(-(min(case["history"] + 8, case["window"] + 1)) // 128) * 128
    pooled = (case["history"] + 8) // case["pool"] + 8 if case["pool"] else 0
    g, b = _gen(seed, 1), case["batch"]
    parts = [_bf16(g, b, KV_HEADS, r, D) for r in (ring, ring, pooled, pooled)]
    for p in parts[2:]:
        p.mul_(case["pool"] ** -0.5 if case["pool"] else 1.0)  # means of that many rows
    return ring, pooled, parts, _bf16(g, b, (HEADS + 2 * KV_HEADS) * D + 128)


def _window_freq():
    return (500000.0 ** (-2.0 * torch.arange(D // 2, dtype=torch.float64) / D)).float().to(_device())


def _prepare_window(case, seed):
    ring, pooled, parts, proj = _window_parts(case, seed)
    b, freq = case["batch"], _window_freq()
    slabs = torch.cat([p.flatten(1) for p in parts], 1).contiguous()
    a = tl.TmWindowAttentionParams()
    a.heads, a.kv_heads, a.dim, a.vdim, a.rot_dims, a.inv_freq = HEADS, KV_HEADS, D, D, D, freq.data_ptr()
    a.scale, a.softcap, a.window, a.pool, a.ring, a.pool_rows = D ** -0.5, case["softcap"], case["window"], case["pool"], ring, pooled
    rows = KV_HEADS * D * 2
    a.k_off, a.v_off, a.pooled_k_off, a.pooled_v_off = 0, rows * ring, 2 * rows * ring, rows * (2 * ring + pooled)
    a.q_col, a.k_col, a.v_col, a.g_col = 0, HEADS * D, (HEADS + KV_HEADS) * D, (HEADS + 2 * KV_HEADS) * D
    out = torch.empty(b, HEADS * D, dtype=torch.bfloat16, device=_device())
    return dict(call=_call(proj, out, [case["history"]] * b, [1] * b, slabs, True), params=a, out=out, keep=(proj, slabs, freq))


def _exact_window(case, seed):
    ring, pooled, (rk, rv, pk, pv), proj = _window_parts(case, seed)
    at, window, pool = case["history"], case["window"], case["pool"]
    y, b = proj.double(), case["batch"]
    angle = at * _window_freq().double()
    cos, sin = angle.cos(), angle.sin()

    def turn(v):
        u, w = v[..., 0::2], v[..., 1::2]
        return torch.stack([u * cos - w * sin, u * sin + w * cos], -1).flatten(-2)

    q = turn(y[:, :HEADS * D].view(b, HEADS, D)).view(b, KV_HEADS, HEADS // KV_HEADS, D)
    k = turn(y[:, HEADS * D:(HEADS + KV_HEADS) * D].view(b, KV_HEADS, 1, D))
    v = y[:, (HEADS + KV_HEADS) * D:(HEADS + 2 * KV_HEADS) * D].view(b, KV_HEADS, 1, D)
    seen = torch.arange(max(0, at - window + 1), at, device=y.device) % ring
    blocks = max(0, (at - window + 1) // pool) if pool else 0
    keys = torch.cat([pk[:, :, :blocks].double(), rk[:, :, seen].double(), k], 2)
    values = torch.cat([pv[:, :, :blocks].double(), rv[:, :, seen].double(), v], 2)
    s = q @ keys.transpose(-1, -2) * D ** -0.5
    if case["softcap"]:
        s = case["softcap"] * torch.tanh(s / case["softcap"])
    o = (torch.softmax(s, -1) @ values).view(b, HEADS, D)
    return (o * torch.sigmoid(y[:, (HEADS + 2 * KV_HEADS) * D:][:, :HEADS, None])).view(b, -1)


def _delta_parts(case, seed):
    g, n = _gen(seed, 2), DELTA_HEADS * DELTA_DIM
    proj = _randn(g, case["batch"] * case["tokens"], 5 * n + DELTA_RANK)
    proj[:, 5 * n:].tanh_()
    w2 = (_randn(g, n, DELTA_RANK) * DELTA_RANK ** -0.5).to(torch.bfloat16)
    w0, a_bias, norm = _randn(g, n) * 1.5 - 1.0, _randn(g, n), 1 + 0.2 * _randn(g, n)
    return proj.to(torch.bfloat16), w2, w0, a_bias, norm


def _prepare_delta(case, seed):
    proj, w2, w0, a_bias, norm = _delta_parts(case, seed)
    n, b, t = DELTA_HEADS * DELTA_DIM, case["batch"], case["tokens"]
    d = tl.TmDeltaRuleParams()
    d.heads, d.dim, d.rank, d.w2, d.w2_ld = DELTA_HEADS, DELTA_DIM, DELTA_RANK, w2.data_ptr(), DELTA_RANK
    d.w0, d.a_bias, d.norm = w0.data_ptr(), a_bias.data_ptr(), norm.data_ptr()
    d.norm_eps, d.unit_eps, d.decay_scale, d.state_off = 1e-6, 1e-6, math.exp(-0.5), 0
    d.r_col, d.k_col, d.v_col, d.a_col, d.g_col, d.w1_col = (i * n for i in range(6))
    out = torch.empty(b * t, n, dtype=torch.bfloat16, device=_device())
    slabs = torch.zeros(b, n * DELTA_DIM, device=_device())
    return dict(call=_call(proj, out, [0] * b, [t] * b, slabs, False), params=d, out=out, slabs=slabs, keep=(proj, w2, w0, a_bias, norm))


def _exact_delta(case, seed):
    proj, w2, w0, a_bias, norm = (x.double() for x in _delta_parts(case, seed))
    H, E, b, t = DELTA_HEADS, DELTA_DIM, case["batch"], case["tokens"]
    n = H * E
    w = torch.exp(-math.exp(-0.5) * torch.sigmoid(proj[:, 5 * n:] @ w2.T + w0)).view(b, t, H, E)
    a = torch.sigmoid(proj[:, 3 * n:4 * n] + a_bias).view(b, t, H, E)
    r, k, v = (proj[:, i * n:(i + 1) * n].view(b, t, H, E) for i in range(3))
    u = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
    S = torch.zeros(b, H, E, E, dtype=torch.float64, device=proj.device)  # [key, value]
    left = torch.stack([-(a * u), k], -1)                                   # [b, t, H, key, 2]
    o = torch.empty(b, t, H, E, dtype=torch.float64, device=proj.device)
    for i in range(t):
        seen = u[:, i, :, None] @ S                                         # [b, H, 1, value]
        S = w[:, i, :, :, None] * S + left[:, i] @ torch.cat([seen, v[:, i, :, None]], 2)
        o[:, i] = (r[:, i, :, None] @ S)[:, :, 0]
    o = o / torch.sqrt((o * o).mean(-1, keepdim=True) + 1e-6)
    out = o.view(b * t, n) * norm * torch.sigmoid(proj[:, 4 * n:5 * n])
    return {"out": out, "state": S.transpose(-1, -2).reshape(b, -1)}


def _chunk_parts(case, seed):
    g = _gen(seed, 3)
    proj = _bf16(g, case["batch"] * case["tokens"], (HEADS + 2 * KV_HEADS) * D)
    return proj, _randn(g, HEADS) - 4, _randn(g, HEADS, HEADS)


def _prepare_chunk(case, seed):
    proj, bias, talk = _chunk_parts(case, seed)
    b, t, half = case["batch"], case["tokens"], talk.half()
    a = tl.TmChunkAttentionParams()
    a.heads, a.kv_heads, a.dim, a.vdim, a.scale, a.chunk = HEADS, KV_HEADS, D, D, D ** -0.5, case["chunk"]
    a.bias, a.talk, a.talk_half = bias.data_ptr(), talk.data_ptr(), half.data_ptr()
    a.ring = -(-t // 128) * 128
    a.k_off, a.v_off = 0, KV_HEADS * a.ring * D * 2
    a.q_col, a.k_col, a.v_col = 0, HEADS * D, (HEADS + KV_HEADS) * D
    slabs = torch.zeros(b, 2 * KV_HEADS * a.ring * D, dtype=torch.bfloat16, device=_device())
    out = torch.empty(b * t, HEADS * D, dtype=torch.bfloat16, device=_device())
    return dict(call=_call(proj, out, [0] * b, [t] * b, slabs, False), params=a, out=out, slabs=slabs, keep=(proj, bias, talk, half))


def _exact_chunk(case, seed):
    proj, bias, talk = (x.double() for x in _chunk_parts(case, seed))
    b, t, rep, c = case["batch"], case["tokens"], HEADS // KV_HEADS, case["chunk"]
    q = proj[:, :HEADS * D].view(b, t, HEADS, D)
    k, v = (proj[:, (HEADS + i * KV_HEADS) * D:(HEADS + (i + 1) * KV_HEADS) * D].view(b, t, KV_HEADS, D) for i in range(2))
    out = torch.empty(b, t, HEADS, D, dtype=torch.float64, device=proj.device)
    for s in range(b):
        for lo in range(0, t, c):
            for q0 in range(lo, min(t, lo + c), 256):
                q1 = min(t, lo + c, q0 + 256)
                keys, values = (x[s, lo:q1].repeat_interleave(rep, 1).transpose(0, 1) for x in (k, v))
                w = torch.sigmoid(q[s, q0:q1].transpose(0, 1) @ keys.transpose(1, 2) * D ** -0.5 + bias[:, None, None])
                w.masked_fill_(torch.arange(lo, q1, device=w.device)[None, :] > torch.arange(q0, q1, device=w.device)[:, None], 0.0)
                w = (talk @ w.view(HEADS, -1)).view_as(w)
                out[s, q0:q1] = (w @ values).transpose(0, 1)
    ring = -(-t // 128) * 128
    slabs = torch.zeros(b, 2, KV_HEADS, ring, D, dtype=torch.float64, device=proj.device)
    slabs[:, 0, :, :t], slabs[:, 1, :, :t] = k.transpose(1, 2), v.transpose(1, 2)
    return {"out": out.view(b * t, -1), "cache": slabs.view(b, -1)}


def _expert_parts(case, seed):
    g, t = _gen(seed, 4), case["tokens"]
    we = torch.empty(EXPERTS, 2 * EXPERT_FF, WIDTH, dtype=torch.bfloat16, device=g.device)
    wd = torch.empty(EXPERTS, WIDTH, EXPERT_FF, dtype=torch.bfloat16, device=g.device)
    for e in range(EXPERTS):
        we[e] = _randn(g, 2 * EXPERT_FF, WIDTH) * WIDTH ** -0.5
        wd[e] = _randn(g, WIDTH, EXPERT_FF) * EXPERT_FF ** -0.5
    x, z = _randn(g, t, WIDTH), _randn(g, t, EXPERTS + IDENTITY)
    inp, gate = _bf16(g, t, WIDTH), _bf16(g, t, WIDTH)
    return we, wd, x, z, inp, gate, 0.1 * _randn(g, WIDTH), 0.01 * _randn(g, EXPERTS + IDENTITY), 1 + 0.1 * _randn(g, WIDTH)


def _prepare_experts(case, seed):
    we, wd, x, z, inp, gate, gate_bias, correction, norm = keep = _expert_parts(case, seed)
    out, live = torch.empty_like(inp), torch.empty_like(x)
    m = tl.TmMoeParams()
    m.tokens, m.width, m.ff, m.experts, m.identity, m.top = case["tokens"], WIDTH, EXPERT_FF, EXPERTS, IDENTITY, TOP
    m.groups, m.keep, m.limit, m.slope, m.mult, m.norm_eps = EXPERT_GROUPS, EXPERT_KEEP, LIMIT, SLOPE, MULT, NORM_EPS
    m.x, m.logits, m.logits_ld, m.input, m.input_ld = live.data_ptr(), z.data_ptr(), z.shape[1], inp.data_ptr(), WIDTH
    m.gate, m.gate_ld, m.gate_bias, m.correction, m.norm_weight = gate.data_ptr(), WIDTH, gate_bias.data_ptr(), correction.data_ptr(), norm.data_ptr()
    m.w_experts, m.w_down, m.norm_out, m.dtype = we.data_ptr(), wd.data_ptr(), out.data_ptr(), tl.TM_DTYPE_BF16
    return dict(params=m, x=x, live=live, out=out, keep=keep)


def _exact_experts(case, seed):
    we, wd, x, z, inp, gate, gate_bias, correction, norm = _expert_parts(case, seed)
    t, per = case["tokens"], (EXPERTS + IDENTITY) // EXPERT_GROUPS
    s = torch.softmax(z.double(), 1)
    choice = (s + correction.double()).view(t, EXPERT_GROUPS, per)
    kept = torch.zeros(t, EXPERT_GROUPS, dtype=torch.bool, device=z.device).scatter_(1, choice.max(2).values.topk(EXPERT_KEEP, 1).indices, True)
    chosen = choice.masked_fill(~kept[:, :, None], -math.inf).view(t, -1).topk(TOP, 1).indices
    weight = torch.zeros_like(s).scatter_(1, chosen, s.gather(1, chosen))
    h = inp.double()
    y = weight[:, EXPERTS:].sum(1, keepdim=True) * h
    for e in range(EXPERTS):
        rows = weight[:, e].nonzero()[:, 0]
        if len(rows):
            p = h[rows] @ we[e].double().T
            a, u = p[:, 0::2].clamp(max=LIMIT), p[:, 1::2].clamp(-LIMIT, LIMIT)
            y[rows] += weight[rows, e, None] * ((a * torch.sigmoid(SLOPE * a) * (u + 1)) @ wd[e].double().T)
    x = x.double() + MULT * torch.sigmoid(gate.double() + gate_bias.double()) * y
    return {"x": x, "normed": x / torch.sqrt((x * x).mean(1, keepdim=True) + NORM_EPS) * norm.double()}


# -------------------------------------------------------------------------------------------------------------- interface
def prepare(case, seed):
    kind = case["kind"]
    if kind == "linear":
        g, n, k, t = _gen(seed, 0), case["n"], case["k"], case["tokens"]
        w = _linear(g, n, k)
        return dict(kind=kind, op=turbomind.LlamaLinear(_device().index), weight=w, tokens=t, x=_randn(g, t, k).half(),
                    out=torch.empty(t, n // 2 if case["silu"] else n, dtype=torch.float16, device=_device()),
                    type=turbomind.LlamaLinear.kFusedSiluFfn if case["silu"] else turbomind.LlamaLinear.kGemm)
    if kind in ("decode", "prefill"):
        return dict(kind=kind, llama=_Llama(case, seed))
    if kind == "dense":
        g, n, k, t = _gen(seed, 0), case["n"], case["k"], case["tokens"]
        w = (_randn(g, n, k) * k ** -0.5).to(torch.bfloat16)
        state = dict(w=w, x=_bf16(g, t, k), out=torch.empty(t, n, dtype=torch.bfloat16, device=_device()), sizes=(t, n, k))
    else:
        state = dict(window=_prepare_window, delta=_prepare_delta, chunk=_prepare_chunk, experts=_prepare_experts)[kind](case, seed)
    return dict(state, kind=kind, handle=tl.default_handle(_device().index))


def run(state):
    kind = state["kind"]
    if kind == "linear":
        state["op"].forward(state["out"], state["x"], state["tokens"], state["weight"], state["type"])
        return state["out"]
    if kind == "decode":
        s = state["llama"]
        with torch.cuda.stream(s.stream):
            # the sequences' lengths and the step counter, as a scheduler sets them before every step
            s.state.lengths.copy_(s.lengths)
            s.state.step.zero_()
            s.model.decode(s.state, 1)
        out = {"logits": s.state.logits}
        if not s.case["int8"]:
            out["rows"] = [c[b, :, :, s.cached[b]] for b in range(_returned(s.case)) for c in (s.state.k_cache, s.state.v_cache)]
        return out
    if kind == "prefill":
        s = state["llama"]
        s.state.lengths.copy_(s.lengths)
        out = {"hidden": s.model.prefill(s.state, s.tokens, keep_hidden=True)}
        if not s.case["int8"]:
            out["keys"], out["values"] = s.state.k_cache, s.state.v_cache
        return out
    h, st = state["handle"].ptr, _stream()
    if kind == "dense":
        t, n, k = state["sizes"]
        tl.check(tl.lib.tm_gemm_dense(h, state["out"].data_ptr(), n, 0, state["x"].data_ptr(), k, state["w"].data_ptr(), k, t, n, k,
                                      tl.TM_DTYPE_BF16, st), "tm_gemm_dense")
        return state["out"]
    if kind == "window":
        tl.check(tl.lib.tm_window_attention(h, C.byref(state["params"]), C.byref(state["call"]), st), "tm_window_attention")
        return state["out"]
    if kind == "delta":
        tl.check(tl.lib.tm_delta_rule(h, C.byref(state["params"]), C.byref(state["call"]), st), "tm_delta_rule")
        return {"out": state["out"], "state": state["slabs"]}
    if kind == "chunk":
        tl.check(tl.lib.tm_chunk_attention(h, C.byref(state["params"]), C.byref(state["call"]), st), "tm_chunk_attention")
        return {"out": state["out"], "cache": state["slabs"]}
    state["live"].copy_(state["x"])  # the residual stream as the layer ahead left it
    tl.check(tl.lib.tm_moe(h, C.byref(state["params"]), st), "tm_moe")
    return {"x": state["live"], "normed": state["out"]}


def exact(case, seed):
    kind = case["kind"]
    if kind == "linear":
        g = _gen(seed, 0)
        w = _exact_weight(g, case["n"], case["k"])
        y = _randn(g, case["tokens"], case["k"]).half().double() @ w
        return _silu_pairs(y) if case["silu"] else y
    if kind in ("decode", "prefill"):
        return _exact_llama(case, seed)
    if kind == "dense":
        g = _gen(seed, 0)
        w = (_randn(g, case["n"], case["k"]) * case["k"] ** -0.5).to(torch.bfloat16).double()
        return _bf16(g, case["tokens"], case["k"]).double() @ w.T
    return dict(window=_exact_window, delta=_exact_delta, chunk=_exact_chunk, experts=_exact_experts)[kind](case, seed)


def work(case):
    kind = case["kind"]
    if kind == "linear":
        n, k, t = case["n"], case["k"], case["tokens"]
        return dict(bytes=n * k / 2 + n * k / GROUP * 4 + 2 * t * k + 2 * t * n / (2 if case["silu"] else 1), flops=2 * t * n * k)
    if kind in ("decode", "prefill"):
        cfg, layers, e = SIZES[case["size"]], case["layers"], 1 if case["int8"] else 2
        cached, new = _lengths(case)
        t, weights = sum(new), sum(n * k for n, k in _layer_shapes(cfg))
        pairs = sum(n * c + n * (n + 1) // 2 for c, n in zip(cached, new))
        kv = 2 * cfg.kv_head_num * D * e * layers * (sum(cached) + t)  # rows of earlier tokens read, those of the new ones written
        nbytes = layers * weights * (0.5 + 4 / GROUP) + kv + 2 * t * cfg.hidden
        flops = 2 * t * layers * weights + 4 * D * cfg.head_num * layers * pairs
        if kind == "decode":
            return dict(bytes=nbytes + VOCAB * (2 * cfg.hidden + 4 * t), flops=flops + 2 * t * VOCAB * cfg.hidden)
        return dict(bytes=nbytes + 2 * t * cfg.hidden, flops=flops)
    if kind == "dense":
        n, k, t = case["n"], case["k"], case["tokens"]
        return dict(bytes=2 * (n * k + t * k + t * n), flops=2 * t * n * k)
    if kind == "window":
        at, b = case["history"], case["batch"]
        keys = min(at, case["window"] - 1) + (max(0, (at - case["window"] + 1) // case["pool"]) if case["pool"] else 0) + 1
        return dict(bytes=b * (4 * KV_HEADS * keys * D + 2 * (2 * HEADS + 2 * KV_HEADS) * D), flops=4 * D * HEADS * b * keys)
    if kind == "delta":
        n, rows, b = DELTA_HEADS * DELTA_DIM, case["batch"] * case["tokens"], case["batch"]
        return dict(bytes=2 * rows * (6 * n + DELTA_RANK) + 4 * b * n * DELTA_DIM + 2 * n * DELTA_RANK, flops=rows * n * (7 * DELTA_DIM + 2 * DELTA_RANK))
    if kind == "chunk":
        t, c = case["tokens"], case["chunk"]
        pairs = case["batch"] * sum(m * (m + 1) // 2 for m in [c] * (t // c) + [t % c])
        rows = case["batch"] * t
        return dict(bytes=2 * rows * (2 * HEADS + 4 * KV_HEADS) * D, flops=pairs * HEADS * (4 * D + 2 * HEADS))
    t = case["tokens"]
    share = TOP / (EXPERTS + IDENTITY)  # of the experts a token takes; used: those that some token takes
    used = EXPERTS * (1 - (1 - share) ** t)
    return dict(bytes=used * 6 * EXPERT_FF * WIDTH + t * WIDTH * 14, flops=6 * t * TOP * EXPERTS / (EXPERTS + IDENTITY) * EXPERT_FF * WIDTH)


def tolerance(case):
    """About four times the largest error against ``exact`` over the listed and drawn cases.  Whole models add up the fp16 rounding
    of every layer; with an int8 cache a rounding that falls the other way is worth a step of 1/127 of the range."""
    kind = case["kind"]
    if kind == "decode":
        return {"rel": 3e-2 if case["layers"] > 8 else 1.5e-2}
    if kind == "prefill":
        return {"rel": 3e-2 if case["int8"] else 1.6e-2}
    return {"rel": dict(linear=1.5e-3, dense=7e-3, window=1.1e-2, delta=7e-3, chunk=1e-2, experts=7e-3)[kind]}
