"""The work that programs built on this framework have it do, as cases to time and to compare.

Three families, at the sizes of the configurations that `bench.py` and `bench_lm.py` run:

* ``sid``: trie-constrained semantic-ID beam search with the 28-layer FP8 decoder (hidden 2048). A pass is one wave of
  decode steps over prompts that are in the cache already, or a whole request: prompts, first level from their last
  tokens, decode steps.
* ``dibepel`` and ``kotipel``: the 16/32-bit decoders behind the step engine. A pass opens its requests, feeds their prompts
  (whole, or in portions), runs ``new`` one-token steps over all of them and closes them. The tokens are given, as when
  continuations are scored, so that every pass does the same work; the logits of every step are returned.

Everything is made from the seed: weights, prompts, catalog."""

import math

import torch

DEVICE = "cuda:0"
VOCAB = 32768
TOKEN_BASE = 151936  # of the SID tokens; ordinary tokens are below
HIDDEN, Q_HEADS, KV_HEADS, HEAD_DIM, FF, SID_LAYERS = 2048, 16, 8, 128, 6144, 28
# width, heads, kv heads, ff, and for Kotipel the heads of the gated linear attention and of the state-space recurrence
SIZES = {"1.7b": (2048, 16, 8, 6144, 16, 64), "8b": (4096, 32, 8, 12288, 32, 128)}
WINDOW, KEEP, CHUNK, SIDE, RANK = 1024, 4, 1024, 256, 16
DTYPES = {"bf16": torch.bfloat16, "f32": torch.float32}


def _sid(name, requests, beams, shortest, longest, shared, levels, width, items, prefill):
    case = dict(family="sid", requests=requests, beams=beams, shortest=shortest, longest=longest, shared=shared, levels=levels,
                width=width, items=items, prefill=prefill)
    return dict(case, name=name) if name else case


def _lm(name, family, size, layers, dtype, requests, shortest, longest, new, portion, every):
    case = dict(family=family, size=size, layers=layers, dtype=dtype, requests=requests, shortest=shortest, longest=longest, new=new,
                portion=portion, every=every)
    return dict(case, name=name) if name else case


def listed():
    return [
        # one user waits for recommendations: a single request's beams, every product has 512 rows
        _sid("sid_wave_1x512", 1, 512, 640, 640, 64, 3, 8192, 1_000_000, False),
        # a few users with short histories and the smaller beam width, prompts included; no row count is a multiple of 32
        _sid("sid_request_7x50", 7, 50, 33, 300, 20, 3, 8192, 200_000, True),
        # a saturated server: 32 requests of 512 beams, prompts of 128 to 1024 tokens in the cache
        _sid("sid_wave_32x512", 32, 512, 128, 1024, 64, 3, 8192, 1_000_000, False),
        # long histories: the prompts are most of the work; four levels of 4096 codes
        _sid("sid_request_8x128_long", 8, 128, 1024, 3072, 64, 4, 4096, 1_000_000, True),
        # one conversation: a prompt of a page or so and a short answer, token after token
        _lm("dibepel_chat_1", "dibepel", "1.7b", 8, "bf16", 1, 777, 777, 24, 0, 0),
        # many requests at once: ragged prompts, then decoding as one batch
        _lm("dibepel_batch_64", "dibepel", "1.7b", 8, "bf16", 64, 40, 260, 16, 0, 0),
        # one long document, the logits of every 64th token
        _lm("dibepel_document_8192", "dibepel", "1.7b", 8, "bf16", 1, 8192, 8192, 0, 0, 64),
        # the smallest call: a short question and a few tokens of answer
        _lm("kotipel_chat_1", "kotipel", "1.7b", 8, "bf16", 1, 37, 37, 24, 0, 0),
        _lm("kotipel_batch_48", "kotipel", "1.7b", 8, "bf16", 48, 50, 333, 16, 0, 0),
        _lm("kotipel_document_8192", "kotipel", "1.7b", 8, "bf16", 1, 8192, 8192, 0, 0, 64),
        # the larger layers: ragged prompts in portions of 1024 tokens, then a few tokens each
        _lm("kotipel_8b_portions", "kotipel", "8b", 4, "bf16", 5, 500, 3001, 8, 1024, 0),
        # 32-bit arithmetic throughout, for checking a model: short prompts and a few tokens
        _lm("dibepel_f32", "dibepel", "1.7b", 4, "f32", 3, 50, 201, 6, 0, 0),
    ]


def draw(rng):
    def log(lo, hi):
        return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))

    family = rng.choice(["sid", "dibepel", "kotipel"])
    if family == "sid":
        requests = log(1, 32)
        beams = log(16, min(512, 8192 // requests))
        longest = min(log(48, 3072), 16384 // requests)
        shortest = log(max(32, longest // 8), longest)
        return _sid(None, requests, beams, shortest, longest, rng.randrange(0, min(65, shortest)), rng.choice([3, 4]),
                    rng.choice([4096, 8192]), log(50_000, 1_000_000), rng.random() < 0.5)
    dtype = "f32" if rng.random() < 0.15 else "bf16"
    if dtype == "f32":
        longest = log(16, 250)
        return _lm(None, family, "1.7b", 4, dtype, rng.randrange(1, 4), log(8, longest), longest, rng.randrange(2, 8), 0, 0)
    size = rng.choice(["1.7b", "1.7b", "8b"])
    requests = log(1, 64)
    longest = log(24, 8192 // requests)
    new = 0 if longest > 4000 else rng.randrange(4, 25)
    return _lm(None, family, size, 8 if size == "1.7b" else 4, dtype, requests, log(max(8, longest // 6), longest), longest, new,
               rng.choice([0, 0, 512, 1024]), 0 if new else 64)


# ---- what both sides need: sizes, configurations, weights, tokens ------------------------------------------------------
def _lengths(case):
    """Prompt lengths from the shortest to the longest, spread over their logarithm, in an order of their own."""
    n, lo, hi = case["requests"], case["shortest"], case["longest"]
    if n == 1:
        return [hi]
    step = next(s for s in (5, 7, 11, 13, 1) if math.gcd(s, n) == 1)
    return [round(lo * (hi / lo) ** ((i * step % n) / (n - 1))) for i in range(n)]


def _lm_config(case):
    width, heads, kv, ff, linear, ssm = SIZES[case["size"]]
    layers = []
    for i in range(case["layers"]):
        first = i % 2 == 0
        if case["family"] == "dibepel" and first:
            kind, mixer = "attention", dict(heads=heads, kv_heads=kv, dim=64, vdim=128, scale=64 ** -0.5, diff=0.2,
                                            mask=dict(size=WINDOW, keep_first=KEEP))
        elif case["family"] == "dibepel":
            kind, mixer = "attention_2", dict(heads=heads, kv_heads=kv, dim=128, vdim=128, scale=128 ** -0.5, conv=4,
                                              mask=dict(size=CHUNK))
        elif first:
            kind, mixer = "mamba2", dict(heads=ssm, vdim=64, state=128, groups=8, conv=4, norm_groups=1)
        else:
            rot = dict(dims=128, base=5e5, scaling=dict(factor=8.0, low=1.0, high=4.0, original=8192))
            kind, mixer = "parallel", dict(left=dict(heads=heads, kv_heads=kv, dim=128, vdim=128, rot=rot, scale=128 ** -0.5),
                                           right=dict(heads=linear, dim=64, vdim=128, tau=16.0))
        layers.append(dict(type=kind, mixer=mixer, mlp=dict(kind="dense", ff=ff, limit=7.0)))
    cfg = dict(vocab=VOCAB, width=width, norm=dict(eps=1e-5), layers=layers)
    if case["family"] == "dibepel":
        return dict(cfg, architecture="Dibepel", embedding=dict(scale=1.0))
    return dict(cfg, architecture="Kotipel", token_side=dict(dim=SIDE))


def _lm_shapes(case):
    """Name and shape of every tensor of a checkpoint."""
    cfg = _lm_config(case)
    w, out = cfg["width"], {"embed": (VOCAB, cfg["width"]), "final.norm": (cfg["width"],)}
    if case["family"] == "dibepel":
        out["head"] = (VOCAB, w)
    else:
        out["side.embed"] = (VOCAB, len(cfg["layers"]) * SIDE)
    for i, e in enumerate(cfg["layers"]):
        m, ff, p = e["mixer"], e["mlp"]["ff"], f"l{i}."
        mix = {}
        if case["family"] == "dibepel":
            maps = 2 if e["type"] == "attention" else 1
            q, k, v = m["heads"] * maps * m["dim"], m["kv_heads"] * maps * m["dim"], m["kv_heads"] * m["vdim"]
            mix = {"q": (q, w), "k": (k, w), "v": (v, w), "o": (w, m["heads"] * m["vdim"])}
            if maps == 2:
                mix.update({n: (m["dim"],) for n in ("lq1", "lk1", "lq2", "lk2")})
            else:
                mix.update({"q.conv": (q, 4), "k.conv": (k, 4), "v.conv": (v, 4), "talk": (m["heads"], m["heads"])})
            out.update({p + "rg1": (w, w), p + "rg1.b": (w,), p + "rg2": (w, w), p + "rg2.b": (w,)})
        elif e["type"] == "mamba2":
            inner, h = m["heads"] * m["vdim"], (m["heads"],)
            channels = inner + 2 * m["groups"] * m["state"]
            mix = {"in": (inner + channels + m["heads"], w), "conv": (channels, 4), "conv.b": (channels,), "dt_bias": h, "A_log": h,
                   "D": h, "norm": (inner,), "o": (w, inner)}
        else:
            a, g = m["left"], m["right"]
            q, k, n, v = a["heads"] * a["dim"], a["kv_heads"] * a["dim"], g["heads"] * g["dim"], g["heads"] * g["vdim"]
            mix = {"left.q": (q, w), "left.k": (k, w), "left.v": (k, w), "left.q.norm": (q,), "left.k.norm": (k,),
                   "left.g": (a["heads"], w), "left.o": (w, q), "left.out": (w,), "right.q": (n, w), "right.k": (n, w),
                   "right.v": (v, w), "right.g": (v, w), "right.o": (w, v), "right.norm": (g["vdim"],), "right.a1": (RANK, w),
                   "right.a2": (n, RANK), "right.a2.b": (n,), "right.out": (w,)}
        out[p + "norm1"] = (w,)
        out.update({p + "mix." + n: s for n, s in mix.items()})
        out.update({p + "mlp.gate": (ff, w), p + "mlp.up": (ff, w), p + "mlp.down": (w, ff)})
        if case["family"] == "kotipel":
            out.update({p + "norm2": (w,), p + "side.gate": (SIDE, w), p + "side.proj": (w, SIDE), p + "side.norm": (w,)})
    return out


def _lm_tensors(case, seed):
    """A checkpoint's tensors: matrices of 1 / sqrt(fan in), norms around what they are stored around, decays that forget within
    tens to thousands of tokens."""
    g = torch.Generator(device=DEVICE)
    g.manual_seed(seed)
    out = {}
    for name, shape in _lm_shapes(case).items():
        t = torch.randn(shape, generator=g, device=DEVICE, dtype=torch.bfloat16 if len(shape) == 2 else torch.float32)
        if name.endswith(("norm", "norm1", "norm2", "left.out", "right.out")):
            t = 0.1 * t if case["family"] == "dibepel" else 1 + 0.2 * t
        elif name.endswith((".b", "D")):
            t = (0.1 if case["family"] == "dibepel" else 0.5) * t
        elif name.endswith(("lq1", "lk1", "lq2", "lk2")):
            t = 0.1 * t
        elif name.endswith("dt_bias"):
            t = t - 2
        elif name.endswith("A_log"):
            t = 0.7 * t
        elif name.endswith(".conv"):
            t = 0.5 * t
        elif name not in ("embed", "side.embed"):
            t = t * shape[-1] ** -0.5
        out[name] = t.to(torch.bfloat16)
    return out


def _lm_tokens(case, seed):
    """Per request its prompt and the tokens that follow."""
    g = torch.Generator().manual_seed(seed + 1)
    return [torch.randint(0, VOCAB, (n + case["new"],), generator=g).tolist() for n in _lengths(case)]


def _wanted(case, n):
    """Places of a prompt of ``n`` tokens whose logits are asked for."""
    return sorted(set(range(case["every"] - 1, n, case["every"])) | {n - 1}) if case["every"] else [n - 1]


def _portions(case):
    """Per step the (first, last) tokens of every request's prompt."""
    lens, size = _lengths(case), case["portion"] or case["longest"]
    return [[(min(s, n), min(s + size, n)) for n in lens] for s in range(0, max(lens), size)]


# ---- the framework's side ----------------------------------------------------------------------------------------------
def prepare(case, seed):
    """The server as it stands before the call: model, caches and captured steps, and the tokens of the requests."""
    if case["family"] == "sid":
        from flashrec_b200.decoder import Qwen3Config
        from flashrec_b200.sid_decode import SidDecodeEngine
        from flashrec_b200.trie import build_trie_device

        levels, width = case["levels"], case["width"]
        g = torch.Generator(device=DEVICE)
        g.manual_seed(seed)
        items = torch.randint(0, width, (case["items"], levels), generator=g, device=DEVICE, dtype=torch.int32)
        trie = build_trie_device(items, [width] * levels, TOKEN_BASE)
        cfg = Qwen3Config(hidden_size=HIDDEN, num_attention_heads=Q_HEADS, num_key_value_heads=KV_HEADS, head_dim=HEAD_DIM,
                          intermediate_size=FF, num_hidden_layers=SID_LAYERS, vocab_size=TOKEN_BASE + levels * width)
        eng = SidDecodeEngine(cfg, case["requests"], case["beams"], _lengths(case), [width] * levels, TOKEN_BASE, trie, DEVICE,
                              shared_prefix=case["shared"], seed=seed, level0_from_prefill=case["prefill"])
        if case["prefill"]:
            eng.prefill()
        eng.capture()
        return dict(case=case, engine=eng, items=items)
    from flashrec_b200 import dibepel, kotipel
    from flashrec_b200.engine import LMEngine, StepEntry

    cfg, tensors = _lm_config(case), _lm_tensors(case, seed)
    if case["family"] == "dibepel":
        model = dibepel.DibepelForCausalLM(dibepel.DibepelConfig.from_json(cfg), tensors, DTYPES[case["dtype"]], DEVICE)
    else:
        model = kotipel.KotipelForCausalLM(kotipel.KotipelConfig.from_json(cfg), tensors, DTYPES[case["dtype"]], DEVICE)
    n, toks = case["requests"], _lm_tokens(case, seed)
    eng = LMEngine(model, sum(-(-len(t) // 64) * 64 for t in toks), n, max(len(t) for t in toks))
    if case["new"]:  # the decode step of this batch is captured when a server starts
        eng.step([StepEntry(r, [0], [0]) for r in range(n)])
        for r in range(n):
            eng.finish(r)
    return dict(case=case, engine=eng, tokens=toks)


def run(state):
    case, eng = state["case"], state["engine"]
    if case["family"] == "sid":
        if case["prefill"]:
            eng.prefill()
        eng.run(host_io=False)
        return dict(scores=[o.vals for o in eng.outs], tokens=eng.final_tokens)
    from flashrec_b200.engine import StepEntry

    toks, lens, out = state["tokens"], _lengths(case), []
    for spans in _portions(case):
        entries = []
        for r, (a, b) in enumerate(spans):
            if b > a:
                entries.append(StepEntry(r, toks[r][a:b], [w - a for w in _wanted(case, lens[r]) if a <= w < b]))
        out.append(eng.step(entries))
    for i in range(case["new"]):
        out.append(eng.step([StepEntry(r, [toks[r][lens[r] + i]], [0]) for r in range(case["requests"])]))
    for r in range(case["requests"]):
        eng.finish(r)
    return out


# ---- what a pass cannot do without -------------------------------------------------------------------------------------
def work(case):
    lens = _lengths(case)
    if case["family"] == "sid":
        rows, n, steps = case["requests"] * case["beams"], case["requests"], case["levels"]
        layer = HIDDEN * (Q_HEADS + 2 * KV_HEADS) * HEAD_DIM + HIDDEN * Q_HEADS * HEAD_DIM + 3 * HIDDEN * FF
        kv = 2 * KV_HEADS * HEAD_DIM * SID_LAYERS  # bytes of a token's keys and values
        flops = byts = 0
        if case["prefill"]:
            own = [lens[0]] + [m - case["shared"] for m in lens[1:]]
            pairs = sum(o * (m - o) + o * (o + 1) // 2 for o, m in zip(own, lens))
            flops += 2 * sum(own) * layer * SID_LAYERS + 4 * pairs * Q_HEADS * HEAD_DIM * SID_LAYERS + 2 * n * case["width"] * HIDDEN
            byts += layer * SID_LAYERS + case["width"] * HIDDEN + sum(own) * kv
            steps -= 1
        unique = case["shared"] + sum(m - case["shared"] for m in lens)
        pairs = sum(lens) * case["beams"]
        per = 2 * rows * (layer * SID_LAYERS + case["width"] * HIDDEN) + 4 * pairs * Q_HEADS * HEAD_DIM * SID_LAYERS
        flops += per * steps
        byts += (layer * SID_LAYERS + case["width"] * HIDDEN + (unique + rows) * kv) * steps
        return dict(bytes=byts, flops=flops)
    es = DTYPES[case["dtype"]].itemsize
    cfg, shapes = _lm_config(case), _lm_shapes(case)
    mats = sum(s[0] * s[1] for n, s in shapes.items() if n.startswith("l") and len(s) == 2 and "conv" not in n)
    tokens, w = sum(lens) + case["requests"] * case["new"], cfg["width"]
    wanted = sum(len(_wanted(case, n)) for n in lens) + case["requests"] * case["new"]
    flops = 2 * mats * tokens + 2 * wanted * VOCAB * w
    steps = len(_portions(case)) + case["new"]
    byts = steps * (mats + VOCAB * w) * es + wanted * VOCAB * 4
    for e in cfg["layers"]:
        m = e["mixer"]

        def seen(p, kind=e["type"]):  # keys that the query at position p sees
            return p % CHUNK + 1 if kind == "attention_2" else min(p + 1, WINDOW + KEEP) if kind == "attention" else p + 1

        a = m["left"] if e["type"] == "parallel" else m
        if e["type"] != "mamba2":
            maps = 2 if e["type"] == "attention" else 1
            cols = maps * (a["dim"] + a["vdim"])
            pairs = sum(seen(p) for n in lens for p in range(n + case["new"]))
            flops += 2 * pairs * a["heads"] * cols
            read = sum(seen(n + i) for n in lens for i in range(case["new"]))
            byts += (read + tokens) * a["kv_heads"] * (maps * a["dim"] + a["vdim"]) * es
        s = (m["heads"], m["state"], m["vdim"]) if e["type"] == "mamba2" else \
            (m["right"]["heads"], m["right"]["dim"], m["right"]["vdim"]) if e["type"] == "parallel" else (0, 0, 0)
        flops += 4 * tokens * s[0] * s[1] * s[2]
        byts += case["requests"] * (2 * case["new"] + 1) * s[0] * s[1] * s[2] * 4
    return dict(bytes=byts, flops=flops)


def tolerance(case):
    """Measured against ``exact``, times four: the bf16 models are 0.5 to 0.9 % off in the norm and 5 % of the root mean square
    in the worst logit, float32 1.5e-6 and 7e-6. Beam scores are 0.3 to 1 % off what unrounded activations give, and less from
    another order of sums; beams that are closer than that may change places."""
    if case["family"] == "sid":
        return dict(rel=1e-2, max=0.1, differ=0.01)
    return dict(rel=6e-6, max=3e-5) if case["dtype"] == "f32" else dict(rel=3e-2, max=0.2)


# ---- the same in 64 bits -----------------------------------------------------------------------------------------------
def exact(case, seed):
    w = work(case)
    if w["flops"] > 4e14:
        return None
    if case["family"] == "sid":
        return _sid_exact(case, seed)
    lens, toks = _lengths(case), _lm_tokens(case, seed)
    longest = max(len(t) for t in toks)
    ids = torch.tensor([t + [0] * (longest - len(t)) for t in toks], device=DEVICE)  # causal: what pads the end is not seen
    tensors = _lm_tensors(case, seed)
    x = _lm_exact(case, tensors, ids)
    head = tensors["head" if case["family"] == "dibepel" else "embed"].double()
    out = []
    for spans in _portions(case):
        at = [(r, p) for r, (a, b) in enumerate(spans) for p in _wanted(case, lens[r]) if a <= p < b]
        out.append(torch.stack([x[r, p] for r, p in at]) @ head.T if at else torch.empty((0, VOCAB), device=DEVICE).double())
    for i in range(case["new"]):
        out.append(torch.stack([x[r, n + i] for r, n in enumerate(lens)]) @ head.T)
    return out


def _rms(x, eps=1e-5):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _conv(u, w, b=None):
    y = sum(torch.nn.functional.pad(u, (0, 0, j, 0))[:, :u.shape[1]] * w[:, w.shape[1] - 1 - j] for j in range(w.shape[1]))
    return y if b is None else torch.nn.functional.silu(y + b)


def _weights(q, k, visible, at, scale, slopes=None):
    """q [B, H, n, d] of the places ``at``, k [B, H, T, d]: softmax over the visible keys."""
    s = q @ k.transpose(-1, -2) * scale
    if slopes is not None:
        s = s - slopes[:, None, None] * (at[:, None] - torch.arange(k.shape[2], device=DEVICE))
    return torch.softmax(s.masked_fill(~visible, float("-inf")), dim=-1)


def _attend(q, k, v, m, kind, talk=None, lam=0.0):
    """q [B, T, maps, H, d], k [B, T, maps, G, d], v [B, T, G, e] -> [B, T, H, e], a block of queries at a time."""
    b, t, heads = q.shape[0], q.shape[1], q.shape[3]
    rep = heads // k.shape[3]
    slopes = torch.tensor([2.0 ** (-8.0 * (h + 1) / heads) for h in range(heads)], device=DEVICE).double() if kind == "talk" else None
    j = torch.arange(t, device=DEVICE)
    out = torch.empty((b, t, heads, v.shape[-1]), dtype=torch.float64, device=DEVICE)
    step = max(16, (1 << 28) // (t * heads * 4))
    for r in range(b):
        kr = [k[r:r + 1, :, i].repeat_interleave(rep, 2).transpose(1, 2) for i in range(k.shape[2])]
        vr = v[r:r + 1].repeat_interleave(rep, 2).transpose(1, 2)
        for s in range(0, t, step):
            at = j[s:s + step]
            hi = int(at[-1]) + 1
            i = at[:, None]
            vis = j[None, :hi] <= i
            if kind == "diff":
                vis = vis & ((i - j[None, :hi] < WINDOW) | (j[None, :hi] < KEEP))
            if kind == "talk":
                vis = vis & (i // CHUNK == j[None, :hi] // CHUNK)
            p = [_weights(q[r:r + 1, s:s + step, n].transpose(1, 2), kr[n][:, :, :hi], vis, at, m["scale"], slopes)
                 for n in range(len(kr))]
            w = p[0] - lam * p[1] if kind == "diff" else torch.einsum("hg,bgij->bhij", talk, p[0]) if kind == "talk" else p[0]
            out[r:r + 1, s:s + step] = (w @ vr[:, :, :hi]).transpose(1, 2)
    return out


def _recur(q, k, u, decay):
    """S <- decay S + k u^T, o = S^T q, token after token; q, k [B, T, H, N], u [B, T, H, V], decay [B, T, H, N or 1]."""
    b, t, h, n = k.shape
    s = torch.zeros((b, h, n, u.shape[-1]), dtype=torch.float64, device=DEVICE)
    out = torch.empty_like(u)
    for i in range(t):
        s = s * decay[:, i, :, :, None] + k[:, i, :, :, None] * u[:, i, :, None, :]
        out[:, i] = (q[:, i, :, None, :] @ s)[:, :, 0]
    return out


def _rotate(x, freqs):
    """x [B, T, H, d]: dimension i turns with i + d / 2."""
    a = torch.arange(x.shape[1], device=DEVICE).double()[:, None] * freqs
    c, s, half = a.cos()[:, None], a.sin()[:, None], x.shape[-1] // 2
    return torch.cat([x[..., :half] * c - x[..., half:] * s, x[..., half:] * c + x[..., :half] * s], dim=-1)


def _frequencies(rot):
    f = rot["base"] ** (-torch.arange(0, rot["dims"], 2, device=DEVICE).double() / rot["dims"])
    sc, length = rot["scaling"], 2 * math.pi / f
    s = (sc["original"] / length - sc["low"]) / (sc["high"] - sc["low"])
    mid = (1 - s) * f / sc["factor"] + s * f
    return torch.where(length > sc["original"] / sc["low"], f / sc["factor"], torch.where(length < sc["original"] / sc["high"], f, mid))


def _lm_exact(case, tensors, ids):
    """The final norm's output [B, T, width] of whole sequences."""
    cfg, silu, softplus = _lm_config(case), torch.nn.functional.silu, torch.nn.functional.softplus
    b, t = ids.shape
    x = tensors["embed"][ids].double()
    for i, e in enumerate(cfg["layers"]):
        W = lambda n, p=f"l{i}.": tensors[p + n].double()  # noqa: E731
        m, heads = e["mixer"], lambda y, *s: y.view(b, t, *s)  # noqa: E731
        if case["family"] == "dibepel":
            h = _rms(x) * (1 + W("norm1"))
            q, k, v = h @ W("mix.q").T, h @ W("mix.k").T, h @ W("mix.v").T
            H, G, d = m["heads"], m["kv_heads"], m["dim"]
            if e["type"] == "attention":
                lam = math.exp((W("mix.lq1") * W("mix.lk1")).sum()) - math.exp((W("mix.lq2") * W("mix.lk2")).sum()) + m["diff"]
                o = _attend(heads(q, H, 2, d).transpose(2, 3), heads(k, G, 2, d).transpose(2, 3), heads(v, G, m["vdim"]), m, "diff", lam=lam)
                o = _rms(o) * (1 - m["diff"])
            else:
                q, k, v = _conv(q, W("mix.q.conv")), _conv(k, W("mix.k.conv")), _conv(v, W("mix.v.conv"))
                o = _attend(heads(q, 1, H, d), heads(k, 1, G, d), heads(v, G, m["vdim"]), m, "talk", talk=W("mix.talk"))
            y = torch.sigmoid(h @ W("rg1").T + W("rg1.b")) * (o.reshape(b, t, -1) @ W("mix.o").T)
            ff = (silu(h @ W("mlp.gate").T) * (h @ W("mlp.up").T)) @ W("mlp.down").T
            x = x + y + torch.sigmoid(h @ W("rg2").T + W("rg2.b")) * ff
            continue
        h = _rms(x) * W("norm1")
        if e["type"] == "mamba2":
            H, V, N, G = m["heads"], m["vdim"], m["state"], m["groups"]
            z, u, dt = torch.split(h @ W("mix.in").T, [H * V, H * V + 2 * G * N, H], dim=-1)
            xs, bb, cc = torch.split(_conv(u, W("mix.conv"), W("mix.conv.b")), [H * V, G * N, G * N], dim=-1)
            dt = softplus(dt + W("mix.dt_bias"))
            xs, bb, cc = heads(xs, H, V), heads(bb, G, N).repeat_interleave(H // G, 2), heads(cc, G, N).repeat_interleave(H // G, 2)
            o = _recur(cc, bb, xs * dt[..., None], torch.exp(-torch.exp(W("mix.A_log")) * dt)[..., None]) + W("mix.D")[:, None] * xs
            x = x + (_rms(o.reshape(b, t, -1) * silu(z)) * W("mix.norm")) @ W("mix.o").T
        else:
            a, g = m["left"], m["right"]
            f = _frequencies(a["rot"])
            q = _rotate(heads(_rms(h @ W("mix.left.q").T) * W("mix.left.q.norm"), a["heads"], a["dim"]), f)
            k = _rotate(heads(_rms(h @ W("mix.left.k").T) * W("mix.left.k.norm"), a["kv_heads"], a["dim"]), f)
            o = _attend(q[:, :, None], k[:, :, None], heads(h @ W("mix.left.v").T, a["kv_heads"], a["vdim"]), a, "plain")
            left = (o * torch.sigmoid(h @ W("mix.left.g").T)[..., None]).reshape(b, t, -1) @ W("mix.left.o").T
            n, d = g["heads"], g["dim"]
            z = (h @ W("mix.right.a1").T) @ W("mix.right.a2").T + W("mix.right.a2.b")
            o = _recur(heads(h @ W("mix.right.q").T, n, d) * d ** -0.5, heads(h @ W("mix.right.k").T, n, d),
                       heads(h @ W("mix.right.v").T, n, g["vdim"]), heads(torch.exp(-softplus(-z) / g["tau"]), n, d))
            right = ((_rms(o) * W("mix.right.norm")).reshape(b, t, -1) * silu(h @ W("mix.right.g").T)) @ W("mix.right.o").T
            x = x + 0.5 * (_rms(left) * W("mix.left.out") + _rms(right) * W("mix.right.out"))
        h = _rms(x) * W("norm2")
        gate, up = (h @ W("mlp.gate").T).clamp(max=7.0), (h @ W("mlp.up").T).clamp(-7.0, 7.0)
        x = x + (gate * torch.sigmoid(1.702 * gate) * (up + 1)) @ W("mlp.down").T
        side = torch.nn.functional.gelu(x @ W("side.gate").T, approximate="tanh") * tensors["side.embed"][ids][..., i * SIDE:(i + 1) * SIDE]
        x = x + _rms(side @ W("side.proj").T) * W("side.norm")
    final = tensors["final.norm"].double()
    return _rms(x) * (1 + final if case["family"] == "dibepel" else final)


def _sid_exact(case, seed):
    """Sorted scores of every level with the stored e4m3 weights and prompt keys, nothing else rounded; no tokens: beams whose
    scores are closer than the rounding of 8-bit activations change places."""
    state = prepare(case, seed)
    eng, n, bw, width = state["engine"], case["requests"], case["beams"], case["width"]
    lens, layers, G, D = _lengths(case), eng.model.layers, KV_HEADS, HEAD_DIM

    def dense(w, s):
        return w.double() * s.double().reshape(-1, 1)

    def matrices(l):
        a, mlp = l.self_attn, l.mlp
        gu = dense(mlp._gu_w, mlp._gu_s)  # blocks of 128 gate rows and 128 up rows
        gate, up = gu.view(-1, 2, 128, HIDDEN).unbind(1)
        return (dense(a.qkv_proj._fp8_weight.t(), a.qkv_proj._fp8_scale), dense(a.o_proj._fp8_weight.t(), a.o_proj._fp8_scale),
                gate.reshape(-1, HIDDEN), up.reshape(-1, HIDDEN), dense(mlp.down_proj._fp8_weight.t(), mlp.down_proj._fp8_scale))

    freqs = 1e6 ** (-torch.arange(0, D, 2, device=DEVICE).double() / D)

    def turn(x, pos):  # x [T, H, D]
        a = pos.double()[:, None, None] * freqs
        x1, x2 = x[..., :D // 2], x[..., D // 2:]
        return torch.cat([x1 * a.cos() - x2 * a.sin(), x2 * a.cos() + x1 * a.sin()], dim=-1)

    def forward(x, pos, attend):
        for i, l in enumerate(layers):
            qkv_w, o_w, gate, up, down = matrices(l)
            qkv = (_rms(x, 1e-6) @ qkv_w.T).view(x.shape[0], Q_HEADS + 2 * G, D)
            q, k = turn(_rms(qkv[:, :Q_HEADS], 1e-6), pos), turn(_rms(qkv[:, Q_HEADS:Q_HEADS + G], 1e-6), pos)
            x = x + attend(i, q, k, qkv[:, Q_HEADS + G:]).reshape(x.shape[0], -1) @ o_w.T
            h = _rms(x, 1e-6)
            x = x + (torch.nn.functional.silu(h @ gate.T) * (h @ up.T)) @ down.T
        return _rms(x, 1e-6)

    def soft(q, k, v, hidden=None):  # q [T, Hq, D], k, v [S, G, D]
        qg = q.view(q.shape[0], G, -1, D).permute(1, 2, 0, 3)
        s = qg @ k.permute(1, 2, 0)[:, None] / math.sqrt(D)
        s = s if hidden is None else s.masked_fill(hidden, float("-inf"))
        return s, qg

    # keys and values of every prompt: as the cache holds them, or computed from the prompts' tokens
    table = eng.req_to_token[eng.rows:].long()
    prompts = [[(eng.pool.k[i][table[r, :m]].double(), eng.pool.v[i][table[r, :m]].double()) for r, m in enumerate(lens)]
               for i in range(len(layers))] if not case["prefill"] else [[None] * n for _ in layers]
    first = []
    if case["prefill"]:
        g = torch.Generator().manual_seed(seed + 17)
        shared = torch.randint(0, TOKEN_BASE, (case["shared"],), generator=g)
        for r, m in enumerate(lens):
            ids = torch.cat([shared[:m], torch.randint(0, TOKEN_BASE, (m - min(case["shared"], m),), generator=g)]).to(DEVICE)
            hidden = torch.ones((m, m), dtype=torch.bool, device=DEVICE).triu(1)

            def attend(i, q, k, v, r=r, hidden=hidden):
                prompts[i][r] = (k, v)
                s, _ = soft(q, k, v, hidden)
                return (torch.softmax(s, -1) @ v.transpose(0, 1)[:, None]).permute(2, 0, 1, 3).reshape(q.shape)

            first.append(forward(eng.model.embed_tokens[ids].double(), torch.arange(m, device=DEVICE), attend)[-1])
    # legal codes: sorted prefixes of the catalog
    prefixes, key = [], torch.zeros(case["items"], dtype=torch.int64, device=DEVICE)
    for l in range(case["levels"]):
        key = key * width + state["items"][:, l].long()
        prefixes.append(torch.unique(key))
    codes = torch.arange(width, device=DEVICE)

    def extend(cum, node, hidden, level):
        """cum, node [n, rows]; hidden [n * rows, H] -> scores, parents, nodes, codes of the best beams"""
        head = dense(eng.head._level_weights[level], eng.head._level_scales[level])
        vals, par, nod, cod = [], [], [], []
        for r in range(n):
            rows = cum.shape[1]
            lp = torch.log_softmax(hidden[r * rows:(r + 1) * rows] @ head.T, -1)
            cand = node[r][:, None] * width + codes
            pre = prefixes[level]
            at = torch.searchsorted(pre, cand).clamp(max=pre.numel() - 1)
            score = (lp + cum[r][:, None]).masked_fill(pre[at] != cand, float("-inf")).reshape(-1)
            best = torch.topk(score, min(bw, score.numel()))
            v, idx = best.values, best.indices
            if idx.numel() < bw:
                v = torch.cat([v, v.new_full((bw - v.numel(),), float("-inf"))])
                idx = torch.cat([idx, idx.new_zeros(bw - idx.numel())])
            vals.append(v), par.append(idx // width), cod.append(idx % width), nod.append(cand.reshape(-1)[idx])
        return [torch.stack(y) for y in (vals, par, nod, cod)]

    scores = []
    cum, node = torch.zeros((n, 1), dtype=torch.float64, device=DEVICE), torch.zeros((n, 1), dtype=torch.int64, device=DEVICE)
    tok = torch.full((n, 1), TOKEN_BASE, device=DEVICE)
    window = [None] * len(layers)  # the decoded tokens' keys and values [n, rows, steps, G, D]
    start = 0
    if case["prefill"]:
        cum, _, node, code = extend(cum, node, torch.stack(first), 0)
        scores.append(cum)
        tok, start = TOKEN_BASE + code, 1
    for step in range(start, case["levels"]):
        rows = cum.shape[1]

        def attend(i, q, k, v):
            k, v = k.view(n, rows, 1, G, D), v.view(n, rows, 1, G, D)
            if window[i] is not None:
                k, v = torch.cat([window[i][0], k], 2), torch.cat([window[i][1], v], 2)
            window[i] = (k, v)
            out = []
            for r in range(n):
                pk, pv = prompts[i][r]
                s, qg = soft(q[r * rows:(r + 1) * rows], pk, pv)
                own = torch.einsum("gqbd,bsgd->gqbs", qg, k[r]) / math.sqrt(D)
                p = torch.softmax(torch.cat([s, own], -1), -1)
                o = p[..., :s.shape[-1]] @ pv.transpose(0, 1)[:, None] + torch.einsum("gqbs,bsgd->gqbd", p[..., s.shape[-1]:], v[r])
                out.append(o.permute(2, 0, 1, 3).reshape(rows, -1))
            return torch.cat(out)

        pos = torch.tensor(lens, device=DEVICE).repeat_interleave(rows) + step - start
        hidden = forward(eng.model.embed_tokens[tok.reshape(-1)].double(), pos, attend)
        cum, par, node, code = extend(cum, node, hidden, step)
        pick = torch.arange(n, device=DEVICE)[:, None]
        window = [(k[pick, par], v[pick, par]) for k, v in window]
        scores.append(cum)
        tok = TOKEN_BASE + step * width + code
    return dict(scores=scores, tokens=None)
