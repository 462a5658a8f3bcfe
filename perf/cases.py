"""Workloads of the engine: scheduled steps of a decoder (prompts, chunks of long prompts, decoding, verification, mixed batches) over
their real sizes, and the feed-forward projections of the block-quantised preset.

A step is described by the rows that it takes: `prompt` rows of one sequence that has `prompt_context` tokens in its cache already,
and `rows` rows of each of `seqs` further sequences with up to `context` cached tokens.  `layers` of the named model's layers run; what
lies in the caches before the step is drawn at random with the distributions that the layers write.
"""
import math
import zlib

import torch

PAGE = 16
EPS = 1e-6
HIDDEN = {"4b": 2560, "27b": 5120}
FF = {"4b": 9216, "27b": 17408}
VOCAB = 151936
HYBRID = {"4b": dict(hk=16, hv=32, hq=16, hkv=4), "27b": dict(hk=16, hv=48, hq=24, hkv=4)}      # head sizes 128 and 256
GEBUZEN = {"4b": dict(hq=16, hkv=4, h=32), "27b": dict(hq=24, hkv=4, h=48)}
RANK, TAU, BLOCK = 16, 16.0, 4096
ACT_SCALE = 8.0 / 192


def step(family, model, weights, layers, kv, prompt=0, prompt_context=0, seqs=0, rows=1, context=0):
    return dict(family=family, model=model, weights=weights, layers=layers, kv=kv, prompt=prompt, prompt_context=prompt_context,
                seqs=seqs, rows=rows, context=context)


def listed():
    def named(name, case):
        return dict(case, name=name)
    return [
        # one user's chat: a token of a small bf16 model, and of a large one quantised to 4 bits
        named("decode-4b", step("hybrid", "4b", "bf16", 8, "bf16", seqs=1, context=2048)),
        named("decode-27b-nvfp4", step("hybrid", "27b", "nvfp4", 4, "bf16", seqs=1, context=4096)),
        # the rows of a drafted block, checked in one step
        named("verify-4b", step("hybrid", "4b", "bf16", 8, "bf16", seqs=1, rows=8, context=1501)),
        # a short question, a whole prompt, and a chunk late in a long one with 8-bit pages
        named("question-4b", step("hybrid", "4b", "bf16", 8, "fp8_e4m3", prompt=37)),
        named("prompt-4b", step("hybrid", "4b", "bf16", 8, "bf16", prompt=2048)),
        named("chunk-27b", step("hybrid", "27b", "bf16", 4, "fp8_e4m3", prompt=2048, prompt_context=6144)),
        # servers: a few users, many with long contexts in 8-bit pages, and a prompt arriving among decoding users
        named("serve-4b", step("hybrid", "4b", "bf16", 8, "bf16", seqs=12, context=3001)),
        named("serve-27b", step("hybrid", "27b", "bf16", 4, "fp8_e4m3", seqs=32, context=8192)),
        named("mixed-4b", step("hybrid", "4b", "bf16", 8, "bf16", prompt=777, seqs=15, context=2500)),
        # another model family: attention and gated linear attention side by side
        named("gebuzen-prompt-4b", step("gebuzen", "4b", "bf16", 4, "bf16", prompt=1500)),
        named("gebuzen-serve-4b", step("gebuzen", "4b", "bf16", 4, "bf16", seqs=24, context=3500)),
        # the feed-forward of a prompt with 4-bit and 8-bit weights
        named("ff-27b-nvfp4", step("ff", "27b", "nvfp4", 1, "bf16", prompt=2048)),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.4)))))
    kind = rng.choice(("decode", "decode", "verify", "prompt", "prompt", "chunk", "serve", "serve", "mixed", "gebuzen", "gebuzen", "ff"))
    model = rng.choice(("4b", "4b", "27b"))
    layers = 8 if model == "4b" else 4
    kv = rng.choice(("bf16", "fp8_e4m3"))
    if kind == "decode":
        weights = "nvfp4" if model == "27b" else "bf16"
        return step("hybrid", model, weights, layers, kv, seqs=1, context=size(64, 8192))
    if kind == "verify":
        return step("hybrid", model, "bf16", layers, "bf16", seqs=1, rows=rng.randint(2, 16), context=size(64, 8192))
    if kind == "prompt":
        return step("hybrid", model, "bf16", layers, kv, prompt=size(20, 2048))
    if kind == "chunk":
        return step("hybrid", model, "bf16", layers, kv, prompt=size(200, 2048), prompt_context=size(64, 6144))
    if kind == "serve":
        return step("hybrid", model, "bf16", layers, kv, seqs=size(2, 64), context=size(256, 8192))
    if kind == "mixed":
        return step("hybrid", "4b", "bf16", 8, kv, prompt=size(100, 1500), seqs=size(1, 48), context=size(256, 4096))
    if kind == "gebuzen":
        if rng.random() < 0.5:
            return step("gebuzen", "4b", "bf16", 4, "bf16", prompt=size(20, 2048))
        return step("gebuzen", "4b", "bf16", 4, "bf16", seqs=size(1, 64), context=size(256, 4000))
    return step("ff", "27b", "nvfp4", 1, "bf16", prompt=size(2, 2048))


# ---------------------------------------------------------------- the step's rows
def sequences(c):
    """(cached tokens, rows, first row whose logits are read) of the step's sequences; sequence i has slot i."""
    out = [(c["prompt_context"], c["prompt"], c["prompt"] - 1)] if c["prompt"] else []
    for i in range(c["seqs"]):
        share = ((i + 1) * 0.618034) % 1.0 if c["seqs"] > 1 else 1.0
        out.append((max(1, int(c["context"] * (0.05 + 0.95 * share))), c["rows"], 0))
    return out


def pages_of(c, seed):
    """Pages of every sequence, scattered as in a server that has run for a while; page 0 is not handed out."""
    need = [-(-(ctx + n) // PAGE) for ctx, n, _ in sequences(c)]
    at = torch.randperm(sum(need), generator=torch.Generator().manual_seed(seed)) + 1
    return [list(map(int, p)) for p in torch.split(at, need)]


def token_ids(c, seed):
    g = torch.Generator().manual_seed(seed + 1)
    return [torch.randint(0, VOCAB, (n,), generator=g).tolist() for _, n, _ in sequences(c)]


# ---------------------------------------------------------------- random tensors, each from the seed and its name
def normal(seed, name, shape, std=1.0, mean=0.0, dtype=torch.bfloat16):
    g = torch.Generator(device="cuda").manual_seed((seed * 1000003 + zlib.crc32(name.encode())) & 0x7FFFFFFF)
    t = torch.empty(shape, dtype=dtype, device="cuda").normal_(mean, std, generator=g)
    return t


def weight(seed, name, shape):
    if name.endswith("A_log"):
        return normal(seed, name, shape, 0.8, -0.5)
    if name.endswith("dt_bias"):
        return normal(seed, name, shape, 0.5)
    if name.endswith("conv1d.weight"):
        return normal(seed, name, shape, 0.3)
    if name.endswith("linear_attn.norm.weight"):
        return normal(seed, name, shape, 0.05, 1.0)
    if name.endswith("norm.weight"):
        return normal(seed, name, shape, 0.05)
    if name.endswith("embed_tokens.weight"):
        return normal(seed, name, shape)
    # what returns to the residual stream is small beside it, as in models that have been trained
    return normal(seed, name, shape, 0.007 if name.endswith(("out_proj.weight", "o_proj.weight", "down_proj.weight")) else 0.02)


def gebuzen_weight(seed, name, shape):
    if name == "embed":
        return normal(seed, name, shape)
    if name.endswith("a2.b"):
        return normal(seed, name, shape, 1.0, 2.0)
    if name.endswith((".sink", ".b")):
        return normal(seed, name, shape, 0.5)
    return normal(seed, name, shape, 0.1, 1.0) if len(shape) == 1 else normal(seed, name, shape, shape[1] ** -0.5)


# ---------------------------------------------------------------- block formats
def e4m3(x):
    return x.clamp(-448, 448).to(torch.float8_e4m3fn)


def e2m1(x):
    """Codes of the nearest 4-bit values, ties to the even code."""
    m = x.abs()
    code = torch.zeros_like(m, dtype=torch.uint8)
    for i, (edge, open_) in enumerate(((0.25, True), (0.75, False), (1.25, True), (1.75, False), (2.5, True), (3.5, False), (5.0, True))):
        code = torch.where(m > edge if open_ else m >= edge, torch.full_like(code, i + 1), code)
    return code + 8 * ((x < 0) & (code > 0)).to(torch.uint8)


def e2m1_value(code):
    t = torch.tensor([0, 0.5, 1, 1.5, 2, 3, 4, 6, -0.0, -0.5, -1, -1.5, -2, -3, -4, -6], dtype=torch.float64, device=code.device)
    return t[code.long()]


def mx_exponent(amax):
    """Smallest e with amax / 2^e <= 448."""
    m, e = torch.frexp(amax)
    return (e - 9 + (2 * m > 1.75).to(e.dtype)).clamp(-126, 126)


def block_format(name, layer):
    if "in_proj_a" in name or "in_proj_b" in name:
        return "bf16"
    if "embed_tokens" in name or "lm_head" in name:
        return "mxfp8"
    if any(s in name for s in ("down_proj", "in_proj", "out_proj")):
        return "mxfp8" if layer % 4 == 0 else "nvfp4"
    return "nvfp4"


TENSOR_SCALE = 2.0 ** -12


def block_codes(w, fmt):
    """(codes, block scales) as a quantised checkpoint holds them."""
    n, k = w.shape
    codes, scales = [], []
    for part in torch.split(w, 16384):
        v = part.float()
        if fmt == "nvfp4":
            v = v.reshape(-1, k // 16, 16)
            s = e4m3(v.abs().amax(-1) / 6 / TENSOR_SCALE)
            q = e2m1(v / (s.float() * TENSOR_SCALE)[..., None]).reshape(-1, k)
            codes.append(q[:, 0::2] | (q[:, 1::2] << 4))
            scales.append(s.view(torch.uint8))
        else:
            v = v.reshape(-1, k // 32, 32)
            e = mx_exponent(v.abs().amax(-1))
            codes.append(e4m3(v / torch.ldexp(torch.ones_like(v[..., 0]), e)[..., None]).view(torch.uint8).reshape(-1, k))
            scales.append((e + 127).to(torch.uint8))
    return torch.cat(codes), torch.cat(scales)


def block_values(codes, scales, fmt):
    n = codes.shape[0]
    if fmt == "nvfp4":
        q = torch.stack([codes & 15, codes >> 4], -1).reshape(n, -1, 16)
        return (e2m1_value(q) * (scales.view(torch.float8_e4m3fn).double() * TENSOR_SCALE)[..., None]).reshape(n, -1)
    v = codes.view(torch.float8_e4m3fn).double().reshape(n, -1, 32)
    return (v * torch.ldexp(torch.ones_like(v[..., 0]), scales.int() - 127)[..., None]).reshape(n, -1)


class Checkpoint:
    """Source of the hybrid decoder's weights: plain tensors, and projections as a quantised model directory would give them."""

    def __init__(self, shapes, weights, seed):
        self.shapes, self.weights, self.seed = shapes, weights, seed

    def tensor(self, name):
        return weight(self.seed, name, self.shapes[name])

    def linear(self, parts, role, layer, interleave=False):
        from phaseshift_b200.quant.formats import QuantizedTensor
        ws = [self.tensor(name)[slice(rr.start, rr.stop) if rr is not None else slice(None)] for name, rr, _ in parts]
        fmt = "bf16" if self.weights == "bf16" else block_format(parts[0][0], layer)
        got = [(w, None) if fmt == "bf16" else block_codes(w, fmt) for w in ws]
        k = ws[0].shape[1]

        def join(ts):
            if ts[0] is None or len(ts) == 1:
                return ts[0]
            return torch.stack(ts, 1).reshape(-1, ts[0].shape[1]) if interleave else torch.cat(ts)
        codes, scales = join([c for c, _ in got]), join([s for _, s in got])
        return QuantizedTensor(fmt, (codes.shape[0], k), k, codes.contiguous(), scales, TENSOR_SCALE if fmt == "nvfp4" else 1.0)


# ---------------------------------------------------------------- caches before the step
def cached_rows(c, seed, layer, which, heads, dim):
    """Pool [pages, heads, PAGE, dim] of a layer as it is before the step: values, or (codes, row scales) in 8 bits."""
    n = 1 + sum(map(len, pages_of(c, seed)))
    v = normal(seed, "%s%d" % (which, layer), (n, heads, PAGE, dim))
    if c["kv"] == "bf16":
        return v, None
    v = v.float()
    scale = v.abs().amax(-1) / 448
    return e4m3(v / scale[..., None]), scale


def recurrent_rows(c, seed, layer, shape):
    return normal(seed, "state%d" % layer, shape, 5.0 if c["family"] == "gebuzen" else 0.3, dtype=torch.float32)


def conv_rows(c, seed, layer, channels):
    """The last three inputs of the short convolution: [sequences, 3, channels], the oldest first."""
    return normal(seed, "conv%d" % layer, (len(sequences(c)), 3, channels))


def fill_caches(c, seed, st):
    seqs = sequences(c)
    for i, kv in enumerate(st.kv):
        if kv is not None:
            for pool, scales, which in ((kv.k, kv.k_scale, "k"), (kv.v, kv.v_scale, "v"))[:1 if kv.v is kv.k else 2]:
                pool.zero_()
                v, s = cached_rows(c, seed, i, which, pool.shape[1], pool.shape[3])
                pool[:len(v)].view(v.dtype).copy_(v)
                if s is not None:
                    scales.fill_(1.0)
                    scales[:len(s)].copy_(s)
    for i, g in enumerate(st.gdn):
        if g is None:
            continue
        g.rec.copy_(recurrent_rows(c, seed, i, g.rec.shape))
        for slot, (ctx, _, _) in enumerate(seqs):
            if ctx == 0:
                g.rec[slot].zero_()
        if g.conv is not None:
            h = HYBRID[c["model"]]
            rows = conv_rows(c, seed, i, (2 * h["hk"] + h["hv"]) * 128)
            q, k, v = (t.reshape(len(seqs), 3, -1, 128) for t in torch.split(rows, [h["hk"] * 128, h["hk"] * 128, h["hv"] * 128], 2))
            rep = h["hv"] // h["hk"]
            per_head = torch.cat([q.repeat_interleave(rep, 2), k.repeat_interleave(rep, 2), v], 3)
            for slot, (ctx, _, _) in enumerate(seqs):
                for j in range(3):
                    if ctx - 3 + j >= 0:
                        g.conv[slot, :, (ctx - 3 + j) % g.conv.shape[2]].copy_(per_head[slot, j])


# ---------------------------------------------------------------- the measured calls
def prepare(case, seed):
    from phaseshift_b200.runtime.batch import SeqRows
    from phaseshift_b200.runtime.engine import Engine
    from phaseshift_b200.runtime.state import StateConfig
    c, device = case, torch.device("cuda", torch.cuda.current_device())
    if c["family"] == "gebuzen":
        from phaseshift_b200.models.gebuzen import config, weights
        cfg = getattr(config, "gebuzen_%s_config" % c["model"])()
        cfg.layers = cfg.layers[:c["layers"]]
        shapes = weights.tensor_shapes(cfg)
        w = weights.build_engine_weights(cfg, lambda name: gebuzen_weight(seed, name, shapes[name]), device)
    else:
        from phaseshift_b200.models.qwen35 import config, weights
        more = dict(vocab_size=1024) if c["family"] == "ff" else {}
        cfg = getattr(config, "qwen35_%s_config" % c["model"])(num_hidden_layers=c["layers"], **more)
        w = weights.build_engine_weights(cfg, Checkpoint(weights.hf_tensor_shapes(cfg), c["weights"], seed), c["weights"], device,
                                         layout="both" if c["weights"] != "bf16" else None)
    seqs = sequences(c)
    longest = max(ctx + n for ctx, n, _ in seqs)
    eng = Engine(w, device, StateConfig(max_slots=len(seqs), max_seq_len=longest + 1024, page_tokens=PAGE, kv_dtype=c["kv"],
                                        kv_capacity_tokens=sum(ctx + n + PAGE for ctx, n, _ in seqs)), calibrate=c["family"] != "ff")
    if c["family"] == "ff":
        layer = w.layers[0]
        layer.gate_up.act_scale = layer.down.act_scale = ACT_SCALE
        return dict(case=c, engine=eng, layer=layer, x=normal(seed, "x", (c["prompt"], HIDDEN[c["model"]])))
    eng.apply_block_updates([(slot, block, page) for slot, pages in enumerate(pages_of(c, seed)) for block, page in enumerate(pages)])
    rows = [SeqRows(slot, ctx, ids, output_rows=range(first, n)) for slot, ((ctx, n, first), ids) in enumerate(zip(seqs, token_ids(c, seed)))]
    s = dict(case=c, engine=eng, rows=rows, new=[slot for slot, (ctx, _, _) in enumerate(seqs) if ctx == 0])
    run(s)                                    # an engine in service has seen a step of this size
    fill_caches(c, seed, eng.state)
    return s


def run(state):
    eng = state["engine"]
    if "layer" in state:
        x, layer = state["x"], state["layer"]
        act = eng.ops.linear(x, layer.gate_up, name="act", norm_w=layer.post_norm, eps=EPS, swiglu=True)
        return {"act": act, "out": eng.ops.linear(act, layer.down, name="out", residual=x)}
    for slot in state["new"]:
        eng.state.reset_slot(slot)
    _, out, status = eng.run_rows(state["rows"], want_logits=True)
    if status:
        raise RuntimeError("the step reported status %d" % status)
    pools = [p for kv in eng.state.kv if kv is not None for p in ((kv.k,) if kv.v is kv.k else (kv.k, kv.v))]
    scales = [s for kv in eng.state.kv if kv is not None and kv.k_scale is not None for s in (kv.k_scale, kv.v_scale)]
    return {"logits": out.logits, "states": [g.rec for g in eng.state.gdn if g is not None],
            "pools": [p.view(torch.float8_e4m3fn) if p.dtype == torch.uint8 else p for p in pools], "scales": scales}


# ---------------------------------------------------------------- what a pass cannot do without
def work(case):
    c = case
    H, F = HIDDEN[c["model"]], FF[c["model"]]
    if c["family"] == "ff":
        M = c["prompt"]
        return {"bytes": H * 2 * F * 0.5625 + H * F * 33 / 32 + 2 * M * (2 * H + F), "flops": 2.0 * M * 3 * H * F}
    seqs = sequences(c)
    M = sum(n for _, n, _ in seqs)
    n_out = sum(n - first for _, n, first in seqs)
    byte = 0.5625 if c["weights"] == "nvfp4" else 2
    params = flops = nbytes = 0.0
    for i in range(c["layers"]):
        attention = True
        if c["family"] == "gebuzen":
            g = GEBUZEN[c["model"]]
            hq, hkv, pools = g["hq"], g["hkv"], 1
            params += H * (g["hq"] * 512 + g["hkv"] * 256 + g["h"] * 640 + RANK) + 3 * H * F
            states = g["h"]
        else:
            g = HYBRID[c["model"]]
            hq, hkv, pools, attention = g["hq"], g["hkv"], 2, (i + 1) % 4 == 0
            params += 3 * H * F + (H * (3 * hq + 2 * hkv) * 256 if attention else H * (2 * g["hk"] + 3 * g["hv"]) * 128 + 2 * H * g["hv"])
            states = 0 if attention else g["hv"]
        flops += M * states * 7.0 * 128 * 128
        nbytes += len(seqs) * states * 2 * 4 * 128 * 128
        if attention:
            seen = [(ctx % BLOCK if c["family"] == "gebuzen" else ctx, n) for ctx, n, _ in seqs]
            flops += sum(4.0 * hq * 256 * (n * ctx + n * (n + 1) / 2) for ctx, n in seen)
            nbytes += sum(pools * hkv * 256 * (ctx + n) for ctx, n in seen) * (1 if c["kv"] == "fp8_e4m3" else 2)
    head = H * VOCAB * (33 / 32 if c["weights"] == "nvfp4" else 2)
    return {"bytes": params * byte + head + nbytes + n_out * VOCAB * 4 + M * H * 2, "flops": flops + 2.0 * params * M + 2.0 * H * VOCAB * n_out}


def tolerance(case):
    # measured against 64 bits: 0.4 to 1.3 % after several layers of bf16 activations (codes of 8-bit rows: up to 2.5 %); two such
    # results differ by up to twice that
    return {"rel": 0.03, "max": 0.5, "differ": 0.0}


# ---------------------------------------------------------------- the same in 64 bits
def exact(case, seed):
    c = case
    with torch.no_grad():
        if c["family"] == "ff":
            return exact_ff(c, seed)
        return Exact(c, seed).gebuzen() if c["family"] == "gebuzen" else Exact(c, seed).hybrid()


def silu(x):
    return x * torch.sigmoid(x)


def rms(x):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + EPS)


def quantised_rows(x, fmt):
    """Activations as the block-scaled products take them; the 4-bit format has one fixed scale above its block scales."""
    v = x.float()
    if fmt == "nvfp4":
        b = v.reshape(len(v), -1, 16)
        s = e4m3(b.abs().amax(-1) / (6 * ACT_SCALE)).double() * ACT_SCALE
        q = e2m1_value(e2m1(torch.where(s > 0, 1 / s, 0)[..., None] * b)) * s[..., None]
    else:
        b = v.reshape(len(v), -1, 32)
        s = torch.ldexp(torch.ones_like(b[..., 0]), mx_exponent(b.abs().amax(-1)))[..., None]
        q = e4m3(b / s).double() * s
    return q.reshape(len(v), -1)


def exact_ff(c, seed):
    H, F = HIDDEN[c["model"]], FF[c["model"]]
    x = normal(seed, "x", (c["prompt"], H)).double()
    pre = "model.language_model.layers.0."
    w = {n: block_values(*block_codes(weight(seed, pre + "mlp.%s_proj.weight" % n, s), f), f)
         for n, s, f in (("gate", (F, H), "nvfp4"), ("up", (F, H), "nvfp4"), ("down", (H, F), "mxfp8"))}
    norm = weight(seed, pre + "post_attention_layernorm.weight", (H,)).double()
    h = quantised_rows((x.float() * (1 + norm.float())), "nvfp4")
    r = torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + EPS)
    act = silu(h @ w["gate"].T * r) * (h @ w["up"].T * r)
    return {"act": act, "out": quantised_rows(act.bfloat16(), "mxfp8") @ w["down"].T + x}


class Exact:
    def __init__(self, c, seed):
        self.c, self.seed, self.seqs, self.pages = c, seed, sequences(c), pages_of(c, seed)
        self.H, self.F = HIDDEN[c["model"]], FF[c["model"]]
        self.ids = torch.tensor(sum(token_ids(c, seed), []), device="cuda")
        self.states, self.pools, self.scales = [], [], []

    def each(self):
        """(sequence, cached tokens, its rows of the step)."""
        at = 0
        for i, (ctx, n, _) in enumerate(self.seqs):
            yield i, ctx, slice(at, at + n)
            at += n

    def w(self, name, *shape, layer=0):
        """A projection's weights as the checkpoint's format holds them."""
        if self.c["family"] == "gebuzen":
            return gebuzen_weight(self.seed, name, shape).double()
        t = weight(self.seed, "model.language_model." + name, shape)
        fmt = block_format(name, layer)
        if self.c["weights"] == "bf16" or fmt == "bf16" or len(shape) != 2:
            return t.double()
        return block_values(*block_codes(t, fmt), fmt)

    def head(self, h, name):
        rows = [s.start + j for (i, _, s), (_, n, first) in zip(self.each(), self.seqs) for j in range(first, n)]
        return {"logits": h[rows] @ self.w(name, VOCAB, self.H).T, "states": self.states, "pools": self.pools, "scales": self.scales}

    def pool(self, layer, which, heads, new):
        """Append the step's rows [rows, heads, 256]; what each sequence then sees: [tokens, heads, 256] for every sequence."""
        pool, scale = cached_rows(self.c, self.seed, layer, which, heads, 256)
        pool = pool.double()
        new = new.bfloat16().double()
        if scale is not None:
            scale = scale.double()
            s = new.abs().amax(-1) / 448
            new = e4m3((new / s[..., None]).float()).double()
        out = []
        for i, ctx, rows in self.each():
            pos = torch.arange(ctx, ctx + rows.stop - rows.start, device="cuda")
            page = torch.tensor(self.pages[i], device="cuda")
            pool[page[pos // PAGE], :, pos % PAGE] = new[rows]
            if scale is not None:
                scale[page[pos // PAGE], :, pos % PAGE] = s[rows]
            seen = pool[page] * scale[page][..., None] if scale is not None else pool[page]
            out.append(seen.transpose(1, 2).reshape(-1, heads, 256)[:ctx + len(pos)])
        # pools and scales are compared over the pages that the sequences hold; the engine's have some to spare
        spare = -(-sum(ctx + n + PAGE for ctx, n, _ in self.seqs) // PAGE) + 1 + len(self.seqs) - len(pool)
        self.pools.append(torch.cat([pool, pool.new_zeros(spare, *pool.shape[1:])]))
        if scale is not None:
            self.scales.append(torch.cat([scale, scale.new_ones(spare, *scale.shape[1:])]))
        return out

    def attend(self, q, ks, vs, block=0, sink=None):
        """q [rows, heads, 256]; causal, inside blocks of `block` positions where one is given."""
        out = torch.empty_like(q)
        rep = q.shape[1] // ks[0].shape[1]
        for i, ctx, rows in self.each():
            n = rows.stop - rows.start
            pos, at = torch.arange(ctx, ctx + n, device="cuda"), torch.arange(ctx + n, device="cuda")
            hidden = at[None] > pos[:, None]
            if block:
                hidden |= at[None] // block != pos[:, None] // block
            for h in range(q.shape[1]):
                s = (q[rows, h] @ ks[i][:, h // rep].T / 16).masked_fill(hidden, -math.inf)
                if sink is not None:
                    s = torch.cat([s, sink[h].expand(n, 1)], 1)
                out[rows, h] = torch.softmax(s, 1)[:, :ctx + n] @ vs[i][:, h // rep]
        return out

    # ---- the hybrid decoder
    def hybrid(self):
        c, H, F = self.c, self.H, self.F
        x = weight(self.seed, "model.language_model.embed_tokens.weight", (VOCAB, H))
        if c["weights"] != "bf16":
            codes, scales = block_codes(x, "mxfp8")
            x = block_values(codes[self.ids], scales[self.ids], "mxfp8")
        else:
            x = x[self.ids].double()
        for i in range(c["layers"]):
            p = "layers.%d." % i
            n = rms(x) * (1 + self.w(p + "input_layernorm.weight", H))
            x = x + (self.attention(i, p + "self_attn.", n) if (i + 1) % 4 == 0 else self.delta(i, p + "linear_attn.", n))
            n = rms(x) * (1 + self.w(p + "post_attention_layernorm.weight", H))
            p += "mlp."
            y = silu(n @ self.w(p + "gate_proj.weight", F, H, layer=i).T) * (n @ self.w(p + "up_proj.weight", F, H, layer=i).T)
            x = x + y @ self.w(p + "down_proj.weight", H, F, layer=i).T
        return self.head(rms(x) * (1 + self.w("norm.weight", H)), "lm_head.weight")

    def attention(self, i, p, n):
        h = HYBRID[self.c["model"]]
        q, gate = (n @ self.w(p + "q_proj.weight", h["hq"] * 512, self.H, layer=i).T).reshape(len(n), -1, 512).split(256, 2)
        k, v = ((n @ self.w(p + s + "_proj.weight", h["hkv"] * 256, self.H, layer=i).T).reshape(len(n), -1, 256) for s in "kv")
        pos = torch.cat([torch.arange(ctx, ctx + r.stop - r.start) for _, ctx, r in self.each()]).to("cuda")
        turn = pos[:, None, None] * 1e7 ** (-torch.arange(32, dtype=torch.float64, device="cuda") / 32)

        def turned(t, name):
            t = rms(t) * (1 + self.w(p + name, 256))
            a, b, rest = t[..., :32], t[..., 32:64], t[..., 64:]
            return torch.cat([a * turn.cos() - b * turn.sin(), b * turn.cos() + a * turn.sin(), rest], -1)
        ks = self.pool(i, "k", h["hkv"], turned(k, "k_norm.weight"))
        vs = self.pool(i, "v", h["hkv"], v)
        o = self.attend(turned(q, "q_norm.weight"), ks, vs) * torch.sigmoid(gate)
        return o.reshape(len(n), -1) @ self.w(p + "o_proj.weight", self.H, h["hq"] * 256, layer=i).T

    def delta(self, i, p, n):
        h = HYBRID[self.c["model"]]
        hk, hv, H = h["hk"], h["hv"], self.H
        channels = (2 * hk + hv) * 128
        qkv = n @ self.w(p + "in_proj_qkv.weight", channels, H, layer=i).T
        z = n @ self.w(p + "in_proj_z.weight", hv * 128, H, layer=i).T
        beta = torch.sigmoid(n @ self.w(p + "in_proj_b.weight", hv, H).T)
        a = n @ self.w(p + "in_proj_a.weight", hv, H).T + self.w(p + "dt_bias", hv)
        decay = torch.exp(-torch.exp(self.w(p + "A_log", hv)) * torch.nn.functional.softplus(a))
        taps = self.w(p + "conv1d.weight", channels, 1, 4)[:, 0]
        before = conv_rows(self.c, self.seed, i, channels).double()
        S = recurrent_rows(self.c, self.seed, i, (len(self.seqs), hv, 128, 128)).double()
        o = torch.empty(len(n), hv, 128, dtype=torch.float64, device="cuda")
        for s, ctx, r in self.each():
            m = r.stop - r.start
            past = before[s] * (torch.arange(3, device="cuda") >= 3 - ctx)[:, None]
            if ctx == 0:
                S[s] = 0
            t = torch.cat([past, qkv[r]])
            t = silu(sum(t[j:j + m] * taps[:, j] for j in range(4)))
            q, k, v = (u.reshape(m, -1, 128) for u in t.split([hk * 128, hk * 128, hv * 128], 1))
            q, k = ((u * torch.rsqrt(u.pow(2).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(hv // hk, 1) for u in (q, k))
            state = S[s]
            for j in range(m):
                state = state * decay[r][j][:, None, None]
                d = (v[j] - (k[j][:, None] @ state)[:, 0]) * beta[r][j][:, None]
                state = torch.baddbmm(state, k[j][:, :, None], d[:, None])
                o[r.start + j] = (q[j][:, None] @ state)[:, 0]
            S[s] = state
        self.states.append(S)
        o = rms(o * 128 ** -0.5) * self.w(p + "norm.weight", 128) * silu(z.reshape(len(n), hv, 128))
        return o.reshape(len(n), -1) @ self.w(p + "out_proj.weight", H, hv * 128, layer=i).T

    # ---- attention and gated linear attention side by side
    def gebuzen(self):
        H, F, g = self.H, self.F, GEBUZEN[self.c["model"]]
        x = gebuzen_weight(self.seed, "embed", (VOCAB, H))[self.ids].double()
        for i in range(self.c["layers"]):
            p = "l%d.mix." % i
            n = rms(x) * self.w("l%d.norm1" % i, H)
            q, k = ((n @ self.w(p + "left." + s, h * 256, H).T + self.w(p + "left." + s + ".b", h * 256)).reshape(len(n), -1, 256)
                    for s, h in (("q", g["hq"]), ("k", g["hkv"])))
            ks = self.pool(i, "k", g["hkv"], k)
            a = self.attend(q, ks, ks, BLOCK, self.w(p + "left.sink", g["hq"])).reshape(len(n), -1) @ self.w(p + "left.o", H, g["hq"] * 256).T
            b = self.linear_attention(i, p + "right.", n, g["h"])
            x = x + 0.25 * (rms(a) * self.w(p + "left.out", H) + rms(b) * self.w(p + "right.out", H))
            n = rms(x) * self.w("l%d.norm2" % i, H)
            p = "l%d.mlp." % i
            x = x + 0.5 * ((torch.relu(n @ self.w(p + "gate", F, H).T) * (n @ self.w(p + "up", F, H).T)) @ self.w(p + "down", H, F).T)
        return self.head(rms(x) * self.w("final.norm", H), "head")

    def linear_attention(self, i, p, n, heads):
        H = self.H
        q, k, v, gate = ((n @ self.w(p + s, heads * 128, H).T).reshape(len(n), heads, 128) for s in "qkvg")
        z = (n @ self.w(p + "a1", RANK, H).T) @ self.w(p + "a2", heads * 128, RANK).T + self.w(p + "a2.b", heads * 128)
        decay = (torch.sigmoid(z) ** (1 / TAU)).reshape(len(n), heads, 128)
        S = recurrent_rows(self.c, self.seed, i, (len(self.seqs), heads, 128, 128)).double()
        o = torch.empty_like(v)
        for s, ctx, r in self.each():
            state = S[s] if ctx else torch.zeros_like(S[s])
            for j in range(r.start, r.stop):
                state = torch.baddbmm(state * decay[j][:, :, None], k[j][:, :, None], v[j][:, None])
                o[j] = (q[j][:, None] @ state)[:, 0]
            S[s] = state
        self.states.append(S)
        o = rms(o * 128 ** -0.5) * self.w(p + "norm", 128) * silu(gate)
        return o.reshape(len(n), -1) @ self.w(p + "o", H, heads * 128).T
