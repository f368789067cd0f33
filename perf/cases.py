"""Performance cases: the work a user of the engine has it do, at the served model's own layer shapes.

A pass goes through the public entry points (``Engine.prefill`` / ``decode`` / ``draft_batch`` / ``verify_batch`` /
``accept_batch``, ``VisionEncoder.encode``, the tensor-level wrappers of ``ops.kernels``).  Engine cases hold a slice of
the model: a text of layer letters (``g`` = gated delta net, ``q`` = sparse attention; every layer also has its expert
block and two hyper-connection mixers) with the full widths, 512 experts, the whole vocabulary and random-init weights.
``exact`` is the same mathematics in plain 64-bit torch.
"""
import math

import torch
import torch.nn.functional as F

from qwb200.engine.engine import Engine, EngineOptions
from qwb200.engine.state_io import StateIO
from qwb200.engine.weights_prep import prep_moe
from qwb200.models.config import ModelConfig, ShardConfig
from qwb200.models.ngram import NgramHasher
from qwb200.models.ple import PleTable
from qwb200.models.weights import synth_experts, synth_globals, synth_layer
from qwb200.ops import kernels as K
from qwb200.vision.encoder import VisionConfig, VisionEncoder, synth_vision_weights

DEV = "cuda:0"
FULL = ModelConfig.full()
PLE_ROWS = 1 << 16
STEPS = 4                     # tokens generated per stream in a pass of a decode case

# rows of a layer's projection weight matrices (N, K): attention and linear-attention projections, their output
# projections, router + shared expert, PLE key / value, vision MLP
DENSE = {"gdn_proj": (16480, 2560), "qsa_proj": (13952, 2560), "out": (2560, 6144), "router": (1793, 2560),
         "shared_down": (2560, 640), "ple": (12800, 2560), "mixer_down": (324, 10240), "mixer_up": (10240, 320),
         "vit_qkv": (3456, 1152), "vit_fc1": (4304, 1152), "vit_fc2": (1152, 4304)}


def listed():
    return [
        # one user chatting: batch-1 decode behind a 4k context, token by token (two of the model's twelve 4-layer groups)
        {"name": "decode-1", "kind": "decode", "layers": "gggqgggq", "streams": 1, "context": 4096},
        # eight users at once, one row each
        {"name": "decode-8", "kind": "decode", "layers": "gggq", "streams": 8, "context": 1021},
        # speculative decoding, one stream: five drafts and the pending token in one verification step, part accepted
        {"name": "verify-1x6", "kind": "verify", "layers": "gggq", "streams": 1, "run": 6, "context": 4096},
        # four streams of the same
        {"name": "verify-4x6", "kind": "verify", "layers": "gggq", "streams": 4, "run": 6, "context": 2300},
        # the draft side of it: one pass of the MTP head over the streams
        {"name": "draft-4", "kind": "draft", "layers": "g", "streams": 4, "context": 1500},
        # the tail of a follow-up turn: a short prompt through the token-major path
        {"name": "prefill-100", "kind": "prefill", "layers": "gggq", "tokens": 100, "base": 0},
        # an ordinary prompt of odd length
        {"name": "prefill-1021", "kind": "prefill", "layers": "gggq", "tokens": 1021, "base": 0},
        # one full chunk of a long prompt
        {"name": "prefill-4096", "kind": "prefill", "layers": "gggq", "tokens": 4096, "base": 0},
        # a chunk deep inside a long prompt: two attention layers behind 16k tokens
        {"name": "attention-deep", "kind": "prefill", "layers": "qq", "tokens": 2048, "base": 16384},
        # an uploaded 720p picture through the vision tower
        {"name": "vision-720p", "kind": "vision", "h": 44, "w": 80},
        # the routed and shared experts of one layer for the rows of a speculative step
        {"name": "experts-6", "kind": "experts", "rows": 6},
        # one linear-attention projection of an ordinary prompt
        {"name": "dense-777", "kind": "dense", "which": "gdn_proj", "tokens": 777},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["decode", "verify", "draft", "prefill", "prefill", "vision", "experts", "dense"])
    if kind == "decode":
        return {"kind": kind, "layers": rng.choice(["gg", "qq", "gggq"]), "streams": _log(rng, 1, 16), "context": _log(rng, 70, 3000)}
    if kind == "verify":
        return {"kind": kind, "layers": rng.choice(["gg", "qq", "gggq"]), "streams": rng.randint(1, 4), "run": rng.randint(2, 6),
                "context": _log(rng, 70, 5000)}
    if kind == "draft":
        return {"kind": kind, "layers": "g", "streams": rng.randint(1, 8), "context": _log(rng, 70, 3000)}
    if kind == "prefill":
        tokens = _log(rng, 64, 3500)
        return {"kind": kind, "layers": rng.choice(["gg", "qq", "gggq"]), "tokens": tokens, "base": rng.choice([0, 0, _log(rng, 70, 4000)])}
    if kind == "vision":
        return {"kind": kind, "h": 2 * rng.randint(4, 22), "w": 2 * rng.randint(4, 40)}
    if kind == "experts":
        return {"kind": kind, "rows": _log(rng, 1, 32)}
    return {"kind": "dense", "which": rng.choice(sorted(DENSE)), "tokens": _log(rng, 16, 4096)}


# ---------------------------------------------------------------------------------------------------- preparation
def _config(case):
    types = tuple("qsa" if c == "q" else "gdn" for c in case["layers"])
    return ModelConfig(n_layers=len(types), layer_types=types, mtp=case["kind"] == "draft")


def _tokens(cfg, seed, n):
    g = torch.Generator().manual_seed(1000 + seed)
    return torch.randint(0, cfg.vocab, (n,), generator=g).tolist()


def _streams(case, cfg, seed):
    """Per stream: the context, and the tokens the pass feeds behind it."""
    feed = {"decode": STEPS, "verify": case.get("run", 0), "draft": 1, "prefill": case.get("tokens", 0)}[case["kind"]]
    out = []
    for s in range(case.get("streams", 1)):
        base = case["context"] if "context" in case else case["base"]
        t = _tokens(cfg, seed * 64 + s, base + feed)
        out.append((t[:base], t[base:]))
    return out


def _accepted(case):
    """Rows of each stream's run that a verification case keeps: all, some or one, as it falls."""
    return [1 + (s * 2 + 2) % case["run"] for s in range(case["streams"])]


def _dense_inputs(case, seed):
    n, k = DENSE[case["which"]]
    g = torch.Generator(device=DEV).manual_seed(seed)
    x = torch.randn(case["tokens"], k, generator=g, device=DEV).to(torch.bfloat16)
    w = (torch.randn(n, k, generator=g, device=DEV) * 0.02).to(torch.bfloat16)
    return x, w


def _expert_inputs(case, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    w = synth_experts(FULL, g, 0.02, DEV, False, "")
    w["down"] = (torch.randn(FULL.hidden, FULL.ffn, generator=g, device=DEV) * 0.02).to(torch.bfloat16)
    w["rs"] = (torch.randn(FULL.n_experts + 1 + 2 * FULL.ffn, FULL.hidden, generator=g, device=DEV) * 0.02).to(torch.bfloat16)
    x = torch.randn(case["rows"], FULL.hidden, generator=g, device=DEV).to(torch.bfloat16)
    return w, x


def _vision_inputs(case, seed):
    """The tower's weights (the names and shapes of a one-block synthetic tower, repeated) and the patches of a picture."""
    cfg = VisionConfig()
    shapes = {n: t.shape for n, t in synth_vision_weights(VisionConfig(depth=1), 0).items()}
    g = torch.Generator(device=DEV).manual_seed(seed)
    w = {}
    for name, shape in shapes.items():
        for b in range(cfg.depth) if ".blocks." in name else [0]:
            r = torch.randn(shape, generator=g, device=DEV)
            if name.endswith("bias"):
                r = r * 0.05
            elif "norm" in name:
                r = 1.0 + r * 0.05
            else:
                r = r * (0.1 if "pos_embed" in name else 1.0 / math.sqrt(r[0].numel()))
            w[name.replace(".blocks.0.", f".blocks.{b}.")] = r.to(torch.bfloat16)
    patches = (torch.rand(case["h"] * case["w"], cfg.patch_in, generator=g, device=DEV) * 2 - 1)
    return cfg, w, patches


def prepare(case, seed):
    kind = case["kind"]
    if kind == "dense":
        x, w = _dense_inputs(case, seed)
        n = w.shape[0]                                  # rows of the result lie 16-byte aligned, as in the engine's buffers
        out = torch.empty(x.shape[0], (n + 7) // 8 * 8, device=DEV)[:, :n]
        return {"kind": kind, "x": x, "w": w, "out": out}
    if kind == "experts":
        w, x = _expert_inputs(case, seed)
        c, E = FULL, FULL.n_experts
        named = {"gate.weight": w["rs"][:E], "shared_expert_gate.weight": w["rs"][E:E + 1],
                 "shared_expert.gate_proj.weight": w["rs"][E + 1:E + 1 + c.ffn], "shared_expert.up_proj.weight": w["rs"][E + 1 + c.ffn:],
                 "shared_expert.down_proj.weight": w["down"], **{n: t for n, t in w.items() if n.startswith("experts.")}}
        return {"kind": kind, "x": x, "w": prep_moe(named, "", ShardConfig(c, 1, 0), DEV)}
    if kind == "vision":
        cfg, w, patches = _vision_inputs(case, seed)
        return {"kind": kind, "tower": VisionEncoder(cfg, w, DEV), "patches": patches, "h": case["h"], "w": case["w"]}
    cfg = _config(case)
    streams = _streams(case, cfg, seed)
    longest = max(len(a) + len(b) for a, b in streams)
    eng = Engine.synthetic(cfg, EngineOptions(slots=len(streams), slot_tokens=longest + 8, use_graphs=True, save_gdn=kind == "verify"),
                           device=DEV, seed=seed, ple_rows=PLE_ROWS)
    io = StateIO(eng.dm)
    for s, (context, _) in enumerate(streams):
        eng.reset(s)
        if context:
            eng.prefill(s, context, want_logits=False)
    return {"kind": kind, "engine": eng, "io": io, "streams": streams, "accept": _accepted(case) if kind == "verify" else None,
            "snapshots": [io.snapshot_save(s) for s in range(len(streams))], "run": case.get("run", 0)}


# ---------------------------------------------------------------------------------------------------- one pass
def _rewind(st):
    """Every slot back to the end of its context, as a session does before a regenerated answer."""
    for s, (context, _) in enumerate(st["streams"]):
        st["io"].snapshot_restore(s, st["snapshots"][s])
        del st["engine"].slot[s].tokens[len(context):]


def _state(st, fed):
    """The slots' state behind a pass: delta-net states, and the key / value rows of the fed tokens of every attention layer."""
    dm, out = st["engine"].dm, {}
    for i, t in enumerate(dm.gdn_S):
        out[f"delta{i}"] = t
    for i in range(dm.cfg.n_qsa):
        for name, pages in (("k", dm.k_dev[i]), ("v", dm.v_dev[i])):
            rows = pages.view(len(st["streams"]), dm.slot_tokens, -1)
            base = len(st["streams"][0][0])
            out[f"{name}{i}"] = rows[:, base:base + fed]
    return out


def run(st):
    kind = st["kind"]
    if kind == "dense":
        return K.gemm_bf16_tc(st["x"], st["w"], out=st["out"])
    if kind == "experts":
        w, c = st["w"], FULL
        rs = K.gemv_bf16(w["Wrs"], st["x"])
        pair_expert, pair_w, shared = K.moe_route(rs, c.n_experts, c.top_k, c.ffn)
        return K.moe_experts_pair(w["w13"], w["s13"], w["w2"], w["s2"], st["x"], pair_expert, pair_w, c.ffn, c.hidden, w["Wsd"], shared)
    if kind == "vision":
        return st["tower"].encode(st["patches"], st["h"], st["w"])
    eng, streams = st["engine"], st["streams"]
    slots = list(range(len(streams)))
    logits = eng.dm.buf["logits"]
    if kind == "draft":
        eng.draft_batch(slots, [feed[0] for _, feed in streams], 1)
        return {"logits": logits[:len(slots)], "hidden": eng.dm.buf["hidden_out"][:len(slots)]}
    _rewind(st)
    if kind == "prefill":
        out = eng.prefill(0, streams[0][1])
        return {"logits": out, **_state(st, len(streams[0][1]))}
    if kind == "decode":
        rows = []
        for j in range(STEPS):
            eng.decode(slots, [feed[j] for _, feed in streams])
            rows.append(logits[:len(slots)].clone())
        return {"logits": torch.stack(rows), **_state(st, STEPS)}
    runs = [feed for _, feed in streams]
    n = eng.verify_batch(slots, runs)
    eng.accept_batch(slots, runs, st["accept"])
    return {"logits": logits[:n], **_state(st, st["run"])}


# ---------------------------------------------------------------------------------------------------- what a pass needs
def _layer_dense(q):
    """Dense weights of a layer (attention part, two mixers, router, shared expert), in values."""
    n = DENSE["qsa_proj" if q else "gdn_proj"]
    mats = [n, DENSE["out"], DENSE["router"], DENSE["shared_down"]] + 2 * [DENSE["mixer_down"], DENSE["mixer_up"]]
    return sum(a * b for a, b in mats)


EXPERT = 3 * 640 * 2560                                 # values of one routed expert
EXPERT_BYTES = EXPERT / 2 + EXPERT / 128 * 2


def _distinct(rows):
    """Experts of a layer that `rows` rows of ten choices each touch, on average."""
    return 512 * (1 - (1 - 10 / 512) ** rows)


def work(case):
    kind = case["kind"]
    if kind == "dense":
        (n, k), t = DENSE[case["which"]], case["tokens"]
        return {"bytes": 2 * (n * k + t * k) + 4 * t * n, "flops": 2 * t * n * k}
    if kind == "experts":
        r = case["rows"]
        dense = 1793 * 2560 + 2560 * 640
        return {"bytes": _distinct(r) * EXPERT_BYTES + 2 * dense + r * 2560 * 6, "flops": 2 * r * (10 * EXPERT + dense)}
    if kind == "vision":
        c, L = VisionConfig(), case["h"] * case["w"]
        block = 4 * c.dim * c.dim + 2 * c.dim * c.mlp
        weights = c.depth * block + c.patch_in * c.dim + 16 * c.dim * c.dim + 4 * c.dim * c.out_dim
        flops = 2 * L * (c.depth * block + c.patch_in * c.dim + 4 * c.dim * c.dim + c.dim * c.out_dim) + c.depth * 4 * L * L * c.dim
        return {"bytes": 2 * weights + 4 * L * c.patch_in + L * c.out_dim, "flops": flops}
    streams = case.get("streams", 1)
    fed = {"decode": STEPS, "verify": case.get("run", 0), "draft": 1, "prefill": case.get("tokens", 0)}[kind]
    base = case["context"] if "context" in case else case["base"]
    steps = STEPS if kind == "decode" else 1
    rows = streams * fed // steps                       # rows of a step
    head = rows if kind != "prefill" else 1
    total = {"bytes": 0.0, "flops": 0.0}
    layers = "q" if kind == "draft" else case["layers"]
    for i, c in enumerate(layers):
        dense = _layer_dense(c == "q") + (2 * 2560 * 2560 if kind == "draft" else 0) + (12800 * 2560 if i == 1 else 0)
        seen = sum(min(base + j + 1, 2048 + 3) for j in range(0, fed, max(1, fed // 64))) / len(range(0, fed, max(1, fed // 64)))
        if c == "q":
            once = min(base + fed, seen * fed)          # key / value rows: each read once where rows share them
            mem = streams * (once * 2 * 512 * 2 + (base + fed) / 4 * 256 if base + fed > 2048 else once * 2048)
            mul = rows * (4 * seen * 24 * 256 + (2 * (base + fed) / 4 * 512 if base + fed > 2048 else 0))
        else:
            mem = streams * 2 * 48 * 128 * 128 * 4
            mul = rows * 48 * 128 * 128 * 6
        total["bytes"] += steps * (2 * dense + _distinct(rows) * EXPERT_BYTES + mem)
        total["flops"] += steps * (2 * rows * (dense + 10 * EXPERT) + mul)
    mixer = 320 * 10240 * 2
    total["bytes"] += steps * (2 * (248320 * 2560 + mixer) + head * 248320 * 4)
    total["flops"] += steps * 2 * head * (248320 * 2560 + mixer)
    return total


def tolerance(case):
    kind = case["kind"]
    # each about four times what another order of the sums, or the 64-bit reference, was seen to differ by
    if kind == "dense":
        return {"rel": 2e-5, "max": 1e-3}               # bf16 inputs, fp32 sums and outputs
    if kind == "experts":
        return {"rel": 1e-4, "max": 2e-3}               # the same, with a rounding of the hidden values to bf16
    if kind == "vision":
        return {"rel": 2e-2, "max": 0.3}                # bf16 activations through 27 blocks
    return {"rel": 3e-2, "max": 0.9}                    # bf16 activations, and experts and tokens chosen by them


# ---------------------------------------------------------------------------------------------------- 64-bit reference
def _rms(x, eps):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps)


def _rope(c, x, pos):
    half = c.rope_dim // 2
    inv = c.rope_theta ** (-2.0 * torch.arange(half, dtype=torch.float64, device=x.device) / c.rope_dim)
    a = (pos.double()[:, None] * inv).view([len(pos)] + [1] * (x.dim() - 2) + [half])
    x1, x2 = x[..., :half], x[..., half:2 * half]
    return torch.cat([x1 * a.cos() - x2 * a.sin(), x2 * a.cos() + x1 * a.sin(), x[..., 2 * half:]], -1)


def _q4(packed, scale):
    """Values of int4 words (element i of a word in bits 4i..4i+3, stored + 8), one scale per 128 columns."""
    nib = (packed.unsqueeze(-1) >> (4 * torch.arange(8, device=packed.device, dtype=torch.int32))) & 15
    v = (nib - 8).double().reshape(packed.shape[0], -1, 128)
    return (v * scale.double().unsqueeze(-1)).reshape(packed.shape[0], -1)


class _Exact:
    """One sequence through the sliced model in 64 bits; keeps what the outputs need of the layers' states."""

    def __init__(self, cfg, w, table):
        self.c, self.w, self.table = cfg, w, table
        self.delta, self.keys, self.values = [], [], []

    def W(self, name):
        return self.w[name].double()

    def mix(self, p, X, inject=True):
        c = self.c
        xn = (_rms(X.view(-1, c.hc, c.hidden), c.eps) * (1 + self.W(p + "hc_norm.weight").view(c.hc, c.hidden))).reshape(-1, c.hch)
        u = F.silu(xn @ self.W(p + "input_mix_weight_down.weight").T / c.hc)
        gate = torch.sigmoid(u @ self.W(p + "input_mix_weight_up.weight").T)
        y = (gate * xn).view(-1, c.hc, c.hidden).mean(1)
        return (y, xn @ self.W(p + "block_inject_weight.weight").T) if inject else y

    def add(self, X, out, inj):
        return X + ((2 * torch.sigmoid(inj / self.c.hc)).unsqueeze(-1) * out.unsqueeze(1)).reshape(X.shape)

    def ple(self, X, tokens):
        c, p = self.c, f"layers.{self.c.ple_layer}.ple."
        ids = torch.from_numpy(NgramHasher(c).ids_for([], tokens)) % self.table.shape[0]
        e = self.table[ids.to(self.table.device)].view(torch.float8_e4m3fn).float().double().reshape(len(tokens), -1) * 0.25
        shape = (c.hc, c.hidden)
        key = _rms((e @ self.W(p + "key_proj.weight").T).view(-1, *shape), c.eps) * (1 + self.W(p + "norm_key.weight").view(shape))
        query = _rms(X.view(-1, *shape), c.eps) * (1 + self.W(p + "norm_query.weight").view(shape))
        s = (key * query).sum(-1) / math.sqrt(c.hidden)
        gate = torch.sigmoid(torch.sign(s) * s.abs().clamp_min(1e-6).sqrt())
        gv = gate.unsqueeze(-1) * (e @ self.W(p + "value_proj.weight").T).unsqueeze(1)
        nc = (_rms(gv, c.eps) * (1 + self.W(p + "norm_conv.weight").view(shape))).reshape(-1, c.hch)
        back = (c.ple_conv - 1) * c.ple_dilation
        seq = torch.cat([nc.new_zeros(back, c.hch), nc])
        cw = self.W(p + "conv1d.weight").view(c.hch, c.ple_conv)
        conv = sum(cw[:, i] * seq[i * c.ple_dilation:i * c.ple_dilation + len(tokens)] for i in range(c.ple_conv))
        return X + gv.reshape(-1, c.hch) + F.silu(conv)

    def gdn(self, p, x, keep):
        c, T = self.c, x.shape[0]
        pre = x @ self.W(p + "in_proj_qkv.weight").T
        seq = torch.cat([pre.new_zeros(c.gdn_conv - 1, c.gdn_qkv), pre])
        cw = self.W(p + "conv1d.weight").view(c.gdn_qkv, c.gdn_conv)
        qkv = F.silu(sum(cw[:, i] * seq[i:i + T] for i in range(c.gdn_conv)))
        q, k, v = (t.view(T, -1, c.gdn_dim) for t in qkv.split([c.gdn_key, c.gdn_key, c.gdn_val], 1))
        q = q * torch.rsqrt(q.pow(2).sum(-1, keepdim=True) + c.eps) / math.sqrt(c.gdn_dim)
        k = k * torch.rsqrt(k.pow(2).sum(-1, keepdim=True) + c.eps)
        rep = c.gdn_v_heads // c.gdn_qk_heads
        q, k = q.repeat_interleave(rep, 1), k.repeat_interleave(rep, 1)
        a = x @ self.W(p + "in_proj_a.weight").T + self.W(p + "dt_bias")
        decay = torch.exp(-torch.exp(self.W(p + "A_log")) * F.softplus(a))[:, :, None, None]
        beta = torch.sigmoid(x @ self.W(p + "in_proj_b.weight").T)[:, :, None]
        S = x.new_zeros(c.gdn_v_heads, c.gdn_dim, c.gdn_dim)
        o = torch.empty_like(v)
        for t in range(T):
            S = S * decay[t]
            d = (v[t] - torch.bmm(k[t].unsqueeze(1), S).squeeze(1)) * beta[t]
            S = torch.baddbmm(S, k[t].unsqueeze(2), d.unsqueeze(1))
            o[t] = torch.bmm(q[t].unsqueeze(1), S).squeeze(1)
            if t == keep:
                self.delta.append(S.clone())
        z = torch.sigmoid(x @ self.W(p + "in_proj_z.weight").T)
        return ((_rms(o, c.eps) * self.W(p + "norm.weight")).reshape(T, -1) * z) @ self.W(p + "out_proj.weight").T

    def qsa(self, p, x):
        c, T, D = self.c, x.shape[0], self.c.head_dim
        pos = torch.arange(T, device=x.device)
        qg = (x @ self.W(p + "q_proj.weight").T).view(T, c.q_heads, 2, D)
        q = _rope(c, _rms(qg[:, :, 0], c.eps) * (1 + self.W(p + "q_norm.weight")), pos)
        k = (x @ self.W(p + "k_proj.weight").T).view(T, c.kv_heads, D)
        k = _rope(c, _rms(k, c.eps) * (1 + self.W(p + "k_norm.weight")), pos)
        v = (x @ self.W(p + "v_proj.weight").T).view(T, c.kv_heads, D)
        self.keys.append(k.reshape(T, -1))
        self.values.append(v.reshape(T, -1))
        iqk = x @ self.W(p + "indexer.index_qk_proj.weight").T
        iq = iqk[:, :c.idx_heads * c.idx_dim].view(T, c.idx_heads, c.idx_dim)
        iq = _rope(c, _rms(iq, c.eps) * (1 + self.W(p + "indexer.q_layernorm.weight")), pos)
        r, ng = c.idx_ratio, T // c.idx_ratio
        raw = iqk[:ng * r, c.idx_heads * c.idx_dim:].view(ng, r, c.idx_dim).mean(1)
        ck = _rope(c, _rms(raw, c.eps) * (1 + self.W(p + "indexer.k_layernorm.weight")), pos[:ng * r:r])
        rep = c.q_heads // c.kv_heads
        kh, vh = k.permute(1, 2, 0).repeat_interleave(rep, 0), v.permute(1, 0, 2).repeat_interleave(rep, 0)
        out = torch.empty(T, c.q_heads * D, dtype=x.dtype, device=x.device)
        for a in range(0, T, 256):
            b = min(T, a + 256)
            rows = pos[a:b]
            seen = pos[None, :b] <= rows[:, None]
            groups = (rows + 1) // r                                          # complete groups of each row
            if int(groups[-1]) > c.idx_topk_blocks:
                n = int(groups[-1])
                s = torch.relu(torch.einsum("thd,gd->tgh", iq[a:b], ck[:n])).sum(-1)
                s = s.masked_fill(torch.arange(n, device=x.device)[None] >= groups[:, None], -1.0)
                best = torch.sort(-s, dim=1, stable=True).indices[:, :c.idx_topk_blocks]
                chosen = torch.zeros_like(s, dtype=torch.bool).scatter_(1, best, True) | (groups <= c.idx_topk_blocks)[:, None]
                by_token = F.pad(chosen.repeat_interleave(r, 1), (0, max(0, b - n * r)))[:, :b]
                seen &= by_token | (pos[None, :b] >= (groups * r)[:, None])
            w = torch.bmm(q[a:b].permute(1, 0, 2), kh[:, :, :b]) / math.sqrt(D)
            w = torch.softmax(w.masked_fill(~seen, -math.inf), -1)
            out[a:b] = torch.bmm(w, vh[:, :b]).permute(1, 0, 2).reshape(b - a, -1)
        return (out * torch.sigmoid(qg[:, :, 1]).reshape(T, -1)) @ self.W(p + "o_proj.weight").T

    def moe(self, p, x):
        c = self.c
        pr = torch.softmax(x @ self.W(p + "gate.weight").T, -1)
        idx = torch.sort(-pr, dim=-1, stable=True).indices[:, :c.top_k]
        wgt = pr.gather(1, idx)
        wgt = wgt / wgt.sum(-1, keepdim=True)
        out = torch.zeros_like(x)
        for e in torch.unique(idx).tolist():
            rows, at = torch.nonzero(idx == e, as_tuple=True)
            g, u, d = (_q4(self.w[p + f"experts.{n}.weight_packed"][e], self.w[p + f"experts.{n}.weight_scale"][e])
                       for n in ("gate_proj", "up_proj", "down_proj"))
            h = F.silu(x[rows] @ g.T) * (x[rows] @ u.T)
            out.index_add_(0, rows, (h @ d.T) * wgt[rows, at].unsqueeze(-1))
        s = p + "shared_expert"
        h = F.silu(x @ self.W(s + ".gate_proj.weight").T) * (x @ self.W(s + ".up_proj.weight").T)
        return out + torch.sigmoid(x @ self.W(s + "_gate.weight").T) * (h @ self.W(s + ".down_proj.weight").T)

    def layer(self, p, X, attend):
        y, inj = self.mix(p + "attn_hyper_connection.", X)
        X = self.add(X, attend(y), inj)
        y, inj = self.mix(p + "mlp_hyper_connection.", X)
        return self.add(X, self.moe(p + "mlp.", y), inj)

    def forward(self, tokens, keep):
        """The residual streams behind the last layer, of every token; the delta-net states behind token ``keep``."""
        c = self.c
        X = self.W("embed_tokens.weight")[torch.tensor(tokens, device=DEV)].repeat(1, c.hc)
        for L in range(c.n_layers):
            p = f"layers.{L}."
            if L == c.ple_layer:
                X = self.ple(X, tokens)
            X = self.layer(p, X, (lambda y: self.qsa(p + "self_attn.", y)) if c.is_qsa(L) else (lambda y: self.gdn(p + "linear_attn.", y, keep)))
        return X

    def head(self, X, mixer="hyper_connection_mixer."):
        return self.mix(mixer, X, False) @ self.W("lm_head.weight").T

    def mtp(self, X, following):
        c = self.c
        hn = _rms(X, c.eps) * (1 + self.W("mtp.pre_fc_norm_hidden.weight"))
        en = _rms(self.W("embed_tokens.weight")[torch.tensor(following, device=DEV)], c.eps) * (1 + self.W("mtp.pre_fc_norm_embedding.weight"))
        fh = hn.view(-1, c.hc, c.hidden) @ self.W("mtp.fc_hidden.weight").T
        X = (fh + (en @ self.W("mtp.fc_embedding.weight").T).unsqueeze(1)).reshape(len(following), c.hch)
        return self.layer("mtp.layers.0.", X, lambda y: self.qsa("mtp.layers.0.self_attn.", y))


def _exact_vision(case, seed):
    cfg, w, patches = _vision_inputs(case, seed)
    W = lambda n: w["model.visual." + n].double()      # noqa: E731
    h, wd, D, H = case["h"], case["w"], cfg.dim, cfg.heads
    hd, n, m, side = D // H, h * wd, cfg.merge, cfg.grid_side
    i = torch.arange(n, device=DEV)                     # patches come window by window, m x m each
    block = i // (m * m)
    row = block // (wd // m) * m + i // m % m
    col = block % (wd // m) * m + i % m

    def taps(at, size):                                 # bilinear taps with aligned corners, in 32 bits as positions are
        f = at.float() * (side - 1) / max(size - 1, 1)
        lo = f.floor().long().clamp_max(side - 1)
        return lo, (f.floor().long() + 1).clamp_max(side - 1), (f - f.floor()).double()[:, None]
    y0, y1, fy = taps(row, h)
    x0, x1, fx = taps(col, wd)
    t = W("pos_embed.weight").view(side, side, D)
    place = (t[y0, x0] * (1 - fx) + t[y0, x1] * fx) * (1 - fy) + (t[y1, x0] * (1 - fx) + t[y1, x1] * fx) * fy
    x = patches.to(torch.bfloat16).double() @ W("patch_embed.proj.weight").reshape(D, -1).T + W("patch_embed.proj.bias") + place
    inv = 10000.0 ** (-4.0 * torch.arange(hd // 4, dtype=torch.float64, device=DEV) / hd)
    ang = torch.cat([row.double()[:, None] * inv, col.double()[:, None] * inv], 1)[:, None]

    def rope(v):
        a, b = v.view(n, H, 2, hd // 2).unbind(2)
        return torch.cat([a * ang.cos() - b * ang.sin(), b * ang.cos() + a * ang.sin()], -1).transpose(0, 1)

    def norm(v, p):
        return F.layer_norm(v, (D,), W(p + ".weight"), W(p + ".bias"), cfg.eps)

    def linear(v, p):
        return v @ W(p + ".weight").T + W(p + ".bias")
    for b in range(cfg.depth):
        p = f"blocks.{b}."
        q, k, v = linear(norm(x, p + "norm1"), p + "attn.qkv").split(D, 1)
        q, k, v = rope(q), rope(k), v.reshape(n, H, hd).transpose(0, 1)
        att = torch.softmax(torch.bmm(q, k.transpose(1, 2)) / math.sqrt(hd), -1)
        x = x + linear(torch.bmm(att, v).transpose(0, 1).reshape(n, D), p + "attn.proj")
        x = x + linear(F.gelu(linear(norm(x, p + "norm2"), p + "mlp.linear_fc1"), approximate="tanh"), p + "mlp.linear_fc2")
    y = norm(x, "merger.norm").view(n // (m * m), D * m * m)
    return linear(F.gelu(linear(y, "merger.linear_fc1")), "merger.linear_fc2")


@torch.no_grad()
def exact(case, seed):
    kind = case["kind"]
    if kind == "dense":
        x, w = _dense_inputs(case, seed)
        return x.double() @ w.double().T
    if kind == "experts":
        w, x = _expert_inputs(case, seed)
        c, E = FULL, FULL.n_experts
        w.update({"gate.weight": w["rs"][:E], "shared_expert_gate.weight": w["rs"][E:E + 1],
                  "shared_expert.gate_proj.weight": w["rs"][E + 1:E + 1 + c.ffn], "shared_expert.up_proj.weight": w["rs"][E + 1 + c.ffn:],
                  "shared_expert.down_proj.weight": w["down"]})
        return _Exact(c, w, None).moe("", x.double())
    if kind == "vision":
        return _exact_vision(case, seed)
    cfg = _config(case)
    w = synth_globals(cfg, seed, device=DEV)
    for L in range(cfg.n_layers):
        w.update(synth_layer(cfg, L, seed, device=DEV, exact=False))
    if cfg.mtp:
        w.update(synth_layer(cfg, cfg.n_layers, seed, device=DEV, exact=False, prefix="mtp.layers.0.", qsa=True))
    table = PleTable.synthetic(cfg, rows=PLE_ROWS, layout="f8", seed=seed).shards[0]["weight_f8"].to(DEV)
    logits, hidden, models = [], [], []
    for s, (context, feed) in enumerate(_streams(case, cfg, seed)):
        m = _Exact(cfg, w, table)
        n = len(context)
        if kind == "draft":
            X = m.mtp(m.forward(context, -1), context[1:] + feed)[-1:]
            hidden.append(X.view(1, cfg.hc, cfg.hidden))
            logits.append(m.head(X, "mtp.hyper_connection_mixer."))
            continue
        X = m.forward(context + feed, n + (_accepted(case)[s] if kind == "verify" else len(feed)) - 1)
        logits.append(m.head(X[-1:] if kind == "prefill" else X[n:]))
        m.keys, m.values = [t[n:] for t in m.keys], [t[n:] for t in m.values]
        models.append(m)
    if kind == "draft":
        return {"logits": torch.cat(logits), "hidden": torch.cat(hidden)}
    out = {"logits": logits[0][0] if kind == "prefill" else torch.stack(logits, 1) if kind == "decode" else torch.cat(logits)}
    for i in range(cfg.n_gdn):
        out[f"delta{i}"] = torch.stack([m.delta[i] for m in models])
    for i in range(cfg.n_qsa):
        out[f"k{i}"] = torch.stack([m.keys[i] for m in models])
        out[f"v{i}"] = torch.stack([m.values[i] for m in models])
    return out
