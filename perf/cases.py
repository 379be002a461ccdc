"""Timed cases of the framework on one GPU: the layers of a training step, the update and hash that end it, and three
whole calls (a quantised micro-batch, a tiny fp32 micro-batch, scoring without gradients).

Sizes come from the recipes in ``open_transformers_b200/configs``: width 2048 with 16 query heads x 128 sharing 4, SwiGLU
5632, vocabulary 128 256, 4 x 4096 tokens per micro-batch; width 768 with 12 heads x 64 sharing 4, SwiGLU 2048; and the
two-layer width-256 decoder of the fp32 reproducibility gate.
"""
import math
import zlib

import torch

from open_transformers_b200.config import load_config
from open_transformers_b200.models.fused_loss import fused_ce_z_loss
from open_transformers_b200.ops import autograd as A
from open_transformers_b200.ops import functional as K
from open_transformers_b200.train.engine import TrainEngine

DEV = "cuda"
BF16, F32, F64 = torch.bfloat16, torch.float32, torch.float64
EPS = 1e-5
Z_COEFF = 1e-4
THETA = 500000.0
SHARDS = 8  # virtual ranks whose gradients one update folds (configs/run/single_node_8xb200.yaml)


def listed():
    return [
        # attention of one full-causal layer of the 1B recipe, forward and backward, at the training micro-batch
        {"name": "attn_full", "kind": "attn", "B": 4, "T": 4096, "H": 16, "Hkv": 4, "D": 128, "window": 0, "norm": True},
        # four of five layers of that recipe attend to a 512-key window
        {"name": "attn_window", "kind": "attn", "B": 4, "T": 4096, "H": 16, "Hkv": 4, "D": 128, "window": 512, "norm": True},
        # the 100M recipe's heads at a sequence that is no multiple of a tile (fine-tuning on whole documents)
        {"name": "attn_ragged", "kind": "attn", "B": 2, "T": 1000, "H": 12, "Hkv": 4, "D": 64, "window": 512, "norm": True},
        # pre-norm feed-forward sublayer with its residual, forward and backward with weight gradients: 1B recipe
        {"name": "ffn_1b", "kind": "ffn", "tokens": 16384, "d": 2048, "F": 5632},
        # the same sublayer of the 100M recipe on an odd number of tokens
        {"name": "ffn_small", "kind": "ffn", "tokens": 1111, "d": 768, "F": 2048},
        # vocabulary projection, fused cross-entropy + z-loss and their backward: the largest single layer of a step
        {"name": "head_loss", "kind": "head", "tokens": 16384, "d": 2048, "V": 128256},
        # micro-batch of a model with int8 (LSQ) projections, int8 P V attention, QK-norm gains and embedding norm, as
        # configs/train/1b_repop.yaml trains it, cut to two layers and a small vocabulary
        {"name": "micro_qat", "kind": "micro", "recipe": "1b_repop", "B": 2, "T": 4096, "layers": 2, "vocab": 8192, "accum": 1},
        # micro-batch of the fp32 reproducibility gate (configs/train/tiny_cpu.yaml): the smallest training call
        {"name": "micro_tiny_fp32", "kind": "micro", "recipe": "tiny_cpu", "B": 4, "T": 512, "layers": 2, "vocab": 1024, "accum": 1},
        # scoring / one decode position: the 100M model's logits for one prompt, no gradients (there is no KV cache)
        {"name": "logits_prompt", "kind": "logits", "recipe": "100m_smoke_repop", "B": 1, "T": 333, "layers": 6, "vocab": 128256},
        # end of a step: fold of 8 virtual ranks' gradients, global norm, clip, AdamW and the bf16 weights
        {"name": "update", "kind": "update", "layers": 2, "vocab": 8192},
        # chained hash of the whole training state (weights, moments, gradient), every step of an audited run
        {"name": "state_hash", "kind": "hash", "layers": 2, "vocab": 8192},
    ]


def _log(rng, lo, hi, step=1):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / step)) * step))


def draw(rng):
    kind = rng.choice(["attn", "attn", "ffn", "ffn", "head", "micro", "micro", "logits", "update", "hash"])
    if kind == "attn":
        D, H, Hkv = rng.choice([(128, 16, 4), (64, 12, 4), (64, 4, 4)])
        T = _log(rng, 33, 4096, rng.choice([1, 64]))
        return {"kind": kind, "B": rng.randint(1, max(1, min(8, 16384 // T))), "T": T, "H": H, "Hkv": Hkv, "D": D,
                "window": rng.choice([0, 512]), "norm": rng.random() < 0.75}
    if kind == "ffn":
        d, F = rng.choice([(2048, 5632), (768, 2048), (256, 704)])
        return {"kind": kind, "tokens": _log(rng, 64, 16384), "d": d, "F": F}
    if kind == "head":
        d, V = rng.choice([(2048, 128256), (768, 128256), (256, 1024)])
        return {"kind": kind, "tokens": _log(rng, 64, 8192), "d": d, "V": V}
    if kind == "micro":
        if rng.random() < 0.5:
            return {"kind": kind, "recipe": "tiny_cpu", "B": rng.randint(1, 4), "T": _log(rng, 32, 512), "layers": 2, "vocab": 1024,
                    "accum": rng.randint(1, 4)}
        T = _log(rng, 128, 4096, 64)
        return {"kind": kind, "recipe": "1b_repop", "B": rng.randint(1, max(1, min(4, 8192 // T))), "T": T, "layers": 2, "vocab": 8192,
                "accum": rng.randint(1, 4)}
    if kind == "logits":
        return {"kind": kind, "recipe": "100m_smoke_repop", "B": rng.randint(1, 2), "T": _log(rng, 16, 2048), "layers": 6, "vocab": 128256}
    return {"kind": kind, "layers": rng.randint(1, 3), "vocab": 1024 * rng.randint(4, 12)}


# ------------------------------------------------------------------------------------------------ inputs
def _gen(seed, what):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 1000003 + zlib.crc32(what.encode()))
    return g


def _randn(seed, what, shape, dtype=BF16, std=1.0):
    return (torch.randn(shape, generator=_gen(seed, what), device=DEV, dtype=F32) * std).to(dtype)


def _tokens(seed, what, shape, vocab):
    return torch.randint(0, vocab, shape, generator=_gen(seed, what), device=DEV)


def _recipe(case):
    """Plain numbers of the model a whole-call case builds (the recipes' values, with the case's cuts)."""
    r = case.get("recipe", "open1b_b200")
    if r == "tiny_cpu":
        m = dict(d=256, H=4, Hkv=4, D=64, F=704, theta=10000.0, window=0, every=1, qk_norm=False, gain=False, qat=False, emb_norm=False, bf16=False)
    elif r == "100m_smoke_repop":
        m = dict(d=768, H=12, Hkv=4, D=64, F=2048, theta=THETA, window=512, every=5, qk_norm=True, gain=False, qat=False, emb_norm=False, bf16=True)
    elif r == "1b_repop":
        m = dict(d=2048, H=16, Hkv=4, D=128, F=5632, theta=THETA, window=512, every=5, qk_norm=True, gain=True, qat=True, emb_norm=True, bf16=True)
    else:
        m = dict(d=2048, H=16, Hkv=4, D=128, F=5632, theta=THETA, window=512, every=5, qk_norm=True, gain=False, qat=False, emb_norm=False, bf16=True)
    m.update(L=case["layers"], V=case["vocab"])
    return m


def _config(case):
    r = case.get("recipe", "open1b_b200")
    over = ["model.n_layers=%d" % case["layers"], "model.vocab_size=%d" % case["vocab"], "run.dp_replicate_size=1"]
    if case["kind"] in ("micro", "logits"):
        over += ["run.virtual_dp_size=1", "run.dp_shard_size=1", "run.activation_checkpoint=false"]
    else:
        over += ["run.virtual_dp_size=%d" % SHARDS, "run.dp_shard_size=%d" % SHARDS]
    if r == "100m_smoke_repop":
        over += ["model.qat.enabled=false"]
    return load_config(r, over)


def _shapes(m):
    lin = lambda i, n, o, k: [("blocks.%d.%s.weight" % (i, n), (o, k))] + ([("blocks.%d.%s.weight_scale" % (i, n), (o,))] if m["qat"] else [])  # noqa: E731
    out = [("embedding.tok_embeddings.weight", (m["V"], m["d"])), ("embedding.output.weight", (m["V"], m["d"])), ("norm_out.weight", (m["d"],))]
    if m["emb_norm"]:
        out.append(("emb_norm.weight", (m["d"],)))
    for i in range(m["L"]):
        out += [("blocks.%d.norm1.weight" % i, (m["d"],)), ("blocks.%d.norm2.weight" % i, (m["d"],))]
        out += lin(i, "attn.wq", m["H"] * m["D"], m["d"]) + lin(i, "attn.wk", m["Hkv"] * m["D"], m["d"]) + lin(i, "attn.wv", m["Hkv"] * m["D"], m["d"])
        out += lin(i, "attn.wo", m["d"], m["H"] * m["D"]) + lin(i, "ffn.w_gate_up", 2 * m["F"], m["d"]) + lin(i, "ffn.w_down", m["d"], m["F"])
        if m["gain"]:
            out += [("blocks.%d.attn.q_norm.weight" % i, (m["D"],)), ("blocks.%d.attn.k_norm.weight" % i, (m["D"],))]
    return out


def _weights(m, seed):
    """fp32 masters of every parameter: matrices as initialised (0.02), gains around one, step sizes from their matrices."""
    w = {}
    for name, shape in _shapes(m):
        if name.endswith("weight_scale"):
            ref = w[name[: -len("_scale")]].to(BF16).float()
            w[name] = ref.abs().mean(1) * (2.0 / math.sqrt(127.0))
        elif len(shape) == 1:
            w[name] = 1.0 + _randn(seed, name, shape, F32, 0.1)
        else:
            w[name] = _randn(seed, name, shape, F32, 0.02)
    return w


def _engine(case, seed, moments=False):
    m = _recipe(case)
    eng = TrainEngine(_config(case), DEV, init=False)
    w = _weights(m, seed)
    assert sorted(w) == sorted(eng.names)
    for i, name in enumerate(eng.names):
        if moments:
            eng.load_parameter_state(i, w[name], *_moments(seed, name, w[name].shape))
        else:
            eng.load_parameter_state(i, w[name], None, None)
    eng.refresh_compute_weights()
    return eng


def _moments(seed, name, shape):
    return _randn(seed, name + ".m", shape, F32, 1e-4), _randn(seed, name + ".v", shape, F32, 1e-4).square_()


def prepare(case, seed):
    k = case["kind"]
    if k == "attn":
        n = (case["H"] + 2 * case["Hkv"]) * case["D"]
        cos, sin = K.rope_tables(case["T"], case["D"], THETA, DEV)
        return {"case": case, "qkv": _randn(seed, "qkv", (case["B"], case["T"], n)).requires_grad_(), "cos": cos, "sin": sin,
                "dO": _randn(seed, "dO", (case["B"], case["T"], case["H"] * case["D"]))}
    if k == "ffn":
        d, F, t = case["d"], case["F"], case["tokens"]
        s = {"case": case, "x": _randn(seed, "x", (t, d)).requires_grad_(), "dy": _randn(seed, "dy", (t, d))}
        for name, shape, std in (("gain", (d,), 0.1), ("gate_up", (2 * F, d), 0.02), ("down", (d, F), 0.02)):
            master = _randn(seed, name, shape, F32, std)
            if name == "gain":
                master += 1.0
            s[name] = (master.requires_grad_(), master.detach().to(BF16), A.GradSlot(torch.empty(shape, dtype=F32, device=DEV)))
        return s
    if k == "head":
        w = _randn(seed, "w", (case["V"], case["d"]), BF16, 0.02)
        # the parameter autograd sees; its gradient goes to the slot, as in the training engine
        return {"case": case, "h": _randn(seed, "h", (case["tokens"], case["d"])).requires_grad_(), "w": w, "master": w.float().requires_grad_(),
                "labels": _tokens(seed, "labels", (case["tokens"],), case["V"]), "slot": A.GradSlot(torch.empty(w.shape, dtype=F32, device=DEV))}
    if k in ("micro", "logits"):
        ids = _tokens(seed, "ids", (case["B"], case["T"]), case["vocab"])
        return {"case": case, "eng": _engine(case, seed), "ids": ids, "labels": _tokens(seed, "labels", (case["B"], case["T"]), case["vocab"])}
    eng = _engine(case, seed, moments=True)
    eng.opt_step = 100
    if k == "update":
        for v, g in enumerate(eng.grads):
            for i, name in enumerate(eng.names):
                view = eng.layout.view(g, i)
                view.copy_(_randn(seed, "%s.g%d" % (name, v), tuple(view.shape), F32, 1e-4))
    else:
        for i, name in enumerate(eng.names):
            view = eng.layout.view(eng.grad_red, i)
            view.copy_(_randn(seed, name + ".g", tuple(view.shape), F32, 1e-4))
    return {"case": case, "eng": eng}


def _store(slot):
    """First micro-batch of a step: the gradient slot is stale and its first writer stores."""
    slot.fresh, slot.written = True, False
    return slot


def run(s):
    case = s["case"]
    k = case["kind"]
    if k == "attn":
        o = A.attention(s["qkv"], s["cos"], s["sin"], case["H"], case["Hkv"], case["D"], case["window"], case["norm"], EPS)
        (dqkv,) = torch.autograd.grad(o, s["qkv"], s["dO"])
        return {"o": o.detach(), "dqkv": dqkv}
    if k == "ffn":
        gain, gu, dn = s["gain"], s["gate_up"], s["down"]
        h = A.rms_norm(s["x"], gain[0], gain[1], _store(gain[2]), EPS)
        h = A.swiglu(A.linear(h, gu[0], gu[1], _store(gu[2])))
        y = A.linear(h, dn[0], dn[1], _store(dn[2]), residual=s["x"])
        (dx,) = torch.autograd.grad(y, s["x"], s["dy"])
        return {"y": y.detach(), "dx": dx, "gain": gain[2].buf, "gate_up": gu[2].buf, "down": dn[2].buf}
    if k == "head":
        logits = A.linear(s["h"], s["master"], s["w"], _store(s["slot"]))
        ce, z = fused_ce_z_loss(logits, s["labels"], Z_COEFF)
        (dh,) = torch.autograd.grad(ce + z, s["h"])
        return {"ce": ce.detach(), "z": z.detach(), "dh": dh, "dw": s["slot"].buf}
    eng = s["eng"]
    if k == "micro":
        eng.zero_grads()
        ce, z = eng.forward_backward(0, s["ids"], s["labels"], case["accum"])
        return {"ce": ce.detach(), "z": z.detach(), "grads": {n: eng.layout.view(eng.grads[0], i) for i, n in enumerate(eng.names)}}
    if k == "logits":
        with torch.no_grad():
            eng.model.eval()
            return {"logits": eng.model(s["ids"]).logits}
    if k == "update":
        norm = eng.reduce_gradients()
        eng.optimizer_step(4.5e-4, eng.clip_coefficient(norm, 1.0))
        return {"norm": norm, "grad": eng.grad_red, "master": {n: eng.layout.view(eng.master, i) for i, n in enumerate(eng.names)},
                "m": eng.m1, "v": eng.m2, "weights": eng.compute}
    return {"hash": torch.tensor(list(bytes.fromhex(eng.sharded_state_hash(None, None, tensor_digest="tree"))), dtype=torch.int64)}


# --------------------------------------------------------------------------------- what a pass cannot do without
def _pairs(T, window):
    """Query-key pairs of one head of one causal (windowed) sequence."""
    w = T if window == 0 else min(window, T)
    return w * (w + 1) // 2 + (T - w) * w


def _params(m):
    return sum(math.prod(s) for _, s in _shapes(m))


def _forward_work(m, B, T):
    """(FLOPs, bytes) of one forward pass: matrix products and attention; weights, tokens and logits once each."""
    t, e = B * T, 2 if m["bf16"] else 4
    mats = m["L"] * (m["d"] * (m["H"] + 2 * m["Hkv"]) * m["D"] + m["H"] * m["D"] * m["d"] + 3 * m["d"] * m["F"]) + m["V"] * m["d"]
    pairs = 0
    for i in range(m["L"]):
        full = i % m["every"] == m["every"] - 1 or i == m["L"] - 1
        pairs += B * m["H"] * _pairs(T, 0 if full else m["window"])
    return 2.0 * t * mats + 4.0 * pairs * m["D"], e * (mats + t * m["d"] + t * m["V"])


def work(case):
    k = case["kind"]
    if k == "attn":
        t, D = case["B"] * case["T"], case["D"]
        pairs = case["B"] * case["H"] * _pairs(case["T"], case["window"])
        return {"flops": 14.0 * pairs * D, "bytes": 2.0 * t * D * (2 * (case["H"] + 2 * case["Hkv"]) + 2 * case["H"])}
    if k == "ffn":
        t, d, F = case["tokens"], case["d"], case["F"]
        return {"flops": 18.0 * t * d * F, "bytes": 2.0 * 4 * t * d + 3 * d * F * (2 + 4)}
    if k == "head":
        t, d, V = case["tokens"], case["d"], case["V"]
        return {"flops": 6.0 * t * d * V, "bytes": 2.0 * 2 * t * d + V * d * (2 + 4)}
    m = _recipe(case)
    n = _params(m)
    if k == "micro":
        f, _ = _forward_work(m, case["B"], case["T"])
        e = 2 if m["bf16"] else 4
        # backward: twice the products of the forward, attention 2.5 x; weights read, gradients written
        return {"flops": 3.0 * f, "bytes": float(n * (e + 4))}
    if k == "logits":
        f, b = _forward_work(m, case["B"], case["T"])
        return {"flops": f, "bytes": float(b)}
    if k == "update":
        return {"bytes": float(n * (4 * SHARDS + 4 + 3 * 8 + 2)), "flops": 0.0}
    return {"bytes": 16.0 * n, "flops": 0.0}


def tolerance(case):
    k = case["kind"]
    if k == "hash":
        return "exact"
    if k == "update":
        return {"rel": 1e-5}
    if k == "micro":
        return {"rel": 1e-5} if case["recipe"] == "tiny_cpu" else {"rel": 0.03}
    if k == "logits":
        return {"rel": 0.02}
    return {"rel": 0.01}


# ------------------------------------------------------------------------------------------- the same in 64 bits
def _rms64(x, g=None):
    y = x * torch.rsqrt(x.square().mean(-1, keepdim=True) + EPS)
    return y if g is None else y * g


def _rope64(x, theta):
    """x [B, T, heads, D]: element pairs (2j, 2j + 1) turn by t * theta^(-2j / D); tables rounded to fp32 once."""
    T, D = x.shape[1], x.shape[3]
    ang = torch.arange(T, device=DEV, dtype=F64)[:, None] / theta ** (torch.arange(D // 2, device=DEV, dtype=F64) * 2 / D)
    c, s = (f.float().double()[None, :, None, :] for f in (ang.cos(), ang.sin()))
    a, b = x[..., 0::2], x[..., 1::2]
    return torch.stack([a * c - b * s, a * s + b * c], -1).flatten(-2)


class _Attend64(torch.autograd.Function):
    """Softmax attention of q [B, H, T, D] over k, v [B, Hkv, T, D], a block of queries at a time in both directions."""

    STEP = 512

    @staticmethod
    def _p(q, k, i, window):
        T, D = k.shape[-2], k.shape[-1]
        s = (q[..., i:i + _Attend64.STEP, :] @ k.transpose(-1, -2)) / math.sqrt(D)
        qi, kj = torch.arange(i, i + s.shape[-2], device=DEV)[:, None], torch.arange(T, device=DEV)[None]
        dead = (kj > qi) | ((kj <= qi - window) if window else False)
        return torch.softmax(s.masked_fill(dead, -math.inf), -1)

    @staticmethod
    def forward(ctx, q, k, v, window):
        ctx.save_for_backward(q, k, v)
        ctx.window = window
        G = q.shape[1] // k.shape[1]
        o = torch.empty_like(q)
        for b in range(q.shape[0]):
            for h in range(q.shape[1]):
                for i in range(0, q.shape[2], _Attend64.STEP):
                    o[b, h, i:i + _Attend64.STEP] = _Attend64._p(q[b, h], k[b, h // G], i, window) @ v[b, h // G]
        return o

    @staticmethod
    def backward(ctx, do):
        q, k, v = ctx.saved_tensors
        G, D = q.shape[1] // k.shape[1], q.shape[-1]
        dq, dk, dv = torch.zeros_like(q), torch.zeros_like(k), torch.zeros_like(v)
        for b in range(q.shape[0]):
            for h in range(q.shape[1]):
                g = h // G
                for i in range(0, q.shape[2], _Attend64.STEP):
                    rows = slice(i, i + _Attend64.STEP)
                    p, d = _Attend64._p(q[b, h], k[b, g], i, ctx.window), do[b, h, rows]
                    dv[b, g] += p.T @ d
                    dp = d @ v[b, g].T
                    ds = p * (dp - (p * dp).sum(-1, keepdim=True)) / math.sqrt(D)
                    dq[b, h, rows] = ds @ k[b, g]
                    dk[b, g] += ds.T @ q[b, h, rows]
        return dq, dk, dv, None


def _attention64(qkv, H, Hkv, D, window, norm, theta, gains=None):
    B, T, _ = qkv.shape
    q, k, v = qkv.split([H * D, Hkv * D, Hkv * D], -1)
    q, k, v = q.reshape(B, T, H, D), k.reshape(B, T, Hkv, D), v.reshape(B, T, Hkv, D)
    if norm:
        q, k = _rms64(q, gains[0] if gains else None), _rms64(k, gains[1] if gains else None)
    q, k = _rope64(q, theta), _rope64(k, theta)
    o = _Attend64.apply(q.transpose(1, 2), k.transpose(1, 2), v.transpose(1, 2), window)
    return o.transpose(1, 2).reshape(B, T, H * D)


def _swiglu64(gu):
    g, u = gu.chunk(2, -1)
    return torch.nn.functional.silu(g) * u


class _Quant64(torch.autograd.Function):
    """W8A8 product with learned steps: straight through the rounding, gradients as the learned-step method defines them."""

    @staticmethod
    def forward(ctx, x, w, s):
        sa = (x.abs().max() / 127.0).clamp_min(1.2e-38)
        xq, t = (x / sa).round().clamp(-127, 127), w / s[:, None]
        wh = t.round().clamp(-127, 127) * s[:, None]
        ctx.save_for_backward(xq * sa, wh, t, s)
        return (xq * sa) @ wh.T

    @staticmethod
    def backward(ctx, dy):
        xh, wh, t, s = ctx.saved_tensors
        G = dy.reshape(-1, dy.shape[-1]).T @ xh.reshape(-1, xh.shape[-1])
        inside = t.abs() <= 127
        ds = (G * torch.where(inside, t.round() - t, torch.sign(t) * 127)).sum(1) / math.sqrt(t.shape[1] * 127.0)
        return dy @ wh, G * inside, ds


def _model64(m, w, ids):
    def lin(x, name):
        if m["qat"]:
            return _Quant64.apply(x, w[name + ".weight"], w[name + ".weight_scale"])
        return x @ w[name + ".weight"].T

    x = w["embedding.tok_embeddings.weight"][ids]
    if m["emb_norm"]:
        x = _rms64(x, w["emb_norm.weight"])
    for i in range(m["L"]):
        b = "blocks.%d." % i
        full = i % m["every"] == m["every"] - 1 or i == m["L"] - 1
        h = _rms64(x, w[b + "norm1.weight"])
        qkv = torch.cat([lin(h, b + "attn." + n) for n in ("wq", "wk", "wv")], -1)
        gains = (w[b + "attn.q_norm.weight"], w[b + "attn.k_norm.weight"]) if m["gain"] else None
        x = x + lin(_attention64(qkv, m["H"], m["Hkv"], m["D"], 0 if full else m["window"], m["qk_norm"], m["theta"], gains), b + "attn.wo")
        x = x + lin(_swiglu64(lin(_rms64(x, w[b + "norm2.weight"]), b + "ffn.w_gate_up")), b + "ffn.w_down")
    return _rms64(x, w["norm_out.weight"]) @ w["embedding.output.weight"].T


def _loss64(logits, labels, z_coeff):
    lse = torch.logsumexp(logits, -1)
    return (lse - logits.gather(-1, labels[..., None])[..., 0]).mean(), z_coeff * lse.square().mean()


def exact(case, seed):
    k = case["kind"]
    if k == "attn":
        qkv = _randn(seed, "qkv", (case["B"], case["T"], (case["H"] + 2 * case["Hkv"]) * case["D"])).double().requires_grad_()
        dO = _randn(seed, "dO", (case["B"], case["T"], case["H"] * case["D"])).double()
        o = _attention64(qkv, case["H"], case["Hkv"], case["D"], case["window"], case["norm"], THETA)
        (dqkv,) = torch.autograd.grad(o, qkv, dO)
        return {"o": o.detach(), "dqkv": dqkv}
    if k == "ffn":
        d, F, t = case["d"], case["F"], case["tokens"]
        x, dy = _randn(seed, "x", (t, d)).double().requires_grad_(), _randn(seed, "dy", (t, d)).double()
        gain = (_randn(seed, "gain", (d,), F32, 0.1) + 1.0).to(BF16).double().requires_grad_()
        gu = _randn(seed, "gate_up", (2 * F, d), F32, 0.02).to(BF16).double().requires_grad_()
        dn = _randn(seed, "down", (d, F), F32, 0.02).to(BF16).double().requires_grad_()
        y = x + _swiglu64(_rms64(x, gain) @ gu.T) @ dn.T
        dx, a, b, c = torch.autograd.grad(y, (x, gain, gu, dn), dy)
        return {"y": y.detach(), "dx": dx, "gain": a, "gate_up": b, "down": c}
    if k == "head":
        t, d, V = case["tokens"], case["d"], case["V"]
        h, w = _randn(seed, "h", (t, d)).double(), _randn(seed, "w", (V, d), BF16, 0.02).double()
        labels = _tokens(seed, "labels", (t,), V)
        ce, z = torch.zeros((), dtype=F64, device=DEV), torch.zeros((), dtype=F64, device=DEV)
        dh, dw = torch.empty_like(h), torch.zeros_like(w)
        for i in range(0, t, 2048):  # rows are independent but for the weight gradient
            rows = slice(i, min(i + 2048, t))
            x = h[rows] @ w.T
            lse = torch.logsumexp(x, -1)
            ce += (lse - x.gather(-1, labels[rows, None])[:, 0]).sum() / t
            z += Z_COEFF * lse.square().sum() / t
            g = torch.exp(x - lse[:, None]) * ((1 + 2 * Z_COEFF * lse) / t)[:, None]
            g[torch.arange(g.shape[0], device=DEV), labels[rows]] -= 1.0 / t
            dh[rows] = g @ w
            dw += g.T @ h[rows]
        return {"ce": ce, "z": z, "dh": dh, "dw": dw}
    if k == "hash":
        return None
    m = _recipe(case)
    w = _weights(m, seed)
    if k == "update":
        return _update64(m, w, seed)
    w = {n: (v.to(BF16) if m["bf16"] else v).double() for n, v in w.items()}
    ids, labels = _tokens(seed, "ids", (case["B"], case["T"]), m["V"]), _tokens(seed, "labels", (case["B"], case["T"]), m["V"])
    if k == "logits":
        with torch.no_grad():
            return {"logits": _model64(m, w, ids)}
    for v in w.values():
        v.requires_grad_()
    ce, z = _loss64(_model64(m, w, ids), labels, Z_COEFF)
    names = sorted(w)
    if m["qat"]:
        # int8 P V quantises the values block by block in the forward pass only, and a rounding to int8 that falls the
        # other way travels through every layer after it: the gradients have no plain counterpart, the losses do
        return {"ce": ce.detach(), "z": z.detach(), "grads": None}
    grads = torch.autograd.grad((ce + z) / case["accum"], [w[n] for n in names])
    return {"ce": ce.detach(), "z": z.detach(), "grads": dict(zip(names, grads))}


def _update64(m, w, seed):
    """Norm and masters after the update; the other outputs are the engine's flat buffers, in an order of its own."""
    red = {}
    for name, shape in _shapes(m):
        red[name] = sum(_randn(seed, "%s.g%d" % (name, v), shape, F32, 1e-4).double() for v in range(SHARDS)) / SHARDS
    norm = math.sqrt(sum(float(g.square().sum()) for g in red.values()))
    lr, b1, b2, t = 4.5e-4, 0.9, 0.95, 101
    master = {}
    for name, shape in _shapes(m):
        g, p = red[name] * min(1.0, 1.0 / (norm + 1e-6)), w[name].double()
        m1, m2 = (x.double() for x in _moments(seed, name, shape))
        m1, m2 = b1 * m1 + (1 - b1) * g, b2 * m2 + (1 - b2) * g * g
        if len(shape) > 1 and "tok_embeddings" not in name:
            p = p * (1 - lr * 0.1)
        master[name] = p - lr * (m1 / (1 - b1 ** t)) / ((m2 / (1 - b2 ** t)).sqrt() + 1e-8)
    return {"norm": norm, "grad": None, "master": master, "m": None, "v": None, "weights": None}
