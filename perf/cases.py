"""Performance cases: the layers and ops a training or evaluation program spends its time in.

Each case goes through the public entry points (`bux_b200.ops`, `bux_b200.models.Model`) with the
shapes of this repository's architectures: Qwen3-30B-A3B (d 2048, 32/4 heads of 128, 128 experts of
768, vocabulary 151936), Llama-3-8B (d 4096, 32/8 heads of 128, feed-forward 14336) and
gpt-oss-20b (64/8 heads of 64, window 128, sinks, 32 experts of 2880). A training case is the
forward and the backward and returns the output and every gradient; an evaluation case is the
forward alone. Upstream gradients are given, as the layer above would hand them down.
"""

from __future__ import annotations

import math

import torch
import torch.nn.functional as F

from bux_b200 import ops
from bux_b200.lang import compile as compile_bux
from bux_b200.models import Model

DEV = "cuda"


def listed():
    return [
        # Qwen3-30B-A3B's attention in training: 4096-token rows, 8 query heads per key head
        {"name": "attn_train", "kind": "attention", "b": 2, "t": 4096, "h": 32, "g": 4, "d": 128,
         "window": 0, "sinks": False, "docs": 0, "train": True},
        # gpt-oss-20b's local layers in training: heads of 64, a 128-token window, learned sinks
        {"name": "attn_window_sinks", "kind": "attention", "b": 2, "t": 4096, "h": 64, "g": 8, "d": 64,
         "window": 128, "sinks": True, "docs": 0, "train": True},
        # Llama-3-8B's attention on documents packed into one row of odd length
        {"name": "attn_packed", "kind": "attention", "b": 1, "t": 6137, "h": 32, "g": 8, "d": 128,
         "window": 0, "sinks": False, "docs": 5, "train": True},
        # Llama-3-8B's feed-forward projection in bf16 training
        {"name": "linear_bf16", "kind": "linear", "m": 8192, "k": 4096, "n": 14336, "fmt": "bf16", "train": True},
        # a fused qkv projection of a handful of tokens (sampling, the last rows of an evaluation)
        {"name": "linear_small", "kind": "linear", "m": 16, "k": 4096, "n": 6144, "fmt": "bf16", "train": False},
        # Qwen3-30B-A3B's qkv projection in MXFP8 training (a weight gathered for the block)
        {"name": "linear_mxfp8", "kind": "linear", "m": 16384, "k": 2048, "n": 5120, "fmt": "mxfp8", "train": True},
        # Qwen3-30B-A3B's expert layer in MXFP8 training
        {"name": "moe_mxfp8", "kind": "moe", "t": 16384, "d": 2048, "f": 768, "e": 128, "k": 8, "act": "swish",
         "limit": 0.0, "up_offset": 0.0, "fmt": "mxfp8", "train": True},
        # gpt-oss-20b's expert layer in bf16 on an odd, small number of tokens
        {"name": "moe_bf16_ragged", "kind": "moe", "t": 777, "d": 2880, "f": 2880, "e": 32, "k": 4, "act": "quick_gelu",
         "limit": 7.0, "up_offset": 1.0, "fmt": "bf16", "train": True},
        # the output matrix and the loss over Qwen3's vocabulary, logits never whole
        {"name": "head_loss", "kind": "head", "t": 4096, "d": 2048, "v": 151936},
        # the pre-norm of a block's stream
        {"name": "rmsnorm", "kind": "rmsnorm", "t": 16384, "d": 2048},
        # per-head norm and rotation of Qwen3's queries
        {"name": "qk_norm_rope", "kind": "rope", "b": 2, "t": 4096, "h": 32, "d": 128},
        # a whole small dense model, loss and all gradients: short rows, many launches
        {"name": "model_train", "kind": "model", "b": 1, "t": 509, "d": 1024, "f": 3072, "v": 8192, "blocks": 2},
    ]


def _log(rng, lo, hi, step=1):
    return max(1, int(math.exp(rng.uniform(math.log(lo), math.log(hi))) // step)) * step


def draw(rng):
    kind = rng.choice(["attention", "attention", "linear", "linear", "moe", "moe", "head", "rmsnorm", "rope", "model"])
    if kind == "attention":
        h, g, d = rng.choice([(32, 4, 128), (32, 8, 128), (64, 8, 64), (16, 8, 128)])
        docs = rng.choice([0, 0, rng.randint(2, 9)])
        return {"kind": kind, "b": rng.randint(1, 2), "t": _log(rng, 100, 4096), "h": h, "g": g, "d": d,
                "window": rng.choice([0, 0, 128, 1024]), "sinks": d == 64, "docs": docs, "train": rng.random() < 0.7}
    if kind == "linear":
        fmt = rng.choice(["bf16", "mxfp8"])
        k, n = rng.choice([(2048, 5120), (4096, 6144), (4096, 2048), (4096, 14336), (14336, 4096)])
        return {"kind": kind, "m": _log(rng, 1, 8192), "k": k, "n": n, "fmt": fmt, "train": rng.random() < 0.6}
    if kind == "moe":
        if rng.random() < 0.5:
            return {"kind": kind, "t": _log(rng, 16, 16384), "d": 2048, "f": 768, "e": 128, "k": 8, "act": "swish",
                    "limit": 0.0, "up_offset": 0.0, "fmt": rng.choice(["bf16", "mxfp8"]), "train": rng.random() < 0.7}
        return {"kind": kind, "t": _log(rng, 16, 4096), "d": 2880, "f": 2880, "e": 32, "k": 4, "act": "quick_gelu",
                "limit": 7.0, "up_offset": 1.0, "fmt": "bf16", "train": rng.random() < 0.7}
    if kind == "head":
        d, v = rng.choice([(2048, 151936), (4096, 128256), (2880, 201088), (1024, 8192)])
        return {"kind": kind, "t": _log(rng, 64, 2048), "d": d, "v": v}
    if kind == "rmsnorm":
        return {"kind": kind, "t": _log(rng, 1, 32768), "d": rng.choice([1024, 2048, 2880, 4096])}
    if kind == "rope":
        h, d = rng.choice([(32, 128), (4, 128), (8, 128), (64, 64)])
        return {"kind": kind, "b": rng.randint(1, 2), "t": _log(rng, 16, 4096), "h": h, "d": d}
    return {"kind": kind, "b": rng.randint(1, 2), "t": _log(rng, 32, 2048), "d": 1024, "f": 3072, "v": 8192, "blocks": 2}


# ------------------------------------------------------------------ inputs
def _rand(gen, *shape, std=1.0, dtype=torch.bfloat16):
    return (torch.randn(*shape, generator=gen, device=DEV, dtype=torch.float32) * std).to(dtype)


def _document_ids(case, gen):
    """Rows cut into `docs` documents at random places: ids that never fall along a row."""
    b, t, docs = case["b"], case["t"], case["docs"]
    cuts = torch.zeros(b, t, dtype=torch.int32, device=DEV)
    at = torch.randint(1, t, (b, docs - 1), generator=gen, device=DEV)
    cuts.scatter_(1, at, 1)
    return torch.cumsum(cuts, 1, dtype=torch.int32)


def _rope_tables(b, t, d):
    inv = 1e6 ** (-torch.arange(0, d, 2, dtype=torch.float32, device=DEV) / d)
    angle = torch.arange(t, dtype=torch.float32, device=DEV)[:, None] * inv
    angle = angle.expand(b, t, d // 2).contiguous()
    return angle.cos(), angle.sin()


MODEL = """
d_model    = {d}
vocab_size = {v}
norm  = rmsnorm(eps=1e-6)
attn  = gqa(num_heads=8, num_kv_heads=2, head_dim=128, qk_norm=norm, rope=rope(base=1000000))
ffn   = gated_mlp(intermediate_size={f}, activation=swish)
block = [norm attn] [norm ffn]
model = embed block^{blocks} norm head
"""


def prepare(case, seed):
    gen = torch.Generator(device=DEV).manual_seed(int(seed))
    kind = case["kind"]
    s = {"case": case}
    if kind == "attention":
        b, t, h, g, d = (case[n] for n in ("b", "t", "h", "g", "d"))
        s["q"], s["k"], s["v"] = _rand(gen, b, t, h, d), _rand(gen, b, t, g, d), _rand(gen, b, t, g, d)
        s["sinks"] = _rand(gen, h, dtype=torch.float32) if case["sinks"] else None
        s["segments"] = _document_ids(case, gen) if case["docs"] > 1 else None
        s["dy"] = _rand(gen, b, t, h, d, std=0.1)
        s["inputs"] = [s[n] for n in ("q", "k", "v", "sinks") if s[n] is not None]
    elif kind == "linear":
        m, k, n = case["m"], case["k"], case["n"]
        s["x"], s["w"] = _rand(gen, m, k), _rand(gen, n, k, std=0.02)
        s["dy"] = _rand(gen, m, n, std=0.1)
        s["inputs"] = [s["x"], s["w"]]
    elif kind == "moe":
        t, d, f, e = case["t"], case["d"], case["f"], case["e"]
        s["x"] = _rand(gen, t, d)
        s["w_gu"], s["w_down"] = _rand(gen, e, 2 * f, d, std=0.02), _rand(gen, e, d, f, std=0.02)
        # a router that favours some experts
        logits = _rand(gen, t, e, dtype=torch.float32) + _rand(gen, 1, e, std=0.5, dtype=torch.float32)
        top, s["experts"] = logits.topk(case["k"], dim=-1)
        s["weights"] = torch.softmax(top, -1)
        s["dy"] = _rand(gen, t, d, std=0.1)
        s["inputs"] = [s["x"], s["w_gu"], s["w_down"], s["weights"]]
    elif kind == "head":
        t, d, v = case["t"], case["d"], case["v"]
        s["x"], s["w"] = _rand(gen, t, d), _rand(gen, v, d, std=0.02)
        s["targets"] = torch.randint(0, v, (t,), generator=gen, device=DEV)
        s["mask"] = torch.rand(t, generator=gen, device=DEV) < 0.95
        s["inputs"] = [s["x"], s["w"]]
    elif kind == "rmsnorm":
        t, d = case["t"], case["d"]
        s["x"], s["w"] = _rand(gen, 1, t, d), 1 + _rand(gen, d, std=0.1, dtype=torch.float32)
        s["dy"] = _rand(gen, 1, t, d, std=0.1)
        s["inputs"] = [s["x"], s["w"]]
    elif kind == "rope":
        b, t, h, d = (case[n] for n in ("b", "t", "h", "d"))
        s["x"], s["w"] = _rand(gen, b, t, h, d), 1 + _rand(gen, d, std=0.1, dtype=torch.float32)
        s["cos"], s["sin"] = _rope_tables(b, t, d)
        s["dy"] = _rand(gen, b, t, h, d, std=0.1)
        s["inputs"] = [s["x"], s["w"]]
    else:
        arch = compile_bux(MODEL.format(**{n: case[n] for n in ("d", "v", "f", "blocks")}), filename="case.bux")
        s["model"] = Model(arch, dtype=torch.bfloat16, seed=int(seed) % (1 << 31), device=DEV)
        s["ids"] = torch.randint(0, case["v"], (case["b"], case["t"]), generator=gen, device=DEV)
        s["targets"] = torch.randint(0, case["v"], (case["b"] * case["t"],), generator=gen, device=DEV)
        s["inputs"] = list(s["model"].parameters())
    if case.get("train", True):
        for x in s["inputs"]:
            x.requires_grad_(True)
    return s


# ------------------------------------------------------------------ one pass
def _forward(s):
    c, kind = s["case"], s["case"]["kind"]
    if kind == "attention":
        return ops.attention(s["q"], s["k"], s["v"], causal=True, window=c["window"] or None, sinks=s["sinks"],
                             segments=s["segments"])
    if kind == "linear":
        return ops.linear(s["x"], s["w"], fmt=c["fmt"])
    if kind == "moe":
        return ops.moe_experts(s["x"], s["w_gu"], s["w_down"], s["weights"], s["experts"], act=c["act"],
                               limit=c["limit"] or None, up_offset=c["up_offset"], fmt=c["fmt"])
    if kind == "head":
        loss, count = ops.cross_entropy_head(s["x"], s["w"], s["targets"], s["mask"])
        return loss / count
    if kind == "rmsnorm":
        return ops.rmsnorm(s["x"], s["w"], 1e-6)
    if kind == "rope":
        return ops.rmsnorm_rope(s["x"], s["w"], s["cos"], s["sin"], 1e-6)
    ctx = s["model"](s["ids"], training=True)
    head = ctx.heads[0]
    loss, count = ops.cross_entropy_head(head.hidden.reshape(-1, c["d"]), head.weight, s["targets"])
    return loss / count


def run(state):
    if not state["case"].get("train", True):
        with torch.no_grad():
            return [_forward(state)]
    y = _forward(state)
    return [y.detach(), *torch.autograd.grad(y, state["inputs"], state.get("dy"))]


# ------------------------------------------------------------------ what a pass cannot do without
def work(case):
    kind = case["kind"]
    train = case.get("train", True)
    if kind == "attention":
        b, t, h, g, d = (case[n] for n in ("b", "t", "h", "g", "d"))
        docs = max(1, case["docs"])
        seen = t / docs                                    # keys a query may see on average, twice over
        pairs = t * seen / 2
        if case["window"]:
            pairs = min(pairs, t * case["window"])
        q, kv = 2 * b * t * h * d, 2 * b * t * g * d       # bytes
        return {"bytes": 2 * q + 2 * kv + (2 * q + 2 * kv if train else 0),
                "flops": 2 * b * h * pairs * d * (7 if train else 2)}
    if kind == "linear":
        m, k, n = case["m"], case["k"], case["n"]
        one = 2 * (m * k + n * k + m * n)
        return {"bytes": one * (2 if train else 1), "flops": 2 * m * n * k * (3 if train else 1)}
    if kind == "moe":
        t, d, f, e, k = (case[n] for n in ("t", "d", "f", "e", "k"))
        one = 2 * (3 * min(e, t * k) * f * d + 2 * t * d) + 12 * t * k
        return {"bytes": one * (2 if train else 1), "flops": 2 * t * k * 3 * f * d * (3 if train else 1)}
    if kind == "head":
        t, d, v = case["t"], case["d"], case["v"]
        return {"bytes": 2 * 2 * (t * d + v * d), "flops": 3 * 2 * t * d * v}
    if kind == "rmsnorm":
        t, d = case["t"], case["d"]
        return {"bytes": 8 * t * d, "flops": 12 * t * d}
    if kind == "rope":
        n = case["b"] * case["t"] * case["h"] * case["d"]
        return {"bytes": 8 * n + 4 * case["b"] * case["t"] * case["d"], "flops": 20 * n}
    tokens, d, f, v = case["b"] * case["t"], case["d"], case["f"], case["v"]
    block = 1536 * d + 1024 * d + 3 * f * d
    weights = case["blocks"] * block + v * d
    return {"bytes": 2 * 2 * (weights + v * d),
            "flops": 6 * tokens * weights + case["blocks"] * 7 * case["b"] * 8 * case["t"] ** 2 * 128}


def tolerance(case):
    """Against the library path of the same ops (other kernels, sums in another order) bf16 outputs
    differ by up to 0.005, the model's gradients by up to 0.022."""
    kind = case["kind"]
    if kind == "model":
        return {"rel": 0.03, "max": 0.9}   # bf16 roundings travel through two blocks and back
    if case.get("fmt") == "mxfp8" and kind == "moe":
        # a value next to a rounding boundary of E4M3 (three mantissa bits) may take either code
        return {"rel": 0.02, "max": 0.8}
    return {"rel": 0.01, "max": 0.4}


# ------------------------------------------------------------------ the same in 64 bits
def _rms64(x, w, eps=1e-6):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * w


def _rope64(x, cos, sin):
    a, b = x.chunk(2, -1)
    c, s = cos.double().unsqueeze(-2), sin.double().unsqueeze(-2)
    return torch.cat((a * c - b * s, a * s + b * c), -1)


def _attend64(q, k, v, window=0, sinks=None, segments=None):
    """One batch row, a query head at a time: q [t, h, d], k and v [t, g, d]."""
    t, h, d = q.shape
    per = h // k.shape[1]
    i = torch.arange(t, device=q.device)
    hidden = i[None, :] > i[:, None]
    if window:
        hidden |= i[None, :] <= i[:, None] - window
    if segments is not None:
        hidden |= segments[None, :] != segments[:, None]
    outs = []
    for j in range(h):
        s = (q[:, j] @ k[:, j // per].t()) * d ** -0.5
        s = s.masked_fill(hidden, float("-inf"))
        if sinks is not None:
            s = torch.cat((s, sinks[j].expand(t, 1)), -1)
        outs.append(torch.softmax(s, -1)[:, :t] @ v[:, j // per])
    return torch.stack(outs, 1)


def _exact_attention(s):
    """Heads are independent of one another: their graphs are walked one group at a time."""
    c = s["case"]
    per = c["h"] // c["g"]
    wide = {n: s[n].detach().double() for n in ("q", "k", "v", "dy")}
    out = torch.empty_like(wide["q"])
    grads = {n: torch.zeros_like(wide[n]) for n in ("q", "k", "v")}
    sinks = s["sinks"].detach().double() if s["sinks"] is not None else None
    dsinks = torch.zeros_like(sinks) if sinks is not None else None
    for b in range(c["b"]):
        seg = s["segments"][b] if s["segments"] is not None else None
        for h in range(c["h"]):
            g = h // per
            q = wide["q"][b, :, h:h + 1].clone().requires_grad_(True)
            k = wide["k"][b, :, g:g + 1].clone().requires_grad_(True)
            v = wide["v"][b, :, g:g + 1].clone().requires_grad_(True)
            sk = sinks[h:h + 1].clone().requires_grad_(True) if sinks is not None else None
            with torch.enable_grad():
                y = _attend64(q, k, v, c["window"], sk, seg)
            out[b, :, h:h + 1] = y.detach()
            if c["train"]:
                got = torch.autograd.grad(y, [q, k, v] + ([sk] if sk is not None else []), wide["dy"][b, :, h:h + 1])
                grads["q"][b, :, h:h + 1] = got[0]
                grads["k"][b, :, g:g + 1] += got[1]
                grads["v"][b, :, g:g + 1] += got[2]
                if sk is not None:
                    dsinks[h:h + 1] += got[3]
    if not c["train"]:
        return [out]
    return [out, grads["q"], grads["k"], grads["v"]] + ([dsinks] if dsinks is not None else [])


def _exact_moe(s):
    c = s["case"]
    x, wts, dy = s["x"].detach().double(), s["weights"].detach().double(), s["dy"].double()
    f, train = c["f"], c["train"]
    out, dx, dwts = torch.zeros_like(x), torch.zeros_like(x), torch.zeros_like(wts)
    dgu, ddown = torch.zeros_like(s["w_gu"], dtype=torch.float32), torch.zeros_like(s["w_down"], dtype=torch.float32)
    for e in range(c["e"]):
        tok, pick = (s["experts"] == e).nonzero(as_tuple=True)
        if tok.numel() == 0:
            continue
        w1 = s["w_gu"][e].detach().double().requires_grad_(train)
        w2 = s["w_down"][e].detach().double().requires_grad_(train)
        xe, we = x[tok].requires_grad_(train), wts[tok, pick].requires_grad_(train)
        with torch.enable_grad():
            h = xe @ w1.t()
            gate, up = h[:, :f], h[:, f:]
            if c["limit"]:
                gate, up = gate.clamp(max=c["limit"]), up.clamp(-c["limit"], c["limit"])
            act = F.silu(gate) if c["act"] == "swish" else gate * torch.sigmoid(1.702 * gate)
            y = (act * (up + c["up_offset"])) @ w2.t() * we[:, None]
        out.index_add_(0, tok, y.detach())
        if train:
            gx, g1, g2, gw = torch.autograd.grad(y, [xe, w1, w2, we], dy[tok])
            dx.index_add_(0, tok, gx)
            dwts[tok, pick] = gw
            dgu[e], ddown[e] = g1.float(), g2.float()
    return [out, dx, dgu, ddown, dwts] if train else [out]


def _exact_head(x, w, targets, mask, chunk=512):
    """Mean loss and its gradients, a chunk of tokens at a time."""
    x, w = x.detach().double(), w.detach().double()
    keep = torch.ones(x.shape[0], device=x.device, dtype=torch.float64) if mask is None else mask.double()
    n = keep.sum()
    loss, dx, dw = x.new_zeros(()), torch.empty_like(x), torch.zeros_like(w)
    for a in range(0, x.shape[0], chunk):
        z = x[a:a + chunk] @ w.t()
        logz = torch.logsumexp(z, -1)
        t = targets[a:a + chunk].long()[:, None]
        loss += ((logz - z.gather(1, t)[:, 0]) * keep[a:a + chunk]).sum()
        z = torch.exp(z - logz[:, None])
        z.scatter_add_(1, t, -torch.ones_like(t, dtype=z.dtype))
        z *= (keep[a:a + chunk] / n)[:, None]
        dx[a:a + chunk] = z @ w
        dw += z.t() @ x[a:a + chunk]
    return loss / n, dx, dw


def _exact_model(s):
    c = s["case"]
    p = {n: x.detach().double().requires_grad_(True) for n, x in s["model"].named_parameters()}
    names = list(p)
    cos, sin = _rope_tables(c["b"], c["t"], 128)
    b, t = c["b"], c["t"]
    with torch.enable_grad():
        x = p["graph.items.0.tokens.embedding"][s["ids"]]
        for i in range(c["blocks"]):
            a = f"graph.items.1.items.{i}.items.0.body.items."
            m = f"graph.items.1.items.{i}.items.1.body.items."
            q, k, v = (_rms64(x, p[a + "0.scale"]) @ p[a + "1.qkv.weight"].t()).split((1024, 256, 256), -1)
            q = _rope64(_rms64(q.view(b, t, 8, 128), p[a + "1.q_norm.scale"]), cos, sin)
            k = _rope64(_rms64(k.view(b, t, 2, 128), p[a + "1.k_norm.scale"]), cos, sin)
            o = torch.stack([_attend64(q[r], k[r], v.view(b, t, 2, 128)[r]) for r in range(b)])
            x = x + o.reshape(b, t, 1024) @ p[a + "1.o.weight"].t()
            gate, up = (_rms64(x, p[m + "0.scale"]) @ p[m + "1.gate_up.weight"].t()).chunk(2, -1)
            x = x + (F.silu(gate) * up) @ p[m + "1.down.weight"].t()
        x = _rms64(x, p["graph.items.2.scale"])
        loss = F.cross_entropy(x.reshape(b * t, -1) @ p["graph.items.3.proj.weight"].t(), s["targets"])
    return [loss.detach(), *torch.autograd.grad(loss, [p[n] for n in names])]


def exact(case, seed):
    s = prepare(case, seed)
    kind = case["kind"]
    if kind == "attention":
        return _exact_attention(s)
    if kind == "moe":
        return _exact_moe(s)
    if kind == "head":
        return list(_exact_head(s["x"], s["w"], s["targets"], s["mask"]))
    if kind == "model":
        return _exact_model(s)
    wide = [x.detach().double().requires_grad_(True) for x in s["inputs"]]
    with torch.enable_grad():
        if kind == "linear":
            y = wide[0] @ wide[1].t()
        elif kind == "rmsnorm":
            y = _rms64(wide[0], wide[1])
        else:
            y = _rope64(_rms64(wide[0], wide[1]), s["cos"], s["sin"])
    if not case.get("train", True):
        return [y.detach()]
    return [y.detach(), *torch.autograd.grad(y, wide, s["dy"].double())]
