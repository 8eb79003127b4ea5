"""The work that a user of this framework has it do, as cases that can be timed and compared.

A window of a node is inner steps (blocks of the decoder forward and backward, the head with its loss, AdamW),
then the compression of the window's pseudo-gradient, the exchange, and the outer step over the peers' payloads;
a validator adds forward passes, and a node that trains with Muon orthogonalises its weight gradients.  Each case
runs one of these through the entry point that the model, the engine or the optimizer uses for it.

``listed`` holds the cases, ``draw`` gives further ones of the same ranges, ``prepare`` makes what a program has in
hand before the call, ``run`` is one pass, ``work`` is what a pass cannot do without, ``tolerance`` how far two
correct implementations may be apart, ``exact`` the same outputs in 64 bits from plain torch."""

from __future__ import annotations

import math

import torch

from templar_b200.models.llama import ModelArgs, build_model
from templar_b200.muon import newton_schulz
from templar_b200.ops import functional as OF
from templar_b200.parallel.window_engine import EngineConfig, WindowEngine
from templar_b200.utils.synthetic import synthetic_payload

DEV = "cuda"
EPS = 1e-5


# ------------------------------------------------------------------------------------------ cases
def listed():
    return [
        # the attention part of a 1B block on the benchmark's micro-batch of 8 x 2048 tokens, forward and backward
        {"name": "attention_1b", "op": "attention", "batch": 8, "seq": 2048, "dim": 2048, "heads": 16, "kv": 16},
        # the same part of an 8B block (grouped queries) on one sequence of 1024 tokens: a short micro-batch of a large model
        {"name": "attention_8b", "op": "attention", "batch": 1, "seq": 1024, "dim": 4096, "heads": 32, "kv": 8},
        # a block of the 150M model, whose heads are 64 wide, on 8 x 1024 tokens
        {"name": "attention_150m", "op": "attention", "batch": 8, "seq": 1024, "dim": 768, "heads": 12, "kv": 12},
        # the feed-forward part of a 1B block on the same micro-batch, forward and backward
        {"name": "ffn_1b", "op": "ffn", "tokens": 16384, "dim": 2048, "hidden": 8192},
        # the feed-forward part of a 150M block on one sequence of 2048 tokens
        {"name": "ffn_150m", "op": "ffn", "tokens": 2048, "dim": 768, "hidden": 3072},
        # residual add and norm at the 8B width, forward and backward, two sequences of 2048 tokens
        {"name": "norm_8b", "op": "norm", "tokens": 4096, "dim": 4096},
        # the smallest call: residual add and norm of the 150M model on two sequences of 256 tokens
        {"name": "norm_150m", "op": "norm", "tokens": 512, "dim": 768},
        # output projection, loss and their backward at the 1B width and vocabulary, four sequences of 2048 tokens
        {"name": "head_1b", "op": "head", "tokens": 8192, "dim": 2048, "vocab": 32000},
        # compression of a window's pseudo-gradient with 8-bit codes: the 1B widths with 4 of the 16 blocks
        {"name": "compress_1b", "op": "compress", "dim": 2048, "hidden": 8192, "heads": 16, "layers": 4, "vocab": 32000, "topk": 32, "quantize": True},
        # the outer step over eight peers' payloads on the same parameters
        {"name": "outer_1b", "op": "outer", "dim": 2048, "hidden": 8192, "heads": 16, "layers": 4, "vocab": 32000, "topk": 32, "peers": 8},
        # Muon's orthogonalisation of the gradient of a 1B gate projection
        {"name": "orthogonalise_1b", "op": "orthogonalise", "rows": 8192, "cols": 2048},
        # a validator's forward pass of the whole 150M model on its sample of 8 x 2048 tokens, logits out
        {"name": "logits_150m", "op": "logits", "batch": 8, "seq": 2048, "dim": 768, "hidden": 3072, "heads": 12, "layers": 12, "vocab": 32000},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# (dim, hidden, heads, kv heads): the widths of the model presets, and two generic ones between them
_WIDTHS = [(768, 3072, 12, 12), (1024, 2816, 8, 8), (1536, 4096, 12, 4), (2048, 8192, 16, 16), (4096, 14336, 32, 8)]


def _seq(rng, most):
    """Sequence lengths: mostly multiples of 128 as a packed data loader cuts them, one in four odd (a text as it comes)."""
    s = _log(rng, 128, most)
    return s if rng.random() < 0.25 else max(128, s // 128 * 128)


def draw(rng):
    op = rng.choice(["attention", "attention", "ffn", "ffn", "norm", "norm", "head", "compress", "outer", "orthogonalise", "logits"])
    if op == "attention":
        dim, _, heads, kv = rng.choice(_WIDTHS)
        seq = _seq(rng, 2048)
        most = min(8, 16384 * 2048 // (dim * seq * max(1, dim // 2048)))
        return {"op": op, "batch": rng.randint(1, max(1, most)), "seq": seq, "dim": dim, "heads": heads, "kv": kv}
    if op == "ffn":
        dim, hidden, _, _ = rng.choice(_WIDTHS)
        return {"op": op, "tokens": _log(rng, 256, min(16384, 16384 * 2048 * 8192 // (dim * hidden))), "dim": dim, "hidden": hidden}
    if op == "norm":
        return {"op": op, "tokens": _log(rng, 256, 16384), "dim": rng.choice([768, 1024, 1536, 2048, 4096, 8192])}
    if op == "head":
        return {"op": op, "tokens": _log(rng, 256, 8192), "dim": rng.choice([768, 1024, 1536, 2048]), "vocab": 32000}
    if op in ("compress", "outer"):
        dim, hidden, heads, _ = rng.choice(_WIDTHS[:4])
        c = {"op": op, "dim": dim, "hidden": hidden, "heads": heads, "layers": rng.randint(1, 4), "vocab": rng.choice([2048, 8064, 32000]),
             "topk": rng.choice([16, 32, 64])}
        return dict(c, quantize=rng.random() < 0.75) if op == "compress" else dict(c, peers=rng.randint(2, 8))
    if op == "orthogonalise":
        dim, hidden, _, _ = rng.choice(_WIDTHS[:4])
        rows, cols = rng.choice([(hidden, dim), (dim, hidden), (dim, dim // 2)])
        return {"op": op, "rows": rows, "cols": cols}
    dim, hidden, heads, _ = rng.choice(_WIDTHS[:2])
    return {"op": op, "batch": rng.randint(1, 8), "seq": _seq(rng, 2048), "dim": dim, "hidden": hidden, "heads": heads,
            "layers": rng.randint(2, 12), "vocab": 32000}


# ------------------------------------------------------------------------------------------ inputs
class _Gen:
    def __init__(self, seed):
        self.g = torch.Generator(device=DEV).manual_seed(int(seed))

    def normal(self, *shape, std=1.0, dtype=torch.bfloat16):
        return torch.randn(*shape, generator=self.g, device=DEV).mul_(std).to(dtype)

    def weight(self, *shape, std=0.02):
        return self.normal(*shape, std=std).requires_grad_()

    def tokens(self, vocab, *shape):
        return torch.randint(0, vocab, shape, generator=self.g, device=DEV)


def _main_grad(w):
    """Weight gradients accumulate in fp32 buffers, as under the engine's flat store."""
    return torch.zeros(w.shape, dtype=torch.float32, device=DEV)


def _engine(c, seed, **cfg):
    args = ModelArgs(dim=c["dim"], n_layers=c["layers"], n_heads=c["heads"], vocab_size=c["vocab"], intermediate_size=c["hidden"])
    model = build_model(args, device=DEV, seed=int(seed))            # fp32 initial values; the engine keeps the bf16 copy
    return model, WindowEngine(model, EngineConfig(**cfg), device=DEV)


@torch.no_grad()
def _window_state(eng, g):
    """A window that is about to close: weights moved by the inner steps, and an error feedback from earlier windows."""
    eng.snapshot()
    eng.store.master_shard.add_(g.normal(eng.store.master_shard.numel(), std=1e-3, dtype=torch.float32))
    eng.ef.copy_(g.normal(eng.ef.numel(), std=2e-3, dtype=torch.float32))


def prepare(case, seed):
    c, g = case, _Gen(seed)
    op = c["op"]
    s = {"case": c}
    if op == "attention":
        B, S, D, H, KV = c["batch"], c["seq"], c["dim"], c["heads"], c["kv"]
        hd = D // H
        s["x"] = g.normal(B, S, D).requires_grad_()
        # projections wide enough that scores spread as in a trained model: entropy well below the uniform one
        s["wqkv"] = g.weight((H + 2 * KV) * hd, D, std=1.2 / math.sqrt(D))
        s["wo"] = g.weight(D, H * hd)
        s["dy"] = g.normal(B, S, D, std=1e-3)
        s["cos"], s["sin"] = OF.rope_tables(S, hd, 10000.0, DEV)
        s["mg_qkv"], s["mg_o"] = _main_grad(s["wqkv"]), _main_grad(s["wo"])
    elif op == "ffn":
        T, D, Fd = c["tokens"], c["dim"], c["hidden"]
        s["x"] = g.normal(T, D).requires_grad_()
        s["w13"], s["w2"] = g.weight(2 * Fd, D), g.weight(D, Fd)
        s["dy"] = g.normal(T, D, std=1e-3)
        s["mg13"], s["mg2"] = _main_grad(s["w13"]), _main_grad(s["w2"])
    elif op == "norm":
        T, D = c["tokens"], c["dim"]
        s["res"], s["delta"] = g.normal(T, D, std=2.0).requires_grad_(), g.normal(T, D).requires_grad_()
        s["w"] = (1 + 0.1 * g.normal(D, dtype=torch.float32)).to(torch.bfloat16).requires_grad_()
        s["dh"], s["dy"] = g.normal(T, D, std=1e-3), g.normal(T, D, std=1e-3)
        s["mg"] = _main_grad(s["w"])
    elif op == "head":
        T, D, V = c["tokens"], c["dim"], c["vocab"]
        s["x"] = g.normal(T, D).requires_grad_()
        s["w"] = g.weight(V, D, std=D ** -0.5)
        s["labels"] = g.tokens(V, T)
        s["labels"][::17] = -100                      # padding positions carry no label
        s["mg"] = _main_grad(s["w"])
    elif op == "compress":
        s["model"], s["eng"] = _engine(c, seed, topk=c["topk"], max_peers=1, quantize=c["quantize"])
        _window_state(s["eng"], g)
    elif op == "outer":
        s["model"], s["eng"] = _engine(c, seed, topk=c["topk"], max_peers=c["peers"])
        _window_state(s["eng"], g)
        for j in range(c["peers"]):
            s["eng"].load_peer_payload(j, synthetic_payload(s["eng"].layout, int(seed) * 64 + j, device=DEV, scale=1e-3 * (1 + 0.1 * j)))
    elif op == "orthogonalise":
        s["g"] = g.normal(c["rows"], c["cols"], std=1e-3)
    else:
        s["model"], s["eng"] = _engine(c, seed)
        s["tokens"] = g.tokens(c["vocab"], c["batch"], c["seq"])
    return s


# ------------------------------------------------------------------------------------------ one pass
def run(s):
    c = s["case"]
    op = c["op"]
    if op == "attention":
        y = OF.attention_block(s["x"], s["wqkv"], s["wo"], s["cos"], s["sin"], c["heads"], c["kv"], c["dim"] // c["heads"], s["mg_qkv"], s["mg_o"])
        (dx,) = torch.autograd.grad(y, (s["x"],), s["dy"])
        return {"y": y.detach(), "dx": dx, "dwqkv": s["mg_qkv"], "dwo": s["mg_o"]}
    if op == "ffn":
        y = OF.feed_forward(s["x"], s["w13"], s["w2"], s["mg13"], s["mg2"])
        (dx,) = torch.autograd.grad(y, (s["x"],), s["dy"])
        return {"y": y.detach(), "dx": dx, "dw13": s["mg13"], "dw2": s["mg2"]}
    if op == "norm":
        h, y = OF.add_rmsnorm(s["res"], s["delta"], s["w"], EPS, s["mg"])
        dres, ddelta = torch.autograd.grad((h, y), (s["res"], s["delta"]), (s["dh"], s["dy"]))
        return {"h": h.detach(), "y": y.detach(), "dres": dres, "ddelta": ddelta, "dw": s["mg"]}
    if op == "head":
        loss = OF.cross_entropy(OF.linear(s["x"], s["w"], s["mg"]), s["labels"])
        (dx,) = torch.autograd.grad(loss, (s["x"],))
        return {"loss": loss.detach(), "dx": dx, "dw": s["mg"]}
    if op == "compress":
        eng = s["eng"]
        eng.compress()
        return {"idx": eng.own_idx, "val": eng.own_val, "ef": eng.ef}
    if op == "outer":
        eng = s["eng"]
        eng.outer_step(c["peers"], include_own=False)
        return {"master": eng.store.master_shard, "weights": eng.store.compute}
    if op == "orthogonalise":
        return newton_schulz(s["g"])
    with torch.no_grad():
        return s["model"](s["tokens"])


# ------------------------------------------------------------------------------------------ work and tolerance
def _n_params(c):
    d, f, v, n = c["dim"], c["hidden"], c["vocab"], c["layers"]
    return n * (4 * d * d + 3 * d * f + 2 * d) + 2 * v * d + d


def work(case):
    c = case
    op = c["op"]
    if op == "attention":
        B, S, D, H, KV = c["batch"], c["seq"], c["dim"], c["heads"], c["kv"]
        T, hd = B * S, D // H
        wide = (H + 2 * KV) * hd
        gemms = 3 * 2.0 * T * D * (wide + H * hd)
        core = 3.5 * 2.0 * B * H * hd * S * (S + 1)            # two products forward, five backward, over the causal half
        return {"bytes": 2.0 * T * D * 4 + (2 + 4 + 4) * D * (wide + H * hd), "flops": gemms + core}
    if op == "ffn":
        T, D, Fd = c["tokens"], c["dim"], c["hidden"]
        return {"bytes": 2.0 * T * D * 4 + (2 + 4 + 4) * 3.0 * D * Fd, "flops": 3 * 2.0 * T * D * 3 * Fd}
    if op == "norm":
        T, D = c["tokens"], c["dim"]
        return {"bytes": 2.0 * T * D * 7 + 10.0 * D, "flops": 20.0 * T * D}
    if op == "head":
        T, D, V = c["tokens"], c["dim"], c["vocab"]
        return {"bytes": 2.0 * T * D * 2 + 8.0 * T + (2 + 4 + 4) * float(V) * D, "flops": 3 * 2.0 * T * D * V}
    if op == "compress":
        n = _n_params(c)
        return {"bytes": n * (4 * 4 + c["topk"] / 4096 * (1.5 + 4 + (1 if c["quantize"] else 0))), "flops": n * 2.0 * 128 * 2}
    if op == "outer":
        n = _n_params(c)
        return {"bytes": n * (4 + 4 + 2 + c["peers"] * c["topk"] / 4096 * 5.5), "flops": n * 2.0 * 128}
    if op == "orthogonalise":
        m, k = sorted((c["rows"], c["cols"]))
        # X X^T and A A are symmetric: half their products, then the full B X
        return {"bytes": 4.0 * m * k, "flops": 5 * (m * m * k + m * m * m + 2.0 * m * m * k)}
    T, S, D = c["batch"] * c["seq"], c["seq"], c["dim"]
    n = c["layers"] * (4 * D * D + 3 * D * c["hidden"]) + c["vocab"] * D
    return {"bytes": 2.0 * n + 8.0 * T + 2.0 * T * c["vocab"] + 2.0 * T * D, "flops": 2.0 * T * n + c["layers"] * 2.0 * T * (S + 1) * D}


def tolerance(case):
    """About four times what the path differs by from 64 bits (measured at the listed cases and drawn ones), and for the
    error feedback and the master weights, which are 32-bit sums, a little over that."""
    return {"attention": {"rel": 2e-2, "max": 0.3}, "ffn": {"rel": 1e-2, "max": 0.15}, "norm": {"rel": 8e-3, "max": 0.05},
            "head": {"rel": 7e-3, "max": 0.2}, "compress": {"rel": 1.5e-3, "max": 0.5, "differ": 1e-3},
            "outer": {"rel": 5e-4, "max": 1e-2}, "orthogonalise": {"rel": 2e-2, "max": 0.3}, "logits": {"rel": 3e-2, "max": 0.5}}[case["op"]]


# ------------------------------------------------------------------------------------------ the same in 64 bits
def _f64(t):
    return t.detach().double()


def _rotate(x, cos, sin):
    """Pairs (2i, 2i+1) of [..., S, hd] turned by the position's angles."""
    a, b = x[..., 0::2], x[..., 1::2]
    return torch.stack((a * cos - b * sin, a * sin + b * cos), dim=-1).flatten(-2)


def _attend(q, k, v, cos, sin):
    """Causal attention of [H, S, hd] queries on [KV, S, hd] keys and values, one head at a time."""
    H, S, hd = q.shape
    rep = H // k.shape[0]
    hide = torch.ones(S, S, dtype=torch.bool, device=q.device).triu(1)
    q, k = _rotate(q, cos, sin), _rotate(k, cos, sin)
    out = []
    for h in range(H):
        scores = (q[h] @ k[h // rep].t()) / math.sqrt(hd)
        out.append(torch.softmax(scores.masked_fill(hide, -math.inf), dim=-1) @ v[h // rep])
    return torch.stack(out)


def _heads(x, n, hd):
    return x.view(x.shape[0], n, hd).transpose(0, 1)


def _exact_attention(s, c):
    H, KV = c["heads"], c["kv"]
    hd = c["dim"] // H
    wqkv, wo = _f64(s["wqkv"]).requires_grad_(), _f64(s["wo"]).requires_grad_()
    cos, sin = _f64(s["cos"]), _f64(s["sin"])
    ys, dxs = [], []
    for b in range(c["batch"]):
        x = _f64(s["x"][b]).requires_grad_()
        qkv = x @ wqkv.t()
        q, k, v = qkv.split([H * hd, KV * hd, KV * hd], dim=-1)
        q, k, v = _heads(q, H, hd), _heads(k, KV, hd), _heads(v, KV, hd)
        y = _attend(q, k, v, cos, sin).transpose(0, 1).reshape(-1, H * hd) @ wo.t()
        y.backward(_f64(s["dy"][b]))
        ys.append(y.detach())
        dxs.append(x.grad)
    return {"y": torch.stack(ys), "dx": torch.stack(dxs), "dwqkv": wqkv.grad, "dwo": wo.grad}


def _exact_ffn(s, c):
    x, w13, w2 = (_f64(s[k]).requires_grad_() for k in ("x", "w13", "w2"))
    gate, up = (x @ w13.t()).chunk(2, dim=-1)
    y = (gate * torch.sigmoid(gate) * up) @ w2.t()
    y.backward(_f64(s["dy"]))
    return {"y": y.detach(), "dx": x.grad, "dw13": w13.grad, "dw2": w2.grad}


def _exact_norm(s, c):
    res, delta, w = (_f64(s[k]).requires_grad_() for k in ("res", "delta", "w"))
    h = res + delta
    y = h * torch.rsqrt(h.square().mean(-1, keepdim=True) + EPS) * w
    torch.autograd.backward((h, y), (_f64(s["dh"]), _f64(s["dy"])))
    return {"h": h.detach(), "y": y.detach(), "dres": res.grad, "ddelta": delta.grad, "dw": w.grad}


def _exact_head(s, c):
    x, w = _f64(s["x"]).requires_grad_(), _f64(s["w"]).requires_grad_()
    n = (s["labels"] != -100).sum().item()
    total = 0.0
    for lo in range(0, c["tokens"], 2048):
        part = torch.nn.functional.cross_entropy(x[lo: lo + 2048] @ w.t(), s["labels"][lo: lo + 2048], ignore_index=-100, reduction="sum") / n
        part.backward()
        total += part.item()
    return {"loss": torch.tensor(total, dtype=torch.float64, device=DEV), "dx": x.grad, "dw": w.grad}


def _dct_matrix(n):
    k = torch.arange(n, dtype=torch.float64, device=DEV).view(-1, 1)
    f = torch.cos(math.pi * (2 * torch.arange(n, dtype=torch.float64, device=DEV) + 1) * k / (2 * n)) * math.sqrt(2.0 / n)
    f[0] = math.sqrt(1.0 / n)
    return f


def _to_chunks(x, spec):
    """[rows, cols] as [chunks, h, w]."""
    return x.view(spec.rows // spec.h, spec.h, spec.cols // spec.w, spec.w).transpose(1, 2).reshape(-1, spec.h, spec.w)


def _from_chunks(y, spec):
    return y.view(spec.rows // spec.h, spec.cols // spec.w, spec.h, spec.w).transpose(1, 2).reshape(-1)


def _inverse(coef, spec):
    return _dct_matrix(spec.h).t() @ coef.view(-1, spec.h, spec.w) @ _dct_matrix(spec.w)


def _exact_compress(s, c):
    """The error feedback alone: neither the order of a chunk's entries nor the choice between two coefficients that agree
    to the last bits is part of what the call promises."""
    eng, layout = s["eng"], s["eng"].layout
    ef = _f64(eng.ef) * eng.cfg.momentum_decay + (_f64(eng.theta0) - _f64(eng.store.master_shard))
    for spec in layout.specs:
        at = slice(spec.offset, spec.offset + spec.numel)
        chunks = _to_chunks(ef[at].view(spec.rows, spec.cols), spec)
        coef = (_dct_matrix(spec.h) @ chunks @ _dct_matrix(spec.w).t()).view(-1, spec.h * spec.w)
        k = spec.topk(c["topk"])
        idx = torch.topk(coef.abs(), k, dim=-1).indices
        kept = torch.gather(coef, 1, idx)
        if c["quantize"]:
            bins = eng.cfg.quant_bins
            shift = kept.mean()
            off = kept - shift
            step = eng.cfg.quant_range * (off.square().sum() / (off.numel() - 1)).sqrt() / bins
            code = (off / step + bins // 2).round().clamp(0, bins - 1).long()
            table = torch.zeros(bins, dtype=torch.float64, device=DEV).scatter_add_(0, code.view(-1), off.view(-1))
            table /= torch.bincount(code.view(-1), minlength=bins).clamp(min=1)
            kept = table[code] + shift
        sent = torch.zeros_like(coef).scatter_(1, idx, kept)
        ef[at] -= _from_chunks(_inverse(sent, spec), spec)
    return {"idx": None, "val": None, "ef": ef}


def _exact_outer(s, c):
    eng, layout = s["eng"], s["eng"].layout
    master = _f64(eng.theta0)
    for spec in layout.specs:
        k, n = spec.topk(c["topk"]), spec.h * spec.w
        vals, places = [], []
        for j in range(c["peers"]):
            idx, val = eng.peer_idx[j], eng.peer_val[j]
            vo, io = layout.val_off[spec.name], layout.idx_off[spec.name]
            vals.append(_f64(val[vo: vo + spec.n_chunks * k]).view(-1, k))
            three = idx[io: io + spec.n_chunks * k // 2 * 3].view(-1, 3).long()
            places.append(torch.stack((three[:, 0] | (three[:, 1] & 15) << 8, three[:, 1] >> 4 | three[:, 2] << 4), dim=1).view(-1, k))
        norms = torch.stack([v.norm() for v in vals])
        scale = (norms.median() / (norms + 1e-8)).clamp(max=1.0)
        place = torch.cat(places, dim=1)
        total = torch.zeros(spec.n_chunks, n, dtype=torch.float64, device=DEV)
        count = torch.zeros_like(total)
        total.scatter_add_(1, place, torch.cat([v * f for v, f in zip(vals, scale)], dim=1))
        count.scatter_add_(1, place, torch.ones_like(place, dtype=torch.float64))
        grad = _from_chunks(_inverse(total / count.clamp(min=1), spec), spec)
        master[spec.offset: spec.offset + spec.numel] -= eng.cfg.outer_lr * grad
    return {"master": master, "weights": master.clone()}


_NS = [(4.0848, -6.8946, 2.9270), (3.9505, -6.3029, 2.6377), (3.7418, -5.5913, 2.3037), (2.8769, -3.1427, 1.2046), (2.8366, -3.0525, 1.2012)]


def _exact_orthogonalise(s, c):
    x = _f64(s["g"])
    turn = x.shape[0] > x.shape[1]
    x = x.t() if turn else x
    x = x / (x.norm() + 1e-7)
    for a, b, d in _NS:
        m = x @ x.t()
        x = a * x + (b * m + d * m @ m) @ x
    return x.t() if turn else x


@torch.no_grad()
def _exact_logits(s, c):
    model = s["model"]
    H, hd = c["heads"], c["dim"] // c["heads"]
    w = {n: _f64(p) for n, p in model.named_parameters()}
    pos = torch.arange(c["seq"], dtype=torch.float64, device=DEV)
    angle = pos[:, None] * (10000.0 ** (-torch.arange(0, hd, 2, dtype=torch.float64, device=DEV) / hd))
    cos, sin = angle.cos(), angle.sin()

    def norm(h, name):
        return h * torch.rsqrt(h.square().mean(-1, keepdim=True) + EPS) * w[name]

    out = []
    for b in range(c["batch"]):
        h = w["tok_embeddings.weight"][s["tokens"][b]]
        for i in range(c["layers"]):
            p = f"layers.{i}."
            x = norm(h, p + "attention_norm.weight")
            q, k, v = (_heads(x @ w[p + f"attention.{n}.weight"].t(), H, hd) for n in ("wq", "wk", "wv"))
            h = h + _attend(q, k, v, cos, sin).transpose(0, 1).reshape(c["seq"], -1) @ w[p + "attention.wo.weight"].t()
            x = norm(h, p + "ffn_norm.weight")
            gate = x @ w[p + "feed_forward.w1.weight"].t()
            h = h + (gate * torch.sigmoid(gate) * (x @ w[p + "feed_forward.w3.weight"].t())) @ w[p + "feed_forward.w2.weight"].t()
        out.append(norm(h, "norm.weight") @ w["output.weight"].t())
    return torch.stack(out)


def exact(case, seed):
    s = prepare(case, seed)
    return {"attention": _exact_attention, "ffn": _exact_ffn, "norm": _exact_norm, "head": _exact_head, "compress": _exact_compress,
            "outer": _exact_outer, "orthogonalise": _exact_orthogonalise, "logits": _exact_logits}[case["op"]](s, case)
