"""The work that training and evaluation runs of this framework spend their time on, as timed cases.

Each case is one layer, one whole forward pass or one optimizer step, called the way a program calls it, at the
sizes of the repository's configurations (the 1.1 B and 8 B decoders, the small 768-wide decoder of the
sample run, the sparse mixture-of-experts layer) and at sizes between and beyond them.  Activations and weights are bf16, as in
every GPU run; optimizer state is fp32.
"""
from __future__ import annotations

import math

import torch

from lightron_b200.config import ModelArgs
from lightron_b200.models.llama import LightronTransformer, flatten_parameters, init_weights
from lightron_b200.models.moe import MoEFeedForward
from lightron_b200.ops import functional as OF
from lightron_b200.optim import DistributedAdamW

BF16 = torch.bfloat16
EPS = 1e-5
THETA = 10000.0


def listed():
    return [
        # evaluation of one short prompt with the small decoder: 12 layers of tiny kernels, launches count
        dict(name="model_eval_small", kind="model", B=1, S=128, dim=768, layers=12, heads=12, kv=12, vocab=32000),
        # the sample run's attention layer: micro-batch 4 of 128 tokens, forward and backward
        dict(name="attn_layer_small", kind="attn_layer", B=4, S=128, dim=768, heads=12, kv=12),
        # the small decoder's feed-forward over a ragged number of tokens
        dict(name="mlp_small_ragged", kind="mlp", T=1000, dim=768, hidden=2048),
        # residual add + norm of the 1.1 B decoder at its training batch
        dict(name="norm_1b", kind="norm", T=16384, dim=2048),
        # causal attention of the 1.1 B decoder at its training batch (8 x 2048 tokens, grouped heads)
        dict(name="attn_1b_train", kind="attn", B=8, S=2048, heads=32, kv=4, d=64, grad=True),
        # causal attention of the 8 B decoder at its training sequence
        dict(name="attn_8b_train", kind="attn", B=1, S=8192, heads=32, kv=8, d=128, grad=True),
        # evaluation batch of ragged length: forward only
        dict(name="attn_8b_eval_ragged", kind="attn", B=3, S=1531, heads=32, kv=8, d=128, grad=False),
        # feed-forward of the 1.1 B decoder at its training batch
        dict(name="mlp_1b", kind="mlp", T=16384, dim=2048, hidden=5632),
        # LM head and loss of the 1.1 B decoder, half its training batch
        dict(name="head_1b", kind="head", T=8192, dim=2048, vocab=32000),
        # embedding lookup and its gradient; token frequencies fall off as in text (Zipf-Mandelbrot)
        dict(name="embedding_1b", kind="embedding", T=16384, dim=2048, vocab=32000),
        # one optimizer step of the small decoder (134 M parameters, fp32 master and moments)
        dict(name="optimizer_small", kind="optimizer", dim=768, layers=12, heads=12, vocab=32000),
        # a mixture-of-experts layer, 8 experts, 2 per token, all on one GPU
        dict(name="moe_8x", kind="moe", T=4096, dim=2048, hidden=4096, experts=8, topk=2),
    ]


def _log_int(rng, lo, hi, step=1):
    v = math.exp(rng.uniform(math.log(lo), math.log(hi + step)))
    return max(lo, min(hi, int(v) // step * step))


def draw(rng):
    kind = rng.choice(["model", "attn_layer", "mlp", "norm", "attn", "attn", "head", "embedding", "optimizer", "moe"])
    if kind == "norm":
        return dict(kind=kind, T=_log_int(rng, 16, 16384), dim=_log_int(rng, 256, 4096, 8))
    if kind == "attn":
        d = rng.choice([64, 128])
        kv = rng.choice([2, 4, 8])
        heads = kv * rng.choice([1, 4, 8] if kv < 8 else [1, 4])
        S = _log_int(rng, 64, 8192 if d == 128 else 4096)
        return dict(kind=kind, B=rng.randint(1, max(1, min(8, 8192 // S))), S=S, heads=heads, kv=kv, d=d, grad=rng.random() < 0.7)
    if kind == "attn_layer":
        heads, d = rng.choice([(12, 64), (16, 64), (32, 64), (16, 128)])
        kv = rng.choice([4, heads])
        S = _log_int(rng, 64, 2048)
        return dict(kind=kind, B=rng.randint(1, max(1, min(8, 8192 // S))), S=S, dim=heads * d, heads=heads, kv=kv)
    if kind == "mlp":
        dim, hidden = rng.choice([(768, 2048), (1024, 2816), (2048, 5632), (4096, 14336)])
        return dict(kind=kind, T=_log_int(rng, 16, 16384 if dim <= 2048 else 2048), dim=dim, hidden=hidden)
    if kind == "head":
        return dict(kind=kind, T=_log_int(rng, 64, 4096), dim=rng.choice([768, 1024, 2048]), vocab=rng.choice([8192, 32000, 50264]))
    if kind == "embedding":
        return dict(kind=kind, T=_log_int(rng, 64, 16384), dim=rng.choice([768, 1024, 2048, 4096]), vocab=rng.choice([8192, 32000]))
    if kind == "optimizer":
        dim, heads = rng.choice([(256, 4), (512, 8), (768, 12), (1024, 16)])
        return dict(kind=kind, dim=dim, layers=rng.randint(1, 12), heads=heads, vocab=rng.choice([8192, 32000]))
    if kind == "model":
        dim, heads = rng.choice([(768, 12), (1024, 16), (2048, 32)])
        S = _log_int(rng, 32, 1024)
        return dict(kind=kind, B=rng.randint(1, max(1, min(4, 2048 // S))), S=S, dim=dim, layers=rng.randint(2, 12), heads=heads,
                    kv=rng.choice([4, heads]), vocab=rng.choice([8192, 32000]))
    return dict(kind="moe", T=_log_int(rng, 64, 4096), dim=rng.choice([768, 1024, 2048]), hidden=rng.choice([2048, 4096]),
                experts=rng.choice([4, 8]), topk=2)


# ---- inputs ------------------------------------------------------------------------------------


class _Draws:
    """bf16 normal tensors on the GPU from one seeded generator."""

    def __init__(self, seed):
        self.g = torch.Generator(device="cuda").manual_seed(int(seed))

    def __call__(self, *shape, std=1.0):
        return (torch.randn(*shape, generator=self.g, device="cuda", dtype=torch.float32) * std).to(BF16)

    def ints(self, hi, *shape):
        return torch.randint(0, hi, shape, generator=self.g, device="cuda")

    def text_like(self, vocab, n):
        """Ids whose frequency falls off as 1 / (rank + 50): the most frequent one is 0.3 % of 32000."""
        cum = torch.cumsum(1.0 / torch.arange(50, vocab + 50, device="cuda", dtype=torch.float64), 0)
        u = torch.rand(n, generator=self.g, device="cuda", dtype=torch.float64) * cum[-1]
        rank = torch.searchsorted(cum, u).clamp_max(vocab - 1)
        return torch.randperm(vocab, generator=self.g, device="cuda")[rank]


def _leaf(t):
    return t.detach().requires_grad_(True)


def _args(c):
    return ModelArgs(dim=c["dim"], n_layers=c["layers"], n_heads=c["heads"], n_kv_heads=c.get("kv", c["heads"]), vocab_size=c["vocab"],
                     norm_eps=EPS, max_seq_len=max(c.get("S", 128), 16), rope_theta=THETA)


def _rope_tables(S, d, dtype=torch.float32):
    inv = 1.0 / (THETA ** (torch.arange(0, d, 2, device="cuda", dtype=torch.float64) / d))
    ang = torch.outer(torch.arange(S, device="cuda", dtype=torch.float64), inv)
    return ang.cos().to(dtype).contiguous(), ang.sin().to(dtype).contiguous()


def prepare(case, seed):
    c, rnd = dict(case), _Draws(seed)
    kind = c["kind"]
    s = {"case": c}
    if kind == "norm":
        s.update(x=_leaf(rnd(c["T"], c["dim"])), res=_leaf(rnd(c["T"], c["dim"], std=3.0)), w=_leaf(1 + rnd(c["dim"], std=0.1)),
                 dh=rnd(c["T"], c["dim"]), dy=rnd(c["T"], c["dim"]))
    elif kind == "attn":
        B, S, hq, hkv, d = c["B"], c["S"], c["heads"], c["kv"], c["d"]
        s.update(q=rnd(B, S, hq, d), k=rnd(B, S, hkv, d), v=rnd(B, S, hkv, d))
        if c["grad"]:
            s.update(q=_leaf(s["q"]), k=_leaf(s["k"]), v=_leaf(s["v"]), do=rnd(B, S, hq, d))
    elif kind == "attn_layer":
        H, hq, hkv = c["dim"], c["heads"], c["kv"]
        d = H // hq
        wqkv = rnd((hq + 2 * hkv) * d, H, std=H ** -0.5)
        s.update(x=_leaf(rnd(c["B"] * c["S"], H)), wq=_leaf(wqkv[:hq * d]), wk=_leaf(wqkv[hq * d:(hq + hkv) * d]),
                 wv=_leaf(wqkv[(hq + hkv) * d:]), wo=_leaf(rnd(H, hq * d, std=H ** -0.5)), dy=rnd(c["B"] * c["S"], H),
                 rope=_rope_tables(c["S"], d))
    elif kind == "mlp":
        H, I = c["dim"], c["hidden"]
        w13 = rnd(2 * I, H, std=H ** -0.5)
        s.update(x=_leaf(rnd(c["T"], H)), w1=_leaf(w13[:I]), w3=_leaf(w13[I:]), w2=_leaf(rnd(H, I, std=I ** -0.5)), dy=rnd(c["T"], H))
    elif kind == "head":
        s.update(x=_leaf(rnd(c["T"], c["dim"])), w=_leaf(rnd(c["vocab"], c["dim"], std=c["dim"] ** -0.5)), tgt=rnd.ints(c["vocab"], c["T"]))
    elif kind == "embedding":
        s.update(tok=rnd.text_like(c["vocab"], c["T"]), w=_leaf(rnd(c["vocab"], c["dim"], std=0.02)), dy=rnd(c["T"], c["dim"]))
    elif kind == "optimizer":
        model = LightronTransformer(_args(c), dtype=BF16, device="cuda")
        init_weights(model, seed=int(seed) & 0xFFFF)
        opt = DistributedAdamW(model, lr=3e-4, weight_decay=0.01)
        opt.step_count = 10
        opt.flat_grads.copy_(rnd(opt.flat_grads.numel(), std=1e-2))
        opt.exp_avg.normal_(0.0, 3e-3, generator=rnd.g)
        opt.exp_avg_sq.normal_(0.0, 1e-2, generator=rnd.g).square_()
        s.update(model=model, opt=opt)
    elif kind == "model":
        model = LightronTransformer(_args(c), dtype=BF16, device="cuda").eval()
        init_weights(model, seed=int(seed) & 0xFFFF)
        flatten_parameters(model)
        s.update(model=model, tokens=rnd.ints(c["vocab"], c["B"], c["S"]))
    else:
        H, I, E = c["dim"], c["hidden"], c["experts"]
        args = ModelArgs(dim=H, n_layers=1, n_heads=H // 64, vocab_size=256, intermediate_size=I, moe_num_experts=E,
                         moe_topk=c["topk"], moe_layer_freq=1)
        ctx = LightronTransformer(ModelArgs(dim=64, n_layers=0, n_heads=1, vocab_size=64)).ctx
        layer = MoEFeedForward(args, ctx, dtype=BF16, device="cuda")
        flatten_parameters(layer)
        with torch.no_grad():
            for n, p in layer.named_parameters():
                p.copy_(rnd(*p.shape, std=p.shape[1] ** -0.5))
        for p in layer.parameters():
            p.grad = None
        s.update(layer=layer, x=_leaf(rnd(c["T"], H)), dy=rnd(c["T"], H))
    return s


# ---- one pass ------------------------------------------------------------------------------------


def run(s):
    c = s["case"]
    kind = c["kind"]
    if kind == "norm":
        h, y = OF.add_rmsnorm(s["x"], s["res"], s["w"], EPS)
        dx, dres, dw = torch.autograd.grad([h, y], [s["x"], s["res"], s["w"]], [s["dh"], s["dy"]])
        return {"h": h, "y": y, "dx": dx, "dres": dres, "dw": dw}
    if kind == "attn":
        if not c["grad"]:
            with torch.no_grad():
                return {"o": OF.flash_attention(s["q"], s["k"], s["v"], causal=True)}
        o = OF.flash_attention(s["q"], s["k"], s["v"], causal=True)
        dq, dk, dv = torch.autograd.grad(o, [s["q"], s["k"], s["v"]], s["do"])
        return {"o": o, "dq": dq, "dk": dk, "dv": dv}
    if kind == "attn_layer":
        hq, hkv = c["heads"], c["kv"]
        ins = [s["x"], s["wq"], s["wk"], s["wv"], s["wo"]]
        qkv = OF.linear(*ins[:4])
        o = OF.rope_attention_qkv(qkv, *s["rope"], None, c["B"], c["S"], hq, hkv, c["dim"] // hq)
        y = OF.linear(o, s["wo"])
        return dict(zip(("y", "dx", "dwq", "dwk", "dwv", "dwo"), (y, *torch.autograd.grad(y, ins, s["dy"]))))
    if kind == "mlp":
        ins = [s["x"], s["w1"], s["w3"], s["w2"]]
        y = OF.swiglu_mlp(*ins)
        return dict(zip(("y", "dx", "dw1", "dw3", "dw2"), (y, *torch.autograd.grad(y, ins, s["dy"]))))
    if kind == "head":
        loss = OF.cross_entropy(OF.linear(s["x"], s["w"]), s["tgt"], n_valid_total=c["T"])
        dx, dw = torch.autograd.grad(loss, [s["x"], s["w"]])
        return {"loss": loss, "dx": dx, "dw": dw}
    if kind == "embedding":
        e = OF.embedding(s["tok"], s["w"])
        return {"e": e, "dw": torch.autograd.grad(e, s["w"], s["dy"])[0]}
    if kind == "optimizer":
        opt = s["opt"]
        opt.step()
        return {"params": opt.flat_params, "master": opt.master, "exp_avg": opt.exp_avg, "exp_avg_sq": opt.exp_avg_sq}
    if kind == "model":
        with torch.no_grad():
            return {"logits": s["model"](s["tokens"])}
    layer = s["layer"]
    names, ps = zip(*layer.named_parameters())
    y = layer(s["x"])
    grads = torch.autograd.grad([y, layer.last_aux_loss], [s["x"], *ps], [s["dy"], torch.ones_like(layer.last_aux_loss)])
    return {"y": y, "aux": layer.last_aux_loss, "dx": grads[0], **{"d" + n: g for n, g in zip(names, grads[1:])}}


# ---- what a pass cannot do without -----------------------------------------------------------------


def _sizes(c):
    """Parameters of a decoder."""
    return _args(c).num_params()


def work(case):
    c = case
    kind = c["kind"]
    if kind == "norm":
        n = c["T"] * c["dim"]
        return {"bytes": 2 * n * (2 + 2 + 2 + 1), "flops": 0}          # x, res -> h, y; dh, dy -> one gradient for x and res
    if kind in ("attn", "attn_layer"):
        B, S, hq, hkv = c["B"], c["S"], c["heads"], c["kv"]
        d = c["d"] if kind == "attn" else c["dim"] // hq
        grad = kind == "attn_layer" or c["grad"]
        core = 4.0 * B * hq * (S * (S + 1) / 2) * d * (3.5 if grad else 1.0)
        if kind == "attn":
            qkv = B * S * (hq + 2 * hkv) * d
            o = B * S * hq * d
            return {"bytes": 2 * (qkv + o + ((qkv + o) if grad else 0)), "flops": core}
        T, H = B * S, c["dim"]
        w = ((hq + 2 * hkv) * d + hq * d) * H
        return {"bytes": 2 * (4 * T * H + 2 * w), "flops": core + 3 * 2.0 * T * w}
    if kind == "mlp":
        w = 3 * c["dim"] * c["hidden"]
        return {"bytes": 2 * (4 * c["T"] * c["dim"] + 2 * w), "flops": 3 * 2.0 * c["T"] * w}
    if kind == "head":
        w = c["dim"] * c["vocab"]
        return {"bytes": 2 * (2 * c["T"] * c["dim"] + 2 * w), "flops": 3 * 2.0 * c["T"] * w}
    if kind == "embedding":
        n = c["T"] * c["dim"]
        return {"bytes": 8 * c["T"] + 2 * (3 * n + c["vocab"] * c["dim"]), "flops": 0}
    if kind == "optimizer":
        return {"bytes": _sizes(c) * (2 + 12 + 12 + 2), "flops": 0}    # gradient, fp32 state in and out, bf16 parameter out
    if kind == "model":
        n = _sizes(c) - c["vocab"] * c["dim"]
        T = c["B"] * c["S"]
        return {"bytes": 2 * (n + T * c["vocab"]), "flops": 2.0 * T * n + c["layers"] * 2.0 * T * (c["S"] + 1) * c["dim"]}
    w = 3 * c["dim"] * c["hidden"]
    return {"bytes": 2 * (4 * c["T"] * c["dim"] + 2 * c["experts"] * w), "flops": 3 * 2.0 * c["T"] * c["topk"] * w}


# About four times the distance to 64 bits that was measured, rounded; bf16 has 8 significant bits.
_TOLERANCE = {
    "norm": {"rel": 1.2e-2, "max": 0.05},
    "attn": {"rel": 1.6e-2, "max": 0.3},
    "attn_layer": {"rel": 2e-2, "max": 0.3},
    "mlp": {"rel": 1.6e-2, "max": 0.3},
    "head": {"rel": 1.6e-2, "max": 0.3},
    # gradient rows of frequent tokens may be summed in bf16, in any order
    "embedding": {"rel": 3e-2, "max": 0.95},
    "optimizer": {"rel": 1e-4, "max": 1e-2},
    "model": {"rel": 3e-2, "max": 0.3},
    "moe": {"rel": 2e-2, "max": 0.4},
}


def tolerance(case):
    return _TOLERANCE[case["kind"]]


# ---- the same in 64 bits ------------------------------------------------------------------------


def _d(t):
    return t.detach().double()


def _d_leaf(t):
    return _d(t).requires_grad_(True)


def _norm64(h, w):
    return h * torch.rsqrt(h.square().mean(-1, keepdim=True) + EPS) * w


def _rope64(t, S):
    """[B, S, h, d], interleaved pairs."""
    cos, sin = _rope_tables(S, t.shape[-1], torch.float64)
    cos, sin = cos[None, :, None, :], sin[None, :, None, :]
    a, b = t[..., 0::2], t[..., 1::2]
    return torch.stack((a * cos - b * sin, a * sin + b * cos), -1).flatten(-2)


def _attention64(q, k, v, do=None):
    """Causal attention head by head; with ``do`` also the gradients.  [B, S, h, d] in and out."""
    B, S, hq, d = q.shape
    rep = hq // k.shape[2]
    sc = d ** -0.5
    mask = torch.ones(S, S, dtype=torch.bool, device=q.device).triu(1)
    o, dq, dk, dv = torch.empty_like(q), torch.empty_like(q), torch.zeros_like(k), torch.zeros_like(v)
    for b in range(B):
        for h in range(hq):
            kk, vv = k[b, :, h // rep], v[b, :, h // rep]
            p = (q[b, :, h] @ kk.T).mul_(sc).masked_fill_(mask, -math.inf).softmax(-1)
            o[b, :, h] = p @ vv
            if do is not None:
                g = do[b, :, h]
                dv[b, :, h // rep] += p.T @ g
                ds = (g @ vv.T).sub_((g * o[b, :, h]).sum(-1, keepdim=True)).mul_(p).mul_(sc)
                dq[b, :, h] = ds @ kk
                dk[b, :, h // rep] += ds.T @ q[b, :, h]
    return (o, dq, dk, dv) if do is not None else o


class _Attention64(torch.autograd.Function):
    @staticmethod
    def forward(ctx, q, k, v):
        ctx.save_for_backward(q, k, v)
        return _attention64(q, k, v)

    @staticmethod
    def backward(ctx, do):
        return _attention64(*ctx.saved_tensors, do)[1:]


def _attn_layer64(x, wqkv, wo, B, S, hq, hkv):
    d = wo.shape[1] // hq
    q, k, v = (x @ wqkv.T).view(B, S, hq + 2 * hkv, d).split([hq, hkv, hkv], 2)
    return _Attention64.apply(_rope64(q, S), _rope64(k, S), v).reshape(B * S, hq * d) @ wo.T


def _mlp64(x, w1, w3, w2):
    return (torch.nn.functional.silu(x @ w1.T) * (x @ w3.T)) @ w2.T


def exact(case, seed):
    s = prepare(case, seed)
    c = s["case"]
    kind = c["kind"]
    if kind == "norm":
        x, res, w = _d_leaf(s["x"]), _d_leaf(s["res"]), _d_leaf(s["w"])
        h = x + res
        y = _norm64(h, w)
        dx, dres, dw = torch.autograd.grad([h, y], [x, res, w], [_d(s["dh"]), _d(s["dy"])])
        return {"h": h, "y": y, "dx": dx, "dres": dres, "dw": dw}
    if kind == "attn":
        q, k, v = _d(s["q"]), _d(s["k"]), _d(s["v"])
        if not c["grad"]:
            return {"o": _attention64(q, k, v)}
        return dict(zip(("o", "dq", "dk", "dv"), _attention64(q, k, v, _d(s["do"]))))
    if kind == "attn_layer":
        ins = [_d_leaf(s[n]) for n in ("x", "wq", "wk", "wv", "wo")]
        y = _attn_layer64(ins[0], torch.cat(ins[1:4]), ins[4], c["B"], c["S"], c["heads"], c["kv"])
        return dict(zip(("y", "dx", "dwq", "dwk", "dwv", "dwo"), (y, *torch.autograd.grad(y, ins, _d(s["dy"])))))
    if kind == "mlp":
        ins = [_d_leaf(s[n]) for n in ("x", "w1", "w3", "w2")]
        y = _mlp64(*ins)
        return dict(zip(("y", "dx", "dw1", "dw3", "dw2"), (y, *torch.autograd.grad(y, ins, _d(s["dy"])))))
    if kind == "head":
        x, w = _d_leaf(s["x"]), _d_leaf(s["w"])
        loss = torch.nn.functional.cross_entropy(x @ w.T, s["tgt"])
        dx, dw = torch.autograd.grad(loss, [x, w])
        return {"loss": loss, "dx": dx, "dw": dw}
    if kind == "embedding":
        w = _d(s["w"])
        return {"e": w[s["tok"]], "dw": torch.zeros_like(w).index_add_(0, s["tok"], _d(s["dy"]))}
    if kind == "optimizer":
        opt = s["opt"]
        b1, b2 = opt.betas
        t = opt.step_count + 1
        g = _d(opt.flat_grads)
        m = b1 * _d(opt.exp_avg) + (1 - b1) * g
        v = b2 * _d(opt.exp_avg_sq) + (1 - b2) * g * g
        p = _d(opt.master) * (1 - opt.lr * opt.weight_decay) - opt.lr / (1 - b1 ** t) * m / ((v / (1 - b2 ** t)).sqrt() + opt.eps)
        return {"params": p, "master": p, "exp_avg": m, "exp_avg_sq": v}
    if kind == "model":
        sd = {n: _d(p) for n, p in s["model"].named_parameters()}
        with torch.no_grad():
            h = sd["tok_embeddings.weight"][s["tokens"].reshape(-1)]
            for i in range(c["layers"]):
                w = {n[len(f"layers.{i}."):]: p for n, p in sd.items() if n.startswith(f"layers.{i}.")}
                h = h + _attn_layer64(_norm64(h, w["attention_norm.weight"]),
                                      torch.cat([w[f"attention.w{n}.weight"] for n in "qkv"]), w["attention.wo.weight"],
                                      c["B"], c["S"], c["heads"], c["kv"])
                h = h + _mlp64(_norm64(h, w["ffn_norm.weight"]), *(w[f"feed_forward.w{n}.weight"] for n in (1, 3, 2)))
            return {"logits": (_norm64(h, sd["norm.weight"]) @ sd["output.weight"].T).view(c["B"], c["S"], -1)}
    layer, E, k = s["layer"], c["experts"], c["topk"]
    names = [n for n, _ in layer.named_parameters()]
    ps = {n: _d_leaf(p) for n, p in layer.named_parameters()}
    x = _d_leaf(s["x"])
    probs = (x @ ps["gate.weight"].T).softmax(-1)
    wts, idx = probs.topk(k, -1)
    y = torch.zeros_like(x)
    for e in range(E):
        tok, slot = (idx == e).nonzero(as_tuple=True)
        out = _mlp64(x[tok], *(ps[f"experts.{e}.w{n}.weight"] for n in (1, 3, 2)))
        y = y.index_add(0, tok, out * wts[tok, slot].unsqueeze(-1))
    frac = torch.bincount(idx.reshape(-1), minlength=E).double() / (x.shape[0] * k)
    aux = E * (frac * probs.mean(0)).sum()
    grads = torch.autograd.grad([y, aux], [x, *(ps[n] for n in names)], [_d(s["dy"]), torch.ones_like(aux)])
    return {"y": y, "aux": aux, "dx": grads[0], **{"d" + n: g for n, g in zip(names, grads[1:])}}
