"""The work that a training program has this framework do on one GPU, as cases that can be
timed and compared: single operators and blocks of the decoder through :mod:`monarch_b200.ops`,
and whole forward/backward passes through :class:`monarch_b200.models.LlamaEngine`.

Every case is a dict of plain values; ``kind`` says which path it takes:

* ``linear``     forward, input gradient and weight gradient of one linear layer
* ``attention``  causal grouped-query attention on a fused qkv buffer, with or without its
                 backward
* ``norm``       RMSNorm forward and backward (the residual gradient added in the backward)
* ``swiglu``     the gated activation, forward and backward
* ``loss``       final norm, logits, cross-entropy and the three gradients
* ``adamw``      the optimizer on one flat parameter unit
* ``model``      ``LlamaEngine.forward_backward`` on a whole small model, gradients returned
"""
import math

import torch

from monarch_b200 import ops
from monarch_b200.models import LlamaConfig, LlamaEngine, LocalParamStore, ParamLayout

bf16 = torch.bfloat16
EPS = 1e-5


def listed():
    return [
        # smallest calls: the "tiny" preset (d 256) with a ragged handful of tokens; latency
        dict(name="linear_tiny", kind="linear", tokens=200, n_in=256, n_out=768),
        # an ordinary batch that fills no whole number of tiles: the qkv projection of the
        # 1B shape (d 2048, 32+2*8 heads of 64) on 1000 tokens
        dict(name="linear_ragged", kind="linear", tokens=1000, n_in=2048, n_out=3072),
        # the largest linear of the 8B shape that is no vocabulary head: the down projection
        dict(name="linear_8b_down", kind="linear", tokens=8192, n_in=14336, n_out=4096),
        # attention of the 8B shape at its training length
        dict(name="attention_8b", kind="attention", batch=1, seq=8192, heads=32, kv_heads=8,
             hd=128, train=True),
        # attention of the 1B shape: heads of 64, micro-batch of 2
        dict(name="attention_1b", kind="attention", batch=2, seq=4096, heads=32, kv_heads=8,
             hd=64, train=True),
        # short multi-head attention (the 13B shape's heads on one of four tensor-parallel
        # ranks): an odd number of row blocks, few blocks in all
        dict(name="attention_short", kind="attention", batch=2, seq=640, heads=10, kv_heads=10,
             hd=128, train=True),
        # the norm between the blocks of the 8B shape
        dict(name="norm_8b", kind="norm", tokens=8192, d=4096),
        # the gated activation of the 8B shape
        dict(name="swiglu_8b", kind="swiglu", tokens=8192, ffn=14336),
        # the head of the 1B shape: vocabulary 128256 on half a micro-batch
        dict(name="loss_1b", kind="loss", tokens=4096, d=2048, vocab=128256),
        # the optimizer on one decoder layer of the 1B shape (60.8 M parameters)
        dict(name="adamw_layer", kind="adamw", n=60821504, grad="bf16"),
        # a whole step of the "tiny" preset: launches and host work
        dict(name="model_tiny", kind="model", batch=2, seq=128, vocab=512, d=256, layers=2,
             heads=4, kv_heads=2, ffn=512),
        # one decoder layer of the 8B shape (recomputed in the backward as in training)
        # between a small vocabulary's embedding and head
        dict(name="model_8b_layer", kind="model", batch=1, seq=4096, vocab=2048, d=4096, layers=1,
             heads=32, kv_heads=8, ffn=14336),
    ]


def _log(rng, lo, hi, mult=1):
    """A multiple of ``mult`` in [lo, hi], spread over the logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return int(min(hi, max(lo, round(v / mult) * mult)))


def draw(rng):
    kind = rng.choice(["linear", "linear", "attention", "attention", "norm", "swiglu", "loss",
                       "adamw", "model"])
    if kind == "linear":
        while True:
            c = dict(kind=kind, tokens=_log(rng, 1, 8192), n_in=_log(rng, 256, 14336, 8),
                     n_out=_log(rng, 256, 28672, 8))
            if c["tokens"] * c["n_in"] * c["n_out"] <= 8192 * 4096 * 14336:
                return c
    if kind == "attention":
        while True:
            kv = rng.choice([1, 2, 4, 5, 8, 10])
            c = dict(kind=kind, batch=rng.choice([1, 1, 2, 3]), seq=_log(rng, 128, 8192, 128),
                     heads=kv * rng.choice([1, 2, 3, 4, 8]), kv_heads=kv,
                     hd=rng.choice([64, 128]), train=rng.random() < 0.75)
            if c["heads"] <= 40 and \
                    c["batch"] * c["heads"] * c["hd"] * c["seq"] ** 2 <= 32 * 128 * 8192 ** 2:
                return c
    if kind == "norm":
        return dict(kind=kind, tokens=_log(rng, 1, 8192), d=_log(rng, 256, 8192, 8))
    if kind == "swiglu":
        return dict(kind=kind, tokens=_log(rng, 1, 8192), ffn=_log(rng, 512, 14336, 8))
    if kind == "loss":
        while True:
            c = dict(kind=kind, tokens=_log(rng, 16, 8192), d=_log(rng, 256, 4096, 8),
                     vocab=_log(rng, 512, 128256, 8))
            if c["tokens"] * c["d"] * c["vocab"] <= 4096 * 2048 * 128256:
                return c
    if kind == "adamw":
        return dict(kind=kind, n=_log(rng, 8192, 60821504), grad=rng.choice(["bf16", "fp32"]))
    hd = rng.choice([64, 128])
    kv = rng.choice([1, 2, 4])
    heads = kv * rng.choice([1, 2, 4])
    return dict(kind=kind, batch=rng.choice([1, 2]), seq=_log(rng, 128, 2048, 128),
                vocab=_log(rng, 512, 8192, 8), d=heads * hd, layers=rng.choice([1, 2]),
                heads=heads, kv_heads=kv, ffn=_log(rng, 512, 4096, 8))


# ------------------------------------------------------------------------------- inputs
def _rand(g, *shape, std=1.0, dtype=bf16):
    t = torch.empty(*shape, dtype=torch.float32, device="cuda")
    return t.normal_(0.0, std, generator=g).to(dtype)


def _ids(g, n, hi):
    return torch.randint(0, hi, (n,), generator=g, device="cuda")


def prepare(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    k = case["kind"]
    s = {"case": case}
    if k == "linear":
        T, I, O = case["tokens"], case["n_in"], case["n_out"]
        s.update(x=_rand(g, T, I), w=_rand(g, O, I, std=0.02), dy=_rand(g, T, O),
                 dw=torch.zeros(O, I, dtype=bf16, device="cuda"))
    elif k == "attention":
        B, S, H, HK, D = (case[n] for n in ("batch", "seq", "heads", "kv_heads", "hd"))
        s.update(qkv=_rand(g, B * S, (H + 2 * HK) * D), do=_rand(g, B * S, H * D))
    elif k == "norm":
        T, d = case["tokens"], case["d"]
        s.update(x=_rand(g, T, d), w=(1 + _rand(g, d, std=0.1, dtype=torch.float32)).to(bf16),
                 dy=_rand(g, T, d), dres=_rand(g, T, d),
                 dw=torch.zeros(d, dtype=bf16, device="cuda"))
    elif k == "swiglu":
        T, F = case["tokens"], case["ffn"]
        s.update(gu=_rand(g, T, 2 * F), dh=_rand(g, T, F))
    elif k == "loss":
        T, d, V = case["tokens"], case["d"], case["vocab"]
        s.update(x=_rand(g, T, d), w=(1 + _rand(g, d, std=0.1, dtype=torch.float32)).to(bf16),
                 head=_rand(g, V, d, std=0.02), targets=_ids(g, T, V),
                 dw=torch.zeros(d, dtype=bf16, device="cuda"),
                 dhead=torch.zeros(V, d, dtype=bf16, device="cuda"))
    elif k == "adamw":
        n = case["n"]
        f32 = torch.float32
        s.update(p=_rand(g, n, std=0.02, dtype=f32), m=_rand(g, n, std=1e-4, dtype=f32),
                 v=_rand(g, n, std=1e-4, dtype=f32).square_(),
                 grad=_rand(g, n, std=1e-3, dtype=bf16 if case["grad"] == "bf16" else f32),
                 pb=torch.zeros(n, dtype=bf16, device="cuda"), step=0)
    else:
        cfg = LlamaConfig(vocab=case["vocab"], d=case["d"], n_layers=case["layers"],
                          n_heads=case["heads"], n_kv_heads=case["kv_heads"], ffn=case["ffn"])
        store = LocalParamStore(ParamLayout(cfg), "cuda", seed=seed)
        B, S = case["batch"], case["seq"]
        s.update(cfg=cfg, store=store, engine=LlamaEngine(cfg, store, S),
                 tokens=_ids(g, B * S, cfg.vocab).view(B, S),
                 targets=_ids(g, B * S, cfg.vocab).view(B, S))
    return s


# ----------------------------------------------------------------------------- one pass
def run(s):
    c = s["case"]
    k = c["kind"]
    if k == "linear":
        y = ops.gemm(s["x"], s["w"])
        dx = ops.gemm(s["dy"], s["w"], b_mn=True)
        ops.gemm(s["dy"], s["x"], a_mn=True, b_mn=True, out=s["dw"])
        return {"y": y, "dx": dx, "dw": s["dw"]}
    if k == "attention":
        o, ctx = ops.attention_fwd(s["qkv"], c["batch"], c["seq"], c["heads"], c["kv_heads"],
                                   c["hd"], need_bwd=c["train"])
        if not c["train"]:
            return {"o": o}
        return {"o": o, "dqkv": ops.attention_bwd(ctx, s["do"])}
    if k == "norm":
        y, rstd = ops.rmsnorm_fwd(s["x"], s["w"], EPS)
        dx = ops.rmsnorm_bwd(s["dy"], s["x"], s["w"], rstd, s["dw"], dres=s["dres"])
        return {"y": y, "rstd": rstd, "dx": dx, "dw": s["dw"]}
    if k == "swiglu":
        return {"h": ops.swiglu_fwd(s["gu"]), "dgu": ops.swiglu_bwd(s["gu"], s["dh"])}
    if k == "loss":
        hf, rstd = ops.rmsnorm_fwd(s["x"], s["w"], EPS)
        logits = ops.gemm(hf, s["head"])
        loss = ops.cross_entropy_(logits, s["targets"], 1.0 / c["tokens"])
        dhf = ops.gemm(logits, s["head"], b_mn=True)
        ops.gemm(logits, hf, a_mn=True, b_mn=True, out=s["dhead"])
        dx = ops.rmsnorm_bwd(dhf, s["x"], s["w"], rstd, s["dw"])
        return {"loss": loss, "dlogits": logits, "dx": dx, "dw": s["dw"], "dhead": s["dhead"]}
    if k == "adamw":
        s["step"] += 1
        ops.adamw_(s["p"], s["m"], s["v"], s["grad"], s["pb"], lr=1e-4, step=s["step"],
                   grad_scale=0.5)
        return {"p": s["p"], "m": s["m"], "v": s["v"], "pb": s["pb"]}
    loss = s["engine"].forward_backward(s["tokens"], s["targets"])
    out = {"loss": loss}
    st = s["store"]
    for ui, u in enumerate(st.layout.units):
        for name, t in st.unit_grads(ui).items():
            out[f"{u.name}.{name}"] = t
    return out


# ------------------------------------------------------------- what a pass cannot do without
def _attn_flops(B, S, H, hd):
    return 2.0 * B * H * S * (S + 1) * hd      # causal: q k^T and p v


def work(case):
    k = case["kind"]
    if k == "linear":
        T, I, O = case["tokens"], case["n_in"], case["n_out"]
        return {"bytes": 2.0 * (2 * T * I + 2 * T * O + 2 * O * I), "flops": 6.0 * T * I * O}
    if k == "attention":
        B, S, H, HK, D = (case[n] for n in ("batch", "seq", "heads", "kv_heads", "hd"))
        f, q, kv = _attn_flops(B, S, H, D), 2.0 * B * S * H * D, 2.0 * B * S * 2 * HK * D
        if not case["train"]:
            return {"bytes": 2 * q + kv, "flops": f}
        return {"bytes": 4 * q + 2 * kv, "flops": 3.5 * f}
    if k == "norm":
        T, d = case["tokens"], case["d"]
        return {"bytes": 10.0 * T * d + 4.0 * T + 4.0 * d, "flops": 15.0 * T * d}
    if k == "swiglu":
        T, F = case["tokens"], case["ffn"]
        return {"bytes": 2.0 * T * F * 6, "flops": 20.0 * T * F}
    if k == "loss":
        T, d, V = case["tokens"], case["d"], case["vocab"]
        return {"bytes": 2.0 * (2 * T * d + 2 * V * d + T * V), "flops": 6.0 * T * d * V}
    if k == "adamw":
        gb = 2 if case["grad"] == "bf16" else 4
        return {"bytes": (24.0 + gb + 2) * case["n"], "flops": 15.0 * case["n"]}
    B, S, V, d, L = (case[n] for n in ("batch", "seq", "vocab", "d", "layers"))
    H, HK, F = case["heads"], case["kv_heads"], case["ffn"]
    hd, T = d // H, B * S
    per = (H + 2 * HK) * hd * d + H * hd * d + 3 * F * d
    params = L * (per + 2 * d) + 2 * V * d + d
    return {"bytes": 4.0 * params + 16.0 * T,
            "flops": 6.0 * T * (L * per + V * d) + 3.5 * L * _attn_flops(B, S, H, hd)}


def tolerance(case):
    """About four times the distance to the 64-bit result that the bf16 results show (their
    last rounding alone is 1.7e-3); sums over whole tensors of fp32 values are closer."""
    k = case["kind"]
    if k == "linear":
        return {"rel": 7e-3, "max": 0.05}
    if k == "attention":
        return {"rel": 1e-2, "max": 0.25}
    if k in ("norm", "swiglu"):
        return {"rel": 7e-3, "max": 0.05}
    if k == "loss":
        return {"rel": 1e-2, "max": 0.25}
    if k == "adamw":
        return {"rel": 7e-3, "max": 0.05}
    return {"rel": 3e-2, "max": 0.5}


# ------------------------------------------------------------------- the result in 64 bits
def _norm64(x, w, eps=EPS):
    rstd = torch.rsqrt(x.square().mean(-1, keepdim=True) + eps)
    return x * rstd * w, rstd.squeeze(-1)


def _head64(q, k, v, do, scale):
    """Causal attention of one head: q, k, v, do [S, hd] -> o, dq, dk, dv (or None)."""
    S = q.shape[0]
    s = (q @ k.t()).mul_(scale)
    s.masked_fill_(torch.ones(S, S, dtype=torch.bool, device=q.device).triu_(1), -math.inf)
    p = torch.softmax(s, dim=-1)
    del s
    o = p @ v
    if do is None:
        return o, None, None, None
    dv = p.t() @ do
    dp = do @ v.t()
    ds = p.mul_(dp.sub_((do * o).sum(-1, keepdim=True))).mul_(scale)
    return o, ds @ k, ds.t() @ q, dv


def _attention64(qkv, do, B, S, H, HK, D):
    """qkv, do of any float type -> o, dqkv in 64 bits (dqkv None without do)."""
    T = B * S
    o = torch.empty(T, H * D, dtype=torch.float64, device=qkv.device)
    dqkv = None if do is None else torch.zeros(T, (H + 2 * HK) * D, dtype=torch.float64,
                                               device=qkv.device)
    for b in range(B):
        r = slice(b * S, (b + 1) * S)
        for h in range(H):
            j = h // (H // HK)
            cq = slice(h * D, (h + 1) * D)
            ck = slice((H + j) * D, (H + j + 1) * D)
            cv = slice((H + HK + j) * D, (H + HK + j + 1) * D)
            oh, dq, dk, dv = _head64(qkv[r, cq].double(), qkv[r, ck].double(),
                                     qkv[r, cv].double(),
                                     None if do is None else do[r, cq].double(), D ** -0.5)
            o[r, cq] = oh
            if do is not None:
                dqkv[r, cq] = dq
                dqkv[r, ck] += dk
                dqkv[r, cv] += dv
    return o, dqkv


class _Attention64(torch.autograd.Function):
    @staticmethod
    def forward(ctx, qkv, dims):
        ctx.dims = dims
        ctx.save_for_backward(qkv)
        return _attention64(qkv, None, *dims)[0]

    @staticmethod
    def backward(ctx, do):
        return _attention64(ctx.saved_tensors[0], do, *ctx.dims)[1], None


def _rope64(x, S, theta):
    """x [T, heads, hd], rotate-half, position = row modulo S."""
    T, _, hd = x.shape
    inv = theta ** (-torch.arange(0, hd, 2, dtype=torch.float64, device=x.device) / hd)
    ang = (torch.arange(T, device=x.device) % S).double()[:, None, None] * inv
    a, b = x[..., : hd // 2], x[..., hd // 2:]
    return torch.cat([a * ang.cos() - b * ang.sin(), b * ang.cos() + a * ang.sin()], dim=-1)


def _model64(s, case):
    cfg, st = s["cfg"], s["store"]
    B, S = case["batch"], case["seq"]
    H, HK, D, F = cfg.n_heads, cfg.n_kv_heads, cfg.d // cfg.n_heads, cfg.ffn
    w = {}
    for ui, u in enumerate(st.layout.units):
        for name, t in st.unit_params(ui).items():
            w[f"{u.name}.{name}"] = t.detach().double().requires_grad_(True)
    x = w["embed.embed"][s["tokens"].reshape(-1)]
    for i in range(cfg.n_layers):
        p = f"layer{i}."
        qkv = _norm64(x, w[p + "attn_norm"], cfg.eps)[0] @ w[p + "wqkv"].t()
        qk, v = qkv.split([(H + HK) * D, HK * D], dim=1)
        qk = _rope64(qk.reshape(B * S, H + HK, D), S, cfg.theta).reshape(B * S, -1)
        x = x + _Attention64.apply(torch.cat([qk, v], dim=1), (B, S, H, HK, D)) @ w[p + "wo"].t()
        gate, up = (_norm64(x, w[p + "mlp_norm"], cfg.eps)[0] @ w[p + "w_gu"].t()).split(F, dim=1)
        x = x + (torch.nn.functional.silu(gate) * up) @ w[p + "w_down"].t()
    logits = _norm64(x, w["head.final_norm"], cfg.eps)[0] @ w["head.lm_head"].t()
    loss = torch.nn.functional.cross_entropy(logits, s["targets"].reshape(-1))
    loss.backward()
    return {"loss": loss.detach(), **{n: t.grad for n, t in w.items()}}


def exact(case, seed):
    s = prepare(case, seed)
    k = case["kind"]
    if k == "linear":
        x, w, dy = s["x"].double(), s["w"].double(), s["dy"].double()
        return {"y": x @ w.t(), "dx": dy @ w, "dw": dy.t() @ x}
    if k == "attention":
        o, dqkv = _attention64(s["qkv"], s["do"] if case["train"] else None, case["batch"],
                               case["seq"], case["heads"], case["kv_heads"], case["hd"])
        return {"o": o, "dqkv": dqkv} if case["train"] else {"o": o}
    if k == "norm":
        x, w = s["x"].double().requires_grad_(True), s["w"].double().requires_grad_(True)
        y, rstd = _norm64(x, w)
        y.backward(s["dy"].double())
        return {"y": y.detach(), "rstd": rstd.detach(), "dx": x.grad + s["dres"].double(),
                "dw": w.grad}
    if k == "swiglu":
        gu = s["gu"].double().requires_grad_(True)
        gate, up = gu.split(case["ffn"], dim=1)
        h = torch.nn.functional.silu(gate) * up
        h.backward(s["dh"].double())
        return {"h": h.detach(), "dgu": gu.grad}
    if k == "loss":
        x, w, head = (s[n].double().requires_grad_(True) for n in ("x", "w", "head"))
        logits = _norm64(x, w)[0] @ head.t()
        logits.retain_grad()
        rows = torch.nn.functional.cross_entropy(logits, s["targets"], reduction="none")
        rows.mean().backward()
        return {"loss": rows.detach(), "dlogits": logits.grad, "dx": x.grad, "dw": w.grad,
                "dhead": head.grad}
    if k == "adamw":
        p, m, v, gr = (s[n].double() for n in ("p", "m", "v", "grad"))
        gr = gr * 0.5
        m = 0.9 * m + 0.1 * gr
        v = 0.95 * v + 0.05 * gr * gr
        p = p * (1 - 1e-4 * 0.1) - 1e-4 / (1 - 0.9) * m / ((v / (1 - 0.95)).sqrt() + 1e-8)
        return {"p": p, "m": m, "v": v, "pb": p}
    return _model64(s, case)
