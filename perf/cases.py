"""The work that users of this library have it do, as cases that can be timed one by one: attention under
``torch.func.jvp`` (forward and reverse, the denoiser's and longer sequences, equal and unequal lengths, the head
dimensions in use), attention without tangents, the fused pointwise chain of a denoiser block, the vocabulary-side ends
of the training step, a sampling pass of the denoiser, and the training objective with its gradients.

Sizes are those of the configurations, tests and benchmark of this repository (12 heads of 64 channels at lengths 128 and
256, 16 heads of 64 or 128 channels at 2048, a vocabulary of 30522, hidden size 768) and generic ones around them.

Tolerances, from comparing each path once with the same formulas in 64 bits (relative 2-norm errors): attention outputs and
gradients up to 2.5e-3 in bf16 (bf16 operands of the second product and a bf16 result) and 3e-4 in fp16; the pointwise chain
up to 2.5e-3; the vocabulary-side results up to 2.8e-3 (bf16 gradients); the denoiser's logits 1.2e-2 (twelve bf16 blocks);
the step's gradients 1.3e-2 and its self-distillation loss 1.3e-2 against the plain formulas in 32 bits.  The bounds are
about four times that.
"""
import math

import torch

from semicat_b200 import dual_ops, ops, rotary, safe_sdpa_jvp, sdpa_jvp, train_step, vocab_ops
from semicat_b200.ddp import FlatGradients

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}


def listed():
    return [
        # the smallest call: a few heads of a small model, where only latency and launches count
        {"name": "attn_tiny_d32", "kind": "attention", "entry": "sdpa", "B": 2, "H": 4, "Lq": 64, "Lk": 64, "D": 32, "dtype": "bf16", "cot": "both"},
        # one rank's share of the text8-shaped run on 8 GPUs (8 self-distillation samples of length 256), last layer: only
        # the tangent output has a cotangent
        {"name": "attn_share_L256", "kind": "attention", "entry": "safe", "B": 8, "H": 12, "Lq": 256, "Lk": 256, "D": 64, "dtype": "bf16", "cot": "tangent"},
        # the benchmark's operator workload on fixed buffers (pre-marshalled calls, as in its loop): memory-bound lengths
        {"name": "attn_plan_L128", "kind": "plan", "B": 64, "H": 12, "Lq": 128, "Lk": 128, "D": 64, "dtype": "bf16", "cot": "both"},
        # heads of 32 channels, a small model at a full batch
        {"name": "attn_d32_L256", "kind": "attention", "entry": "sdpa", "B": 32, "H": 8, "Lq": 256, "Lk": 256, "D": 32, "dtype": "bf16", "cot": "both"},
        # long sequences, both head dimensions of the length sweep
        {"name": "attn_long_d64", "kind": "attention", "entry": "safe", "B": 8, "H": 16, "Lq": 2048, "Lk": 2048, "D": 64, "dtype": "bf16", "cot": "both"},
        {"name": "attn_long_d128", "kind": "attention", "entry": "safe", "B": 8, "H": 16, "Lq": 2048, "Lk": 2048, "D": 128, "dtype": "bf16", "cot": "both"},
        # unequal, odd lengths in fp16
        {"name": "attn_ragged_fp16", "kind": "attention", "entry": "sdpa", "B": 4, "H": 10, "Lq": 777, "Lk": 1533, "D": 64, "dtype": "fp16", "cot": "both"},
        # the cross-entropy branch of the training step: attention without tangents, forward and reverse
        {"name": "attn_primal_L128", "kind": "attention", "entry": "safe", "B": 192, "H": 12, "Lq": 128, "Lk": 128, "D": 64, "dtype": "bf16", "cot": "primal"},
        # the fused pointwise chain of one denoiser block on (primal, tangent) pairs, forward and reverse
        {"name": "block_ops", "kind": "block_ops", "B": 128, "S": 128, "C": 768, "H": 12, "dual": True, "p": 0.1},
        # the vocabulary-side ends of the step: 16 self-distillation and 48 cross-entropy samples
        {"name": "vocabulary", "kind": "vocabulary", "sd": 16, "ce": 48, "L": 128, "V": 30522, "eps": 0.0},
        # sampling: one pass of the denoiser without gradients at a small batch
        {"name": "denoiser_sample", "kind": "denoiser", "B": 8, "L": 128, "V": 30522, "blocks": 12},
        # the training objective with all gradients, replayed from a CUDA graph as the training loop of the benchmark does
        {"name": "train_step", "kind": "train_step", "B": 128, "L": 128, "V": 30522, "blocks": 12, "p": 0.1},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["attention", "plan", "block_ops", "vocabulary", "denoiser", "train_step"], [10, 3, 3, 2, 1, 1])[0]
    if kind in ("attention", "plan"):
        D = rng.choice([64, 64, 64, 128, 128, 32, 48, 96, 16])
        Lq = _log(rng, 32, 4096 if D in (64, 128) else 512)
        if rng.random() < 0.5:
            Lq = max(64, Lq // 64 * 64)
        Lk = Lq if rng.random() < 0.7 else max(16, int(Lq * rng.uniform(0.4, 2.0)))
        H = rng.choice([4, 6, 8, 12, 16])
        # tokens x heads up to those of the largest length-2048 case, products up to its products
        most = min(8 * 16 * 2048 / (H * max(Lq, Lk)), 8 * 16 * 2048 ** 2 * 128 / (float(H) * Lq * Lk * D), 256)
        if D not in (64, 128):
            most = min(most, 32)
        B = _log(rng, 1, max(most, 1))
        c = {"kind": kind, "B": B, "H": H, "Lq": Lq, "Lk": Lk, "D": D, "dtype": rng.choice(["bf16", "bf16", "bf16", "fp16"]),
             "cot": rng.choice(["both", "both", "tangent", "primal"])}
        if kind == "attention":
            c["entry"] = rng.choice(["sdpa", "safe"])
        return c
    if kind == "block_ops":
        C = rng.choice([256, 512, 768, 768, 1024])
        return {"kind": kind, "B": _log(rng, 2, 256), "S": _log(rng, 50, 256), "C": C, "H": C // 64, "dual": rng.random() < 0.7,
                "p": rng.choice([0.0, 0.1])}
    if kind == "vocabulary":
        n = _log(rng, 2, 16)
        return {"kind": kind, "sd": n, "ce": 3 * n, "L": _log(rng, 32, 160), "V": rng.choice([30522, _log(rng, 512, 50257)]),
                "eps": rng.choice([0.0, 0.1])}
    c = {"kind": kind, "B": _log(rng, 1, 32), "L": _log(rng, 64, 256), "V": rng.choice([27, 30522, _log(rng, 512, 30000)]),
         "blocks": rng.randint(4, 12)}
    if kind == "train_step":
        c["B"] = max(4, c["B"])
        c["p"] = rng.choice([0.0, 0.1])
    return c


# ------------------------------------------------------------------------------------------------------------ inputs
def _normal(gen, shape, scale=1.0, dtype=torch.bfloat16):
    return (torch.randn(shape, device="cuda", generator=gen) * scale).to(dtype)


def _denoiser(c, seed, p):
    torch.manual_seed(seed)
    rms = c["V"] < 512
    with torch.device("cuda"):
        net = train_step.DiT(c["V"], 768, 128, c["blocks"], 12, dropout=p, length=c["L"], embed_type="rms" if rms else "naive")
    with torch.no_grad():  # a trained model's gates and head are not zero
        for q in net.parameters():
            if not q.any():
                q.normal_(0.0, 0.05)
    return net


def _attention_inputs(c, gen):
    B, H, D, dt = c["B"], c["H"], c["D"], DTYPES[c["dtype"]]
    mk = lambda L, s: _normal(gen, (B, L, H, D), s, dt)  # the denoiser's memory order
    q, k, v = mk(c["Lq"], D ** -0.5), mk(c["Lk"], 1.0), mk(c["Lk"], 1.0)
    tq, tk, tv = mk(c["Lq"], 0.1), mk(c["Lk"], 0.1), mk(c["Lk"], 0.1)
    return q, k, v, tq, tk, tv, mk(c["Lq"], 1.0), mk(c["Lq"], 1.0)


def prepare(c, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind = c["kind"]
    if kind in ("attention", "plan"):
        q, k, v, tq, tk, tv, g_o, g_to = _attention_inputs(c, gen)
        B, H = c["B"], c["H"]
        st = {"case": c}
        if kind == "attention":
            to = (lambda t: t) if c["entry"] == "safe" else (lambda t: t.transpose(1, 2))
            st["fn"] = safe_sdpa_jvp if c["entry"] == "safe" else sdpa_jvp
            st["x"] = [to(t).requires_grad_(True) for t in (q, k, v)]
            if c["cot"] != "primal":
                st["t"] = [to(t).requires_grad_(True) for t in (tq, tk, tv)]
            st["g_o"], st["g_to"] = to(g_o), to(g_to)
            return st
        q, k, v, tq, tk, tv, g_o, g_to = (t.transpose(1, 2) for t in (q, k, v, tq, tk, tv, g_o, g_to))
        like = lambda t: torch.empty_like(t)
        st["o"], st["to"] = like(q), like(q)
        st["lse"] = torch.zeros(B, H, ops.stat_len(c["Lq"]), device="cuda")
        st["mu"] = torch.zeros_like(st["lse"])
        st["grads"] = [like(t) for t in (q, k, v, tq, tk, tv)]
        if c["cot"] == "primal":
            for t in st["grads"][3:]:
                t.zero_()  # not written without a cotangent on the tangent output
        st["plan"] = ops.Plan(q, k, v, tq, tk, tv, st["o"], st["to"], st["lse"], st["mu"], g_o=None if c["cot"] == "tangent" else g_o,
                              g_to=None if c["cot"] == "primal" else g_to, grads=st["grads"])
        return st
    if kind == "block_ops":
        B, S, C, H = c["B"], c["S"], c["C"], c["H"]
        norm = torch.nn.LayerNorm(C, device="cuda")
        with torch.no_grad():
            norm.weight.normal_(1.0, 0.1, generator=gen)
            norm.bias.normal_(0.0, 0.1, generator=gen)
        ang = torch.arange(S, device="cuda")[:, None] / (10000 ** (torch.arange(0, C // H, 2, device="cuda") / (C // H)))[None]
        shapes = {"x": (B, S, C), "qkv": (B, S, 3, H, C // H), "branch": (B, S, C), "mlp": (B, S, 4 * C), "mod": (B, 1, 3 * C)}
        prim = {n: _normal(gen, s, 0.2 if n == "mod" else 1.0).requires_grad_(True) for n, s in shapes.items()}
        tang = {n: _normal(gen, s, 0.1).requires_grad_(True) for n, s in shapes.items()} if c["dual"] else None
        outs = [(B, S, C)] + [(B, S, H, C // H)] * 3 + [(B, S, C), (B, S, 4 * C)]
        return {"case": c, "seed": seed, "norm": norm, "cos": ang.cos(), "sin": ang.sin(), "prim": prim, "tang": tang,
                "g": [_normal(gen, s) for s in outs], "gt": [_normal(gen, s) for s in outs] if c["dual"] else None}
    if kind == "vocabulary":
        sd, ce, L, V = c["sd"], c["ce"], c["L"], c["V"]
        W = vocab_ops.padded(V)
        noise = torch.randn(sd + ce, L, W, device="cuda", generator=gen)[..., :V]
        ids = torch.randint(0, V, (sd + ce, L), device="cuda", generator=gen)
        t = torch.rand(sd + ce, device="cuda", generator=gen)
        mk = lambda n, s: _normal(gen, (n, L, W), s)
        return {"case": c, "x0": noise, "ids": ids, "t": t, "s": torch.rand(sd, device="cuda", generator=gen) * t[:sd],
                "pred": mk(ce, 1.0).requires_grad_(True), "l": mk(sd, 1.0).requires_grad_(True), "tl": mk(sd, 0.5).requires_grad_(True),
                "target": mk(sd, 1.0)}
    net = _denoiser(c, seed, c.get("p", 0.0))
    x1 = torch.randint(0, c["V"], (c["B"], c["L"]), device="cuda", generator=gen)
    noise = train_step.draw_noise(x1, c["V"], generator=gen)
    st = {"case": c, "seed": seed, "net": net, "x1": x1, "noise": noise}
    if kind == "denoiser":
        net.eval()
        st["s"], st["t"] = noise["u_sd"] * noise["t_sd"], noise["t_sd"]
        return st
    # As in the benchmark's loop: the step runs a few times, is captured once, and every later step replays it on the
    # same token and noise buffers (a loop with new data copies it into them).
    st["flat"] = FlatGradients(net.parameters())
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        for _ in range(2):
            _objective(st)
    torch.cuda.current_stream().wait_stream(side)
    torch.cuda.synchronize()
    st["graph"] = torch.cuda.CUDAGraph()
    with torch.cuda.graph(st["graph"]):
        st["loss"] = _objective(st)
    return st


def _objective(st):
    st["flat"].zero()
    vf, sd = train_step.model_step(st["net"], st["x1"], st["noise"], primal_attention="lib")
    train_step.total_loss(vf, sd).backward()
    return vf.detach(), sd.detach()


# ------------------------------------------------------------------------------------------------------------ one pass
def _chain(norm, cos, sin, p, x, qkv, branch, mlp, mod):
    shift, scale, gate = mod.chunk(3, dim=2)
    return (dual_ops.ln_modulate(x, norm, shift, scale), *rotary.rotary_qkv(qkv, cos, sin, torch.bfloat16),
            dual_ops.gated_residual(x, branch, gate, p, True), dual_ops.gelu_tanh(mlp))


def run(st):
    c = st["case"]
    kind = c["kind"]
    if kind == "plan":
        st["plan"].forward()
        st["plan"].backward()
        return [st["o"], st["to"], st["lse"], st["mu"], *st["grads"]]
    if kind == "attention":
        if c["cot"] == "primal":
            y = st["fn"](*st["x"])
            return [y.detach(), *torch.autograd.grad(y, st["x"], st["g_o"])]
        y, ty = torch.func.jvp(st["fn"], tuple(st["x"]), tuple(st["t"]))
        outs, gs = ([y, ty], [st["g_o"], st["g_to"]]) if c["cot"] == "both" else ([ty], [st["g_to"]])
        return [y.detach(), ty.detach(), *torch.autograd.grad(outs, st["x"] + st["t"], gs)]
    if kind == "block_ops":
        torch.cuda.manual_seed(st["seed"])  # the same dropout masks in every pass over this state
        names = list(st["prim"])
        fn = lambda *a: _chain(st["norm"], st["cos"], st["sin"], c["p"], *a)
        prim = [st["prim"][n] for n in names]
        with dual_ops.dropout_seed(torch.device("cuda")):
            if c["dual"]:
                tang = [st["tang"][n] for n in names]
                ys, tys = torch.func.jvp(fn, tuple(prim), tuple(tang))
                outs, gs, wrt = [*ys, *tys], [*st["g"], *st["gt"]], [*prim, *tang]
            else:
                outs, gs, wrt = list(fn(*prim)), st["g"], prim
            wrt = [*wrt, st["norm"].weight, st["norm"].bias]
            grads = torch.autograd.grad(outs, wrt, gs)
        return [*(t.detach() for t in outs), *grads]
    if kind == "vocabulary":
        sd, V = c["sd"], c["V"]
        x0, ids, t, s = st["x0"], st["ids"], st["t"], st["s"]
        xt = vocab_ops.interpolate_cast(x0[sd:], ids[sd:], t[sd:])
        ce = vocab_ops.cross_entropy_padded(st["pred"], ids[sd:], V, c["eps"])
        xs = vocab_ops.interpolate_cast(x0[:sd], ids[:sd], s)
        xst, lse = vocab_ops.flow_map_input(st["l"], x0[:sd], ids[:sd], s, t[:sd])
        lag = vocab_ops.sd_lag_loss(st["l"], st["tl"], st["target"], x0[:sd], ids[:sd], s, t[:sd], lse)
        grads = torch.autograd.grad(ce + lag, [st["pred"], st["l"], st["tl"]])
        return [xt, ce.detach(), xs, xst, lse, lag.detach(), *grads]
    if kind == "denoiser":
        rms = c["V"] < 512
        with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
            if rms:
                x = train_step.interpolate(st["noise"]["x0"], st["x1"], st["s"].view(-1, 1, 1))
            else:
                x = vocab_ops.interpolate_cast(st["noise"]["x0"], st["x1"], st["s"])
            return st["net"](x, st["s"], st["t"], attention="lib")
    torch.cuda.manual_seed(st["seed"])  # the same dropout masks in every pass over this state
    st["graph"].replay()
    return [*st["loss"], st["flat"].flat]


# ------------------------------------------------------------------------------------------------------------ necessary work
def work(c):
    kind = c["kind"]
    if kind in ("attention", "plan"):
        B, H, Lq, Lk, D = c["B"], c["H"], c["Lq"], c["Lk"], c["D"]
        fwd_units, bwd_units = (6, {"both": 15, "tangent": 13, "primal": 5}[c["cot"]])
        if c["cot"] == "primal" and kind == "attention":
            fwd_units = 2
        tq, tk = 2.0 * B * H * Lq * D, 2.0 * B * H * Lk * D
        dual = kind == "plan" or c["cot"] != "primal"
        # inputs and cotangents read once, outputs and gradients written once
        n_g = 2 if c["cot"] == "both" else 1
        grads = 2 if c["cot"] != "primal" else 1
        nq = (2 + 2 if dual else 1 + 1) + n_g + grads
        nk = (4 if dual else 2) + 2 * grads
        return {"flops": 2.0 * B * H * Lq * Lk * D * (fwd_units + bwd_units), "bytes": nq * tq + nk * tk}
    if kind == "block_ops":
        e = 2.0 * c["B"] * c["S"] * c["C"]
        # per direction: x, qkv (3), branch, mlp (4) in; h, q, k, v, z, act (4) out; reverse: those outputs' cotangents in,
        # inputs again, gradients out
        return {"bytes": e * (9 + 9 + 9 + 9) * (2 if c["dual"] else 1), "flops": 0.0}
    if kind == "vocabulary":
        sd, ce, V = c["sd"] * c["L"], c["ce"] * c["L"], c["V"]
        # noise once, 16-bit inputs of the network out, logits in, gradients out
        return {"bytes": (sd + ce) * V * 4.0 + (sd + ce) * V * 2.0 + ce * V * 4.0 + sd * V * (2.0 + 3 * 2.0 + 2 * 2.0), "flops": 0.0}
    C, V, L, nb = 768, c["V"], c["L"], c["blocks"]
    tokens = float(c["B"] * L)
    fwd = 2.0 * (12 * nb * C * C + 2 * V * C) + 4.0 * L * C * nb  # per token, without the small conditioning layers
    params = 12.0 * nb * C * C + 2 * V * C + nb * 128 * 6 * C
    if kind == "denoiser":
        return {"flops": tokens * fwd, "bytes": params * 4 + tokens * V * (4.0 + 2.0)}
    n_sd = int(0.25 * c["B"]) * L
    n_ce = tokens - n_sd
    emb = 2.0 * V * C
    # cross-entropy: forward, two products per layer backward (none towards the input); self-distillation: primal and
    # tangent forward (the input has no tangent), the target pass, primal and tangent backward
    flops = n_ce * (3 * fwd - emb) + n_sd * ((2 * fwd - emb) + fwd + (4 * fwd - 3 * emb))
    return {"flops": flops, "bytes": params * 8 + tokens * V * (4.0 + 2 * 2.0)}


def tolerance(c):
    kind = c["kind"]
    if kind in ("attention", "plan"):
        return {"rel": 0.01 if c["dtype"] == "bf16" else 0.0012}
    if kind == "block_ops":
        return {"rel": 0.01}
    if kind == "vocabulary":
        return {"rel": 0.01}
    return {"rel": 0.05}


# ------------------------------------------------------------------------------------------------------------ in 64 bits
def exact(c, seed):
    """What ``run`` returns, from plain torch in 64 bits; ``None`` for what depends on generated dropout masks and for the
    training step."""
    kind = c["kind"]
    if kind in ("attention", "plan"):
        return _exact_attention(c, seed)
    if kind == "block_ops":
        return _exact_block(c, prepare(c, seed))
    if kind == "vocabulary":
        return _exact_vocabulary(c, prepare(c, seed))
    return _exact_denoiser(c, prepare(c, seed)) if kind == "denoiser" else None


def _exact_attention(c, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    x = [t.transpose(1, 2) for t in _attention_inputs(c, gen)]
    B, H, Lq, Lk, D = c["B"], c["H"], c["Lq"], c["Lk"], c["D"]
    r = D ** -0.5
    outs = [torch.zeros(t.shape, dtype=torch.float64, device="cuda") for t in (x[0], x[0], *x[:6])]
    y, ty, dq, dk, dv, dtq, dtk, dtv = outs
    stats = torch.zeros(2, B, H, -(-Lq // 128) * 128, dtype=torch.float64, device="cuda")
    T = lambda t: t.transpose(-1, -2)
    for b in range(B):
        step = max(1, int(2e8 // (Lq * Lk)))
        for h in range(0, H, step):
            i = (b, slice(h, h + step))
            q, k, v, tq, tk, tv, g, G = (t[i].double() for t in x)
            s = (q @ T(k)) * r
            stats[0][i][:, :Lq] = lse = s.logsumexp(-1)
            p = torch.exp(s.sub_(lse[..., None]))
            n = (tq @ T(k) + q @ T(tk)) * r
            mu = (p * n).sum(-1, keepdim=True)
            stats[1][i][:, :Lq] = mu[..., 0]
            n -= mu
            y[i] = p @ v
            ty[i] = (p * n) @ v + p @ tv
            if c["cot"] == "primal":
                dv[i] = T(p) @ g
                w = p * (g @ T(v) - (g * y[i]).sum(-1, keepdim=True)) * r
                dq[i], dk[i] = w @ k, T(w) @ q
                continue
            if c["cot"] == "tangent":
                g = torch.zeros_like(g)
            a = G @ T(v) - (G * y[i]).sum(-1, keepdim=True)
            w = (a * n + G @ T(tv) + g @ T(v) - (G * ty[i] + g * y[i]).sum(-1, keepdim=True)) * p * r
            dtv[i] = T(p) @ G
            dv[i] = T(p * n) @ G + T(p) @ g
            u = a.mul_(p).mul_(r)
            dtq[i], dtk[i] = u @ k, T(u) @ q
            dq[i], dk[i] = u @ tk + w @ k, T(u) @ tq + T(w) @ q
    if c["kind"] == "plan":
        return [y, ty, *stats, *outs[2:]]
    if c["entry"] == "safe":
        y, ty, *grads = [t.transpose(1, 2) for t in outs]
    else:
        grads = outs[2:]
    return [y, *grads[:3]] if c["cot"] == "primal" else [y, ty, *grads]


def _rotate(t, cos, sin):
    t1, t2 = t.chunk(2, dim=-1)
    cos, sin = cos[None, :, None], sin[None, :, None]
    return torch.cat((t1 * cos - t2 * sin, t1 * sin + t2 * cos), dim=-1)


def _exact_block(c, st):
    F = torch.nn.functional
    cos, sin = st["cos"].double(), st["sin"].double()
    C = c["C"]

    def chain(w, b, x, qkv, branch, mlp, mod):
        shift, scale, gate = mod.chunk(3, dim=2)
        q, k, v = qkv.unbind(2)
        return (F.layer_norm(x, (C,), w, b, st["norm"].eps) * (1 + scale) + shift, _rotate(q, cos, sin), _rotate(k, cos, sin),
                v.clone(), x + branch * gate, F.gelu(mlp, approximate="tanh"))

    leaf = lambda t: t.detach().double().requires_grad_(True)
    prim = [leaf(t) for t in st["prim"].values()]
    wb = [leaf(st["norm"].weight), leaf(st["norm"].bias)]
    g = [t.double() for t in st["g"]]
    if c["dual"]:
        tang = [leaf(t) for t in st["tang"].values()]
        ys, tys = torch.func.jvp(lambda *a: chain(*wb, *a), tuple(prim), tuple(tang))
        outs, wrt = [*ys, *tys], [*prim, *tang, *wb]
        g += [t.double() for t in st["gt"]]
    else:
        outs, wrt = list(chain(*wb, *prim)), [*prim, *wb]
    grads = list(torch.autograd.grad(outs, wrt, g))
    outs = [t.detach() for t in outs]
    if c["p"] > 0:  # the gated residual and the gradients of its branch and of the modulation depend on the masks
        for i in range(0, len(outs), 6):
            outs[i + 4] = None
        for i in range(0, len(grads) - 2, 5):
            grads[i + 2] = grads[i + 4] = None
    return [*outs, *grads]


def _exact_vocabulary(c, st):
    sd, V = c["sd"], c["V"]
    W = st["pred"].shape[-1]
    pad = lambda t: torch.nn.functional.pad(t, (0, W - V))
    col = lambda t: t.double().view(-1, 1, 1)

    def mix(x0, ids, t):
        x = x0.double() * (1 - col(t))
        return x.scatter_add_(-1, ids[..., None], col(t).expand(*ids.shape, 1).contiguous())

    def smooth(ids, logp):
        return -((1 - c["eps"]) * logp.gather(-1, ids[..., None])[..., 0] + c["eps"] * logp.mean(-1)).mean()

    ids, s, t = st["ids"], st["s"], st["t"][:sd]
    xt = pad(mix(st["x0"][sd:], ids[sd:], st["t"][sd:]))
    pred = st["pred"].detach().double().requires_grad_(True)
    ce = smooth(ids[sd:], pred[..., :V].log_softmax(-1))
    d_pred, = torch.autograd.grad(ce, [pred])
    xs = mix(st["x0"][:sd], ids[:sd], s)
    l, tl = (st[n].detach().double().requires_grad_(True) for n in ("l", "tl"))
    p, u = l[..., :V].softmax(-1), tl[..., :V]
    ddt = 1 / (1 - col(s) + 1e-8)
    dt = (col(t) - col(s)) * ddt
    xst = (xs + dt * (p - xs)).detach()
    dv = ddt * (p - xs) + dt * p * (u - (p * u).sum(-1, keepdim=True))
    lag = ((1 - col(t)) * dv - st["target"][..., :V].double().softmax(-1) + xst).square().sum(-1).mean()
    d_l, d_tl = torch.autograd.grad(lag, [l, tl])
    lse = l.detach()[..., :V].logsumexp(-1).flatten()
    return [xt, ce.detach(), pad(xs), pad(xst), lse, lag.detach(), d_pred, d_l, d_tl]


def _exact_denoiser(c, st):
    F = torch.nn.functional
    w = {n: t.double() for n, t in st["net"].state_dict().items()}
    lin = lambda n, x: F.linear(x, w[n + ".weight"], w.get(n + ".bias"))
    norm = lambda n, x: F.layer_norm(x, x.shape[-1:], w[n + ".weight"], w[n + ".bias"])
    gelu = lambda x: F.gelu(x, approximate="tanh")
    B, L, V = c["B"], c["L"], c["V"]
    s, t = st["s"].double(), st["t"].double()

    def clock(n, v):
        a = v[:, None] * w[n + ".freqs"][None]
        return lin(n + ".mlp.2", F.silu(lin(n + ".mlp.0", torch.cat((a.cos(), a.sin()), -1))))

    x = st["noise"]["x0"].double() * (1 - s.view(-1, 1, 1))
    x.scatter_add_(-1, st["x1"][..., None], s.view(-1, 1, 1).expand(B, L, 1).contiguous())
    cond = F.silu(clock("s_map", s)) + F.silu(clock("t_map", t - s))
    with torch.no_grad():
        if V < 512:
            h = lin("embed.proj", x * torch.rsqrt(s ** 2 + (1 - s) ** 2 * V + 1e-6).view(-1, 1, 1))
            h = h + 0.1 * lin("embed.mlp.2", gelu(lin("embed.mlp.0", h)))
            h = (1 + lin("embed.gamma", cond)[:, None]) * h + lin("embed.beta", cond)[:, None]
            h = F.rms_norm(h, h.shape[-1:], w["embed.norm.weight"], 1e-8)
        else:
            h = lin("embed.seq", x * V ** -0.5)
        for i in range(c["blocks"]):
            n = "blocks.%d." % i
            sh1, sc1, g1, sh2, sc2, g2 = lin(n + "ada", cond)[:, None].chunk(6, dim=2)
            q, k, v = lin(n + "attn_qkv", norm(n + "norm1", h) * (1 + sc1) + sh1).view(B, L, 3, 12, 64).unbind(2)
            q, k, v = (z.transpose(1, 2) for z in (_rotate(q, w["cos"], w["sin"]), _rotate(k, w["cos"], w["sin"]), v))
            a = (torch.softmax(q @ k.transpose(-1, -2) / 8, -1) @ v).transpose(1, 2).reshape(B, L, 768)
            h = h + lin(n + "attn_out", a) * g1
            m = lin(n + "mlp.2", gelu(lin(n + "mlp.0", norm(n + "norm2", h) * (1 + sc2) + sh2)))
            h = h + m * g2
        shift, scale = lin("ada_out", cond)[:, None].chunk(2, dim=2)
        return lin("head", norm("norm_out", h) * (1 + scale) + shift)
