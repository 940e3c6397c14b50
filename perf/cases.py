"""Work whose speed matters to a user of memarch_b200: the layers a training run spends its time in, over the sizes
the registry's models have (`tiny` at width 256 up to the 2048-wide anchor-MoE model), and one whole small model.

`listed()` are fixed cases, `draw(rng)` gives another one of the same ranges, `prepare` builds what a program holds
before the call, `run` makes one pass through the public entry points, `exact` states the same result in 64 bits.
"""
from __future__ import annotations

import math

import torch
import torch.nn.functional as F

from memarch_b200 import OptConfig, build, ops
from memarch_b200.models.blocks import LightBlock
from memarch_b200.models.moe import AnchorMoE
from memarch_b200.optim import Instinct

DEV = "cuda"
VOCAB = 50304


def listed():
    return [
        # a light layer of the `tiny` model, one small training batch: launches and latency
        dict(name="block_tiny", op="block", d=256, B=4, T=512, window=128, relu2=False, train=True),
        # a light layer of the 2048-wide model at its training batch (32 texts x 1024 words, plain causal)
        dict(name="block_train", op="block", d=2048, B=32, T=1024, window=2048, relu2=False, train=True),
        # a light layer of the long-context model: 16 384-word texts, sliding window of 256
        dict(name="block_long", op="block", d=1024, B=2, T=16384, window=256, relu2=False, train=True),
        # evaluation of the same layer on texts of an odd length, no gradients
        dict(name="block_eval", op="block", d=1024, B=3, T=3001, window=256, relu2=False, train=False),
        # a heavy layer of the 2048-wide model on the anchors of a training batch (256 of 1024 words per text)
        dict(name="moe_train", op="moe", d=2048, B=32, A=256, E=8, frozen=0, relu2=True),
        # a heavy layer under wave training: half of the experts sit in the frozen int8 bank
        dict(name="moe_bank", op="moe", d=768, B=16, A=205, E=16, frozen=8, relu2=False),
        # output head + cross-entropy with the pointer mixture, 2048 wide plus the frequency column
        dict(name="head_mix", op="head", d=2064, N=8192, mix=True),
        # the head of a small model on one short batch
        dict(name="head_small", op="head", d=256, N=1000, mix=False),
        # optimizer step of one heavy layer's expert tables (bf16 weights with fp32 copies)
        dict(name="opt_experts", op="opt", d=2048, E=8, H=6144),
        # optimizer step of one light layer's matrices (fp32 weights with the bf16 copies the products read)
        dict(name="opt_block", op="opt", d=1024, E=0, H=4096),
        # keys-and-locks search over a long-context batch
        dict(name="locks_long", op="locks", B=4, T=16384),
        # the dense control model of the registry, one training step's loss and gradients
        dict(name="dense_lm", op="lm", B=8, T=512),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["block", "block", "block", "moe", "moe", "head", "head", "opt", "opt", "locks", "lm"])
    if op == "block":
        d = rng.choice([256, 512, 768, 1024, 2048])
        tokens = _log(rng, 300, 24576 if d <= 1024 else 16384)
        T = min(tokens, _log(rng, 100, 16384))
        return dict(op=op, d=d, B=max(1, tokens // T), T=T, window=rng.choice([128, 256, 256, 2048]),
                    relu2=rng.random() < 0.25, train=rng.random() < 0.7)
    if op == "moe":
        d = rng.choice([256, 768, 1024, 2048])
        E = rng.choice([4, 8, 16])
        return dict(op=op, d=d, B=rng.randint(2, 32), A=rng.randint(16, 256 if d < 2048 else 200), E=E,
                    frozen=rng.choice([0, 0, E // 2]), relu2=rng.random() < 0.5)
    if op == "head":
        return dict(op=op, d=rng.choice([256, 512, 768, 1024, 1040, 2064]), N=8 * _log(rng, 16, 900), mix=rng.random() < 0.5)
    if op == "opt":
        d = rng.choice([256, 384, 512, 768, 1024, 2048])
        E = rng.choice([0, 4, 8])
        return dict(op=op, d=d, E=E, H=d * rng.choice([2, 3, 4]))
    if op == "locks":
        T = _log(rng, 200, 16384)
        return dict(op=op, B=max(1, min(32, rng.randint(1, 65536 // T))), T=T)
    return dict(op=op, B=rng.randint(1, 8), T=rng.randint(100, 512))


# ------------------------------------------------------------------------------------------------ inputs
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _randn(g, *shape):
    return torch.randn(*shape, device=DEV, generator=g)


def _zipf(g, *shape):
    """Word ids with a Zipf-like marginal."""
    u = torch.rand(*shape, device=DEV, generator=g, dtype=torch.float64)
    return (torch.exp(u * math.log(VOCAB - 7)).long() - 1).clamp(0, VOCAB - 1)


def _text(g, B, T):
    """Zipf words in which runs copied from earlier in the text are mixed in, as in real text."""
    x = _zipf(g, B, T)
    t = torch.arange(T, device=DEV)[None]
    n = -(-T // 64)
    at = torch.randint(0, 56, (B, n), device=DEV, generator=g).repeat_interleave(64, 1)[:, :T]      # a run per 64 words
    back = torch.randint(1, T, (B, n), device=DEV, generator=g).repeat_interleave(64, 1)[:, :T]
    copied = (t % 64 >= at) & (t % 64 < at + 6) & (t - back >= 0)
    return torch.where(copied, x.gather(1, (t - back).clamp(min=0)), x)


class _State:
    pass


def prepare(case, seed):
    s, g, op = _State(), _gen(seed), case["op"]
    s.case = case
    torch.manual_seed(seed)
    if op == "block":
        d, B, T = case["d"], case["B"], case["T"]
        with torch.device(DEV):
            s.block = LightBlock(d, d // 64, ("relu2",) if case["relu2"] else ())
        s.x = _randn(g, B, T, d)
        s.dy = _randn(g, B, T, d) * 1e-2
        # the bf16 copies of the weights that a trained model carries
        s.block(_randn(g, 1, 8, d), case["window"])
        if case["train"]:
            s.x.requires_grad_()
        else:
            s.block.eval()
    elif op == "moe":
        d, B, A, E = case["d"], case["B"], case["A"], case["E"]
        with torch.device(DEV):
            s.moe = AnchorMoE(d, E=E, k_avg=2, bank=True, act="relu2" if case["relu2"] else "swiglu",
                              w_dtype=torch.bfloat16, bank_q="int8")
        if case["frozen"]:
            s.moe.rebank([e < case["frozen"] for e in range(E)])
        s.x = _randn(g, B, A, d).requires_grad_()
        s.dy = _randn(g, B, A, d) * 1e-2
        # surprise of the anchors; the last places of a text may be empty (-1)
        filled = torch.randint(A // 2, A + 1, (B, 1), device=DEV, generator=g)
        sur = torch.rand(B, A, device=DEV, generator=g) * 8 + 2
        s.sur = torch.where(torch.arange(A, device=DEV)[None] < filled, sur, torch.full_like(sur, -1.0))
    elif op == "head":
        d, N = case["d"], case["N"]
        s.h = _randn(g, N, d).bfloat16().requires_grad_()
        s.w = (_randn(g, VOCAB, d) * d ** -0.5).requires_grad_()
        s.y = _zipf(g, N)
        s.gate = s.hit = None
        if case["mix"]:
            s.gate = (torch.rand(N, device=DEV, generator=g) * 0.4).requires_grad_()
            s.hit = (torch.rand(N, device=DEV, generator=g) > 0.7).float()
    elif op == "opt":
        d, H = case["d"], case["H"]
        shapes = [(case["E"], d, H), (case["E"], H, d)] if case["E"] else [(3 * d, d), (d, d), (2 * H, d), (d, H)]
        s.p, s.g = [], []
        for sh in shapes:
            w = _randn(g, *sh) * sh[-1] ** -0.5
            s.p.append(torch.nn.Parameter(w.bfloat16() if case["E"] else w))
            s.g.append((_randn(g, *sh) * 1e-3).bfloat16())
        if not case["E"]:
            for p in s.p:
                ops.basic.weight_bf16(p, direct=True)          # the bf16 copy that the products read
        s.opt = Instinct(s.p, OptConfig(lr=6e-4, norm="hs", scale=0.12, m_bf16=True, rel_every=8))
        for m in s.opt.m:
            m.copy_(_randn(g, *m.shape) * 5e-4)
        s.opt.prepare(torch.tensor(3.0, device=DEV), _randn(g, 64))
        s.opt.finish()
    elif op == "locks":
        s.x = _text(g, case["B"], case["T"])
        s.bucket = torch.randint(0, 8, (VOCAB,), device=DEV, generator=g)
    elif op == "lm":
        with torch.device(DEV):
            s.model = build("transformer", VOCAB)
        s.x = _zipf(g, case["B"], case["T"] + 1)
    return s


# ------------------------------------------------------------------------------------------------ one pass
def _named_grads(params, grads):
    return {n.replace(".weight", ""): g for (n, _), g in zip(params, grads)}


def run(s):
    case, op = s.case, s.case["op"]
    if op == "block":
        if not case["train"]:
            with torch.no_grad():
                return {"y": s.block(s.x, case["window"])}
        y = s.block(s.x, case["window"])
        ps = list(s.block.named_parameters())
        gr = torch.autograd.grad(y, [s.x] + [p for _, p in ps], s.dy)
        return {"y": y, "dx": gr[0], **_named_grads(ps, gr[1:])}
    if op == "moe":
        y = s.moe(s.x, s.sur)
        ps = list(s.moe.named_parameters())
        gr = torch.autograd.grad([y, s.moe.aux], [s.x] + [p for _, p in ps], [s.dy, torch.full_like(s.moe.aux, 0.01)])
        return {"y": y, "aux": s.moe.aux, "dropped": s.moe.dropped, "dx": gr[0], **_named_grads(ps, gr[1:])}
    if op == "head":
        loss = ops.linear_ce(s.h, s.w, s.y, gate=s.gate, hit=s.hit) / case["N"]
        gr = torch.autograd.grad(loss, [s.h, s.w] + ([s.gate] if case["mix"] else []))
        return {"loss": loss, "dh": gr[0], "dw": gr[1], **({"dgate": gr[2]} if case["mix"] else {})}
    if op == "opt":
        for p, g in zip(s.p, s.g):
            s.opt.update(p, g)
        kept = s.opt.w if case["E"] else [p._bf16_shadow for p in s.p]
        return {"p": [p.detach() for p in s.p], "copy": list(kept), "m": list(s.opt.m)}
    if op == "locks":
        cand, on, bk, src = ops.find_locks(s.x, VOCAB, 3, s.bucket)
        return {"cand": cand, "on": on, "bucket": bk, "src": src}
    out, _ = s.model(s.x[:, :-1])
    loss = s.model.train_loss(out, s.x[:, 1:])
    ps = list(s.model.named_parameters())
    gr = torch.autograd.grad(loss, [p for _, p in ps])
    return {"out": out, "loss": loss, **_named_grads(ps, gr)}


# ------------------------------------------------------------------------------------------------ what a pass cannot do without
def _pairs(T, window):
    """Visible (query, key) pairs of one text and head."""
    W = min(T, window)
    return T * W - W * (W - 1) // 2


def _capacity(case):
    return int(1.25 * case["B"] * case["A"] * 2 / case["E"]) + 1


def work(case):
    op = case["op"]
    if op == "block":
        d, M = case["d"], case["B"] * case["T"]
        hid = 6 * d if case["relu2"] else 4 * d
        up = hid if case["relu2"] else 2 * hid
        weights = d * (4 * d + up + hid)
        attn = 4 * case["B"] * d * _pairs(case["T"], case["window"])
        if not case["train"]:
            return dict(bytes=4 * weights + 8 * M * d, flops=2 * M * weights + attn)
        return dict(bytes=2 * 4 * weights + 16 * M * d, flops=6 * M * weights + 3.5 * attn)
    if op == "moe":
        d, N, E = case["d"], case["B"] * case["A"], case["E"]
        live = E - case["frozen"]
        hid = 3 * d if case["relu2"] else 2 * d
        per = d * (hid if case["relu2"] else 2 * hid) + hid * d
        # three quarters of the places are filled on average; two experts per filled place; frozen experts' tables get no gradient
        rows = 0.75 * 2 * N
        return dict(bytes=16 * N * d + per * (4 * live + case["frozen"]), flops=2 * rows * per * (3 * live + 2 * case["frozen"]) / E)
    if op == "head":
        return dict(bytes=4 * case["N"] * case["d"] + 8 * VOCAB * case["d"], flops=6 * case["N"] * case["d"] * VOCAB)
    if op == "opt":
        d, H = case["d"], case["H"]
        n = 2 * case["E"] * d * H if case["E"] else 4 * d * d + 3 * d * H
        # read: gradient, momentum, fp32 weight; written: momentum, fp32 weight, bf16 copy
        return dict(bytes=n * (2 + 2 + 4 + 2 + 4 + 2), flops=12 * n)
    if op == "locks":
        return dict(bytes=case["B"] * case["T"] * (8 + 3 * (8 + 8 + 1) + 8), flops=0)
    d, L, M = 512, 8, case["B"] * case["T"]
    weights = L * 16 * d * d
    return dict(bytes=8 * (weights + 2 * VOCAB * d), flops=6 * M * (weights + d * VOCAB) + 3.5 * L * 4 * case["B"] * d * _pairs(case["T"], case["T"]))


def tolerance(case):
    return TOLERANCE[case["op"]]


# about four times what the path shows against itself with other summation orders and against 64 bits
TOLERANCE = {
    "block": {"rel": 2e-2},                # bf16 products and activations
    "moe": {"rel": 4e-2},                  # int8 rows of the frozen bank, bf16 elsewhere
    "head": {"rel": 2e-2},                 # bf16 logits and their gradients
    "opt": {"rel": 1e-3, "max": 2e-2},     # bf16 momentum and weight copies may round the other way
    "locks": "exact",
    "lm": {"rel": 4e-2},                   # eight layers of bf16
}


# ------------------------------------------------------------------------------------------------ the same in 64 bits
def _rms64(x, w):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + torch.finfo(torch.float32).eps) * w


def _rope64(t):
    """t (B,T,H,hd), interleaved pairs; the angles are the fp32 tables the model is defined with."""
    T, hd = t.shape[1], t.shape[3]
    inv = 1.0 / 10000.0 ** (torch.arange(0, hd, 2, device=t.device).float() / hd)
    ang = torch.arange(T, device=t.device).float()[:, None] * inv[None]
    c, s = ang.cos().double()[:, None], ang.sin().double()[:, None]
    a, b = t[..., 0::2], t[..., 1::2]
    return torch.stack([a * c - b * s, a * s + b * c], -1).flatten(-2)


def _attn64(q, k, v, window):
    """q, k, v (1,T,H,hd): causal attention over the last `window` words, block of queries by block."""
    T, hd = q.shape[1], q.shape[3]
    W = min(window, T)
    out = []
    step = 512
    for q0 in range(0, T, step):
        q1 = min(T, q0 + step)
        k0 = max(0, q0 - W + 1)
        sc = torch.einsum("qhd,khd->hqk", q[0, q0:q1], k[0, k0:q1]) * hd ** -0.5
        i, j = torch.arange(q0, q1, device=q.device)[:, None], torch.arange(k0, q1, device=q.device)[None]
        p = sc.masked_fill((j > i) | (i - j >= W), float("-inf")).softmax(-1)
        out.append(torch.einsum("hqk,khd->qhd", p, v[0, k0:q1]))
    return torch.cat(out)[None]


def _block64(x, P, heads, window, relu2):
    """One text (1,T,d) through a light block; P: name -> 64-bit weight."""
    _, T, d = x.shape
    qkv = (_rms64(x, P["n1.weight"]) @ P["qkv.weight"].t()).view(1, T, 3, heads, d // heads)
    a = _attn64(_rope64(qkv[:, :, 0]), _rope64(qkv[:, :, 1]), qkv[:, :, 2], window)
    x = x + a.reshape(1, T, d) @ P["o.weight"].t()
    u = _rms64(x, P["n2.weight"]) @ P["up.weight"].t()
    if relu2:
        h = u.relu().square()
    else:
        gate, lin = u.chunk(2, -1)
        h = F.silu(gate) * lin
    return x + h @ P["down.weight"].t()


def _leaf64(t):
    return t.detach().double().requires_grad_()


def _exact_block(s, case):
    P = {n: _leaf64(p) for n, p in s.block.named_parameters()}
    y, dx = [], []
    for b in range(case["B"]):
        x = _leaf64(s.x[b:b + 1])
        with torch.set_grad_enabled(case["train"]):
            yb = _block64(x, P, case["d"] // 64, case["window"], case["relu2"])
        y.append(yb.detach())
        if case["train"]:
            yb.backward(s.dy[b:b + 1].double())
            dx.append(x.grad)
    if not case["train"]:
        return {"y": torch.cat(y)}
    return {"y": torch.cat(y), "dx": torch.cat(dx), **{n.replace(".weight", ""): p.grad for n, p in P.items()}}


def _exact_moe(s, case):
    m, E, C = s.moe, case["E"], _capacity(case)
    d, N = case["d"], case["B"] * case["A"]
    P = {n: _leaf64(p) for n, p in m.named_parameters()}
    x = _leaf64(s.x)
    xf = _rms64(x, P["norm.weight"]).view(N, d)
    # who goes where is decided on the bf16 rows that the router sees
    seen = (xf.detach().bfloat16().double() @ P["router.weight"].detach().t())
    probs = (xf @ P["router.weight"].t()).softmax(-1)
    choice = seen.topk(2, -1).indices
    real = (s.sur.view(N) >= 0)
    top = probs.gather(1, choice)
    w = top / top.sum(-1, keepdim=True) * real[:, None]
    hot = F.one_hot(choice, E) * real[:, None, None]
    place = (hot.view(2 * N, E).cumsum(0) - hot.view(2 * N, E)).view(N, 2, E)
    served = (hot * (place < C)).bool()                                     # (N,2,E)
    cnt = hot.double().sum((0, 1))
    aux = E * (cnt / cnt.sum() * ((probs * real[:, None]).sum(0) / real.sum())).sum()
    y = torch.zeros(N, d, device=DEV, dtype=torch.float64)
    for e in range(E):
        if e in m.L:
            up, down = P["up"][m.L.index(e)], P["down"][m.L.index(e)]
        else:
            f = m.Fz.index(e)
            up = m.up_f[f].double() * m.up_fs[f].double()
            down = m.down_f[f].double() * m.down_fs[f].double()
        rows = served[:, :, e].any(1).nonzero()[:, 0]
        u = xf[rows] @ up
        if case["relu2"]:
            h = u.relu().square()
        else:
            a, b = u.chunk(2, -1)
            h = F.silu(a) * b
        mine = (w * served[:, :, e]).sum(1)[rows]
        y = y.index_add(0, rows, h @ down * mine[:, None])
    y = x + y.view_as(x)
    gr = torch.autograd.grad([y, aux], [x] + list(P.values()), [s.dy.double(), torch.full_like(aux, 0.01)])
    dropped = 1 - served.sum().double() / hot.sum()
    return {"y": y, "aux": aux, "dropped": dropped, "dx": gr[0], **_named_grads(list(P.items()), gr[1:])}


def _ce64(h, w, y, gate, hit):
    """Summed loss and gradients of the (mixture) cross-entropy, rows in chunks."""
    dh, dw, dg, total = torch.empty_like(h), torch.zeros_like(w), None if gate is None else torch.empty_like(gate), 0.0
    for i in range(0, h.shape[0], 2048):
        r = slice(i, i + 2048)
        lo = (h[r] @ w.t()).log_softmax(-1)
        n = lo.shape[0]
        at = torch.arange(n, device=h.device)
        lpy = lo[at, y[r]]
        G = lo.exp_()
        G[at, y[r]] -= 1
        if gate is None:
            total = total - lpy.sum()
        else:
            py = lpy.exp()
            mixed = (1 - gate[r]) * py + gate[r] * hit[r]
            total = total - mixed.log().sum()
            G *= ((1 - gate[r]) * py / mixed)[:, None]
            dg[r] = (py - hit[r]) / mixed
        dh[r] = G @ w
        dw += G.t() @ h[r]
    return total, dh, dw, dg


def _exact_opt(s, case):
    out = {"p": [], "copy": [], "m": []}
    lr = 6e-4 * 0.12
    for i, (p, g) in enumerate(zip(s.p, s.g)):
        rms = lambda t, a: t.pow(2).mean(a, keepdim=True).sqrt() + 1e-8
        m = 0.9 * s.opt.m[i].double() + 0.1 * g.double()
        w = (s.opt.w[i] if case["E"] else p.detach()).double()
        table = not case["E"] and p.shape[0] >= 10000          # stepped like a word table: row norm, no decay
        u = m / rms(m, 1)
        if not table:
            u = u / rms(u, 2 if case["E"] else 0)
            u = u / rms(u, 1)
        w = w * (1 if table else 1 - lr * 0.1 / 0.12) - lr * u
        out["p"].append(w)
        out["copy"].append(w)
        out["m"].append(m)
    return out


def _exact_lm(s, case):
    P = {n: _leaf64(p) for n, p in s.model.named_parameters()}
    x = F.embedding(s.x[:, :-1], P["emb.weight"])
    hs = []
    for b in range(case["B"]):
        h = x[b:b + 1]
        for l in range(8):
            own = {n[len("blocks.%d." % l):]: p for n, p in P.items() if n.startswith("blocks.%d." % l)}
            h = _block64(h, own, 8, case["T"], False)
        hs.append(h)
    out = _rms64(torch.cat(hs), P["norm.weight"])
    M = case["B"] * case["T"]
    total, dh, dw, _ = _ce64(out.detach().view(M, -1), P["head.weight"].detach(), s.x[:, 1:].reshape(-1), None, None)
    names = [n for n in P if n != "head.weight"]
    gr = dict(zip(names, torch.autograd.grad(out, [P[n] for n in names], (dh / M).view_as(out))))
    gr["head.weight"] = dw / M
    return {"out": out, "loss": total / M, **{n.replace(".weight", ""): gr[n] for n in P}}


def _exact_locks(s):
    """Last earlier occurrence of the same 1-, 2- and 3-gram, by a dictionary per text."""
    x = s.x.cpu().tolist()
    B, T = s.x.shape
    cand, on, src = (torch.zeros(B, T, 3, dtype=torch.long) for _ in range(3))
    for b in range(B):
        last = [{}, {}, {}]
        for t in range(T):
            for n in range(3):
                if t < n:
                    continue
                key = tuple(x[b][t - n:t + 1])
                j = last[n].get(key)
                if j is not None:
                    src[b, t, n], cand[b, t, n], on[b, t, n] = j + 1, x[b][j + 1], 1
                last[n][key] = t
    on[..., 0] *= (1 - on[..., 1]) * (1 - on[..., 2])
    on[..., 1] *= 1 - on[..., 2]
    return {"cand": cand, "on": on.bool(), "bucket": s.bucket.cpu()[s.x.cpu()], "src": src}


def exact(case, seed):
    s, op = prepare(case, seed), case["op"]
    if op == "block":
        return _exact_block(s, case)
    if op == "moe":
        return _exact_moe(s, case)
    if op == "head":
        N = case["N"]
        total, dh, dw, dg = _ce64(s.h.detach().double(), s.w.detach().double(), s.y,
                                  s.gate.detach().double() if case["mix"] else None, s.hit.double() if case["mix"] else None)
        return {"loss": total / N, "dh": dh / N, "dw": dw / N, **({"dgate": dg / N} if case["mix"] else {})}
    if op == "opt":
        return _exact_opt(s, case)
    if op == "locks":
        return _exact_locks(s)
    return _exact_lm(s, case)
