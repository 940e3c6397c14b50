"""The row, search, routing, optimizer and attention kernels at the sizes where they can go wrong: edges of tiles and chunks,
remainders, the smallest and largest of a range, every branch of a dispatch - against the PyTorch statements."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return ((a.double() - b.double()).norm() / b.double().norm().clamp(min=1e-30)).item()


# ------------------------------------------------------------------------------------------------ keys and locks
def _share0_words(T, count):
    """Words whose 1-gram key belongs to share 0 of a text of T words: they overflow that share's table."""
    shares, out, mask, w = T // 256 + 1, [], (1 << 64) - 1, 0
    while len(out) < count:
        k = w * 0x9E3779B97F4A7C15 & mask
        k ^= k >> 29
        h = (k * 0xBF58476D1CE4E5B9 & mask) >> 32
        if h * shares >> 32 == 0:
            out.append(w)
        w += 1
    return torch.tensor(out)


@pytest.mark.parametrize("text", ["zipf", "same", "pair", "distinct", "overflow"])
@pytest.mark.parametrize("B,T,n_keys", [(1, 1, 3), (3, 2, 2), (2, 5, 3), (3, 127, 1), (2, 128, 3), (2, 257, 3), (2, 4099, 3), (1, 30000, 3), (1, 30001, 3)])
def test_lock_find_tables_and_scan(text, B, T, n_keys):
    from memarch_b200.ops import anchors, ref
    g = torch.Generator().manual_seed(T)
    V = 1 << 20
    if text == "zipf":
        x = (torch.exp(torch.rand(B, T, generator=g) * 8).long() - 1)
    elif text == "same":
        x = torch.full((B, T), V - 1)
    elif text == "pair":
        x = (torch.arange(T)[None] % 2 + torch.arange(B)[:, None]).long()
    elif text == "distinct":
        x = torch.stack([torch.randperm(max(T, 8), generator=g)[:T] for _ in range(B)])
    else:
        words = _share0_words(T, 700)
        x = words[torch.randint(0, 700, (B, T), generator=g)]
    bucket = torch.randint(0, 9, (1000,), generator=g)
    for lb in (None, bucket):
        got = anchors.find_locks(x.cuda(), V, n_keys, None if lb is None else lb.cuda())
        want = ref.find_locks(x, V, max(n_keys, 2), lb)
        for a, b, per_key in zip(got, want, (True, True, False, True)):
            if per_key and n_keys == 1:
                continue                                        # the statement has at least two key lengths
            assert torch.equal(a.cpu(), b)
    if n_keys == 1:
        got, want = anchors.find_locks(x.cuda(), V, 1, None), ref.find_locks(x, V, 2, None)
        assert torch.equal(got[0][..., 0].cpu(), want[0][..., 0]) and torch.equal(got[3][..., 0].cpu(), want[3][..., 0])


@pytest.mark.parametrize("B,T", [(2, 700), (1, 1), (1, 30001)])
def test_lock_buckets_of_ids_outside_the_table(B, T):
    """Tables and scan: ids past the table take its last entry, negative ones count from its end, ids below that set the status
    word; memory before the table is never read."""
    from memarch_b200.ops import _ext, anchors, ref
    g = torch.Generator().manual_seed(T)
    x = torch.randint(-40, 90, (B, T), generator=g)
    x[0, 0] = -40
    bucket = torch.randint(0, 9, (40,), generator=g)
    mem = torch.full((120,), -77)                        # entries around the table that must not turn up
    mem[40:80] = bucket
    table = mem.cuda()[40:80]
    got, want = anchors.find_locks(x.cuda(), 50304, 3, table), ref.find_locks(x, 50304, 3, bucket)
    for a, b in zip(got, want):
        assert torch.equal(a.cpu(), b)
    assert _ext.C().lock_status(0) == 0
    x[-1, -1] = -41
    bk = anchors.find_locks(x.cuda(), 50304, 3, table)[2]
    assert bk[-1, -1].item() == bucket[0].item() and _ext.C().lock_status(0) == 1 and _ext.C().lock_status(0) == 0


@pytest.mark.parametrize("T", [40, 2500])
@pytest.mark.parametrize("low", [-(1 << 20), -(1 << 20) - 1, (1 << 21) - 3, 1 << 30, (1 << 31) - 12])
def test_lock_ids_outside_the_vocabulary(T, low):
    """Words are told apart by their whole id, also where ids differ by a multiple of 2^21."""
    from memarch_b200.ops import anchors, ref
    g = torch.Generator().manual_seed(T)
    x = torch.randint(0, 6, (2, T), generator=g) + torch.where(torch.rand(2, T, generator=g) < 0.5, low, low + (1 << 21) if low < 1 << 30 else 3)
    x[1] = torch.randint(0, 6, (T,), generator=g)         # the other text is an ordinary one
    ids, compact = x.unique(return_inverse=True)          # the statement packs n-grams into 64 bits: small ids for it
    cand, on, bk, src = ref.find_locks(compact, ids.numel(), 3, None)
    want = torch.where(src > 0, ids[cand], torch.zeros_like(cand)), on, bk, src
    for a, b in zip(anchors.find_locks(x.cuda(), 50304, 3, None), want):
        assert torch.equal(a.cpu(), b)


# ------------------------------------------------------------------------------------------------ RMSNorm, cross-entropy rows
@pytest.mark.parametrize("n,d", [(1, 8), (3, 256), (5, 264), (17, 512), (9, 520), (33, 1024), (2, 1032), (700, 2048), (3, 2056), (4, 4096), (5, 4104), (2, 8192), (3, 8200), (5000, 64)])
def test_rmsnorm_widths(n, d):
    from memarch_b200.ops import _ext
    C = _ext.C()
    g = torch.Generator(device="cuda").manual_seed(d)
    x, w = torch.randn(n, d, device="cuda", generator=g), torch.rand(d, device="cuda", generator=g) + 0.5
    y, dy, add = (torch.randn(n, d, device="cuda", generator=g) for _ in range(3))
    yb, dyb = y.bfloat16(), dy.bfloat16()
    xs = (x.double() + yb.double()).requires_grad_()
    wd = w.double().requires_grad_()
    ref = xs * torch.rsqrt(xs.pow(2).mean(-1, keepdim=True) + 1e-6) * wd
    h, out, rstd = C.add_rmsnorm_fwd(x, yb, w, 1e-6)
    assert _rel(h, xs.detach()) < 1e-6 and _rel(out, ref.detach()) < 4e-3           # bf16 rounding: 2^-9 per element
    out32, _ = C.rmsnorm_fwd(h, w, 1e-6, False)
    assert _rel(out32, ref.detach()) < 1e-6
    outb, _ = C.rmsnorm_fwd(h.bfloat16(), w, 1e-6, True)
    assert _rel(outb, ref.detach()) < 8e-3
    if d > 8192:
        return
    ref.backward(dyb.double())
    for a in (None, add):
        dx, dw, lo = C.rmsnorm_bwd(dyb, h, w, rstd, a, True)
        want = xs.grad if a is None else xs.grad + a.double()
        assert _rel(dx, want) < 1e-5 and _rel(lo, want) < 4e-3 and _rel(dw, wd.grad) < 1e-5


@pytest.mark.parametrize("n,V", [(1, 8), (3, 9), (5, 4096), (4, 16384 + 8), (2, 16389), (3, 50304)])
def test_ce_rows_sizes(n, V):
    from memarch_b200.ops import _ext
    g = torch.Generator(device="cuda").manual_seed(V)
    lg = torch.empty(n, (V + 7) // 8 * 8, device="cuda", dtype=torch.bfloat16)[:, :V]
    lg.copy_(torch.randn(n, V, device="cuda", generator=g) * 4)
    y = torch.randint(0, V, (n,), device="cuda", generator=g)
    y[0], y[-1] = V - 1, 0
    x = lg.double().requires_grad_()
    loss = torch.nn.functional.cross_entropy(x, y, reduction="none")
    loss.sum().backward()
    out = torch.empty(n, device="cuda")
    _ext.C().ce_rows(lg, y, out, None, None, None)
    assert _rel(out, loss.detach()) < 1e-5 and _rel(lg, x.grad) < 4e-3


# ------------------------------------------------------------------------------------------------ split contraction
@pytest.mark.parametrize("M,N,K", [(256, 8, 2048), (264, 256, 2056), (1000, 256, 50304), (512, 1536, 4096), (300, 264, 8200), (2048, 2048, 2048)])
def test_gemm_split_contraction(M, N, K):
    """Few output tiles and a long contraction: all operand layouts, bf16 / fp32 / accumulating outputs."""
    from memarch_b200.ops import gemm
    g = torch.Generator(device="cuda").manual_seed(K)
    A, B = (torch.randn(r, K, device="cuda", generator=g).bfloat16() for r in (M, N))
    want = A.double() @ B.double().t()
    for a_mn in (False, True):
        for b_mn in (False, True):
            a = A.t().contiguous() if a_mn else A
            b = B.t().contiguous() if b_mn else B
            if (a_mn and M % 8) or (b_mn and N % 8):
                continue
            assert _rel(gemm(a, b, a_mn=a_mn, b_mn=b_mn), want) < 4e-3
            assert _rel(gemm(a, b, a_mn=a_mn, b_mn=b_mn, out_dtype=torch.float32), want) < 1e-5
            acc = torch.ones(M, N, device="cuda")
            gemm(a, b, a_mn=a_mn, b_mn=b_mn, out=acc, out_dtype=torch.float32, accumulate=True)
            assert _rel(acc, want + 1) < 1e-5


@pytest.mark.parametrize("M,N,K", [(256, 8, 2048), (1000, 256, 50304), (256, 1024, 2048), (512, 1536, 4096), (300, 264, 8200)])
def test_gemm_split_contraction_repeats(M, N, K):
    """The parts of a cut contraction are added in a fixed order: the same call gives the same bits."""
    from memarch_b200.ops import gemm
    g = torch.Generator(device="cuda").manual_seed(N)
    a, b = (torch.randn(r, K, device="cuda", generator=g).bfloat16() for r in (M, N))
    for kw in (dict(), dict(out_dtype=torch.float32), dict(out_dtype=torch.float32, accumulate=True)):
        def call():
            out = torch.full((M, N), 0.5, device="cuda") if "accumulate" in kw else None
            return gemm(a, b, out=out, **kw)
        first = call()
        assert all(torch.equal(call(), first) for _ in range(20))


@pytest.mark.parametrize("K,kernels", [(1024, 1), (4096, 2)])
def test_launches_of_split_products_are_counted(K, kernels):
    from memarch_b200.ops import _ext, gemm
    a, b = (torch.zeros(512, K, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    n = _ext.launches()
    gemm(a, b)
    assert _ext.launches() - n == kernels


@pytest.mark.parametrize("M,N,K,kernels", [(256, 256, 1984, 1), (256, 256, 1985, 2), (1024, 1024, 2048, 1), (1024, 1024, 3072, 2), (4096, 512, 2048, 1), (4096, 512, 3072, 1),
                                           (4096, 512, 4096, 2), (255, 256, 8192, 1), (9472, 256, 16384, 2), (9473, 256, 16384, 1)])
def test_products_are_cut_where_it_pays(M, N, K, kernels):
    """The line between whole and cut products (a cut one is two kernels), and the result on both sides of it."""
    from memarch_b200.ops import _ext, gemm
    K8 = (K + 7) // 8 * 8
    g = torch.Generator(device="cuda").manual_seed(M)
    a, b = torch.randn(M, K8, device="cuda", generator=g).bfloat16(), torch.randn(N, K8, device="cuda", generator=g).bfloat16()
    n = _ext.launches()
    out = gemm(a, b)
    assert _ext.launches() - n == kernels
    rows = torch.arange(0, M, max(1, M // 64), device="cuda")
    assert _rel(out[rows], a[rows].double() @ b.double().t()) < 4e-3


# ------------------------------------------------------------------------------------------------ narrow tiles
@pytest.mark.parametrize("M,N,K", [(2048, 256, 256), (257, 264, 128), (4095, 512, 520), (1001, 136, 64), (256, 1024, 2048), (9472, 256, 64), (513, 8, 16)])
def test_gemm_narrow_tiles(M, N, K):
    """128-column tiles and their neighbours under the rule, any number of rows: plain, relu2 and SwiGLU epilogues both ways."""
    from memarch_b200.ops import gemm, linear
    from memarch_b200.ops.basic import ffn
    g = torch.Generator(device="cuda").manual_seed(M)
    x, w = torch.randn(M, K, device="cuda", generator=g).bfloat16(), torch.randn(N, K, device="cuda", generator=g) * K ** -0.5
    wd = torch.randn(K, N // 2, device="cuda", generator=g) * N ** -0.5
    go = torch.randn(M, N, device="cuda", generator=g).bfloat16()
    xd, w2 = x.double(), w.bfloat16().double()
    assert _rel(gemm(x, w.bfloat16()), xd @ w2.t()) < 4e-3
    assert _rel(gemm(x, w.bfloat16(), out_dtype=torch.float32), xd @ w2.t()) < 1e-5
    xg, wg = x.clone().requires_grad_(), w.clone().requires_grad_()
    linear(xg, wg).backward(go)
    assert _rel(xg.grad, go.double() @ w2) < 4e-3 and _rel(wg.grad, go.double().t() @ xd) < 4e-3
    for act in ("swiglu", "relu2"):
        H = N // 2 if act == "swiglu" else N
        down = wd if act == "swiglu" else torch.cat([wd, wd], 1)
        gy = torch.randn(M, K, device="cuda", generator=g).bfloat16()
        got, want = [], []
        for native in (True, False):
            a, u, v = x.clone(), w.clone(), down.clone()
            if not native:
                a, u, v = xd.clone(), w2.clone(), down.bfloat16().double()
            a.requires_grad_(), u.requires_grad_(), v.requires_grad_()
            if native:
                y = ffn(a, u, v, act)
            else:
                p = a @ u.t()
                y = (torch.nn.functional.silu(p[:, :H]) * p[:, H:] if act == "swiglu" else p.relu().square()) @ v.t()
            y.backward(gy.to(y.dtype))
            (got if native else want).extend([y, a.grad, u.grad, v.grad])
        # bf16 hidden activations and pre-activations: two to three roundings of 2^-9 along the chain
        for q, r in zip(got, want):
            assert _rel(q, r) < 1e-2


@pytest.mark.parametrize("M", [128, 129, 133, 200, 255])
@pytest.mark.parametrize("act", [None, "swiglu", "relu2"])
def test_few_ragged_rows_on_the_single_cta_kernel(M, act):
    """128 to 255 rows, most of them no multiple of 8: plain and activation epilogues, input and weight gradients."""
    from memarch_b200.ops import basic
    g = torch.Generator(device="cuda").manual_seed(M)
    K, H = 136, 72
    N = 2 * H if act == "swiglu" else H * 2
    x = torch.randn(M, K, device="cuda", generator=g).bfloat16()
    w = (torch.randn(N, K, device="cuda", generator=g) * K ** -0.5).bfloat16()
    res = []
    for own in (True, False):
        a, u = (t.clone() if own else t.double() for t in (x, w))
        a.requires_grad_(), u.requires_grad_()
        if own:
            y = basic.linear(a, u) if act is None else basic.linear_act(a, u, act)
        else:
            p = a @ u.t()
            y = p if act is None else torch.nn.functional.silu(p[:, :H]) * p[:, H:] if act == "swiglu" else p.relu().square()
        go = torch.randn(y.shape, device="cuda", generator=torch.Generator(device="cuda").manual_seed(3)).bfloat16()
        y.backward(go.to(y.dtype))
        res.append([y.detach(), a.grad, u.grad])
    # bf16 pre-activations, activations and their gradients: two to three roundings of 2^-9 along the chain
    for p, q in zip(*res):
        assert _rel(p, q) < 1e-2


# ------------------------------------------------------------------------------------------------ routing
@pytest.mark.parametrize("N,d,E,k,C", [(1, 8, 1, 1, 1), (31, 64, 3, 2, 7), (33, 256, 8, 2, 64), (100, 264, 48, 4, 3), (700, 2048, 8, 2, 176), (257, 512, 128, 8, 9), (4000, 768, 16, 2, 626)])
def test_route_and_slot_fused(N, d, E, k, C):
    """Every output and both gradients of the fused router against the PyTorch statement (fp32 router product)."""
    from memarch_b200 import ops
    from memarch_b200.ops import ref
    g = torch.Generator().manual_seed(N + E)
    x = torch.randn(N, d, generator=g).bfloat16()
    w = torch.randn(E, d, generator=g) * d ** -0.5
    real = torch.rand(N, generator=g) > 0.2
    k_tok = torch.randint(1, k + 1, (N,), generator=g) * real
    gw, gt, gp = torch.randn(N, k, generator=g), torch.randn(E * C, generator=g), torch.randn(N, E, generator=g)
    xc, wc = x.float().requires_grad_(), w.clone().requires_grad_()
    probs, top_e, keep, wt, e_flat, aux = ref.moe_route(xc, wc, real, k_tok, k, E)
    table, _, flat, dropped = ref.moe_slots(e_flat, wt.detach(), E, C)
    ok = flat < E * C
    wtab = torch.zeros(E * C + 1).scatter(0, flat.reshape(-1), (wt * ok).reshape(-1))[:-1]
    ((wt * gw).sum() + (wtab * gt).sum() + (probs * gp).sum() + 3 * aux).backward()
    xg, wg = x.cuda().requires_grad_(), w.cuda().requires_grad_()
    o = ops.route_and_slot(xg, wg, real.cuda(), k_tok.cuda(), k, E, C, want_counts=True)
    assert torch.equal(o[1].cpu(), table) and torch.equal(o[3].cpu(), flat)
    assert torch.equal(o[7].cpu().long(), torch.bincount(flat[ok] // C, minlength=E))
    for a, b in ((o[0], wt), (o[2], wtab), (o[6], probs)):
        assert (a.cpu() - b).abs().max() < 1e-5
    assert abs(float(o[4]) - float(aux)) < 1e-5 * max(1.0, float(aux)) and abs(float(o[5]) - float(dropped)) < 1e-6
    ((o[0] * gw.cuda()).sum() + (o[2] * gt.cuda()).sum() + (o[6] * gp.cuda()).sum() + 3 * o[4]).backward()
    assert _rel(xg.grad.cpu(), xc.grad) < 4e-3 and _rel(wg.grad.cpu(), wc.grad) < 1e-4


@pytest.mark.parametrize("N,E,k,C", [(32768, 8, 2, 9000), (32769, 8, 2, 8000), (70001, 64, 4, 4000), (40000, 128, 8, 2500), (33000, 1, 1, 30000)])
def test_route_places_of_many_tokens(N, E, k, C):
    """Both sides of the line from which on the blocks' numbers are added up once: places, filled counts, dropped share and the auxiliary
    loss from the kernel's own choices."""
    from memarch_b200 import ops
    from memarch_b200.ops import ref
    g = torch.Generator(device="cuda").manual_seed(N)
    x = torch.randn(N, 16, device="cuda", generator=g).bfloat16()
    w = torch.randn(E, 16, device="cuda", generator=g) * 0.5
    real, k_tok = torch.rand(N, device="cuda", generator=g) > 0.2, torch.randint(0, k + 1, (N,), device="cuda", generator=g)
    wt, table, wtab, flat, aux, dropped, probs, counts = ops.route_and_slot(x, w, real, k_tok, k, E, C, want_counts=True)
    top = probs.topk(k, 1).indices
    keep = torch.arange(k, device="cuda")[None] < k_tok[:, None]
    e_flat = torch.where(keep, top, torch.full_like(top, E))
    t2, _, f2, d2 = ref.moe_slots(e_flat.cpu(), wt.detach().cpu(), E, C)
    assert torch.equal(table.cpu(), t2) and torch.equal(flat.cpu(), f2) and abs(float(dropped) - float(d2)) < 1e-6
    cnt = torch.bincount(e_flat[keep], minlength=E)
    assert torch.equal(counts.long(), cnt.clamp(max=C))
    want = E * (cnt.double() / cnt.sum() * (probs.double() * real[:, None]).sum(0) / real.sum()).sum()
    assert abs(float(aux) - float(want)) < 1e-4 * float(want)


@pytest.mark.parametrize("N,d,E", [(8192, 2048, 8), (5000, 264, 16), (40000, 512, 128)])
def test_router_gradients_repeat(N, d, E):
    """The router weight's gradient is summed over the tokens in a fixed order: the same call gives the same bits.  The last size
    has runs of more than 64 tokens."""
    from memarch_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(N)
    x = torch.randn(N, d, device="cuda", generator=g).bfloat16()
    w = torch.randn(E, d, device="cuda", generator=g) * d ** -0.5
    real, k_tok = torch.rand(N, device="cuda", generator=g) > 0.1, torch.full((N,), 2, device="cuda")
    gw, gp = torch.randn(N, 2, device="cuda", generator=g), torch.randn(N, E, device="cuda", generator=g)

    def grads():
        xg, wg = x.clone().requires_grad_(), w.clone().requires_grad_()
        o = ops.route_and_slot(xg, wg, real, k_tok, 2, E, N // E)
        torch.autograd.backward([o[0], o[6]], [gw, gp])
        return xg.grad, wg.grad
    first = grads()
    for _ in range(10):
        assert all(torch.equal(a, b) for a, b in zip(grads(), first))
    # against the sum over the tokens in 64 bits, from the same gradient of the logits
    p = torch.softmax(x.double() @ w.double().t(), 1).requires_grad_()
    top, idx = p.topk(2, 1)
    dp, = torch.autograd.grad([top / top.sum(1, keepdim=True), p], p, [gw.double(), gp.double()])
    dl = p.detach() * (dp - (dp * p.detach()).sum(1, keepdim=True))
    assert _rel(first[1], dl.t() @ x.double()) < 1e-4


# ------------------------------------------------------------------------------------------------ expert rows
@pytest.mark.parametrize("N,d,E,C,k", [(1, 8, 1, 1, 1), (37, 264, 3, 7, 2), (300, 1032, 8, 64, 2), (65, 2048, 4, 33, 4), (50, 100, 2, 9, 2), (500, 768, 2, 100, 8)])
def test_expert_row_moves(N, d, E, C, k):
    """Gather, weighted combine and their gradients with empty places, dropped and unwanted choices; widths that are no multiple
    of 8 take the element-wise kernels."""
    from memarch_b200.ops import moe as ops_moe
    g = torch.Generator().manual_seed(N * d)
    S = E * C
    place = torch.randperm(max(S, N * k) + 3, generator=g)[:N * k].view(N, k)
    flat = torch.where(place < S, place, torch.full_like(place, S))
    table = torch.full((S + 1,), N)
    table[flat.reshape(-1)] = torch.arange(N)[:, None].expand(N, k).reshape(-1)
    table = table[:-1].contiguous()
    x, ye, w = torch.randn(N, d, generator=g).bfloat16(), torch.randn(S, d, generator=g).bfloat16(), torch.rand(S, generator=g)
    gx, go = torch.randn(S, d, generator=g).bfloat16(), torch.randn(N, d, generator=g).bfloat16()
    res = []
    for dev in ("cuda", "cpu"):
        a, b, c = (t.to(dev).clone().requires_grad_() for t in (x, ye, w))
        f, t = flat.to(dev), table.to(dev)
        xe = ops_moe.slot_gather(a, t, f)
        y = ops_moe.combine(b, c, f, t, N)
        xe.backward(gx.to(dev)), y.backward(go.to(dev))
        res.append([xe, y, a.grad, b.grad, c.grad])
    for i, (a, b) in enumerate(zip(*res)):
        assert a.dtype == b.dtype and a.shape == b.shape
        if i == 0:
            assert torch.equal(a.cpu(), b)
        else:
            assert _rel(a.cpu(), b) < 4e-3


@pytest.mark.parametrize("E,C,d", [(1, 1, 8), (3, 7, 264), (8, 1025, 768), (5, 63, 2048), (2, 9, 100)])
def test_expert_error_probe(E, C, d):
    from memarch_b200.models.moe import _ErrProbe
    g = torch.Generator(device="cuda").manual_seed(C)
    x = torch.randn(E, C, d, device="cuda", generator=g).bfloat16().requires_grad_()
    grad = torch.randn(E, C, d, device="cuda", generator=g).bfloat16()
    buf = torch.rand(E, device="cuda", generator=g)
    want = 0.9 * buf.double() + 0.1 * grad.double().norm(dim=-1).mean(1)
    _ErrProbe.apply(x, buf).backward(grad)
    assert torch.equal(x.grad, grad) and (buf.double() - want).abs().max() < 1e-5 * want.max()


# ------------------------------------------------------------------------------------------------ frozen bank
@pytest.mark.parametrize("E,C,d", [(3, 7, 264), (8, 1025, 768), (2, 9, 100), (2, 1, 9)])
def test_bank_group_moves(E, C, d):
    """Groups to the learning and the frozen experts and back; groups that are no multiple of 16 bytes take the general ops."""
    from memarch_b200.models.moe import _JoinGroups, _SplitGroups
    g = torch.Generator(device="cuda").manual_seed(C)
    x = torch.randn(E, C, d, device="cuda", generator=g).bfloat16().requires_grad_()
    grad = torch.randn(E, C, d, device="cuda", generator=g).bfloat16()
    order = torch.randperm(E, device="cuda", generator=g)
    l, f = order[:E // 2].contiguous(), order[E // 2:].contiguous()
    xl, xf = _SplitGroups.apply(x, l, f)
    assert torch.equal(xl, x[l]) and torch.equal(xf, x[f])
    y = _JoinGroups.apply(xl * 2, xf * 3, l, f)
    y.backward(grad)
    scale = torch.full((E, 1, 1), 2.0, device="cuda").index_fill_(0, f, 3.0).bfloat16()
    assert torch.equal(y, x * scale) and torch.equal(x.grad, grad * scale)


@pytest.mark.parametrize("F,I,O", [(1, 1, 8), (3, 33, 264), (4, 768, 1536)])
def test_bank_dequantise(F, I, O):
    from memarch_b200.ops import _ext
    g = torch.Generator(device="cuda").manual_seed(I)
    q = torch.randint(-127, 128, (F, I, O), device="cuda", generator=g).to(torch.int8)
    s = torch.rand(F, 1, O, device="cuda", generator=g).bfloat16()
    assert torch.equal(_ext.C().dequant_i8(q, s), q.to(torch.bfloat16) * s)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("R,K", [(1, 8), (9, 264), (2000, 1536), (5, 100)])
def test_quantised_rows(R, K, dtype):
    """Both row kernels and the PyTorch statement give the same bytes (zero rows and the largest element included)."""
    from memarch_b200.ops import _ext, int8
    g = torch.Generator(device="cuda").manual_seed(K)
    x = (torch.randn(R, K, device="cuda", generator=g) * 3).to(dtype)
    x[R // 2] = 0
    q, s = int8.quant_rows(x)
    q0, s0 = _ext.C().quant_rows_i8(x)
    assert torch.equal(q, q0) and torch.equal(s, s0)


@pytest.mark.parametrize("act", ["swiglu", "relu2"])
@pytest.mark.parametrize("E,C,d,H", [(2, 255, 64, 64), (2, 256, 64, 64), (3, 300, 128, 200), (1, 513, 72, 136)])
def test_expert_ffn_backward_epilogue(E, C, d, H, act):
    from memarch_b200.ops.moe import expert_ffn
    g = torch.Generator(device="cuda").manual_seed(C)
    x = torch.randn(E, C, d, device="cuda", generator=g).bfloat16()
    up = (torch.randn(E, d, 2 * H if act == "swiglu" else H, device="cuda", generator=g) * d ** -0.5).bfloat16()
    down = (torch.randn(E, H, d, device="cuda", generator=g) * H ** -0.5).bfloat16()
    gy = torch.randn(E, C, d, device="cuda", generator=g).bfloat16()
    res = []
    for native in (True, False):
        t = [v.clone() if native else v.double() for v in (x, up, down)]
        [v.requires_grad_() for v in t]
        if native:
            y = expert_ffn(*t, act)
        else:
            p = t[0] @ t[1]
            y = (torch.nn.functional.silu(p[..., :H]) * p[..., H:] if act == "swiglu" else p.relu().square()) @ t[2]
        y.backward(gy.to(y.dtype))
        res.append([y] + [v.grad for v in t])
    # bf16 activations, pre-activations and their gradients: two to three roundings of 2^-9 along the chain
    for a, b in zip(*res):
        assert _rel(a, b) < 1e-2


# ------------------------------------------------------------------------------------------------ optimizer
@pytest.mark.parametrize("shape,bf16", [((1190, 2048), False), ((1200, 1540), True), ((2500, 6144), True), ((1300, 4100), False), ((1024, 4096), False),
                                        ((3072, 1024), False), ((5, 700, 1540), True), ((3, 640, 2304), True), ((12000, 512), False), ((260, 256), False),
                                        ((4, 1024, 256), True), ((4, 592, 256), True), ((3, 789, 256), True), ((2500, 256), False)])
def test_instinct_streamed_forms(shape, bf16):
    """One step on the kernels against the PyTorch statement: whole and cut rows, expert borders inside a block, all width classes."""
    from memarch_b200.config import OptConfig
    from memarch_b200.optim import Instinct
    g = torch.Generator(device="cuda").manual_seed(sum(shape))
    p0 = torch.randn(*shape, device="cuda", generator=g) * 0.05
    grad = (torch.randn(*shape, device="cuda", generator=g) * 1e-3).bfloat16()
    m0 = torch.randn(*shape, device="cuda", generator=g) * 1e-3
    got = []
    for own in (True, False):
        p = torch.nn.Parameter(p0.bfloat16() if bf16 else p0.clone())
        opt = Instinct([p], OptConfig(lr=1e-2, norm="hs", scale=0.12, m_bf16=True, rel_every=1 << 30))
        opt.n_step = 1
        opt.m[0].copy_(m0)
        kind, wd, vocab = opt.spec(p)
        opt._sync_lr()
        with torch.no_grad():
            (opt._update_cuda if own else opt._update_ref)(0, p, grad, kind, 0.1 if wd else 0.0, opt._lr_t, False)
        got.append((opt.w[0] if bf16 else p.detach(), opt.m[0]))
    step = (got[1][0] - (p0.bfloat16().float() if bf16 else p0))
    assert ((got[0][0] - got[1][0]).norm() / step.norm()).item() < 1e-4          # fp32 sums in another order
    # the momentum does not depend on them, but the kernels form 1 - beta in fp32 (2.4e-7 off 0.1 relative) and fuse a
    # multiply-add: the fp32 value moves by less than 1e-7 |g|, its bf16 rounding by one ulp (2^-7 of the value) at most
    a, b = got[0][1].float(), got[1][1].float()
    assert ((a - b).abs() <= 2.0 ** -7 * b.abs() + 1e-7 * grad.float().abs()).all()


@pytest.mark.parametrize("norm,shape", [("row", (1024, 4096)), ("row", (3000, 2048)), ("row", (64, 65536)), ("tensor", (1024, 2048)), ("hs", (12000, 512))])
def test_instinct_row_norms_repeat(norm, shape):
    """Steps whose norms are taken over rows or the whole weight alone (the last one is a word table) give the same bits on every call."""
    from memarch_b200.config import OptConfig
    from memarch_b200.optim import Instinct
    g = torch.Generator(device="cuda").manual_seed(shape[0])
    p0, grad = torch.randn(*shape, device="cuda", generator=g) * 0.05, (torch.randn(*shape, device="cuda", generator=g) * 1e-3).bfloat16()
    m0, res = torch.randn(*shape, device="cuda", generator=g) * 1e-3, []
    for _ in range(8):
        p = torch.nn.Parameter(p0.clone())
        opt = Instinct([p], OptConfig(lr=1e-2, norm=norm, scale=0.12, m_bf16=True, rel_every=1 << 30))
        opt.n_step = 1
        opt.m[0].copy_(m0)
        kind, wd, vocab = opt.spec(p)
        assert kind in ("row", "tensor", "vocab")
        opt._sync_lr()
        with torch.no_grad():
            opt._update_cuda(0, p, grad, kind, 0.1 if wd else 0.0, opt._lr_t, False)
        res.append(p.detach().clone())
    assert all(torch.equal(a, res[0]) for a in res[1:])


# ------------------------------------------------------------------------------------------------ attention
@pytest.mark.parametrize("B,T,H,window,half", [(1, 1, 1, 0, False), (2, 63, 3, 0, True), (1, 64, 2, 0, False), (2, 65, 1, 0, False), (1, 127, 3, 5, True), (2, 128, 2, 0, True),
                                               (2, 129, 2, 0, False), (1, 300, 2, 1, False), (1, 511, 2, 64, False), (1, 700, 2, 100, True), (2, 900, 3, 129, False),
                                               (8, 260, 20, 0, False), (6, 520, 24, 0, True), (10, 400, 20, 130, False)])
def test_attention_on_packed_projections(B, T, H, window, half):
    """Rotation, attention and the gradient of the packed projections; the last three have more tiles than CTAs, in pairs
    (causal, odd and even numbers of tiles) and singly (window)."""
    from memarch_b200.ops import _ext, ref
    from memarch_b200.ops.attention import _QkvAttn
    g = torch.Generator(device="cuda").manual_seed(T)
    qkv = torch.randn(B, T, 3, H, 64, device="cuda", generator=g).bfloat16().requires_grad_()
    go = torch.randn(B, T, H * 64, device="cuda", generator=g).bfloat16()
    o = _QkvAttn.apply(qkv, window, half)
    o.backward(go)
    torch.cuda.synchronize()
    assert _ext.C().attn_status_read() == 0 and _ext.C().attn_bwd_status_read() == 0
    x = qkv.detach().float().requires_grad_()
    r = ref.window_attention(x[:, :, 0], x[:, :, 1], x[:, :, 2], window or None, half).reshape(B, T, H * 64)
    r.backward(go.float())
    assert _rel(o, r.detach()) < 1e-2                                             # bf16 q, k, P and output
    for i in range(3):
        a, b = qkv.grad[:, :, i], x.grad[:, :, i]
        assert (a.double() - b.double()).norm() < 2e-2 * max(b.double().norm(), 1e-2 * x.grad.double().norm()), i


def _held():
    return torch.cuda.memory_stats()["requested_bytes.all.current"]


@pytest.mark.parametrize("window", [0, 100])
@pytest.mark.parametrize("half", [False, True])
def test_attention_keeps_one_packed_array(window, half):
    """What stays on the device for the backward pass: the output, its log-sums and one packed array with q and k rotated; without a
    backward pass the result alone.  The projections themselves are not written to."""
    from memarch_b200.ops.attention import _QkvAttn
    leaf = torch.randn(2, 500, 3, 8, 64, device="cuda").bfloat16().requires_grad_()
    _QkvAttn.apply(leaf.detach(), window, half)                       # the rotation's tables
    size = lambda t: t.numel() * t.element_size()
    for grad in (False, True):
        with torch.set_grad_enabled(grad):
            m0 = _held()
            qkv = leaf * 1.0
            before = qkv.detach().clone()
            o = _QkvAttn.apply(qkv, window, half)
            assert torch.equal(qkv, before)
            del qkv, before                                           # the caller is done with the projections
            assert _held() - m0 <= size(o) + grad * (size(leaf) + 2 * 8 * 500 * 4) + 4 * 512
            del o


def test_light_layer_keeps_one_packed_array():
    """The attention half keeps the norm's output, one packed array, the attention's output and its result."""
    from memarch_b200.models.blocks import LightBlock
    from memarch_b200.ops import layer
    M, d = 2 * 512, 512
    with torch.device("cuda"):
        b = LightBlock(d, 8)
    x = torch.randn(2, 512, d, device="cuda", requires_grad=True)
    run = lambda: layer.attn_half(x, None, b.n1.weight, b.qkv.weight, b.o.weight, 1e-6, 0, False)
    run()                                                             # the weights' bf16 copies
    m0 = _held()
    out = run()
    kept = _held() - m0
    assert len(out) == 2 and kept <= (2 + 6 + 2 + 2) * M * d + (8 + 1) * M * 4 + 8 * 512


# ------------------------------------------------------------------------------------------------ light layer halves
@pytest.mark.parametrize("d,B,T,window,blk,half,defer", [(128, 2, 129, 64, (), False, True), (256, 1, 257, 2048, ("relu2",), False, False), (64, 3, 100, 7, (), True, False),
                                                         (128, 1, 600, 2048, (), False, True), (192, 2, 300, 128, ("relu2",), True, True)])
@pytest.mark.parametrize("mode", ["train", "first", "sink", "eval"])
def test_light_layer_halves_match_single_ops(monkeypatch, d, B, T, window, blk, half, defer, mode):
    """One native call per half against the sequence of single ops: outputs, gradients, gradients handed to the optimizer;
    lengths that the own attention does not serve take the feed-forward half alone."""
    from memarch_b200.models.blocks import LightBlock
    from memarch_b200.ops import basic, layer
    torch.manual_seed(d + T)
    with torch.device("cuda"):
        b = LightBlock(d, d // 64, blk, rope_half=half)
    x0 = torch.randn(B, T, d, device="cuda")
    p0 = None if mode == "first" else torch.randn(B, T, d, device="cuda").bfloat16()
    go, gy = torch.randn(B, T, d, device="cuda"), torch.randn(B, T, d, device="cuda").bfloat16()
    res = []
    for native in (True, False):
        if not native:
            monkeypatch.setattr(layer, "attn_half_ok", lambda *a: False)
            monkeypatch.setattr(layer, "ffn_half_ok", lambda *a: False)
        taken = {}
        if mode == "sink":
            monkeypatch.setattr(basic, "WEIGHT_GRAD_SINK", lambda w, g: taken.__setitem__(id(w), g.clone()) or g.dtype == torch.bfloat16)
        b.zero_grad(set_to_none=True)
        if mode == "eval":
            with torch.no_grad():
                out = b(x0, window, p0, defer)
            res.append(list(out) if defer else [out])
            continue
        x, p = x0.clone().requires_grad_(), None if p0 is None else p0.clone().requires_grad_()
        out = b(x, window, p, defer)
        torch.autograd.backward(list(out) if defer else [out], [go, gy] if defer else [go])
        grads = [x.grad] + ([] if p is None else [p.grad])
        for w in b.parameters():
            if mode == "sink" and w.dim() == 2:
                assert w.grad is None and taken[id(w)].dtype == torch.bfloat16
                grads.append(taken[id(w)])
            else:
                grads.append(w.grad)
        res.append((list(out) if defer else [out]) + grads)
    for a, c in zip(*res):
        # the same kernels on the same bf16 operands; a weight gradient is rounded to bf16 on one side (2^-9 per element), and
        # causal texts of up to 512 words differ by nothing else
        assert a.dtype == c.dtype and _rel(a, c) < 6e-3


@pytest.mark.parametrize("keeps", [True, False])
def test_light_layer_hands_gradients_over_early(monkeypatch, keeps):
    """A weight's gradient reaches the optimizer before the rest of its half is enqueued: between two offers the native call
    allocates what it goes on with.  A gradient that the optimizer declines goes to `.grad`."""
    from memarch_b200.models.blocks import LightBlock
    from memarch_b200.ops import basic
    with torch.device("cuda"):
        b = LightBlock(128, 2)
    names = {id(p): n for n, p in b.named_parameters()}
    seen = []

    def sink(w, g):
        seen.append((names[id(w)], torch.cuda.memory_stats()["allocation.all.allocated"]))
        return keeps
    x = torch.randn(2, 200, 128, device="cuda", requires_grad=True)
    monkeypatch.setattr(basic, "WEIGHT_GRAD_SINK", sink)
    y = b(x, 64)
    y.backward(torch.ones_like(y))
    end = torch.cuda.memory_stats()["allocation.all.allocated"]
    assert [n for n, _ in seen] == ["down.weight", "up.weight", "o.weight", "qkv.weight"]
    at = [c for _, c in seen] + [end]
    # after the offer of `down`: the input gradient and that of `up`; of `up`: the norm's; of `o`: the packed gradient, statistics,
    # input gradient and that of `qkv`; of `qkv`: the norm's
    assert [q - p >= k for p, q, k in zip(at, at[1:], (2, 2, 4, 2))] == [True] * 4
    assert all((p.grad is None) == keeps for n, p in b.named_parameters() if n in dict(seen))


def test_light_layer_halves_leave_other_cases_alone():
    """Frozen weights, a stream without a gradient, bf16 streams and short batches stay on the single ops."""
    from memarch_b200.models.blocks import LightBlock
    from memarch_b200.ops import layer
    with torch.device("cuda"):
        b = LightBlock(128, 2)
    ok = lambda x: layer.attn_half_ok(x, None, b.n1.weight, b.qkv.weight, b.o.weight, 2, 64)
    x = torch.randn(2, 200, 128, device="cuda")
    assert not ok(x) and ok(x.clone().requires_grad_()) and not ok(x[:1].clone().requires_grad_()) and not ok(x.bfloat16().requires_grad_())
    b.o.weight.requires_grad_(False)
    assert not ok(x.clone().requires_grad_())
    with torch.no_grad():
        assert ok(x)


@pytest.mark.parametrize("train", [True, False])
@pytest.mark.parametrize("what", ["x", "pending", "norm", "up"])
def test_light_layer_refuses_forward_mode(train, what):
    """No forward-mode derivative is implemented: one that is asked for is refused, with and without gradients, not dropped."""
    import torch.autograd.forward_ad as fw
    from memarch_b200.models.blocks import LightBlock
    with torch.device("cuda"):
        b = LightBlock(128, 2)
    x = torch.randn(2, 200, 128, device="cuda", requires_grad=True)
    pending = torch.randn_like(x).bfloat16()
    with torch.set_grad_enabled(train), fw.dual_level():
        dual = lambda t: fw.make_dual(t.detach(), torch.ones_like(t))
        if what == "norm":
            del b.n2.weight
            b.n2.weight = dual(torch.ones(128, device="cuda"))
        if what == "up":
            w = b.up.weight
            del b.up.weight
            b.up.weight = dual(w)
        with pytest.raises((RuntimeError, NotImplementedError), match="jvp|forward.mode|forward AD"):
            b(dual(x) if what == "x" else x, 64, pending=dual(pending) if what == "pending" else pending)


@pytest.mark.parametrize("train", [True, False])
def test_light_layer_with_strided_norm_weights(train):
    """Norm weights that are views with a stride give what their contiguous copies give."""
    from memarch_b200.models.blocks import LightBlock
    torch.manual_seed(5)
    with torch.device("cuda"):
        b = LightBlock(128, 2)
    wide = torch.rand(2, 128, 4, device="cuda") + 0.5
    x, go = torch.randn(2, 200, 128, device="cuda"), torch.randn(2, 200, 128, device="cuda")
    res = []
    for take in (lambda w: w[:, 0], lambda w: w[:, 0].contiguous()):
        b.n1.weight, b.n2.weight = (torch.nn.Parameter(take(w)) for w in wide)
        b.zero_grad(set_to_none=True)
        with torch.set_grad_enabled(train):
            a = x.clone().requires_grad_()
            y = b(a, 64)
        if train:
            y.backward(go)
        res.append([y.detach(), a.grad, b.n1.weight.grad, b.n2.weight.grad, b.qkv.weight.grad] if train else [y])
    for p, q in zip(*res):
        assert torch.equal(p, q)


# ------------------------------------------------------------------------------------------------ padded groups
@pytest.mark.parametrize("E,C,counts", [(1, 256, [3]), (3, 2561, [2561, 0, 257]), (8, 600, [0, 600, 256, 255, 1, 0, 512, 300]), (128, 257, "mixed"), (130, 300, "mixed"), (2, 300, [0, 0])])
@pytest.mark.parametrize("act", ["swiglu", "relu2"])
def test_expert_ffn_counts_order(E, C, counts, act):
    """Row tiles of padding are dealt out after the others: same results as without counts, empty groups and more groups than
    the counted order takes included."""
    from memarch_b200.ops.moe import expert_ffn
    g = torch.Generator(device="cuda").manual_seed(E)
    d, H = 64, 136
    cnt = (torch.arange(E, device="cuda") * 37 % (C + 1) if counts == "mixed" else torch.tensor(counts, device="cuda")).int()
    live = (torch.arange(C, device="cuda")[None] < cnt[:, None])[..., None]
    x = torch.randn(E, C, d, device="cuda", generator=g).bfloat16() * live
    up = (torch.randn(E, d, 2 * H if act == "swiglu" else H, device="cuda", generator=g) * d ** -0.5).bfloat16()
    down = (torch.randn(E, H, d, device="cuda", generator=g) * H ** -0.5).bfloat16()
    gy = torch.randn(E, C, d, device="cuda", generator=g).bfloat16() * live
    res = []
    for c in (cnt, None):
        t = [v.clone().requires_grad_() for v in (x, up, down)]
        y = expert_ffn(*t, act, counts=c)
        y.backward(gy)
        res.append([y] + [v.grad for v in t])
    for a, b in zip(*res):
        assert torch.equal(a, b) or _rel(a, b) < 1e-5


# ------------------------------------------------------------------------------------------------ activation backward
@pytest.mark.parametrize("M,H,K", [(256, 8, 64), (300, 72, 64), (513, 200, 136), (1000, 264, 2048), (4000, 1032, 72), (9473, 512, 64)])
@pytest.mark.parametrize("b_mn", [True, False])
def test_gemm_activation_backward(M, H, K, b_mn):
    """Two warps per 32 accumulator rows: ragged rows and columns, narrow and wide tiles, more tiles than CTA pairs."""
    from memarch_b200.ops import gemm
    g = torch.Generator(device="cuda").manual_seed(M)
    dy, w = torch.randn(M, K, device="cuda", generator=g).bfloat16(), (torch.randn(H, K, device="cuda", generator=g) * K ** -0.5).bfloat16()
    pre = torch.randn(M, 2 * H, device="cuda", generator=g).bfloat16()
    dh = dy.double() @ w.double().t()
    wm = w.t().contiguous() if b_mn else w
    gate, up = pre.double().chunk(2, 1)
    s = gate.sigmoid()
    want = torch.cat([dh * up * s * (1 + gate * (1 - s)), dh * gate * s], 1)
    # one rounding to bf16 (2^-9)
    assert _rel(gemm(dy, wm, b_mn=b_mn, epi=5, aux=pre), want) < 4e-3
    p2 = pre[:, :H].contiguous()
    assert _rel(gemm(dy, wm, b_mn=b_mn, epi=2, aux=p2), dh * 2 * p2.double().relu()) < 4e-3


@pytest.mark.parametrize("direct", [False, True])
@pytest.mark.parametrize("gate", [-3.0, -6.0, -9.0, -20.0, -80.0, -200.0, 9.0, 200.0])
def test_swiglu_backward_of_extreme_gates(gate, direct):
    """The sigmoid's relative error stays at that of fp32 where it is small: grouped (experts) and plain products, both epilogues."""
    from memarch_b200.ops import _ext, gemm
    g = torch.Generator(device="cuda").manual_seed(1)
    E, M, H, K = 2, 300, 72, 64
    dy, w = torch.randn(E, M, K, device="cuda", generator=g).bfloat16(), (torch.randn(E, H, K, device="cuda", generator=g) * K ** -0.5).bfloat16()
    pre = torch.randn(E, M, 2 * H, device="cuda", generator=g) * 0.2
    pre[..., :H] += gate
    pre = pre.bfloat16()
    dh = dy.double() @ w.double().mT
    a, u = pre.double().chunk(2, -1)
    s = a.sigmoid()
    want = torch.cat([dh * u * s * (1 + a * (1 - s)), dh * a * s], -1)
    if direct:
        _ext.C().gemm_set_debug(8, 0)
    try:
        got = gemm(dy, w, groups=E, epi=5, aux=pre), gemm(dy[0].contiguous(), w[0].contiguous(), epi=5, aux=pre[0].contiguous())
    finally:
        _ext.C().gemm_set_debug(0, 0)
    for o, r in zip(got, (want, want[0])):
        for c, t in zip(o.double().chunk(2, -1), r.chunk(2, -1)):
            # one rounding to bf16 (2^-9) and three of fp32; results below bf16's normal range (2^-126) count as zero
            assert (c - t).norm() < 3e-3 * t.norm() + 1e-30


# ------------------------------------------------------------------------------------------------ head
@pytest.mark.parametrize("N,V,d,chunk", [(1, 16, 16, 4096), (300, 1000, 24, 128), (513, 264, 136, 512), (40, 104, 64, 7)])
@pytest.mark.parametrize("wdt", [torch.float32, torch.bfloat16])
def test_linear_ce_chunks(N, V, d, chunk, wdt):
    """Chunks of any length, the first one writes the weight gradient; scaled, repeated and differentiable upstream gradients."""
    from memarch_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(N)
    h = torch.randn(N, d, device="cuda", generator=g).bfloat16().requires_grad_()
    w = (torch.randn(V, d, device="cuda", generator=g) * d ** -0.5).to(wdt).requires_grad_()
    y = torch.randint(0, V, (N,), device="cuda", generator=g)
    loss = ops.linear_ce(h, w, y, chunk=chunk) * 0.37
    hd, wd = h.detach().double().requires_grad_(), w.detach().bfloat16().double().requires_grad_()
    want = torch.nn.functional.cross_entropy(hd @ wd.t(), y, reduction="sum") * 0.37
    gh, gw = torch.autograd.grad(want, (hd, wd))
    assert abs(loss.item() - want.item()) < 2e-3 * max(1.0, abs(want.item()))
    for _ in range(2):
        a, b = torch.autograd.grad(loss, (h, w), retain_graph=True)
        # bf16 logits (2^-9 of values up to 4) and bf16 gradients of them
        assert a.dtype == h.dtype and b.dtype == wdt and _rel(a, gh) < 2e-2 and _rel(b, gw) < 2e-2
    a2, = torch.autograd.grad(loss, (h,), create_graph=True)
    assert torch.allclose(a2, a, rtol=1e-2, atol=1e-6)


# ------------------------------------------------------------------------------------------------ operands off the 16-byte boundary
@pytest.mark.parametrize("M", [301, 304])
def test_operands_off_the_boundary(M):
    """Inputs and gradients that start between two 16-byte pieces are copied, not refused."""
    from memarch_b200 import ops
    from memarch_b200.models.blocks import LightBlock
    shift = lambda t: torch.empty(t.numel() + 1, device="cuda", dtype=t.dtype)[1:].view(t.shape).copy_(t)
    g = torch.Generator(device="cuda").manual_seed(M)
    x, w, gy = (torch.randn(s, 64, device="cuda", generator=g).bfloat16() for s in (M, 64, M))
    y = torch.randint(0, 64, (M,), device="cuda", generator=g)
    torch.manual_seed(M)
    with torch.device("cuda"):
        b = LightBlock(64, 1)
    res = []
    for move in (shift, lambda t: t.clone()):
        a, u, f = (move(t).requires_grad_() for t in (x, w, x.float()[None]))
        o = ops.linear(a, u)
        o.backward(move(gy))
        q = ops.ffn(a, u, u, "relu2")
        q.backward(move(gy))
        loss = ops.linear_ce(a, u, y)
        loss.backward()
        h, p = b(f, 16, None, True)
        torch.autograd.backward([h, p], [f.detach() * 0.5, move(gy[None])])
        res.append([o, q, loss, a.grad, u.grad, h, p, f.grad])
    for s, t in zip(*res):
        assert torch.equal(s, t) or _rel(s, t) < 1e-5


@pytest.mark.parametrize("B,T", [(1, 40), (2, 130)])
def test_single_ops_off_the_boundary(B, T):
    """The row operations one by one and a light layer of few rows: operands, gradients and norm weights that start between two
    16-byte pieces are copied before any kernel sees them."""
    from memarch_b200 import ops
    from memarch_b200.models.blocks import LightBlock
    from memarch_b200.ops import basic
    from memarch_b200.ops.attention import attention
    shift = lambda t: torch.empty(t.numel() + 1, device="cuda", dtype=t.dtype)[1:].view(t.shape).copy_(t)
    g = torch.Generator(device="cuda").manual_seed(T)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
    x, y, w, go, qkv = rnd(B, T, 64), rnd(B, T, 64).bfloat16(), rnd(64) + 2, rnd(B, T, 64), rnd(B, T, 3, 2, 64).bfloat16()
    torch.manual_seed(T)
    with torch.device("cuda"):
        b = LightBlock(64, 1)
    res = []
    for move in (shift, lambda t: t.clone()):
        out = []

        def run(f, *ts, grad):
            ts = [move(t).requires_grad_() for t in ts]
            o = f(*ts)
            for q, r in zip(o if isinstance(o, tuple) else (o,), grad):
                q.backward(move(r.to(q.dtype)), retain_graph=True)
                out.append(q.detach())
            out.extend(t.grad for t in ts)
        run(lambda a, u: ops.rmsnorm(a, u, 1e-6), x, w, grad=[go])
        run(lambda a, u: ops.rmsnorm(a, u, 1e-6), y, w, grad=[go])
        run(lambda a, q, u: ops.add_rmsnorm(a, q, u, 1e-6), x, y, w, grad=[go, go])
        run(ops.resid_add, x, y, grad=[go])
        run(basic.relu2, y, grad=[go])
        run(basic.swiglu, y, grad=[go[..., :32].contiguous()])
        run(lambda a: attention(a, 33), qkv, grad=[rnd(1).new_ones(B, T, 128)])
        b.zero_grad(set_to_none=True)
        b.n1.weight, b.n2.weight = (torch.nn.Parameter(move(w)) for _ in range(2))
        run(lambda a: b(a, 2048), x, grad=[go])
        res.append(out + [v.grad for v in b.parameters()])
    assert len(res[0]) == len(res[1])
    for p, q in zip(*res):
        assert _rel(p, q) < 1e-3                                  # the same arithmetic on copied operands
