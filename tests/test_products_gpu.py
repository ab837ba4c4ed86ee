"""The float32 products and attention, the many-token product's stores, the experts' product for few tokens and kernels of the
recurrent and latent layers, each alone against float64, at the edges of their tiles, stages and dispatch lines. Limits: a float32 sum of K products in any order is within
about sqrt(K) / 2 roundings of 2^-24 of sqrt(sum of squares); outputs rounded to bfloat16 are within 2^-9 of their size."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda"
BF = torch.bfloat16


def ops():
    from xpu_serve_b200.ops import lib
    return lib


def gap(got, ref):
    assert torch.isfinite(got).all()
    return (got.double() - ref).abs().max().item() / max(ref.abs().max().item(), 1e-30)


def f32_limit(K):
    # (the largest of many differences, about 5 deviations, over the largest result)
    return 5.0 * math.sqrt(K) / 2.0 * 2.0 ** -24 / 2.0 + 2.0 ** -23


# ------------------------------------------------------------------------------------------- float32 product
@pytest.mark.parametrize("M,N,K", [(1, 1, 4), (1, 8, 32), (3, 7, 36), (4, 9, 1024), (5, 1030, 1028), (8, 40, 2052), (9, 15, 1020),
                                   (16, 2500, 96), (17, 33, 64), (40, 4736, 40), (63, 65, 100), (64, 4800, 33), (65, 64, 32),
                                   (130, 129, 68), (200, 56900, 16), (224, 1024, 36), (225, 1024, 36), (300, 2048, 64), (700, 2050, 40)])
def test_float32_product(M, N, K):
    ld = (K + 3) // 4 * 4 + 4
    x = torch.randn(M, ld, device=DEV)[:, :K]
    w = torch.randn(N, ld, device=DEV)[:, :K]
    bias = torch.randn(N, device=DEV)
    out = torch.full((M, N + 3), 7.0, device=DEV)[:, :N]
    ops().gemm_generic(x, w, out, bias)
    assert gap(out, x.double() @ w.double().T + bias.double()) <= f32_limit(K)
    # the order of the sums is the same for every number of rows and on rows that no 16-byte copy takes
    for rows in {1, min(M, 6), min(M, 12), min(M, 64)}:
        some = torch.empty(rows, N, device=DEV)
        ops().gemm_generic(x[:rows], w, some, bias)
        assert torch.equal(some, out[:rows])
    odd_x, odd_w = torch.randn(M, K + 1, device=DEV)[:, :K], torch.randn(N, K + 1, device=DEV)[:, :K]
    odd_x.copy_(x), odd_w.copy_(w)
    if (K + 1) % 4:
        other = torch.empty(M, N, device=DEV)
        ops().gemm_generic(odd_x, odd_w, other, bias)
        assert torch.equal(other, out)


@pytest.mark.skipif(torch.cuda.device_count() < 2, reason="needs two devices")
@pytest.mark.parametrize("M", [3, 200])
def test_float32_product_on_each_device_of_a_process(M):
    for d in range(2):
        with torch.cuda.device(d):
            x, w, out = torch.randn(M, 64, device=f"cuda:{d}"), torch.randn(200, 64, device=f"cuda:{d}"), torch.empty(M, 200, device=f"cuda:{d}")
            ops().gemm_generic(x, w, out)
            assert gap(out, x.double() @ w.double().T) <= f32_limit(64)


# ------------------------------------------------------------------------------------------ float32 attention
@pytest.mark.parametrize("H,G,D,DV,planes,window,keep,plus,cap", [
    (4, 2, 64, 64, 2, 0, 0, 0, 0.0), (3, 1, 20, 36, 2, 0, 0, 0, 0.0), (2, 2, 128, 64, 2, 50, 0, 0, 0.0), (6, 2, 8, 12, 2, 33, 70, 1, 0.0),
    (2, 1, 256, 256, 2, -100, 0, 0, 30.0), (4, 4, 32, 32, 1, 40, 10, 0, 0.0)])
@pytest.mark.parametrize("lens", [(1, 1), (5, 200), (31, 33, 64, 300)])
def test_float32_attention(H, G, D, DV, planes, window, keep, plus, cap, lens):
    page, T = 64, sum(min(3, n) for n in lens)
    P = -(-max(lens) // page)
    pages = torch.randperm(P * len(lens), device=DEV).to(torch.int32).view(len(lens), P)
    # a page holds its keys [G, page, D], then its values [G, page, DV]
    pool = torch.randn(P * len(lens), G * page * (D + (DV if planes == 2 else 0)), device=DEV)
    seq = torch.tensor([s for s, n in enumerate(lens) for _ in range(min(3, n))], dtype=torch.int32, device=DEV)
    pos = torch.tensor([n - 1 - i for n in lens for i in reversed(range(min(3, n)))], dtype=torch.int32, device=DEV)
    q = torch.randn(T, H, D, device=DEV)
    gate = torch.randn(T, H, device=DEV)
    out = torch.empty(T, H, DV, device=DEV)
    scale = D ** -0.5
    storage = pool.view(-1, planes, G, page, D) if D == DV or planes == 1 else pool
    # (window: the kernels' own number: above 0 a window, below 0 a block of so many positions)
    ops()._check(ops().load().xs_attention_generic(
        q.data_ptr(), storage.data_ptr(), pages.data_ptr(), P, seq.data_ptr(), pos.data_ptr(), gate.data_ptr(), H, out.data_ptr(), H * DV,
        T, H, G, D, DV, planes, page, scale, cap, window, keep, plus, 0, 0, ops()._stream()))
    ref = torch.empty(T, H, DV, dtype=torch.float64, device=DEV)
    for t in range(T):
        p, s = int(pos[t]), int(seq[t])
        lo = max(0, p - window + 1) if window > 0 else p - p % -window if window < 0 else 0
        keys = [j for j in range(p + 1) if j >= lo or j < keep]
        for h in range(H):
            g = h // (H // G)
            rows = [(int(pages[s, j // page]), j % page) for j in keys]
            k = torch.stack([pool[a, (g * page + b) * D:(g * page + b) * D + D] for a, b in rows]).double()
            at = G * page * D if planes == 2 else 0
            v = torch.stack([pool[a, at + (g * page + b) * DV:at + (g * page + b) * DV + DV] for a, b in rows]).double()
            z = k @ q[t, h].double() * scale
            z = cap * torch.tanh(z / cap) if cap > 0 else z
            if plus:
                e = torch.exp(z - z.max().clamp(min=0.0))
                w = e / (e.sum() + torch.exp(-z.max().clamp(min=0.0)))
            else:
                w = torch.softmax(z, 0)
            ref[t, h] = w @ v * torch.sigmoid(gate[t, h].double())
    assert gap(out, ref) <= 4e-6      # (scores of a few units: 2^-24 of them through the exponential, on top of the sums)


@pytest.mark.parametrize("H,G,D,DV,window,keep,plus", [(8, 4, 64, 64, 0, 0, 0), (8, 2, 32, 20, 300, 70, 1), (6, 2, 128, 64, 0, 0, 0),
                                                       (4, 2, 256, 256, 0, 0, 0)])
@pytest.mark.parametrize("keys", [1, 33, 130, 520, 700])
def test_float32_attention_does_not_depend_on_the_step(H, G, D, DV, window, keep, plus, keys):
    """A token alone and among more (token, head) pairs than a launch gives a warp a group: the same bits."""
    page, P, T = 64, 11, 200
    pool = torch.randn(2 * P, G * page * (D + DV), device=DEV)
    pages = torch.randperm(2 * P, device=DEV).to(torch.int32).view(2, P)
    q = torch.randn(T, H, D, device=DEV)
    seq = (torch.arange(T, device=DEV) % 2).to(torch.int32)
    pos = torch.randint(0, 700, (T,), device=DEV).to(torch.int32)
    pos[77] = keys - 1
    assert T * H > 4 * 148 >= H

    def attend(t0, n):
        out = torch.empty(n, H, DV, device=DEV)
        qs, ss, ps = q[t0:t0 + n].contiguous(), seq[t0:t0 + n].clone(), pos[t0:t0 + n].clone()
        ops()._check(ops().load().xs_attention_generic(
            qs.data_ptr(), pool.data_ptr(), pages.data_ptr(), P, ss.data_ptr(), ps.data_ptr(), None, 0, out.data_ptr(), H * DV, n, H, G, D,
            DV, 2, page, D ** -0.5, 0.0, window, keep, plus, 0, 0, ops()._stream()))
        torch.cuda.synchronize()
        return out

    assert torch.equal(attend(77, 1)[0], attend(0, T)[77])


@pytest.mark.parametrize("plus", [0, 1])
@pytest.mark.parametrize("keys", [5, 64, 90, 600])
def test_float32_attention_of_values_that_are_not_finite(plus, keys):
    """Against the kernel of other alignments: an infinite value of the last key, keys whose scores are minus infinity."""
    H, D, page, P = 2, 64, 64, 10
    pool = torch.randn(P, 2, H, page, D, device=DEV)
    pages, seq = torch.arange(P, dtype=torch.int32, device=DEV).view(1, P), torch.zeros(1, dtype=torch.int32, device=DEV)
    pos = torch.tensor([keys - 1], dtype=torch.int32, device=DEV)
    flat_q = torch.randn(H * D + 1, device=DEV)
    flat_q[::8] = flat_q[::8].abs() + 0.1
    flat_q[1:] = flat_q[:-1].clone()

    def both():
        res = []
        for off in (0, 1):                # (the second on an odd word: the general kernel)
            q = flat_q.clone()[1:].clone() if off == 0 else flat_q[1:]
            out = torch.empty(1, H, D, device=DEV)
            ops()._check(ops().load().xs_attention_generic(
                q.data_ptr(), pool.data_ptr(), pages.data_ptr(), P, seq.data_ptr(), pos.data_ptr(), None, 0, out.data_ptr(), H * D, 1, H, H, D,
                D, 2, page, D ** -0.5, 0.0, 0, 0, plus, 0, 0, ops()._stream()))
            res.append(out)
        return res

    pool[(keys - 1) // page, 1, :, (keys - 1) % page, 7] = math.inf
    got, want = both()
    assert bool((want[..., 7] == math.inf).all()) and torch.equal(got.isinf(), want.isinf())
    fine = torch.isfinite(want)
    assert (got[fine] - want[fine]).abs().max() <= 4e-6 * want[fine].abs().max()
    if keys > 64 or plus:
        # (only the keys behind position 31 where the denominator has no term of its own, so that the general kernel's first block has a maximum)
        pool[:, 1].clamp_(-9.0, 9.0)
        first = 0 if plus else 32
        hidden = torch.arange(P * page, device=DEV).view(P, page)
        pool[:, 0, :, :, 0] = torch.where(((hidden >= first) & (hidden < 64))[:, None], torch.tensor(-math.inf, device=DEV), pool[:, 0, :, :, 0])
        got, want = both()
        assert torch.isfinite(want).all() and torch.isfinite(got).all()
        assert (got - want).abs().max() <= 4e-6 * want.abs().max().clamp(min=1e-6)


# --------------------------------------------------------------------------- tcgen05 product, many tokens: the store paths
@pytest.mark.parametrize("T,N", [(65, 48), (128, 272), (129, 256), (300, 528), (1000, 80)])
@pytest.mark.parametrize("pad", [0, 8, 1])
@pytest.mark.parametrize("form", ["store", "store32", "swiglu", "swiglu32", "clamped"])
def test_many_token_product_stores(T, N, pad, form):
    """Rows of the output on 32-byte, 16-byte and odd boundaries, tiles that end inside 32 columns."""
    K = 72
    x, w = torch.randn(T, K, device=DEV).to(BF), torch.randn(N, K, device=DEV).to(BF)
    gated = not form.startswith("store")
    cols, dtype = N // 2 if gated else N, torch.float32 if form.endswith("32") else BF
    out = torch.full((T, (cols + 15) // 16 * 16 + pad), 7.0, device=DEV, dtype=dtype)
    if form == "clamped":
        ops().gemm_tc_clamped(x, w, out[:, :cols], 1.5, 1.702, 1.0)
    else:
        ops().gemm_tc(x, w, out[:, :cols], epilogue=ops().EPI_SWIGLU if gated else ops().EPI_STORE)
    ref = x.double() @ w.double().T
    if gated:
        g, u = ref.view(T, N // 16, 2, 8).unbind(2)
        g, u = g.reshape(T, cols), u.reshape(T, cols)
        if form == "clamped":
            g, u = g.clamp(max=1.5), u.clamp(-1.5, 1.5)
            ref = g * torch.sigmoid(1.702 * g) * (u + 1.0)
        else:
            ref = g * torch.sigmoid(g) * u
    # (the exponential's and the reciprocal's few units in the last place on top of the sums)
    assert gap(out[:, :cols], ref) <= (2.0 ** -8 if dtype == BF else f32_limit(K) + 2.0 ** -20)
    assert bool((out[:, cols:] == 7.0).all())


@pytest.mark.parametrize("dtype", [torch.float32, BF])
@pytest.mark.parametrize("N,pad", [(16, 0), (64, 0), (96, 8), (272, 3)])
@pytest.mark.parametrize("act", ["silu", "clamped"])
def test_gated_epilogue_far_gates(dtype, N, pad, act):
    """Gates where the exponential is zero, huge or infinite, on the 32-column stores (rows on 32 bytes) and off them."""
    gates = torch.tensor([0.0, -1.0, -50.0, -80.0, -88.0, -88.6, -100.0, -3e4, 80.0, 100.0, 3e4], device=DEV)
    T, K = 130, 16
    x = torch.zeros(T, K, device=DEV, dtype=BF)
    x[:, 0] = gates[torch.arange(T, device=DEV) % len(gates)].to(BF)
    x[:, 1] = 3.0
    w = torch.zeros(N // 16, 2, 8, K, device=DEV, dtype=BF)
    w[:, 0, :, 0], w[:, 1, :, 1] = 1.0, 1.0
    w = w.view(N, K)
    out = torch.empty(T, N // 2 + pad, device=DEV, dtype=dtype)[:, :N // 2]
    g = x[:, :1].double()
    if act == "clamped":
        ops().gemm_tc_clamped(x, w, out, 7.0, 1.702, 1.0)
        want = g.clamp(max=7.0) * torch.sigmoid(1.702 * g.clamp(max=7.0)) * 4.0
    else:
        ops().gemm_tc(x, w, out, epilogue=ops().EPI_SWIGLU)
        want = g * torch.sigmoid(g) * 3.0
    assert torch.isfinite(out).all()
    # (the exponential's argument is some tens, rounded to 2^-24 of itself; far out only its size counts)
    limit = want.abs() * (2.0 ** -8 if dtype == BF else 2.0 ** -17) + 1e-30
    assert ((out.double() - want).abs() <= limit).all()


@pytest.mark.parametrize("T", [7, 130, 400])      # (the epilogues of few tokens, of many and of pairs of CTAs)
@pytest.mark.parametrize("act", ["silu", "clamped"])
def test_gated_epilogue_rounds_once(T, act):
    """bfloat16 outputs are the float32 outputs rounded: the gated unit is no less exact where its result is rounded."""
    N, K = 1024, 256
    x, w = torch.randn(T, K, device=DEV).to(BF), (torch.randn(N, K, device=DEV) * 0.125).to(BF)
    exact, rounded = torch.empty(T, N // 2, device=DEV), torch.empty(T, N // 2, device=DEV, dtype=BF)
    for out in (exact, rounded):
        if act == "clamped":
            ops().gemm_tc_clamped(x, w, out, 7.0, 1.702, 1.0)
        else:
            ops().gemm_tc(x, w, out, epilogue=ops().EPI_SWIGLU)
    assert torch.equal(rounded, exact.to(BF))


# ------------------------------------------------------------------------------------------- few tokens' experts
@pytest.mark.parametrize("T,top,E,F,H", [(1, 1, 1, 8, 8), (1, 4, 16, 1024, 2048), (7, 3, 5, 24, 40), (8, 2, 3, 40, 264), (9, 1, 1, 16, 512),
                                         (16, 4, 6, 56, 96), (17, 2, 4, 48, 1032), (32, 5, 7, 72, 328)])
@pytest.mark.parametrize("act", ["silu", "clamped", "relu_squared"])
def test_experts_of_few_tokens(T, top, E, F, H, act):
    top = min(top, E)
    x = torch.randn(T, H + 8, device=DEV).to(BF)[:, :H]
    ids = torch.stack([torch.randperm(E, device=DEV)[:top] for _ in range(T)]).to(torch.int32).reshape(-1)
    if T * top > 3:
        ids[2] = -1
    gate, up = (torch.randn(E, F, H, device=DEV).to(BF) * H ** -0.5 for _ in range(2))
    down = (torch.randn(E, H, F, device=DEV) * F ** -0.5).to(BF)
    glu = act != "relu_squared"
    w = torch.stack([gate.view(E, F // 8, 8, H), up.view(E, F // 8, 8, H)], 2).reshape(E, 2 * F, H).contiguous() if glu else up.contiguous()
    hidden = torch.zeros(T * top, F, device=DEV, dtype=BF)
    clamp = (1.0, 1.702, 1.0) if act == "clamped" else None
    ops().moe_few_rows(x, top, w, hidden, ids, T, glu=glu, clamp=clamp, relu_squared=not glu)
    out = torch.zeros(T * top, H, device=DEV, dtype=BF)
    ops().moe_few_rows(hidden, 1, down, out, ids, T, glu=False)
    for i in range(T * top):
        e = int(ids[i])
        if e < 0:
            assert not hidden[i].any() and not out[i].any()
            continue
        u = up[e].double() @ x[i // top].double()
        g = gate[e].double() @ x[i // top].double()
        if act == "silu":
            ref = g * torch.sigmoid(g) * u
        elif act == "clamped":
            g, u = g.clamp(max=1.0), u.clamp(-1.0, 1.0)
            ref = g * torch.sigmoid(1.702 * g) * (u + 1.0)
        else:
            ref = u.clamp(min=0.0) ** 2
        assert gap(hidden[i], ref) <= 2.0 ** -8 and gap(out[i], down[e].double() @ hidden[i].double()) <= 2.0 ** -8
    wts = torch.rand(T * top, device=DEV)
    y = torch.empty(T, H, device=DEV, dtype=BF)
    ops().moe_combine(out, ids, wts, y, top, in_place=True, passed=x)
    rows = torch.where((ids >= 0)[:, None], out.double(), x.double().repeat_interleave(top, 0))
    assert gap(y, (rows * wts.double()[:, None]).view(T, top, H).sum(1)) <= 2.0 ** -8


@pytest.mark.parametrize("E,top", [(5, 5), (9, 3), (40, 8), (64, 2), (130, 6), (256, 16), (300, 4)])
@pytest.mark.parametrize("router", ["top", "sigmoid", "softmax", "groups"])
def test_choices_are_experts_and_differ(E, top, router):
    """Whatever the logits are: NaN, infinite, equal."""
    inf, nan = math.inf, math.nan
    rows = [torch.full((E,), nan), torch.full((E,), -inf), torch.full((E,), inf), torch.zeros(E), torch.randn(E), torch.randn(E), torch.randn(E)]
    rows[4][::2] = nan
    rows[5][1:] = -inf
    rows[6][: E - 1] = nan
    rows += [torch.randn(E) for _ in range(8 - len(rows))]
    logits = torch.stack(rows).to(DEV)
    T = logits.shape[0]
    ids = torch.full((T * top,), 12345, dtype=torch.int32, device=DEV)
    wts = torch.empty(T * top, device=DEV)
    if router == "top":
        ops().moe_route(logits, top, ids, wts)
    else:
        groups = next(g for g in (4, 3, 2, 1) if E % g == 0) if router == "groups" else 1
        keep = next(k for k in range(1, groups + 1) if k * (E // groups) >= top)
        ops().moe_route_grouped(logits, top, ids, wts, experts=E, score="softmax" if router == "softmax" else "sigmoid",
                                groups=groups, keep=keep, group_top=2, renorm=True, renorm_eps=0.0)
    got = ids.view(T, top).tolist()
    for t, choices in enumerate(got):
        assert all(0 <= e < E for e in choices) and len(set(choices)) == top, (t, choices)
    assert torch.isnan(wts.view(T, top)[0]).all()      # a token of NaNs stays one
    want = torch.topk(logits[7], top).indices.tolist()
    assert router == "groups" or got[7] == want


def test_a_token_of_nan_leaves_the_others_alone():
    T, top, E, F, H = 8, 8, 16, 40, 264
    x, w = torch.randn(T, H, device=DEV).to(BF), torch.randn(E, F, H, device=DEV).to(BF)
    logits = torch.randn(T, E, device=DEV)
    logits[:, 0] = 9.0                 # everybody names expert 0
    logits[0] = math.nan
    ids, wts = torch.empty(T * top, dtype=torch.int32, device=DEV), torch.empty(T * top, device=DEV)
    ops().moe_route_grouped(logits, top, ids, wts, experts=E)
    out = torch.full((T * top, F), math.nan, device=DEV, dtype=BF)
    ops().moe_few_rows(x, top, w, out, ids, T, glu=False)
    ref = torch.einsum("tkfh,th->tkf", w.double()[ids.view(T, top).long()], x.double()).reshape(T * top, F)
    assert gap(out, ref) <= 2.0 ** -8
    with pytest.raises(ops().KernelError, match="choices"):
        ops().moe_few_rows(x, top, w, out, ids, 7, glu=False)


@pytest.mark.parametrize("T,clamped", [(150, False), (300, False), (300, True)])
@pytest.mark.parametrize("out_dtype", [BF, torch.float32])
def test_gated_epilogue_over_all_gates(T, clamped, out_dtype):
    """Gates from the most negative to the largest, where e^-g leaves the normal numbers and where the division takes over; NaN stays
    NaN. Every result is its own quotient: half a unit in the last place of the stored type, and e^-g's few units of float32."""
    g = torch.cat([torch.linspace(-100, 20, T - 12), torch.tensor([-3.3e38, -1e30, -200.0, -88.5, -87.0, -86.9, 0.0, -0.0, 1e-38, 100.0, 1e30, 1e38])])
    x = torch.zeros(T, 64, device=DEV, dtype=BF)
    x[:, 0], x[:, 1] = g.to(DEV), torch.linspace(-3, 3, T, device=DEV)
    x[5, 0] = math.nan
    w = torch.zeros(8, 2, 8, 64, device=DEV, dtype=BF)
    w[:, 0, :, 0] = w[:, 1, :, 1] = 1.0
    out = torch.zeros(T, 64, device=DEV, dtype=out_dtype)
    g, u = x[:, :1].double(), x[:, 1:2].double()
    if clamped:
        ops().gemm_tc_clamped(x, w.view(128, 64), out, 7.0, 1.702, 1.0)
        g, u, a = g.clamp(max=7.0), u.clamp(-7.0, 7.0) + 1.0, 1.702
    else:
        ops().gemm_tc(x, w.view(128, 64), out, epilogue=ops().EPI_SWIGLU)
        a = 1.0
    ref = (g * torch.sigmoid(a * g) * u).expand(T, 64)
    keep = torch.arange(T, device=DEV) != 5
    assert bool(out[5].isnan().all()) or clamped
    if not clamped:
        # (e^-g beyond the largest number: the quotient is 0; 1e-36 covers it)
        assert bool(((out.double() - ref).abs()[keep] <= (2.0 ** -8 if out_dtype == BF else 2.0 ** -18) * ref.abs()[keep] + 1e-36).all())
    else:
        assert bool(((out.double() - ref).abs()[keep] <= 2.0 ** -8 * ref.abs()[keep] + 1e-35).all())


@pytest.mark.parametrize("M,F,K", [(1, 8, 8), (3, 24, 264), (8, 1024, 2048), (8, 16, 8192), (9, 40, 1032), (16, 1024, 2048)])
@pytest.mark.parametrize("slices", [1, 4])
def test_clamped_unit_of_few_rows(M, F, K, slices):
    slices = slices if K > 1024 else 1
    x, w = torch.randn(M, K, device=DEV).to(BF), (torch.randn(2 * F, K, device=DEV) * (2.0 / K) ** 0.5).to(BF)
    scratch = torch.zeros(ops().gemm_small_m_scratch_bytes(M, 2 * F, slices), device=DEV, dtype=torch.uint8)
    out = torch.full((M, F + 8), 7.0, device=DEV, dtype=BF)
    for _ in range(2):
        ops().gemm_small_m_clamped(x, w, out[:, :F], 1.5, 1.702, 1.0, ksplit=slices, scratch=scratch if slices > 1 else None)
    g, u = (x.double() @ w.double().T).view(M, F // 8, 2, 8).unbind(2)
    g, u = g.reshape(M, F).clamp(max=1.5), u.reshape(M, F).clamp(-1.5, 1.5)
    assert gap(out[:, :F], g * torch.sigmoid(1.702 * g) * (u + 1.0)) <= 2.0 ** -8
    assert bool((out[:, F:] == 7.0).all())


def test_experts_rows_do_not_depend_on_the_step():
    E, F, H, top = 6, 64, 256, 2
    x = torch.randn(8, H, device=DEV).to(BF)
    ids = torch.randint(0, E, (8,), device=DEV)
    ids = torch.stack([ids, (ids + 1) % E], 1).to(torch.int32).reshape(-1)
    w = torch.randn(E, F, H, device=DEV).to(BF)
    whole, one = torch.empty(16, F, device=DEV, dtype=BF), torch.empty(2, F, device=DEV, dtype=BF)
    ops().moe_few_rows(x, top, w, whole, ids, 8, glu=False)
    for t in range(8):
        ops().moe_few_rows(x[t:t + 1], top, w, one, ids[2 * t:2 * t + 2].contiguous(), 1, glu=False)
        assert torch.equal(one, whole[2 * t:2 * t + 2])


@pytest.mark.parametrize("T,top,E,N,K", [(1, 1, 3, 16, 8), (1, 4, 16, 2048, 520), (2, 2, 9, 2032, 64), (8, 4, 16, 200, 1000), (8, 2, 40, 1040, 2048),
                                         (5, 5, 150, 144, 2816), (9, 2, 4, 272, 72), (16, 4, 16, 256, 2048), (16, 2, 5, 130, 2056), (8, 1, 2, 48, 4096),
                                         (3, 2, 4, 40, 9400)])
def test_streamed_experts_at_their_lines(T, top, E, N, K):
    """Four and eight warps a CTA, one and two groups of eight rows, K past whole stages, rows of x that leave room for two CTAs
    an SM, for one or for none. One infinite input: its row alone is affected, and stays infinite where the sign is certain."""
    x, w = torch.randn(T, K, device=DEV).to(BF), (torch.randn(E, N, K, device=DEV) / math.sqrt(K)).to(BF)
    ids = torch.stack([torch.randperm(E, device=DEV)[:top] for _ in range(T)]).to(torch.int32)
    ids[0, 0] = -1
    ids = ids.reshape(-1)
    out = torch.full((T * top, N), 7.0, device=DEV, dtype=BF)
    ops().moe_few_rows(x, top, w, out, ids, T, glu=False)
    ref = torch.einsum("rnk,rk->rn", w[ids.long().clamp(min=0)].double(), x.double().repeat_interleave(top, 0))
    met = ids >= 0
    assert gap(out[met], ref[met]) <= 2.0 ** -8 if bool(met.any()) else True
    assert bool((out[~met] == 7.0).all())
    x[T - 1, K - 1] = math.inf
    again = torch.full_like(out, 7.0)
    ops().moe_few_rows(x, top, w, again, ids, T, glu=False)
    assert torch.equal(again[:(T - 1) * top], out[:(T - 1) * top])
    last = met[(T - 1) * top:]
    sign = w[ids[(T - 1) * top:].long().clamp(min=0), :, K - 1].sign()
    assert bool((again[(T - 1) * top:] == sign * math.inf)[last].logical_or(sign[last] == 0).all())


# ------------------------------------------------------------------------- kernels of the recurrent and latent layers
@pytest.mark.parametrize("lens", [[1], [64, 65, 1, 700], [130] * 5])
@pytest.mark.parametrize("H,R,Dr,window", [(16, 512, 64, 0), (3, 128, 32, 100), (16, 64, 0, 64), (5, 512, 64, 0)])
def test_latent_attention_of_single_tokens_in_parts(lens, H, R, Dr, window):
    """As many parts as pages, fewer, and more than there are: those without a page write nothing. Weights and outputs are
    bfloat16: about 2^-8 of the norm."""
    n, W = len(lens), R + Dr
    pages = [-(-l // 64) for l in lens]
    pool = torch.randn(sum(pages), 1, 1, 64, W, device=DEV).to(BF)
    table, order, at = torch.full((n, max(pages) + 1), -1, dtype=torch.int32), torch.randperm(sum(pages)).to(torch.int32), 0
    for i, c in enumerate(pages):
        table[i, :c], at = order[at:at + c], at + c
    ql, qr = torch.randn(n, H, R, device=DEV).to(BF), torch.randn(n, H, Dr, device=DEV).to(BF)
    cu, kv = (torch.tensor(a, dtype=torch.int32, device=DEV) for a in (range(n + 1), lens))
    sink = torch.rand(H, device=DEV)
    for splits in (1, 2, 3, 11, 64):
        out = torch.full((n, H, R), math.nan, device=DEV, dtype=BF)
        scratch = torch.full((max(1, ops().latent_attention_mma_scratch_bytes(n * H, R, splits)),), 255, dtype=torch.uint8, device=DEV)
        ops().latent_attention_mma(ql, qr, pool, table.to(DEV), cu, kv, None, sink, out, scratch, n, 1, 64, W ** -0.5, window, splits)
        for i, l in enumerate(lens):
            keys = pool[table[i, :pages[i]].long().to(DEV), 0, 0].reshape(-1, W)[max(0, l - window) if window else 0:l].double()
            sc = torch.cat([torch.cat([ql[i], qr[i]], -1).double() @ keys.T * W ** -0.5, sink.double()[:, None]], 1)
            ref = sc.softmax(-1)[:, :-1] @ keys[:, :R]
            assert ((out[i].double() - ref).norm() / ref.norm()).item() < 2.0 ** -7, (splits, i)


@pytest.mark.parametrize("B,M,N,K", [(1, 1, 1, 8), (16, 8, 512, 128), (3, 9, 33, 520), (2, 16, 31, 1032), (4, 5, 100, 24)])
def test_batched_product_of_few_rows(B, M, N, K):
    x = torch.randn(M, B, K + 8, device=DEV).to(BF).transpose(0, 1)[:, :, :K]
    w = torch.randn(B, N, K + 16, device=DEV).to(BF)[:, :, :K]
    out = torch.empty(M, B, N, device=DEV, dtype=BF).transpose(0, 1)
    ops().gemm_batched(x, w, out)
    assert gap(out, x.double() @ w.double().transpose(1, 2)) <= 2.0 ** -8


@pytest.mark.parametrize("groups,part", [(2, 4), (3, 100), (16, 128), (5, 132), (8, 512), (2, 516), (2, 1024)])
@pytest.mark.parametrize("act", [None, 0, 1])
@pytest.mark.parametrize("dtype", [torch.float32, BF])
def test_grouped_norm(groups, part, act, dtype):
    T, W, eps = 5, groups * part, 1e-5
    x, w = torch.randn(T, W, device=DEV), torch.rand(W, device=DEV) + 0.5
    y = torch.empty(T, W, device=DEV, dtype=dtype)
    gate = torch.randn(T, W + 3, device=DEV).to(dtype)[:, 3:] if act is not None else None
    ops()._check(ops().load().xs_grouped_rmsnorm(x.data_ptr(), w.data_ptr(), y.data_ptr(), W, ops()._code(y), T, W, groups, eps,
                                                 ops()._ptr(gate), 0 if gate is None else gate.stride(0), act or 0, ops()._stream()))
    v = x.double().view(T, groups, part)
    ref = (v * torch.rsqrt((v * v).mean(-1, keepdim=True) + eps)).view(T, W) * w.double()
    if gate is not None:
        z = gate.double()
        ref = ref * torch.sigmoid(z) * (z if act == 1 else 1.0)
    assert gap(y, ref) <= (2.0 ** -8 if dtype == BF else 2e-6)


@pytest.mark.parametrize("heads,P,N,G,seqs", [(4, 4, 1, 2, 1), (6, 64, 128, 3, 8), (2, 20, 37, 1, 3), (3, 132, 300, 3, 2), (2, 1024, 16, 1, 1),
                                              (2, 7, 301, 1, 2)])
@pytest.mark.parametrize("dtype", [torch.float32, BF])
def test_mamba2_step(heads, P, N, G, seqs, dtype):
    inner = heads * P
    C = inner + 2 * G * N
    r = lambda *s: torch.randn(*s, device=DEV)                                     # noqa: E731
    xbc, proj = r(seqs, C).to(dtype), r(seqs, inner + C + heads).to(dtype)
    bias, a_log, skip, state0 = r(heads), r(heads) * 0.5, r(heads), r(seqs + 2, heads, N, P)
    slots = torch.randperm(seqs + 2, device=DEV)[:seqs].to(torch.int32)
    cu = torch.arange(seqs + 1, dtype=torch.int32, device=DEV)
    state, y = state0.clone(), torch.empty(seqs, inner, device=DEV)
    ops().mamba2_scan(xbc, proj, inner + C, bias, a_log, skip, state, cu, slots, y, heads, P, N, G, single=True)
    x = xbc.double()[:, :inner].view(seqs, heads, P)
    Bm, Cm = (m.view(seqs, G, N).repeat_interleave(heads // G, 1) for m in xbc.double()[:, inner:].split(G * N, 1))
    dt = torch.nn.functional.softplus(proj.double()[:, inner + C:] + bias.double())
    s = state0[slots.long()].double() * torch.exp(-torch.exp(a_log.double()) * dt)[..., None, None] + (dt[..., None] * Bm)[..., None] * x[:, :, None]
    want = ((s * Cm[..., None]).sum(2) + skip.double()[:, None] * x).reshape(seqs, inner)
    want = want * torch.nn.functional.silu(proj.double()[:, :inner])
    assert gap(y, want) <= 4e-6 and gap(state[slots.long()], s) <= 2e-6
    rest = torch.tensor([i for i in range(seqs + 2) if i not in set(slots.tolist())], device=DEV)
    assert torch.equal(state[rest], state0[rest])


@pytest.mark.parametrize("heads,P,N,G,seqs", [(4, 4, 4, 2, 1), (6, 64, 128, 3, 8), (2, 20, 36, 1, 3), (3, 132, 200, 3, 2), (2, 256, 16, 1, 1),
                                              (4, 30, 200, 4, 5), (2, 260, 64, 1, 2), (2, 20, 37, 1, 3), (2, 33, 150, 2, 2), (4, 3, 1, 2, 1)])
@pytest.mark.parametrize("dtype", [torch.float32, BF])
def test_mamba2_step_is_the_scan_of_one_token(heads, P, N, G, seqs, dtype):
    """A token's outputs and state do not depend on whether its step holds single tokens only: the same bits."""
    inner = heads * P
    C = inner + 2 * G * N
    r = lambda *s: torch.randn(*s, device=DEV)                                     # noqa: E731
    xbc, proj = r(seqs, C).to(dtype), r(seqs, inner + C + heads).to(dtype)
    bias, a_log, skip, state = r(heads), r(heads) * 0.5, r(heads), r(seqs, heads, N, P)
    slots, cu = torch.arange(seqs, dtype=torch.int32, device=DEV), torch.arange(seqs + 1, dtype=torch.int32, device=DEV)
    got = []
    for single in (True, False):
        s, y = state.clone(), torch.empty(seqs, inner, device=DEV)
        ops().mamba2_scan(xbc, proj, inner + C, bias, a_log, skip, s, cu, slots, y, heads, P, N, G, single=single)
        got.append((s, y))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])


@pytest.mark.parametrize("chunk,lens", [(4, [100, 3, 33]), (8, [64, 65, 8]), (1, [17, 1])])
def test_mamba2_carry_over_many_chunks(chunk, lens):
    """More chunks than the carry asks for at one time, and one more or fewer. Every token's update and every chunk's carry rounds once
    against the largest state, and an output sums N products: at most T + N roundings."""
    heads, P, N, G = 4, 12, 20, 2
    inner, T = heads * P, sum(lens)
    C = inner + 2 * G * N
    r = lambda *s: torch.randn(*s, device=DEV)                                     # noqa: E731
    xbc, proj, bias, a_log, skip = r(T, C), r(T, inner + C + heads), r(heads), r(heads) * 0.5, r(heads)
    state = r(len(lens), heads, N, P)
    want, states, starts, rows, first, t = [], [], [0], [], [0], 0
    for i, n in enumerate(lens):
        rows += [(i, t + k, min(chunk, n - k)) for k in range(0, n, chunk)]
        first.append(len(rows))
        s = state[i].double()
        for _ in range(n):
            x = xbc[t].double()[:inner].view(heads, P)
            Bm, Cm = (m.view(G, N).repeat_interleave(heads // G, 0) for m in xbc[t].double()[inner:].split(G * N))
            dt = torch.nn.functional.softplus(proj[t].double()[inner + C:] + bias.double())
            s = s * torch.exp(-torch.exp(a_log.double()) * dt)[:, None, None] + (dt[:, None] * Bm)[..., None] * x[:, None]
            y = ((s * Cm[..., None]).sum(1) + skip.double()[:, None] * x).reshape(inner)
            want.append(y * torch.nn.functional.silu(proj[t].double()[:inner]))
            t += 1
        starts.append(t)
        states.append(s)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)                # noqa: E731
    out = torch.empty(T, inner, device=DEV)
    ops().mamba2_scan(xbc, proj, inner + C, bias, a_log, skip, state, i32(starts), i32(range(len(lens))), out, heads, P, N, G,
                      chunks=(i32(rows), i32(first), torch.empty(len(rows), heads, N, P, device=DEV),
                              torch.empty(len(rows), heads, device=DEV)))
    limit = (max(lens) + N) * 2.0 ** -24
    assert gap(out, torch.stack(want)) <= limit and gap(state, torch.stack(states)) <= limit


def test_mamba2_step_of_more_tokens_than_sequences_is_refused():
    heads, P, N, G, T, seqs = 2, 8, 16, 1, 5, 3
    inner = heads * P
    C = inner + 2 * G * N
    r = lambda *s: torch.randn(*s, device=DEV)                                     # noqa: E731
    cu = torch.tensor([0, 1, 3, 5], dtype=torch.int32, device=DEV)
    y = torch.full((T, inner), 7.0, device=DEV)
    with pytest.raises(ops().KernelError, match="5 tokens"):
        ops().mamba2_scan(r(T, C), r(T, inner + C + heads), inner + C, r(heads), r(heads), r(heads), r(seqs, heads, N, P), cu,
                          torch.arange(seqs, dtype=torch.int32, device=DEV), y, heads, P, N, G, single=True)
    assert bool((y == 7.0).all())


@pytest.mark.parametrize("taps,C,col0,seqs", [(1, 16, 8, 2), (2, 24, 0, 1), (3, 1032, 16, 5), (4, 64, 8, 8), (5, 48, 8, 3), (4, 20, 4, 3)])
@pytest.mark.parametrize("dtype", [torch.float32, BF])
def test_mamba2_conv_of_single_tokens(taps, C, col0, seqs, dtype):
    proj, w, bias = torch.randn(seqs, col0 + C + 8, device=DEV).to(dtype), torch.randn(C, taps, device=DEV), torch.randn(C, device=DEV)
    state0 = torch.randn(seqs + 2, max(taps - 1, 1), C, device=DEV).to(dtype)
    slots = torch.randperm(seqs + 2, device=DEV)[:seqs].to(torch.int32)
    seq, cu = torch.arange(seqs, dtype=torch.int32, device=DEV), torch.arange(seqs + 1, dtype=torch.int32, device=DEV)
    state, out = state0.clone(), torch.empty(seqs, C, device=DEV, dtype=dtype)
    before = ops().launches
    ops().mamba2_conv(proj, col0, w, bias, state, seq, cu, slots, out, single=True)
    # (the state is moved on by the filter's own kernel in bfloat16, up to four taps, in 16-byte pieces)
    assert ops().launches - before == (1 if taps == 1 or (dtype == BF and taps <= 4 and C % 8 == 0 and col0 % 8 == 0) else 2)
    new = proj[:, None, col0:col0 + C]
    rows = torch.cat([state0[slots.long()][:, :taps - 1], new], 1)
    acc = (rows.double() * w.double().T[None]).sum(1) + bias.double()
    assert gap(out, acc * torch.sigmoid(acc)) <= (2.0 ** -8 if dtype == BF else 2e-6)
    want = state0.clone()
    if taps > 1:
        want[slots.long()] = rows[:, 1:]
    assert torch.equal(state, want)
