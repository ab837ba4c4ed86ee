"""Products and attention in float32, each alone against float64, at the edges of their tiles, stages and dispatch lines. Limits:
a float32 sum of K products in any order is within about sqrt(K) / 2 roundings of 2^-24 of sqrt(sum of squares)."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda"


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
                                   (130, 129, 68), (200, 56900, 16)])
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
