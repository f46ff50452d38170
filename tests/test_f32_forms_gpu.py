"""The forms of the 32-bit path's kernels (wide and narrow tiles of the products, staged tokens of the router, warps of
eight queries of the attention): every form against float64 within the bound of a chain of additions, and the same bits
from every form."""

import os
import subprocess
import sys

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
UNIT = 2.0 ** -24


def F():
    from mini_infer_b200.ops import functional
    return functional


def rnd(*shape, seed=0, scale=1.0):
    return (torch.randn(*shape, generator=torch.Generator().manual_seed(seed)) * scale).to(DEV)


def within_chain(out, a, w):
    """A chain of K fused multiply-adds is off by at most K units of sum |a||w|."""
    ref = a.double() @ w.double().T
    bound = a.shape[1] * UNIT * (a.double().abs() @ w.double().abs().T) + 1e-30
    assert bool(((out.double() - ref).abs() <= bound).all())


# rows: one, a narrow tile's last, one more, the narrow form's last, one more, a wide tile's edges; columns and inner sizes that fill no tile
@pytest.mark.parametrize("T", [1, 16, 17, 32, 33, 64, 65, 200])
@pytest.mark.parametrize("N,K", [(33, 4), (64, 68), (129, 100), (320, 63), (200, 2050), (19200, 36)])
def test_dense_forms(T, N, K):
    a, w = rnd(T, K, seed=1), rnd(N, K, seed=2)
    out = F().dense_f32(a, w)
    within_chain(out, a, w)
    for lo, hi in ((0, min(T, 5)), (T - 1, T), (max(0, T - 20), T)):
        assert torch.equal(F().dense_f32(a[lo:hi].contiguous(), w), out[lo:hi])


def test_dense_rows_that_are_not_aligned():
    flat, w = rnd(40 * 64 + 1, seed=3), rnd(70, 64, seed=4)
    a = flat[1:].view(40, 64)
    assert torch.equal(F().dense_f32(a, w), F().dense_f32(a.clone(), w))


@pytest.mark.parametrize("counts", [[0, 1, 0, 16, 17], [64, 65, 0, 0, 3], [3] * 40 + [0, 8], [200, 0, 15]])
@pytest.mark.parametrize("nout,K", [(32, 64), (45, 68), (130, 36), (70, 33)])
@pytest.mark.parametrize("paired", [False, True])
def test_grouped_forms(counts, nout, K, paired):
    E, n, T = len(counts), sum(counts), 50
    x, w = rnd(T, K, seed=5), rnd(E, (2 if paired else 1) * nout, K, seed=6)
    gather = torch.randint(0, T, (n,), generator=torch.Generator().manual_seed(7)).to(torch.int32).to(DEV)
    offsets = torch.tensor([sum(counts[:e]) for e in range(E + 1)], dtype=torch.int32, device=DEV)
    scale = rnd(n, seed=8).abs() if paired else None
    out = F().grouped_gemm_plain(x, gather, w, offsets, n, paired, torch.float32, row_scale=scale)
    for e in range(E):
        lo, hi = int(offsets[e]), int(offsets[e + 1])
        if lo == hi:
            continue
        rows = x[gather[lo:hi].long()].contiguous()
        z = F().dense_f32(rows, w[e].contiguous())
        within_chain(z, rows, w[e])
        if not paired:
            assert torch.equal(out[lo:hi], z)
            # whatever else is in the step: the expert's rows one by one
            one = F().grouped_gemm_plain(rows[-1:].contiguous(), None, w[e:e + 1].contiguous(),
                                         torch.tensor([0, 1], dtype=torch.int32, device=DEV), 1, False, torch.float32)
            assert torch.equal(one[0], out[hi - 1])
        else:
            g, u = (z.double() * scale[lo:hi, None].double()).chunk(2, 1)
            ref = g * torch.sigmoid(g) * u
            assert bool(((out[lo:hi].double() - ref).abs() <= 16 * UNIT * (g.abs() + 1) * u.abs() + 1e-30).all())


@pytest.mark.parametrize("rows", [3, 200])
@pytest.mark.parametrize("paired", [False, True])
def test_grouped_product_over_nothing(rows, paired):
    x, w = torch.empty(rows, 0, device=DEV), torch.empty(2, 40, 0, device=DEV)
    offsets = torch.tensor([0, 1, rows], dtype=torch.int32, device=DEV)
    out = F().grouped_gemm_plain(x, None, w, offsets, rows, paired, torch.float32)
    assert torch.equal(out, torch.zeros(rows, 20 if paired else 40, device=DEV))


@pytest.mark.parametrize("T", [33, 40, 77, 512])
@pytest.mark.parametrize("H,E,gated", [(64, 5, True), (1028, 16, False), (2048, 60, True), (2052, 33, True)])
def test_router_of_many_tokens_adds_as_that_of_few(T, H, E, gated):
    x, w, g = rnd(T, H, seed=9), rnd(E, H, seed=10, scale=0.05), rnd(H, seed=11, scale=0.05) if gated else None
    whole = F().moe_router(x, w, g, 2, False, want_probs=True)
    few = [F().moe_router(x[lo:lo + 8].contiguous(), w, g, 2, False, want_probs=True) for lo in range(0, T, 8)]
    for i, got in enumerate(whole):
        if got is not None:
            assert torch.equal(got, torch.cat([f[i] for f in few]))


# the staged rows take H / 32 KiB of shared memory beside 1 KiB of the kernel's own: the sizes at which the two together
# pass 48 KiB (1504, 1508), at which the rows alone do (1536, 1540), and the largest that the router takes
@pytest.mark.parametrize("H", [1504, 1508, 1536, 1540, 6400])
def test_router_rows_at_the_limits_of_shared_memory(H):
    """In a process of its own: a larger size before it would have raised the kernel's limit for good."""
    code = f"""
import torch
from mini_infer_b200.ops import functional as F
x, w = torch.randn(40, {H}, device="cuda:0"), torch.randn(9, {H}, device="cuda:0") * 0.05
whole = F.moe_router(x, w, None, 2, False, want_probs=True)
few = [F.moe_router(x[lo:lo + 8].contiguous(), w, None, 2, False, want_probs=True) for lo in range(0, 40, 8)]
for i, got in enumerate(whole):
    assert got is None or torch.equal(got, torch.cat([f[i] for f in few]))
"""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    subprocess.run([sys.executable, "-c", code], check=True, cwd=root, timeout=300)


@pytest.mark.parametrize("d", [144, 146, 148])
def test_tiled_attention_at_the_limit_of_shared_memory(d):
    """Rows of 146 numbers and what the kernel has beside them pass 48 KiB together, neither by itself (a process of its
    own, as above)."""
    code = f"""
import torch
from mini_infer_b200.ops import functional as F
q, k, v = (torch.randn(s, device="cuda:0") for s in ((16, 2, {d}), (1, 2, 16, {d}), (1, 2, 16, {d})))
i32 = lambda t: torch.tensor(t, dtype=torch.int32, device="cuda:0")
out = F.attention(q, k, v, i32([[0]]), i32([0, 16]), i32([16]), 16, 0)
later = torch.ones(16, 16, dtype=torch.bool, device="cuda:0").triu(1)
s = (torch.einsum("qhd,hkd->hqk", q.double(), k[0].double()) * {d} ** -0.5).masked_fill(later, -torch.inf)
ref = torch.einsum("hqk,hkd->qhd", torch.softmax(s, -1), v[0].double())
assert float((out - ref).abs().max()) <= 3e-6 * float(ref.abs().max())
"""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    subprocess.run([sys.executable, "-c", code], check=True, cwd=root, timeout=300)


@pytest.mark.parametrize("d,nh,nkv,page,window", [(64, 4, 2, 16, 0), (128, 2, 1, 16, 0), (128, 3, 3, 8, 40), (64, 2, 2, 32, 17)])
def test_attention_of_every_cut(d, nh, nkv, page, window):
    lengths, S = [1, 7, 8, 33, 64, 95], 95
    k, v = rnd(1, S, nkv, d, seed=12)[0], rnd(1, S, nkv, d, seed=13)[0]
    q = rnd(S, nh, d, seed=14)
    pages = -(-S // page)
    order = list(range(pages))[::-1]
    kc, vc = torch.zeros(pages, nkv, page, d, device=DEV), torch.zeros(pages, nkv, page, d, device=DEV)
    for p in range(S):
        kc[order[p // page], :, p % page], vc[order[p // page], :, p % page] = k[p], v[p]
    i32 = lambda t: torch.tensor(t, dtype=torch.int32, device=DEV)
    table = i32([order])
    whole = F().attention(q, kc, vc, table, i32([0, S]), i32([S]), S, window)
    at = torch.arange(S, device=DEV)
    seen = (at[None] <= at[:, None]) & ((at[None] > at[:, None] - window) if window else torch.ones(S, S, dtype=torch.bool, device=DEV))
    for h in range(nh):
        s = (q[:, h].double() @ k[:, h // (nh // nkv)].double().T) * d ** -0.5
        ref = torch.softmax(s.masked_fill(~seen, -torch.inf), -1) @ v[:, h // (nh // nkv)].double()
        assert float((whole[:, h].double() - ref).abs().max()) <= 3e-6 * float(ref.abs().max())
    lo = 0
    for hi in lengths:              # the same prompt in portions
        out = F().attention(q[lo:hi].contiguous(), kc, vc, table, i32([0, hi - lo]), i32([hi]), hi - lo, window)
        assert torch.equal(out, whole[lo:hi])
        lo = hi
    # several requests in one step, one of them with one token
    two = F().attention(torch.cat([q[94:95], q[30:64]]).contiguous(), kc, vc, table.expand(2, -1).contiguous(), i32([0, 1, 35]),
                        i32([95, 64]), 34, window)
    assert torch.equal(two, torch.cat([whole[94:95], whole[30:64]]))


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("key,window", [(20, 0), (9, 0), (70, 24)])
def test_values_that_are_not_finite_stay_with_their_queries(d, key, window):
    """A query is as it was unless its block of 16 reaches the key: the tiles of the general kernel, which heads of other
    sizes take, leave out what lies behind their 16 queries."""
    S, nh, page = 96, 2, 16
    q, k, v = rnd(S, nh, d, seed=15), rnd(S // page, nh, page, d, seed=16), rnd(S // page, nh, page, d, seed=17)
    i32 = lambda t: torch.tensor(t, dtype=torch.int32, device=DEV)
    run = lambda: F().attention(q, k, v, i32([list(range(S // page))]), i32([0, S]), i32([S]), S, window)
    clean = run()
    v[key // page, :, key % page, 3] = float("inf")
    out = run()
    before = key // 16 * 16
    assert torch.equal(out[:before], clean[:before])
    if window:                  # tiles of 32 keys that no query of a block of 16 sees any more
        first = (key // 32 * 32 + 32 + window - 1) // 16 * 16 + 16
        assert torch.equal(out[first:], clean[first:])
    sees = slice(key, min(S, key + (window or S)))
    assert not bool(torch.isfinite(out[sees, :, 3]).any())
    rest = [c for c in range(d) if c != 3]
    assert torch.equal(out[:, :, rest], clean[:, :, rest])
