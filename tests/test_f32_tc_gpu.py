"""Products of the 32-bit path on tensor cores (inner sizes from 512 up): every form against float64 and with the same bits,
grouped as dense, rows that TMA does not take, and operands that are not finite."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
UNIT = 2.0 ** -23


def F():
    from mini_infer_b200.ops import functional
    return functional


def rnd(*shape, seed=0, scale=1.0):
    return (torch.randn(*shape, generator=torch.Generator().manual_seed(seed)) * scale).to(DEV)


def near(out, a, w):
    """Per element: what the halves leave out, 3 * 2^-21 of a term; additions that truncate inside a chunk of 32 (12, each of
    at most 8 numbers aligned to the largest: two units of the sum of absolute values at most), and the additions of chunks
    and parts.  As a whole: nearer than the chain of multiply-adds, which is 4.0e-7 off at K = 512 and more above."""
    ref = a.double() @ w.double().T
    chunks = -(-a.shape[1] // 32)
    units = 12 + 24 + chunks / 4 + 1 + 4
    assert bool(((out.double() - ref).abs() <= units * UNIT * (a.double().abs() @ w.double().abs().T) + 1e-30).all())
    if out.numel() > 500:
        assert float((out.double() - ref).norm() / ref.norm()) < 2.5e-7


# rows: one, the tiles' last and one more; columns and inner sizes that fill no tile, chunk or part; parts without a chunk
@pytest.mark.parametrize("T", [1, 16, 17, 33, 64, 65, 200])
@pytest.mark.parametrize("N,K", [(1, 512), (129, 516), (200, 1030), (384, 2048), (257, 544)])
def test_every_form_gives_the_same_bits(T, N, K):
    a, w = rnd(T, K, seed=1), rnd(N, K, seed=2)
    out = F().dense_f32(a, w)
    near(out, a, w)
    for nt in (16, 32, 64, 128):
        if nt >= 64 and T <= 32:
            continue                       # (no room for the rows' halves is asked for)
        for split in (1, 2, 4) if nt < 128 else (1,):
            got = F().f32_tc_form(a, None, w, None, torch.empty_like(out), T, False, rows_per_tile=nt, blocks_per_tile=split)
            assert torch.equal(got, out), (nt, split)
    for lo, hi in ((0, 1), (T - 1, T), (max(0, T - 20), T)):
        assert torch.equal(F().dense_f32(a[lo:hi].contiguous(), w), out[lo:hi])
    F().check_tc_status()


def test_rows_that_are_not_aligned():
    flat, w = rnd(40 * 512 + 1, seed=3), rnd(70 * 512 + 1, seed=4)
    a, b = flat[1:].view(40, 512), w[1:].view(70, 512)
    assert torch.equal(F().dense_f32(a, b), F().dense_f32(a.clone(), b.clone()))


@pytest.mark.parametrize("T", [1, 33, 130])
@pytest.mark.parametrize("nout,K", [(45, 516), (200, 1026)])
def test_paired_dense_product(T, nout, K):
    from mini_infer_b200.parts.base import linear_swiglu
    x, w = rnd(T, K, seed=11), rnd(2 * nout, K, seed=12, scale=K ** -0.5)
    assert torch.equal(linear_swiglu(x, w, torch.float32), F().swiglu(F().dense_f32(x, w)))


@pytest.mark.parametrize("T", [3, 40])
def test_products_of_heads(T):
    H, N, K = 3, 50, 512
    x, w = rnd(T, H * K + 8, seed=5), rnd(H, N, K, seed=6)
    for col in (0, 8, 1):                  # (1: rows that are not aligned)
        out = F().dense_f32_heads(x, w, x_col=col)
        for h in range(H):
            rows = x[:, col + h * K:col + (h + 1) * K].contiguous()
            assert torch.equal(out[:, h * N:(h + 1) * N], F().dense_f32(rows, w[h].contiguous()))


@pytest.mark.parametrize("counts", [[0, 1, 0, 16, 17], [64, 65, 0, 0, 3], [3] * 40 + [0, 8], [200, 0, 15], [129, 130]])
@pytest.mark.parametrize("nout,K", [(64, 512), (45, 516), (200, 1026)])
@pytest.mark.parametrize("paired", [False, True])
def test_grouped(counts, nout, K, paired):
    E, n, T = len(counts), sum(counts), 50
    x, w = rnd(T, K, seed=5), rnd(E, (2 if paired else 1) * nout, K, seed=6, scale=K ** -0.5)
    gather = torch.randint(0, T, (n,), generator=torch.Generator().manual_seed(7)).to(torch.int32).to(DEV)
    offsets = torch.tensor([sum(counts[:e]) for e in range(E + 1)], dtype=torch.int32, device=DEV)
    scale = rnd(n, seed=8).abs() if paired else None
    out = F().grouped_gemm_plain(x, gather, w, offsets, n, paired, torch.float32, row_scale=scale)
    for nt, split in ((16, 2), (32, 1), (64, 4), (128, 1)):
        if K % 4 == 0 and (nt < 64 or n > 32):
            got = F().f32_tc_form(x, gather, w, offsets, torch.empty_like(out), n, paired, None, scale, nt, split)
            assert torch.equal(got, out), (nt, split)
    for e in range(E):
        lo, hi = int(offsets[e]), int(offsets[e + 1])
        if lo == hi:
            continue
        rows = x[gather[lo:hi].long()].contiguous()
        z = F().dense_f32(rows, w[e].contiguous())
        near(z, rows, w[e])
        if not paired:
            assert torch.equal(out[lo:hi], z)
        else:
            g, u = (z.double() * scale[lo:hi, None].double()).chunk(2, 1)
            ref = g * torch.sigmoid(g) * u
            assert bool(((out[lo:hi].double() - ref).abs() <= 8 * UNIT * (g.abs() + 1) * u.abs() + 1e-30).all())
    F().check_tc_status()


@pytest.mark.parametrize("T", [5, 70])
def test_values_that_are_not_finite(T):
    """An infinity, a NaN of any bits and a sum that overflows reach the elements that multiply-adds let them reach."""
    N, K = 130, 512
    a, w = rnd(T, K, seed=9), rnd(N, K, seed=10)
    clean = F().dense_f32(a, w)
    a[0, 3], a[2, 100], w[7, 50] = torch.inf, torch.nan, -torch.inf
    a[3].view(torch.int32)[9] = 0x7f800001
    w[9].view(torch.int32)[8] = 0x7fffffff
    w[5, 3] = 0.0                          # inf * 0
    a[4] = 1e25
    w[11], w[12, :256], w[12, 256:] = 1e25, 1e25, -1e25
    w[20] = w[20].bfloat16().float()       # (its lo is all zeros)
    ref = (a.double() @ w.double().T).float()
    out = F().dense_f32(a, w)
    assert torch.equal(out.isnan() | (torch.arange(N, device=DEV) == 12) & (torch.arange(T, device=DEV) == 4)[:, None],
                       ref.isnan() | (torch.arange(N, device=DEV) == 12) & (torch.arange(T, device=DEV) == 4)[:, None])
    assert torch.equal(out.isposinf(), ref.isposinf()) or bool((out.isposinf() != ref.isposinf()).nonzero().eq(
        torch.tensor([4, 12], device=DEV)).all())
    assert torch.equal(out.isneginf(), ref.isneginf())
    rows, cols = [r for r in range(T) if r not in (0, 2, 3, 4)], [c for c in range(N) if c not in (5, 7, 9, 11, 12, 20)]
    assert torch.equal(out[rows][:, cols], clean[rows][:, cols])


def test_largest_and_smallest_values():
    """The largest finite number (its hi rounds up to infinity) and numbers whose lo is not normal."""
    a, w = torch.zeros(2, 512, device=DEV), torch.zeros(3, 512, device=DEV)
    a[0, 0], a[1, 1] = 3.4028234663852886e38, 1.2345678e-36
    w[0, 0], w[1, 0], w[2, 1] = 1.0, 0.3333333, 1.0
    ref = (a.double() @ w.double().T)
    out = F().dense_f32(a, w).double()
    assert bool(((out - ref).abs() <= 3 * 2.0 ** -21 * ref.abs()).all())
