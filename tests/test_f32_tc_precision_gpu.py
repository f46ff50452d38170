"""Float32 products on tensor cores against float64 and against the chain of multiply-adds that smaller inner sizes take: rows
of few numbers, of many, of numbers near the smallest; products that go in bands."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
T, N, K = 96, 130, 512


def F():
    from mini_infer_b200.ops import functional
    return functional


def chain(a, w):
    """One chain of fused multiply-adds per element (a product of two float32 numbers is exact in float64)."""
    s = torch.zeros(a.shape[0], w.shape[0], device=DEV)
    a, w = a.double(), w.double()
    for k in range(a.shape[1]):
        s = (s.double() + a[:, k:k + 1] * w[:, k]).float()
    return s


def off(out, ref):
    return float((out.double() - ref).norm() / ref.norm())


def rows_of(numbers, g):
    a = torch.zeros(T, K)
    for t in range(T):
        a[t, torch.randperm(K, generator=g)[:numbers]] = torch.randn(numbers, generator=g)
    return a


@pytest.mark.parametrize("numbers", [1, 2, 3, 8, 32, 200, K])
def test_no_further_off_than_the_chain(numbers):
    g = torch.Generator().manual_seed(numbers)
    a, w = rows_of(numbers, g).to(DEV), torch.randn(N, K, generator=g).to(DEV)
    ref = a.double() @ w.double().T
    # (one number a row: both are rounded once, but for sums cut off 2^-33 below; one result in 1,000 differs)
    assert off(F().dense_f32(a, w), ref) <= off(chain(a, w), ref) * (1.002 if numbers == 1 else 1.0)


def test_a_number_times_one_is_the_number():
    g = torch.Generator().manual_seed(0)
    a, w = torch.zeros(T, K), torch.randn(N, K, generator=g)
    at = torch.randint(0, K, (T,), generator=g)
    a[torch.arange(T), at] = 1.0
    for rows in (1, 20, T):
        assert torch.equal(F().dense_f32(a[:rows].to(DEV), w.to(DEV)).cpu(), w[:, at[:rows]].T)


@pytest.mark.parametrize("scale_a,scale_w", [(1e-38, 1.0), (1e-41, 1.0), (1.0, 1e-38), (1e-38, 1e30), (1e-20, 1e-20), (1e18, 1e18), (1e37, 1e-3)])
def test_small_and_large_numbers(scale_a, scale_w):
    """Parts of the smallest numbers are normal numbers; what is beyond the parts' range is a chain."""
    g = torch.Generator().manual_seed(3)
    a, w = (torch.randn(T, K, generator=g) * scale_a).to(DEV), (torch.randn(N, K, generator=g) * scale_w).to(DEV)
    ref = a.double() @ w.double().T
    assert off(F().dense_f32(a, w), ref) <= off(chain(a, w), ref)


def test_product_in_bands():
    """More rows than the scratch for their parts holds (128 MB): the same bits as by themselves."""
    F_, rows, K4 = F(), 50000, 513
    for k in (K, K4):                                  # (513: rows that are not aligned)
        x, w = torch.randn(rows, k, device=DEV), torch.randn(24, k, device=DEV)
        out = F_.dense_f32(x, w)
        assert F_.library().mi_f32_tc_scratch(rows, k, 0, 1, -1) * 4 <= 128 << 20
        for lo in (0, 100, 21000, 25000, 43600, 49950):
            assert torch.equal(F_.dense_f32(x[lo:lo + 50].contiguous(), w), out[lo:lo + 50])
    rows = 50000
    x, w = torch.randn(300, K, device=DEV), torch.randn(3, 24, K, device=DEV)
    gather = torch.randint(0, 300, (rows,), dtype=torch.int32, device=DEV)
    offsets = torch.tensor([0, 21843, 21844, 49999], dtype=torch.int32, device=DEV)
    out = F_.grouped_gemm_plain(x, gather, w, offsets, rows, False, torch.float32)
    for e in range(3):
        every = F_.dense_f32(x, w[e].contiguous())
        lo, hi = int(offsets[e]), int(offsets[e + 1])
        assert torch.equal(out[lo:hi], every[gather[lo:hi].long()])
    F_.check_tc_status()
