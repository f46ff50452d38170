"""What the float32 products on tensor cores refuse before a launch, and which rows they read."""

import pytest
import torch

from mini_infer_b200.ops import functional as F


class Reached(Exception):
    pass


def form(monkeypatch, a, w, n, offsets=None, paired=False, gather=None, on_cpu=True):
    def library():
        raise Reached
    monkeypatch.setattr(F, "library", library)
    if on_cpu:                               # everything but the device is looked at
        chk = F._chk
        monkeypatch.setattr(F, "_chk", lambda t, what, *rest: None if t is None else chk(Cuda(t), what, *rest))
    out = torch.zeros(n, w.shape[-2] // (2 if paired else 1))
    return F.f32_tc_form(a, gather, w, offsets, out, n, paired)


class Cuda:
    def __init__(self, t):
        self.t, self.is_cuda, self.shape, self.dtype, self.is_contiguous = t, True, t.shape, t.dtype, t.is_contiguous


def test_operands_that_are_refused(monkeypatch):
    x, w = torch.zeros(4, 512), torch.zeros(6, 512)
    i32 = lambda n: torch.zeros(n, dtype=torch.int32)
    with pytest.raises(RuntimeError, match="CUDA"):
        form(monkeypatch, x, w, 4, on_cpu=False)
    with pytest.raises(Reached):
        form(monkeypatch, x, w, 4, paired=True)
    with pytest.raises(Reached):             # (rows beyond the experts' need no rows of x)
        form(monkeypatch, x, w.view(2, 3, 512), 9, offsets=i32(3))
    for bad in (dict(a=x.double(), w=w, n=4), dict(a=x, w=w.bfloat16(), n=4), dict(a=x, w=torch.zeros(6, 516), n=4),
                dict(a=x, w=torch.zeros(512, 6).T, n=4), dict(a=x, w=w, n=5), dict(a=x, w=w, n=5, gather=i32(4)),
                dict(a=x, w=w.view(2, 3, 512), n=4, offsets=i32(4)), dict(a=x, w=w, n=4, offsets=i32(2))):
        with pytest.raises((TypeError, ValueError)):
            form(monkeypatch, **bad)


@pytest.mark.gpu
def test_rows_without_an_expert_are_not_read(monkeypatch):
    """`n_rows` may be larger than what the experts have: of the rows behind theirs nothing is read or split."""
    n, live, K, dev = 300, 170, 512, "cuda:0"
    g = torch.Generator().manual_seed(1)
    x, w = torch.randn(30, K, generator=g).to(dev), torch.randn(3, 40, K, generator=g).to(dev)
    gather = torch.randint(0, 30, (n,), generator=g).to(torch.int32).to(dev)
    offsets = torch.tensor([0, 5, 5, live], dtype=torch.int32, device=dev)
    kept = []

    def scratch(t, rows, *sizes):
        room = F.library().mi_f32_tc_scratch(rows, *sizes)
        kept.append(torch.full((room,), -1, dtype=torch.int32, device=dev).view(torch.float32))
        return kept[-1]

    monkeypatch.setattr(F, "_f32_scratch", scratch)
    out = F.grouped_gemm_plain(x, gather, w, offsets, n, False, torch.float32)
    written = int((kept[0].view(torch.int32) != -1).sum())
    assert 0 < written <= live * K * 6 // 4
    for e in range(3):
        lo, hi = int(offsets[e]), int(offsets[e + 1])
        ref = x[gather[lo:hi].long()].double() @ w[e].double().T
        assert float((out[lo:hi].double() - ref).norm()) <= 1e-6 * float(ref.norm())
    F.check_tc_status()
