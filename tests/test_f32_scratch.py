"""The scratch of a float32 product belongs to the call until its kernels are queued: nothing that the call allocates, nor another
thread while the library runs, can be given the same memory."""

import weakref

import pytest
import torch

from mini_infer_b200.ops import functional as F


class Library:
    """Stands in for the CUDA library: notes whether the scratch is still held when a product is queued."""

    def __init__(self):
        self.scratch, self.held = None, []

    def mi_f32_tc_min_inner(self):
        return 512

    def mi_f32_tc_scratch(self, rows, K, *_):
        return 2 * rows * K

    def __getattr__(self, name):
        def queue(*args):
            self.held.append(self.scratch() is not None)
            return 0
        return queue


@pytest.mark.parametrize("call", ["dense", "heads", "grouped", "paired"])
def test_scratch_is_held_while_a_product_is_queued(call, monkeypatch):
    lib = Library()
    made, order = F._f32_scratch, []

    def scratch(*args):
        t = made(*args)
        lib.scratch = weakref.ref(t)
        order.append("scratch")
        return t

    word = F._status_word
    monkeypatch.setattr(F, "library", lambda: lib)
    monkeypatch.setattr(F, "_chk", lambda *a, **k: None)
    monkeypatch.setattr(F, "_stream", lambda: 0)
    monkeypatch.setattr(F, "_tc_status", {})
    monkeypatch.setattr(F, "_tc_pending", False)
    monkeypatch.setattr(F, "_f32_scratch", scratch)
    monkeypatch.setattr(F, "_status_word", lambda dev: (order.append("status"), word(dev))[1])
    x, w = torch.zeros(40, 512), torch.zeros(8, 512)
    if call == "dense":
        F.dense_f32(x, w)
    elif call == "heads":
        F.dense_f32_heads(x.view(20, 1024), w.view(2, 4, 512))
    elif call == "grouped":
        F.f32_tc_form(x, None, w.view(2, 4, 512), torch.zeros(3, dtype=torch.int32), torch.zeros(40, 4), 40, False)
    else:
        F.f32_tc_form(x, None, w, None, torch.zeros(40, 4), 40, True)
    assert lib.held == [True]
    assert order == ["status", "scratch"]


@pytest.mark.gpu
def test_first_product_of_a_device(monkeypatch):
    """The word for waits is made by the first product, whose scratch comes from the same small blocks of the allocator."""
    monkeypatch.setattr(F, "_tc_status", {})
    g = torch.Generator().manual_seed(0)
    x, w = torch.randn(40, 2048, generator=g).to("cuda:0"), torch.randn(64, 2048, generator=g).to("cuda:0")
    out = F.dense_f32(x, w)
    assert float((out.double() - x.double() @ w.double().T).norm()) < 1e-6 * float(out.norm())
    F.check_tc_status()


@pytest.mark.gpu
def test_small_inner_sizes_need_no_word(monkeypatch):
    monkeypatch.setattr(F, "_tc_status", {})
    F.dense_f32(torch.randn(3, 64, device="cuda:0"), torch.randn(5, 64, device="cuda:0"))
    assert not F._tc_status
