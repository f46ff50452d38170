"""Forms of the recurrent mixers' small kernels that a size chooses: the convolution over a window in registers (four taps,
whole fours of channels) and the gated norm with a warp per group."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def i32(v):
    return torch.tensor(v, dtype=torch.int32, device=DEV)


@pytest.mark.parametrize("lengths", [[1], [2, 1, 3], [7, 8, 9], [40, 1, 300], [2000]])
@pytest.mark.parametrize("C", [4, 516, 4096])
@pytest.mark.parametrize("biased", [False, True])
def test_convolution_of_four_taps(lengths, C, biased):
    from mini_infer_b200.ops import functional as F
    g = torch.Generator().manual_seed(C + sum(lengths))
    rnd = lambda *s: torch.randn(*s, generator=g).to(DEV)
    T, B = sum(lengths), len(lengths)
    x, w, bias = rnd(T, C + 8), rnd(C, 4), rnd(C) if biased else None
    state = rnd(B + 1, 3 * C + 4)
    slots = i32(list(range(B, 0, -1)))
    starts = i32([sum(lengths[:b]) for b in range(B + 1)])
    req = torch.repeat_interleave(torch.arange(B), torch.tensor(lengths)).int().to(DEV)
    st = state.clone()
    out = F.causal_conv_silu(x, 4, C, w, bias, st, 4, starts, req, slots)
    for b, n in enumerate(lengths):
        lo, slot = int(starts[b]), int(slots[b])
        rows = torch.cat([state[slot, 4:].view(3, C), x[lo:lo + n, 4:4 + C]]).double()
        z = sum(rows[j:j + n] * w[:, j].double() for j in range(4)) + (bias.double() if biased else 0)
        # four products and a bias in float32, then silu
        assert float((out[lo:lo + n].double() - z * torch.sigmoid(z)).abs().max()) <= 2.0 ** -21 * float(z.abs().max() + 1)
        assert torch.equal(st[slot, 4:].view(3, C), rows[-3:].float())


@pytest.mark.parametrize("T,groups,gs", [(1, 1, 4), (3, 5, 64), (9, 16, 128), (130, 3, 100), (5, 2, 132)])
@pytest.mark.parametrize("before,silu", [(True, False), (False, False), (False, True)])
@pytest.mark.parametrize("act", [torch.float32, torch.bfloat16])
def test_gated_norm_of_small_groups(T, groups, gs, before, silu, act):
    from mini_infer_b200.ops import functional as F
    g = torch.Generator().manual_seed(T + gs)
    n = groups * gs
    y, gate, w = (torch.randn(*s, generator=g).to(DEV) for s in ((T, n), (T, n + 4), (n,)))
    out = F.gated_group_rmsnorm(y, gate, 4, w, groups, before, 1e-6, act, silu_after=silu)
    z, q = y.double(), gate[:, 4:].double()
    if before:
        z = z * q * torch.sigmoid(q)
    z = z.view(T, groups, gs)
    z = (z / (z.pow(2).mean(-1, keepdim=True) + 1e-6).sqrt()).view(T, n) * w.double()
    if not before:
        z = z * torch.sigmoid(q) * (q if silu else 1)
    tol = 2.0 ** -18 if act == torch.float32 else 2.0 ** -8
    assert float(((out.double() - z).abs() / (z.abs() + 1e-2)).max()) <= tol
