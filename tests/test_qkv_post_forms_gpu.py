"""Bias, rotation and cache write of many tokens (a block per token) and of few: the same bits."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("nh,nkv,d", [(4, 2, 64), (3, 1, 128), (2, 2, 24), (1, 1, 264), (5, 0, 64)])
@pytest.mark.parametrize("bias,rope", [(None, True), (torch.float32, True), (torch.bfloat16, False)])
def test_many_tokens_as_few(dtype, nh, nkv, d, bias, rope):
    from mini_infer_b200.ops import functional as F
    g = torch.Generator().manual_seed(d + nh)
    rnd = lambda *s: torch.randn(*s, generator=g).to(DEV)
    T, ps, pages = 130, 16, 12
    qkv, pos = rnd(T, (nh + 2 * nkv) * d), torch.randint(0, 5000, (T,), generator=g).to(torch.int32).to(DEV)
    b = None if bias is None else rnd((nh + 2 * nkv) * d).to(bias)
    inv = (10000.0 ** (-torch.arange(d // 2) * 2.0 / d)).float().to(DEV) if rope else None
    slots = torch.randperm(ps * pages, generator=g)[:T].to(torch.int32).to(DEV)
    slots[7] = -1
    got = []
    for cuts in ([0, 130], [0, 63, 66, 130], [0, 1, 64, 130]):
        kc, vc = (torch.zeros(pages, max(nkv, 1), ps, d, dtype=dtype, device=DEV) for _ in range(2))
        q = [F.qkv_post(qkv[lo:hi].contiguous(), b, pos[lo:hi].contiguous(), inv, d if rope else 0,
                        slots[lo:hi].contiguous() if nkv else None, kc if nkv else None, vc if nkv else None, nh, nkv, d, ps, dtype)
             for lo, hi in zip(cuts, cuts[1:])]
        got.append((torch.cat(q), kc, vc))
    for other in got[1:]:
        assert all(torch.equal(x, y) for x, y in zip(got[0], other))
