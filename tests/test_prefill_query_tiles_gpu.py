"""The tcgen05 prefill attention in every pairing of query tiles (one alone, far apart, neighbours), which the number of
heads and the length choose: ragged requests against plain attention in float32."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def i32(v):
    return torch.tensor(v, dtype=torch.int32, device=DEV)


# (heads, key heads): 60 heads x 3 tiles fill more than one wave alone and less than one in pairs; 80 heads do not
@pytest.mark.parametrize("nh,nkv", [(2, 1), (60, 4), (80, 80)])
@pytest.mark.parametrize("q_lens,past", [([300], [0]), ([129], [70]), ([257, 1, 128], [0, 500, 63]), ([384, 400], [33, 0])])
@pytest.mark.parametrize("window", [0, 150])
@pytest.mark.parametrize("d", [64, 128])
def test_pairs_of_query_tiles(nh, nkv, q_lens, past, window, d):
    from mini_infer_b200.ops import functional as F
    g = torch.Generator(device=DEV).manual_seed(nh + len(q_lens) + window)
    page, ends = 16, [p + n for p, n in zip(past, q_lens)]
    counts = [-(-e // page) for e in ends]
    order = torch.randperm(sum(counts), generator=torch.Generator().manual_seed(1)).tolist()
    table, at = torch.full((len(ends), max(counts)), -1, dtype=torch.int32), 0
    for b, n in enumerate(counts):
        table[b, :n] = torch.tensor(order[at:at + n], dtype=torch.int32)
        at += n
    kc, vc = (torch.randn(sum(counts), nkv, page, d, generator=g, device=DEV).bfloat16() for _ in range(2))
    q = torch.randn(sum(q_lens), nh, d, generator=g, device=DEV).bfloat16()
    starts = [sum(q_lens[:b]) for b in range(len(q_lens) + 1)]
    out = F.prefill_attention_tc(q, kc, vc, table.to(DEV), i32(starts), i32(ends), max(q_lens), window)
    F.check_tc_status()
    for b, (lo, hi) in enumerate(zip(starts, starts[1:])):
        rows = table[b, :counts[b]].long().to(DEV)
        k, v = (c[rows].transpose(1, 2).reshape(-1, nkv, d)[:ends[b]].float().repeat_interleave(nh // nkv, 1) for c in (kc, vc))
        s = torch.einsum("qhd,khd->hqk", q[lo:hi].float(), k) * d ** -0.5
        pos, key = torch.arange(past[b], ends[b], device=DEV)[:, None], torch.arange(ends[b], device=DEV)[None]
        s = s.masked_fill((key > pos) | ((key <= pos - window) if window else (key < 0)), -torch.inf)
        ref = torch.einsum("hqk,khd->qhd", torch.softmax(s, -1), v)
        # weights and result are rounded to bfloat16: half a unit in the last place (2^-9) each, of values up to max |v|
        assert float((out[lo:hi].float() - ref).abs().max()) <= 2.0 ** -8 * float(v.abs().max())
