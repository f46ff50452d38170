"""Decode attention whose splits go as clusters in one launch: the same bits as in two launches, over lengths around the splits'
edges, windows, chunks, an added key with and without scores, capped scores and gates."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
D, PAGE = 128, 16


def F():
    from mini_infer_b200.ops import functional
    return functional


FORMS = {"plain": {}, "window": {"window": 100}, "narrow": {"window": 5}, "chunk": {"chunk": 160}, "cap": {"softcap": 8.0},
         "sink": {"sink": True}, "scores and gates": {"sink": True, "sink_score": True, "gate": True}}


@pytest.mark.parametrize("form", list(FORMS))
@pytest.mark.parametrize("nh,nkv", [(3, 1), (8, 2), (4, 4)])
@pytest.mark.parametrize("split,lengths", [(128, [1, 127, 160, 161, 900]), (256, [64, 320, 321, 2047]), (512, [640, 641, 3000, 7])])
def test_joined_as_in_two_launches(split, lengths, nh, nkv, form):
    g = torch.Generator().manual_seed(split + nh)
    rnd = lambda *s: torch.randn(*s, generator=g).to(DEV)
    i32 = lambda t: torch.as_tensor(t, dtype=torch.int32, device=DEV)
    B = len(lengths)
    counts = [-(-n // PAGE) for n in lengths]
    table = torch.full((B, max(counts)), -1, dtype=torch.int32)
    order, at = torch.randperm(sum(counts), generator=g).to(torch.int32), 0
    for b, n in enumerate(counts):
        table[b, :n] = order[at:at + n]
        at += n
    q, k, v = rnd(B, nh, D).bfloat16(), rnd(sum(counts), nkv, PAGE, D).bfloat16(), rnd(sum(counts), nkv, PAGE, D).bfloat16()
    kw = dict(FORMS[form])
    if kw.get("sink_score"):
        kw["sink_score"] = rnd(nh)
    if kw.get("gate"):
        kw["gate"] = rnd(B, nh + 3)
        kw["gate_col"] = 3
    outs = []
    for splits in (-(-max(lengths) // split), 8, 9):
        joined = bool(F().library().mi_attn_decode_joined(D, B * nh, splits))
        assert joined == (splits <= 8)
        po, pml = rnd(B * nh * splits * D), rnd(B * nh * splits * 2)
        before = po.clone()
        outs.append(F().decode_attention(q, k, v, table.to(DEV), i32(range(B + 1)), i32(lengths), po, pml, splits, split=split, **kw))
        assert torch.equal(po, before) == joined          # (the scratch is not touched)
    assert torch.equal(outs[0], outs[2]) and torch.equal(outs[1], outs[2])
    if form == "plain":
        for b, n in enumerate(lengths):
            pages = table[b, :counts[b]].long().to(DEV)
            kk, vv = (x[pages].transpose(1, 2).reshape(-1, nkv, D)[:n].double().repeat_interleave(nh // nkv, 1) for x in (k, v))
            s = torch.softmax(torch.einsum("hd,nhd->hn", q[b].double(), kk) * D ** -0.5, -1)
            ref = torch.einsum("hn,nhd->hd", s, vv)
            # the result is rounded to bfloat16
            assert float((outs[0][b].double() - ref).abs().max()) <= 2.0 ** -8 * float(ref.abs().max()) + 1e-5


def test_which_split_goes_as_clusters():
    f = F()
    got = [f.decode_joined_split(*a) for a in ((1, 8, 128, 300), (1, 8, 128, 1025), (8, 16, 128, 600), (8, 16, 128, 2048),
                                               (64, 16, 128, 3000), (1, 8, 64, 300), (1, 8, 128, 5000))]
    assert got == [128, 256, 256, 512, None, None, None]
