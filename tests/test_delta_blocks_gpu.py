"""The delta rule walked in blocks of eight tokens: against the recurrence in float64 and no further from it than the walk
token by token, at lengths around a block's edges, from states that are not zero."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def recurrence(qkv, beta_raw, a_raw, a_log, dt_bias, S, H, G, d, dv, scale):
    qkv, beta, S = qkv.double(), torch.sigmoid(beta_raw.double()), S.double().clone()
    g = torch.exp(-torch.exp(a_log.double()) * torch.nn.functional.softplus(a_raw.double() + dt_bias.double()))
    unit = lambda t: t / (t.pow(2).sum(-1, keepdim=True) + 1e-6).sqrt()
    n = qkv.shape[0]
    q = (unit(qkv[:, :G * d].view(n, G, d)) * scale).repeat_interleave(H // G, 1)
    k = unit(qkv[:, G * d:2 * G * d].view(n, G, d)).repeat_interleave(H // G, 1)
    v = qkv[:, 2 * G * d:2 * G * d + H * dv].view(n, H, dv)
    out = []
    for t in range(n):
        S = S * g[t][:, None, None]
        u = beta[t][:, None] * (v[t] - torch.einsum("hkv,hk->hv", S, k[t]))
        S = S + k[t][:, :, None] * u[:, None]
        out.append(torch.einsum("hkv,hk->hv", S, q[t]).reshape(-1))
    return torch.stack(out), S


@pytest.mark.parametrize("lengths", [[8], [1, 7, 9], [16, 61, 3], [200]])
@pytest.mark.parametrize("H,G,d,dv", [(2, 1, 64, 64), (3, 3, 128, 20), (4, 2, 128, 128), (1, 1, 64, 33)])
@pytest.mark.parametrize("decay", [-4.0, 0.0, 3.0])
def test_blocks_against_the_recurrence(lengths, H, G, d, dv, decay):
    from mini_infer_b200.ops import functional as F
    g = torch.Generator().manual_seed(sum(lengths) + d + dv)
    rnd = lambda *s: torch.randn(*s, generator=g).to(DEV)
    T, B, ch = sum(lengths), len(lengths), 2 * G * d + H * dv
    qkv, raw = rnd(T, ch + 4), rnd(T, 2 * H + 3)
    a_log, dt_bias = rnd(H) * 0.3 + decay, rnd(H)
    state = rnd(B + 1, H * d * dv + 5)
    slots = torch.arange(B, 0, -1, dtype=torch.int32, device=DEV)
    starts = torch.tensor([sum(lengths[:b]) for b in range(B + 1)], dtype=torch.int32, device=DEV)
    error = {}
    for blocks in (0, max(lengths)):
        st = state.clone()
        out = F.delta_scan(qkv, raw, 1, raw, H + 2, a_log, dt_bias, st, 5, starts, slots, H, G, d, dv, d ** -0.5,
                           form="head_decay", blocks_of=blocks)
        diff = ref_sq = 0.0
        for b, n in enumerate(lengths):
            lo, slot = int(starts[b]), int(slots[b])
            o, S = recurrence(qkv[lo:lo + n], raw[lo:lo + n, 1:1 + H], raw[lo:lo + n, H + 2:2 * H + 2], a_log, dt_bias,
                              state[slot, 5:].view(H, d, dv), H, G, d, dv, d ** -0.5)
            for got, ref in ((out[lo:lo + n], o), (st[slot, 5:].view(H, d, dv), S)):
                diff += float((got.double() - ref).pow(2).sum())
                ref_sq += float(ref.pow(2).sum())
        assert torch.equal(st[0], state[0]) and torch.equal(st[:, :5], state[:, :5])
        error[bool(blocks)] = (diff / ref_sq) ** 0.5
    print(lengths, H, G, d, dv, decay, error)
    # sums of d numbers in float32, in two orders: half a unit of rounding per addition, added as a random walk
    assert error[True] <= max(1.5 * error[False], 2.0 ** -24 * d ** 0.5)


@pytest.mark.parametrize("d", [64, 128])
def test_the_length_given_sizes_the_launch_only(d):
    from mini_infer_b200.ops import functional as F
    g = torch.Generator().manual_seed(d)
    rnd = lambda *s: torch.randn(*s, generator=g).to(DEV)
    lengths, H, G, dv = [131, 9], 4, 2, 48
    T, starts = sum(lengths), torch.tensor([0, 131, 140], dtype=torch.int32, device=DEV)
    slots = torch.tensor([1, 0], dtype=torch.int32, device=DEV)
    qkv, raw, a_log, dt_bias, state = rnd(T, 2 * G * d + H * dv), rnd(T, 2 * H), rnd(H) * 0.3, rnd(H), rnd(2, H * d * dv)
    got = []
    for blocks_of in (131, 1, 17, 1000):
        st = state.clone()
        junk = torch.full((1 << 22,), float("nan"), device=DEV)       # what the scratch finds
        del junk
        got.append((F.delta_scan(qkv, raw, 0, raw, H, a_log, dt_bias, st, 0, starts, slots, H, G, d, dv, d ** -0.5,
                                 form="head_decay", blocks_of=blocks_of), st))
    for out, st in got[1:]:
        assert torch.equal(out, got[0][0]) and torch.equal(st, got[0][1])


@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
@pytest.mark.parametrize("where", ["value", "key", "query", "strength", "decay"])
def test_tokens_before_one_that_is_not_finite_stay_as_they_are(where, bad):
    from mini_infer_b200.ops import functional as F
    g = torch.Generator().manual_seed(5)
    rnd = lambda *s: torch.randn(*s, generator=g).to(DEV)
    n, H, G, d, dv, at = 21, 2, 1, 64, 32, 13
    i32 = lambda t: torch.tensor(t, dtype=torch.int32, device=DEV)
    qkv, raw, a_log, dt_bias, state = rnd(n, 2 * G * d + H * dv), rnd(n, 2 * H), rnd(H) * 0.3, rnd(H), rnd(1, H * d * dv)
    run = lambda: F.delta_scan(qkv, raw, 0, raw, H, a_log, dt_bias, state.clone(), 0, i32([0, n]), i32([0]), H, G, d, dv,
                               d ** -0.5, form="head_decay", blocks_of=n)
    clean = run()
    if where in ("strength", "decay"):
        raw[at, 0 if where == "strength" else H] = bad
    else:
        qkv[at, {"query": 7, "key": G * d + 7, "value": 2 * G * d + 7}[where]] = bad
    out = run()
    assert torch.equal(out[:at], clean[:at])
    if where == "value":                # one column of one head
        others = [c for c in range(H * dv) if c != 7]
        assert not torch.isfinite(out[at, 7]) and torch.equal(out[:, others], clean[:, others])


@pytest.mark.parametrize("lengths,blocks", [([47], 0), ([48], 48), ([48, 48], 48), ([100, 1], 100), ([1] * 7 + [48], 0),
                                             ([1] * 7 + [69], 69), ([1] * 31 + [100], 0), ([1] * 31 + [141], 141),
                                             ([8] * 31 + [48], 48), ([40] * 8, 0)])
def test_which_steps_walk_in_blocks(lengths, blocks):
    from types import SimpleNamespace
    from mini_infer_b200.parts.recurrent import GatedDelta
    ctx = SimpleNamespace(num_tokens=sum(lengths), num_requests=len(lengths), max_q_len=max(lengths))
    layer = lambda act, d: SimpleNamespace(rt=SimpleNamespace(act=act), d=d)
    assert GatedDelta._blocks_of(layer(torch.bfloat16, 128), ctx) == blocks
    assert GatedDelta._blocks_of(layer(torch.bfloat16, 96), ctx) == 0
    assert GatedDelta._blocks_of(layer(torch.float32, 128), ctx) == 0


def test_blocks_are_refused_where_they_are_not_built():
    from mini_infer_b200.ops import functional as F
    z = torch.zeros(8, 400, device=DEV)
    i = torch.tensor([0, 8], dtype=torch.int32, device=DEV)
    for form, d in (("channel_decay", 64), ("head_decay", 96)):
        n = 64 if form == "channel_decay" else 1
        with pytest.raises(ValueError, match="blocks"):
            F.delta_scan(z, z, 0, z, 0, torch.zeros(1, device=DEV), torch.zeros(n, device=DEV), torch.zeros(1, d * 16, device=DEV),
                         0, i, i[:1].contiguous(), 1, 1, d, 16, 1.0, form=form, blocks_of=8)
