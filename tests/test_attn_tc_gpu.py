"""Prompt attention of the hybrid models on tcgen05 (heads of 128 channels) against the float64 oracles: windows, chunks, sinks, gates per
channel and per head, one to all query heads on a key head, portions that start and end anywhere in a 64-token page, windows inside,
on and outside page borders, with a mild and with a sharp softmax. Pages start out full of NaN, so nothing past the newest token or
in front of the window may be touched by a product."""
import pytest
import torch

import dibedra_cases
import dibedra_oracle
import seq_cases
import seq_oracle
from livecc_b200.checkpoint import synthetic_seq_tensors
from livecc_b200.config import SeqModelConfig

pytestmark = pytest.mark.gpu
# bf16 storage and bf16 softmax weights: the bound that the other bf16 tests of these models use for the worst row
BF16_TOL = 4e-2


def _check(d, oracle, cuts, n, seed):
    from livecc_b200.seq_engine import SeqLMForCausalLM

    cfg = SeqModelConfig.from_json(d)
    t = synthetic_seq_tensors(cfg, seed=seed)
    toks = seq_cases.tokens(n, d["vocab"], seed=seed)
    want = oracle.forward(d, t, toks)
    want = (want[0] if isinstance(want, tuple) else want).double()
    m = SeqLMForCausalLM.from_state_dict(cfg, t, "bfloat16", max_tokens=n + 64)
    for pages in (m.pool.k, m.pool.v):
        for x in (pages.values() if isinstance(pages, dict) else pages):
            if x is not None:
                x.fill_(float("nan"))
    c, rows, lo = m.new_cache(), [], 0
    for hi in list(cuts) + [n]:
        rows.append(m.forward_step([(c, toks[lo:hi])], [list(range(hi - lo))]).cpu())
        lo = hi
    c.release()
    got = torch.cat(rows).double()
    err = (got - want).pow(2).mean(-1).sqrt() / want.pow(2).mean(-1).sqrt().clamp_min(1e-30)
    assert bool(torch.isfinite(got).all()) and float(err.max()) < BF16_TOL, (float(err.max()), int(err.argmax()))


CUTS = [16, 33, 97, 161, 164, 228]      # portions of 16, 17, 64, 64, 3, 64 and the rest


@pytest.mark.parametrize("heads,kv_heads,window,scale,cuts,n", [
    (8, 1, 1000, 0.09, CUTS, 300),      # a window that reaches back to the start
    (8, 1, 64, 0.09, CUTS, 300), (8, 2, 65, 0.5, CUTS, 300), (4, 4, 63, 0.09, CUTS, 300), (6, 2, 10, 0.5, CUTS, 300),
    (16, 2, 100, 0.09, [], 513), (7, 1, 130, 0.5, [1], 290), (3, 1, 1, 0.09, [40], 80), (16, 1, 200, 0.09, [255], 271),
])
def test_windows_and_channel_gates(heads, kv_heads, window, scale, cuts, n):
    d = dibedra_cases.config([dibedra_cases.att(heads=heads, kv_heads=kv_heads, dim=128, window=window, rot_dims=64, scale=scale) for _ in range(2)], width=64)
    _check(d, dibedra_oracle, cuts, n, seed=heads + window)


@pytest.mark.parametrize("heads,kv_heads,chunk,scale,cuts,n", [
    (8, 1, 64, 0.09, CUTS, 300), (4, 2, 100, 0.5, CUTS, 300), (2, 2, 1024, 0.09, [], 400), (16, 2, 40, 0.5, [129], 280),
])
def test_chunks_sinks_and_head_gates(heads, kv_heads, chunk, scale, cuts, n):
    d = seq_cases.config([seq_cases.par(heads=heads, kv_heads=kv_heads, dim=128, vdim=128, chunk=chunk, scale=scale) for _ in range(2)], width=40)
    _check(d, seq_oracle, cuts, n, seed=heads + chunk)


def _op_case(S, past, Hq, G, seed, vscale=1.0):
    g = torch.Generator().manual_seed(seed)
    pages = (past + S + 63) // 64
    order = torch.randperm(pages, generator=g)
    kv = torch.full((2, pages, G, 64, 128), float("nan"))
    flat = torch.randn((2, G, past + S, 128), generator=g)
    flat[1] *= vscale
    flat = flat.to(torch.bfloat16).float()
    for t in range(past + S):
        kv[:, order[t // 64], :, t % 64] = flat[:, :, t]
    q = torch.randn((S, Hq, 128), generator=g).to(torch.bfloat16).float()
    return q.cuda(), kv[0].bfloat16().cuda(), kv[1].bfloat16().cuda(), order.int().cuda(), flat.double().cuda()


def _op_want(q, flat, past, scale, chunk, window, sink, gate):
    S, Hq, _ = q.shape
    k, v = (x.repeat_interleave(Hq // flat.shape[1], 0) for x in flat)
    s = torch.einsum("shd,htd->hst", q.double(), k) * scale
    i, j = torch.arange(past, past + S, device="cuda")[:, None], torch.arange(past + S, device="cuda")[None]
    see = (j <= i) & ((j > i - window) if window else True) & ((j // chunk == i // chunk) if chunk else True)
    s = s.masked_fill(~see, float("-inf"))
    m = s.amax(-1, keepdim=True).clamp_min(0.0 if sink else -1e300)
    p = (s - m).exp()
    o = torch.einsum("hst,htd->shd", p / (p.sum(-1, keepdim=True) + ((-m).exp() if sink else 0.0)), v)
    return o if gate is None else o * torch.sigmoid(gate.double()).view(S, Hq, -1)


@pytest.mark.parametrize("S,past,Hq,G,chunk,window", [(70, 0, 8, 1, 100, 30), (130, 77, 4, 2, 128, 64), (65, 191, 6, 2, 64, 1000), (200, 300, 16, 2, 150, 149), (17, 63, 3, 1, 16, 5)])
@pytest.mark.parametrize("sink", [False, True])
@pytest.mark.parametrize("gated", [0, 1, 2])
def test_window_and_chunks_together(ctx, S, past, Hq, G, chunk, window, sink, gated):
    q, k, v, table, flat = _op_case(S, past, Hq, G, S + past)
    gate = None if not gated else torch.randn((S, Hq * (128 if gated == 2 else 1)), device="cuda").bfloat16()
    if gated == 1:    # (a gate per head is one column of a wider row in the models)
        gate = torch.cat([gate, gate], 1)[:, :Hq]
    got = ctx.attn_masked(q, k, v, table, past, 0.09, chunk=chunk, window=window, sink=sink, gate=gate, gate_channel=gated == 2)
    want = _op_want(q, flat, past, 0.09, chunk, window, sink, gate)
    # softmax weights and the result are rounded to bf16 (2^-9 each, weights relative to values of size 1)
    assert bool(((got.double() - want).abs() <= 2.0 ** -8 * (want.abs() + 1.0) * 1.5).all())


@pytest.mark.parametrize("gated", [1, 2])
def test_gates_that_are_nearly_shut(ctx, gated):
    """sigmoid(-88) is 6e-39, a normal quotient of a denominator past 2^126: values of 1e30 come out as 6e-9, not as zeros."""
    q, k, v, table, flat = _op_case(80, 20, 4, 1, 3, vscale=1e30)
    gate = torch.full((80, 4 * (128 if gated == 2 else 1)), -88.0, device="cuda").bfloat16()
    got = ctx.attn_masked(q, k, v, table, 20, 0.09, gate=gate, gate_channel=gated == 2).double()
    want = _op_want(q, flat, 20, 0.09, 0, 0, False, gate)
    assert bool(((got - want).abs() <= 2.0 ** -8 * 1.5 * (want.abs() + 1e30 * 6e-39)).all()) and float(got.abs().max()) > 1e-9
