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
