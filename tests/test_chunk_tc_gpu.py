"""The block form of the state-space recurrence on bf16 rows (tensor-core products of values cut in three) against the float64 oracle: sizes at
the edges of its tiles of 64 rows, 64 channels and 64 / 128 key channels, several heads per group, short last blocks, states that enter
from an earlier portion. What bf16 storage allows is the bound; the same rows token by token are no closer to the oracle."""
import pytest
import torch

import seq_cases
import seq_oracle
from livecc_b200.checkpoint import synthetic_seq_tensors
from livecc_b200.config import SeqModelConfig

pytestmark = pytest.mark.gpu
BF16_TOL = 4e-2


def _errors(d, n, portions, seed):
    from livecc_b200.seq_engine import SeqLMForCausalLM

    cfg = SeqModelConfig.from_json(d)
    t = synthetic_seq_tensors(cfg, seed=seed)
    toks = seq_cases.tokens(n, d["vocab"], seed=seed)
    want = seq_oracle.forward(d, t, toks)[0].double()
    m = SeqLMForCausalLM.from_state_dict(cfg, t, "bfloat16", max_tokens=n + 64)
    out = []
    for cuts in portions:
        c, rows, lo = m.new_cache(), [], 0
        for hi in list(cuts) + [n]:
            rows.append(m.forward_step([(c, toks[lo:hi])], [list(range(hi - lo))]).cpu())
            lo = hi
        c.release()
        got = torch.cat(rows).double()
        assert bool(torch.isfinite(got).all())
        out.append((got - want).pow(2).mean(-1).sqrt() / want.pow(2).mean(-1).sqrt().clamp_min(1e-30))
    return out


@pytest.mark.parametrize("heads,vdim,state,groups,n,cut", [
    (4, 64, 128, 1, 130, 65), (8, 64, 64, 8, 192, 64), (2, 72, 136, 2, 193, 128), (6, 8, 16, 3, 100, 33), (3, 128, 72, 1, 129, 1), (2, 16, 256, 1, 64, 40),
])
def test_block_form_on_tensor_cores(heads, vdim, state, groups, n, cut):
    d = seq_cases.config([seq_cases.ssd(heads=heads, vdim=vdim, state=state, groups=groups, conv=4, norm_groups=1) for _ in range(2)], width=48)
    whole, parts, single = _errors(d, n, [[], [cut], range(1, n)], seed=heads + state)
    for e in (whole, parts):
        assert float(e.max()) < BF16_TOL and float(e.median()) < 1.2 * float(single.median()) + 1e-4, (float(e.max()), float(e.median()), float(single.median()))
