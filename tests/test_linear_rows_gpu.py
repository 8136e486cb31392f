"""Few-row products of the hybrid models at the limits of their forms (columns per warp, warps per column), in one row and in several: the output head's
store against float64 torch, and a row's bits whatever stands beside it."""
import pytest
import torch

import seq_cases
import seq_oracle as O
from livecc_b200.checkpoint import synthetic_seq_tensors
from livecc_b200.config import SeqModelConfig
from test_seq_gpu import BF16_TOL, F32_TOL, rel, run

pytestmark = pytest.mark.gpu


# k of a product (the model's width, the feed-forward's) around 1024, 2048, 4096 and 6144 in bf16 and half of that in fp32; columns (vocabulary, 2 x ff)
# around 888, 1024, 1184, 2048, 2664, 4096, 4608 and 8192
@pytest.mark.parametrize("width,ff,vocab", [(512, 1016, 4095), (520, 2048, 4097), (1016, 2056, 8191), (1024, 4096, 8193), (1032, 4104, 4096), (2048, 6144, 8192), (264, 6152, 333),
                                            (1024, 2048, 888), (1024, 2056, 896), (1024, 1032, 1184), (1032, 4096, 1192), (2048, 512, 2664), (2048, 4096, 2672),
                                            (4096, 1024, 4608), (4096, 1016, 4616), (2056, 264, 2048)])
def test_products_at_the_limits_of_their_forms(width, ff, vocab):
    from livecc_b200.seq_engine import SeqLMForCausalLM

    d = seq_cases.config([seq_cases.ssd(heads=2, vdim=8, state=8, groups=1, norm_groups=1, ff=ff)], width=width, vocab=vocab, softcap=6.0)
    cfg = SeqModelConfig.from_json(d)
    t = synthetic_seq_tensors(cfg, seed=9)
    toks = seq_cases.tokens(12, vocab, seed=ff)
    want, _ = O.forward(d, t, toks)
    for dtype, tol in (("float32", F32_TOL), ("bfloat16", BF16_TOL)):
        m = SeqLMForCausalLM.from_state_dict(cfg, t, dtype)
        assert rel(run(m, toks, [1, 3, 8]), want) < tol        # products of 1, 2, 5 and 4 rows
        alone = []
        for n in (1, 2, 4, 8):                                  # the same token behind the same row, n sequences in one step
            caches = [m.new_cache() for _ in range(n)]
            for c in caches:
                m.forward_step([(c, toks[:1])], [[0]])
            alone.append(m.forward_step([(c, toks[1:2]) for c in caches], [[0]] * n).cpu())
            for c in caches:
                c.release()
        for got in alone:
            assert all(torch.equal(row, alone[0][0]) for row in got)
