"""Row lists of routed layers against the oracle: numbers of experts either side of a warp and at the largest router, lists without rows, dense lists (fp32)
and lists padded to whole tiles (bf16 on the tensor cores)."""
import pytest

import dibedra_cases as K
import dibedra_oracle as O
from livecc_b200.checkpoint import synthetic_seq_tensors
from livecc_b200.config import SeqModelConfig
from test_dibedra_gpu import F32_TOL, bf16_ok, build, rel, run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("experts,identity,top,dtype", [(1, 0, 1, "float32"), (31, 1, 2, "float32"), (32, 0, 3, "float32"), (33, 0, 2, "float32"), (65, 3, 2, "float32"),
                                                        (509, 3, 2, "float32"), (31, 1, 2, "bfloat16"), (32, 0, 3, "bfloat16"), (65, 0, 2, "bfloat16")])
def test_lists_of_many_experts(experts, identity, top, dtype):
    ff = 64 if dtype == "bfloat16" else 6
    d = K.config([K.att(heads=2, kv_heads=1, dim=8, window=40, mlp=K.moe(experts=experts, top=top, ff=ff, limit=1.0, identity=identity))], width=64, vocab=64)
    tensors = synthetic_seq_tensors(SeqModelConfig.from_json(d), seed=25)
    toks = K.tokens(300, d["vocab"], seed=experts)
    want = O.forward(d, tensors, toks)
    got = run(build(d, tensors, dtype), toks, [])
    assert rel(got, want) < F32_TOL if dtype == "float32" else bf16_ok(got, want)
