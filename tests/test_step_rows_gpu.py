"""Row kernels of a decode step at the widths where their forms meet, the output head's store, and few-row products whose warps share columns, against float64."""
import pytest
import torch

import seq_cases
import seq_oracle as O
from livecc_b200.checkpoint import synthetic_seq_tensors
from livecc_b200.config import SeqModelConfig
from test_seq_gpu import BF16_TOL, F32_TOL, rel, run

pytestmark = pytest.mark.gpu


# widths on and off 4-column boundaries, at the ends of the register forms (2 and 4 or 8 pieces of 256 x 4 or 256 columns) and one past them
@pytest.mark.parametrize("width", [24, 255, 512, 514, 1024, 2046, 2048, 2052, 4096, 4100])
def test_widths_of_the_row_kernels(width):
    from livecc_b200.seq_engine import SeqLMForCausalLM

    heads = dict(heads=2, kv_heads=1, dim=12, vdim=8) if width % 4 else dict(heads=4, kv_heads=2, dim=16, vdim=8)
    d = seq_cases.config([seq_cases.par(**heads, ff=None)], width=width, vocab=70, softcap=8.0)
    cfg = SeqModelConfig.from_json(d)
    t = synthetic_seq_tensors(cfg, seed=3)
    toks = seq_cases.tokens(5, 70, seed=width)
    want, _ = O.forward(d, t, toks)
    for dtype, tol in (("float32", F32_TOL), ("bfloat16", BF16_TOL)):
        m = SeqLMForCausalLM.from_state_dict(cfg, t, dtype)
        assert rel(run(m, toks, [3, 4]), want) < tol


# head sizes of the q/k norm's register forms: 2 x 1024 and 4 x 1024 query columns, one past them, and columns off 4-element boundaries
@pytest.mark.parametrize("heads,kv,dim", [(2, 1, 10), (8, 2, 256), (9, 3, 228), (16, 4, 256), (17, 1, 256), (4, 4, 260)])
def test_widths_of_the_query_and_key_norm(heads, kv, dim):
    from livecc_b200.seq_engine import SeqLMForCausalLM

    d = seq_cases.config([seq_cases.par(heads=heads, kv_heads=kv, dim=dim, vdim=8, scale=dim ** -0.5, ff=None)], width=40)
    cfg = SeqModelConfig.from_json(d)
    t = synthetic_seq_tensors(cfg, seed=3)
    toks = seq_cases.tokens(6, 96, seed=dim)
    want, _ = O.forward(d, t, toks)
    for dtype, tol in (("float32", F32_TOL), ("bfloat16", BF16_TOL)):
        m = SeqLMForCausalLM.from_state_dict(cfg, t, dtype)
        assert rel(run(m, toks, [4, 5]), want) < tol


@pytest.mark.parametrize("cap,scale", [(8.0, 1.0), (8.0, 0.7), (0.0, 0.7)])
@pytest.mark.parametrize("vocab", [32, 200, 203, 1000])
@pytest.mark.parametrize("rows", [9, 64, 129])
def test_cap_and_scale_of_many_rows_equal_those_of_one(rows, vocab, cap, scale):
    """Logits of many rows are capped and scaled in the product's store (or behind it where the tensor cores do not take the sizes), those of one row in
    another kernel's. The two sums differ by the order of 72 products, which neither a cap (slope at most 1) nor a scale below 1 widens; tanh rounds at 2^-22."""
    from livecc_b200.seq_engine import SeqLMForCausalLM

    d = seq_cases.config([seq_cases.ssd(heads=2, vdim=8, state=8, groups=1)], width=72, vocab=vocab, softcap=cap)
    d["logit_scale"] = scale
    cfg = SeqModelConfig.from_json(d)
    assert cfg.logit_scale == scale
    m = SeqLMForCausalLM.from_state_dict(cfg, synthetic_seq_tensors(cfg, seed=3), "bfloat16")
    toks = seq_cases.tokens(rows, vocab, seed=rows)

    def logits(want):
        c = m.new_cache()
        out = m.forward_step([(c, toks)], [want])
        c.release()
        return out

    many = logits(list(range(rows)))
    for k in (0, rows // 2, rows - 1):
        assert (many[k] - logits([k])[0]).abs().max() <= 72 * 2.0 ** -23 * 1.25 * 72 ** 0.5 + cap * 2.0 ** -22


# either side of the rows from which the embedding takes four columns per thread, widths off 4 and past a pass of 1024; norm groups of a warp: up to 128, 256, 512, and past it
@pytest.mark.parametrize("rows,width", [(148, 24), (149, 24), (149, 255), (150, 1028), (149, 252), (149, 256), (148, 256), (150, 260)])
def test_embedding_of_many_rows(rows, width):
    from livecc_b200.seq_engine import SeqLMForCausalLM

    heads = dict(heads=2, kv_heads=1, dim=12, vdim=8) if width % 4 else dict(heads=4, kv_heads=2, dim=16, vdim=8)
    d = seq_cases.config([seq_cases.par(**heads, ff=None)], width=width, vocab=70, softcap=8.0)
    cfg = SeqModelConfig.from_json(d)
    t = synthetic_seq_tensors(cfg, seed=3)
    toks = seq_cases.tokens(rows, 70, seed=width)
    want, _ = O.forward(d, t, toks)
    for dtype, tol in (("float32", F32_TOL), ("bfloat16", BF16_TOL)):
        m = SeqLMForCausalLM.from_state_dict(cfg, t, dtype)
        assert rel(run(m, toks, [rows]), want) < tol


@pytest.mark.parametrize("heads,vdim,groups", [(1, 132, 1), (2, 128, 1), (4, 65, 1), (4, 128, 1), (8, 128, 2), (4, 129, 1)])
def test_groups_of_the_gated_norm(heads, vdim, groups):
    from livecc_b200.seq_engine import SeqLMForCausalLM

    d = seq_cases.config([seq_cases.ssd(heads=heads, vdim=vdim, state=16, groups=1, norm_groups=groups)], width=40, vocab=70)
    cfg = SeqModelConfig.from_json(d)
    t = synthetic_seq_tensors(cfg, seed=5)
    toks = seq_cases.tokens(35, 70, seed=vdim)
    want, _ = O.forward(d, t, toks)
    for dtype, tol in (("float32", F32_TOL), ("bfloat16", BF16_TOL)):
        m = SeqLMForCausalLM.from_state_dict(cfg, t, dtype)
        assert rel(run(m, toks, [33, 34, 35]), want) < tol


@pytest.mark.parametrize("heads,vdim", [(4, 128), (4, 65)])
def test_gated_norm_has_the_same_bits_for_few_and_many_rows(heads, vdim):
    """8 groups of rows: more than 2960 (row, group) pairs go a warp to a group, fewer a CTA; both sum in one order. The scan in front is cut at the same
    blocks of 64 rows, and the products behind one row alone are those of many on the CUDA cores (fp32 storage)."""
    from livecc_b200.seq_engine import SeqLMForCausalLM

    d = seq_cases.config([seq_cases.ssd(heads=8 * heads, vdim=vdim, state=8, groups=1, norm_groups=8)], width=24, vocab=40)
    cfg = SeqModelConfig.from_json(d)
    m = SeqLMForCausalLM.from_state_dict(cfg, synthetic_seq_tensors(cfg, seed=5), "float32", max_tokens=512)
    toks = seq_cases.tokens(394, 40, seed=vdim)
    many, few = run(m, toks, [384]), run(m, toks, [128, 256, 384])
    assert torch.equal(many[:384], few[:384])


@pytest.mark.parametrize("rows,width", [(296, 260), (297, 260), (297, 1028), (297, 1030), (1184, 2052), (1185, 2052)])
@pytest.mark.parametrize("branches", [1, 2])
def test_post_norms_with_and_without_kept_weights(rows, width, branches):
    """Rows from which the norms' weights are no longer kept in registers, in rows of one, two and four pieces, on and off 4-column boundaries."""
    from livecc_b200.seq_engine import SeqLMForCausalLM

    layer = (seq_cases.ssd(heads=2, vdim=8, state=8, groups=1, norm_groups=1) if branches == 1 else
             seq_cases.par(**(dict(heads=2, kv_heads=1, dim=10, vdim=8) if width % 4 else dict(heads=4, kv_heads=2, dim=16, vdim=8)), ff=None))
    d = seq_cases.config([layer], width=width, vocab=70)
    cfg = SeqModelConfig.from_json(d)
    t = synthetic_seq_tensors(cfg, seed=3)
    toks = seq_cases.tokens(rows, 70, seed=width)
    want, _ = O.forward(d, t, toks)
    for dtype, tol in (("float32", F32_TOL), ("bfloat16", BF16_TOL)):
        m = SeqLMForCausalLM.from_state_dict(cfg, t, dtype, max_tokens=2048)
        assert rel(run(m, toks, [rows]), want) < tol


@pytest.mark.parametrize("width", [260, 1030, 1536])
def test_post_norms_have_the_same_bits_for_few_and_many_rows(width):
    """320 rows load the norms' weights behind the sums, 256 and 64 in front. The scans in front are cut at the same blocks of 64 rows, and the products in
    fp32 storage are those of many rows on the CUDA cores."""
    from livecc_b200.seq_engine import SeqLMForCausalLM

    par = seq_cases.par(**(dict(heads=2, kv_heads=1, dim=10, vdim=8) if width % 4 else dict(heads=4, kv_heads=2, dim=16, vdim=8)), ff=None)
    d = seq_cases.config([seq_cases.ssd(heads=2, vdim=8, state=8, groups=1, norm_groups=1), par], width=width, vocab=40)
    cfg = SeqModelConfig.from_json(d)
    m = SeqLMForCausalLM.from_state_dict(cfg, synthetic_seq_tensors(cfg, seed=5), "float32", max_tokens=512)
    toks = seq_cases.tokens(320, 40, seed=width)
    many, few = run(m, toks, [320]), run(m, toks, [256, 320])
    assert torch.equal(many, few)
