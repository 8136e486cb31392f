"""One token of a gated recurrence in one kernel (decode steps of state-space and linear-attention layers), at the sizes it takes: against the float64
oracle token by token behind a prompt, against the kernels that longer portions use, and in batches beside prompts."""
import re
from pathlib import Path

import pytest
import torch

import seq_cases
import seq_oracle as O
from livecc_b200 import _cabi
from livecc_b200.checkpoint import synthetic_seq_tensors
from livecc_b200.config import SeqModelConfig
from test_seq_gpu import BF16_TOL, F32_TOL, rel, run

pytestmark = pytest.mark.gpu
CSRC = Path(__file__).resolve().parent.parent / "livecc_b200" / "csrc"

# layers whose recurrence the kernel takes: 1, 2, 4 and 8 pieces of state per thread, states of 32, 64 and 128, 2 to 4 taps, one and several key
# groups per norm group, one and several clusters
TAKEN = {
    "ssd_1": seq_cases.ssd(heads=4, vdim=64, state=32, groups=4, conv=3, norm_groups=1),
    "ssd_2": seq_cases.ssd(heads=16, vdim=32, state=64, groups=2, conv=4, norm_groups=2, ff=24),
    "ssd_4": seq_cases.ssd(heads=8, vdim=32, state=128, groups=1, conv=2, norm_groups=1),
    "ssd_8": seq_cases.ssd(heads=16, vdim=64, state=128, groups=4, conv=4, norm_groups=2),
    "gla_1": seq_cases.par(r_heads=2, r_dim=128, r_vdim=64, chunk=40),
    "gla_2": seq_cases.par(r_heads=1, r_dim=64, r_vdim=256, chunk=40),
    "gla_4": seq_cases.par(r_heads=3, r_dim=128, r_vdim=256, chunk=40, ff=None),
}
LEFT = {   # a size next to a limit: the kernels of longer portions serve it
    "taps_5": seq_cases.ssd(heads=4, vdim=64, state=32, groups=4, conv=5, norm_groups=1),
    "group_over_norms": seq_cases.ssd(heads=8, vdim=64, state=32, groups=1, conv=4, norm_groups=2),
    "state_48": seq_cases.ssd(heads=4, vdim=64, state=48, groups=4, conv=4, norm_groups=1),
    "gla_vdim_48": seq_cases.par(r_heads=2, r_dim=128, r_vdim=48, chunk=40),
}


def build(layer, dtype):
    from livecc_b200.seq_engine import SeqLMForCausalLM

    d = seq_cases.config([layer, layer], width=64)
    cfg = SeqModelConfig.from_json(d)
    tensors = synthetic_seq_tensors(cfg, seed=23)
    return SeqLMForCausalLM.from_state_dict(cfg, tensors, dtype), d, tensors


def launches(m, toks):
    c = m.new_cache()
    m.forward_step([(c, toks[:-1])], [[0]])
    before = _cabi.launch_count()
    m.forward_step([(c, toks[-1:])], [[0]])
    c.release()
    return _cabi.launch_count() - before


@pytest.mark.parametrize("name", list(TAKEN) + list(LEFT))
def test_steps_match_the_oracle(name):
    layer = TAKEN.get(name) or LEFT[name]
    toks = seq_cases.tokens(52, 96, seed=5)
    for dtype, tol in (("float32", F32_TOL), ("bfloat16", BF16_TOL)):
        m, d, tensors = build(layer, dtype)
        want, _ = O.forward(d, tensors, toks)
        assert rel(run(m, toks, [40] + list(range(41, 52))), want) < tol, dtype      # 40 rows together, then one by one
        assert rel(run(m, toks, list(range(1, 52))), want) < tol, dtype              # from an empty state
    per = 2 * (3 if layer["type"] == "mamba2" else 2)                                # links that became one, in two layers
    other = build(next(iter(LEFT.values())) if layer["type"] == "mamba2" else LEFT["gla_vdim_48"], "float32")[0]
    extra = 2 * 4 if layer["mlp"] and layer["type"] == "mamba2" else (-2 * 4 if layer["type"] == "parallel" and not layer["mlp"] else 0)
    assert launches(m, toks) - extra == launches(other, toks) - (per if name in TAKEN else 0)


@pytest.mark.parametrize("name", ["ssd_2", "gla_2"])
def test_a_token_beside_a_prompt_has_its_own_bits(name):
    m, d, _ = build(TAKEN[name], "bfloat16")
    a, b = seq_cases.tokens(30, 96, seed=1), seq_cases.tokens(21, 96, seed=2)

    def after(order):
        ca, cb = m.new_cache(), m.new_cache()
        m.forward_step([(ca, a[:-2])], [[0]])
        reqs = [(ca, a[-2:-1]), (cb, b)]
        m.forward_step(reqs if order else [reqs[0]], [[0]] * (2 if order else 1))
        out = m.forward_step([(ca, a[-1:])], [[0]]).cpu()
        ca.release(), cb.release()
        return out

    assert torch.equal(after(True), after(False))


def test_fresh_rows_are_read_behind_the_wait():
    """Read from the source: what the kernel in front writes (projections and decay rows) is not touched before chain_begin."""
    src = re.sub(r"//[^\n]*", "", (CSRC / "recurrent_step.cu").read_text())
    body = src[src.index("scan_step_kernel(const __grid_constant__"):]
    early, late = body[:body.index("chain_begin();")], body[body.index("chain_begin();"):]
    for fresh in ("a.u", "a.k", "a.c,", "a.dec", "a.gate"):
        assert not re.search(re.escape(fresh) + r"(?![a-z_])", early), fresh
        assert fresh == "a.c," or re.search(re.escape(fresh) + r"(?![a-z_])", late), fresh
    assert "__ldg" not in body and "ld_stream16" not in body and "__restrict__" not in body
