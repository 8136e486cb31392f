"""Chained launches of the hybrid sequence models, read from the sources: a kernel that lies on the SMs while the one before it still writes
may take the non-coherent read path (ld.global.nc: explicit, `__ldg`, or a load through a `const __restrict__` parameter) for weights and
tables alone."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "livecc_b200" / "csrc"
FILES = ["rowops", "recurrent", "recurrent_step", "recurrent_chunked", "attn_local", "attn_latent", "hyper", "moe", "rotary", "linear_any"]

# `__restrict__` parameters that no kernel or copy of a pass writes before the kernel reads them: weights and tables, and what it only writes
WEIGHTS = {
    "embed_sinusoid_kernel": "table inv_freq", "postnorm_residual_kernel": "wa wb w", "postnorm_branch_kernel": "ls w",
    "gated_group_norm_kernel": "w", "gated_group_norm4_kernel": "w", "gather_rmsnorm_kernel": "w", "slice_rmsnorm_kernel": "w",
    "branch_norm_residual_kernel": "w", "causal_conv_kernel": "w b", "causal_conv_long_kernel": "w b", "ssm_step_decay_kernel": "dt_bias a_log",
    "gla_decay_kernel": "bias", "qk_headnorm_rope_append_kernel": "qn_w kn_w inv_freq", "qk_norm_kv_append_kernel": "qn_w kn_w",
    "attn_chunk_sink_kernel": "sink", "attn_rows_kernel": "sink", "attn_split_kernel": "sink", "latent_kv_append_kernel": "norm_w inv_freq", "hyper_boundary_kernel": "prev next w",
    "moe_route_kernel": "correction", "moe_route_small_kernel": "correction", "rotary_pack_kernel": "inv_freq",
    "linear_tile_kernel": "W bias", "linear_rows_kernel": "W bias",
}
WRITTEN = {
    "embed_sinusoid_kernel": "x32 xa", "postnorm_residual_kernel": "xa", "postnorm_branch_kernel": "xa", "gated_group_norm_kernel": "out",
    "gated_group_norm4_kernel": "out", "glu_gelu_tanh_kernel": "out", "gather_rmsnorm_kernel": "out", "slice_rmsnorm_kernel": "out",
    "gather_norm_kernel": "out", "residual_norm_kernel": "xa", "glu_clamp_swish_kernel": "out", "branch_norm_residual_kernel": "xa",
    "sandwich_residual_kernel": "xa", "causal_conv_kernel": "out", "causal_conv_long_kernel": "out", "ssm_step_decay_kernel": "dt_out decay_out",
    "gla_decay_kernel": "decay_out", "qk_headnorm_rope_append_kernel": "q_out k_pages v_pages", "qk_norm_kv_append_kernel": "q_out k_pages v_pages",
    "attn_chunk_sink_kernel": "out", "attn_rows_kernel": "out part counters", "attn_split_kernel": "out part counters",
    "diff_combine_kernel": "out",
    "latent_kv_append_kernel": "q_out k_pages", "hyper_boundary_kernel": "xa sum_out", "moe_route_kernel": "sel weight shared_gate counts rank",
    "moe_route_small_kernel": "sel weight shared_gate row_off pos src_row", "moe_index_kernel": "row_off pos src_row tile_group",
    "moe_gather_kernel": "out", "rotary_pack_kernel": "out fill_out", "linear_tile_kernel": "C", "linear_rows_kernel": "C",
}


def kernels(name):
    """(kernel name, parameter text, body) of every __global__ function of a file."""
    src = re.sub(r"//[^\n]*", "", (CSRC / f"{name}.cu").read_text())
    out = []
    for m in re.finditer(r"__global__\s+void\s+(?:__cluster_dims__\([^)]*\)\s*)?(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s*)?(\w+)\(([^{]*)\)\s*\{", src):
        depth, i = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(src[i], 0)
            i += 1
        out.append((m.group(1), m.group(2), src[m.end():i]))
    return src, out


# What is touched in front of the wait, per kernel: elements of arrays in the launch parameters, shared memory behind a pointer in a struct, and
# loads of what nothing writes while the kernel in front runs. Nothing at all may be stored to global memory there.
PARAMETERS = {"attn_prefill_tc_kernel": {"p.ps.st"}}
SHARED = {"gemm_swap_kernel": {"g.flag"}}
EARLY_LOADS = {
    "linear_rows_kernel": {"W"},                          # weights
    # weights, and the state and the carried inputs: their one writer is the same layer's kernel of the step before, a whole step of kernels away
    "scan_step_kernel": {"a.conv_w", "a.conv_b", "a.dt_bias", "a.a_log", "a.skip", "a.norm_w", "a.carry", "a.state"},
    # the form with windows reads its sequence's scalars; it is launched in the ordinary way (test_prompt_attention_is_launched_in_the_ordinary_way)
    "attn_prefill_tc_kernel": {"lp.pos.finished", "lp.pos.kv_len"},
}


def touched_before_the_wait(body):
    """(loaded, stored): the pointers through which global memory is reached in front of a kernel's chain_begin; a block's statements behind a
    chain_wait() of its own do not count. Shared memory, local arrays and pointers to either are left out, a pointer that is a local name for
    an offset into another counts as that one."""
    text = body[:body.index("chain_begin(")]
    while "chain_wait();" in text:
        at = i = text.index("chain_wait();")
        depth = 0
        while i < len(text) and depth >= 0:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        text = text[:at] + text[i - 1:]
    near = set(re.findall(r"__shared__[^;]*?(\w+)\[", text)) | {"smem_raw"}
    for decl in re.findall(r"__shared__([^;]*);", text):
        near |= set(re.findall(r"(\w+)\s*(?:\[|,|$)", decl))
    near |= set(re.findall(r"\b(?:float4?|uint4|int|uint32_t)\s+(\w+)\[", text)) | set(re.findall(r"\b(?:float|int)\s[^;=(]*?,\s*(\w+)\[", text))
    for decl in re.findall(r"\bfloat ((?:\w+\[[^;]*?)+);", text):
        near |= set(re.findall(r"(\w+)(?:\[\w+\])+", decl))
    names = {}
    for m in re.finditer(r"(?:\*|\bauto)\s*(?:const\s+)?(?:__restrict__\s+)?(\w+)\s*=\s*([^;]*);", text):
        sources = [x for x in re.findall(r"[A-Za-z_][\w.]*", m.group(2))]
        first = next((x for x in sources if x in near or x in names or "." in x), None)
        if first in near:
            near.add(m.group(1))
        elif first:
            names[m.group(1)] = names.get(first, first)
    loaded, stored = set(), set()
    access = [(m.group(1), m.end()) for m in re.finditer(r"\b([A-Za-z_]\w*(?:\.\w+)*)\s*\[", text)]
    access += [(m.group(1), m.end()) for m in re.finditer(r"(?<=[=(,&|?:!])\s*\*\s*([A-Za-z_]\w*(?:\.\w+)*)", text)]
    access += [(m.group(1), m.end()) for m in re.finditer(r"[;{}]\s*\*\s*([A-Za-z_]\w*(?:\.\w+)*)", text)]
    access += [(m.group(1), m.end()) for m in re.finditer(r"(?:ld_stream16|__ldg|ldf|ld4)\(\s*&?([A-Za-z_]\w*(?:\.\w+)*)", text)]
    for name, end in access:
        if name in near:
            continue
        depth = text[end - 1] == "["
        while depth:
            depth += {"[": 1, "]": -1}.get(text[end], 0)
            end += 1
        into = stored if re.match(r"\s*(?:\.\w+\s*)?(?:[-+*/|&^]?=(?!=)|\+\+|--)", text[end:]) else loaded
        into.add(names.get(name, name))
    calls = set(re.findall(r"\b(tma_\w+|cp_async\w*|st_\w+|stf|st4|atomic\w+|red_\w+|mbar_wait\w*)\(", text))
    calls |= {a for a in re.findall(r'asm volatile\("([^"]*)', text) if "global" in a or "bulk" in a}
    return loaded, stored | calls


def check_before_the_wait(kernel, body):
    loaded, stored = touched_before_the_wait(body)
    stored -= SHARED.get(kernel, set())
    assert not stored, f"{kernel} writes in front of its wait: {sorted(stored)}"
    allowed = PARAMETERS.get(kernel, set()) | EARLY_LOADS.get(kernel, set())
    assert loaded <= allowed, f"{kernel} reads in front of its wait: {sorted(loaded - allowed)}"


@pytest.mark.parametrize("name", FILES)
def test_chained_kernels_wait_and_name_what_was_written_before(name):
    src, found = kernels(name)
    chained = set(re.findall(r"chained\(\s*(\w+)", src))
    assert chained and chained <= {k for k, _, _ in found}
    for kernel, params, body in found:
        if kernel not in chained:
            continue
        begin = re.findall(r"chain_begin\(([^)]*)\);", body)
        assert len(begin) == 1, kernel
        if kernel not in EARLY_LOADS:
            assert body.lstrip().startswith("chain_begin("), kernel
        check_before_the_wait(kernel, body)
        restrict = set(re.findall(r"\*\s*__restrict__\s+(\w+)", params))
        named = set(filter(None, re.split(r"[,\s]+", begin[0])))
        rest = set((WEIGHTS.get(kernel, "") + " " + WRITTEN.get(kernel, "")).split())
        assert named | rest == restrict and not named & rest, f"{kernel}: {sorted(restrict - named - rest)} may be read non-coherently"


@pytest.mark.parametrize("name", FILES)
def test_explicit_non_coherent_loads_are_of_weights(name):
    src, _ = kernels(name)
    allowed = {"linear_any": ["W + (size_t)wrow(r) * ldw + k"], "attn_local": ["row + min(dist, len - 1)"]}   # weights; the distance table
    loads = [a for a in re.findall(r"(?:ld_stream16|__ldg)\(((?:[^()]|\([^()]*\))*)\)", src)]
    assert [a for a in loads if a not in allowed.get(name, [])] == []


def test_the_kernel_behind_a_copy_a_clear_a_fork_or_a_join_is_not_chained():
    """lcc_seq_forward copies and clears through helpers that break the chain; a fork's or a join's wait on another stream's event is followed
    by a break before anything is launched."""
    src = re.sub(r"//[^\n]*", "", (CSRC / "seq_model.cu").read_text())
    for helper in re.findall(r"\n(?:int|void) \w+\([^)]*cudaStream_t s\) \{[^{}]*cudaMem(?:cpy|set)Async[^{}]*\}", src):
        assert helper.index("Async") < helper.index("chain_break()")
    forward = src[src.index("int lcc_seq_forward("):]
    assert not re.search(r"cudaMem(?:cpy|set)\w*\(", forward)
    waits = [w for w in re.finditer(r"cudaStreamWaitEvent\((\S+), m->(ev_\w+), 0\)", forward)]
    assert len(waits) == 4
    for w in waits:
        rest = forward[w.end():]
        # the branch that forks from the main stream goes on there (same predecessor kernel); its first launch on the side stream follows a break
        stop = rest.index("chain_break()")
        between = rest[:stop]
        if w.group(2) == "ev_join" or "fork_ff" not in forward[max(0, w.start() - 120):w.start()]:
            assert "STEP(" not in between, w.group(0)
        else:
            assert not re.search(r"STEP\([^;]*\bfs\b", between), w.group(0)


def test_prompt_attention_is_launched_in_the_ordinary_way():
    """Its few large CTAs would be placed on the SMs that the kernel in front leaves free, two to an SM."""
    src, found = kernels("attn_local")
    for kernel in ("attn_chunk_sink_mma_kernel", "attn_chunk_sink_tiled_kernel"):
        assert not re.search(rf"chained\(\s*{kernel}", src)
        assert all("chain_begin" not in body for k, _, body in found if k == kernel)
    src, _ = kernels("attention_prefill_tc")      # the tcgen05 form with windows
    assert "attn_prefill_tc_kernel<true><<<" in src and "chained(attn_prefill_tc_kernel<true>" not in src
