"""Chained launches of the vision tower and the prefill, read from the sources: which data a kernel may read non-coherently, what it touches before it waits
(nothing that another kernel of the pass writes or still reads), and that tensor memory is taken before the next kernel is let in."""
import re

import pytest

from test_chain_cpu import CSRC, check_before_the_wait, kernels

FILES = ["gemm_tcgen05", "elementwise", "attention", "attention_tc", "attention_prefill_tc"]
# `__restrict__` parameters that nothing of the pass writes while the kernel is on the SMs (weights, tables), and those that are only written
WEIGHTS = {"norm_rows_kernel": "w b", "norm_rows_warp_kernel": "w b", "vit_rope_table_kernel": "inv_freq", "embed_gather_kernel": "table",
           "mrope_kv_write_kernel": "inv_freq", "splitk_reduce_kernel": "bias", "gemm_bf16_tn_kernel": "bias", "gemm2_bf16_tn_kernel": "bias",
           "gemm_swap_kernel": "bias"}
WRITTEN = {"norm_rows_kernel": "y", "norm_rows_warp_kernel": "y", "vit_rope_table_kernel": "cos_t sin_t", "embed_gather_kernel": "out",
           "video_rank_kernel": "rank", "mrope_kv_write_kernel": "kc vc", "flash_merge_kernel": "out"}


@pytest.mark.parametrize("name", FILES)
def test_chained_kernels_wait_and_name_what_was_written_before(name):
    src, found = kernels(name)
    chained = set(re.findall(r"chained\(\s*(\w+)", src)) - {"kern"}
    if "chained(kern" in src or "chain_next()" in src:      # launched through a local name: every kernel of the file that waits
        chained |= {k for k, _, b in found if "chain_begin(" in b}
    assert chained and chained <= {k for k, _, _ in found}
    for kernel, params, body in found:
        begin = re.findall(r"chain_begin\(([^)]*)\);", body)
        if kernel not in chained:
            assert not begin, kernel
            continue
        assert len(begin) == 1, kernel
        at = body.index("chain_begin(")
        restrict = set(re.findall(r"\*\s*__restrict__\s+(\w+)", params))
        named = set(filter(None, re.split(r"[,\s]+", begin[0])))
        if kernel == "gemm_bf16_tn_kernel":                  # the row lists' tiles: a local copy of the parameter is what is read
            assert "const int* tile_group = tile_groups;" in body[:at] and body.count("tile_groups") == 1
            restrict = restrict - {"tile_groups"} | {"tile_group"}
        rest = set((WEIGHTS.get(kernel, "") + " " + WRITTEN.get(kernel, "")).split())
        assert named | rest == restrict, f"{kernel}: {sorted(restrict - named - rest)}"
        if "tmem_alloc" in body:
            alloc = body.index("tmem_alloc")
            assert alloc < at and re.search(r"__syncthreads\(\)|cluster_sync_all\(\)", body[alloc:at]), kernel
            assert "residual" not in body[:at], kernel
        else:
            assert body.lstrip().startswith("chain_begin("), kernel
        check_before_the_wait(kernel, body)


def test_scopes_end_with_the_pass():
    """A scope is a local of the two passes; copies and clears inside one would have to break the chain."""
    src = re.sub(r"//[^\n]*", "", (CSRC / "model.cu").read_text())
    for fn in ("static int vit_forward_impl(", "static int prefill_impl("):
        at = src.index(fn)
        body = src[at:src.index("\n}", at)]
        assert body.count("ChainScope chain;") == 1 and not re.search(r"cudaMem(?:cpy|set)", body[body.index("ChainScope"):])
    assert src.count("ChainScope") == 2
