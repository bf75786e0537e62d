"""Rules of the CUDA sources that a run on a GPU cannot show broken: what a kernel may touch before others have started or ended."""

import os
import re

from conftest import ROOT

CSRC = os.path.join(ROOT, "backendbench_b200", "csrc")


def _source(name):
    text = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*", "", text)


def _body(text, name):
    """The body of the function `name`, braces and all."""
    at = re.search(r"\b" + name + r"\([^;{]*\{", text)
    depth, i = 1, at.end()
    while depth:
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        i += 1
    return text[at.end() - 1 : i]


def test_a_comparison_writes_its_neighbours_memory_only_when_that_runs():
    text = _source("evalk.cu")
    kernel, publish = _body(text, "allclose_kernel"), _body(text, "publish")
    assert 0 <= kernel.find("cluster_started_arrive()") < kernel.find("ld_stream") < kernel.find("publish<")
    assert 0 <= publish.find("cluster_started_wait()") < publish.find("map_shared_rank")
    assert "return" not in kernel[: kernel.find("cluster_started_arrive()")] and publish.find("return") > publish.find("cluster_started_wait()")


def _kernels(text):
    """name -> (parameters, body) of every __global__ function"""
    found = {}
    for m in re.finditer(r"__global__[^;{]*?\b(\w+)\(([^;{]*)\)\s*\{", re.sub(r"__launch_bounds__\((?:[^()]|\([^()]*\))*\)", "", text)):
        found[m.group(1)] = (m.group(2), _body(text, m.group(1)))
    return found


# Operands of a call whose first kernel is launched the ordinary way, behind everything earlier: none of its kernels writes them.
READ_ONLY_ALL_ALONG = {"index", "src", "self", "idx", "grad"}


def test_what_the_grid_before_may_still_write_is_not_read_as_if_it_were_constant():
    early = {}
    for name in sorted(os.listdir(CSRC)):
        if name.endswith(".cu"):
            text = _source(name)
            kernels = _kernels(text)
            for launched in re.findall(r"launch_after\((\w+)\b", text):
                assert launched not in kernels or "after_grids_before()" in kernels[launched][1], launched
            early.update({k: v for k, v in kernels.items() if "after_grids_before()" in v[1]})
    assert {"ew_unary_vec", "gemm_few_rows", "gemm_tcgen05_kernel", "splitk_reduce", "layernorm_bwd_finalize", "binned_sort", "binned_replay", "emb_sort", "emb_replay", "chain_assign"} <= set(early)
    for name, (parameters, body) in early.items():
        constant = set(re.findall(r"const\s+[\w:]+(?:\s+[\w:]+)*\s*\*\s*__restrict__\s+(\w+)", parameters))
        assert constant <= READ_ONLY_ALL_ALONG, (name, constant)
        after = body[body.find("after_grids_before()") :]
        assert set(re.findall(r"\b(?:__ldg|__ldcs|ld_keep|ld_stream)\(\W*(\w+)", after)) <= READ_ONLY_ALL_ALONG, name
        assert ("_after(" in after or "_after_f(" in after) == ("waited(" in after), name


def test_bins_without_a_control_block_do_not_look_into_one():
    kernels = _kernels(_source("scatter_add.cu"))
    for name in ("binned_sort", "binned_replay"):
        body = kernels[name][1]
        assert body.count("ctl[") == body.count("ctl && ctl[") == 1, name
    for name in ("chain_link", "chain_replay", "chain_count", "chain_assign", "chain_fill"):
        assert "ctl &&" not in kernels[name][1], name
