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
    assert 0 <= kernel.find("cluster_started_arrive()") < kernel.find("ld_stream") < kernel.find("publish(")
    assert 0 <= publish.find("cluster_started_wait()") < publish.find("map_shared_rank")
    assert "return" not in kernel[: kernel.find("cluster_started_arrive()")] and publish.find("return") > publish.find("cluster_started_wait()")
