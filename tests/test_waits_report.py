"""Every kernel whose device-side waits may give up says so in the status words that blr_workspace_status and blr_blast_static_status read.  (Read from the
sources: making a wait of each kernel run out would take a switch in the kernels that leaves a copy out.)"""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mem_efficient_blr_b200", "csrc")
WAITS = re.compile(r"\b(mbar_wait\w*|wait_counter)\(")
REPORTS = re.compile(r"atomicExch\(p\.(status|counters \+ 3), 1u\)")


def _kernels():
    """(file, name, body) of every __global__ function: up to the closing brace in the first column."""
    for f in sorted(os.listdir(CSRC)):
        if f.endswith(".cu"):
            text = open(os.path.join(CSRC, f)).read()
            for m in re.finditer(r"__global__[^;{]*?\b(\w+_kernel)\(", text):
                yield f, m.group(1), text[m.start():text.index("\n}", m.start())]


WAITING = [k for k in _kernels() if WAITS.search(k[2])]


def test_the_waiting_kernels_are_found():
    assert {f for f, _, _ in WAITING} >= {"stream_kernel.cu", "blast_cluster.cu", "blast_split.cu", "skinny.cu", "umma_gemm.cu", "umma_pair.cu", "umma_wq.cu",
                                          "couple.cu"}


@pytest.mark.parametrize("f,name,body", WAITING, ids=[k[1] for k in WAITING])
def test_a_kernel_that_gave_up_reports(f, name, body):
    assert REPORTS.search(body)


def test_the_pipelines_hand_the_status_word_on():
    text = open(os.path.join(CSRC, "pipeline.cu")).read()
    assert "p.status = status;" in text
    without = [c for c in re.findall(r"run_gemm\((?:[^()]|\([^()]*\))*\)", text) if "stream, nullptr" in c]
    assert len(without) == 1 and "W, w_layout, 1, O, I, x" in without[0]  # (a dense call has no workspace)
    api = open(os.path.join(CSRC, "c_api.cu")).read()
    for call in ("pipeline_blast_small(x", "pipeline_blast(static", "pipeline_monarch(static", "pipeline_low_rank(static"):
        assert "w.counters + 255" in api[api.index(call):api.index(";", api.index(call))]
