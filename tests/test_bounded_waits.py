"""The persistent GEMM's waits end: read from the source, as a wait that runs out cannot be timed to fall between two warps."""
from __future__ import annotations

import os
import re

import renee_b200

CSRC = os.path.join(os.path.dirname(renee_b200.__file__), "ops", "csrc")
BARRIER = r"\bmeet_rows\(|\bbar\.|barrier\.(cta|cluster|sync)|__syncthreads|cluster_sync_all"


def _source(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def test_a_staging_warp_whose_wait_ran_out_still_comes_to_every_meeting():
    """The logits' staging warps of 32 rows meet at barriers without a time limit.  A warp whose bounded wait has run out, while its
    neighbours' ended just in time, must come to all of them: under the same condition, as often per tile, and in every later tile."""
    src = _source("gemm.cu")
    at = src.index("if (!__all_sync(0xffffffffu, ok))")
    tmem = src.index("tc::tc_fence_after();", at)
    expired, staged = src[at:tmem], src[src.index("if (STAGED && staging) {", tmem): src.index("if (EPI == E_TOPK) {", tmem)]
    assert "tma_store_2d" in staged                                # the slice is the staged epilogue
    meetings = len(re.findall(r"\bmeet_rows\(", staged))
    assert meetings == len(re.findall(BARRIER, staged)) == 2
    assert "if (pos_end > pos_more) {" in staged and "if (EPI == E_SIGMOID_POS && p.pos_labels != nullptr) {" in staged
    assert not re.search(r"\b(break|continue|return|goto)\b[^;]*;", staged)
    expired = expired[: expired.index("} else {")]
    assert re.findall(r"if \(([^{;]*)\) break;", expired) == ["EPI != E_SIGMOID_POS"] and expired.count("break;") == 1
    assert "if (staging && p.pos_labels != nullptr && pos_end > pos_more) {" in expired
    assert len(re.findall(r"\bmeet_rows\(", expired)) == meetings and "aborted = true;" in expired and "continue;" in expired


def test_every_mbarrier_wait_has_the_time_limit():
    """``mbar_try_wait`` is called by the bounded wait alone."""
    for name in sorted(os.listdir(CSRC)):
        src = _source(name)
        calls = len(re.findall(r"\bmbar_try_wait\(", src))
        assert calls == (3 if name == "tc.cuh" else 0), name       # its definition and the two places in mbar_wait
        assert "mbarrier.test_wait" not in src
