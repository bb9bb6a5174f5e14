"""Barriers on which the other CTA of a pair arrives are signalled and awaited at cluster scope."""
import os
import re

import batchgen_b200

CSRC = os.path.join(os.path.dirname(batchgen_b200.__file__), "ops", "csrc")


def _source(name):
    return re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())


def test_arrivals_in_another_cta_are_at_cluster_scope():
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".cuh")):
            for ins in re.findall(r"mbarrier\.arrive[\w.:]*", _source(name)):
                if "shared::cluster" in ins:
                    assert re.search(r"\.(release|relaxed)\.cluster\.", ins), (name, ins)


def test_relaxed_arrivals_stand_behind_the_fence_of_the_reads_they_report():
    assert re.search(r"tc_fence_before\(\);\s*__syncwarp\(\);\s*if \(lane == 0\) pair::arrive_cluster\(", _source("gemm_bf16_pair.cu"))
    assert _source("gemm_bf16_pair.cu").count("arrive_cluster(") == 1


def test_waits_of_a_pair_acquire_at_cluster_scope():
    wait = re.search(r"bool wait_cluster\(.*?\n}", _source("pair.cuh"), re.S).group(0)
    attempt = re.search(r"(\w+)\(bar, parity\)\) return true", wait).group(1)
    assert "mbarrier.try_wait.parity.acquire.cluster" in re.search(r"bool %s\(.*?\n}" % attempt, _source("pair.cuh"), re.S).group(0)
    kernel = _source("gemm_bf16_pair.cu")
    assert re.search(r"pair::commit\(&ss\.empty", kernel) and re.search(r"leader_addr\(&ss\.tmem_empty", kernel)
    assert "pair::wait_cluster(&ss.tmem_empty" in kernel and not re.search(r"\bmbar_wait\(", kernel)
