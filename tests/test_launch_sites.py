"""Every kernel a step can contain goes through launch_dep / launch_plain / launch_cluster, which add it to a recorded step."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tinyflow_b200", "csrc")
# never part of a recorded step: the data-parallel exchange (not recorded), the bounded-wait probe
ELSEWHERE = {"dp_nccl.cu", "gemm_tcgen05.cu:barrier_timeout_probe_kernel"}


def test_no_launch_bypasses_a_recording():
    found = []
    for name in sorted(os.listdir(CSRC)):
        text = open(os.path.join(CSRC, name)).read()
        code = re.sub(r"//[^\n]*", "", text)
        for m in re.finditer(r"(\w+)(?:<[^<>;]*>)?<<<", code):
            if name not in ELSEWHERE and "%s:%s" % (name, m.group(1)) not in ELSEWHERE:
                found.append((name, m.group(1)))
        if name != "common.h" and re.search(r"cudaLaunchKernel|cudaLaunchCooperative", code):
            found.append((name, "cudaLaunch..."))
    assert not found
