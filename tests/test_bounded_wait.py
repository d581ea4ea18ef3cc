"""Bounded waits of the roles of a kernel's block (amca3d_gb300/csrc/bounded_wait.h): where a wait runs out or is aborted
while some lanes of a warp already find their barrier complete, the warp's lanes all get one verdict."""
import os
import re
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_lanes_that_wait_together_get_one_verdict(tmp_path):
    exe = str(tmp_path / "bounded_wait")
    subprocess.run(["g++", "-std=c++17", "-O2", "-pthread", os.path.join(HERE, "bounded_wait.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True, timeout=120).stdout
    rows = [line.split() for line in out.splitlines()]
    assert [r[0] for r in rows] == ["done", "abort_before_some", "runs_out_for_some", "runs_out_for_all"]
    assert all(int(split) == 0 and int(wrong) == 0 for _, _, split, wrong in rows), rows


def test_the_warps_that_share_instructions_wait_together():
    """In the inference kernel only the weight and MMA roles, one thread each, may wait lane by lane."""
    src = open(os.path.join(HERE, "..", "amca3d_gb300", "csrc", "surrogate.cu")).read()
    body = src[src.index("mlp_infer_kernel(const"):]
    body = body[:body.index("\n}\n")]
    single, warps = body.split("// ---- features, epilogues, results ----")
    assert re.search(r"\bwait\(", single) and not re.search(r"\bwait\(", warps)
    assert len(re.findall(r"\bwait_warp\(", warps)) >= 5
