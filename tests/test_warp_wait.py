"""Bounded waits of a warp end the same way in all its lanes
(difx_b200/csrc/gx_warp_wait.h, used by the X-steps' stage rings): the header is
compiled for the host, where 32 threads stand for the lanes.  Lanes that decide
alone part at the barriers as soon as one lane's wait runs out; voting lanes never do."""
import os
import re
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(not os.path.exists("/usr/bin/g++"), reason="no C++ compiler")
def test_lanes_leave_together(tmp_path):
    exe = str(tmp_path / "model")
    subprocess.run(["/usr/bin/g++", "-O1", "-std=c++17", os.path.join(ROOT, "tests", "host", "warp_wait_model.cpp"), "-o", exe,
                    "-lpthread"], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, check=True, timeout=120).stdout
    patterns, voting, alone = map(int, out.split())
    assert patterns == 6 and voting == 0
    assert alone == patterns   # what the vote is there for


@pytest.mark.parametrize("source,kernel", [("gx_xstep.cu", "xmac_fp32_kernel"), ("gx_tcxmac.cu", "xmac_tc_kernel")])
def test_stages_end_by_vote(source, kernel):
    """In the kernels whose warps wait per lane, no bare full-mask barrier ends a stage."""
    src = open(os.path.join(ROOT, "difx_b200", "csrc", source)).read()
    body = src[src.index(kernel + "("):]
    body = re.sub(r"//[^\n]*", "", body[:body.index("\n}\n")])
    assert "mbar_wait(" in body and "stage_end(" in body
    assert "__syncwarp" not in body
