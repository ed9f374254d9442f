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
def test_whole_warps_wait_by_vote(source, kernel):
    """A wait before the kernel's full-mask warp barriers is the voting one."""
    src = open(os.path.join(ROOT, "difx_b200", "csrc", source)).read()
    body = src[src.index(kernel + "("):]
    body = re.sub(r"//[^\n]*", "", body[:body.index("\n}\n")])
    waits = [m.start() for m in re.finditer(r"mbar_wait\(", body)]
    for b in (m.start() for m in re.finditer(r"__syncwarp\(\)", body)):
        loop = body.rindex("for (", 0, body.rindex("mbar_wait", 0, b))
        assert not [w for w in waits if loop < w < b], "a lane-by-lane wait before a warp barrier"
