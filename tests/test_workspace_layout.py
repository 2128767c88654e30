"""Layout of the plan's device header that the one-tile-per-CTA kernels rest on,
checked by a host compiler.

A CTA must have read the launch number and the count of launches that used the
group sums before it publishes anything: the last tile advances both as soon as
it has seen every other tile. The kernels read them by one 16-byte load, on
which every publication depends.
"""
import os
import subprocess

from gpuprefixsums_gb300 import build as B

CHECK = """
#include <cstddef>
#include "gps_internal.h"
using gps::WsHeader;
static_assert(offsetof(WsHeader, mid_launch) % 16 == 0, "one aligned 16-byte word");
static_assert(offsetof(WsHeader, sums_launch) == offsetof(WsHeader, mid_launch) + 8, "its second half");
static_assert(alignof(WsHeader) % 16 == 0, "in every header");
"""


def test_launch_number_and_set_count_are_one_16_byte_word(tmp_path):
    src = tmp_path / "layout.cpp"
    src.write_text(CHECK)
    res = subprocess.run(["g++", "-std=c++17", "-fsyntax-only", "-I", B.CSRC_DIR, "-I", B.INCLUDE_DIR,
                          "-I", os.path.join(B.cuda_home(), "include"), str(src)], capture_output=True, text=True)
    assert res.returncode == 0, res.stderr[-2000:]
