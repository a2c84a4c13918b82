"""Waits on a tile copy that end a warp's work must end it for the whole warp.

A warp of the octet kernels goes on to full-mask votes and shuffles after a
wait, so its lanes have to leave together when one of them runs out of polls.
That cannot be made to happen on a GPU without breaking a kernel; this reads
the source: the octet kernels branch only on the form that votes
(mbar_wait_warp, whose agreement yk_wait_selftest checks on the GPU).
"""
import os
import re

CSRC = os.path.join(os.path.dirname(__file__), "..", "yukawamd_b200", "csrc")


def test_octet_waits_agree_in_the_warp():
    text = open(os.path.join(CSRC, "yk_octets.cuh")).read()
    branches = re.findall(r"if \(!(mbar_wait_\w+)\(", text)
    assert len(branches) == 2 and set(branches) == {"mbar_wait_warp"}
    common = open(os.path.join(CSRC, "yk_common.cuh")).read()
    body = common[common.index("bool mbar_wait_warp("):]
    assert "__all_sync(0xffffffffu, mbar_wait_bounded(" in body[:body.index("\n}")]
