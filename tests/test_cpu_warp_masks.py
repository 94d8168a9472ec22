"""Masks of warp shuffles are taken by a ballot that all lanes reach.  __activemask
names the lanes that happen to run together, which inside a branch may be some of
those that take it: a shuffle under such a mask can read a lane outside it, whose
value is undefined (a spin would walk with another's draws)."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dsim_gb300", "csrc")


def _code(path):
    text = open(path, encoding="utf-8").read()
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", text, flags=re.S)


def test_no_mask_of_the_lanes_that_happen_to_run():
    files = [f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh", ".h"))]
    assert files
    assert [f for f in files if "__activemask" in _code(os.path.join(CSRC, f))] == []
