"""The ensemble's gather + update reads what it overwrites by ordinary loads, checked in the source.

Its last stage forms U_old (src/fv.cc:1626-1630) from the step's starting state Q[0] and
writes the new state into Q[0].  ld2 and ldh go through __ldg, which is defined only for
memory that the whole kernel leaves alone, so they must not read Q[0] there.  That a load
moved past a store is up to the compiler, and no run shows that it may.
"""
import os
import re

PATH = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tensum_b200", "csrc", "tg_batch.cuh")


def test_u_old_is_read_by_ordinary_loads():
    with open(PATH) as fh:
        text = re.sub(r"//[^\n]*", "", fh.read())
    body = text[re.search(r"\)\s*kb_gather_update\(", text).start():text.index("__global__ void kb_step_end")]
    names = re.findall(r"(\w+)\s*=\s*L\.Q\[0\]", body)
    assert names                                           # U_old is formed from Q[0]
    for n in names:
        loads = re.findall(r"(\w+)(?:<H>)?\(" + n + r"\b", body)
        assert loads and set(loads) == {"ldh_rw"}, (n, loads)
    rw = re.search(r"void ldh_rw\(.*?\n}", text, re.S).group(0)
    assert "__ldg" not in rw and "ld2(" not in rw
