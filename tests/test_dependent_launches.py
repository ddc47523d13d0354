"""Kernels that may start before their predecessor has ended, checked in the source.

With programmatic stream serialization only griddepcontrol.wait (pdl_wait) makes the
predecessor's writes visible, whatever else shows that they have been made.  So every
function that waits does so unconditionally and before it reads the done flag, the state
records or anything derived from them; a kernel that triggers its successor early waits
too.  No run can fail for a wait that is missing here (a stale line is excluded by
practice, not by the model), so the rule is held in the text.
"""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tensum_b200", "csrc")
# reads of what a step changes
STATE = re.compile(r"\*\s*done\b|\bs\.|\bsc->|\b(?:load_prim|load_ent|load_grad_vertex|ld4|bflux_one|viscous_one|stage)\s*[<(]")


def _block(text, at):
    """The text from the brace at or after `at` to its partner."""
    a = text.index("{", at)
    depth = 0
    for i in range(a, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return text[a:i + 1]
    raise AssertionError("unbalanced braces")


def _functions():
    out = []
    for f in ("tg_kernels.cuh", "tg_tiles.cuh"):
        with open(os.path.join(CSRC, f)) as fh:
            text = re.sub(r"//[^\n]*", "", fh.read())
        text = re.sub(r"__launch_bounds__\((?:[^()]|\([^()]*\))*\)", "", text)
        for m in re.finditer(r"__(?:global|device)__[^;{}]*?\b(\w+)\s*\(([^;{}]*)\)\s*\{", text):
            if m.group(1) not in ("pdl_wait", "pdl_trigger"):
                out.append((m.group(1), m.group(2), _block(text, m.end() - 1)))
    return out


def _without_lambdas(body):
    while True:
        m = re.search(r"auto\s+\w+\s*=\s*\[&\]\s*\([^)]*\)\s*\{", body)
        if not m:
            return body
        b = _block(body, m.end() - 1)
        at = body.index(b, m.end() - 1)
        body = body[:m.start()] + body[at + len(b):]


DEPENDENT = [(n, a, _without_lambdas(b)) for n, a, b in _functions() if "pdl_wait" in b or "pdl_trigger" in b]


def test_the_step_kernels_are_found():
    names = {n for n, _, _ in DEPENDENT}
    assert {"tile_grad", "k_tile_flux", "k_stage_head", "k_bflux", "k_dt", "k_dt_final", "k_step_begin", "k_strong_bc"} <= names


@pytest.mark.parametrize("name,args,body", DEPENDENT, ids=[n for n, _, _ in DEPENDENT])
def test_waits_before_it_reads_the_state(name, args, body):
    m = re.search(r"(?:^|[;{}])\s*pdl_wait\(\);", body)
    assert m, f"{name} has no unconditional pdl_wait()"
    early = STATE.search(body[:m.end()])
    assert not early, f"{name} reads {early.group(0)!r} before pdl_wait()"


@pytest.mark.parametrize("name,args,body", DEPENDENT, ids=[n for n, _, _ in DEPENDENT])
def test_promises_no_read_only_memory(name, args, body):
    """It may be resident while its predecessor writes: __restrict__ and __ldg let a load move
    ahead of the wait (the tile records, which no kernel writes, are read by load_rec)."""
    assert "__restrict__" not in args
    assert "__ldg" not in body
