"""The small batches' kernels overlap their predecessors (programmatic dependent launch): before
pdl_wait() they may touch only what no kernel writes.  Nothing of that shows in results, since a
stale line is a matter of timing, so the source is checked."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "denise-black-edition_b200", "csrc")


def _written():
    """The members of Inst that kernels may write: its pointers to non-constant data."""
    text = open(os.path.join(CSRC, "dn_kernels.cuh")).read()
    text = re.sub(r"//[^\n]*", "", text[text.index("struct Inst {"):])
    text = text[:text.index("\n};")]
    names = [n for d in text.split(";") if "*" in d and "const " not in d for n in re.findall(r"\*\s*(\w+)", d)]
    assert {"vx", "syy", "psi_vxxs", "sec", "flag", "snap_scale"} <= set(names)
    return r"I\.(?:" + "|".join(names) + r")\b"


def _kernels():
    text = open(os.path.join(CSRC, "dn_kernels_small.cuh")).read()
    text = re.sub(r"//[^\n]*", "", text)
    return {m.group(1): m.group(0) for m in
            re.finditer(r"__global__ void [^(]*\(\d+, \d+\) (k_\w+)\(.*?\n}\n", text, flags=re.S)}


@pytest.mark.parametrize("name", ["k_update_v2_small", "k_update_s_el2_small"])
def test_nothing_written_is_touched_before_the_wait(name):
    body = _kernels()[name]
    waits = [m.start() for m in re.finditer(r"pdl_wait\(\)", body)]
    assert len(waits) == 2   # a block without work, and the first row of the others
    before = body[:waits[0]] + body[body.index("}", waits[0]):waits[1]]
    touched = re.findall(_written(), before)
    assert not touched, touched
    # every way out of the kernel passes a wait
    assert "return" not in body[:waits[0]] and "return" not in body[body.index("}", waits[0]):waits[1]]
