"""Rules of the tensor-core kernels that no GPU run can show without hanging one,
checked in their source: an MMA and every commit that waits for it are issued by
the same lane, and a bounded wait has one outcome for a warp that goes on to
warp-wide instructions.
"""
import os
import re
import sys

import numpy as np
import pytest

PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "geodynamo.jl_b200")
CSRC = os.path.join(PKG, "csrc")
sys.path.insert(0, PKG)
import workloads  # noqa: E402
FILES = ("gd_legendre_tc.cu", "gd_ozaki.cu")


def _code(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def _guards(code):
    """The innermost `if` condition in front of each MMA issue and commit inside a kernel."""
    out = []
    for k in re.finditer(r"\b(mma_commit|mma_i8|issue_chunk|issue_products)\(", code):
        if re.search(r"__forceinline__ void $", code[:k.start()]):
            continue  # the definition
        i, depth = k.start(), 0
        # outwards to the statement or block whose condition names a lane
        while i > 0:
            i -= 1
            if code[i] == "}":
                depth += 1
            elif code[i] == "{" or (code[i] == ")" and depth == 0):
                if code[i] == "{" and depth > 0:
                    depth -= 1
                    continue
                head = code[:i + 1] if code[i] == ")" else code[:i]
                m = re.search(r"if \((lane == 0|elect_one\(\))[^;{}]*\)?\s*$", head)
                if m:
                    out.append((k.group(1), m.group(1)))
                    break
    return out


@pytest.mark.parametrize("name", FILES)
def test_commits_come_from_the_lane_that_issues(name):
    guards = _guards(_code(name))
    issued = {g for op, g in guards if op != "mma_commit"}
    commits = [g for op, g in guards if op == "mma_commit"]
    assert len(issued) == 1 and len(commits) >= 3
    assert set(commits) == issued, guards


@pytest.mark.parametrize("name", FILES)
def test_waits_ahead_of_warp_wide_instructions_have_one_outcome(name):
    """Per-lane outcomes only where no warp-wide instruction follows: the loaders of
    the analysis, and the drain of its stages, which a block-wide vote follows."""
    per_lane = {"&empty[g]", "&empty[(gs + T - q) & 1]"}
    used = re.findall(r"(?:[!=] ?|&& |\? |: )mbar_wait\(([^,]+),", _code(name))
    assert set(used) <= per_lane, used
    assert len(re.findall(r"mbar_wait_warp\(", _code(name))) >= 4


@pytest.mark.gpu
@pytest.mark.parametrize("omit", [0, 3])
def test_failed_vector_synthesis_drains_and_recovers(gdb, omit):
    """The drain after an expired wait in the vector form, with MMAs issued before
    it (omit 3) and with none: the error is reported, the next call is right."""
    g = gdb.SHTnsKitConfig(130, 132, 288, 33, precision="mixed")
    re, im = workloads.transform_batch(130, 130, 33, 2, seed=3)
    coef = (re[0], im[0], re[1], im[1])
    want = g.synth_vector(*coef)
    g.set_fault_test(wait_cycles=1 << 24, omit_step=omit)
    with pytest.raises(gdb.GeoDynamoError) as e:
        g.synth_vector(*coef)
    assert e.value.status == 3 and "wait expired" in str(e.value)
    g.set_fault_test(0, -1)
    for x, y in zip(g.synth_vector(*coef), want):
        assert np.array_equal(x, y)
    g.close()
