"""The compile-time plans of the passes without functors (QSM_FIXED_PLANS_MORE_0..3 in
csrc/fft_engine.cuh) must equal the host planner's output for each length, as
test_fixed_plans.py checks for the other two lists, and no length may be in two lists."""
import os
import re
import shutil
import subprocess

import pytest

from test_fixed_plans import CSRC, HARNESS, listed_plans


def more_plans():
    src = open(os.path.join(CSRC, "fft_engine.cuh")).read()
    out = []
    for g in range(4):
        m = re.search(r"#define QSM_FIXED_PLANS_MORE_%d\(X\)(.*?)(?:\n\n|\n//|\n#)" % g, src, re.S)
        assert m, g
        out += [tuple(int(v) for v in e)
                for e in re.findall(r"X\((\d+),\s*(\d+),\s*(\d+),\s*(\d+),\s*(\d+)\)", m.group(1).replace("\\\n", " "))]
    return out


def test_lists_share_no_length():
    more = [e[0] for e in more_plans()]
    other = [e[0] for lst in listed_plans().values() for e in lst]
    assert len(set(more)) == len(more) and not set(more) & set(other)


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host C++ compiler")
def test_plans_match_the_planner(tmp_path):
    harness = tmp_path / "plan_harness.cpp"
    harness.write_text(HARNESS)
    exe = tmp_path / "plan_harness"
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", CSRC, str(harness), os.path.join(CSRC, "fft_plan.cpp"),
                    "-o", str(exe)], check=True)
    plans = more_plans()
    lines = subprocess.run([str(exe)] + [str(p[0]) for p in plans], check=True, capture_output=True,
                           text=True).stdout.splitlines()
    for (n, t, *radices), line in zip(plans, lines):
        got = [int(v) for v in line.split()]
        assert got == [n, t] + [r for r in radices if r > 1], (line, n, t, radices)
