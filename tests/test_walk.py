"""The 64-ary walk of the trace kernel against the reference's depth-first
search on random trees and rays (outside, inside, on node planes, along
axes and diagonals), on the host: same candidates, same order, same
parameters; a ray the walk hands back has only taken candidates of the
search's prefix."""
import os
import subprocess

import vt_fixtures as F


def test_walk_yields_the_depth_first_candidates(tmp_path):
    exe = str(tmp_path / "walk_check")
    subprocess.run(["g++", "-std=c++17", "-O1", "-ffp-contract=off", "-I", "/usr/local/cuda/include", "-I",
                    os.path.join(F.ROOT, "visualtur_b200", "csrc"), os.path.join(F.ROOT, "tests", "walk_check.cpp"),
                    "-o", exe], check=True)
    run = subprocess.run([exe], capture_output=True, text=True)
    assert run.returncode == 0, run.stdout
    rows = {r.split()[0]: [int(v) for v in r.split()[1:]] for r in run.stdout.split("\n") if r}
    assert len(rows) == 8
    for name in ("outside", "inside", "far"):
        rays, cands, ties = rows[name]
        assert cands > rays and ties < rays // 1000      # general rays are walked, not handed back
    assert rows["axis"][2] == rows["axis"][0]            # non-finite products go to the literal search
