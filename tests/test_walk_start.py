"""Points from which every ray's 64-ary walk ends at once (ties_at_start), on
random trees and rays on the host (tests/start_check.cpp)."""
import os
import subprocess

import vt_fixtures as F


def test_points_where_every_ray_ties(tmp_path):
    exe = str(tmp_path / "start_check")
    subprocess.run(["g++", "-std=c++17", "-O1", "-ffp-contract=off", "-I", "/usr/local/cuda/include", "-I",
                    os.path.join(F.ROOT, "visualtur_b200", "csrc"), os.path.join(F.ROOT, "tests", "start_check.cpp"),
                    "-o", exe], check=True)
    run = subprocess.run([exe], capture_output=True, text=True)
    assert run.returncode == 0, run.stdout
    rows = {r.split()[0]: [int(v) for v in r.split()[1:]] for r in run.stdout.split("\n") if r}
    points, rays, ties = rows["named"]
    assert points > 1000 and ties > 0.8 * rays      # the others leave the volume or its set cells at once
    points, rays, ties = rows["other"]
    assert points > 1000 and ties <= rays // 1000
