"""The builder's child search by rank against its search over ranges, on
random levels on the host (tests/search_check.cpp)."""
import os
import subprocess

import vt_fixtures as F


def test_search_by_rank_equals_search_over_ranges(tmp_path):
    exe = str(tmp_path / "search_check")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", "/usr/local/cuda/include", "-I",
                    os.path.join(F.ROOT, "visualtur_b200", "csrc"), os.path.join(F.ROOT, "tests", "search_check.cpp"),
                    "-o", exe], check=True)
    run = subprocess.run([exe], capture_output=True, text=True)
    assert run.returncode == 0, run.stdout
    assert int(run.stdout.split()[0]) > 100000
