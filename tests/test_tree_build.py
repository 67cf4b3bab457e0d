"""The 64-ary candidate tree of the trace kernel as made when a renderer is
opened (tests/tree_build_check.cpp)."""
import os
import subprocess

import vt_fixtures as F


def test_tree_build(tmp_path):
    """The same nodes as from a node's 64 cells one by one, in less than a
    fifth of the time (octants looked up cell by cell but in one pass of eight
    each: half; by whole octants and set cells only: a sixteenth)."""
    exe = str(tmp_path / "tree_build_check")
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", "/usr/local/cuda/include", "-I",
                    os.path.join(F.ROOT, "visualtur_b200", "csrc"), os.path.join(F.ROOT, "tests", "tree_build_check.cpp"),
                    "-o", exe], check=True)
    run = subprocess.run([exe], capture_output=True, text=True)
    assert run.returncode == 0, run.stdout
    trees, nodes, cells, built = (float(v) for v in run.stdout.split())
    assert trees > 400 and nodes > 30000
    assert built < 0.2 * cells
