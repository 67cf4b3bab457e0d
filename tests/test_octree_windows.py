"""Range arrays of more words than the builder makes at a time: the blocks a
window is made from, on the host (tests/window_check.cpp), and the file of a
volume of noise against the reference's algorithm on the CPU."""
import filecmp
import os
import subprocess

import numpy as np
import pytest

import vt_fixtures as F


def test_blocks_of_a_window(tmp_path):
    exe = str(tmp_path / "window_check")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(F.ROOT, "visualtur_b200", "csrc"),
                    os.path.join(F.ROOT, "tests", "window_check.cpp"), "-o", exe], check=True)
    run = subprocess.run([exe], capture_output=True, text=True)
    assert run.returncode == 0, run.stdout
    levels, windows, _ = (int(v) for v in run.stdout.split())
    assert levels == 4000 and windows > 10 * levels


@pytest.mark.gpu
@pytest.mark.parametrize("shape, p", [((256, 256, 256), 0.05), ((128, 256, 200), 0.2), ((256, 256, 256), 0.002)])
def test_noise_of_many_windows(shape, p, workdir, cuda):
    import visualtur_b200 as vt
    from oracle import oracle as orc
    vol = (np.random.default_rng(6).random(shape) < p).astype(np.uint8) * 255
    a, b = workdir + "/noise.oct", workdir + "/noise_cpu.oct"
    vt.build_octree(vt.FileManager.wrap(vol), 128.0, a)
    orc.build_octree(vol, 128.0, b)
    assert os.path.getsize(a) > 1 << 18
    assert filecmp.cmp(a, b, shallow=False)
