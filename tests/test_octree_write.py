"""The octree file takes its path's place when it is whole
(tests/write_check.cpp): a build whose device work fails half way leaves what
was there, and paths that were written into still are."""
import os
import stat
import struct
import subprocess

import pytest

import vt_fixtures as F

OK, FETCH, OPEN, SHORT = range(4)
WANT = struct.pack("<ifi3ii", 919278872, 0.5, 8, 7, 5, 8, 3)
for _words in ((512, 513, 600, 601, 700, 700), (64, 65, 80, 80), (8, 9), (1, 1)):
    WANT += struct.pack("<i%dQ" % len(_words), len(_words), *_words)


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("write") / "write_check")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(F.ROOT, "visualtur_b200", "csrc"),
                    os.path.join(F.ROOT, "tests", "write_check.cpp"), "-o", exe], check=True)

    def run(path, fail=-1):
        out = subprocess.run([exe, str(path), str(fail)], capture_output=True, text=True, check=True).stdout.split()
        return int(out[0]), int(out[1])
    return run


@pytest.mark.parametrize("fail", [0, 4, 11])
def test_failed_ranges_leave_the_path(fail, check, tmp_path):
    old, new = tmp_path / "old.oct", tmp_path / "new.oct"
    old.write_bytes(b"an earlier octree")
    assert check(old, fail)[0] == FETCH and old.read_bytes() == b"an earlier octree"
    assert check(new, fail)[0] == FETCH and not new.exists()
    assert sorted(p.name for p in tmp_path.iterdir()) == ["old.oct"]


def test_file(check, tmp_path):
    new, old = tmp_path / "a.oct", tmp_path / "b.oct"
    assert check(new) == (OK, 12) and new.read_bytes() == WANT
    umask = os.umask(0)
    os.umask(umask)
    assert stat.S_IMODE(new.stat().st_mode) == 0o666 & ~umask
    old.write_bytes(b"x" * 1000)
    old.chmod(0o640)
    assert check(old) == (OK, 12) and old.read_bytes() == WANT and stat.S_IMODE(old.stat().st_mode) == 0o640
    assert sorted(p.name for p in tmp_path.iterdir()) == ["a.oct", "b.oct"]


def test_paths_that_are_written_into(check, tmp_path):
    """links, devices, and a directory that takes no new file"""
    real, sym, hard = tmp_path / "real.oct", tmp_path / "sym.oct", tmp_path / "hard.oct"
    real.write_bytes(b"")
    sym.symlink_to(real)
    assert check(sym) == (OK, 12) and sym.is_symlink() and real.read_bytes() == WANT
    real.write_bytes(b"")
    os.link(real, hard)
    assert check(hard) == (OK, 12) and real.read_bytes() == WANT and real.stat().st_nlink == 2
    assert check("/dev/null") == (OK, 12) and stat.S_ISCHR(os.stat("/dev/null").st_mode)
    long = tmp_path / ("n" * 250)                 # no room in the name for more
    long.write_bytes(b"")
    assert check(long) == (OK, 12) and long.read_bytes() == WANT


def test_paths_that_cannot_be_written(check, tmp_path):
    assert check(tmp_path / "no" / "a.oct")[0] == OPEN
    assert check(tmp_path)[0] == OPEN
    if os.path.exists("/dev/full"):
        assert check("/dev/full")[0] == SHORT
