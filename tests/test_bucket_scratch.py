"""Bounds of the bucket kernel's scratch (csrc/zg_bucket.cuh, FbScratch).

The kernel's source on host threads, with a scratch of exactly the asked size
and poisoned gaps between its blocks: buckets of odd counts in both sort units
(one slot more each than half their entries), one segment and several, whose
ends cut buckets, and each batch size.
"""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def runner(tmp_path_factory):
    cxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else shutil.which("g++")
    exe = str(tmp_path_factory.mktemp("emu") / "bucket_scratch")
    subprocess.run([cxx, "-std=c++20", "-O1", "-fsanitize=address,undefined", "-fno-sanitize=alignment", "-Wno-unknown-pragmas",
                    "-o", exe, os.path.join(HERE, "emu", "bucket_scratch.cpp"), "-lpthread"], check=True)
    return exe


@pytest.mark.parametrize("e0,e1,cap,group,task", [
    (1, 1, 0, 1, 64), (1, 1, 0, 2, 32), (3, 1, 0, 1, 96), (1, 0, 0, 2, 64), (0, 0, 64, 1, 64),
    (5, 7, 0, 2, 96), (5, 7, 1777, 1, 32), (3, 3, 1024, 2, 64), (1, 1, 333, 1, 64), (9, 0, 4001, 2, 48),
])
def test_scratch_bounds(runner, e0, e1, cap, group, task):
    r = subprocess.run([runner, str(e0), str(e1), str(cap), str(group), str(task)], capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
