"""Long runs of one bucket in the affine bucket kernel (csrc/zg_bucket.cuh).

A level's additions of one bucket are listed by the bucket's owner or, from
FB_RUN_PAIRS on, by the whole CTA (up to FB_RUNS_MAX runs a turn). The
kernel's source runs on host threads (tests/emu) under the address and
undefined-behaviour sanitizers: runs one shorter, equal and one longer than
the line, more runs than the CTA takes, and one bucket with every entry.
"""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def runner(tmp_path_factory):
    cxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else shutil.which("g++")
    exe = str(tmp_path_factory.mktemp("emu") / "bucket_ranges")
    subprocess.run([cxx, "-std=c++20", "-O1", "-fsanitize=address,undefined", "-fno-sanitize=alignment", "-Wno-unknown-pragmas",
                    "-o", exe, os.path.join(HERE, "emu", "bucket_ranges.cpp"), "-lpthread"], check=True)
    return exe


@pytest.mark.parametrize("form,group", [("edge", 1), ("edge", 3), ("one", 1), ("one", 2), ("many", 1), ("many", 3),
                                        ("few", 2)])
def test_long_runs(runner, form, group):
    r = subprocess.run([runner, form, str(group), "7"], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
