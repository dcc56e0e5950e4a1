"""The affine bucket kernel (csrc/zg_bucket.cuh) on host threads.

tests/emu runs the kernel's own source as one CTA of 128 host threads, under
the address and undefined-behaviour sanitizers, and compares every row and
column sum with plain XYZZ additions of the same buckets: chunk and wide
items, merged units, buckets that run over several segments, repeated and
opposite points (doubling, cancellation), and empty items.
"""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def runner(tmp_path_factory):
    cxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else shutil.which("g++")
    exe = str(tmp_path_factory.mktemp("emu") / "bucket_accum")
    subprocess.run([cxx, "-std=c++20", "-O1", "-fsanitize=address,undefined", "-fno-sanitize=alignment", "-Wno-unknown-pragmas",
                    "-o", exe, os.path.join(HERE, "emu", "bucket_accum.cpp"), "-lpthread"], check=True)
    return exe


@pytest.mark.parametrize("kind,group", [("chunk", 1), ("chunk", 3), ("small", 2), ("small", 3), ("wide", 1),
                                        ("wide", 4), ("merged", 2), ("skewed", 1), ("skewed", 4), ("empty", 2)])
def test_bucket_sums(runner, kind, group):
    r = subprocess.run([runner, kind, str(group), "11"], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
