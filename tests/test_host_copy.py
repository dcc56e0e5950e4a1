"""Host threads of a call (csrc/zg_host.hpp): small copies stay on the caller's
thread (starting threads cost a 128 x 1024 recovery more than the copy), large
ones share a few, every byte arrives once, and a throwing call is reported."""
import os
import shutil
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def test_copies_and_threads(tmp_path):
    cxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else shutil.which("g++")
    exe = str(tmp_path / "host_copy")
    subprocess.run([cxx, "-std=c++17", "-O1", "-fsanitize=address,undefined", "-o", exe,
                    os.path.join(HERE, "emu", "host_copy.cpp"), "-lpthread"], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
