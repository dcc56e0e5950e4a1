"""The factor tables that zg_ntt keeps: bounded per device, with the same
results where there is no room for them, and built without harm to a stream
capture. Each test has a process of its own (the tables last as long as it)."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))

COMMON = """
import sys
sys.path[:0] = [{root!r}, {here!r}]
import numpy as np, torch, __graft_entry__, zgo
pkg = __graft_entry__.load_package()
lib, oracle = pkg.lib(), zgo.Oracle()
def data(seed, n):
    x = np.random.default_rng(seed).integers(0, 256, (n, 32), dtype=np.uint8)
    x[:, 31] &= 0x1f
    return x.tobytes()
def dev(b):
    return torch.from_numpy(np.frombuffer(b, np.uint8).copy()).cuda()
def ntt(t, log_n, inverse=0, coset=0, stream=None):
    rc = lib.zg_ntt(t.data_ptr(), log_n, 1, inverse, coset, stream)
    assert rc == 0, lib.zg_last_error()
def check(log_n, inverse, coset):
    b = data(log_n, 1 << log_n)
    t = dev(b)
    ntt(t, log_n, inverse, coset)
    torch.cuda.synchronize()
    assert t.cpu().numpy().tobytes() == oracle.ntt(b, bool(inverse), coset, 1 << log_n), (log_n, inverse, coset)
"""


def run(body):
    code = COMMON.format(root=os.path.dirname(HERE), here=HERE) + body
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-2000:]


def test_tables_are_bounded_and_the_rest_runs_without():
    # both directions of 2^22 take the whole allowance
    run("""
t = dev(data(1, 1 << 22))
a, b = t.clone(), t.clone()
ntt(t, 22)
ntt(t, 22, 1)
torch.cuda.synchronize()
assert torch.equal(a, t)
free0 = torch.cuda.mem_get_info()[0]
for log_n in (12, 13, 17, 18):
    for inverse, coset in ((0, 0), (1, 0), (0, 1), (0, 2)):
        check(log_n, inverse, coset)
ntt(b, 21), ntt(b, 21, 1), ntt(b, 21, 0, 1), ntt(b, 22, 0, 2)
torch.cuda.synchronize()
torch.cuda.empty_cache()
held = free0 - torch.cuda.mem_get_info()[0]
assert held < 64 << 20, held
""")


def test_other_direction_is_captured_first():
    run("""
b = data(3, 1 << 13)
t, w = dev(b), dev(b)
s = torch.cuda.Stream()
ntt(w, 13, 0, 0, s.cuda_stream)
s.synchronize()
g = torch.cuda.CUDAGraph()
with torch.cuda.graph(g, stream=s):
    ntt(t, 13, 1, 0, s.cuda_stream)
g.replay()
torch.cuda.synchronize()
assert t.cpu().numpy().tobytes() == oracle.ntt(b, True)
""")
