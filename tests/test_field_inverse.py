"""The field inverse (Fp::inverse, csrc/zg_field.cuh).

The host path runs compiled, against a^(p - 2). A model with Python integers
restates the division steps and checks what the packed words and limbs rely
on: the halves of 15 steps' matrix rows fit 16 bits, |f| and |g| stay below
2^256, |d| and |e| at most 11 p, and 20 batches end with f = +-1, g = 0. The
device forms (predicated steps, four lanes per value) are checked by
zg_selftest.
"""
import os
import random
import shutil
import subprocess

import pytest

import zgo

HERE = os.path.dirname(os.path.abspath(__file__))


def test_host_inverse_matches_exponentiation(tmp_path):
    cxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else shutil.which("g++")
    exe = str(tmp_path / "field_inverse")
    subprocess.run([cxx, "-std=c++20", "-O1", "-fsanitize=address,undefined", "-o", exe,
                    os.path.join(HERE, "emu", "field_inverse.cpp"), "-lpthread"], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr


M32 = (1 << 32) - 1


def steps15(k0, x, y, nd2):
    """15 steps from step k0 on: words, delta and the two matrix rows"""
    U, Q = (1, 0), (0, 1)
    for k in range(k0, k0 + 15):
        odd = y >> k & 1
        swap = odd and nd2 < 0
        if odd:
            s = -1 if swap else 1
            y = (y + s * x) & M32
            Q = (Q[0] + s * U[0], Q[1] + s * U[1])
        if swap:
            x = (x + y) & M32
            U = (U[0] + Q[0], U[1] + Q[1])
            nd2 = -nd2
        nd2 -= 2
        x = x << 1 & M32
        if k < k0 + 14:
            U = (2 * U[0], 2 * U[1])
    # what the 16-bit halves of a word hold
    assert max(map(abs, U)) <= 1 << 14
    assert abs(Q[0]) + abs(Q[1]) <= 1 << 15 and all(-(1 << 15) <= q < 1 << 15 for q in Q)
    return x, y, nd2, (2 * U[0], 2 * U[1]), Q


def inverse_model(P, a):
    pinv = pow(P, -1, 1 << 30)

    def mod_row(u, d, v, e):
        t = u * d + v * e
        k = -t * pinv & ((1 << 30) - 1)
        if k >= 1 << 29:
            k -= 1 << 30
        assert (t + k * P) % (1 << 30) == 0
        return (t + k * P) >> 30

    f, g, d, e, nd2 = P, a, 0, pow(2, 542, P), -1
    for _ in range(20):
        x, y, nd2, (u1, v1), (q1, r1) = steps15(0, f & M32, g & M32, nd2)
        x, y, nd2, (u2, v2), (q2, r2) = steps15(15, x, y, nd2)
        u, v = u2 * u1 + v2 * q1, u2 * v1 + v2 * r1
        q, r = q2 * u1 + r2 * q1, q2 * v1 + r2 * r1
        assert abs(u) + abs(v) <= 1 << 30 and abs(q) + abs(r) <= 1 << 30
        assert (u * f + v * g) % (1 << 30) == 0 and (q * f + r * g) % (1 << 30) == 0
        f, g = (u * f + v * g) >> 30, (q * f + r * g) >> 30
        d, e = mod_row(u, d, v, e), mod_row(q, d, r, e)
        assert max(abs(f), abs(g)) < 1 << 256 and max(abs(d), abs(e)) <= 11 * P
    assert g == 0 and (abs(f) == 1 or a == 0)
    out = mod_row(-1 if f < 0 else 1, d, 0, 0)
    assert -P < out < P
    return out + P if out < 0 else out


@pytest.mark.parametrize("P", [zgo.Q_MOD, zgo.R_MOD])
def test_division_steps_model(P):
    rng = random.Random(30)
    vals = list(range(0, 9)) + [1 << k for k in range(9, 254)] + [P // 2, P // 2 + 1, P // 3]
    vals += [rng.randrange(P) for _ in range(600)] + [rng.getrandbits(40) for _ in range(60)]
    vals += [P - x for x in vals if 0 < x < P]
    r2 = pow(2, 512, P)
    for a in vals:
        if a < P:
            assert inverse_model(P, a) == (pow(a, -1, P) * r2 % P if a else 0)
