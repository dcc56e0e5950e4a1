"""Exact-integer model of the FP64-pipe product (csrc/zg_field_f64.cuh), Fq and Fr.

The device routine holds the operands in 51-bit limbs, splits every limb
product with two FMAs (exact, so the integer halves below are what the device
computes), lets two products of a column share one high and one low sum, and
adds the sums' bit patterns to 64-bit columns. This test restates the schedule
with Python integers: the result against a * b / 2^256 mod p, the sums' ranges
that keep the doubles exact, the number of sums per column that the columns'
initial values cancel, and the constants written in Limbs51. The device
routine itself is checked by zg_selftest (checks 1 and 8).
"""
import random

import pytest

import zgo

M51 = (1 << 51) - 1
M64 = (1 << 64) - 1
KL = 0x4330000000000000  # bit pattern of the double 2^52
KH = 0x4660000000000000  # bit pattern of the double 2^103
NLOW = [1, 2, 3, 4, 5, 5, 4, 3, 2, 0]
NHIGH = [0, 2, 3, 4, 5, 6, 5, 4, 3, 2]
# the constants written in Limbs51<FqCfg> / Limbs51<FrCfg>
DEVICE_CONSTS = {
    zgo.Q_MOD: ([0x8C16D87CFD47, 0x22D0E3951A784, 0x60561765E05AA, 0x14DC2822DB40, 0x30644E72E131A],
                0x20782E4866389, 0x20782E4866389),
    zgo.R_MOD: ([0x1F593F0000001, 0x10F372E12287C, 0x6056174A0CFA1, 0x14DC2822DB40, 0x30644E72E131A],
                0x1F593EFFFFFFF, 0x1F593EFFFFFFF),
}


def mont_mul_model(P, a, b):
    PL, p51, p52 = DEVICE_CONSTS[P]
    A = [(a >> (51 * k)) & M51 for k in range(4)] + [a >> 204]
    B = [(b >> (51 * k)) & M51 for k in range(4)] + [b >> 204]
    assert max(A[4], B[4]) <= M51
    t = [(-NLOW[c] * KL - NHIGH[c] * KH) & M64 for c in range(10)]
    true = [0] * 10
    sums = [[0] * 10, [0] * 10]

    def low(c, v):
        assert v < 1 << 52  # 2^52 + v is an exact double with unit spacing
        t[c] = (t[c] + KL + v) & M64
        true[c] += v
        sums[0][c] += 1

    def high(c, v):
        assert v < 1 << 52  # 2^103 + 2^51 v stays below 2^104
        t[c] = (t[c] + KH + v) & M64
        true[c] += v
        sums[1][c] += 1

    def one(c, x, y):
        low(c, x * y & M51)
        high(c + 1, x * y >> 51)

    def two(c, x, y, z, w):
        assert x * y < 1 << 102 and z * w < 1 << 102
        low(c, (x * y & M51) + (z * w & M51))
        high(c + 1, (x * y >> 51) + (z * w >> 51))

    def carry(c):  # column c is a multiple of 2^51 once m p_0's low half is in
        t[c + 1] = (t[c + 1] + ((t[c] + M51 & M64) >> 51)) & M64
        true[c + 1] += true[c] + M51 >> 51

    m = [0] * 5

    def quot(c):
        m[c] = (t[c] & M51) * p51 & M51
        high(c + 1, m[c] * PL[0] >> 51)
        carry(c)

    one(0, A[0], B[0])
    quot(0)
    two(1, A[0], B[1], A[1], B[0])
    one(1, m[0], PL[1])
    quot(1)
    two(2, A[0], B[2], A[1], B[1])
    two(2, A[2], B[0], m[0], PL[2])
    one(2, m[1], PL[1])
    quot(2)
    two(3, A[0], B[3], A[1], B[2])
    two(3, A[2], B[1], A[3], B[0])
    two(3, m[0], PL[3], m[1], PL[2])
    one(3, m[2], PL[1])
    quot(3)
    two(4, A[0], B[4], A[1], B[3])
    two(4, A[2], B[2], A[3], B[1])
    two(4, A[4], B[0], m[0], PL[4])
    two(4, m[1], PL[3], m[2], PL[2])
    one(4, m[3], PL[1])
    two(5, A[1], B[4], A[2], B[3])
    two(5, A[3], B[2], A[4], B[1])
    two(5, m[1], PL[4], m[2], PL[3])
    one(5, m[3], PL[2])
    # t's pending initial values are multiples of 2^52: the low bits are true
    u = ((t[4] & ((1 << 52) - 1)) ^ ((t[5] & 1) << 51))
    m[4] = u * p52 & ((1 << 52) - 1)
    high(5, m[4] * PL[0] >> 51)
    carry(4)
    one(5, m[4], PL[1])
    two(6, A[2], B[4], A[3], B[3])
    two(6, A[4], B[2], m[2], PL[4])
    one(6, m[3], PL[3])
    one(6, m[4], PL[2])
    two(7, A[3], B[4], A[4], B[3])
    one(7, m[3], PL[4])
    one(7, m[4], PL[3])
    one(8, A[4], B[4])
    one(8, m[4], PL[4])
    assert sums == [NLOW, NHIGH]
    assert t == true and max(true) < 1 << 57
    assert t[5] & 1 == 0
    r = sum(t[c] << (51 * (c - 5)) for c in range(5, 10)) >> 1
    assert r < 2 * P
    return r - P if r >= P else r


@pytest.mark.parametrize("P", [zgo.Q_MOD, zgo.R_MOD])
def test_device_constants(P):
    limbs, p51, p52 = DEVICE_CONSTS[P]
    assert sum(x << (51 * k) for k, x in enumerate(limbs)) == P
    assert (P * p51 + 1) % (1 << 51) == 0 and (P * p52 + 1) % (1 << 52) == 0


@pytest.mark.parametrize("P", [zgo.Q_MOD, zgo.R_MOD])
def test_model_matches_montgomery_product(P):
    rng = random.Random(51)
    edge = [0, 1, 2, P - 1, P - 2, (1 << 253) - 1, 1 << 200, M51, M51 << 51]
    pairs = [(x, y) for x in edge for y in edge]
    pairs += [(rng.randrange(P), rng.randrange(P)) for _ in range(3000)]
    rinv = pow(2, -256, P)
    for a, b in pairs:
        assert mont_mul_model(P, a, b) == a * b * rinv % P
