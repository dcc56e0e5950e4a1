// Keccak-256 (Keccak-f[1600], rate 136 bytes, original 0x01 padding) as used
// by the reference's Merkle tree (tiny-keccak 2.0.2 `Keccak::v256`,
// crates/encoder/src/utils.rs:45-66; keccak-hash 0.10 `keccak`,
// crates/encoder/src/merkle/slice.rs:95). State lives in 25 64-bit
// registers.
#pragma once
#include <stdint.h>

namespace zg {

__device__ __constant__ uint64_t KECCAK_RC_DEV[24] = {
    0x0000000000000001ULL, 0x0000000000008082ULL, 0x800000000000808aULL, 0x8000000080008000ULL,
    0x000000000000808bULL, 0x0000000080000001ULL, 0x8000000080008081ULL, 0x8000000000008009ULL,
    0x000000000000008aULL, 0x0000000000000088ULL, 0x0000000080008009ULL, 0x000000008000000aULL,
    0x000000008000808bULL, 0x800000000000008bULL, 0x8000000000008089ULL, 0x8000000000008003ULL,
    0x8000000000008002ULL, 0x8000000000000080ULL, 0x000000000000800aULL, 0x800000008000000aULL,
    0x8000000080008081ULL, 0x8000000000008080ULL, 0x0000000080000001ULL, 0x8000000080008008ULL};

// rotation by a constant as two funnel shifts of the 32-bit halves (written
// with 64-bit shifts, the rounds came out 15 % longer)
__device__ __forceinline__ uint64_t k_rotl(uint64_t x, int s) {
  uint32_t lo = (uint32_t)x, hi = (uint32_t)(x >> 32);
  if (s >= 32) {
    const uint32_t t = lo;
    lo = hi;
    hi = t;
  }
  return (uint64_t)__funnelshift_l(lo, hi, s & 31) << 32 | __funnelshift_l(hi, lo, s & 31);
}

// One round. Theta's d_x = c_(x-1) ^ rotl(c_(x+1), 1) is never formed: both
// terms go into each lane's XOR, one three-input logic operation per half.
__device__ __forceinline__ void keccak_round(uint64_t a[25], uint64_t rc) {
  const uint64_t c0 = a[0] ^ a[5] ^ a[10] ^ a[15] ^ a[20];
  const uint64_t c1 = a[1] ^ a[6] ^ a[11] ^ a[16] ^ a[21];
  const uint64_t c2 = a[2] ^ a[7] ^ a[12] ^ a[17] ^ a[22];
  const uint64_t c3 = a[3] ^ a[8] ^ a[13] ^ a[18] ^ a[23];
  const uint64_t c4 = a[4] ^ a[9] ^ a[14] ^ a[19] ^ a[24];
  const uint64_t r0 = k_rotl(c0, 1), r1 = k_rotl(c1, 1), r2 = k_rotl(c2, 1), r3 = k_rotl(c3, 1), r4 = k_rotl(c4, 1);
  // rho + pi: b[y + 5((2x + 3y) % 5)] = rotl(a[x + 5y], r[x][y])
  uint64_t b[25];
  b[0] = a[0] ^ c4 ^ r1;
  b[10] = k_rotl(a[1] ^ c0 ^ r2, 1);
  b[20] = k_rotl(a[2] ^ c1 ^ r3, 62);
  b[5] = k_rotl(a[3] ^ c2 ^ r4, 28);
  b[15] = k_rotl(a[4] ^ c3 ^ r0, 27);
  b[16] = k_rotl(a[5] ^ c4 ^ r1, 36);
  b[1] = k_rotl(a[6] ^ c0 ^ r2, 44);
  b[11] = k_rotl(a[7] ^ c1 ^ r3, 6);
  b[21] = k_rotl(a[8] ^ c2 ^ r4, 55);
  b[6] = k_rotl(a[9] ^ c3 ^ r0, 20);
  b[7] = k_rotl(a[10] ^ c4 ^ r1, 3);
  b[17] = k_rotl(a[11] ^ c0 ^ r2, 10);
  b[2] = k_rotl(a[12] ^ c1 ^ r3, 43);
  b[12] = k_rotl(a[13] ^ c2 ^ r4, 25);
  b[22] = k_rotl(a[14] ^ c3 ^ r0, 39);
  b[23] = k_rotl(a[15] ^ c4 ^ r1, 41);
  b[8] = k_rotl(a[16] ^ c0 ^ r2, 45);
  b[18] = k_rotl(a[17] ^ c1 ^ r3, 15);
  b[3] = k_rotl(a[18] ^ c2 ^ r4, 21);
  b[13] = k_rotl(a[19] ^ c3 ^ r0, 8);
  b[14] = k_rotl(a[20] ^ c4 ^ r1, 18);
  b[24] = k_rotl(a[21] ^ c0 ^ r2, 2);
  b[9] = k_rotl(a[22] ^ c1 ^ r3, 61);
  b[19] = k_rotl(a[23] ^ c2 ^ r4, 56);
  b[4] = k_rotl(a[24] ^ c3 ^ r0, 14);
#pragma unroll
  for (int y = 0; y < 5; ++y) {
    uint64_t t0 = b[5 * y], t1 = b[5 * y + 1], t2 = b[5 * y + 2], t3 = b[5 * y + 3], t4 = b[5 * y + 4];
    a[5 * y] = t0 ^ (~t1 & t2);
    a[5 * y + 1] = t1 ^ (~t2 & t3);
    a[5 * y + 2] = t2 ^ (~t3 & t4);
    a[5 * y + 3] = t3 ^ (~t4 & t0);
    a[5 * y + 4] = t4 ^ (~t0 & t1);
  }
  a[0] ^= rc;
}

// 24 rounds, two per loop turn: bounded by the ALU pipe's 180 logic and shift
// operations per round (67 clocks per SM and permutation at 64 lanes a
// clock). Measured over 393 216 leaves on a B200: 74 clocks, 4.0 G
// permutations/s; one round per turn 88 clocks (3.4 G/s, theta's d formed:
// 20 operations more and the state moved at every turn), all 24 unrolled 87
// (instruction cache). Rotations as multiplications on the idle multiply
// pipe were slower the more of them there were (77 - 84 clocks).
__device__ __forceinline__ void keccak_f1600(uint64_t a[25]) {
#pragma unroll 1
  for (int round = 0; round < 24; round += 2) {
    keccak_round(a, KECCAK_RC_DEV[round]);
    keccak_round(a, KECCAK_RC_DEV[round + 1]);
  }
}

// keccak256 of exactly 64 bytes given as 8 little-endian words
__device__ __forceinline__ void keccak256_64(const uint64_t in[8], uint64_t out[4]) {
  uint64_t a[25];
#pragma unroll
  for (int i = 0; i < 25; ++i) a[i] = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) a[i] = in[i];
  a[8] = 0x01;                      // padding byte at offset 64
  a[16] = 0x8000000000000000ULL;    // final bit at offset 135
  keccak_f1600(a);
#pragma unroll
  for (int i = 0; i < 4; ++i) out[i] = a[i];
}

// keccak256 of exactly 256 bytes, get(k) = little-endian words 2 k and 2 k + 1
// (word 16's pair is read for each of the two blocks)
template <class Get>
__device__ __forceinline__ void keccak256_256(Get get, uint64_t out[4]) {
  uint64_t a[25];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const ulonglong2 v = get(i);
    a[2 * i] = v.x;
    a[2 * i + 1] = v.y;
  }
  a[16] = get(8).x;
#pragma unroll
  for (int i = 17; i < 25; ++i) a[i] = 0;
  keccak_f1600(a);
  a[0] ^= get(8).y;
#pragma unroll
  for (int i = 9; i < 16; ++i) {
    const ulonglong2 v = get(i);
    a[2 * i - 17] ^= v.x;
    a[2 * i - 16] ^= v.y;
  }
  a[15] ^= 0x01;                    // offset 120 of the second block
  a[16] ^= 0x8000000000000000ULL;
  keccak_f1600(a);
#pragma unroll
  for (int i = 0; i < 4; ++i) out[i] = a[i];
}

}  // namespace zg
