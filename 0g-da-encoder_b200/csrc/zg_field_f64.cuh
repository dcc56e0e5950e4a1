// BN254 Montgomery product (Fq and Fr) on the FP64 pipe (device only).
//
// The integer product (Fp::mul) keeps the integer multiply-add pipe busy; the
// FP64 pipe of the SM (DFMA at the same rate on sm_100a) is idle beside it.
// This product computes the same value (a * b / 2^256 mod p, 8 x 32-bit words)
// with 51-bit limbs held in doubles:
//
//  * operands below 2^255 are split into 5 limbs of 51 bits, each an exact
//    double;
//  * a limb product xy (< 2^102) is split exactly into hi = floor(xy / 2^51)
//    and lo = xy mod 2^51 by two FMAs: h = fma_rz(x, y, 2^103) holds hi in its
//    mantissa, and l = fma(x, y, 2^103 + 2^52 - h) = 2^52 + lo is exact (the
//    split of Emmart, Zheng and Weems, "Faster Modular Exponentiation Using
//    Double Precision Floating Point Arithmetic on the GPU", ARITH 2018);
//  * two products of one column share their sums: the second's FMA starts
//    from the first's h (2^103 + two halves < 2^104, the same binade), and the
//    two low halves meet in one FP64 addition (2^52 + lo + lo' < 2^53);
//  * the bit patterns of the sums (integers offset by the patterns of 2^103
//    and 2^52) go to 64-bit integer column accumulators whose initial values
//    cancel the offsets, multiples of 2^52, so a column's low 52 bits are
//    exact at any time;
//  * Montgomery reduction runs column by column: 4 steps of 51 bits and one of
//    52 (which reads the lowest bit of column 5) remove 256 bits, m = t_k *
//    (-p^-1) by the same split; the low half of m p_0 only completes the
//    column to a multiple of 2^51, so the carry is the rounded-up quotient and
//    that half is never computed;
//  * the result (< 2p) is repacked into 32-bit words and reduced once.
// Column sums stay below 2^57 (at most 18 halves below 2^52 plus a carry).
//
// Why 51 bits: with 52 (one product per h and l, 100 64-bit additions) the
// column additions bound the product, on the ALU pipe that also does the
// shifts and masks: 53 G products/s for a pair on a B200 against 57 - 62 with
// shared sums (360 instructions a product, FP64 pipe 62 % and ALU 50 % busy).
// Paired with an integer product it reaches 65 G/s (56 before): both pipes
// have room left, but an FP64 instruction holds the dispatch port like two
// others, and that is what the pair runs into.
#pragma once
#include "zg_field.cuh"

namespace zg {
namespace f51 {

constexpr uint64_t KL = 0x4330000000000000ull;  // bit pattern of 2^52
constexpr uint64_t KH = 0x4660000000000000ull;  // bit pattern of 2^103
constexpr uint64_t M51 = (1ull << 51) - 1;

// low and high sums that column c receives (the schedule of mont_mul)
__host__ __device__ constexpr int nlow(int c) {
  constexpr int n[10] = {1, 2, 3, 4, 5, 5, 4, 3, 2, 0};
  return n[c];
}
__host__ __device__ constexpr int nhigh(int c) {
  constexpr int n[10] = {0, 2, 3, 4, 5, 6, 5, 4, 3, 2};
  return n[c];
}
__host__ __device__ constexpr uint64_t col_init(int c) {
  return (uint64_t)0 - (uint64_t)nlow(c) * KL - (uint64_t)nhigh(c) * KH;
}

// 51-bit limbs of the modulus, -p^-1 mod 2^51 and mod 2^52 (Fq and Fr)
template <class C> struct Limbs51;
template <> struct Limbs51<FqCfg> {
  static __device__ __forceinline__ double P(int j) {
    return j == 0 ? (double)0x8c16d87cfd47ull
         : j == 1 ? (double)0x22d0e3951a784ull
         : j == 2 ? (double)0x60561765e05aaull
         : j == 3 ? (double)0x14dc2822db40ull
                  : (double)0x30644e72e131aull;
  }
  static constexpr double PINV51 = (double)0x20782e4866389ull;
  static constexpr double PINV52 = (double)0x20782e4866389ull;
};
template <> struct Limbs51<FrCfg> {
  static __device__ __forceinline__ double P(int j) {
    return j == 0 ? (double)0x1f593f0000001ull
         : j == 1 ? (double)0x10f372e12287cull
         : j == 2 ? (double)0x6056174a0cfa1ull
         : j == 3 ? (double)0x14dc2822db40ull
                  : (double)0x30644e72e131aull;
  }
  static constexpr double PINV51 = (double)0x1f593efffffffull;
  static constexpr double PINV52 = (double)0x1f593efffffffull;
};

// exact double of the 52-bit integer hi20:lo (hi20 < 2^20)
__device__ __forceinline__ double u52(uint32_t lo, uint32_t hi20) {
  return __dsub_rn(__hiloint2double((int)(hi20 | 0x43300000u), (int)lo), 0x1p52);
}

template <class C>
__device__ __forceinline__ void split(const Fp<C>& a, double* x) {
  const uint32_t* w = a.v;
  x[0] = u52(w[0], w[1] & 0x7ffffu);
  x[1] = u52(__funnelshift_r(w[1], w[2], 19), __funnelshift_r(w[2], w[3], 19) & 0x7ffffu);
  x[2] = u52(__funnelshift_r(w[3], w[4], 6), (w[4] >> 6) & 0x7ffffu);
  x[3] = u52(__funnelshift_r(w[4], w[5], 25), __funnelshift_r(w[5], w[6], 25) & 0x7ffffu);
  x[4] = u52(__funnelshift_r(w[6], w[7], 12), w[7] >> 12);
}

__device__ __forceinline__ uint64_t bits(double x) { return (uint64_t)__double_as_longlong(x); }

// x y: lo += bits(2^52 + low half), hi += bits(2^103 + 2^51 high half); x y < 2^103
__device__ __forceinline__ void one(double x, double y, uint64_t& lo, uint64_t& hi) {
  const double h = __fma_rz(x, y, 0x1p103);
  lo += bits(__fma_rn(x, y, __dsub_rn(0x1p103 + 0x1p52, h)));
  hi += bits(h);
}
// x y + z w, each below 2^102: one low and one high sum for both
__device__ __forceinline__ void two(double x, double y, double z, double w, uint64_t& lo, uint64_t& hi) {
  const double h = __fma_rz(x, y, 0x1p103);
  const double g = __fma_rz(z, w, h);
  const double l = __fma_rn(x, y, __dsub_rn(0x1p103 + 0x1p52, h));
  lo += bits(__dadd_rn(l, __fma_rn(z, w, __dsub_rn(h, g))));
  hi += bits(g);
}
// (low 51 bits of t) * -p^-1 mod 2^51
template <class C>
__device__ __forceinline__ double quot(uint64_t t) {
  const double u = u52((uint32_t)t, (uint32_t)(t >> 32) & 0x7ffffu);
  const double h = __fma_rz(u, Limbs51<C>::PINV51, 0x1p103);
  return __fma_rn(u, Limbs51<C>::PINV51, __dsub_rn(0x1p103, h));
}

// a * b / 2^256 mod p for a, b < 2p; result < p (p the modulus of C: Fq or Fr)
template <class C>
__device__ __forceinline__ Fp<C> mont_mul(const Fp<C>& a, const Fp<C>& b) {
  typedef Limbs51<C> L;
  double A[5], B[5], m[5], P[5];
  split(a, A);
  split(b, B);
#pragma unroll
  for (int j = 0; j < 5; ++j) P[j] = L::P(j);
  uint64_t t[10];
#pragma unroll
  for (int c = 0; c < 10; ++c) t[c] = col_init(c);

  one(A[0], B[0], t[0], t[1]);
  m[0] = quot<C>(t[0]);
  t[1] += bits(__fma_rz(m[0], P[0], 0x1p103)) + ((t[0] + M51) >> 51);

  two(A[0], B[1], A[1], B[0], t[1], t[2]);
  one(m[0], P[1], t[1], t[2]);
  m[1] = quot<C>(t[1]);
  t[2] += bits(__fma_rz(m[1], P[0], 0x1p103)) + ((t[1] + M51) >> 51);

  two(A[0], B[2], A[1], B[1], t[2], t[3]);
  two(A[2], B[0], m[0], P[2], t[2], t[3]);
  one(m[1], P[1], t[2], t[3]);
  m[2] = quot<C>(t[2]);
  t[3] += bits(__fma_rz(m[2], P[0], 0x1p103)) + ((t[2] + M51) >> 51);

  two(A[0], B[3], A[1], B[2], t[3], t[4]);
  two(A[2], B[1], A[3], B[0], t[3], t[4]);
  two(m[0], P[3], m[1], P[2], t[3], t[4]);
  one(m[2], P[1], t[3], t[4]);
  m[3] = quot<C>(t[3]);
  t[4] += bits(__fma_rz(m[3], P[0], 0x1p103)) + ((t[3] + M51) >> 51);

  two(A[0], B[4], A[1], B[3], t[4], t[5]);
  two(A[2], B[2], A[3], B[1], t[4], t[5]);
  two(A[4], B[0], m[0], P[4], t[4], t[5]);
  two(m[1], P[3], m[2], P[2], t[4], t[5]);
  one(m[3], P[1], t[4], t[5]);
  two(A[1], B[4], A[2], B[3], t[5], t[6]);
  two(A[3], B[2], A[4], B[1], t[5], t[6]);
  two(m[1], P[4], m[2], P[3], t[5], t[6]);
  one(m[3], P[2], t[5], t[6]);
  {
    // the last step clears 52 bits: bit 51 is column 4's plus column 5's lowest
    const double u = u52((uint32_t)t[4], ((uint32_t)(t[4] >> 32) ^ ((uint32_t)t[5] << 19)) & 0xfffffu);
    const double h = __fma_rz(u, L::PINV52, 0x1p104);
    m[4] = __fma_rn(u, L::PINV52, __dsub_rn(0x1p104, h));
  }
  t[5] += bits(__fma_rz(m[4], P[0], 0x1p103)) + ((t[4] + M51) >> 51);
  one(m[4], P[1], t[5], t[6]);
  two(A[2], B[4], A[3], B[3], t[6], t[7]);
  two(A[4], B[2], m[2], P[4], t[6], t[7]);
  one(m[3], P[3], t[6], t[7]);
  one(m[4], P[2], t[6], t[7]);
  two(A[3], B[4], A[4], B[3], t[7], t[8]);
  one(m[3], P[4], t[7], t[8]);
  one(m[4], P[3], t[7], t[8]);
  one(A[4], B[4], t[8], t[9]);
  one(m[4], P[4], t[8], t[9]);

  // normalise columns 5..9 (column 5 is even now); the value is half of
  // sum t_c 2^(51 (c - 5))
  t[6] += t[5] >> 51;
  t[7] += t[6] >> 51;
  t[8] += t[7] >> 51;
  t[9] += t[8] >> 51;
  const uint64_t n5 = t[5] & M51, n6 = t[6] & M51, n7 = t[7] & M51, n8 = t[8] & M51, n9 = t[9];
  Fp<C> r;
  r.v[0] = (uint32_t)(n5 >> 1);
  r.v[1] = (uint32_t)(n5 >> 33) | (uint32_t)(n6 << 18);
  r.v[2] = (uint32_t)(n6 >> 14);
  r.v[3] = (uint32_t)(n6 >> 46) | (uint32_t)(n7 << 5);
  r.v[4] = (uint32_t)(n7 >> 27) | (uint32_t)(n8 << 24);
  r.v[5] = (uint32_t)(n8 >> 8);
  r.v[6] = (uint32_t)(n8 >> 40) | (uint32_t)(n9 << 11);
  r.v[7] = (uint32_t)(n9 >> 21);
  Fp<C> s;
  const uint32_t borrow = Fp<C>::sub_raw(s, r, Fp<C>::modulus());
  return borrow ? r : s;
}

}  // namespace f51
}  // namespace zg
