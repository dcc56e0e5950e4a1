// BN254 prime-field arithmetic for sm_100a: eight 32-bit limbs, Montgomery
// form with R = 2^256 (the same representation as ark-ff's four 64-bit limbs,
// so device buffers and the reference's mont param files share bytes,
// crates/amt/src/prove_params/fast_serde_bn254.rs:139-187).
//
// Multiplication is CIOS Montgomery: per limb b_i one multiply-accumulate row
// t += a * b_i and one reduction row t += m * p. The accumulator is kept as
// two word arrays, one for the products of even limbs and one for those of
// odd limbs (Fp::Acc): each lo/hi pair of a carry chain then fills one aligned
// register pair, so mad.lo.cc / madc.hi.cc issue as ONE wide multiply-add with
// carry. sm_100a runs 32 of those per SM and clock (a lone mad.hi costs the
// same), so the product is bounded by 128 wide + 8 narrow multiply-adds = 4.1
// clocks per SM; measured 4.5 (64 G products/s on a B200, multiply pipe 92 %
// busy), against 6.1 clocks (47 G/s) for one accumulator array, whose odd
// chains straddle the pairs and issue lo and hi apart. (Separate rows for even
// and odd limbs are a published technique of big-number libraries for GPUs
// with multiply-adds on register pairs.) Outputs that are
// written before every input of an asm block has been read are early-clobber
// ("=&r"), so the compiler never assigns them an input's register. Host builds
// use a portable 64-bit path with identical results.
#pragma once
#include <stdint.h>

#ifndef ZG_HD
#define ZG_HD __host__ __device__ __forceinline__
#endif

namespace zg {

struct FqCfg {
  static constexpr uint32_t p0 = 0xd87cfd47u, p1 = 0x3c208c16u, p2 = 0x6871ca8du, p3 = 0x97816a91u,
                            p4 = 0x8181585du, p5 = 0xb85045b6u, p6 = 0xe131a029u, p7 = 0x30644e72u;
  static constexpr uint32_t inv = 0xe4866389u;
  static constexpr uint32_t r2_0 = 0x538afa89u, r2_1 = 0xf32cfc5bu, r2_2 = 0xd44501fbu, r2_3 = 0xb5e71911u,
                            r2_4 = 0x0a417ff6u, r2_5 = 0x47ab1effu, r2_6 = 0xcab8351fu, r2_7 = 0x06d89f71u;
  static constexpr uint32_t one0 = 0xc58f0d9du, one1 = 0xd35d438du, one2 = 0xf5c70b3du, one3 = 0x0a78eb28u,
                            one4 = 0x7879462cu, one5 = 0x666ea36fu, one6 = 0x9a07df2fu, one7 = 0x0e0a77c1u;
  // 2^(30 + 512) mod p, the start of inverse()
  static constexpr uint32_t gcd0 = 0xe0d1e109u, gcd1 = 0x54964889u, gcd2 = 0x580bb0b7u, gcd3 = 0xf5c72b3bu,
                            gcd4 = 0xf3b7923cu, gcd5 = 0x9507f0f3u, gcd6 = 0x65a80820u, gcd7 = 0x03f1b742u;
};
struct FrCfg {
  static constexpr uint32_t p0 = 0xf0000001u, p1 = 0x43e1f593u, p2 = 0x79b97091u, p3 = 0x2833e848u,
                            p4 = 0x8181585du, p5 = 0xb85045b6u, p6 = 0xe131a029u, p7 = 0x30644e72u;
  static constexpr uint32_t inv = 0xefffffffu;
  static constexpr uint32_t r2_0 = 0xae216da7u, r2_1 = 0x1bb8e645u, r2_2 = 0xe35c59e3u, r2_3 = 0x53fe3ab1u,
                            r2_4 = 0x53bb8085u, r2_5 = 0x8c49833du, r2_6 = 0x7f4e44a5u, r2_7 = 0x0216d0b1u;
  static constexpr uint32_t one0 = 0x4ffffffbu, one1 = 0xac96341cu, one2 = 0x9f60cd29u, one3 = 0x36fc7695u,
                            one4 = 0x7879462eu, one5 = 0x666ea36fu, one6 = 0x9a07df2fu, one7 = 0x0e0a77c1u;
  static constexpr uint32_t gcd0 = 0x7d3cafd4u, gcd1 = 0xec641afcu, gcd2 = 0x06b30259u, gcd3 = 0xd72c58d8u,
                            gcd4 = 0x9de13abeu, gcd5 = 0x0a523413u, gcd6 = 0xd945ca5au, gcd7 = 0x0ece42fdu;
};

template <class C>
struct Fp {
  uint32_t v[8];

  ZG_HD static Fp zero() {
    Fp r;
#pragma unroll
    for (int i = 0; i < 8; ++i) r.v[i] = 0;
    return r;
  }
  ZG_HD static Fp modulus() {
    Fp r;
    r.v[0] = C::p0; r.v[1] = C::p1; r.v[2] = C::p2; r.v[3] = C::p3;
    r.v[4] = C::p4; r.v[5] = C::p5; r.v[6] = C::p6; r.v[7] = C::p7;
    return r;
  }
  ZG_HD static Fp one() {
    Fp r;
    r.v[0] = C::one0; r.v[1] = C::one1; r.v[2] = C::one2; r.v[3] = C::one3;
    r.v[4] = C::one4; r.v[5] = C::one5; r.v[6] = C::one6; r.v[7] = C::one7;
    return r;
  }
  ZG_HD static Fp r2() {
    Fp r;
    r.v[0] = C::r2_0; r.v[1] = C::r2_1; r.v[2] = C::r2_2; r.v[3] = C::r2_3;
    r.v[4] = C::r2_4; r.v[5] = C::r2_5; r.v[6] = C::r2_6; r.v[7] = C::r2_7;
    return r;
  }
  ZG_HD bool is_zero() const {
    uint32_t o = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) o |= v[i];
    return o == 0;
  }
  ZG_HD bool operator==(const Fp& o) const {
    uint32_t d = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) d |= v[i] ^ o.v[i];
    return d == 0;
  }
  ZG_HD bool operator!=(const Fp& o) const { return !(*this == o); }

  // ---- add / sub (inputs and outputs fully reduced, in [0, p))
  ZG_HD static Fp add(const Fp& a, const Fp& b) {
    Fp s, t;
    uint32_t carry = add_raw(s, a, b);
    uint32_t borrow = sub_raw(t, s, modulus());
    // keep s when (no carry and borrow) i.e. s < p
    bool keep = (carry == 0) && (borrow != 0);
    return keep ? s : t;
  }
  ZG_HD static Fp sub(const Fp& a, const Fp& b) {
    Fp d, e;
    uint32_t borrow = sub_raw(d, a, b);
    add_raw(e, d, modulus());
    return borrow ? e : d;
  }
  ZG_HD static Fp neg(const Fp& a) {
    if (a.is_zero()) return a;
    Fp r;
    sub_raw(r, modulus(), a);
    return r;
  }
  ZG_HD static Fp dbl(const Fp& a) { return add(a, a); }

  ZG_HD Fp operator+(const Fp& o) const { return add(*this, o); }
  ZG_HD Fp operator-(const Fp& o) const { return sub(*this, o); }
  ZG_HD Fp operator-() const { return neg(*this); }
  ZG_HD Fp operator*(const Fp& o) const { return mul(*this, o); }
  ZG_HD Fp& operator+=(const Fp& o) { *this = add(*this, o); return *this; }
  ZG_HD Fp& operator-=(const Fp& o) { *this = sub(*this, o); return *this; }
  ZG_HD Fp& operator*=(const Fp& o) { *this = mul(*this, o); return *this; }
  ZG_HD Fp sqr() const { return mul(*this, *this); }

  ZG_HD static uint32_t add_raw(Fp& r, const Fp& a, const Fp& b) {
#ifdef __CUDA_ARCH__
    uint32_t c;
    asm("add.cc.u32 %0, %9, %17;\n\t"
        "addc.cc.u32 %1, %10, %18;\n\t"
        "addc.cc.u32 %2, %11, %19;\n\t"
        "addc.cc.u32 %3, %12, %20;\n\t"
        "addc.cc.u32 %4, %13, %21;\n\t"
        "addc.cc.u32 %5, %14, %22;\n\t"
        "addc.cc.u32 %6, %15, %23;\n\t"
        "addc.cc.u32 %7, %16, %24;\n\t"
        "addc.u32 %8, 0, 0;"
        : "=&r"(r.v[0]), "=&r"(r.v[1]), "=&r"(r.v[2]), "=&r"(r.v[3]), "=&r"(r.v[4]), "=&r"(r.v[5]),
          "=&r"(r.v[6]), "=&r"(r.v[7]), "=&r"(c)
        : "r"(a.v[0]), "r"(a.v[1]), "r"(a.v[2]), "r"(a.v[3]), "r"(a.v[4]), "r"(a.v[5]), "r"(a.v[6]),
          "r"(a.v[7]), "r"(b.v[0]), "r"(b.v[1]), "r"(b.v[2]), "r"(b.v[3]), "r"(b.v[4]), "r"(b.v[5]),
          "r"(b.v[6]), "r"(b.v[7]));
    return c;
#else
    uint64_t c = 0;
    for (int i = 0; i < 8; ++i) {
      uint64_t s = (uint64_t)a.v[i] + b.v[i] + c;
      r.v[i] = (uint32_t)s;
      c = s >> 32;
    }
    return (uint32_t)c;
#endif
  }
  // returns 1 on borrow
  ZG_HD static uint32_t sub_raw(Fp& r, const Fp& a, const Fp& b) {
#ifdef __CUDA_ARCH__
    uint32_t c;
    asm("sub.cc.u32 %0, %9, %17;\n\t"
        "subc.cc.u32 %1, %10, %18;\n\t"
        "subc.cc.u32 %2, %11, %19;\n\t"
        "subc.cc.u32 %3, %12, %20;\n\t"
        "subc.cc.u32 %4, %13, %21;\n\t"
        "subc.cc.u32 %5, %14, %22;\n\t"
        "subc.cc.u32 %6, %15, %23;\n\t"
        "subc.cc.u32 %7, %16, %24;\n\t"
        "subc.u32 %8, 0, 0;"
        : "=&r"(r.v[0]), "=&r"(r.v[1]), "=&r"(r.v[2]), "=&r"(r.v[3]), "=&r"(r.v[4]), "=&r"(r.v[5]),
          "=&r"(r.v[6]), "=&r"(r.v[7]), "=&r"(c)
        : "r"(a.v[0]), "r"(a.v[1]), "r"(a.v[2]), "r"(a.v[3]), "r"(a.v[4]), "r"(a.v[5]), "r"(a.v[6]),
          "r"(a.v[7]), "r"(b.v[0]), "r"(b.v[1]), "r"(b.v[2]), "r"(b.v[3]), "r"(b.v[4]), "r"(b.v[5]),
          "r"(b.v[6]), "r"(b.v[7]));
    return c & 1;
#else
    int64_t br = 0;
    for (int i = 0; i < 8; ++i) {
      int64_t s = (int64_t)a.v[i] - b.v[i] - br;
      br = s < 0 ? 1 : 0;
      r.v[i] = (uint32_t)s;
    }
    return (uint32_t)br;
#endif
  }

  // ---- Montgomery multiplication: a * b / R mod p, inputs in [0, p)
  ZG_HD static Fp mul(const Fp& a, const Fp& b) {
#ifdef __CUDA_ARCH__
    Acc t;
    t.first(a, b.v[0]);
#pragma unroll
    for (int i = 1; i < 8; ++i) t.next(a, b.v[i]);
    return t.result();
#else
    return mul_host(a, b);
#endif
  }

#ifndef __CUDA_ARCH__
  // the host product, out of line: inlined into every host use of the
  // extension-field and curve formulas it makes the host object huge and slow
  // to compile, for no speed that matters on the host
  __host__ __attribute__((noinline)) static Fp mul_host(const Fp& a, const Fp& b) {
    uint32_t t[10] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
    const Fp p = modulus();
    for (int i = 0; i < 8; ++i) {
      uint64_t c = 0;
      for (int j = 0; j < 8; ++j) {
        uint64_t s = (uint64_t)a.v[j] * b.v[i] + t[j] + c;
        t[j] = (uint32_t)s;
        c = s >> 32;
      }
      uint64_t s = (uint64_t)t[8] + c;
      t[8] = (uint32_t)s;
      t[9] = (uint32_t)(s >> 32);
      uint32_t m = t[0] * C::inv;
      s = (uint64_t)m * p.v[0] + t[0];
      c = s >> 32;
      for (int j = 1; j < 8; ++j) {
        s = (uint64_t)m * p.v[j] + t[j] + c;
        t[j - 1] = (uint32_t)s;
        c = s >> 32;
      }
      s = (uint64_t)t[8] + c;
      t[7] = (uint32_t)s;
      t[8] = t[9] + (uint32_t)(s >> 32);
    }
    Fp r;
    for (int i = 0; i < 8; ++i) r.v[i] = t[i];
    Fp d;
    uint32_t borrow = sub_raw(d, r, p);
    return (t[8] == 0 && borrow) ? r : d;
  }
#endif

  // two independent products r1 = a*b, r2 = c*d with their CIOS rows
  // interleaved: the two carry chains have no data dependence, so either
  // fills the other's multiply latency.
  ZG_HD static void mul2(const Fp& a, const Fp& b, const Fp& c, const Fp& d, Fp& r1, Fp& r2) {
#ifdef __CUDA_ARCH__
    Acc t, u;
    t.first(a, b.v[0]);
    u.first(c, d.v[0]);
#pragma unroll
    for (int i = 1; i < 8; ++i) {
      t.next(a, b.v[i]);
      u.next(c, d.v[i]);
    }
    r1 = t.result();
    r2 = u.result();
#else
    Fp x = mul(a, b), y = mul(c, d);
    r1 = x;
    r2 = y;
#endif
  }

#ifdef __CUDA_ARCH__
  // CIOS accumulator of one product: the value sum e[k] 2^(32k) +
  // sum o[k] 2^(32(k+1)), so the products of even limbs of a (and p) land on
  // the pairs (e[0],e[1]), (e[2],e[3]), .. and those of odd limbs on
  // (o[0],o[1]), ..: every lo/hi pair of a chain fills one aligned pair of
  // words and issues as one wide multiply-add with carry. Dividing by 2^32
  // after a row renames o to e and e[2..] to o; the leftover word e[1] is
  // added at the head of the next row, its carry entering the odd chain.
  struct Acc {
    uint32_t e[9], o[8];
    // row 0: a * b0, then the reduction row
    __device__ __forceinline__ void first(const Fp& a, uint32_t b) {
#pragma unroll
      for (int k = 0; k < 8; k += 2) {
        const uint64_t x = (uint64_t)a.v[k] * b, y = (uint64_t)a.v[k + 1] * b;
        e[k] = (uint32_t)x;
        e[k + 1] = (uint32_t)(x >> 32);
        o[k] = (uint32_t)y;
        o[k + 1] = (uint32_t)(y >> 32);
      }
      e[8] = 0;
      reduce();
    }
    // the division by 2^32 of the previous row, then the next row
    __device__ __forceinline__ void next(const Fp& a, uint32_t b) {
      const uint32_t low = e[1];
      uint32_t n[8];
#pragma unroll
      for (int k = 0; k < 7; ++k) n[k] = e[k + 2];
      n[7] = 0;
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        e[k] = o[k];
        o[k] = n[k];
      }
      asm("add.cc.u32 %0, %0, %17;\n\t"
          "madc.lo.cc.u32 %9, %19, %22, %9;\n\t"
          "madc.hi.cc.u32 %10, %19, %22, %10;\n\t"
          "madc.lo.cc.u32 %11, %21, %22, %11;\n\t"
          "madc.hi.cc.u32 %12, %21, %22, %12;\n\t"
          "madc.lo.cc.u32 %13, %24, %22, %13;\n\t"
          "madc.hi.cc.u32 %14, %24, %22, %14;\n\t"
          "madc.lo.cc.u32 %15, %26, %22, %15;\n\t"
          "madc.hi.u32 %16, %26, %22, %16;\n\t"
          "mad.lo.cc.u32 %0, %18, %22, %0;\n\t"
          "madc.hi.cc.u32 %1, %18, %22, %1;\n\t"
          "madc.lo.cc.u32 %2, %20, %22, %2;\n\t"
          "madc.hi.cc.u32 %3, %20, %22, %3;\n\t"
          "madc.lo.cc.u32 %4, %23, %22, %4;\n\t"
          "madc.hi.cc.u32 %5, %23, %22, %5;\n\t"
          "madc.lo.cc.u32 %6, %25, %22, %6;\n\t"
          "madc.hi.cc.u32 %7, %25, %22, %7;\n\t"
          "addc.u32 %8, 0, 0;"
          : "+r"(e[0]), "+r"(e[1]), "+r"(e[2]), "+r"(e[3]), "+r"(e[4]), "+r"(e[5]), "+r"(e[6]), "+r"(e[7]),
            "=&r"(e[8]), "+r"(o[0]), "+r"(o[1]), "+r"(o[2]), "+r"(o[3]), "+r"(o[4]), "+r"(o[5]), "+r"(o[6]),
            "+r"(o[7])
          : "r"(low), "r"(a.v[0]), "r"(a.v[1]), "r"(a.v[2]), "r"(a.v[3]), "r"(b), "r"(a.v[4]), "r"(a.v[5]),
            "r"(a.v[6]), "r"(a.v[7]));
      reduce();
    }
    // += m p with m = -e[0] / p mod 2^32, which clears e[0]
    __device__ __forceinline__ void reduce() {
      const uint32_t m = e[0] * C::inv;
      asm("mad.lo.cc.u32 %9, %17, %19, %9;\n\t"
          "madc.hi.cc.u32 %10, %17, %19, %10;\n\t"
          "madc.lo.cc.u32 %11, %17, %21, %11;\n\t"
          "madc.hi.cc.u32 %12, %17, %21, %12;\n\t"
          "madc.lo.cc.u32 %13, %17, %23, %13;\n\t"
          "madc.hi.cc.u32 %14, %17, %23, %14;\n\t"
          "madc.lo.cc.u32 %15, %17, %25, %15;\n\t"
          "madc.hi.u32 %16, %17, %25, %16;\n\t"
          "mad.lo.cc.u32 %0, %17, %18, %0;\n\t"
          "madc.hi.cc.u32 %1, %17, %18, %1;\n\t"
          "madc.lo.cc.u32 %2, %17, %20, %2;\n\t"
          "madc.hi.cc.u32 %3, %17, %20, %3;\n\t"
          "madc.lo.cc.u32 %4, %17, %22, %4;\n\t"
          "madc.hi.cc.u32 %5, %17, %22, %5;\n\t"
          "madc.lo.cc.u32 %6, %17, %24, %6;\n\t"
          "madc.hi.cc.u32 %7, %17, %24, %7;\n\t"
          "addc.u32 %8, %8, 0;"
          : "+r"(e[0]), "+r"(e[1]), "+r"(e[2]), "+r"(e[3]), "+r"(e[4]), "+r"(e[5]), "+r"(e[6]), "+r"(e[7]),
            "+r"(e[8]), "+r"(o[0]), "+r"(o[1]), "+r"(o[2]), "+r"(o[3]), "+r"(o[4]), "+r"(o[5]), "+r"(o[6]),
            "+r"(o[7])
          : "r"(m), "r"(C::p0), "r"(C::p1), "r"(C::p2), "r"(C::p3), "r"(C::p4), "r"(C::p5), "r"(C::p6),
            "r"(C::p7));
    }
    // the value / 2^32 (below 2p), reduced once
    __device__ __forceinline__ Fp result() const {
      Fp r, h;
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        r.v[k] = o[k];
        h.v[k] = e[k + 1];
      }
      add_raw(r, r, h);
      Fp s;
      const uint32_t borrow = sub_raw(s, r, modulus());
      return borrow ? r : s;
    }
  };
#endif

  // canonical (< p) -> Montgomery
  ZG_HD static Fp from_canonical(const Fp& a) { return mul(a, r2()); }
  // Montgomery -> canonical
  ZG_HD Fp to_canonical() const {
    Fp one_raw = zero();
    one_raw.v[0] = 1;
    return mul(*this, one_raw);
  }
  ZG_HD static Fp from_u32(uint32_t x) {
    Fp a = zero();
    a.v[0] = x;
    return from_canonical(a);
  }
  // a^e for a little-endian exponent of n 32-bit words
  ZG_HD Fp pow(const uint32_t* e, int n) const {
    Fp r = one(), b = *this;
    for (int i = 0; i < n; ++i) {
      uint32_t w = e[i];
      for (int k = 0; k < 32; ++k) {
        if (w & 1) r = mul(r, b);
        b = mul(b, b);
        w >>= 1;
      }
    }
    return r;
  }
  ZG_HD Fp pow_u64(uint64_t e) const {
    uint32_t w[2] = {(uint32_t)e, (uint32_t)(e >> 32)};
    return pow(w, 2);
  }
  // Inverse in Montgomery form; inverse(0) = 0. Constant-time division steps
  // (Bernstein and Yang, "Fast constant-time gcd computation and modular
  // inversion", TCHES 2019, with the half-integer delta that needs at most 590
  // steps for 256-bit operands), run 30 at a time on the low words of f and g;
  // each batch of 30 is a 2 x 2 matrix of 31-bit entries that is applied to
  // f, g (signed 30-bit limbs, an exact division by 2^30) and to d, e (the same
  // limbs; a multiple of p makes the division exact). d a = f S and e a = g S
  // mod p hold throughout for the start e = S; 20 batches end with f = +-1,
  // g = 0, so d = +-S / a, and a last division by 2^30 brings |d| <= 11 p
  // (each batch adds up to p / 2) below p.
  // A lone warp's time is the instructions of the 600 steps. x and the matrix'
  // first row double instead of y halving (bit k of y is tested in step k), a
  // row's two entries share a word (15 steps keep them in 16 bits each): 12
  // instructions a step. A lone warp takes 36 000 cycles on a B200 (40 000
  // with two words a row, y halving and 32-bit limbs of d and e), against some
  // 310 000 for the exponentiation by p - 2 (380 products in a row).
  ZG_HD Fp inverse() const {
    int32_t f[9], g[9], d[9], e[9];
    limbs30(modulus(), f);
    limbs30(*this, g);
    limbs30(gcd_start(), e);
#pragma unroll
    for (int i = 0; i < 9; ++i) d[i] = 0;
    int32_t nd2 = -1;  // -2 delta
#pragma unroll 1
    for (int batch = 0; batch < 20; ++batch) {
      uint32_t x = (uint32_t)f[0] | (uint32_t)f[1] << 30, y = (uint32_t)g[0] | (uint32_t)g[1] << 30;
      int32_t u1, v1, q1, r1, u2, v2, q2, r2;
      gcd_steps<0>(x, y, nd2, u1, v1, q1, r1);
      gcd_steps<15>(x, y, nd2, u2, v2, q2, r2);
      const int32_t u = u2 * u1 + v2 * q1, v = u2 * v1 + v2 * r1;
      const int32_t q = q2 * u1 + r2 * q1, r = q2 * v1 + r2 * r1;
      gcd_rows<false>(f, g, u, v, q, r);
      gcd_rows<true>(d, e, u, v, q, r);
    }
    // d / 2^30, with the sign of f
    gcd_rows<true>(d, e, f[8] < 0 ? -1 : 1, 0, 0, 0);
    return from_limbs30(d);
  }
#ifdef __CUDACC__
  // inverse() with the four lanes of a quad (a whole warp calls; a is the same
  // in all four, and so is the result): each lane has the batch's division
  // steps and one column of its matrix, then one of the rows f, g, d, e, whose
  // limbs it exchanges with its neighbour. 26 800 cycles of a lone warp.
  static __device__ __noinline__ Fp inverse_quad(const Fp a) {
    constexpr int32_t M30 = (1 << 30) - 1;
    const uint32_t all = 0xffffffffu, quad = threadIdx.x & 28u, row = threadIdx.x & 3u;
    const bool odd = row & 1u;
    int32_t m[9], p[9];
    {
      const Fp mod = modulus(), start = gcd_start();
      Fp x;
#pragma unroll
      for (int i = 0; i < 8; ++i) x.v[i] = row == 0 ? mod.v[i] : row == 1 ? a.v[i] : row == 2 ? 0u : start.v[i];
      limbs30(x, m);
      limbs30(mod, p);
    }
    int32_t nd2 = -1;
#pragma unroll 1
    for (int batch = 0; batch <= 20; ++batch) {
      int32_t own, other;  // this row' = own this row + other the neighbour's
      if (batch < 20) {
        const uint32_t w = (uint32_t)m[0] | (uint32_t)m[1] << 30;
        uint32_t x = __shfl_sync(all, w, quad), y = __shfl_sync(all, w, quad + 1);
        uint32_t U = odd ? 0u : 1u, Q = odd ? 1u : 0u;
#pragma unroll
        for (int k = 0; k < 30; ++k) {
          gcd_step(x, y, U, Q, nd2, k);
          U <<= 1;
        }
        own = (int32_t)(odd ? Q : U);
        other = (int32_t)__shfl_xor_sync(all, odd ? U : Q, 1);
      } else {  // the division by 2^30 that ends inverse(), with the sign of f
        own = (int32_t)__shfl_sync(all, (uint32_t)m[8], quad) < 0 ? -1 : 1;
        other = 0;
      }
      int64_t c = 0;
      int32_t k = 0;
#pragma unroll
      for (int i = 0; i < 9; ++i) {
        const int32_t n = (int32_t)__shfl_xor_sync(all, (uint32_t)m[i], 1);
        c += (int64_t)own * m[i] + (int64_t)other * n;
        if (i == 0 && row >= 2) k = (int32_t)((uint32_t)c * C::inv << 2) >> 2;
        c += (int64_t)k * p[i];
        if (i) m[i - 1] = (int32_t)c & M30;
        c >>= 30;
      }
      m[8] = (int32_t)c;
    }
    Fp r = from_limbs30(m);
#pragma unroll
    for (int i = 0; i < 8; ++i) r.v[i] = __shfl_sync(all, r.v[i], quad + 2);
    return r;
  }
#endif
  ZG_HD static Fp gcd_start() {
    Fp r;
    r.v[0] = C::gcd0; r.v[1] = C::gcd1; r.v[2] = C::gcd2; r.v[3] = C::gcd3;
    r.v[4] = C::gcd4; r.v[5] = C::gcd5; r.v[6] = C::gcd6; r.v[7] = C::gcd7;
    return r;
  }
  // 15 division steps, K done before them on these words: x and y are 2^K times
  // their values (mod 2^32). (u, v) and (q, r) receive the rows of
  // 2^15 f' = u f + v g, 2^15 g' = q f + r g. The first row is kept undoubled by
  // the last step, so |u|, |v| <= 2^14 fit their half words; |q| + |r| <= 2^15,
  // and neither is 2^15 alone (u and v are even, the determinant is 2^15).
  template <int K>
  ZG_HD static void gcd_steps(uint32_t& x, uint32_t& y, int32_t& nd2, int32_t& u, int32_t& v, int32_t& q, int32_t& r) {
    uint32_t U = 1u, Q = 1u << 16;
#pragma unroll
    for (int k = K; k < K + 15; ++k) {
      gcd_step(x, y, U, Q, nd2, k);
      if (k < K + 14) U <<= 1;
    }
    u = (int16_t)U;
    v = (int32_t)(U - (uint32_t)u) >> 16;
    q = (int16_t)Q;
    r = (int32_t)(Q - (uint32_t)q) >> 16;
    u *= 2;
    v *= 2;
  }
  // one division step on bit k of y: (x, y) and, alike, the matrix rows (U, Q);
  // nd2 = -2 delta. Predicated: what a lone warp waits for is the chain of
  // instructions from one tested bit to the next.
  ZG_HD static void gcd_step(uint32_t& x, uint32_t& y, uint32_t& U, uint32_t& Q, int32_t& nd2, int k) {
#ifdef __CUDA_ARCH__
    asm("{\n\t.reg .pred o, s, n;\n\t.reg .b32 t;\n\t"
        "and.b32 t, %1, %5;\n\t"
        "setp.ne.u32 o, t, 0;\n\t"
        "setp.lt.and.s32 s|n, %4, 0, o;\n\t"
        "@s sub.u32 %1, %1, %0;\n\t"
        "@n add.u32 %1, %1, %0;\n\t"
        "@s neg.s32 %4, %4;\n\t"
        "@s sub.u32 %3, %3, %2;\n\t"
        "@n add.u32 %3, %3, %2;\n\t"
        "@s add.u32 %0, %0, %1;\n\t"
        "@s add.u32 %2, %2, %3;\n\t"
        "add.s32 %4, %4, -2;\n\t"
        "shl.b32 %0, %0, 1;\n\t}"
        : "+r"(x), "+r"(y), "+r"(U), "+r"(Q), "+r"(nd2)
        : "r"(1u << k));
#else
    const bool odd = (y >> k & 1u) != 0, swap = odd && nd2 < 0;
    if (odd) {
      y = swap ? y - x : y + x;
      Q = swap ? Q - U : Q + U;
    }
    if (swap) {  // x = the old y
      x += y;
      U += Q;
      nd2 = -nd2;
    }
    nd2 -= 2;
    x <<= 1;
#endif
  }
  // a, b = (u a + v b) / 2^30, (q a + r b) / 2^30 in signed 30-bit limbs (limbs 0
  // to 7 in [0, 2^30)), mod p (a multiple of p below 2^29 p makes the division
  // exact) or exact already
  template <bool MOD>
  ZG_HD static void gcd_rows(int32_t* a, int32_t* b, int32_t u, int32_t v, int32_t q, int32_t r) {
    constexpr int32_t M30 = (1 << 30) - 1;
    int32_t p[9], ka = 0, kb = 0;
    limbs30(modulus(), p);
    int64_t ca = (int64_t)u * a[0] + (int64_t)v * b[0], cb = (int64_t)q * a[0] + (int64_t)r * b[0];
    if (MOD) {
      ka = (int32_t)((uint32_t)ca * C::inv << 2) >> 2;
      kb = (int32_t)((uint32_t)cb * C::inv << 2) >> 2;
      ca += (int64_t)ka * p[0];
      cb += (int64_t)kb * p[0];
    }
    ca >>= 30;
    cb >>= 30;
#pragma unroll
    for (int i = 1; i < 9; ++i) {
      ca += (int64_t)u * a[i] + (int64_t)v * b[i];
      cb += (int64_t)q * a[i] + (int64_t)r * b[i];
      if (MOD) {
        ca += (int64_t)ka * p[i];
        cb += (int64_t)kb * p[i];
      }
      a[i - 1] = (int32_t)ca & M30;
      b[i - 1] = (int32_t)cb & M30;
      ca >>= 30;
      cb >>= 30;
    }
    a[8] = (int32_t)ca;
    b[8] = (int32_t)cb;
  }
  // signed 30-bit limbs of a value below 2^256 in absolute terms, p added if
  // it is negative
  ZG_HD static Fp from_limbs30(const int32_t* l) {
    Fp t, s;
#pragma unroll
    for (int i = 0; i < 8; ++i) t.v[i] = (uint32_t)l[i] >> (2 * i) | (uint32_t)l[i + 1] << (30 - 2 * i);
    add_raw(s, t, modulus());
    return l[8] < 0 ? s : t;
  }
  ZG_HD static void limbs30(const Fp& a, int32_t* l) {
#pragma unroll
    for (int i = 0; i < 9; ++i) {
      const int o = 30 * i, w = o >> 5, s = o & 31;
      uint32_t x = a.v[w] >> s;
      if (s > 2 && w + 1 < 8) x |= a.v[w + 1] << (32 - s);
      l[i] = (int32_t)(x & ((1u << 30) - 1));
    }
  }
  // canonical value > (p-1)/2, i.e. ark's "y > -y" (SWFlags::YIsNegative)
  ZG_HD bool canonical_is_negative() const {
    Fp c = to_canonical();
    Fp d = neg(c);  // canonical of -y as integer
    // compare c > d as integers
    for (int i = 7; i >= 0; --i)
      if (c.v[i] != d.v[i]) return c.v[i] > d.v[i];
    return false;
  }
};

typedef Fp<FqCfg> Fq;
typedef Fp<FrCfg> Fr;

}  // namespace zg
