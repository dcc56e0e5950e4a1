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
// chains straddle the pairs and issue lo and hi apart. Outputs that are
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
  // 2^(40 + 512) mod p, the start of inverse()
  static constexpr uint32_t gcd0 = 0x16fe05fbu, gcd1 = 0xda94bc1bu, gcd2 = 0x51de3187u, gcd3 = 0xfdb7603bu,
                            gcd4 = 0xe1594d7eu, gcd5 = 0x5dbd35a2u, gcd6 = 0x9d0994cdu, gcd7 = 0x16579a57u;
};
struct FrCfg {
  static constexpr uint32_t p0 = 0xf0000001u, p1 = 0x43e1f593u, p2 = 0x79b97091u, p3 = 0x2833e848u,
                            p4 = 0x8181585du, p5 = 0xb85045b6u, p6 = 0xe131a029u, p7 = 0x30644e72u;
  static constexpr uint32_t inv = 0xefffffffu;
  static constexpr uint32_t r2_0 = 0xae216da7u, r2_1 = 0x1bb8e645u, r2_2 = 0xe35c59e3u, r2_3 = 0x53fe3ab1u,
                            r2_4 = 0x53bb8085u, r2_5 = 0x8c49833du, r2_6 = 0x7f4e44a5u, r2_7 = 0x0216d0b1u;
  static constexpr uint32_t one0 = 0x4ffffffbu, one1 = 0xac96341cu, one2 = 0x9f60cd29u, one3 = 0x36fc7695u,
                            one4 = 0x7879462eu, one5 = 0x666ea36fu, one6 = 0x9a07df2fu, one7 = 0x0e0a77c1u;
  static constexpr uint32_t gcd0 = 0x82bf4ec7u, gcd1 = 0x9126b014u, gcd2 = 0xf84ec615u, gcd3 = 0x89ec5f7du,
                            gcd4 = 0x2dc5f176u, gcd5 = 0xeeab1253u, gcd6 = 0xc17c9526u, gcd7 = 0x0e680cefu;
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
  // f, g (signed 30-bit limbs, an exact division by 2^30) and to d, e (mod p,
  // f = d x 2^(2k) and g = e x 2^(2k) mod p after k batches: every batch
  // divides d and e by 2^32 in one Montgomery row). 20 batches end with
  // f = +-1, g = 0, so the inverse is +-d for the start e = 2^40 R^2. A lone
  // warp takes 21 us on a B200, against 165 us for the exponentiation by p - 2
  // (380 products in a row).
  ZG_HD Fp inverse() const {
    constexpr int32_t M30 = (1 << 30) - 1;
    int32_t f[9], g[9];
    const Fp p = modulus();
    limbs30(p, f);
    limbs30(*this, g);
    Fp d = zero(), e;
    e.v[0] = C::gcd0; e.v[1] = C::gcd1; e.v[2] = C::gcd2; e.v[3] = C::gcd3;
    e.v[4] = C::gcd4; e.v[5] = C::gcd5; e.v[6] = C::gcd6; e.v[7] = C::gcd7;
    int32_t delta2 = 1;  // 2 delta
#pragma unroll 1
    for (int batch = 0; batch < 20; ++batch) {
      // rows (u, v) and (q, r): 2^30 f' = u f + v g, 2^30 g' = q f + r g
      int32_t u = 1, v = 0, q = 0, r = 1;
      uint32_t x = (uint32_t)f[0] | (uint32_t)f[1] << 30, y = (uint32_t)g[0] | (uint32_t)g[1] << 30;
#pragma unroll 6
      for (int k = 0; k < 30; ++k) {
        const bool odd = (y & 1u) != 0, swap = odd && delta2 > 0;
        const uint32_t ax = odd ? (swap ? 0u - x : x) : 0u;
        const int32_t au = odd ? (swap ? -u : u) : 0, av = odd ? (swap ? -v : v) : 0;
        if (swap) {
          x = y;
          u = q;
          v = r;
          delta2 = -delta2;
        }
        delta2 += 2;
        y = (y + ax) >> 1;
        q += au;
        r += av;
        u *= 2;
        v *= 2;
      }
      const Fp nd = raw_neg(d), ne = raw_neg(e);
      const Fp d1 = gcd_row(u < 0 ? nd : d, v < 0 ? ne : e, u, v);
      e = gcd_row(q < 0 ? nd : d, r < 0 ? ne : e, q, r);
      d = d1;
      int64_t cf = (int64_t)u * f[0] + (int64_t)v * g[0];
      int64_t cg = (int64_t)q * f[0] + (int64_t)r * g[0];
      cf >>= 30;
      cg >>= 30;
#pragma unroll
      for (int i = 1; i < 9; ++i) {
        cf += (int64_t)u * f[i] + (int64_t)v * g[i];
        cg += (int64_t)q * f[i] + (int64_t)r * g[i];
        f[i - 1] = (int32_t)cf & M30;
        g[i - 1] = (int32_t)cg & M30;
        cf >>= 30;
        cg >>= 30;
      }
      f[8] = (int32_t)cf;
      g[8] = (int32_t)cg;
    }
    return f[8] < 0 ? neg(d) : d;
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
  ZG_HD static Fp raw_neg(const Fp& a) {  // p - a for a <= p, not reduced
    Fp r;
    sub_raw(r, modulus(), a);
    return r;
  }
  // (|u| a + |v| b) / 2^32 mod p for a, b <= p and |u| + |v| <= 2^30
  ZG_HD static Fp gcd_row(const Fp& a, const Fp& b, int32_t u, int32_t v) {
    const uint32_t au = (uint32_t)(u < 0 ? -u : u), av = (uint32_t)(v < 0 ? -v : v);
    const Fp p = modulus();
    uint64_t s = (uint64_t)a.v[0] * au + (uint64_t)b.v[0] * av;
    const uint32_t k = (uint32_t)s * C::inv;
    // the low word cancels: its sum with k p_0's is 0 or 2^32
    uint64_t carry = (s >> 32) + (((uint64_t)k * p.v[0]) >> 32) + ((uint32_t)s != 0 ? 1u : 0u);
    Fp t;
#pragma unroll
    for (int i = 1; i < 8; ++i) {
      s = (uint64_t)a.v[i] * au + (uint64_t)b.v[i] * av + carry;
      const uint64_t w = (uint64_t)k * p.v[i] + (uint32_t)s;
      t.v[i - 1] = (uint32_t)w;
      carry = (s >> 32) + (w >> 32);
    }
    t.v[7] = (uint32_t)carry;
    Fp red;
    const uint32_t borrow = sub_raw(red, t, p);
    return borrow ? t : red;
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
