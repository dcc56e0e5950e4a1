// Fp::inverse on the host path against a^(p - 2), Fq and Fr: edge operands,
// every power of two and its negative, and random ones.
#include <cstdio>
#include <random>

#include "cuda_threads.hpp"
#include "../../0g-da-encoder_b200/csrc/zg_field.cuh"
using namespace zg;

template <class F>
int check(const char* name) {
  std::mt19937_64 rng(17);
  const F p = F::modulus();
  std::vector<F> v;
  auto small = [](uint32_t x) {
    F r = F::zero();
    r.v[0] = x;
    return r;
  };
  for (uint32_t x = 0; x < 40; ++x) v.push_back(small(x));
  for (int k = 0; k < 254; ++k) {
    F x = F::zero();
    x.v[k / 32] = 1u << (k % 32);
    F d;
    if (F::sub_raw(d, x, p)) v.push_back(x);
  }
  for (int i = 0; i < 3000; ++i) {
    F x, d;
    for (int k = 0; k < 8; ++k) x.v[k] = (uint32_t)rng();
    x.v[7] &= i % 2 ? 0x3fffffffu : 0xfu;
    if (F::sub_raw(d, x, p)) v.push_back(x);
  }
  for (size_t i = v.size(); i-- > 0;) v.push_back(-v[i]);
  F e;  // p - 2
  F::sub_raw(e, p, small(2));
  int bad = 0;
  for (const F& x : v) {
    const F got = x.inverse();
    F d;
    if (got != x.pow(e.v, 8) || !F::sub_raw(d, got, p)) ++bad;
    if (!x.is_zero() && got * x != F::one()) ++bad;
  }
  printf("%s: %d wrong of %zu\n", name, bad, v.size());
  return bad;
}

int main() { return check<Fq>("Fq") + check<Fr>("Fr") != 0; }
