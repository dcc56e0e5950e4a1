// G1 additions by four lanes, for the places where a few points are added one
// after another and the latency of a point addition counts (AMT trees, the
// combine of few items, sums of partial results).
//
// Lane q = lane mod 4 of a quad holds one XYZZ coordinate of a point (X, Y,
// ZZ, ZZZ). The 14 products of an addition (add-2008-s) are four levels of
// independent products, one per lane and level; the operands between levels
// go through warp shuffles. One addition takes the latency of 4 products
// (about 2 us for a lone warp) instead of 7 pairs (5.5 us), in 16 product
// slots for 14. A doubling takes three levels. All 32 lanes of a warp call
// together.
#pragma once
#include "zg_curve.cuh"

namespace zg {

__device__ __forceinline__ Fq quad_get(const Fq& a, int q) {
  Fq r;
  const int src = (int)(threadIdx.x & 28u) | q;
#pragma unroll
  for (int i = 0; i < 8; ++i) r.v[i] = __shfl_sync(0xffffffffu, a.v[i], src);
  return r;
}
__device__ __forceinline__ Fq lane_xor(const Fq& a, int m) {
  Fq r;
#pragma unroll
  for (int i = 0; i < 8; ++i) r.v[i] = __shfl_xor_sync(0xffffffffu, a.v[i], m);
  return r;
}
// the coordinate of the point `delta` quads further up (its own past the end)
__device__ __forceinline__ Fq quad_down(const Fq& a, int delta) {
  Fq r;
#pragma unroll
  for (int i = 0; i < 8; ++i) r.v[i] = __shfl_down_sync(0xffffffffu, a.v[i], 4 * delta);
  return r;
}
__device__ __forceinline__ Fq quad_sel(bool c, const Fq& a, const Fq& b) {
  Fq r;
#pragma unroll
  for (int i = 0; i < 8; ++i) r.v[i] = c ? a.v[i] : b.v[i];
  return r;
}
// this lane's coordinate of infinity
__device__ __forceinline__ Fq quad_inf() { return (threadIdx.x & 3u) < 2 ? Fq::one() : Fq::zero(); }

// this lane's coordinate of a + b by the one-lane formulas (equal or opposite
// points)
static __device__ __noinline__ Fq quad_add_full(const Fq a, const Fq b) {
  XYZZ p, o;
  p.X = quad_get(a, 0); p.Y = quad_get(a, 1); p.ZZ = quad_get(a, 2); p.ZZZ = quad_get(a, 3);
  o.X = quad_get(b, 0); o.Y = quad_get(b, 1); o.ZZ = quad_get(b, 2); o.ZZZ = quad_get(b, 3);
  p.add(o);
  const uint32_t q = threadIdx.x & 3u;
  return q == 0 ? p.X : q == 1 ? p.Y : q == 2 ? p.ZZ : p.ZZZ;
}

// a + b
static __device__ __noinline__ Fq quad_add(const Fq a, const Fq b) {
  const uint32_t q = threadIdx.x & 3u;
  const bool lo = q < 2;
  const bool a_inf = __shfl_sync(0xffffffffu, (int)a.is_zero(), (int)(threadIdx.x & 28u) | 2) != 0;
  const bool b_inf = __shfl_sync(0xffffffffu, (int)b.is_zero(), (int)(threadIdx.x & 28u) | 2) != 0;
  // U1, S1, U2, S2
  const Fq t1 = Fq::mul(a, lane_xor(b, 2));
  const Fq t1x = lane_xor(t1, 2);
  const Fq d = quad_sel(lo, t1x, t1) - quad_sel(lo, t1, t1x);  // P in lanes 0 and 2, R in lanes 1 and 3
  const bool same = __shfl_sync(0xffffffffu, (int)d.is_zero(), (int)(threadIdx.x & 28u)) != 0;
  // PP, R^2, ZZ1 ZZ2, ZZZ1 ZZZ2
  const Fq t2 = Fq::mul(quad_sel(lo, d, a), quad_sel(lo, d, b));
  const Fq pp = quad_get(t2, 0);
  // PPP, Q, ZZ3, -
  const Fq u1 = quad_get(t1, 0);
  const Fq t3 = Fq::mul(quad_sel(q == 0, d, quad_sel(q == 1, u1, t2)), pp);
  const Fq ppp = quad_get(t3, 0), Q = quad_get(t3, 1);
  const Fq x3 = quad_get(t2, 1) - ppp - (Q + Q);
  const Fq r = quad_get(d, 1);
  // -, S1 PPP, R (Q - X3), ZZZ3
  const Fq t4 = Fq::mul(quad_sel(q == 2, r, quad_sel(q == 1, t1, t2)), quad_sel(q == 2, Q - x3, ppp));
  const Fq y = quad_get(t4, 2) - t4;
  Fq out = quad_sel(q == 0, x3, quad_sel(q == 1, y, quad_sel(q == 2, t3, t4)));
  const bool special = same && !a_inf && !b_inf;
  if (__any_sync(0xffffffffu, special)) {
    const Fq f = quad_add_full(a, b);
    out = quad_sel(special, f, out);
  }
  return quad_sel(b_inf, a, quad_sel(a_inf, b, out));
}

// 2 a
static __device__ __noinline__ Fq quad_dbl(const Fq a) {
  const uint32_t q = threadIdx.x & 3u;
  const Fq a2 = a + a;
  // X^2, V = U^2 (U = 2Y), -, -
  const Fq t1 = Fq::mul(quad_sel(q == 1, a2, a), quad_sel(q == 1, a2, a));
  const Fq v = quad_get(t1, 1), xx = quad_get(t1, 0);
  const Fq m = xx + xx + xx;
  // S = X V, W = U V, ZZ3, M^2
  const Fq t2 = Fq::mul(quad_sel(q == 3, m, quad_sel(q == 1, a2, a)), quad_sel(q == 3, m, v));
  const Fq s = quad_get(t2, 0), w = quad_get(t2, 1);
  const Fq x3 = quad_get(t2, 3) - (s + s);
  // M (S - X3), W Y, -, ZZZ3
  const Fq t3 = Fq::mul(quad_sel(q == 0, m, w), quad_sel(q == 0, s - x3, a));
  const Fq y = quad_get(t3, 0) - t3;
  return quad_sel(q == 0, x3, quad_sel(q == 1, y, quad_sel(q == 2, t2, t3)));
}

// this lane's coordinate of a point in memory
__device__ __forceinline__ Fq quad_load(const XYZZ* p) {
  const uint4* s = reinterpret_cast<const uint4*>(p) + 2 * (threadIdx.x & 3u);
  const uint4 a = s[0], b = s[1];
  Fq r;
  r.v[0] = a.x; r.v[1] = a.y; r.v[2] = a.z; r.v[3] = a.w;
  r.v[4] = b.x; r.v[5] = b.y; r.v[6] = b.z; r.v[7] = b.w;
  return r;
}
__device__ __forceinline__ void quad_store(XYZZ* p, const Fq& c) {
  uint4* d = reinterpret_cast<uint4*>(p) + 2 * (threadIdx.x & 3u);
  d[0] = make_uint4(c.v[0], c.v[1], c.v[2], c.v[3]);
  d[1] = make_uint4(c.v[4], c.v[5], c.v[6], c.v[7]);
}
// an affine point, (0, 0) standing for infinity
__device__ __forceinline__ Fq quad_load_aff(const G1Aff* p) {
  const uint32_t q = threadIdx.x & 3u;
  const uint4* s = reinterpret_cast<const uint4*>(p) + 2 * (q & 1);
  const uint4 a = s[0], b = s[1];
  Fq r;
  r.v[0] = a.x; r.v[1] = a.y; r.v[2] = a.z; r.v[3] = a.w;
  r.v[4] = b.x; r.v[5] = b.y; r.v[6] = b.z; r.v[7] = b.w;
  const unsigned zero = __ballot_sync(0xffffffffu, r.is_zero());
  const bool inf = ((zero >> (threadIdx.x & 28u)) & 3u) == 3u;
  return inf ? quad_inf() : q < 2 ? r : Fq::one();
}
// the sum over the warp's eight quads, in every quad
__device__ __forceinline__ Fq quad_warp_sum(Fq c) {
#pragma unroll 1
  for (int m = 4; m < 32; m <<= 1) c = quad_add(c, lane_xor(c, m));
  return c;
}

}  // namespace zg
