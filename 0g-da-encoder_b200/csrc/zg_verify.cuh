// Device kernels of batched slice verification (zg_verify_slices).
//
// The reference checks one EncodedSlice at a time (EncodedSlice::verify,
// crates/encoder/src/encoder/slice.rs:73-95): a Merkle path
// (merkle/slice.rs:50-104) and an AMT proof of 10 KZG pairing equalities, one
// MSM consistency check and one low-degree pairing test
// (crates/amt/src/verify_params.rs:136-211); its DeferredVerifier
// (deferred_verification.rs:67-146) folds many such checks into random linear
// combinations. Here a whole batch of slices is checked at once:
//  * Merkle paths: one CTA per slice (k_verify_merkle);
//  * MSM checks: sum_i alpha_i (sum_t basis[bi C + t] data_i[t]) over all
//    slices of a coset is ONE MSM over the coset's basis line (scalars
//    alpha_i data_i[t] scattered by k_verify_scalars), run on the context's
//    fixed-base tables;
//  * pairing checks: e(L, g2) prod_g e(-G_g, V_g) prod_c e(-H_c, high_g2_c) = 1
//    with L, G_g, H_c random-weighted G1 sums (k_g1_mul_glv + segment
//    sums), one Miller loop per distinct G2 point (k_miller) and one final
//    exponentiation on the host.
#pragma once
#include "zg_pairing.cuh"
#include "zg_quad.cuh"

namespace zg {

// The curve endomorphism phi(x, y) = (beta x, y) = lambda (x, y), beta^3 = 1 in
// Fq and lambda^3 = 1 in Fr. The random coefficients of the combinations are
// k1 + lambda k2 with k1, k2 of 64 bits: 2^128 different values (no vector of
// the lattice a + lambda b = 0 mod r is that short), and s P takes 64
// doublings and a joint addition of P, phi(P) or P + phi(P) =
// -phi^2(P) = (beta^2 x, -y) per bit, against 128 doublings and 64 additions.
__device__ __forceinline__ Fq glv_beta(int k) {  // beta^k, k = 1, 2 (Montgomery form)
  constexpr uint32_t b1[8] = {0xd782e155u, 0x71930c11u, 0xffbe3323u, 0xa6bb947cu,
                              0xd4741444u, 0xaa303344u, 0x26594943u, 0x2c3b3f0du};
  constexpr uint32_t b2[8] = {0x13e80b9cu, 0x3350c88eu, 0xdb5e56b9u, 0x7dce557cu,
                              0xb615564au, 0x6001b4b8u, 0x020217e0u, 0x2682e617u};
  Fq r;
#pragma unroll
  for (int i = 0; i < 8; ++i) r.v[i] = k == 1 ? b1[i] : b2[i];
  return r;
}
// out[i] = (k1 + lambda k2) P_i for affine P_i (inf[i] != 0: infinity), k1 and
// k2 the two 64-bit halves of the four little-endian words at sc + 4 i
__global__ void __launch_bounds__(128) k_g1_mul_glv(const G1Aff* __restrict__ pts, const uint8_t* __restrict__ inf,
                                                    const uint32_t* __restrict__ sc, XYZZ* __restrict__ out,
                                                    uint32_t n) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  XYZZ acc = XYZZ::inf();
  if (!inf[i]) {
    const G1Aff p = pts[i];
    const Fq x1 = Fq::mul(p.x, glv_beta(1)), x2 = Fq::mul(p.x, glv_beta(2)), yn = -p.y;
    const uint4 w = reinterpret_cast<const uint4*>(sc)[i];
    uint64_t k1 = (uint64_t)w.y << 32 | w.x, k2 = (uint64_t)w.w << 32 | w.z;
#pragma unroll 1
    for (int b = 0; b < 64; ++b, k1 <<= 1, k2 <<= 1) {
      acc = acc.dbl();
      const bool s1 = (int64_t)k1 < 0, s2 = (int64_t)k2 < 0;
      if (s1 || s2) acc.add_affine(s1 ? (s2 ? x2 : p.x) : x1, s1 && s2 ? yn : p.y);
    }
  }
  store_xyzz(out + i, acc);
}
// out[i] = (k1 + lambda k2) sum_{d < m} P_{i stride + d}, k1 and k2 of nw words
// at sc + 2 nw i; one quad per i (zg_quad.cuh)
__global__ void __launch_bounds__(128) k_g1_mul_sum(const G1Aff* __restrict__ pts, const uint8_t* __restrict__ inf,
                                                    uint32_t m, uint32_t stride, const uint32_t* __restrict__ sc,
                                                    int nw, XYZZ* __restrict__ out, uint32_t n) {
  const uint32_t at = (blockIdx.x * blockDim.x + threadIdx.x) / 4, i = min(at, n - 1), q = threadIdx.x & 3;
  Fq p = quad_inf();
#pragma unroll 1
  for (uint32_t d = 0; d < m; ++d) {
    const Fq x = quad_load_aff(pts + (size_t)i * stride + d);
    p = quad_add(p, quad_sel(inf[(size_t)i * stride + d] != 0, quad_inf(), x));
  }
  const Fq p1 = q == 0 ? Fq::mul(p, glv_beta(1)) : p;
  const Fq p2 = q == 0 ? Fq::mul(p, glv_beta(2)) : q == 1 ? -p : p;
  const uint32_t *k1 = sc + (size_t)i * 2 * nw, *k2 = k1 + nw;
  Fq acc = quad_inf();
#pragma unroll 1
  for (int b = 32 * nw - 1; b >= 0; --b) {
    acc = quad_dbl(acc);
    const bool s1 = (k1[b >> 5] >> (b & 31)) & 1, s2 = (k2[b >> 5] >> (b & 31)) & 1;
    acc = quad_add(acc, quad_sel(s1, quad_sel(s2, p2, p), quad_sel(s2, p1, quad_inf())));
  }
  if (at < n) quad_store(out + i, acc);
}

// out[g] = sum of terms[k] for k in [off[g], off[g + 1]), one warp per segment
// (eight quads, then their sum): segments run from one term to half the slices
__global__ void __launch_bounds__(128) k_seg_sum(const XYZZ* __restrict__ terms, const uint32_t* __restrict__ off,
                                                 XYZZ* __restrict__ out, uint32_t nseg) {
  const uint32_t g = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (g >= nseg) return;  // uniform per warp
  Fq acc = quad_inf();
#pragma unroll 1
  for (uint32_t k0 = off[g]; k0 < off[g + 1]; k0 += 8) {
    const uint32_t k = k0 + (threadIdx.x & 31) / 4;
    acc = quad_add(acc, k < off[g + 1] ? quad_load(terms + k) : quad_inf());
  }
  acc = quad_warp_sum(acc);
  if ((threadIdx.x & 31) < 4) quad_store(out + g, acc);
}

// Miller inputs: affine (negated when neg[j]) G1 points with infinity flags
__global__ void __launch_bounds__(128) k_pairing_inputs(const XYZZ* __restrict__ in, const uint8_t* __restrict__ neg,
                                                        G1Aff* __restrict__ out, uint8_t* __restrict__ inf, uint32_t n) {
  const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n) return;
  G1Aff a;
  const bool ok = in[j].to_affine(a);
  if (ok && neg[j]) a.y = -a.y;
  if (!ok) { a.x = Fq::zero(); a.y = Fq::zero(); }
  out[j] = a;
  inf[j] = ok ? 0 : 1;
}

// Miller loops by two lanes: lane h = lane mod 2 holds the Fq6 half c_h of
// f = c0 + c1 w, so a square is one Fq6 product per lane and a line product
// one half of the result. All 32 lanes call together.
__device__ __forceinline__ Fq6 pair_other(const Fq6& a) {
  Fq6 r;
  r.c0 = Fq2{lane_xor(a.c0.c0, 1), lane_xor(a.c0.c1, 1)};
  r.c1 = Fq2{lane_xor(a.c1.c0, 1), lane_xor(a.c1.c1, 1)};
  r.c2 = Fq2{lane_xor(a.c2.c0, 1), lane_xor(a.c2.c1, 1)};
  return r;
}
__device__ __forceinline__ Fq6 fq6_sel(bool c, const Fq6& a, const Fq6& b) {
  Fq6 r;
  r.c0 = Fq2{quad_sel(c, a.c0.c0, b.c0.c0), quad_sel(c, a.c0.c1, b.c0.c1)};
  r.c1 = Fq2{quad_sel(c, a.c1.c0, b.c1.c0), quad_sel(c, a.c1.c1, b.c1.c1)};
  r.c2 = Fq2{quad_sel(c, a.c2.c0, b.c2.c0), quad_sel(c, a.c2.c1, b.c2.c1)};
  return r;
}
static __device__ __noinline__ Fq6 fq6_mul_ool(const Fq6 a, const Fq6 b) { return a * b; }
// f^2: lane 0 forms m = c0 c1, lane 1 s = (c0 + c1)(c0 + v c1);
// c0' = s - m - v m, c1' = 2 m
static __device__ __noinline__ Fq6 pair_sqr(const Fq6 own) {
  const bool h = threadIdx.x & 1;
  const Fq6 oth = pair_other(own);
  // lane 0: c0, c1; lane 1: c0 + c1, c0 + v c1
  const Fq6 p = fq6_mul_ool(fq6_sel(h, own + oth, own), fq6_sel(h, oth + own.mul_v(), oth));
  const Fq6 x = pair_other(p);
  return fq6_sel(h, x + x, x - p - p.mul_v());
}
// f times the line c00 + c01 v + c11 v w: c_h L0 + (v) c_(1-h) c11 v
static __device__ __noinline__ Fq6 pair_line(const Fq6 own, const Fq c00, const Fq2 c01, const Fq2 c11) {
  const bool h = threadIdx.x & 1;
  const Fq6 u = pair_other(own).mul_bv(c11);
  return own.mul_ab(c00, c01) + fq6_sel(h, u, u.mul_v());
}

// f[j] = Miller function of (P_j, Q_j) (miller_tate), two lanes per pair: each
// half of f and, twice, the point T. 6145 pairs leave most of the GPU to
// latency: 24.6 ms with one lane per pair (Fq12 in one thread's registers and
// local memory), 13.2 so.
__global__ void __launch_bounds__(64) k_miller(const G1Aff* __restrict__ Pp, const uint8_t* __restrict__ pinf,
                                               const G2Aff* __restrict__ Qp, Fq12* __restrict__ f, uint32_t n) {
  const uint32_t at = (blockIdx.x * blockDim.x + threadIdx.x) / 2, j = min(at, n - 1);
  const bool h = threadIdx.x & 1;
  const G1Aff P = Pp[j];
  const Fq2 qx = Qp[j].x, qy = Qp[j].y;
  const bool trivial = pinf[j] || Qp[j].inf;
  const uint32_t r[8] = {FrCfg::p0, FrCfg::p1, FrCfg::p2, FrCfg::p3, FrCfg::p4, FrCfg::p5, FrCfg::p6, FrCfg::p7};
  const Fq6 unit = fq6_sel(h, Fq6::zero(), Fq6::one());
  Fq6 own = unit;
  Fq X = P.x, Y = P.y, Z = Fq::one();
#pragma unroll 1
  for (int i = 252; i >= 0; --i) {
    {  // tangent at T, times 2 Y Z^3
      const Fq A = zp_mul(X, X), B = zp_mul(Y, Y), C = zp_mul(B, B), Z2 = zp_mul(Z, Z);
      const Fq E = A + A + A;
      const Fq c00 = zp_mul(X, E) - (B + B);
      const Fq2 c01 = qx.mul_fq(-zp_mul(E, Z2));
      const Fq YZ = zp_mul(Y, Z);
      const Fq Z3 = YZ + YZ;
      const Fq2 c11 = qy.mul_fq(zp_mul(Z3, Z2));
      own = pair_line(pair_sqr(own), c00, c01, c11);
      const Fq XB = X + B;
      const Fq D0 = zp_mul(XB, XB) - A - C;
      const Fq D = D0 + D0;
      const Fq F = zp_mul(E, E);
      X = F - (D + D);
      Fq C8 = C + C;
      C8 = C8 + C8;
      C8 = C8 + C8;
      Y = zp_mul(E, D - X) - C8;
      Z = Z3;
    }
    if ((r[i >> 5] >> (i & 31)) & 1) {  // chord through T and P, times Z H
      const Fq Z2 = zp_mul(Z, Z);
      const Fq H = zp_mul(P.x, Z2) - X;
      const Fq N = zp_mul(zp_mul(P.y, Z2), Z) - Y;
      const Fq ZH = zp_mul(Z, H);
      const Fq6 g = pair_line(own, zp_mul(N, P.x) - zp_mul(ZH, P.y), qx.mul_fq(-N), qy.mul_fq(ZH));
      // T = -P (only at the last bit): the vertical line lies in Fq6
      own = fq6_sel(H.is_zero(), own, g);
      const Fq HH = zp_mul(H, H), HHH = zp_mul(H, HH), V = zp_mul(X, HH);
      X = zp_mul(N, N) - HHH - (V + V);
      Y = zp_mul(N, V - X) - zp_mul(Y, HHH);
      Z = ZH;
    }
  }
  own = fq6_sel(trivial, unit, own);
  if (at < n) (h ? f[j].c1 : f[j].c0) = own;
}

// part[b] = product of f[k] for k = 32 b + t + 32 gridDim.x s: one warp per
// CTA, each lane its own factors, then a tree in shared memory
constexpr int FQ12_PARTS = 64;
__global__ void __launch_bounds__(32) k_fq12_partial(const Fq12* __restrict__ f, uint32_t n, Fq12* __restrict__ part) {
  __shared__ Fq12 sh[32];
  Fq12 acc = Fq12::one();
  for (uint32_t k = 32 * blockIdx.x + threadIdx.x; k < n; k += 32 * gridDim.x) acc = acc * f[k];
  sh[threadIdx.x] = acc;
  __syncwarp();
#pragma unroll 1
  for (int w = 16; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w) sh[threadIdx.x] = sh[threadIdx.x] * sh[threadIdx.x + w];
    __syncwarp();
  }
  if (threadIdx.x == 0) part[blockIdx.x] = sh[0];
}

// out[i] = s_i * g2 for canonical Fr scalars (32 B little-endian each)
__global__ void __launch_bounds__(64) k_g2_mul(const uint8_t* __restrict__ sc, G2Aff g2, G2Aff* __restrict__ out,
                                               uint32_t n) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t* s = reinterpret_cast<const uint32_t*>(sc + (size_t)i * 32);
  G2Jac acc = G2Jac::inf();
  for (int w = 7; w >= 0; --w) {
    const uint32_t word = s[w];
#pragma unroll 1
    for (int b = 31; b >= 0; --b) {
      acc = acc.dbl();
      if ((word >> b) & 1) acc = acc.add_affine(g2.x, g2.y);
    }
  }
  out[i] = acc.to_affine();
}

// Byte offsets inside one serialized EncodedSlice (the layout k_slices writes):
//   0 index | 8 amt.index | 16 commitment | 80 row.index | 88 row len | 96 row
//   | proof len | LR x (commitment_d, quotient_d) | high | roots[3] | proof len
//   | LR x sibling | leaf_index | leaf
struct SliceOffsets {
  uint32_t row, proof, high, roots, mproof, leaf_index, leaf, size;
  __host__ __device__ SliceOffsets(int lr, int lc) {
    row = 96;
    proof = row + (32u << lc) + 8;
    high = proof + 128u * lr;
    roots = high + 64;
    mproof = roots + 96 + 8;
    leaf_index = mproof + 32u * lr;
    leaf = leaf_index + 8;
    size = leaf + 32;
  }
};

__device__ __forceinline__ void keccak_pair(const uint8_t* a, const uint8_t* b, uint8_t* out) {
  uint64_t in[8], h[4];
  for (int k = 0; k < 4; ++k) {
    uint64_t x = 0, y = 0;
    for (int t = 0; t < 8; ++t) {
      x |= (uint64_t)a[8 * k + t] << (8 * t);
      y |= (uint64_t)b[8 * k + t] << (8 * t);
    }
    in[k] = x;
    in[4 + k] = y;
  }
  keccak256_64(in, h);
  for (int k = 0; k < 4; ++k)
    for (int t = 0; t < 8; ++t) out[8 * k + t] = (uint8_t)(h[k] >> (8 * t));
}

// Merkle part of EncodedSlice::verify (merkle/slice.rs:50-104) in the
// reference's order: file root of the slice's roots, leaf index range, the
// row's local root against the leaf, the sibling path against
// roots[leaf_index / R]. Slice j of the batch starts at slices + j * stride
// (16-byte aligned) with the standard layout up to its Merkle proof, whose
// length is nproof[j]. One CTA of 128 threads per slice.
__global__ void __launch_bounds__(128) k_verify_merkle(const uint8_t* __restrict__ slices, uint64_t stride, int lr,
                                                       int lc, const uint32_t* __restrict__ nproof,
                                                       const uint8_t* __restrict__ auth_root,
                                                       int32_t* __restrict__ code) {
  __shared__ __align__(16) uint8_t nodes[2][128 * 32];
  __shared__ int bad_root;
  const SliceOffsets L(lr, lc);
  const uint8_t* s = slices + (uint64_t)blockIdx.x * stride;
  const uint32_t np = nproof[blockIdx.x];  // sibling count (LR in a well-formed slice)
  const uint32_t li_off = L.mproof + 32 * np;
  const uint32_t C = 1u << lc, R = 1u << lr;
  const uint32_t nleaf = C / 8;  // <= 128
  if (threadIdx.x == 0) {
    uint8_t h01[32], fr[32];
    keccak_pair(s + L.roots, s + L.roots + 32, h01);
    keccak_pair(h01, s + L.roots + 64, fr);
    int bad = 0;
    for (int k = 0; k < 32; ++k) bad |= fr[k] != auth_root[k];
    bad_root = bad;
  }
  // leaves: keccak256 of 8 consecutive 32-byte items of the row
  for (uint32_t j = threadIdx.x; j < nleaf; j += blockDim.x) {
    const uint64_t* src = reinterpret_cast<const uint64_t*>(s + L.row + (size_t)j * 256);
    uint64_t h[4];
    keccak256_256([&](int k) { return make_ulonglong2(src[2 * k], src[2 * k + 1]); }, h);
    uint64_t* d = reinterpret_cast<uint64_t*>(nodes[0] + 32 * j);
    for (int k = 0; k < 4; ++k) d[k] = h[k];
  }
  __syncthreads();
  int cur = 0;
  for (uint32_t cnt = nleaf; cnt > 1; cnt >>= 1) {
    for (uint32_t j = threadIdx.x; j < cnt / 2; j += blockDim.x)
      keccak_pair(nodes[cur] + 64 * j, nodes[cur] + 64 * j + 32, nodes[cur ^ 1] + 32 * j);
    __syncthreads();
    cur ^= 1;
  }
  if (threadIdx.x != 0) return;
  int32_t c = 0;
  uint64_t li = 0;
  for (int t = 0; t < 8; ++t) li |= (uint64_t)s[li_off + t] << (8 * t);
  if (bad_root) c = 20;
  else if (li >= 3ull * R) c = 22;
  else {
    int diff = 0;
    for (int k = 0; k < 32; ++k) diff |= nodes[cur][k] != s[li_off + 8 + k];
    if (diff) c = 23;
    else {
      uint8_t acc[32];
      for (int k = 0; k < 32; ++k) acc[k] = s[li_off + 8 + k];
      uint64_t pos = li % R;
      for (uint32_t d = 0; d < np; ++d) {
        const uint8_t* sib = s + L.mproof + 32 * d;
        uint8_t nxt[32];
        if (pos & 1) keccak_pair(sib, acc, nxt);
        else keccak_pair(acc, sib, nxt);
        for (int k = 0; k < 32; ++k) acc[k] = nxt[k];
        pos >>= 1;
      }
      const uint8_t* root = s + L.roots + 32 * (li / R);
      int pd = 0;
      for (int k = 0; k < 32; ++k) pd |= acc[k] != root[k];
      if (pd) c = 24;
    }
  }
  code[blockIdx.x] = c;
}

// scal[coset(j)][bi(j) C + t] = alpha_j * row_j[bitrev(t)] (canonical), row_j
// the row of the slice at position pos[j] of the batch buffer: the
// scalars of the batch's MSM checks (the row is index_reverse'd, encode.rs:225-241).
// alpha in Montgomery form, so one product gives the canonical result.
__global__ void __launch_bounds__(256) k_verify_scalars(const uint8_t* __restrict__ slices, uint64_t stride,
                                                        const uint32_t* __restrict__ pos, int lc,
                                                        const uint32_t* __restrict__ coset,
                                                        const uint32_t* __restrict__ bi, const Fr* __restrict__ alpha,
                                                        uint8_t* __restrict__ scal, uint64_t coset_stride) {
  const uint32_t j = blockIdx.x;
  const uint32_t C = 1u << lc;
  const Fr* row = reinterpret_cast<const Fr*>(slices + (uint64_t)pos[j] * stride + 96);
  const Fr a = alpha[j];
  Fr* dst = reinterpret_cast<Fr*>(scal + coset[j] * coset_stride) + (size_t)bi[j] * C;
  for (uint32_t t = threadIdx.x; t < C; t += blockDim.x) dst[t] = load_fr(row + brev_bits(t, lc)) * a;
}

}  // namespace zg
