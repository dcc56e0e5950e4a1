// Bucket accumulation of the fixed-base MSMs with affine additions.
//
// A work item is FB_BUCKETS = 1024 buckets of (point, window, sign) entries
// (the digit sorts' output); its result is sum_k (k + 1) B_k over the bucket
// sums B_k. Additions are affine: slope = (y2 - y1) / (x2 - x1), 5 products
// and a square per addition once the divisions share one inversion
// (Montgomery's trick, 3 of the 6), against 10 for a mixed XYZZ addition. The
// price is memory: each addition reads its operands twice and keeps a prefix
// product, some 410 bytes of DRAM traffic per entry (140 for running XYZZ
// sums in registers).
// Measured on a B200, the MSM phase of a 1024 x 1024 blob (668 M additions of
// entries, 60 M of the bucket grids): 143 ms with XYZZ bucket tasks, 122 ms
// with affine additions and plain loads, 118 ms at 5 CTAs per SM, 110 ms with
// the next addition's points staged by cp.async and two items per CTA and
// turn, 107 ms without the default 128-byte fetch of each 64-byte point (DRAM
// reads 457 -> 300 bytes per entry) and with lambda and the running inverse
// as one product pair. What bounds it now is power: 980 - 1010 W of the
// board's 1000 W at 1965 MHz (820 W before), the multiply pipe 70 - 76 % busy;
// 5 CTAs per SM run 2 % lower clocks for the same time, 3 CTAs 127 ms.
#pragma once
#include "zg_curve.cuh"

namespace zg {

struct FbAccArgs {
  const G1Aff* tab = nullptr;      // [cosets][Ltot][W][tabN]
  const uint32_t* offs = nullptr;
  const uint16_t* ents = nullptr;    // chunk items
  const uint32_t* ents32 = nullptr;  // wide items (k_wd_sort's lists)
  G1Aff* out = nullptr;            // [cosets * nchunks * lines][FB_OUT] row and column sums
  int lr = 0, lc = 0, lines = 1;   // 2^lr items of each of `lines` lines per coset
  int l0 = 0, Ltot = 1;            // item line l reads table line l0 + l of Ltot per coset
  int ulog = 10;                   // wide items: sort units of 2^ulog points
  int mlog = 0;                    // wide items: 2^mlog consecutive sort units share buckets
  int W = FB_WINDOWS;              // windows per table line (wd_windows(ulog) for wide items)
  uint64_t tabN = 0;               // points per window table (the param line length)
  int group = 1;                   // items per CTA and turn
};

// One launch covers up to FB_MAX_SETS item sets (a blob's chunk items and its
// wide classes, for up to FB_MAX_BLOBS blobs whose MSMs share the launch):
// set k holds items start[k] .. start[k + 1] - 1, described by a[k] with
// local item index u - start[k]. One launch keeps the persistent CTAs busy to
// the end of the whole MSM instead of leaving a partial last round per set. A
// CTA takes its next item from the counter *next (zero at launch): items
// differ in size (a wide unit's block 0 holds the top window's small
// digits), and a fixed item-to-CTA map would give some CTAs every heavy item.
constexpr int FB_MAX_BLOBS = 2;  // blobs per fused MSM launch
constexpr int FB_MAX_SETS = 8 * FB_MAX_BLOBS;
struct FbAccPlan {
  int n = 0;
  uint32_t start[FB_MAX_SETS + 1] = {};
  FbAccArgs a[FB_MAX_SETS];
};

// Task size, a tuning choice within [FB_TASK_MIN, FB_TASK_MAX]: a batch gives
// each thread at most 3/2 of it in additions per shared inversion (96 at the
// default: MSM 109.2 ms against 111.0 at 64 and 113 at 48). The prefix
// products of a batch take 32 bytes each of the CTA's scratch, sized for the
// largest.
constexpr int FB_TASK_MIN = 32;
constexpr int FB_TASK_MAX = 96;
constexpr int FB_TASK_DEFAULT = 64;
__host__ __device__ constexpr uint32_t fb_batch(uint32_t task) { return task * 3 / 2; }

// The grid that reduces an item's buckets: bucket k = 32 a + b, row sums
// R_a = sum_b B_k and column sums C_b = sum_a B_k; sum_k (k + 1) B_k =
// 32 sum_a a R_a + sum_b (b + 1) C_b. FB_OUT points per item: 32 rows, then
// 32 columns.
constexpr int FB_GRID = 32;
constexpr int FB_OUT = 2 * FB_GRID;
static_assert(FB_GRID * FB_GRID == FB_BUCKETS, "buckets fill the grid");

// A CTA works on up to FB_GROUP items of a set at a time (FbAccArgs::group): the
// levels of their trees run together, so the short levels share their
// inversions.
constexpr int FB_GROUP = 4;
// A level's list is written by the threads that own the buckets, but runs of
// FB_RUN_PAIRS additions or more of one bucket by the whole CTA, up to
// FB_RUNS_MAX a level (the owner lists what is beyond): equal digits put
// thousands of entries into one bucket. A 128 x 1024 blob of one byte repeated
// (all digits of all windows equal) takes 46 ms, 97 listed by the owners, of
// one element repeated 15.5 and 19.4 ms; a 1024 x 1024 one 144 and 206, 111 and
// 126 ms. Lines of 32 to 160 pairs time alike.
constexpr uint32_t FB_RUN_PAIRS = 64;
constexpr uint32_t FB_RUNS_MAX = 192;
// Scratch of `ctas` CTAs, for turns of up to `group` items and segments of at
// most `cap` entries, in five blocks (GAP bytes that nothing touches after each).
struct FbScratch {
  uint8_t* base = nullptr;
  uint32_t cap = 0;
  uint32_t group = FB_GROUP;
  uint32_t ctas = 0;
  static constexpr size_t GAP = 16;
  // level-1 sums of a segment: half its entries, an odd one per bucket and sort
  // unit (half a slot each), and a carried sum
  __host__ __device__ uint32_t slots() const { return cap / 2 + group * FB_BUCKETS + 1; }
  // additions per thread and batch: of the longest level (level 1, or the grid's
  // FB_BUCKETS per item)
  __host__ __device__ uint32_t batch() const {
    const uint32_t most = (max2(cap / 2, group * FB_BUCKETS) + FB_ACC_THREADS - 1) / FB_ACC_THREADS;
    return most < fb_batch(FB_TASK_MAX) ? most : fb_batch(FB_TASK_MAX);
  }
  __host__ __device__ size_t off_fin() const { return after(0, (size_t)slots() * sizeof(G1Aff)); }
  __host__ __device__ size_t off_pre() const { return after(off_fin(), (size_t)group * FB_BUCKETS * sizeof(G1Aff)); }
  __host__ __device__ size_t off_list() const { return after(off_pre(), (size_t)batch() * FB_ACC_THREADS * sizeof(Fq)); }
  __host__ __device__ size_t off_dst() const { return after(off_list(), (size_t)(cap / 2) * sizeof(uint2)); }
  // a bucket's slots pair up to at most half of the segment's entries and carry
  __host__ __device__ size_t bytes() const {
    return (after(off_dst(), ((size_t)cap / 2 + 1) * sizeof(uint32_t)) + 255) / 256 * 256;
  }

 private:
  __host__ __device__ static uint32_t max2(uint32_t a, uint32_t b) { return a > b ? a : b; }
  __host__ __device__ static size_t after(size_t at, size_t n) { return (at + n + GAP + 15) / 16 * 16; }
};
// Largest segment: two blocks of 2^16-point units (32 768 entries, half as many
// again in a block 0), four chunks of 1024 points.
constexpr uint32_t FB_CAP_MAX = 98304;
static_assert(FB_CAP_MAX / 2 + FB_GROUP * FB_BUCKETS + 1 < 65536, "slot indexes fit 16 bits");

__device__ __forceinline__ Fq ld_fq(const Fq* p) {
  const uint4* q = reinterpret_cast<const uint4*>(p);
  const uint4 a = q[0], b = q[1];
  Fq r;
  r.v[0] = a.x; r.v[1] = a.y; r.v[2] = a.z; r.v[3] = a.w;
  r.v[4] = b.x; r.v[5] = b.y; r.v[6] = b.z; r.v[7] = b.w;
  return r;
}
__device__ __forceinline__ G1Aff ld_aff(const G1Aff* p) {
  G1Aff r;
  r.x = ld_fq(&p->x);
  r.y = ld_fq(&p->y);
  return r;
}
__device__ __forceinline__ void st_fq(Fq* p, const Fq& x) {
  uint4* q = reinterpret_cast<uint4*>(p);
  q[0] = make_uint4(x.v[0], x.v[1], x.v[2], x.v[3]);
  q[1] = make_uint4(x.v[4], x.v[5], x.v[6], x.v[7]);
}
__device__ __forceinline__ void st_aff(G1Aff* p, const G1Aff& a) {
  st_fq(&p->x, a.x);
  st_fq(&p->y, a.y);
}
// affine infinity is (0, 0), which is not on the curve
__device__ __forceinline__ bool aff_is_inf(const G1Aff& a) { return a.x.is_zero() && a.y.is_zero(); }
__device__ __forceinline__ G1Aff aff_inf() { return G1Aff{Fq::zero(), Fq::zero()}; }

// The cases the slope formula does not cover, taken when x1 = x2 or an x is 0:
// the slope's numerator and (nonzero) denominator, and what the sum is
struct AffCase {
  Fq num, den;
  int sum;  // 0: by the slope; 1: the first point; 2: the second; 3: infinity
};
static __device__ __noinline__ AffCase aff_case(const G1Aff a, const G1Aff b) {
  AffCase r;
  r.num = Fq::zero();
  r.den = Fq::one();
  r.sum = 0;
  if (aff_is_inf(b)) {
    r.sum = 1;
  } else if (aff_is_inf(a)) {
    r.sum = 2;
  } else if (a.x != b.x) {
    r.num = b.y - a.y;
    r.den = b.x - a.x;
  } else if (a.y == b.y) {  // doubling (no point of this curve has y = 0)
    const Fq xx = a.x * a.x;
    r.num = xx + xx + xx;
    r.den = a.y + a.y;
  } else {
    r.sum = 3;
  }
  return r;
}

#ifdef __CUDACC__
__device__ __forceinline__ Fq fq_lane_xor(const Fq& x, int d) {
  Fq r;
#pragma unroll
  for (int i = 0; i < 8; ++i) r.v[i] = __shfl_xor_sync(0xffffffffu, x.v[i], d);
  return r;
}
// the inverse of each lane's c (a whole warp calls): one inversion per quad of
// the four lanes' product, four products in a row more
template <class M>
__device__ __forceinline__ Fq warp_inverse(const Fq& c) {
  const Fq c1 = fq_lane_xor(c, 1), p = M::mul(c, c1), p2 = fq_lane_xor(p, 2);
  return M::mul(M::mul(Fq::inverse_quad(M::mul(p, p2)), p2), c1);
}
#else
template <class M>
Fq warp_inverse(const Fq& c) {
  return c.inverse();
}
#endif

// Inverts every thread's v (nonzero): the threads' values are multiplied into
// 32 products that one warp inverts, `turn` picking the warp. Where a launch
// has few items, these inversions are its time.
template <class M>
__device__ __forceinline__ Fq block_inverse(const Fq& v, Fq* sp, uint32_t turn) {
  constexpr int N = FB_ACC_THREADS / 32;
  sp[threadIdx.x] = v;
  __syncthreads();
  if (threadIdx.x / 32 == turn % N) {
    const uint32_t lane = threadIdx.x % 32;
    Fq c[N];
    c[0] = sp[lane];
#pragma unroll
    for (int i = 1; i < N; ++i) c[i] = M::mul(c[i - 1], sp[lane + 32 * i]);
    Fq inv = warp_inverse<M>(c[N - 1]);
#pragma unroll
    for (int i = N - 1; i >= 1; --i) {
      const Fq x = sp[lane + 32 * i];
      sp[lane + 32 * i] = M::mul(inv, c[i - 1]);
      inv = M::mul(inv, x);
    }
    sp[lane] = inv;
  }
  __syncthreads();
  return sp[threadIdx.x];
}

// exclusive scan over the CTA of two 16-bit counts packed in a word (sums
// below 2^16); *total receives the sum
__device__ __forceinline__ uint32_t block_scan(uint32_t x, uint32_t* wsum, uint32_t* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t incl = x;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= d) incl += y;
  }
  __syncthreads();  // wsum's previous readers are done
  if (lane == 31) wsum[warp] = incl;
  __syncthreads();
  uint32_t before = 0, all = 0;
#pragma unroll
  for (int w = 0; w < FB_ACC_THREADS / 32; ++w) {
    const uint32_t s = wsum[w];
    if (w < warp) before += s;
    all += s;
  }
  *total = all;
  return before + incl - x;
}

// 16 bytes from global to shared memory, asynchronously (a fetch of 64 bytes,
// one point: the default fetches 128, half of it never used for a random
// table point); the thread's own copies have arrived after cp_wait<n> for all
// but its last n groups
__device__ __forceinline__ void cp16(uint4* to, const uint4* from) {
#ifdef __CUDA_ARCH__
  asm volatile("cp.async.cg.shared.global.L2::64B [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(to)), "l"(from)
               : "memory");
#else
  *to = *from;
#endif
}
__device__ __forceinline__ void cp_commit() {
#ifdef __CUDA_ARCH__
  asm volatile("cp.async.commit_group;" ::: "memory");
#endif
}
template <int N>
__device__ __forceinline__ void cp_wait() {
#ifdef __CUDA_ARCH__
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
#endif
}
__device__ __forceinline__ Fq fq_of(const uint4& a, const uint4& b) {
  Fq r;
  r.v[0] = a.x; r.v[1] = a.y; r.v[2] = a.z; r.v[3] = a.w;
  r.v[4] = b.x; r.v[5] = b.y; r.v[6] = b.z; r.v[7] = b.w;
  return r;
}

// A work item's sort output: its bucket offsets and first entry (in elements
// of the set's entries) for each of its sort units, and the table point of
// index 0 and window 0
struct BktItem {
  const uint32_t *offs, *offs2;
  uint32_t ents, ents2, tab;
};
// The lists of a set's items as k_fb_sort (16-bit entries, U) or k_wd_sort (32)
// wrote them: lg bits of point index, then 5 of the window, the sign on top
template <class U>
struct BktLists {
  const U* ents;
  uint32_t lg, N;
  // table point and sign bit of entry e; tab: point of index 0 and window 0
  __device__ __forceinline__ uint32_t point(uint32_t tab, uint32_t e) const {
    const uint32_t v = ents[e], sign = sizeof(U) == 4 ? v & 0x80000000u : (v & 0x8000u) << 16;
    return (tab + ((v >> lg) & 31) * N + (v & ((1u << lg) - 1))) | sign;
  }
};
// What a CTA lists a level with (shared memory). A run: entry or slot of its
// first addition, its tab, number of additions, place in the list | first
// target slot << 16
struct BktShared {
  uint16_t sstart[FB_GROUP * FB_BUCKETS + 1];  // first slot of each bucket
  uint32_t wsum[FB_ACC_THREADS / 32];
  uint4 run[FB_RUNS_MAX];
  uint32_t runs;
  __device__ __forceinline__ bool defer(uint32_t from, uint32_t tab, uint32_t pairs, uint32_t at, uint32_t slot) {
    const uint32_t i = atomicAdd(&runs, 1u);
    if (i < FB_RUNS_MAX) run[i] = make_uint4(from, tab, pairs, at | slot << 16);
    return i < FB_RUNS_MAX;
  }
};
// The listings are functions of their own: inlined, they cost the passes
// registers (a 1024 x 1024 blob of random bytes 106.7 -> 108.5 ms; so 107.0).
// Two pairs are listed at a time, as the stores keep the loads of the next
// pair behind them (32 x 1024 4.95 -> 4.75 ms), and the counts take the offsets
// of eight buckets (1024 x 1024 108.0 -> 107.0).
// Level 1 of entries lo .. hi - 1 of the turn, buckets k0 .. k0 + per - 1 of
// item `it`, whose first entry is the turn's entry `first` (`mine` false: no
// such item): lists the pairs, writes what is alone in its bucket, and sets
// sstart. Returns the number of additions.
template <class U>
static __device__ __noinline__ uint32_t bkt_list_first(BktShared& sh, const BktLists<U> l, const BktItem it, bool mine,
                                                       uint32_t first, uint32_t lo, uint32_t hi, uint32_t k0,
                                                       uint32_t per, const G1Aff* tab, G1Aff* slots, const G1Aff* fin,
                                                       uint2* list, uint32_t* dst) {
  const uint32_t f0 = it.offs[0], f1 = it.offs2 ? it.offs2[0] : 0u;
  // the range of the segment in bucket k, as entry ranges of its two sort units
  struct Part {
    uint32_t e[2], n[2], carry;
  };
  auto part = [&](uint32_t k) {
    Part p = {};
    if (!mine) return p;
    const uint32_t b = k % FB_BUCKETS;
    const uint32_t o0 = it.offs[b], c0 = it.offs[b + 1] - o0;
    const uint32_t o1 = it.offs2 ? it.offs2[b] : 0u, c1 = it.offs2 ? it.offs2[b + 1] - o1 : 0u;
    const uint32_t at = first + (o0 - f0) + (o1 - f1);
    const uint32_t qa = min(max(lo, at) - at, c0 + c1), qb = hi > at ? max(qa, min(hi - at, c0 + c1)) : qa;
    const uint32_t a0 = min(qa, c0), b0 = min(qb, c0);
    p.e[0] = it.ents + o0 + a0;
    p.n[0] = b0 - a0;
    p.e[1] = it.ents2 + o1 + (qa - a0);
    p.n[1] = (qb - b0) - (qa - a0);
    p.carry = at < lo && qb > qa;  // the bucket began in an earlier segment
    return p;
  };
  if (threadIdx.x == 0) sh.runs = 0;  // its last readers are behind a barrier, the next ones behind block_scan's
  uint32_t cnt = 0;  // pairs | slots << 16
#pragma unroll 8
  for (uint32_t k = k0; k < k0 + per; ++k) {
    const Part p = part(k);
    cnt += ((p.n[0] >> 1) + (p.n[1] >> 1)) + ((((p.n[0] + 1) >> 1) + ((p.n[1] + 1) >> 1) + p.carry) << 16);
  }
  uint32_t total;
  const uint32_t at = block_scan(cnt, sh.wsum, &total);
  uint32_t p = at & 0xffffu, sl = at >> 16;
  for (uint32_t k = k0; k < k0 + per; ++k) {
    const Part r = part(k);
    sh.sstart[k] = (uint16_t)sl;
    if (r.carry) st_aff(slots + sl++, ld_aff(fin + k));
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      const uint32_t pairs = r.n[s] >> 1, ptab = it.tab + (s ? 1u << l.lg : 0u);
      uint32_t e = r.e[s];
      if (pairs >= FB_RUN_PAIRS && sh.defer(e, ptab, pairs, p, sl)) {
        p += pairs;
        sl += pairs;
        e += 2 * pairs;
      } else {
        uint32_t i = 0;
        for (; i + 1 < pairs; i += 2, e += 4, p += 2, sl += 2) {
          const uint2 x = make_uint2(l.point(ptab, e), l.point(ptab, e + 1));
          const uint2 y = make_uint2(l.point(ptab, e + 2), l.point(ptab, e + 3));
          list[p] = x;
          list[p + 1] = y;
          dst[p] = sl;
          dst[p + 1] = sl + 1;
        }
        if (i < pairs) {
          list[p] = make_uint2(l.point(ptab, e), l.point(ptab, e + 1));
          dst[p++] = sl++;
          e += 2;
        }
      }
      if (r.n[s] & 1) {
        const uint32_t v = l.point(ptab, e);
        G1Aff q = ld_aff(tab + (v & 0x7fffffffu));
        if (v >> 31) q.y = -q.y;
        st_aff(slots + sl++, q);
      }
    }
  }
  if (threadIdx.x == FB_ACC_THREADS - 1) sh.sstart[k0 + per] = (uint16_t)sl;
  return total & 0xffffu;
}
// the later levels: slots 2^lst apart of each bucket
static __device__ __noinline__ uint32_t bkt_list_next(BktShared& sh, uint32_t k0, uint32_t per, uint32_t lst,
                                                      uint32_t* dst) {
  if (threadIdx.x == 0) sh.runs = 0;
  auto pairs_of = [&](uint32_t k) {
    return ((uint32_t)sh.sstart[k + 1] - sh.sstart[k] + (1u << lst) - 1) >> (lst + 1);
  };
  uint32_t cnt = 0, np;
#pragma unroll 8
  for (uint32_t k = k0; k < k0 + per; ++k) cnt += pairs_of(k);
  uint32_t p = block_scan(cnt, sh.wsum, &np);
  for (uint32_t k = k0; k < k0 + per; ++k) {
    const uint32_t s0 = sh.sstart[k], pairs = pairs_of(k);
    if (pairs >= FB_RUN_PAIRS && sh.defer(s0, 0, pairs, p, 0)) p += pairs;
    else
      for (uint32_t i = 0; i < pairs; ++i) dst[p++] = s0 + (i << (lst + 1));
  }
  return np;
}
// the runs that bkt_list_first left to the CTA
template <class U>
static __device__ __noinline__ void bkt_runs_first(const BktShared& sh, const BktLists<U> l, uint2* list,
                                                   uint32_t* dst) {
  const uint32_t runs = min(sh.runs, FB_RUNS_MAX);
  for (uint32_t r = 0; r < runs; ++r) {
    const uint4 q = sh.run[r];
    const uint32_t p = q.w & 0xffffu;
    for (uint32_t i = threadIdx.x; i < q.z; i += FB_ACC_THREADS) {
      list[p + i] = make_uint2(l.point(q.y, q.x + 2 * i), l.point(q.y, q.x + 2 * i + 1));
      dst[p + i] = (q.w >> 16) + i;
    }
  }
}
// the runs that bkt_list_next left to the CTA
static __device__ __noinline__ void bkt_runs_next(const BktShared& sh, uint32_t lst, uint32_t* dst) {
  const uint32_t runs = min(sh.runs, FB_RUNS_MAX);
  for (uint32_t r = 0; r < runs; ++r) {
    const uint4 q = sh.run[r];
    for (uint32_t i = threadIdx.x; i < q.z; i += FB_ACC_THREADS) dst[(q.w & 0xffffu) + i] = q.x + (i << (lst + 1));
  }
}

// One addition of a level: what its list entry says (read ahead), and where
// its points are
struct BktDesc {
  uint32_t v1, v2, d;
};
struct BktPair {
  const G1Aff *p1, *p2;  // operands
  G1Aff* d;              // target
};

// First pass of a batch: this thread's additions base, base + T, .. (below np,
// at most K): the product of their denominators, the products before each one
// going to the prefix array. The x coordinates of the addition after next
// arrive in stg (two stages of 4 rows) while a product runs.
template <class M, class Fetch, class Locate>
__device__ __forceinline__ Fq bkt_first(Fetch fetch, Locate locate, uint4* pre, uint4 (*stg)[FB_ACC_THREADS],
                                        uint32_t base, uint32_t K, uint32_t np) {
  constexpr uint32_t T = FB_ACC_THREADS;
  const uint32_t tid = threadIdx.x;
  Fq run = Fq::one();
  K = base < np ? min(K, (np - base + T - 1) / T) : 0;
  auto stage = [&](uint32_t k, const BktDesc& c) {
    if (k < K) {
      const BktPair q = locate(base + k * T, c);
      const uint4 *a = reinterpret_cast<const uint4*>(q.p1), *b = reinterpret_cast<const uint4*>(q.p2);
      uint4(*o)[T] = stg + 4 * (k & 1);
      cp16(&o[0][tid], a);
      cp16(&o[1][tid], a + 1);
      cp16(&o[2][tid], b);
      cp16(&o[3][tid], b + 1);
    }
    cp_commit();
  };
  BktDesc c0 = fetch(base, K > 0), c1 = fetch(base + T, K > 1), c2 = fetch(base + 2 * T, K > 2);
  stage(0, c0);
  stage(1, c1);
#pragma unroll 1
  for (uint32_t k = 0; k < K; ++k) {
    const BktDesc c3 = fetch(base + (k + 3) * T, k + 3 < K);
    cp_wait<1>();
    uint4(*o)[T] = stg + 4 * (k & 1);
    const Fq x1 = fq_of(o[0][tid], o[1][tid]), x2 = fq_of(o[2][tid], o[3][tid]);
    Fq den = x2 - x1;
    if (den.is_zero() || x1.is_zero() || x2.is_zero()) {
      const BktPair q = locate(base + k * T, c0);
      G1Aff q1 = ld_aff(q.p1), q2 = ld_aff(q.p2);
      if (c0.v1 >> 31) q1.y = -q1.y;
      if (c0.v2 >> 31) q2.y = -q2.y;
      den = aff_case(q1, q2).den;
    }
    stage(k + 2, c2);  // into the stage whose points den has consumed
    c0 = c1;
    c1 = c2;
    c2 = c3;
    uint4* w = pre + tid + k * 2 * T;
    w[0] = make_uint4(run.v[0], run.v[1], run.v[2], run.v[3]);
    w[T] = make_uint4(run.v[4], run.v[5], run.v[6], run.v[7]);
    run = M::mul(run, den);
  }
  cp_wait<0>();
  __syncwarp();  // the caller goes on to a barrier: lanes of fewer additions wait for the others here
  return run;
}

// Second pass, in reverse: inv is the inverse of the first pass's product;
// each denominator's inverse follows from it and the prefix, and the sum is
// written to its target. The next addition's points and prefix arrive in stg
// (10 rows) behind the products.
template <class M, class Fetch, class Locate>
__device__ __forceinline__ void bkt_second(Fetch fetch, Locate locate, const uint4* pre, uint4 (*stg)[FB_ACC_THREADS],
                                           uint32_t base, uint32_t K, uint32_t np, Fq inv) {
  constexpr uint32_t T = FB_ACC_THREADS;
  const uint32_t tid = threadIdx.x;
  K = base < np ? min(K, (np - base + T - 1) / T) : 0;
  auto stage = [&](uint32_t k, const BktPair& q) {
    const uint4 *a = reinterpret_cast<const uint4*>(q.p1), *b = reinterpret_cast<const uint4*>(q.p2);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      cp16(&stg[i][tid], a + i);
      cp16(&stg[4 + i][tid], b + i);
    }
    const uint4* w = pre + tid + k * 2 * T;
    cp16(&stg[8][tid], w);
    cp16(&stg[9][tid], w + T);
    cp_commit();
  };
  BktDesc c = fetch(base + (K - 1) * T, K > 0), c1 = fetch(base + (K - 2) * T, K > 1);
  if (K > 0) stage(K - 1, locate(base + (K - 1) * T, c));
#pragma unroll 1
  for (uint32_t k = K; k-- > 0;) {
    const BktDesc c2 = fetch(base + (k - 2) * T, k > 1);
    G1Aff* const d = locate(base + k * T, c).d;
    cp_wait<0>();
    const Fq iv = M::mul(inv, fq_of(stg[8][tid], stg[9][tid]));
    G1Aff q1, q2;
    q1.x = fq_of(stg[0][tid], stg[1][tid]);
    q1.y = fq_of(stg[2][tid], stg[3][tid]);
    q2.x = fq_of(stg[4][tid], stg[5][tid]);
    q2.y = fq_of(stg[6][tid], stg[7][tid]);
    if (c.v1 >> 31) q1.y = -q1.y;
    if (c.v2 >> 31) q2.y = -q2.y;
    Fq den = q2.x - q1.x, num = q2.y - q1.y;
    c = c1;
    c1 = c2;
    int sum = 0;
    if (den.is_zero() || q1.x.is_zero() || q2.x.is_zero()) {
      const AffCase ac = aff_case(q1, q2);
      num = ac.num;
      den = ac.den;
      sum = ac.sum;
      // an operand or infinity; the denominator is 1
      if (sum) st_aff(d, sum == 1 ? q1 : sum == 2 ? q2 : aff_inf());
    }
    if (k > 0) stage(k - 1, locate(base + (k - 1) * T, c));  // every staged value is in registers or used
    if (sum == 0) {
      const FqPair li = M::mul2(num, iv, inv, den);
      const Fq lam = li.a;
      inv = li.b;
      G1Aff r;
      r.x = M::mul(lam, lam) - q1.x - q2.x;
      r.y = M::mul(lam, q1.x - r.x) - q1.y;
      st_aff(d, r);
    }
  }
  __syncwarp();
}

// Persistent CTAs over the (chunk, line) work items. Per item, the entries of
// each bucket are summed as a binary tree: level 1 adds entries 2i and 2i + 1
// of a bucket (table points) into slot i of the bucket's slot range (an odd
// last entry is copied), level r + 1 adds slots 2^r apart in place, until one
// sum per bucket is left; then five levels of additions along the rows and
// columns of the 32 x 32 bucket grid leave the item's FB_OUT sums. The
// additions of a level are independent, so they share inversions: a batch
// gives each thread some additions, whose denominators it multiplies
// up in a first pass (keeping the prefix products), one inversion for the CTA
// follows, and a second pass in reverse order recovers each denominator's
// inverse and adds. Items of more than cap entries (skewed digits) run in
// segments whose bucket sums carry over.
// Wide items (ents32 set) are 1024-bucket blocks of a wide unit of 2^(ulog +
// mlog) points whose buckets are those of its 2^mlog sort units of 2^ulog
// points (k_wd_sort; mlog <= 1): item g of a coset is block g & (2^(ulog -
// 10) - 1) of unit g >> (ulog - 10); bucket k's entries are those of sort
// unit 0 followed by those of sort unit 1, indexing the points of the
// merged unit and the W windows of the wide table.
// M is the product kind of the point additions (chosen by the context's
// tuning; identical results).
// A set's `group` items share a CTA's turn.
template <class M>
__global__ void __launch_bounds__(FB_ACC_THREADS, FB_ACC_MIN_CTAS)
    k_fb_accum(const FbAccPlan plan, const FbScratch scratch, uint32_t* __restrict__ next, uint32_t task) {
  constexpr uint32_t T = FB_ACC_THREADS;
  __shared__ uint4 stg[10][T];           // the passes' staging rows
  __shared__ Fq sp[T];
  __shared__ BktShared sh;
  __shared__ uint32_t first[FB_GROUP + 1];  // entries before each item of the group
  __shared__ uint32_t item;
  const uint32_t tid = threadIdx.x;
  uint8_t* const mem = scratch.base + (size_t)blockIdx.x * scratch.bytes();
  G1Aff* const slots = reinterpret_cast<G1Aff*>(mem);
  G1Aff* const fin = reinterpret_cast<G1Aff*>(mem + scratch.off_fin());
  uint4* const pre = reinterpret_cast<uint4*>(mem + scratch.off_pre());
  uint2* const list = reinterpret_cast<uint2*>(mem + scratch.off_list());
  uint32_t* const dst = reinterpret_cast<uint32_t*>(mem + scratch.off_dst());
  const uint32_t cap = scratch.cap;
  const uint32_t batch = fb_batch(min(max(task, (uint32_t)FB_TASK_MIN), (uint32_t)FB_TASK_MAX));
  uint32_t turn = blockIdx.x;
  for (;;) {
    __syncthreads();  // every thread has read the previous group number
    if (tid == 0) item = atomicAdd(next, 1u);
    __syncthreads();
    // group number -> set and its items u0, u0 + groups, ..: spread over the set,
    // as neighbours may all be empty (a scalar vector's zero end) or all full
    uint32_t u0 = item, groups = 0;
    int set = 0;
    for (; set < plan.n; ++set) {
      const uint32_t group = (uint32_t)plan.a[set].group;
      groups = (plan.start[set + 1] - plan.start[set] + group - 1) / group;
      if (u0 < groups) break;
      u0 -= groups;
    }
    if (set >= plan.n) break;
    const FbAccArgs& a = plan.a[set];
    const uint32_t ng = (plan.start[set + 1] - plan.start[set] - u0 + groups - 1) / groups;
    const bool wide = a.ents32 != nullptr;
    const BktLists<uint32_t> lists32{a.ents32, (uint32_t)a.ulog, (uint32_t)a.tabN};
    const BktLists<uint16_t> lists16{a.ents, 10u, (uint32_t)a.tabN};
    // item i of the group
    auto item_of = [&](uint32_t i) {
      const uint32_t u = u0 + i * groups, nch = 1u << a.lr;
      const uint32_t l = u % a.lines, g = u / a.lines;
      const uint32_t coset = g / nch, b = g % nch;
      BktItem it;
      it.offs2 = nullptr;
      it.ents2 = 0;
      it.tab = (coset * a.Ltot + a.l0 + l) * a.W * (uint32_t)a.tabN;
      if (wide) {
        const int bl = a.ulog - 10, ml = a.mlog;
        const uint32_t unit = b >> bl, blk = b & ((1u << bl) - 1);
        const uint32_t cu = coset * ((nch >> bl) << ml) + (unit << ml);  // first sort unit
        it.offs = a.offs + (size_t)cu * ((1u << a.ulog) + 1) + (size_t)blk * FB_BUCKETS;
        it.ents = cu * (uint32_t)wd_unit_ents(a.ulog);
        if (ml) {
          it.offs2 = it.offs + ((1u << a.ulog) + 1);
          it.ents2 = it.ents + (uint32_t)wd_unit_ents(a.ulog);
        }
        it.tab += unit << (a.ulog + ml);
      } else {
        it.offs = a.offs + (size_t)g * (FB_BUCKETS + 1);
        it.ents = g * (FB_WINDOWS << a.lc);
        it.tab += b << a.lc;
      }
      return it;
    };
    if (tid == 0) {
      uint32_t n = 0;
      for (uint32_t i = 0; i < ng; ++i) {
        first[i] = n;
        const BktItem it = item_of(i);
        n += it.offs[FB_BUCKETS] - it.offs[0];
        if (it.offs2) n += it.offs2[FB_BUCKETS] - it.offs2[0];
      }
      first[ng] = n;
    }
    __syncthreads();
    const uint32_t nent = first[ng];
    // this thread's buckets k0 .. k0 + per - 1 are item my's
    const uint32_t per = (ng <= 2 ? ng : 4) * (FB_BUCKETS / T), k0 = tid * per, my = k0 / FB_BUCKETS;
    uint32_t seg = 0, st = 0, lst = 0, h = 0, lh = 0;
    int mode = 0;  // 0: level 1 of segment seg, 1: slots 2^lst apart, 2: grid level of half width h
    for (;;) {
      uint32_t np = 0;
      if (mode == 0) {
        const uint32_t lo = seg * cap, mine = min(my, ng - 1);
        const BktItem it = item_of(mine);
        const uint32_t hi = min(nent, lo + cap);
        np = wide ? bkt_list_first(sh, lists32, it, my < ng, first[mine], lo, hi, k0, per, a.tab, slots, fin, list, dst)
                  : bkt_list_first(sh, lists16, it, my < ng, first[mine], lo, hi, k0, per, a.tab, slots, fin, list, dst);
      } else if (mode == 1) {
        np = bkt_list_next(sh, k0, per, lst, dst);
        if (np == 0) {  // one sum per bucket left
          for (uint32_t k = tid; k < ng * FB_BUCKETS; k += T) {
            if (sh.sstart[k + 1] > sh.sstart[k]) st_aff(fin + k, ld_aff(slots + sh.sstart[k]));
            else if (seg == 0) st_aff(fin + k, aff_inf());
          }
          ++seg;
          if (seg * cap < nent) {
            mode = 0;
          } else {
            mode = 2;
            h = FB_GRID / 2;
            lh = fb_log2(FB_GRID / 2);
          }
          __syncthreads();
          continue;
        }
      } else {
        np = ng * FB_OUT * h;
      }
      __syncthreads();
      if (sh.runs) {  // the same for all threads; 0 in grid levels
        if (mode != 0) bkt_runs_next(sh, lst, dst);
        else if (wide) bkt_runs_first(sh, lists32, list, dst);
        else bkt_runs_first(sh, lists16, list, dst);
        __syncthreads();
      }
      const uint32_t lmode = (uint32_t)mode;
      auto fetch = [&](uint32_t j, bool there) {
        BktDesc c = {0, 0, 0};
        if (there && lmode == 0) {
          const uint2 v = list[j];
          c.v1 = v.x;
          c.v2 = v.y;
        }
        if (there && lmode <= 1) c.d = dst[j];
        return c;
      };
      // the j-th addition of the level, c its list entry
      auto locate = [&](uint32_t j, const BktDesc& c) {
        BktPair r;
        if (lmode == 0) {
          r.p1 = a.tab + (c.v1 & 0x7fffffffu);
          r.p2 = a.tab + (c.v2 & 0x7fffffffu);
          r.d = slots + c.d;
        } else if (lmode == 1) {
          r.d = slots + c.d;
          r.p1 = r.d;
          r.p2 = r.d + st;
        } else {
          // per item FB_BUCKETS slots: rows [32][16], then columns [16][32]
          const uint32_t it = j >> (lh + 6);
          j &= FB_OUT * h - 1;
          const bool col = j >= FB_GRID * h;
          if (col) j -= FB_GRID * h;
          const uint32_t row = j >> lh, in = j & (h - 1);
          r.d = slots + it * FB_BUCKETS + (col ? FB_BUCKETS / 2 + j : row * (FB_GRID / 2) + in);
          r.p1 = h == FB_GRID / 2 ? fin + it * FB_BUCKETS + (col ? j : row * FB_GRID + in) : r.d;
          r.p2 = r.p1 + (col ? FB_GRID * h : h);
        }
        return r;
      };
      const uint32_t nb = (np + T * batch - 1) / (T * batch);
      const uint32_t K = nb ? (np + T * nb - 1) / (T * nb) : 0;
      for (uint32_t base = tid, left = nb; left > 0; --left, base += T * K) {
        const Fq all = bkt_first<M>(fetch, locate, pre, stg, base, K, np);
        bkt_second<M>(fetch, locate, pre, stg, base, K, np, block_inverse<M>(all, sp, turn++));
      }
      __syncthreads();
      if (mode == 0) {
        mode = 1;
        st = 1;
        lst = 0;
      } else if (mode == 1) {
        st *= 2;
        ++lst;
      } else {
        if (h == 1) break;
        h >>= 1;
        --lh;
      }
    }
    // R_a in slot 16 a, C_b in slot 512 + b of the item's slots
    for (uint32_t k = tid; k < ng * FB_OUT; k += T) {
      const uint32_t i = k / FB_OUT, o = k % FB_OUT;
      st_aff(a.out + (size_t)(u0 + i * groups) * FB_OUT + o,
             ld_aff(slots + i * FB_BUCKETS + (o < FB_GRID ? o * (FB_GRID / 2) : FB_BUCKETS / 2 + o - FB_GRID)));
    }
  }
}

}  // namespace zg
