// k_fb_accum on host threads against plain XYZZ sums of the same buckets.
//   bucket_accum KIND GROUP SEED
// KIND: chunk (1024 points), small (32-point chunks), wide (2^11-point units),
// merged (pairs of units), skewed (most digits equal: buckets across several
// segments), empty (no entries). Points repeat within buckets, with both
// signs, so that doublings and cancellations occur.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include <string>

#include "cuda_threads.hpp"
namespace zg {
constexpr int FB_BITS = 11, FB_WINDOWS = 24, FB_BUCKETS = 1024, FB_ACC_THREADS = 128, FB_ACC_MIN_CTAS = 4;
constexpr int fb_log2(int x) { return x <= 1 ? 0 : 1 + fb_log2(x / 2); }
constexpr int wd_windows(int ulog) { return 254 / (ulog + 1) + 1; }
constexpr uint64_t wd_unit_ents(int ulog) { return (uint64_t)wd_windows(ulog) << ulog; }
}  // namespace zg
#include "../../0g-da-encoder_b200/csrc/zg_bucket.cuh"
using namespace zg;

static std::vector<G1Aff> multiples(size_t n) {
  G1Aff g;
  g.x = Fq::from_u32(1);
  g.y = Fq::from_u32(2);
  std::vector<G1Aff> out(n);
  XYZZ p = XYZZ::from_affine(g);
  for (size_t i = 0; i < n; ++i) {
    p.to_affine(out[i]);
    p.add_affine(g.x, g.y);
  }
  return out;
}
static bool same(const XYZZ& p, const G1Aff& q) {
  G1Aff a;
  if (!p.to_affine(a)) return q.x.is_zero() && q.y.is_zero();
  return a.x == q.x && a.y == q.y;
}

int main(int argc, char** argv) {
  const std::string kind = argv[1];
  const uint32_t group = (uint32_t)atoi(argv[2]);
  std::mt19937 rng((unsigned)atoi(argv[3]));
  const bool wide = kind == "wide" || kind == "merged" || kind == "skewed";
  const int lc = kind == "small" ? 5 : 10, ulog = 11, mlog = kind == "merged" || kind == "skewed" ? 1 : 0;
  const uint32_t units = 1u << mlog, unit_points = wide ? 1u << ulog : 1u << lc, buckets = wide ? 1u << ulog : 1024u;
  const uint32_t points = unit_points * units, W = wide ? (uint32_t)wd_windows(ulog) : FB_WINDOWS;
  const uint32_t items = wide ? buckets / 1024 : 1;  // of the same lists for every line
  const std::vector<G1Aff> base = multiples(300);
  std::vector<G1Aff> tab((size_t)3 * W * points);
  for (G1Aff& p : tab) {
    p = base[rng() % base.size()];
    if (rng() % 2) p.y = -p.y;
  }
  const size_t unit_ents = wide ? wd_unit_ents(ulog) : (size_t)FB_WINDOWS << lc;
  std::vector<std::vector<uint32_t>> list((size_t)units * buckets);
  for (uint32_t u = 0; u < units; ++u)
    for (uint32_t p = 0; p < unit_points; ++p)
      for (uint32_t w = 0; w < W; ++w) {
        uint32_t d = rng() % (buckets + 1);
        if (kind == "skewed" && w < W - 4) d = 7;
        else if (w == W - 1) d = rng() % 3;
        if (!d || kind == "empty") continue;
        const uint32_t neg = rng() % 2;
        list[(size_t)u * buckets + d - 1].push_back(wide ? p | w << ulog | neg << 31 : p | w << 10 | neg << 15);
      }
  std::vector<uint32_t> offs, e32(unit_ents * units);
  std::vector<uint16_t> e16(unit_ents * units);
  for (uint32_t u = 0; u < units; ++u) {
    uint32_t at = 0;
    for (uint32_t k = 0; k < buckets; ++k) {
      offs.push_back(at);
      for (uint32_t v : list[(size_t)u * buckets + k]) {
        e32[u * unit_ents + at] = v;
        e16[u * unit_ents + at++] = (uint16_t)v;
      }
    }
    offs.push_back(at);
  }
  FbAccPlan plan;
  const uint32_t lines = 3;  // table lines that read the same lists
  std::vector<G1Aff> out((size_t)items * lines * FB_OUT);
  plan.n = 1;
  plan.start[1] = items * lines;
  FbAccArgs& a = plan.a[0];
  a.tab = tab.data();
  a.offs = offs.data();
  a.ents = wide ? nullptr : e16.data();
  a.ents32 = wide ? e32.data() : nullptr;
  a.out = out.data();
  a.lr = fb_log2((int)items);
  a.lc = lc;
  a.ulog = ulog;
  a.mlog = mlog;
  a.W = (int)W;
  a.lines = a.Ltot = (int)lines;
  a.tabN = points;
  a.group = (int)group;
  FbScratch s;
  s.cap = kind == "skewed" ? 8192 : min(FB_GROUP * W * 1536 << mlog, FB_CAP_MAX);
  std::vector<uint8_t> mem(s.bytes() + 256);
  s.base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(mem.data()) + 255) / 256 * 256);
  uint32_t next = 0;
  run_block(FB_ACC_THREADS, [&] { k_fb_accum<MulImad>(plan, s, &next, 32); });

  int bad = 0;
  for (uint32_t item = 0; item < items * lines; ++item) {
    const uint32_t it = item / lines, line = item % lines;
    std::vector<XYZZ> sum(1024, XYZZ::inf());
    for (uint32_t u = 0; u < units; ++u)
      for (uint32_t k = 0; k < 1024; ++k)
        for (uint32_t v : list[(size_t)u * buckets + it * 1024 + k]) {
          const uint32_t lg = wide ? (uint32_t)ulog : 10u;
          const uint32_t idx = (v & ((1u << lg) - 1)) + u * unit_points, w = (v >> lg) & 31;
          G1Aff q = tab[((size_t)line * W + w) * points + idx];
          if (wide ? v >> 31 : (v >> 15) & 1) q.y = -q.y;
          sum[k].add_affine(q.x, q.y);
        }
    for (int r = 0; r < 32; ++r) {
      XYZZ row = XYZZ::inf(), col = XYZZ::inf();
      for (int c = 0; c < 32; ++c) {
        row.add(sum[32 * r + c]);
        col.add(sum[32 * c + r]);
      }
      bad += !same(row, out[item * FB_OUT + r]) + !same(col, out[item * FB_OUT + 32 + r]);
    }
  }
  printf("%s: %d of %u sums differ\n", kind.c_str(), bad, items * lines * FB_OUT);
  return bad != 0;
}
