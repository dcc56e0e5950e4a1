// k_fb_accum on host threads where single buckets hold long runs of a level's
// additions, against plain XYZZ sums.
//   bucket_ranges FORM GROUP SEED
// FORM: edge (buckets of 2 (FB_RUN_PAIRS - 1) .. 2 (FB_RUN_PAIRS + 1) + 1
// entries), one (every entry in one bucket, several segments), many (more long
// runs in a turn than FB_RUNS_MAX), few (half as many).
#include <cstdio>
#include <cstdlib>
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

int main(int, char** argv) {
  const std::string form = argv[1];
  const uint32_t group = (uint32_t)atoi(argv[2]), points = 1024, items = 3, most = FB_WINDOWS * points;
  std::mt19937 rng((unsigned)atoi(argv[3]));
  std::vector<G1Aff> base(200);
  XYZZ p = XYZZ::from_affine(G1Aff{Fq::from_u32(1), Fq::from_u32(2)});
  for (G1Aff& b : base) {
    p.to_affine(b);
    p.add_affine(Fq::from_u32(1), Fq::from_u32(2));
  }
  std::vector<G1Aff> tab((size_t)FB_WINDOWS * points * items);
  for (G1Aff& q : tab) q = base[rng() % base.size()];
  // entries per bucket
  std::vector<uint32_t> len(1024, 0);
  const uint32_t edge = 2 * FB_RUN_PAIRS;
  if (form == "one") len[517] = most;
  for (uint32_t k = 0, left = most; form != "one" && k < 1024; ++k) {
    uint32_t n = rng() % 3;
    if (form == "edge" && k % 9 == 0) n = edge - 2 + k / 9 % 6;
    if (form == "many" && k % 5 == 0) n = edge;
    if (form == "few" && k % 16 == 0) n = edge + 13;
    left -= len[k] = std::min(n, left);
  }
  // item g's entries: points of its own chunk, in an order of its own
  std::vector<uint32_t> offs;
  std::vector<uint16_t> ents((size_t)most * items);
  for (uint32_t g = 0; g < items; ++g) {
    std::vector<uint16_t> all(most);
    for (uint32_t e = 0; e < most; ++e) all[e] = (uint16_t)(e % points | e / points << 10 | (rng() & 1) << 15);
    std::shuffle(all.begin(), all.end(), rng);
    std::copy(all.begin(), all.end(), ents.begin() + (size_t)g * most);
    uint32_t at = 0;
    for (uint32_t k = 0; k < 1024; at += len[k++]) offs.push_back(at);
    offs.push_back(at);
  }
  FbAccPlan plan;
  std::vector<G1Aff> out((size_t)items * FB_OUT);
  plan.n = 1;
  plan.start[1] = items;
  FbAccArgs& a = plan.a[0];
  a.tab = tab.data();
  a.offs = offs.data();
  a.ents = ents.data();
  a.out = out.data();
  a.lr = 2;  // items 0 .. 2 of a coset
  a.lc = 10;
  a.tabN = (uint64_t)points * items;
  a.group = (int)group;
  FbScratch s;
  s.cap = form == "one" ? 10000 : FB_CAP_MAX;
  std::vector<uint8_t> mem(s.bytes() + 256);
  s.base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(mem.data()) + 255) / 256 * 256);
  uint32_t next = 0;
  run_block(FB_ACC_THREADS, [&] { k_fb_accum<MulImad>(plan, s, &next, 32); });

  auto same = [](const XYZZ& x, const G1Aff& q) {
    G1Aff b;
    return x.to_affine(b) ? b.x == q.x && b.y == q.y : aff_is_inf(q);
  };
  int bad = 0;
  for (uint32_t g = 0; g < items; ++g) {
    std::vector<XYZZ> sum(1024, XYZZ::inf());
    for (uint32_t k = 0; k < 1024; ++k)
      for (uint32_t e = offs[g * 1025 + k]; e < offs[g * 1025 + k + 1]; ++e) {
        const uint16_t v = ents[(size_t)g * most + e];
        G1Aff q = tab[(size_t)(v >> 10 & 31) * a.tabN + g * points + (v & 1023)];
        if (v >> 15) q.y = -q.y;
        sum[k].add_affine(q.x, q.y);
      }
    for (int r = 0; r < 32; ++r) {
      XYZZ row = XYZZ::inf(), col = XYZZ::inf();
      for (int c = 0; c < 32; ++c) {
        row.add(sum[32 * r + c]);
        col.add(sum[32 * c + r]);
      }
      bad += !same(row, out[g * FB_OUT + r]) + !same(col, out[g * FB_OUT + 32 + r]);
    }
  }
  printf("%s: %d of %u sums differ\n", form.c_str(), bad, items * FB_OUT);
  return bad != 0;
}
