// The bounds of k_fb_accum's scratch: merged wide items whose buckets hold odd
// counts of both sort units (the most slots per entry), in segments of given
// sizes, with the gaps between the scratch's blocks poisoned, against plain XYZZ
// sums.
//   bucket_scratch ENTRIES0 ENTRIES1 CAP GROUP TASK
// ENTRIES0/1: entries of each bucket in sort units 0 and 1; CAP 0: one segment
#include <sanitizer/asan_interface.h>

#include <cstdio>
#include <cstdlib>
#include <random>

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
  const uint32_t per[2] = {(uint32_t)atoi(argv[1]), (uint32_t)atoi(argv[2])};
  const uint32_t group = (uint32_t)atoi(argv[4]), task = (uint32_t)atoi(argv[5]);
  constexpr int ulog = 11;
  constexpr uint32_t U = 1u << ulog, W = (uint32_t)wd_windows(ulog), blocks = U / 1024, points = 2 * U;
  std::mt19937 rng(3);
  std::vector<G1Aff> base(150);
  XYZZ p = XYZZ::from_affine(G1Aff{Fq::from_u32(1), Fq::from_u32(2)});
  for (G1Aff& b : base) {
    p.to_affine(b);
    p.add_affine(Fq::from_u32(1), Fq::from_u32(2));
  }
  std::vector<G1Aff> tab((size_t)W * points);
  for (G1Aff& q : tab) q = base[rng() % base.size()];
  std::vector<uint32_t> offs, ents(2 * wd_unit_ents(ulog));
  for (uint32_t u = 0; u < 2; ++u)
    for (uint32_t k = 0; k <= U; ++k) {
      offs.push_back(k * per[u]);
      for (uint32_t i = 0; k < U && i < per[u]; ++i)
        ents[u * wd_unit_ents(ulog) + k * per[u] + i] = rng() % U | rng() % W << ulog | (rng() & 1) << 31;
    }
  FbAccPlan plan;
  std::vector<G1Aff> out((size_t)blocks * FB_OUT);
  plan.n = 1;
  plan.start[1] = blocks;
  FbAccArgs& a = plan.a[0];
  a.tab = tab.data();
  a.offs = offs.data();
  a.ents32 = ents.data();
  a.out = out.data();
  a.lr = fb_log2((int)blocks);
  a.lc = 10;
  a.ulog = ulog;
  a.mlog = 1;
  a.W = (int)W;
  a.tabN = points;
  a.group = (int)group;
  FbScratch s;
  s.group = group;
  s.cap = atoi(argv[3]) ? (uint32_t)atoi(argv[3]) : group * 1024 * (per[0] + per[1]);
  s.ctas = 1;
  std::vector<uint8_t> mem(s.bytes() + 256);
  s.base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(mem.data()) + 255) / 256 * 256);
  const size_t ends[5] = {s.slots() * sizeof(G1Aff), s.off_fin() + group * 1024 * sizeof(G1Aff),
                          s.off_pre() + s.batch() * FB_ACC_THREADS * sizeof(Fq), s.off_list() + s.cap / 2 * sizeof(uint2),
                          s.off_dst() + (s.cap / 2 + 1) * sizeof(uint32_t)};
  const size_t next[5] = {s.off_fin(), s.off_pre(), s.off_list(), s.off_dst(), s.bytes()};
  for (int i = 0; i < 5; ++i) {
    if (next[i] < ends[i] + FbScratch::GAP) return printf("block %d overlaps\n", i), 2;
    ASAN_POISON_MEMORY_REGION(s.base + ends[i], next[i] - ends[i]);
  }
  uint32_t turn = 0;
  run_block(FB_ACC_THREADS, [&] { k_fb_accum<MulImad>(plan, s, &turn, task); });
  ASAN_UNPOISON_MEMORY_REGION(mem.data(), mem.size());

  auto same = [](const XYZZ& x, const G1Aff& q) {
    G1Aff b;
    return x.to_affine(b) ? b.x == q.x && b.y == q.y : aff_is_inf(q);
  };
  int bad = 0;
  for (uint32_t it = 0; it < blocks; ++it) {
    std::vector<XYZZ> sum(1024, XYZZ::inf());
    for (uint32_t u = 0; u < 2; ++u)
      for (uint32_t k = 0; k < 1024; ++k)
        for (uint32_t i = 0; i < per[u]; ++i) {
          const uint32_t v = ents[u * wd_unit_ents(ulog) + (it * 1024 + k) * per[u] + i];
          G1Aff q = tab[(size_t)(v >> ulog & 31) * points + u * U + (v & (U - 1))];
          if (v >> 31) q.y = -q.y;
          sum[k].add_affine(q.x, q.y);
        }
    for (int r = 0; r < 32; ++r) {
      XYZZ row = XYZZ::inf(), col = XYZZ::inf();
      for (int c = 0; c < 32; ++c) {
        row.add(sum[32 * r + c]);
        col.add(sum[32 * c + r]);
      }
      bad += !same(row, out[it * FB_OUT + r]) + !same(col, out[it * FB_OUT + 32 + r]);
    }
  }
  printf("%d of %u sums differ\n", bad, blocks * FB_OUT);
  return bad != 0;
}
