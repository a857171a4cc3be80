// driver.cpp - CPU runs of the commit kernels' warp code (see csmv_prims.cuh beside it).
#include <cstring>
#include <map>
#include <set>

#include "csmv-gpu-stm_gb300/csrc/memcd_kernel.cuh"

using namespace csmv;

// `warps` client warps of one CTA and its commit server run rounds of 32 requests of a cache of
// n_sets sets, round r under the LRU tick ticks[r] (as rounds of overlapping batches do). Returns 0,
// the device error word, or 255 when the run did not end.
extern "C" int emu_memcd(uint32_t warps, uint32_t rounds, const uint32_t* kind, const uint32_t* key,
                         const uint32_t* val, const uint32_t* ticks, uint32_t n_sets, uint64_t seed,
                         uint32_t switch_log2, unsigned long long* tags, uint32_t* recs,
                         uint32_t* found, uint32_t* val_out, uint32_t* log_txn, uint32_t log_cap,
                         uint32_t* outcome, uint32_t* final_ts) {
  std::vector<uint4> k4(rounds * 32), v4(rounds * 64), rec((size_t)n_sets * kWays * kMemcdDepth * 4),
      vo(rounds * 64);
  memcpy(k4.data(), key, k4.size() * 16);
  memcpy(v4.data(), val, v4.size() * 16);
  memcpy(rec.data(), recs, rec.size() * 16);
  std::vector<unsigned long long> cw((size_t)n_sets * kWays), stats(ST_COUNT);
  std::vector<uint32_t> done(1024);
  static GlobalSync gs;
  memset((void*)&gs, 0, sizeof(gs));
  static MemcdShared sm;
  memset((void*)&sm, 0, sizeof(sm));
  MemcdParams p{};
  p.kind = kind;
  p.key = k4.data();
  p.val = v4.data();
  p.n_rounds = rounds;
  p.n_sets = n_sets;
  p.tag = tags;
  p.rec = rec.data();
  p.cw = cw.data();
  p.done = done.data();
  p.done_mask = 1023;
  p.gs = &gs;
  p.found = found;
  p.val_out = vo.data();
  p.log_txn = log_txn;
  p.outcome = outcome;
  p.log = 1;
  p.log_cap = log_cap;
  p.stats = stats.data();
  p.nc = warps;
  p.spin_log2 = 30;
  emu::reset();
  emu::switch_log2 = switch_log2;
  emu::add_warp(0, 0, [&] {  // the commit server, one lane: the next timestamps to each request
    std::vector<uint32_t> seen(warps);
    for (; lane_id() == 0 && sm.done_warps != warps; emu::pause())
      for (uint32_t w = 0; w < warps; w++) {
        const uint32_t req = ld_acquire_cta(&sm.mail[w].req);
        if (req == seen[w]) continue;
        sm.mail[w].base = atomicAdd(&gs.ts_next, (uint32_t)__popc(sm.mail[w].cand));
        st_release_cta(&sm.mail[w].rep, seen[w] = req);
      }
  });
  for (uint32_t w = 0; w < warps; w++)
    emu::add_warp(0, w + 1, [&, w] {
      uint32_t seq = 0;
      for (;;) {
        uint32_t g = 0;
        if (lane_id() == 0) g = atomicAdd(&gs.round_next, 1u);
        g = __shfl_sync(0xFFFFFFFFu, g, 0);
        if (g >= rounds) break;
        if (!memcd_round(p, sm, sm.mail[w], w + 1, g * 32u + lane_id(), seq, ticks[g])) break;
      }
      __syncwarp();
      if (lane_id() == 0) atomicAdd(&sm.done_warps, 1u);
    });
  // What makes failing SETs meet: a warp that reads a withdrawn tag waits there until its holder
  // has let go of the entry; one that has locked an entry waits until a stamp of the set moves.
  auto in = [](const void* q, const auto& v) { return q >= v.data() && q < v.data() + v.size(); };
  emu::on_load = [&](const void* q, bool) {
    const unsigned long long* t = (const unsigned long long*)q;
    if (t < tags || t >= tags + cw.size() * kMemcdDepth || tag_ts(*t) != kEmptyTs) return;
    const unsigned long long* w = &cw[(t - tags) / kMemcdDepth];
    if ((*w >> 32) != 0ull && (emu::rnd() & 3u)) emu::hold([w] { return (*w >> 32) == 0ull; }, 60000);
  };
  emu::on_store = [&](const void* q, unsigned long long v) {
    const uint32_t own = (uint32_t)(v >> 32);
    if (!in(q, cw) || own == 0u || (own & kPendingFlag) || (emu::rnd() & 1u) == 0u) return;
    const size_t e0 = ((const unsigned long long*)q - cw.data()) / kWays * kWays;
    const std::vector<unsigned long long> was(cw.begin() + e0, cw.begin() + e0 + kWays);
    emu::cur->warp->until = [&cw, e0, was] {
      for (int i = 0; i < kWays; i++)
        if ((uint32_t)cw[e0 + i] != (uint32_t)was[i]) return true;
      return false;
    };
    emu::cur->warp->patience = emu::steps + 8000;
  };
  const bool ended = emu::run(seed, 1ull << 28);
  memcpy(recs, rec.data(), rec.size() * 16);
  memcpy(val_out, vo.data(), vo.size() * 16);
  *final_ts = gs.ts_next;
  return ended ? (int)gs.error : 255;
}

// `warps` warps complete the ranges [lo[i], hi[i]] of timestamps after clock0, warp w those with
// i = w, w + warps, ... Counts in *unordered the completion words that a clock store passes while the
// lane that read them has not acquired them (a fence, or the load itself). Returns 0, or 255 when
// the run did not end.
extern "C" int emu_complete(uint32_t warps, uint32_t n, const uint32_t* lo, const uint32_t* hi,
                            uint32_t clock0, uint32_t done_mask, uint64_t seed, uint32_t* clock_end,
                            uint32_t* unordered) {
  std::vector<uint32_t> done(done_mask + 1);
  static GlobalSync gs;
  memset((void*)&gs, 0, sizeof(gs));
  gs.clock = clock0;
  *unordered = 0;
  emu::reset();
  emu::switch_log2 = 2;
  for (uint32_t w = 0; w < warps; w++)
    emu::add_warp(0, w, [&, w] {
      for (uint32_t i = w; i < n; i += warps) complete_range(done.data(), done_mask, &gs, lo[i], hi[i]);
    });
  std::map<const emu::Lane*, std::set<uint32_t>> open;  // words read and not acquired yet
  emu::on_load = [&](const void* q, bool acquire) {
    const uint32_t* d = (const uint32_t*)q;
    if (d < done.data() || d > done.data() + done_mask) return;
    if (acquire)
      open[emu::cur].erase(d - done.data());
    else
      open[emu::cur].insert(d - done.data());
  };
  emu::on_fence = [&] { open[emu::cur].clear(); };
  emu::on_store = [&](const void* q, unsigned long long v) {
    if (q != &gs.clock) return;
    for (auto& [lane, words] : open)
      if (lane->warp == emu::cur->warp)
        for (uint32_t t = (gs.clock + 1u) >> 5; t <= (uint32_t)v >> 5; t++) *unordered += words.count(t & done_mask);
  };
  const bool ended = emu::run(seed, 1ull << 26);
  *clock_end = gs.clock;
  return ended ? 0 : 255;
}

// One attempt of the per-transaction protocol for a round of transfers of nr accounts each (addr
// [32][nr]) whose funds are short, beside nothing else. Counts in *unordered the commit words that a
// lane looks at again without a fence since its first look. Returns the committed lanes.
extern "C" uint32_t emu_short_funds(uint32_t nr, const uint32_t* op, const uint32_t* addr, uint32_t n_items,
                                    const int32_t* value, uint64_t seed, uint32_t* unordered) {
  constexpr int kD = 4, kR = 8;
  std::vector<unsigned long long> slots((size_t)n_items * kD, 0xFFFFFFFFull << 32), cw(n_items), stats(ST_COUNT);
  for (uint32_t i = 0; i < n_items; i++) slots[(size_t)i * kD] = (uint32_t)value[i];
  static GlobalSync gs;
  memset((void*)&gs, 0, sizeof(gs));
  static CtaShared<kR, 2> sm;
  memset((void*)&sm, 0, sizeof(sm));
  std::vector<uint32_t> outcome(32);
  std::vector<int32_t> result(32);
  BankParams p{};
  p.n_items = n_items;
  p.slots = slots.data();
  p.cw = cw.data();
  p.gs = &gs;
  p.outcome = outcome.data();
  p.result = (int32_t*)result.data();
  p.log = 1;
  p.prevalidate = 1;
  p.spin_log2 = 20;
  uint32_t fin = 0;
  *unordered = 0;
  emu::reset();
  emu::add_warp(0, 1, [&] {
    uint32_t a[kR] = {}, seq = 0;
    for (uint32_t k = 0; k < nr; k++) a[k] = addr[lane_id() * nr + k];
    bool tried = false, lost = false, failed = false;
    fin = stamp_attempt<kD, kR, 2, false>(p, sm, sm.mail[0], 1u, lane_id(), op[lane_id()], nr, a, true, false, seq,
                                          tried, lost, failed);
  });
  std::map<const emu::Lane*, std::set<const void*>> open;  // words looked at, no fence since
  emu::on_load = [&](const void* q, bool) {
    if (q >= cw.data() && q < cw.data() + n_items && !open[emu::cur].insert(q).second) ++*unordered;
  };
  emu::on_fence = [&] { open[emu::cur].clear(); };
  return emu::run(seed, 1ull << 24) ? fin : 0u;
}

// TXWriteOverlap of one warp: write sets ws [32][2] of nws[l] addresses.
extern "C" void emu_write_overlap(const uint32_t* ws, const uint32_t* nws, uint32_t active, uint32_t* out) {
  emu::reset();
  emu::add_warp(0, 0, [&] {
    const uint32_t l = lane_id();
    WriteSet<2> x;
    x.n = nws[l];
    for (int k = 0; k < 2; k++) x.addr[k] = ws[2 * l + k];
    out[l] = TXWriteOverlap(x, (active >> l) & 1u);
  });
  emu::run(1, 1ull << 20);
}
