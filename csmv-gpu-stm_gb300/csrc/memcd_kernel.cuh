// memcd_kernel.cuh - transactional set-associative cache (the reference's memcachedGPU driver,
// memcachedGPU/memcdSH.cu:237-448) on the stamp commit protocol (sm_103a).
//
// Reference: four versioned arrays (key, val, ts, state) of one word each per way; a SET reads
// key/state/ts of every way with TXRead, picks the way holding the key (valid) or else the one
// with the smallest LRU timestamp, and writes all four items; a GET reads key/state of each way
// read-only and the value of the first match. Every transaction goes through the single
// commit-server block.
//
// Here an entry (set, way) holds kMemcdDepth versions; version j is
//   tag  (8 bytes): ts << 32 | valid << 31 | 31-bit key hash   - one single-copy-atomic word
//   rec  (64 bytes): {lru, 0, 0, 0}, 16-byte key, 32-byte value
// A writer (holding the entry's lock) empties the victim's tag, fences, writes the record,
// fences and publishes the new tag; a reader re-reads the tag after the record, so a record is
// used only if its tag did not move (a sequence-lock). The tags of a set's 8 ways sit in one
// 128-byte line: a GET reads the ways' commit words, takes each way's latest committed version
// (the one its stamp names) from that line, and reads only the records whose valid hash matches,
// in way order (first full key match wins, as the reference breaks at the first match). A SET
// looks at each way's latest committed
// version (by its commit word), chooses the slot by the reference's rule, locks only that entry,
// takes a commit timestamp from the CTA's server, validates the eight stamps and installs the
// new version. Rounds of 32 requests are warp-uniform GETs or SETs (memcdSH.cu:333-339).
//
// Bound under Zipf(0.99) by the hottest entry's lock, through which its SETs pass one hold after
// the other, and by the GETs that wait for holders. A warp's SETs of one key therefore share a
// hold; a hold is kept to the timestamp draw, the validation and three fences; and records
// are read only where a tag's hash says so. A call of 64 K requests with 1 % SETs on a filled
// table of 2^20 sets took 1.6 to 1.8 ms with one SET a hold and takes 0.24 to 0.27 ms; a serving
// session of 495 K requests with 5 % SETs took 55 to 57 ms and takes 4.6 ms.
#pragma once
#include <cstdint>

#include "bank_kernel.cuh"

namespace csmv {

constexpr int kWays = 8;
constexpr int kMemcdDepth = 2;
constexpr uint32_t kValidBit = 0x80000000u;
constexpr uint32_t kMemcdBackoffLog2 = 6;  // longest pause after lost locks: 64 << this (ns)

struct MemcdParams {
  const uint32_t* kind;  // [n] 0 = GET, 1 = SET
  const uint4* key;      // [n]
  const uint4* val;      // [2n]
  uint32_t n_rounds;
  uint32_t tick;         // LRU timestamp a SET writes (the reference's curr_clock)
  uint32_t n_sets;
  unsigned long long* tag;  // [entry][kMemcdDepth]
  uint4* rec;               // [entry][kMemcdDepth][4]
  unsigned long long* cw;   // [entry] commit words
  uint32_t* done;
  uint32_t done_mask;
  GlobalSync* gs;
  uint32_t* found;       // [n]
  uint4* val_out;        // [2n]
  uint32_t* log_txn;
  uint32_t* outcome;
  uint32_t log, log_base, log_cap;
  unsigned long long* stats;
  uint32_t nc, batch, spin_log2;
};

struct MemcdMail {
  uint32_t req, rep, snap, cand, base, pad[3];
};

struct MemcdShared {
  uint32_t done_warps, pad[3];
  unsigned long long stat[ST_COUNT];
  MemcdMail mail[kMaxClientWarps];
};

// Set of a 16-byte key (the reference takes its one-word key modulo nbSets,
// memcdSH.cu:79-82; the four words are mixed first) and the 31-bit hash kept in the tag.
__host__ __device__ __forceinline__ uint32_t memcd_mix(uint32_t k0, uint32_t k1, uint32_t k2,
                                                       uint32_t k3) {
  uint32_t h = k0 * 0x9E3779B1u ^ k1 * 0x85EBCA6Bu ^ k2 * 0xC2B2AE35u ^ k3 * 0x27D4EB2Fu;
  return h ^ (h >> 16);
}
__host__ __device__ __forceinline__ uint32_t memcd_set_of(uint32_t h, uint32_t n_sets) {
  return h % n_sets;
}
__host__ __device__ __forceinline__ uint32_t memcd_tag_hash(uint32_t h) {
  return (h * 0x2C1B3C6Du) & 0x7FFFFFFFu;
}

__device__ __forceinline__ bool key_eq(uint4 a, uint4 b) {
  return a.x == b.x && a.y == b.y && a.z == b.z && a.w == b.w;
}
__device__ __forceinline__ uint32_t tag_ts(unsigned long long t) { return (uint32_t)(t >> 32); }

// One round of 32 requests (request r on this lane), run until every request has committed.
// Returns false when the warp must stop (device error raised).
__device__ bool memcd_round(const MemcdParams& p, MemcdShared& sm, MemcdMail& ms, uint32_t me,
                            uint32_t r, uint32_t& seq, uint32_t tick) {
  constexpr int D = kMemcdDepth;
  static_assert(D == 2, "two versions an entry");
  constexpr uint32_t FULL = 0xFFFFFFFFu;
  const uint32_t lane = lane_id();
  bool failed = false;
  {
    const uint32_t kind = p.kind[r];
    const bool is_set = __all_sync(0xFFFFFFFFu, kind == 1u);
    if (__any_sync(0xFFFFFFFFu, (kind == 1u) != is_set || kind > 1u)) {  // mixed round
      if (lane == 0) raise_error(&p.gs->error, ERR_DATA);
      return false;
    }
    const uint4 key = p.key[r];
    const uint32_t hmix = memcd_mix(key.x, key.y, key.z, key.w);
    const uint32_t e0 = memcd_set_of(hmix, p.n_sets) * kWays;
    const uint32_t th = memcd_tag_hash(hmix) | kValidBit;
    uint4 nv0 = make_uint4(0, 0, 0, 0), nv1 = nv0;
    if (is_set) {
      nv0 = p.val[2 * r];
      nv1 = p.val[2 * r + 1];
    }
    uint32_t pending = 0xFFFFFFFFu, attempts = 0, lock_fails = 0;
    while (pending) {
      if (lane == 0) atomicAdd(&sm.stat[ST_ROUNDS], 1ull);
      if (++attempts > (1u << 20)) {
        if (lane == 0) raise_error(&p.gs->error, ERR_LIVELOCK);
        failed = true;
        break;
      }
      if (lock_fails) {
        const uint32_t h = (me * 0x9E3779B1u) ^ (attempts * 0x85EBCA6Bu);
        __nanosleep((h >> 16) & ((64u << lock_fails) - 1u));
      }
      const bool mine = (pending >> lane) & 1u;
      uint32_t snap = 0, err = 0;
      if (lane == 0) {  // the device error word beside the clock
        err = ld_relaxed_gpu(&p.gs->error);
        snap = ld_acquire_gpu(&p.gs->clock);
      }
      snap = __shfl_sync(FULL, snap, 0);
      if (__shfl_sync(FULL, err, 0) != 0u) {
        failed = true;
        break;
      }

      if (!is_set) {
        // GET: the latest committed version of each way, read through its commit word and
        // re-checked afterwards (a double collect), serialised at the largest stamp read. The
        // record read is checked by its tag too (several SETs of one key that commit together
        // replace both versions). Locks: a holder with a timestamp above the snapshot commits
        // after it and is ignored; one below it makes the GET retry; one still without a
        // timestamp when the GET looks may commit inside the snapshot and is waited for (bounded).
        bool found = false, aged = false;
        uint32_t smax = 0;
        uint4 o0 = make_uint4(0, 0, 0, 0), o1 = o0;
        if (mine) {
          unsigned long long w1[kWays];
#pragma unroll
          for (int wy = 0; wy < kWays; wy++) w1[wy] = ld_relaxed_gpu(&p.cw[e0 + wy]);
#pragma unroll
          for (int wy = 0; wy < kWays; wy++) {
            for (uint32_t it = 0; it < 512u; it++) {
              const uint32_t own = (uint32_t)(w1[wy] >> 32);
              if (own == 0u || (own & kPendingFlag)) break;
              __nanosleep(64);
              w1[wy] = ld_relaxed_gpu(&p.cw[e0 + wy]);
            }
          }
          fence_acq_rel_gpu();  // versions after the stamps
          unsigned long long tg[kWays * D];
#pragma unroll
          for (int i = 0; i < kWays * D; i += 2)
            ld_relaxed_gpu_v2(p.tag + (size_t)e0 * D + i, tg[i], tg[i + 1]);
          uint32_t hit = 0, second = 0;  // ways whose latest version has the key's hash; its slot
#pragma unroll
          for (int wy = 0; wy < kWays; wy++) {
            const uint32_t st = (uint32_t)w1[wy], own = (uint32_t)(w1[wy] >> 32);
            if (own != 0u && !(own & kPendingFlag)) aged = true;  // still no timestamp: retry
            smax = max(smax, st);
            bool there = false;
#pragma unroll
            for (int q = 0; q < D; q++)
              if (tag_ts(tg[wy * D + q]) == st) {
                there = true;
                second |= (uint32_t)q << wy;
                if ((uint32_t)tg[wy * D + q] == th) hit |= 1u << wy;
              }
            aged |= !there;
          }
#pragma unroll
          for (int wy = 0; wy < kWays; wy++) {
            const uint32_t own = (uint32_t)(w1[wy] >> 32);
            if ((own & kPendingFlag) && (own & ~kPendingFlag) < smax) aged = true;
          }
          uint32_t read = 0;  // ways whose record was read
          for (uint32_t m = aged ? 0u : hit; m && !found; m &= m - 1u) {
            const uint32_t wy = __ffs(m) - 1u;
            const size_t v = (size_t)(e0 + wy) * D + ((second >> wy) & 1u);
            read |= 1u << wy;
            const uint4 kk = ld_relaxed_gpu_v4(p.rec + v * 4 + 1);
            o0 = ld_relaxed_gpu_v4(p.rec + v * 4 + 2);
            o1 = ld_relaxed_gpu_v4(p.rec + v * 4 + 3);
            found = key_eq(kk, key);
          }
          if (!found) o0 = o1 = make_uint4(0, 0, 0, 0);
          fence_acq_rel_gpu();
#pragma unroll
          for (int wy = 0; wy < kWays; wy++) {  // the second collect
            const unsigned long long w2 = ld_relaxed_gpu(&p.cw[e0 + wy]);
            const uint32_t own = (uint32_t)(w2 >> 32);
            if ((uint32_t)w2 != (uint32_t)w1[wy]) aged = true;
            if ((own & kPendingFlag) && (own & ~kPendingFlag) < smax) aged = true;
            // a holder without a timestamp that locked after the first collect draws its
            // timestamp after every stamp read here: it lands above the snapshot
          }
          for (uint32_t m = read; m; m &= m - 1u) {
            const uint32_t wy = __ffs(m) - 1u;
            const unsigned long long t2 =
                ld_relaxed_gpu(p.tag + (size_t)(e0 + wy) * D + ((second >> wy) & 1u));
            uint32_t st = 0;
#pragma unroll
            for (int q = 0; q < kWays; q++) st = wy == (uint32_t)q ? (uint32_t)w1[q] : st;
            if (tag_ts(t2) != st) aged = true;  // the record was being replaced
          }
        }
        const bool done = mine && !aged;
        if (done) {
          p.found[r] = found ? 1u : 0u;
          p.val_out[2 * r] = o0;
          p.val_out[2 * r + 1] = o1;
          // every commit up to the clock read before the first collect was visible to it, so
          // the state read is also the state at that clock when it is the later of the two
          if (p.log) p.outcome[r] = max(smax, snap) | kSnapFlag;
        }
        const uint32_t dm = __ballot_sync(FULL, done);
        const uint32_t am = __ballot_sync(FULL, mine && aged);
        if (lane == 0) {
          stat_add(sm.stat, ST_COMMIT_RO, __popc(dm));
          stat_add(sm.stat, ST_ABORT_DATA_AGE, __popc(am));
        }
        pending &= ~dm;
        continue;
      }

      // SET. The warp's SETs of one key commit together: their lowest lane reads the set, locks
      // the entry and validates for all of them, and they take timestamps in lane order; of the
      // versions they would install one after the other only the last two remain, and only
      // those are written. (Under Zipf(0.99) the hottest key's SETs follow each other through one
      // lock, two of a round's 32 on average.) When lanes with different keys share a set, only
      // the lowest of them takes part this time.
      const uint32_t peers = __match_any_sync(FULL, mine ? e0 : 0x80000000u | lane);
      const uint32_t lead = __ffs(peers) - 1u;
      const uint4 lk = make_uint4(__shfl_sync(FULL, key.x, lead), __shfl_sync(FULL, key.y, lead),
                                  __shfl_sync(FULL, key.z, lead), __shfl_sync(FULL, key.w, lead));
      const uint32_t samem = __ballot_sync(FULL, key_eq(lk, key));
      const bool leader = mine && lane == lead;
      const bool member = mine && (leader || (peers & ~samem) == 0u);
      // the leader reads each way's latest committed version (the one whose ts is the way's
      // stamp) and picks the slot by the reference's rule: the way holding the key (valid), else
      // the smallest LRU timestamp, first on ties (memcdSH.cu:365-387). Records are read only
      // where the tag's hash matches or, without a match, for the LRU timestamps.
      uint32_t stw[kWays];
      unsigned long long pick[kWays];  // tag of each way's latest version
      uint32_t second = 0, used = 0;   // slot of the latest version; ways whose record was read
      bool aborted = false;
      int slot = 0;
#pragma unroll
      for (int wy = 0; wy < kWays; wy++) {
        stw[wy] = 0;
        pick[wy] = 0;
      }
      if (leader) {
        unsigned long long tg[kWays * D];
#pragma unroll
        for (int wy = 0; wy < kWays; wy++) stw[wy] = (uint32_t)ld_relaxed_gpu(&p.cw[e0 + wy]);
        fence_acq_rel_gpu();  // versions after the stamps
#pragma unroll
        for (int i = 0; i < kWays * D; i += 2)
          ld_relaxed_gpu_v2(p.tag + (size_t)e0 * D + i, tg[i], tg[i + 1]);
        uint32_t hit = 0;
#pragma unroll
        for (int wy = 0; wy < kWays; wy++) {
          bool there = false;
#pragma unroll
          for (int q = 0; q < D; q++)
            if (tag_ts(tg[wy * D + q]) == stw[wy]) {
              there = true;
              second |= (uint32_t)q << wy;
              pick[wy] = tg[wy * D + q];
              if ((uint32_t)pick[wy] == th) hit |= 1u << wy;
            }
          aborted |= !there;  // being replaced: retry
        }
        fence_acq_rel_gpu();  // the record loads stay behind the tag loads (sequence lock)
        bool matched = false;
        for (uint32_t m = aborted ? 0u : hit; m && !matched; m &= m - 1u) {
          const uint32_t wy = __ffs(m) - 1u;
          used |= 1u << wy;
          matched = key_eq(ld_relaxed_gpu_v4(p.rec + ((size_t)(e0 + wy) * D + ((second >> wy) & 1u)) * 4 + 1), key);
          if (matched) slot = (int)wy;
        }
        if (!matched && !aborted) {
          uint32_t lru[kWays];
#pragma unroll
          for (int wy = 0; wy < kWays; wy++)
            lru[wy] = ld_relaxed_gpu(reinterpret_cast<const uint32_t*>(
                p.rec + ((size_t)(e0 + wy) * D + ((second >> wy) & 1u)) * 4));
#pragma unroll
          for (int wy = 1; wy < kWays; wy++)
            if (lru[wy] < lru[0]) {
              lru[0] = lru[wy];
              slot = wy;
            }
          used = 0xFFu;
        }
        fence_acq_rel_gpu();
      }
      // the lock, by a CAS that also proves the entry's stamp (so its latest version is the one
      // read), beside a second look at the tags: no record that was read has been replaced
      uint32_t target = e0 + (uint32_t)slot, st0 = 0;
      bool got = false;
      if (leader && !aborted) {
#pragma unroll
        for (int wy = 0; wy < kWays; wy++) st0 = wy == slot ? stw[wy] : st0;
        unsigned long long t2[kWays];
#pragma unroll
        for (int wy = 0; wy < kWays; wy++)
          t2[wy] = (used >> wy) & 1u ? ld_relaxed_gpu(p.tag + (size_t)(e0 + wy) * D + ((second >> wy) & 1u)) : pick[wy];
        const unsigned long long free_w = st0;
        got = atomicCAS(&p.cw[target], free_w, free_w | ((unsigned long long)me << 32)) == free_w;
        bool moved = false;
#pragma unroll
        for (int wy = 0; wy < kWays; wy++) moved |= t2[wy] != pick[wy];
        if (moved) {
          if (got) st_relaxed_gpu(&p.cw[target], free_w);
          got = false;
          aborted = true;
        }
      }
      const uint32_t locked = __ballot_sync(FULL, got);
      const uint32_t agedm = __ballot_sync(FULL, leader && aborted);
      const bool cand_me = member && ((locked >> lead) & 1u);
      const uint32_t cand = __ballot_sync(FULL, cand_me);
      {
        const uint32_t agm = __ballot_sync(FULL, member && ((agedm >> lead) & 1u));
        const uint32_t wwm = __ballot_sync(FULL, member && !cand_me && !((agedm >> lead) & 1u));
        const uint32_t pvm = __ballot_sync(FULL, mine && !member);
        if (lane == 0) {
          stat_add(sm.stat, ST_ABORT_DATA_AGE, __popc(agm));
          stat_add(sm.stat, ST_ABORT_WRITE_WRITE, __popc(wwm));
          stat_add(sm.stat, ST_ABORT_PREVALID, __popc(pvm));
        }
        lock_fails = wwm ? min(lock_fails + 1, kMemcdBackoffLog2) : 0u;
      }
      if (cand == 0) continue;
      // commit timestamps from the CTA's server; meanwhile the version to replace is withdrawn
      // (the older one: no reader uses it). Its tag, which a SET that fails puts back, is read
      // under the lock: a holder before this one may have withdrawn it and put it back at the same
      // stamp. The load and its fence pass under the draw.
      seq++;
      __syncwarp();
      if (lane == 0) {
        ms.snap = snap;
        ms.cand = cand;
        st_release_cta(&ms.req, seq);
      }
      const uint32_t group = peers & cand, n_group = __popc(group), rank = __popc(group & lanemask_lt());
      target = __shfl_sync(FULL, target, lead);
      st0 = __shfl_sync(FULL, st0, lead);
      const uint32_t latest = __shfl_sync(FULL, (second >> slot) & 1u, lead);
      // rank 0 replaces the other version, rank 1 the latest, rank 2 rank 0's, ...
      const uint32_t my_slot = (rank & 1u) ? latest : 1u - latest;
      const bool inst = cand_me && rank + 2u >= n_group;
      const bool early = inst && my_slot != latest;
      unsigned long long* my_tag = p.tag + (size_t)target * D + my_slot;
      constexpr unsigned long long kNoTag = (unsigned long long)kEmptyTs << 32;
      unsigned long long old_tag = kNoTag;
      fence_acq_rel_gpu();  // the leader's, behind its lock: the last holder's tags
      __syncwarp();
      if (early) {
        old_tag = ld_relaxed_gpu(my_tag);
        st_relaxed_gpu(my_tag, kNoTag);  // readers: moving
      }
      fence_acq_rel_gpu();
      bool ok_wait = true;
      if (lane == 0)
        ok_wait = bounded_wait_fast([&] { return ld_acquire_cta(&ms.rep) == seq; }, &p.gs->error,
                                    ERR_WAIT_REPLY, p.spin_log2);
      ok_wait = __shfl_sync(FULL, ok_wait, 0);
      if (!ok_wait) {
        if (early) st_relaxed_gpu(my_tag, old_tag);
        failed = true;
        break;
      }
      (void)ld_acquire_cta(&ms.rep);
      const uint32_t base = ms.base;
      const uint32_t my_ts = base + 1 + __popc(cand & lanemask_lt());
      // the group's first timestamp in its lock (no timestamp of another SET of this cache set
      // lies between the group's), then the leader's validation
      bool valid = cand_me && leader;
      if (valid) {
        st_relaxed_gpu(&p.cw[target], ((unsigned long long)(kPendingFlag | my_ts) << 32) | st0);
        unsigned long long wd[kWays];
#pragma unroll
        for (int wy = 0; wy < kWays; wy++) wd[wy] = ld_relaxed_gpu(&p.cw[e0 + wy]);
#pragma unroll
        for (int wy = 0; wy < kWays; wy++) {
          if (!valid || wy == slot) continue;  // (the target's stamp is held)
          // a lock of an earlier or not yet numbered holder: wait (bounded) for its outcome;
          // a later holder is ordered after this SET and is ignored
          bool settled = false;
          for (uint32_t it = 0; it < 2048; it++) {
            const uint32_t own = (uint32_t)(wd[wy] >> 32);
            if (own == 0u || own == me ||
                ((own & kPendingFlag) && (own & ~kPendingFlag) >= my_ts)) {
              settled = true;
              break;
            }
            __nanosleep(32);
            wd[wy] = ld_relaxed_gpu(&p.cw[e0 + wy]);
          }
          valid = settled && (uint32_t)wd[wy] == stw[wy];
        }
      }
      valid = __shfl_sync(FULL, valid, lead) && cand_me;
      const uint32_t okm = __ballot_sync(FULL, valid);
      if (lane == 0) {
        stat_add(sm.stat, ST_ABORT_READ_WRITE, __popc(cand & ~okm));
        stat_add(sm.stat, ST_COMMIT_UPDATE, __popc(okm));
      }
      if (__any_sync(FULL, valid && inst && !early)) {  // the latest version is replaced too
        if (valid && inst && !early) st_relaxed_gpu(my_tag, kNoTag);
        fence_acq_rel_gpu();
      }
      if (valid && inst) {
        uint4* rec = p.rec + ((size_t)target * D + my_slot) * 4;
        st_relaxed_gpu_v4(rec, make_uint4(tick, 0u, 0u, 0u));
        st_relaxed_gpu_v4(rec + 1, key);
        st_relaxed_gpu_v4(rec + 2, nv0);
        st_relaxed_gpu_v4(rec + 3, nv1);
      }
      fence_acq_rel_gpu();
      if (valid && inst)
        st_relaxed_gpu(my_tag, ((unsigned long long)my_ts << 32) | th);
      else if (early)
        st_relaxed_gpu(my_tag, old_tag);
      fence_acq_rel_gpu();  // with the relaxed store below, the release of the stamp
      __syncwarp();
      const uint32_t last_ts = __shfl_sync(FULL, my_ts, group ? 31u - __clz(group) : lane);
      if (cand_me && leader)
        st_relaxed_gpu(&p.cw[target], (unsigned long long)(valid ? last_ts : st0));
      if (p.log && cand_me) {
        const uint32_t li = my_ts - 1 - p.log_base;
        if (li < p.log_cap)
          p.log_txn[li] = valid ? r : kHole;
        else
          raise_error(&p.gs->error, ERR_CAPACITY);
      }
      if (valid) {
        if (p.log) p.outcome[r] = my_ts;
        p.found[r] = 0u;
        p.val_out[2 * r] = make_uint4(0, 0, 0, 0);
        p.val_out[2 * r + 1] = make_uint4(0, 0, 0, 0);
      }
      __syncwarp();
      fence_acq_rel_gpu();
      complete_range(p.done, p.done_mask, p.gs, base + 1, base + __popc(cand));
      pending &= ~okm;
    }
  }
  return !failed;
}

__device__ void memcd_client(const MemcdParams& p, MemcdShared& sm, uint32_t w) {
  MemcdMail& ms = sm.mail[w];
  const uint32_t lane = lane_id();
  const uint32_t me = blockIdx.x * p.nc + w + 1;
  uint32_t seq = 0;
  for (;;) {
    uint32_t g = 0;
    if (lane == 0) g = atomicAdd(&p.gs->round_next, 1u);
    g = __shfl_sync(0xFFFFFFFFu, g, 0);
    if (g >= p.n_rounds) break;
    if (!memcd_round(p, sm, ms, me, g * 32u + lane, seq, p.tick)) break;
  }
  __syncwarp();
  if (lane == 0) atomicAdd(&sm.done_warps, 1u);
}

__global__ void __launch_bounds__(512, 1) memcd_kernel(MemcdParams p) {
  __shared__ MemcdShared sm;
  const uint32_t warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) sm.done_warps = 0;
  for (uint32_t i = threadIdx.x; i < ST_COUNT; i += blockDim.x) sm.stat[i] = 0;
  for (uint32_t i = threadIdx.x; i < p.nc; i += blockDim.x) {
    sm.mail[i].req = 0;
    sm.mail[i].rep = 0;
  }
  __syncthreads();
  if (warp == 0)
    server_warp_stamp(p.nc, p.batch, p.gs, sm);
  else
    memcd_client(p, sm, warp - 1);
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < ST_COUNT; i += blockDim.x)
    if (sm.stat[i]) atomicAdd(&p.stats[i], sm.stat[i]);
}

// ---------------------------------------------------------------------------------------------
// Serving: a persistent kernel that admits request batches as the host publishes them.
//
// Requests live in a ring ("arena") of pinned, mapped host memory that the kernel reads and
// writes in place (coherent over the C2C link of a Grace-Blackwell node): request i of a batch
// that starts at arena index f is request (f + i) mod arena size. The host publishes a batch by
// filling its descriptor and then bumping ctl->submitted (release). ONE warp (the first client
// warp of CTA 0) is the admitter: it alone polls the host's control words, turns newly
// published batches into rounds of 32 requests appended to the device round queue, and releases
// the queue tail; it runs no rounds. Every other client warp takes a ticket (the next round
// index, one atomic add) and polls the queue tail in device memory until its round exists, then
// runs it with the cache's commit protocol, so rounds of different batches overlap on the device
// and idle warps put no traffic on the host link (and little on the queue's line: a warp polls
// less often the farther its ticket is from the tail). After a round, the warp makes its results
// visible to the host and counts the round off its batch; the batch's last round stamps done_ns
// and sets done (release). Once ctl->stop is set and every published batch is admitted, or when
// the host has published nothing and every round is done for idle_ns (error ERR_WAIT_REQUEST),
// the admitter raises dev->quit; a warp leaves when quit is set and its ticket is past the tail.
// ---------------------------------------------------------------------------------------------
constexpr uint32_t kServeSlots = 1024;  // batch descriptors in flight at most

struct ServeHostCtl {     // mapped host memory
  uint32_t submitted;     // host: batches published
  uint32_t stop;          // host: finish what is published, then return
  uint32_t error;         // device: first device error of the session (0 = none)
  uint32_t pad[13];
};

struct ServeBatchDesc {   // mapped host memory, one per in-flight batch (slot = batch % kServeSlots)
  uint32_t first, n_req, tick, seq;
  unsigned long long admit_ns, done_ns;  // device global timer
  uint32_t done, sets, pad[6];
};

struct alignas(128) ServeDev {  // device memory
  alignas(128) uint32_t admitted;     // batches turned into rounds
  alignas(128) uint32_t q_head;       // round tickets taken
  alignas(128) uint32_t q_tail;       // rounds appended
  alignas(128) uint32_t rounds_done;  // rounds completed
  alignas(128) uint32_t quit;         // no round will be appended any more
};

struct ServeParams {
  ServeHostCtl* ctl;
  ServeBatchDesc* desc;
  ServeDev* dev;
  uint2* rq;             // [q_mask + 1] {first request index, batch slot}
  uint32_t q_mask;
  uint32_t arena_mask;
  uint32_t* remaining;   // [kServeSlots] rounds left per batch
  uint32_t* tick;        // [kServeSlots] LRU tick per batch
  unsigned long long idle_ns;
  uint32_t serial;       // 1: one batch on the device at a time
};

// The admitter's loop, warp-collective: the only reader of the host's control words.
__device__ void serve_admitter(const MemcdParams& p, const ServeParams& s) {
  const uint32_t lane = lane_id();
  uint32_t adm = 0, qt = 0, last_sub = 0;
  unsigned long long idle_since = globaltimer_ns();
  for (;;) {
    uint32_t sub = 0, stop = 0, err = 0, done = 0;
    if (lane == 0) {
      sub = ld_acquire_sys(&s.ctl->submitted);
      stop = ld_acquire_sys(&s.ctl->stop);
      err = ld_relaxed_gpu(&p.gs->error);
      done = ld_relaxed_gpu(&s.dev->rounds_done);
    }
    sub = __shfl_sync(0xFFFFFFFFu, sub, 0);
    stop = __shfl_sync(0xFFFFFFFFu, stop, 0);
    err = __shfl_sync(0xFFFFFFFFu, err, 0);
    done = __shfl_sync(0xFFFFFFFFu, done, 0);
    if (err) {
      if (lane == 0) st_release_sys(&s.ctl->error, err);  // the host sees it without waiting
      break;
    }
    // one batch at a time (s.serial): the next batch's rounds are appended once every round
    // appended so far is done, so a batch runs alone on the device, as a synchronous call would
    const uint32_t admit_to = (s.serial && done != qt) ? adm : (s.serial ? min(sub, adm + 1u) : sub);
    const bool fresh = adm < admit_to;
    for (uint32_t guard = 0; adm < admit_to && guard < kServeSlots; guard++, adm++) {
      const uint32_t slot = adm % kServeSlots;
      uint32_t first = 0, n = 0, tk = 0;
      if (lane == 0) {
        const volatile ServeBatchDesc* d = s.desc + slot;
        first = d->first;
        n = d->n_req;
        tk = d->tick;
      }
      first = __shfl_sync(0xFFFFFFFFu, first, 0);
      n = __shfl_sync(0xFFFFFFFFu, n, 0);
      tk = __shfl_sync(0xFFFFFFFFu, tk, 0);
      const uint32_t rounds = n / 32u;
      for (uint32_t i = lane; i < rounds; i += 32)
        s.rq[(qt + i) & s.q_mask] = make_uint2((first + 32u * i) & s.arena_mask, slot);
      if (lane == 0) {
        s.remaining[slot] = rounds;
        s.tick[slot] = tk;
        s.desc[slot].admit_ns = globaltimer_ns();
      }
      qt += rounds;
    }
    __syncwarp();
    if (fresh && lane == 0) {
      st_relaxed_gpu(&s.dev->admitted, adm);
      __threadfence();
      st_release_gpu(&s.dev->q_tail, qt);  // rounds, counts and ticks before the tail
    }
    const unsigned long long now = globaltimer_ns();
    if (sub != last_sub || done != qt) {  // the host published, or rounds are running: not idle
      last_sub = sub;
      idle_since = now;
    }
    if (stop && adm == sub) break;  // (serial: adm reaches sub only after the last admission)
    if (now - idle_since > s.idle_ns) {
      if (lane == 0) {
        raise_error(&p.gs->error, ERR_WAIT_REQUEST);
        st_release_sys(&s.ctl->error, ERR_WAIT_REQUEST);
      }
      break;
    }
    if (!fresh) __nanosleep(256);
  }
  if (lane == 0) st_release_gpu(&s.dev->quit, 1u);
}

__device__ void serve_client(const MemcdParams& p, const ServeParams& s, MemcdShared& sm,
                             uint32_t w) {
  MemcdMail& ms = sm.mail[w];
  const uint32_t lane = lane_id();
  const uint32_t me = blockIdx.x * p.nc + w + 1;
  uint32_t seq = 0;
  if (blockIdx.x == 0 && w == 0) {
    serve_admitter(p, s);
  } else {
    for (;;) {
      uint32_t state = 0u, first = 0u, slot = 0u;  // 1: a round, 2: leave
      if (lane == 0) {
        const uint32_t ticket = atomicAdd(&s.dev->q_head, 1u);
        for (;;) {
          const uint32_t tail = ld_acquire_gpu(&s.dev->q_tail);
          if (ticket < tail) {
            const uint2 e = s.rq[ticket & s.q_mask];
            first = e.x;
            slot = e.y;
            state = 1u;
            break;
          }
          if (ld_acquire_gpu(&s.dev->quit) && ticket >= ld_acquire_gpu(&s.dev->q_tail)) {
            state = 2u;  // nothing more will be appended
            break;
          }
          if (ld_relaxed_gpu(&p.gs->error)) {
            state = 2u;
            break;
          }
          // the farther back a ticket is, the more rounds must be appended before it: poll
          // less often, so idle warps do not crowd the queue's L2 line
          __nanosleep(min(64u + 32u * (ticket - tail), 8192u));
        }
      }
      state = __shfl_sync(0xFFFFFFFFu, state, 0);
      if (state == 2u) break;
      first = __shfl_sync(0xFFFFFFFFu, first, 0);
      slot = __shfl_sync(0xFFFFFFFFu, slot, 0);
      uint32_t tk = 0;
      if (lane == 0) tk = ld_relaxed_gpu(&s.tick[slot]);
      tk = __shfl_sync(0xFFFFFFFFu, tk, 0);
      if (!memcd_round(p, sm, ms, me, (first + lane) & s.arena_mask, seq, tk)) {
        if (lane == 0) st_release_sys(&s.ctl->error, max(1u, ld_relaxed_gpu(&p.gs->error)));
        break;
      }
      __syncwarp();
      if (lane == 0) {
        __threadfence_system();  // this round's results reach the host before its batch completes
        if (atomicSub(&s.remaining[slot], 1u) == 1u) {
          s.desc[slot].done_ns = globaltimer_ns();
          __threadfence_system();
          st_release_sys(&s.desc[slot].done, 1u);
        }
        atomicAdd(&s.dev->rounds_done, 1u);
      }
    }
  }
  __syncwarp();
  if (lane == 0) atomicAdd(&sm.done_warps, 1u);
}

__global__ void __launch_bounds__(512, 1) memcd_serve_kernel(MemcdParams p, ServeParams s) {
  __shared__ MemcdShared sm;
  const uint32_t warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) sm.done_warps = 0;
  for (uint32_t i = threadIdx.x; i < ST_COUNT; i += blockDim.x) sm.stat[i] = 0;
  for (uint32_t i = threadIdx.x; i < p.nc; i += blockDim.x) {
    sm.mail[i].req = 0;
    sm.mail[i].rep = 0;
  }
  __syncthreads();
  if (warp == 0)
    server_warp_stamp(p.nc, p.batch, p.gs, sm);
  else
    serve_client(p, s, sm, warp - 1);
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < ST_COUNT; i += blockDim.x)
    if (sm.stat[i]) atomicAdd(&p.stats[i], sm.stat[i]);
}

}  // namespace csmv
