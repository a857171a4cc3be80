// csmv_prims.cuh - the stand-in of csrc/csmv_prims.cuh that runs the commit kernels' warp code on
// the CPU: every lane is a fiber, warp collectives are barriers, and each access to memory is a
// point where a seeded scheduler may go on with another lane. Memory itself is sequentially
// consistent; what orders it on the device (fences, acquires) is reported to the test through
// emu::on_*. Used by tests/test_warp_emu.py, which compiles the kernels' headers against it.
#pragma once
#include <ucontext.h>

#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <functional>
#include <memory>
#include <vector>

#define __device__
#define __host__
#define __global__
#define __shared__
#define __forceinline__ inline
#define __align__(n) __attribute__((aligned(n)))
#define __launch_bounds__(...)
#define __restrict__

struct uint2 { uint32_t x, y; };
struct uint4 { uint32_t x, y, z, w; };
inline uint2 make_uint2(uint32_t x, uint32_t y) { return {x, y}; }
inline uint4 make_uint4(uint32_t x, uint32_t y, uint32_t z, uint32_t w) { return {x, y, z, w}; }
template <class T> T min(T a, T b) { return b < a ? b : a; }
template <class T> T max(T a, T b) { return a < b ? b : a; }

namespace emu {

struct Dim { uint32_t x; };

struct Warp {
  uint32_t block, index, runnable = 0xFFFFFFFFu, left = 32, arrived = 0, epoch = 0;
  const char* op = nullptr;
  unsigned long long slot[2][32];
  std::function<bool()> until;  // held up until this is true, or until step `patience`
  uint64_t patience = 0;
};

struct Lane {
  ucontext_t ctx;
  std::vector<char> stack;
  Warp* warp;
  uint32_t lane;
  std::function<void()> body;
};

inline std::vector<std::unique_ptr<Warp>> warps;
inline std::vector<std::unique_ptr<Lane>> lanes;
inline Lane* cur = nullptr;
inline ucontext_t main_ctx;
inline uint64_t rng_state = 1;
inline uint32_t favoured = 0, switch_log2 = 2;
inline uint64_t steps = 0;
// what the test watches: a load (acquire or not), a store, a fence of the current lane
inline std::function<void(const void*, bool)> on_load;
inline std::function<void(const void*, unsigned long long)> on_store;
inline std::function<void()> on_fence;

inline uint32_t rnd() {
  rng_state = rng_state * 6364136223846793005ull + 1442695040888963407ull;
  return (uint32_t)(rng_state >> 33);
}

inline void pause() { swapcontext(&cur->ctx, &main_ctx); }
inline void step() {  // an access to memory
  if ((rnd() & ((1u << switch_log2) - 1u)) == 0u) pause();
}

// The current lane's warp is held up at this point until `until` is true, for `most` steps at most.
inline void hold(std::function<bool()> until, uint64_t most) {
  cur->warp->until = until;
  cur->warp->patience = steps + most;
  pause();
}

inline void entry() {
  cur->body();
  cur->warp->runnable &= ~(1u << cur->lane);
  cur->warp->left--;
  for (;;) pause();
}

inline void add_warp(uint32_t block, uint32_t index, std::function<void()> body) {
  warps.emplace_back(new Warp{block, index});
  for (uint32_t l = 0; l < 32; l++) {
    lanes.emplace_back(new Lane);
    Lane& f = *lanes.back();
    f.stack.resize(128 << 10);
    f.warp = warps.back().get();
    f.lane = l;
    f.body = body;
    getcontext(&f.ctx);
    f.ctx.uc_stack.ss_sp = f.stack.data();
    f.ctx.uc_stack.ss_size = f.stack.size();
    f.ctx.uc_link = nullptr;
    makecontext(&f.ctx, (void (*)())entry, 0);
  }
}

// Runs every warp to its end; false when nothing can go on or `limit` steps were not enough.
inline bool run(uint64_t seed, uint64_t limit) {
  rng_state = seed * 0x9E3779B97F4A7C15ull + 1;
  for (steps = 0; steps < limit; steps++) {
    uint32_t live[64], k = 0;
    bool left = false;
    for (uint32_t w = 0; w < warps.size(); w++) {
      Warp& x = *warps[w];
      left |= x.left != 0;
      if (x.until && (steps >= x.patience || x.until())) x.until = nullptr;
      if (x.runnable && !x.until) live[k++] = w;
    }
    if (k == 0) {
      bool held = false;
      for (auto& x : warps) held |= (bool)x->until;
      if (held) continue;
      return !left;
    }
    // one warp runs ahead of the others for a while, so that they meet at every distance
    if ((rnd() & 63u) == 0u) favoured = rnd() % warps.size();
    uint32_t w = live[rnd() % k];
    if (warps[favoured]->runnable && !warps[favoured]->until && (rnd() & 7u)) w = favoured;
    uint32_t m = warps[w]->runnable, skip = rnd() % __builtin_popcount(m);
    while (skip--) m &= m - 1;
    cur = lanes[w * 32 + __builtin_ctz(m)].get();
    swapcontext(&main_ctx, &cur->ctx);
  }
  return false;
}

inline void reset() {
  warps.clear();
  lanes.clear();
  favoured = 0;
  on_load = nullptr;
  on_store = nullptr;
  on_fence = nullptr;
}

// Barrier of the warp's 32 lanes that leaves each lane's value with all of them.
inline const unsigned long long* exchange(const char* op, unsigned long long v) {
  Warp& w = *cur->warp;
  if (w.arrived == 0)
    w.op = op;
  else if (w.op != op) {
    fprintf(stderr, "lanes of a warp meet at %s and %s\n", w.op, op);
    abort();
  }
  unsigned long long* s = w.slot[w.epoch & 1u];
  s[cur->lane] = v;
  if (++w.arrived == 32) {
    w.arrived = 0;
    w.epoch++;
    w.runnable = 0xFFFFFFFFu;
  } else {
    w.runnable &= ~(1u << cur->lane);
    pause();
  }
  return s;
}

inline Dim tid() { return {cur->warp->index * 32u + cur->lane}; }
inline Dim bid() { return {cur->warp->block}; }
inline Dim bdim() { return {512}; }
inline Dim gdim() { return {1}; }

template <class T> T load(const T* p, bool acquire = false) {
  step();
  const T v = *(const volatile T*)p;
  if (on_load) on_load(p, acquire);
  return v;
}
template <class T> void store(T* p, T v) {
  step();
  if (on_store) on_store(p, v);
  *(volatile T*)p = v;
}
inline void fence() {
  if (on_fence) on_fence();
  step();
}

}  // namespace emu

#define threadIdx (emu::tid())
#define blockIdx (emu::bid())
#define blockDim (emu::bdim())
#define gridDim (emu::gdim())

// ---- warp collectives (full masks only) ------------------------------------------------------
inline void __syncwarp() { emu::exchange("syncwarp", 0); }
inline void __syncthreads() { abort(); }
inline uint32_t __ballot_sync(uint32_t, bool p) {
  const unsigned long long* s = emu::exchange("ballot", p);
  uint32_t m = 0;
  for (int l = 0; l < 32; l++) m |= (uint32_t)s[l] << l;
  return m;
}
inline bool __any_sync(uint32_t, bool p) { return __ballot_sync(0, p) != 0u; }
inline bool __all_sync(uint32_t, bool p) { return __ballot_sync(0, p) == 0xFFFFFFFFu; }
template <class T> T __shfl_sync(uint32_t, T v, uint32_t src) {
  return (T)emu::exchange("shfl", (unsigned long long)v)[src & 31u];
}
template <class T> T __shfl_up_sync(uint32_t, T v, uint32_t d) {
  const unsigned long long* s = emu::exchange("shfl_up", (unsigned long long)v);
  return emu::cur->lane >= d ? (T)s[emu::cur->lane - d] : v;
}
inline uint32_t __match_any_sync(uint32_t, uint32_t v) {
  const unsigned long long* s = emu::exchange("match", v);
  uint32_t m = 0;
  for (int l = 0; l < 32; l++) m |= (uint32_t)((uint32_t)s[l] == v) << l;
  return m;
}
template <class F> uint32_t emu_reduce(const char* op, uint32_t v, F f) {
  const unsigned long long* s = emu::exchange(op, v);
  uint32_t r = (uint32_t)s[0];
  for (int l = 1; l < 32; l++) r = f(r, (uint32_t)s[l]);
  return r;
}
inline uint32_t __reduce_min_sync(uint32_t, uint32_t v) { return emu_reduce("min", v, min<uint32_t>); }
inline uint32_t __reduce_max_sync(uint32_t, uint32_t v) { return emu_reduce("max", v, max<uint32_t>); }
inline uint32_t __reduce_or_sync(uint32_t, uint32_t v) {
  return emu_reduce("or", v, [](uint32_t a, uint32_t b) { return a | b; });
}

// ---- per lane --------------------------------------------------------------------------------
inline int __popc(uint32_t v) { return __builtin_popcount(v); }
inline int __ffs(uint32_t v) { return __builtin_ffs((int)v); }
inline int __ffsll(long long v) { return __builtin_ffsll(v); }
inline int __clz(uint32_t v) { return v ? __builtin_clz(v) : 32; }
inline uint32_t __umulhi(uint32_t a, uint32_t b) { return (uint32_t)(((uint64_t)a * b) >> 32); }
inline void __nanosleep(uint32_t) { emu::pause(); }
inline void __threadfence() { emu::fence(); }
inline void __threadfence_system() { emu::fence(); }
template <class T> T emu_rmw(T* p, T v, T old) {
  if (emu::on_store) emu::on_store(p, v);
  *(volatile T*)p = v;
  return old;
}
template <class T> T atomicCAS(T* p, T want, T v) {
  emu::step();
  const T old = *(volatile T*)p;
  return old == want ? emu_rmw(p, v, old) : old;
}
template <class T> T atomicAdd(T* p, T v) { emu::step(); const T o = *(volatile T*)p; return emu_rmw<T>(p, o + v, o); }
template <class T> T atomicSub(T* p, T v) { emu::step(); const T o = *(volatile T*)p; return emu_rmw<T>(p, o - v, o); }
template <class T> T atomicOr(T* p, T v) { emu::step(); const T o = *(volatile T*)p; return emu_rmw<T>(p, o | v, o); }
template <class T> T atomicExch(T* p, T v) { emu::step(); const T o = *(volatile T*)p; return emu_rmw<T>(p, v, o); }

namespace csmv {

using u64 = unsigned long long;
inline uint32_t lane_id() { return emu::cur->lane; }
inline uint32_t lanemask_lt() { return (1u << emu::cur->lane) - 1u; }
inline uint32_t ld_acquire_gpu(const uint32_t* p) { return emu::load(p, true); }
inline u64 ld_acquire_gpu(const u64* p) { return emu::load(p, true); }
inline uint32_t ld_relaxed_gpu(const uint32_t* p) { return emu::load(p); }
inline u64 ld_relaxed_gpu(const u64* p) { return emu::load(p); }
inline void st_release_gpu(uint32_t* p, uint32_t v) { emu::store(p, v); }
inline void st_release_gpu(u64* p, u64 v) { emu::store(p, v); }
inline void st_relaxed_gpu(uint32_t* p, uint32_t v) { emu::store(p, v); }
inline void st_relaxed_gpu(u64* p, u64 v) { emu::store(p, v); }
inline uint32_t atom_add_acquire_gpu(uint32_t* p, uint32_t v) { return atomicAdd(p, v); }
inline void ld_relaxed_gpu_v2(const u64* p, u64& a, u64& b) {
  a = emu::load(p);
  b = emu::load(p + 1);
}
inline uint4 ld_relaxed_gpu_v4(const uint4* p) {
  return {emu::load(&p->x), emu::load(&p->y), emu::load(&p->z), emu::load(&p->w)};
}
inline void st_relaxed_gpu_v4(uint4* p, uint4 v) {
  emu::store(&p->x, v.x);
  emu::store(&p->y, v.y);
  emu::store(&p->z, v.z);
  emu::store(&p->w, v.w);
}
inline void fence_acq_rel_gpu() { emu::fence(); }
inline void fence_sc_gpu() { emu::fence(); }
inline uint32_t ld_acquire_cta(const uint32_t* p) { return emu::load(p, true); }
inline void st_release_cta(uint32_t* p, uint32_t v) { emu::store(p, v); }
template <bool CLUSTER> uint32_t mail_acquire(const uint32_t* p) { return ld_acquire_cta(p); }
template <bool CLUSTER> void mail_release(uint32_t* p, uint32_t v) { st_release_cta(p, v); }
inline uint32_t ld_acquire_cluster(const uint32_t* p) { return emu::load(p, true); }
inline uint32_t ld_acquire_sys(const uint32_t* p) { return emu::load(p, true); }
inline void st_release_sys(uint32_t* p, uint32_t v) { emu::store(p, v); }
inline u64 globaltimer_ns() { return 0; }
inline void cp_async16(void*, const void*) { abort(); }
inline void cp_async_commit() { abort(); }
inline void cp_async_wait_all() { abort(); }
template <int N> void cp_async_wait_group() { abort(); }

enum : uint32_t {
  ERR_NONE = 0, ERR_WAIT_TURN = 1, ERR_WAIT_CLOCK = 2, ERR_WAIT_REPLY = 3, ERR_WAIT_REQUEST = 4,
  ERR_CAPACITY = 5, ERR_DATA = 6, ERR_LIVELOCK = 7, ERR_WAIT_FLOW = 8
};
inline void raise_error(uint32_t* err, uint32_t code) { atomicCAS(err, 0u, code); }
template <class Pred> bool bounded_wait(Pred pred, uint32_t* err, uint32_t code, uint32_t limit_log2) {
  for (uint64_t it = 0; it < 1ull << limit_log2; it++) {
    if (pred()) return true;
    if (ld_relaxed_gpu(err) != 0) return false;
    emu::pause();
  }
  raise_error(err, code);
  return false;
}
template <class Pred> bool bounded_wait_fast(Pred pred, uint32_t* err, uint32_t code, uint32_t limit_log2) {
  return bounded_wait(pred, err, code, limit_log2);
}

}  // namespace csmv
