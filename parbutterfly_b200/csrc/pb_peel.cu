// Tip (vertex) and wing (edge) peeling on the device.
//
// Semantics (Peel / PeelOrigParallel, butterfly_peel.h:647-711,896-934; PeelE /
// PeelEOrigParallel, butterfly_epeel.h:339-443,519-569; updateBuckets,
// butterfly_putils.h:1027-1115): items start in bucket D = their butterfly count.  Each round
// takes every unpeeled item whose bucket equals the current minimum k (the frontier):
//   tip : for each frontier vertex u and each two-hop neighbour u2 != u, the C(w(u,u2), 2)
//         shared butterflies leave u2's count;
//   wing: each butterfly that contains a frontier edge and no edge peeled in an earlier round
//         is removed once, by its frontier edge of smallest index, and its other edges lose 1.
// Every touched unpeeled item moves to bucket max(count, k).  Buckets are 64-bit (the
// reference's are 32-bit, ligra/bucket.h:15-16, exact only below 2^32 - 1).
//
// Device design: one cooperative persistent kernel runs all rounds.  A round has two phases, each
// closed by one grid barrier whose wait is bounded in time (on expiry the kernel records
// PB_ETIMEOUT and returns; the context stays usable):
//   F: the near list (the unpeeled items whose bucket lies below a window bound) is scanned; the
//      items of bucket k form the frontier, the least other bucket seeds the next minimum;
//   P: the frontier is processed.  The decrement that lowers an item's count also feeds the next
//      minimum and, when it is the one that crosses the window bound, adds the item to the near
//      list, so no pass over touched items follows.
// An item's bucket is max(count, k) (k: the last round's bucket), so it needs no storage.  The
// window advances (one pass over the alive list, a log2 histogram of distances to the minimum)
// when the near list runs dry.
//
// What bounds it: most rounds are light (a few items, 2^12 .. 2^17 probes), so a round's time is
// its chain of dependent L2 round trips (about 0.35 us each) plus the barriers, not its probes.
// The phases are therefore cut to short chains: probes that hit go to a queue of the warp and are
// charged 32 at a time (one chain per 32 hits instead of one per probe step with a hit), a
// barrier is one release add and one acquire poll, and per-round statistics stay in shared
// memory.
#include <algorithm>
#include <functional>
#include <memory>
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "pb_engine.cuh"
#include "pb_prims.cuh"

namespace pb {

namespace {

constexpr int kPT = 512;
constexpr int kPW = kPT / 32;
// Shared-memory table area of a CTA, in 32-bit words (84 KiB; with the fixed part two CTAs fit an
// SM).  Wing: keys, values and hit counters (three equal parts, per CTA or per warp); tip: keys
// and values (power-of-two parts).
constexpr uint32_t kPoolWords = 21504;
constexpr uint32_t kWingSlots = kPoolWords / 3;            // 7168 slots, probe sets up to kWingSet
constexpr uint32_t kWingSet = 4096;
constexpr uint32_t kWingLoad = 4;  // slots per probe-set entry, while they fit
constexpr uint32_t kWingWarpSlots = kPoolWords / 3 / kPW;  // 448 slots, probe sets up to kWingWarpSet
constexpr uint32_t kWingWarpSet = 256;
constexpr uint32_t kTipSlots = 8192;      // two-hop lists of up to 4096 wedges
constexpr uint32_t kTipWarpSlots = 512;   // two-hop lists of up to 256 wedges; 512 with one-word entries
constexpr uint32_t kTipWindow = 2 * kPoolWords;  // 16-bit counters of a window
constexpr int64_t kTipWindows = 4, kTipWindowWedges = 4096;
constexpr uint32_t kEmpty = 0xFFFFFFFFu;
constexpr unsigned long long kInf = ~0ull;
// Item states.  The frontier of round r is marked 1 + (r & 1); the next round turns the marks
// into PEELED, so a mark never outlives the round after its own.
constexpr uint8_t ALIVE = 0, PEELED = 3;
constexpr unsigned ERR_TIMEOUT = 1u;
constexpr unsigned long long kBarrierTimeoutNs = 60ull * 1000000000ull;  // 60 s per wait
constexpr unsigned long long kBarErr = 1ull << 63;  // barrier word: some wait or invariant failed

struct Ctl {
  unsigned long long nm[2];       // next minimum per round parity
  unsigned long long k_lo, win_hi;
  unsigned long long rounds, work;
  // Frontier lists per round parity: items in the high word, their work units in the low word, so
  // that one add gives an item its position and its first unit (units ascend with positions).
  unsigned long long fsmall[2], fbig[2], fhuge[2];
  unsigned cur_small[2], cur_big[2], cur_huge[2];
  unsigned long long huge_sum[2], huge_max[2];  // two-hop lengths of the heavy tip items
  unsigned long long round_est[2];   // summed cost estimate of the round (range mode, tracing)
  unsigned long long near_len;
  unsigned near_done;             // range mode: near items already taken (kept across launches)
  unsigned alive;                 // unpeeled items (written when the kernel ends or pauses)
  unsigned alen[2];               // alive list lengths
  unsigned hist[66];
  unsigned err;
  unsigned long long bar;       // arrivals at grid barriers since the control block was made
  unsigned long long bar_base;  // bar when the current launch began
  unsigned long long round;   // next round to run (kept across launches)
  unsigned alist_cur;         // current alive list (kept across launches)
  unsigned started;           // alive list initialised
  unsigned alive_at_compact;  // unpeeled items when the lists were last compacted
  unsigned min_gain;          // pause for compaction once this many more items are peeled
  // Instrumentation (CTA 0): device time per phase and work counters.
  unsigned trace;                          // phase times are kept
  unsigned long long phase_ns[3];          // advance, F, P
  unsigned long long barrier_timeout_ns;   // bound of every grid-barrier wait
  unsigned test_skip_arrival;              // test hook: CTA 0 never arrives at grid barriers
  unsigned long long scanned, n_small, n_big, n_huge, advances;
  // Phase-P time of the rounds binned by log2 of their estimated work (frontier cost sum).
  unsigned long long pbin_ns[42], pbin_rounds[42], pbin_est[42];
  // Near-window size: at least near_min items, or alive / near_div.
  unsigned near_min, near_div;
  // Range mode (the coarse pass of the two-phase peel): each window is one partition, its
  // frontier every unpeeled item whose count is below the window bound, repeated until no
  // unpeeled item is below it.  The bound is chosen so that the window holds about
  // part_target of estimated work.  npart counts the partitions opened so far.
  unsigned range_mode, npart;
  unsigned long long part_target;  // base target per partition
  // Partitions grow past their opening bound (items fall below it while the partition peels):
  // part_done sums the estimated work actually peeled, part_used the target the partition was
  // opened with, part_ratio_q (x256, smoothed) their ratio, which scales the next target down.
  unsigned long long part_done, part_used, part_ratio_q;
  unsigned long long whist[66];    // estimated work per log2 distance bin
  unsigned long long wsub[256];    // estimated work per linear sub-bin of the chosen octave
  // Wing items per probe structure (warp table, CTA table, dense markers) and their probes;
  // probes that walked the probe set against a binary search (the reverse direction).
  unsigned long long mode_items[3], mode_work[3], rev_work;
};
constexpr unsigned kMaxGroups = 128;  // heavy tip items of one wave
constexpr unsigned kFlatAll = 32;     // rounds of at most this many CTA-level tip items run as one wave
// Pairs per CTA below which tip_items_flat uses fewer CTAs.
constexpr unsigned long long kFlatPairs = 1024;
// Device memory for grid-shared dense counters (one n-sized slice per concurrent heavy tip
// item or per fine-pass instance with a CTA range of its own).
constexpr int64_t kGsharedBudget = int64_t(2) << 30;


// Live adjacency of both sides.  Lists are compacted to their live entries between launches
// of the peeling kernel, so list positions are not edge ids: eidK / eidC carry the output
// edge index of every entry.
struct Lists {
  const uint32_t* offK;  // count side: vertex -> centre ids
  const uint32_t* edgK;
  const uint32_t* eidK;  // count-side entry -> output edge index (wing only)
  const uint32_t* offC;  // centre side: vertex -> count-side ids
  const uint32_t* edgC;
  const uint32_t* eidC;  // centre-side entry -> output edge index (wing only)
  const uint32_t* center_of;  // output edge index -> centre vertex (wing only)
  const uint32_t* u_of;       // output edge index -> count-side vertex (wing only)
  const int64_t* S;      // per count-side vertex then per centre vertex: sum of neighbour degrees (wing)
  const int64_t* wk;     // per count-side vertex: two-hop wedges sum(deg(v) - 1) (tip)
  const uint32_t* info;  // per edge (wing): how its item is peeled (wing_info_kernel)
  int64_t nK, nC;
};
// Lists::info: work units of the item, whether it runs on warps, whether it walks from the centre.
constexpr int64_t kUnitSets = 2;
constexpr uint32_t kInfoUnits = 0x1FFFu, kInfoSmall = 1u << 13, kInfoFromV = 1u << 31;

struct Work {
  int64_t* D;        // final tip / wing numbers (range mode: the counts when the partition opened)
  int64_t* cnt;      // butterfly counts
  uint8_t* state;
  uint32_t* alist[2];
  uint32_t* near;
  // Frontier of a round, per parity: warp-level items from the front, CTA-level items from the
  // back (an item is in one of them).  What phase P needs of an item is written once by phase F:
  // wing: {edge, probe vertex a | from_v << 31, first-level vertex b, first unit}; tip: {vertex,
  // its list start, its degree, two-hop list length (saturated)}.
  uint4* front[2];
  uint4* fhuge[2];       // tip only
  uint32_t* gshared;     // tip: ngroups slices of gshared_stride grid-shared dense counters (zeroed)
  int64_t gshared_stride;
  unsigned ngroups;
  uint32_t* gscratch;  // per-CTA dense scratch (dense counters / probe markers)
  int64_t gscratch_len;
  int tip_cb;          // count bits of a one-word tip table entry (beside a count-side vertex)
  int64_t N;           // items of this instance
  uint32_t item0;      // first item of this instance: its items are items[item0 .. item0 + N)
                       // (item0 .. item0 + N - 1 themselves when items is null)
  const uint32_t* items;
  // Two-phase peel.  Fine pass: every instance is one partition of the coarse pass; part[x]
  // is the partition of item x and my_part this instance's.  Items of lower partitions are
  // peeled, items of higher partitions stay unpeeled for the whole pass (and are never
  // charged), items of my_part follow the exact rounds.  Coarse pass: part_out receives the
  // partition of every item as it is peeled.  level: the live-list version the instance reads.
  const uint32_t* part;
  uint32_t my_part;
  uint32_t* part_out;
  uint32_t level;
  const uint32_t* wgt;  // coarse pass: every item's estimated work (item_weight, capped at 2^32 - 1)
};

// Every CTA belongs to one peel instance (the whole input, or one graph of a batch, each with
// its own control block, lists and rounds): its index within the instance and the instance's
// CTA count, set at kernel start.
__shared__ unsigned s_vb, s_vg;
__device__ __forceinline__ unsigned vblock() { return s_vb; }
__device__ __forceinline__ unsigned vgrid() { return s_vg; }

// Per-CTA copies of the round's parameters (set at the start of every round) and of the
// instance's barrier state.
__shared__ unsigned long long s_win_hi;
__shared__ long long s_k;
__shared__ unsigned s_act;  // state mark of this round's frontier
__shared__ unsigned long long s_bar_target, s_bar_timeout;
__shared__ unsigned s_err, s_skip_arrival, s_trace;

// Statistics of CTA 0 (phase times, round counts) and of every CTA (wing probes), written to the
// control block when the instance ends or pauses.
struct Stats {
  unsigned long long t_last, phase_ns[3];
  unsigned long long pbin_ns[42], pbin_rounds[42], pbin_est[42];
  unsigned long long rounds, scanned, n_small, n_big, n_huge, advances, part_done;
  unsigned long long mode_items[3], mode_work[3], rev_work;
};
__shared__ Stats s_st;

__device__ __forceinline__ unsigned long long globaltimer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// CTA 0 charges the time since its previous mark to phase `ph` (called right after barriers).
// Phase P is also binned by log2 of the round's estimated work (est).
__device__ __forceinline__ void phase_mark(bool trace, int ph, unsigned long long est = 0) {
  if (trace && threadIdx.x == 0) {
    const unsigned long long now = globaltimer_ns();
    if (s_st.t_last) {
      s_st.phase_ns[ph] += now - s_st.t_last;
      if (ph == 2) {
        const int b = est ? min(41, 64 - __clzll(est)) : 0;
        s_st.pbin_ns[b] += now - s_st.t_last;
        s_st.pbin_rounds[b] += 1;
        s_st.pbin_est[b] += est;
      }
    }
    s_st.t_last = now;
  }
}

// Records an error and makes every barrier of the instance fail from here on.
__device__ __noinline__ void raise_err(Ctl* ctl, unsigned code) {
  atomicOr(&ctl->err, code);
  atomicOr(&ctl->bar, kBarErr);
  *(volatile unsigned*)&s_err = 1u;
}

// Control-block words every thread needs after a barrier: read by one warp per CTA (thousands of
// warps reading one address queue up at its L2 slice) and handed on through shared memory.
__shared__ unsigned long long s_words[3];

// Barrier over the CTAs of one peel instance (a cooperative launch keeps every CTA co-resident).
// Arrivals are counted in one 64-bit word that is never reset: a barrier is complete when the
// word reaches the CTA count times the number of barriers so far, so it costs one release add and
// the acquire polls of the word (1.4 us on 148 CTAs).  Bounded: a wait longer than the control block's
// timeout sets ERR_TIMEOUT and returns false.
// w0 .. w2: control-block words that land in s_words (null: none).
__device__ __forceinline__ bool grid_barrier(Ctl* ctl, const unsigned long long* w0 = nullptr,
                                             const unsigned long long* w1 = nullptr,
                                             const unsigned long long* w2 = nullptr) {
  int bad = 0;
  __syncthreads();
  if (threadIdx.x < 32) {
    if (vgrid() == 1) {  // one CTA: a block barrier orders its global memory accesses too
      bad = (int)*(volatile unsigned*)&s_err;
    } else if (threadIdx.x == 0) {
      const unsigned long long target = s_bar_target + vgrid();
      s_bar_target = target;
      // (test hook) without CTA 0's arrivals no barrier completes, so every wait runs out.
      if (!s_skip_arrival)
        asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(&ctl->bar), "l"(1ull) : "memory");
      unsigned long long t0 = 0, seen;
      unsigned polls = 0;
      while (true) {
        asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(seen) : "l"(&ctl->bar) : "memory");
        if (seen >= target) break;  // the error bit is above every count
        if ((++polls & 63u) == 0) {
          const unsigned long long now = globaltimer_ns();
          if (!t0) t0 = now;
          else if (now - t0 > s_bar_timeout) raise_err(ctl, ERR_TIMEOUT);
        }
      }
      bad = (seen & kBarErr) != 0;
    }
    if (w0) {
      __syncwarp();
      const unsigned long long* w = threadIdx.x == 0 ? w0 : (threadIdx.x == 1 ? w1 : w2);
      if (threadIdx.x < 3 && w) s_words[threadIdx.x] = *(const volatile unsigned long long*)w;
    }
  }
  return __syncthreads_or(bad) == 0;
}

// Fibonacci hashing: the high bits of key * 2^32/phi, folded into the table size (any size).
__device__ __forceinline__ uint32_t hslot(uint32_t key, uint32_t size) { return __umulhi(key * 0x9E3779B1u, size); }

// Tables hold at most 4/7 of their slots, so probe sequences stay shorter than the table; the
// bounds turn a broken invariant into a recorded error, not an endless loop.
constexpr unsigned ERR_TABLE = 2u;

__device__ __forceinline__ void t_add(uint32_t* keys, uint32_t* vals, uint32_t size, uint32_t key, Ctl* ctl) {
  uint32_t h = hslot(key, size);
  for (uint32_t probes = 0; probes < size; ++probes) {
    uint32_t k = keys[h];
    if (k == key) { atomicAdd(&vals[h], 1u); return; }
    if (k == kEmpty) {
      uint32_t prev = atomicCAS(&keys[h], kEmpty, key);
      if (prev == kEmpty || prev == key) { atomicAdd(&vals[h], 1u); return; }
    }
    h = h + 1 == size ? 0u : h + 1;
  }
  raise_err(ctl, ERR_TABLE);
}

// The same with one-word entries (key << cb | count; counts of at most 2^cb - 2).
__device__ __forceinline__ void t_add1(uint32_t* tab, uint32_t size, int cb, uint32_t key, Ctl* ctl) {
  uint32_t h = hslot(key, size);
  for (uint32_t probes = 0; probes < size; ++probes) {
    uint32_t k = tab[h];
    if (k == kEmpty) {
      k = atomicCAS(&tab[h], kEmpty, (key << cb) | 1u);
      if (k == kEmpty) return;
    }
    if ((k >> cb) == key) { atomicAdd(&tab[h], 1u); return; }
    h = h + 1 == size ? 0u : h + 1;
  }
  raise_err(ctl, ERR_TABLE);
}

// Unique-key insert of (key, val).
__device__ __forceinline__ void t_put(uint32_t* keys, uint32_t* vals, uint32_t size, uint32_t key, uint32_t val,
                                      Ctl* ctl) {
  uint32_t h = hslot(key, size);
  for (uint32_t probes = 0; probes < size; ++probes) {
    uint32_t prev = atomicCAS(&keys[h], kEmpty, key);
    if (prev == kEmpty) { vals[h] = val; return; }
    h = h + 1 == size ? 0u : h + 1;
  }
  raise_err(ctl, ERR_TABLE);
}

// The same from slot h on, which neither matched nor was empty.
__device__ __forceinline__ uint32_t t_slot_next(const uint32_t* keys, uint32_t size, uint32_t key, uint32_t h) {
  for (uint32_t probes = 1; probes < size; ++probes) {
    h = h + 1 == size ? 0u : h + 1;
    const uint32_t k = keys[h];
    if (k == key) return h;
    if (k == kEmpty) return kEmpty;
  }
  return kEmpty;
}

// Slot of key, or kEmpty when absent.
__device__ __forceinline__ uint32_t t_slot(const uint32_t* keys, uint32_t size, uint32_t key) {
  uint32_t h = hslot(key, size);
  for (uint32_t probes = 0; probes < size; ++probes) {
    const uint32_t k = keys[h];
    if (k == key) return h;
    if (k == kEmpty) return kEmpty;
    h = h + 1 == size ? 0u : h + 1;
  }
  return kEmpty;
}

__device__ __forceinline__ uint32_t np2(uint32_t x) { return x <= 1 ? 1u : 1u << (32 - __clz(x - 1)); }

constexpr uint32_t kQueue = 64;         // entries of a warp's queue (31 left over + 32 pushed)
struct Shared {
  unsigned long long red[32];
  unsigned long long queue[kPW][kQueue];
  uint32_t incl[kPT];
  uint32_t sb[kPT];
  uint32_t len[kPT];
  uint32_t acc[kPT];  // butterflies found through each first-level position of the chunk
  uint4 flat[kMaxGroups];  // tip_items_flat: the items of the wave
  unsigned long long flat_end[kMaxGroups];
  uint32_t scan[32];
  uint32_t item;
  uint32_t list_steps[kPW], list_item[kPW];  // tip_items_lists: the same per warp
  uint32_t flat_steps, flat_item;  // tip_items_flat: steps of this CTA's slice, item of a one-step slice
  unsigned hist[66];
};

// A second-level position with this bit set walks the probe set instead (the reverse direction of
// a wing intersection); list positions stay below 2^31 (2m <= 2^32).
constexpr uint32_t kRevFlag = 0x80000000u;

// A queue of 64-bit entries private to one warp.  push() is called by all lanes; once 32 entries
// are waiting the warp handles them with all lanes at work: f(entry) per lane.  n is the same in
// every lane.
struct WarpQueue {
  unsigned long long* buf;
  unsigned n;
  template <class F>
  __device__ __forceinline__ void push(bool have, unsigned long long x, F&& f) {
    const unsigned bal = __ballot_sync(0xffffffffu, have);
    if (!bal) return;
    if (have) buf[n + __popc(bal & ((1u << lane_id()) - 1u))] = x;
    n += __popc(bal);
    __syncwarp();
    if (n >= 32) {
      n -= 32;
      f(buf[n + lane_id()]);
      __syncwarp();
    }
  }
  template <class F>
  __device__ __forceinline__ void flush(F&& f) {
    __syncwarp();
    if (lane_id() < n) f(buf[lane_id()]);
    n = 0;
    __syncwarp();
  }
};

// Position of this lane's entry in a list of *len entries that the lanes with `have` append to: one
// add per warp (all lanes call it).
template <class T>
__device__ __forceinline__ T warp_append(T* len, bool have) {
  const unsigned bal = __ballot_sync(0xffffffffu, have);
  T base = 0;
  if (bal && lane_id() == (unsigned)(__ffs(bal) - 1)) base = atomicAdd(len, (T)__popc(bal));
  base = __shfl_sync(0xffffffffu, base, bal ? __ffs(bal) - 1 : 0);
  return base + (T)__popc(bal & ((1u << lane_id()) - 1u));
}

// bins[bin] += w (bin < 0: nothing), equal bins of a warp in one shared-memory add: neighbouring
// items lie in few bins, and 64-bit shared-memory adds to one address are served one by one.
__device__ __forceinline__ void warp_bin_add(unsigned long long* bins, int bin, uint32_t w) {
  const unsigned peers = __match_any_sync(0xffffffffu, bin);
  const uint32_t lo = __reduce_add_sync(peers, w & 0xFFFFu), hi = __reduce_add_sync(peers, w >> 16);
  if (bin >= 0 && lane_id() == (unsigned)(__ffs(peers) - 1))
    atomicAdd(&bins[bin], ((unsigned long long)hi << 16) + lo);
}

// The first of `nbins` control-block bins whose running sum (from `cum` on) reaches target, nbins when
// none does, for the whole CTA; cum becomes the sum of the bins before it.  One warp loads the bins
// together: walked one by one, every bin is a round trip (84 us of an advance).
__shared__ unsigned s_bin;
__shared__ unsigned long long s_cum;
template <class T>
__device__ __forceinline__ unsigned find_bin(const T* bins, unsigned nbins, unsigned long long target,
                                             unsigned long long& cum) {
  if (threadIdx.x < 32) {
    const unsigned per = (nbins + 31) / 32, b0 = threadIdx.x * per;
    T v[8];
    unsigned long long sum = 0;
#pragma unroll
    for (unsigned i = 0; i < 8; ++i) {
      v[i] = i < per && b0 + i < nbins ? *(const volatile T*)&bins[b0 + i] : T(0);
      sum += v[i];
    }
    const unsigned long long incl = warp_inclusive_scan(sum) + cum;
    const unsigned reach = __ballot_sync(0xffffffffu, incl >= target);
    if (reach ? threadIdx.x == (unsigned)(__ffs(reach) - 1) : threadIdx.x == 31) {
      unsigned long long run = incl - sum;
      unsigned b = nbins;
#pragma unroll
      for (unsigned i = 0; i < 8; ++i) {
        if (b == nbins && i < per && b0 + i < nbins) {
          if (run + v[i] >= target) b = b0 + i;
          else run += v[i];
        }
      }
      s_bin = b;
      s_cum = run;
    }
  }
  __syncthreads();
  cum = s_cum;
  return s_bin;
}

// Flattened two-level iteration by one warp: first(j, L, sb) gives the second-level range
// [sb, sb + L) of first-level position j in [b, e) (all lanes call it; valid: j < e); f(valid, lo,
// q, x) gets the pairs of position j0 + lo, four steps of 32 loads at a time, and done() runs
// after the last pair of each chunk of 32 positions (all lanes call both).
template <class First, class F, class Done>
__device__ __forceinline__ void warp_iter(uint32_t b, uint32_t e, const uint32_t* __restrict__ arr, First&& first, F&& f,
                                          Done&& done) {
  const unsigned lane = lane_id();
  for (uint32_t j0 = b; j0 < e; j0 += 32) {
    const uint32_t j = j0 + lane;
    uint32_t L = 0, sb = 0;
    first(j, j < e, L, sb);
    const uint32_t incl = warp_inclusive_scan(L);
    const uint32_t excl = incl - L;
    const uint32_t T = __shfl_sync(0xffffffffu, incl, 31);
    for (uint32_t t0 = 0; t0 < T; t0 += 128) {
      uint32_t q[4], x[4], at[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const uint32_t t = t0 + 32 * r + lane;
        uint32_t lo = 0;
#pragma unroll
        for (uint32_t step = 16; step > 0; step >>= 1) {
          uint32_t y = __shfl_sync(0xffffffffu, incl, lo + step - 1);
          if (y <= t) lo += step;
        }
        const uint32_t ex = __shfl_sync(0xffffffffu, excl, lo);
        const uint32_t s = __shfl_sync(0xffffffffu, sb, lo);
        at[r] = lo;
        q[r] = s + (t - ex);
        x[r] = t < T ? arr[q[r] & ~kRevFlag] : 0u;
      }
#pragma unroll
      for (int r = 0; r < 4; ++r)
        if (t0 + 32 * r < T) f(t0 + 32 * r + lane < T, at[r], q[r], x[r]);
    }
    done();
  }
}

// Inclusive scan over the CTA; smem (32 words) may be used again after the caller's next barrier.
__device__ __forceinline__ uint32_t block_incl_scan(uint32_t x, uint32_t* smem, uint32_t& total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const uint32_t incl = warp_inclusive_scan(x);
  if (lane == 31) smem[warp] = incl;
  __syncthreads();
  const uint32_t v = warp_inclusive_scan(lane < nwarps ? smem[lane] : 0u);  // by every warp
  total = __shfl_sync(0xffffffffu, v, nwarps - 1);
  const uint32_t before = __shfl_sync(0xffffffffu, v, warp > 0 ? warp - 1 : 0);
  return incl + (warp > 0 ? before : 0u);
}

// The same iteration by the whole CTA.  Each chunk of kPT first-level positions has its
// second-level ranges cut into pieces of at most kPiece entries; pieces go to the warps in turn
// (they are of one size, so no counter is needed), a warp locates a piece's position once (two
// ballots over the chunk's inclusive piece counts) and walks it with 32 lanes, so consecutive lanes
// read consecutive entries.  piece(lo, k, q, n, x): a piece of position j0 + lo; this lane holds its
// entries k, k + 32, ... below n, at list positions q, q + 32, ..., with values x[0 .. 3] (kEmpty
// beyond the end).
constexpr uint32_t kPiece = 128;

// One warp's part of the pieces of up to 32 positions (lens / starts in shared memory): every warp
// scans the piece counts by itself, so no barrier is needed.
template <class Piece>
__device__ __forceinline__ void few_pieces(uint32_t n, const uint32_t* lens, const uint32_t* starts,
                                           const uint32_t* __restrict__ arr, Piece&& piece) {
  const uint32_t lane = lane_id();
  const uint32_t len = lane < n ? lens[lane] : 0u, beg = lane < n ? starts[lane] : 0u;
  const uint32_t incl = warp_inclusive_scan((len + kPiece - 1) / kPiece);
  const uint32_t T = __shfl_sync(0xffffffffu, incl, 31);
  for (uint32_t p = threadIdx.x >> 5; p < T; p += kPW) {
    const uint32_t lo = (uint32_t)__ffs(__ballot_sync(0xffffffffu, incl > p)) - 1u;
    const uint32_t before = __shfl_sync(0xffffffffu, incl, lo > 0 ? lo - 1 : 0);
    const uint32_t k0 = (p - (lo > 0 ? before : 0u)) * kPiece;
    const uint32_t kend = min(k0 + kPiece, __shfl_sync(0xffffffffu, len, lo));
    const uint32_t sbj = __shfl_sync(0xffffffffu, beg, lo), base = sbj & ~kRevFlag;
    uint32_t x[kPiece / 32];
#pragma unroll
    for (uint32_t r = 0; r < kPiece / 32; ++r) {
      const uint32_t k = k0 + lane + 32 * r;
      x[r] = k < kend ? arr[base + k] : kEmpty;
    }
    piece(lo, k0 + lane, sbj + k0 + lane, kend, x);
  }
}

template <class First, class Piece, class Done>
__device__ __forceinline__ void block_pieces(uint32_t b, uint32_t e, Shared& S, const uint32_t* __restrict__ arr,
                                             First&& first, Piece&& piece, Done&& done) {
  const uint32_t tid = threadIdx.x, lane = tid & 31u;
  for (uint32_t j0 = b; j0 < e; j0 += kPT) {
    const uint32_t j = j0 + tid;
    uint32_t L = 0, sb = 0;
    first(j, j < e, L, sb);
    uint32_t T;
    const uint32_t incl = block_incl_scan((L + kPiece - 1) / kPiece, S.scan, T);
    S.incl[tid] = incl;
    S.sb[tid] = sb;
    S.len[tid] = L;
    __syncthreads();
    for (uint32_t p = tid >> 5; p < T; p += kPW) {
      // The first position whose inclusive count exceeds p, in two ballots.
      const unsigned ge = __ballot_sync(0xffffffffu, S.incl[lane * kPW + kPW - 1] > p);
      uint32_t lo = (__ffs(ge) - 1) * kPW;
      const unsigned in = __ballot_sync(0xffffffffu, lane < kPW && S.incl[lo + (lane & (kPW - 1))] > p);
      lo += __ffs(in) - 1;
      const uint32_t k0 = (p - (lo ? S.incl[lo - 1] : 0u)) * kPiece;
      const uint32_t kend = min(k0 + kPiece, S.len[lo]);
      const uint32_t sbj = S.sb[lo], base = sbj & ~kRevFlag;
      // A piece is 4 x 32 entries: every lane issues its 4 loads before it uses any of them.
      uint32_t x[kPiece / 32];
#pragma unroll
      for (uint32_t r = 0; r < kPiece / 32; ++r) {
        const uint32_t k = k0 + lane + 32 * r;
        x[r] = k < kend ? arr[base + k] : kEmpty;
      }
      piece(lo, k0 + lane, sbj + k0 + lane, kend, x);
    }
    done();
  }
}


// The same with f(valid, lo, q, x) per step of 32 entries.
template <class First, class F, class Done>
__device__ __forceinline__ void block_iter(uint32_t b, uint32_t e, Shared& S, const uint32_t* __restrict__ arr,
                                           First&& first, F&& f, Done&& done) {
  block_pieces(b, e, S, arr, first, [&](uint32_t lo, uint32_t k, uint32_t q, uint32_t n, const uint32_t* x) {
#pragma unroll
    for (uint32_t r = 0; r < kPiece / 32; ++r)
      if ((k & ~31u) + 32 * r < n) f(k + 32 * r < n, lo, q + 32 * r, x[r]);
  }, done);
}

// The same iteration restricted to flattened pair indices [lo, hi) (counted from the first
// pair of [b, e)); every CTA takes one slice of a heavy item.  Four pairs per thread are loaded
// before any of them is used.
template <class First, class F>
__device__ __forceinline__ void block_iter_range(uint32_t b, uint32_t e, Shared& S, const uint32_t* __restrict__ arr,
                                                 uint64_t lo, uint64_t hi, First&& first, F&& f) {
  const uint32_t tid = threadIdx.x;
  uint64_t base = 0;
  for (uint32_t j0 = b; j0 < e && base < hi; j0 += kPT) {
    const uint32_t j = j0 + tid;
    uint32_t L = 0, sb = 0;
    first(j, j < e, L, sb);
    uint32_t T;
    const uint32_t incl = block_incl_scan(L, S.scan, T);
    S.incl[tid] = incl;
    S.sb[tid] = sb;
    __syncthreads();
    const uint64_t tb = lo > base ? lo - base : 0;
    const uint64_t te = (hi - base) < (uint64_t)T ? (hi - base) : (uint64_t)T;
    for (uint64_t t0 = tb; t0 < te; t0 += 4 * kPT) {
      uint32_t x[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const uint64_t tt = t0 + (uint64_t)r * kPT + tid;
        x[r] = kEmpty;
        if (tt < te) {
          const uint32_t t = (uint32_t)tt;
          uint32_t lo2 = 0;
#pragma unroll
          for (uint32_t step = kPT / 2; step > 0; step >>= 1)
            if (S.incl[lo2 + step - 1] <= t) lo2 += step;
          x[r] = arr[S.sb[lo2] + (t - (lo2 ? S.incl[lo2 - 1] : 0u))];
        }
      }
      f(x);
    }
    __syncthreads();
    base += T;
  }
}

// What a thread gathers during a phase P: the least bucket it moved an item to, and the wedges
// or probes it processed.
struct Acc {
  unsigned long long mn;
  unsigned long long work;
};

__device__ __forceinline__ bool mine(const Work& W, uint32_t x) { return !W.part || W.part[x] == W.my_part; }

// Removes `amount` butterflies from item x, which is unpeeled and of this instance.  The decrement
// whose result first lies below the window bound adds the item to the near list (counts only
// fall, so exactly one decrement crosses); items above the bound cannot reach the frontier before
// the next window advance, which reads their counts.
__device__ __forceinline__ long long dec_add(const Work& W, uint32_t x, int64_t amount) {
  return (long long)atomicAdd(reinterpret_cast<unsigned long long*>(&W.cnt[x]), (unsigned long long)(-amount));
}

// What follows the add that returned `old`.
__device__ __forceinline__ void dec_done(const Work& W, Ctl* ctl, Acc& A, uint32_t x, int64_t amount, long long old) {
  const unsigned long long nb = (unsigned long long)max(old - amount, s_k);
  if (nb < s_win_hi) {
    A.mn = min(A.mn, nb);
    if ((unsigned long long)max(old, s_k) >= s_win_hi) W.near[atomicAdd(&ctl->near_len, 1ull)] = x;
  }
}

__device__ __forceinline__ void dec_known(const Work& W, Ctl* ctl, Acc& A, uint32_t x, int64_t amount) {
  dec_done(W, ctl, A, x, amount, dec_add(W, x, amount));
}

__device__ __forceinline__ void dec(const Work& W, Ctl* ctl, Acc& A, uint32_t x, int64_t amount) {
  if (W.state[x] == ALIVE && mine(W, x)) dec_known(W, ctl, A, x, amount);
}

// ---- tip: process one frontier vertex -------------------------------------------------------
struct TipFirst {
  const Lists& G;
  __device__ __forceinline__ void operator()(uint32_t j, bool valid, uint32_t& L, uint32_t& sb) const {
    if (!valid) return;
    const uint32_t v = G.edgK[j];
    sb = G.offC[v];
    L = G.offC[v + 1] - sb;
  }
};

__device__ __forceinline__ bool tip_one_word(const Work& W, uint32_t deg) { return deg < (1u << W.tip_cb) - 1u; }

// Queue entries of tip items: (u2, w) with w wedges to u2.
__device__ __forceinline__ void tip_charge(const Work& W, Ctl* ctl, Acc& A, unsigned long long x) {
  const int64_t w = (int64_t)(x >> 32);
  dec(W, ctl, A, (uint32_t)x, w * (w - 1) / 2);
}

// Table: 2 kTipWarpSlots words.  Entries are one word (u2 << cb | count) when the count, at most the
// degree, fits beside the vertex.
__device__ void tip_item_warp(const Lists& G, const Work& W, Ctl* ctl, const uint4& it, uint32_t* keys, WarpQueue& Q,
                              Acc& A) {
  const unsigned lane = lane_id();
  const uint32_t u = it.x;
  const int64_t wk = G.wk[u];
  const int cb = tip_one_word(W, it.z) ? W.tip_cb : 0;
  uint32_t* vals = keys + kTipWarpSlots;  // two-array tables
  const uint32_t tsize = max(64u, cb ? 2u * (uint32_t)wk : np2(2u * (uint32_t)wk));
  for (uint32_t s = lane; s < tsize; s += 32) {
    keys[s] = kEmpty;
    if (!cb) vals[s] = 0;
  }
  __syncwarp();
  warp_iter(it.y, it.y + it.z, G.edgC, TipFirst{G},
            [&](bool valid, uint32_t, uint32_t, uint32_t u2) {
              if (!valid || u2 == u) return;
              if (cb) t_add1(keys, tsize, cb, u2, ctl);
              else t_add(keys, vals, tsize, u2, ctl);
            },
            [] {});
  __syncwarp();
  auto charge = [&](unsigned long long x) { tip_charge(W, ctl, A, x); };
  for (uint32_t s0 = 0; s0 < tsize; s0 += 32) {
    const uint32_t s = s0 + lane;
    const uint32_t k = s < tsize ? keys[s] : kEmpty;
    const uint32_t w = k == kEmpty ? 0u : (cb ? k & ((1u << cb) - 1u) : vals[s]);
    Q.push(w >= 2, ((unsigned long long)w << 32) | (k >> cb), charge);
  }
  Q.flush(charge);
  if (lane == 0) A.work += (unsigned long long)wk;
}

__device__ void tip_item_block(const Lists& G, const Work& W, Ctl* ctl, uint32_t u, uint32_t* table, Shared& S,
                               WarpQueue& Q, Acc& A) {
  const int64_t wk = G.wk[u];
  const bool hash = (uint64_t)2 * (uint64_t)wk <= (uint64_t)kTipSlots;
  const uint32_t deg = G.offK[u + 1] - G.offK[u];
  // Longer lists: 16-bit counters in shared memory over windows of the vertices, when that takes few
  // windows for the list's length (no atomic leaves the SM); else counters in global memory.
  const int64_t nwin = (G.nK + kTipWindow - 1) / kTipWindow;
  if (!hash && deg <= 0xFFFFu && nwin <= kTipWindows && wk > nwin * kTipWindowWedges) {
    auto charge = [&](unsigned long long x) { tip_charge(W, ctl, A, x); };
    for (int64_t w0 = 0; w0 < G.nK; w0 += kTipWindow) {
      const uint32_t base = (uint32_t)w0, len = (uint32_t)min((int64_t)kTipWindow, G.nK - w0), words = (len + 1) / 2;
      for (uint32_t s = threadIdx.x; s < words; s += kPT) table[s] = 0;
      __syncthreads();
      block_pieces(G.offK[u], G.offK[u + 1], S, G.edgC, TipFirst{G},
                   [&](uint32_t, uint32_t, uint32_t, uint32_t, const uint32_t* x) {
#pragma unroll
                     for (uint32_t r = 0; r < kPiece / 32; ++r) {
                       const uint32_t i = x[r] - base;  // kEmpty lies above every window
                       if (i < len && x[r] != u) atomicAdd(&table[i >> 1], 1u << (16 * (i & 1u)));
                     }
                   },
                   [] { __syncthreads(); });
      __syncthreads();
      for (uint32_t s0 = 0; s0 < words; s0 += kPT) {
        const uint32_t s = s0 + threadIdx.x, c = s < words ? table[s] : 0u;
        Q.push((c & 0xFFFFu) >= 2, ((unsigned long long)(c & 0xFFFFu) << 32) | (base + 2 * s), charge);
        Q.push((c >> 16) >= 2, ((unsigned long long)(c >> 16) << 32) | (base + 2 * s + 1), charge);
      }
      Q.flush(charge);
      __syncthreads();
    }
    if (threadIdx.x == 0) A.work += (unsigned long long)wk;
    return;
  }
  uint32_t* keys = table;
  uint32_t* vals = table + kTipSlots;
  uint32_t* gcnt = W.gscratch + (size_t)blockIdx.x * (size_t)W.gscratch_len;
  const uint32_t tsize = hash ? max(64u, np2(2u * (uint32_t)wk)) : 0u;
  if (hash)
    for (uint32_t s = threadIdx.x; s < tsize; s += kPT) { keys[s] = kEmpty; vals[s] = 0; }
  __syncthreads();
  auto charge = [&](unsigned long long x) { tip_charge(W, ctl, A, x); };
  const auto done = [] { __syncthreads(); };
  block_iter(G.offK[u], G.offK[u + 1], S, G.edgC, TipFirst{G}, [&](bool valid, uint32_t, uint32_t, uint32_t u2) {
    if (!valid || u2 == u) return;
    if (hash) t_add(keys, vals, tsize, u2, ctl);
    else atomicAdd(&gcnt[u2], 1u);
  }, done);
  __syncthreads();
  if (hash) {
    for (uint32_t s0 = 0; s0 < tsize; s0 += kPT) {
      const uint32_t s = s0 + threadIdx.x;
      const uint32_t w = s < tsize ? vals[s] : 0u;
      Q.push(w >= 2, ((unsigned long long)w << 32) | (s < tsize ? keys[s] : 0u), charge);
    }
  } else {
    block_iter(G.offK[u], G.offK[u + 1], S, G.edgC, TipFirst{G}, [&](bool valid, uint32_t, uint32_t, uint32_t u2) {
      uint32_t w = 0;
      if (valid && u2 != u) w = atomicExch(&gcnt[u2], 0u);
      Q.push(w >= 2, ((unsigned long long)w << 32) | u2, charge);
    }, done);
  }
  Q.flush(charge);
  if (threadIdx.x == 0) A.work += (unsigned long long)wk;
  __syncthreads();
}

// Removes j[r] butterflies from x[r] where it is unpeeled (state st[r]): all four adds are under way
// before the first result is looked at.
__device__ __forceinline__ void charge_four(const Work& W, Ctl* ctl, Acc& A, const uint32_t* x, const uint32_t* j,
                                            const uint8_t* st) {
  bool c[4];
  long long old[4];
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    c[r] = j[r] && st[r] == ALIVE && mine(W, x[r]);
    old[r] = c[r] ? dec_add(W, x[r], (int64_t)j[r]) : 0;
  }
#pragma unroll
  for (int r = 0; r < 4; ++r)
    if (c[r]) dec_done(W, ctl, A, x[r], (int64_t)j[r], old[r]);
}

// The tip items of one wave: huge ones, then (rounds that run whole) CTA-level and warp-level ones.
struct TipWave {
  const uint4* huge;
  const uint4* front;  // warp-level items from the front, CTA-level ones back from front[last]
  int64_t last;
  unsigned nh, nb, n;
  __device__ __forceinline__ uint4 item(unsigned i) const {
    return i < nh ? huge[i] : (i < nh + nb ? front[last - (int64_t)(i - nh)] : front[i - nh - nb]);
  }
};

// The items of a wave (at most W.ngroups of them): their flattened two-hop lists are cut into equal slices
// over the instance's CTAs.  Every wedge adds one to the item's grid-shared dense counter of u2;
// the add that returns j removes j butterflies from u2 at once (0 + 1 + ... + (w - 1) = C(w, 2)),
// so one pass and no barrier is needed.  clear: every CTA resets the counters of its slice (after a
// barrier): a slice of one step is remembered in `kept` (4 entries per thread of shared memory, so
// clearing costs no loads: light rounds wait for it), a longer one is walked again.
__device__ void tip_items_flat(const Lists& G, const Work& W, Ctl* ctl, const TipWave& V, bool clear, Shared& S,
                               uint32_t* kept, Acc& A) {
  const unsigned n = V.n;
  if (clear && S.flat_steps <= 1) {  // uniform across the CTA; set by the walk
    if (S.flat_steps == 1) {
      uint32_t* cnt = W.gshared + (size_t)S.flat_item * (size_t)W.gshared_stride;
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const uint32_t x = kept[r * kPT + threadIdx.x];
        if (x != kEmpty) cnt[x] = 0u;
      }
    }
    return;
  }
  if (threadIdx.x < 32) {
    unsigned long long carry = 0;
    for (unsigned i0 = 0; i0 < n; i0 += 32) {
      const unsigned i = i0 + threadIdx.x;
      unsigned long long t = 0;
      if (i < n) {
        const uint4 d = V.item(i);
        t = d.w == 0xFFFFFFFFu ? (unsigned long long)G.wk[d.x] + d.z : d.w;
        S.flat[i] = d;
      }
      t = warp_inclusive_scan(t) + carry;
      if (i < n) S.flat_end[i] = t;
      carry = __shfl_sync(0xffffffffu, t, 31);
    }
  }
  __syncthreads();
  unsigned steps = 0;
  const unsigned long long T = S.flat_end[n - 1];
  const unsigned nuse = (unsigned)min((unsigned long long)vgrid(), T / kFlatPairs + 1ull);
  if (T && vblock() < nuse) {
    const unsigned long long lo = T * vblock() / nuse, hi = T * (vblock() + 1) / nuse;
    for (unsigned i = 0; i < n; ++i) {
      const unsigned long long tb = i ? S.flat_end[i - 1] : 0ull, te = S.flat_end[i];
      if (te <= lo || tb >= hi) continue;  // uniform across the CTA
      const uint32_t u = S.flat[i].x, b = S.flat[i].y;
      uint32_t* cnt = W.gshared + (size_t)i * (size_t)W.gshared_stride;
      block_iter_range(b, b + S.flat[i].z, S, G.edgC, lo > tb ? lo - tb : 0ull, min(hi, te) - tb, TipFirst{G},
                       [&](const uint32_t* x) {
                         if (clear) {
#pragma unroll
                           for (int r = 0; r < 4; ++r)
                             if (x[r] != kEmpty) cnt[x[r]] = 0u;
                           return;
                         }
                         if (steps == 0) {
#pragma unroll
                           for (int r = 0; r < 4; ++r) kept[r * kPT + threadIdx.x] = x[r];
                           if (threadIdx.x == 0) S.flat_item = i;
                         }
                         ++steps;
                         uint32_t j[4];
                         uint8_t st[4];
#pragma unroll
                         for (int r = 0; r < 4; ++r) {
                           j[r] = 0;
                           st[r] = PEELED;
                           if (x[r] != kEmpty && x[r] != u) {
                             j[r] = atomicAdd(&cnt[x[r]], 1u);
                             st[r] = W.state[x[r]];
                           }
                         }
                         charge_four(W, ctl, A, x, j, st);
                       });
    }
  }
  if (!clear && threadIdx.x == 0) {
    S.flat_steps = steps;
    if (vblock() == 0) A.work += T;
  }
  __syncthreads();
}

// The same for light rounds (at most 32 items and kListPairs pairs; false and nothing done
// otherwise): a warp takes a whole list N(v) of an item, or with few lists an equal share of its
// 128-entry steps, so that no scan, search or barrier lies between the item and its wedges.  What a
// warp did in one step is remembered in `kept`; several steps are walked again to clear.  (Tip peel
// of the R-MAT graph with 2^20 edges: 78.0 -> 72.4 ms, of it the clearing in phase F 3.7.)
constexpr unsigned long long kListPairs = 1ull << 15;
__device__ bool tip_items_lists(const Lists& G, const Work& W, Ctl* ctl, const TipWave& V, bool clear, Shared& S,
                                uint32_t* kept, Acc& A) {
  const unsigned n = V.n;
  if (n > 32) return false;
  const unsigned lane = lane_id(), warp = threadIdx.x >> 5;
  uint32_t* mykept = kept + warp * 128;
  if (clear && S.list_steps[warp] <= 1) {
    if (S.list_steps[warp] == 1) {
      uint32_t* cnt = W.gshared + (size_t)S.list_item[warp] * (size_t)W.gshared_stride;
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const uint32_t x = mykept[r * 32 + lane];
        if (x != kEmpty) cnt[x] = 0u;
      }
    }
    return true;
  }
  uint4 d = make_uint4(0, 0, 0, 0);
  if (lane < n) d = V.item(lane);
  const unsigned long long T = warp_sum((unsigned long long)d.w);  // a saturated length is above the limit
  if (T > kListPairs) return false;
  const uint32_t incl = warp_inclusive_scan(d.w ? d.z : 0u);  // lists (none: no live butterfly)
  const uint32_t D = __shfl_sync(0xffffffffu, incl, 31);
  unsigned steps = 0, item = 0;
  if (D) {
    const uint32_t nw = vgrid() * kPW, share = max(1u, nw / D);
    for (uint32_t t = warp * vgrid() + vblock(); t < D * share; t += nw) {
      const uint32_t s = t / D, l = t - s * D;
      const unsigned i = __ffs(__ballot_sync(0xffffffffu, incl > l)) - 1;
      const uint32_t before = __shfl_sync(0xffffffffu, incl, i > 0 ? i - 1 : 0);
      const uint32_t u = __shfl_sync(0xffffffffu, d.x, i);
      const uint32_t v = G.edgK[__shfl_sync(0xffffffffu, d.y, i) + l - (i > 0 ? before : 0u)];
      const uint32_t end = G.offC[v + 1];
      uint32_t* cnt = W.gshared + (size_t)i * (size_t)W.gshared_stride;
      for (uint32_t q = G.offC[v] + s * 128; q < end; q += share * 128) {
        uint32_t x[4], j[4];
        uint8_t st[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) x[r] = q + 32 * r + lane < end ? G.edgC[q + 32 * r + lane] : kEmpty;
        if (clear) {
#pragma unroll
          for (int r = 0; r < 4; ++r)
            if (x[r] != kEmpty) cnt[x[r]] = 0u;
          continue;
        }
        if (steps == 0) {
          item = i;
#pragma unroll
          for (int r = 0; r < 4; ++r) mykept[r * 32 + lane] = x[r];
        }
        ++steps;
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          j[r] = 0;
          st[r] = PEELED;
          if (x[r] != kEmpty && x[r] != u) {
            j[r] = atomicAdd(&cnt[x[r]], 1u);
            st[r] = W.state[x[r]];
          }
        }
        charge_four(W, ctl, A, x, j, st);
      }
    }
  }
  if (!clear) {
    if (lane == 0) {
      S.list_steps[warp] = steps;
      S.list_item[warp] = item;
    }
    if (vblock() == 0 && threadIdx.x == 0) A.work += T;
  }
  return true;
}

// ---- wing: process one frontier edge --------------------------------------------------------
// Orientation A (walk from the centre v): probe set N(u) (centre -> edge), first level N(v)
// (u2, edge e2), second level N(u2) (v2, edge e3), probe v2 -> e4.
// Orientation B (walk from u): probe set N(v) (count-side vertex -> edge), first level N(u)
// (v2, e4), second level N(v2) (u2, e3), probe u2 -> e2.  Both find the same butterflies, and
// run the same code with the two sides' lists exchanged.

// Binary-searching a list of length dbig for each of dsmall keys beats scanning it.
__device__ __forceinline__ bool reverse_cheaper(uint32_t dsmall, uint32_t dbig) {
  return (uint64_t)dsmall * (uint64_t)(33u - __clz(dbig | 1u)) < (uint64_t)dbig;
}

// How edge e stands towards frontier edge e1: ES_GONE (peeled earlier, or in this round's
// frontier with a smaller index: the tie rule), ES_CHARGE (unpeeled, loses the butterfly) or
// ES_KEEP (in this round's frontier with a larger index, or of a higher partition: the butterfly
// exists but the edge is not charged).  Edges of lower partitions are gone.
enum EdgeStatus : uint32_t { ES_GONE = 0, ES_CHARGE = 1, ES_KEEP = 2 };
__device__ __forceinline__ uint32_t edge_status(const Work& W, uint32_t e, uint32_t e1) {
  const uint8_t s = W.state[e];
  if (W.part) {
    const uint32_t p = W.part[e];
    if (p != W.my_part) return p < W.my_part ? ES_GONE : ES_KEEP;
  }
  return s == ALIVE ? ES_CHARGE : (s == s_act && e >= e1 ? ES_KEEP : ES_GONE);
}

enum Level { LV_WARP = 0, LV_BLOCK = 1 };
constexpr unsigned kOneSlice = 128;          // rounds of at most this many CTA-level items: one slice per CTA
constexpr uint32_t kKeepBit = 0x80000000u;   // probe-set edges that are not charged (m < 2^31)
constexpr uint32_t kNoSlot = 0x3FFFu;        // queue entries found through the dense markers

// The units [chunk, chunk_end) of nchunks of one frontier edge, by one warp or one CTA.  Unit s holds
// the first-level positions s, s + nchunks, s + 2 nchunks, ...: list lengths vary smoothly with the
// position (ids are ordered alike in every list), so strided units are of nearly equal work where
// contiguous slices are not.
template <int kLevel>
__device__ void wing_item(const Lists& G, const Work& W, Ctl* ctl, const uint4& E, uint32_t* keys, Shared& S,
                          WarpQueue& Q, Acc& A, uint32_t chunk, uint32_t nchunks, uint32_t chunk_end) {
  constexpr uint32_t cap = kLevel == LV_WARP ? kWingWarpSlots : kWingSlots;
  const uint32_t rank = kLevel == LV_WARP ? lane_id() : threadIdx.x;
  constexpr uint32_t gsize = kLevel == LV_WARP ? 32 : kPT;
  auto sync = [] {
    if (kLevel == LV_WARP) __syncwarp();
    else __syncthreads();
  };
  // Side A holds the probe set N(a) and the second-level lists, side B the first level N(b).
  const bool from_v = (E.y & kInfoFromV) != 0;
  const uint32_t* offA = from_v ? G.offK : G.offC;
  const uint32_t* edgA = from_v ? G.edgK : G.edgC;
  const uint32_t* eidA = from_v ? G.eidK : G.eidC;
  const uint32_t* offB = from_v ? G.offC : G.offK;
  const uint32_t* edgB = from_v ? G.edgC : G.edgK;
  const uint32_t* eidB = from_v ? G.eidC : G.eidK;
  const uint32_t e1 = E.x, a = E.y & ~kInfoFromV, b = E.z;
  const uint32_t pb = offA[a], pe = offA[a + 1], psize = pe - pb;
  const uint32_t b1 = offB[b], d1 = offB[b + 1] - b1;
  const bool hash = kLevel == LV_WARP || psize <= kWingSet;
  uint32_t* mark = W.gscratch + (size_t)blockIdx.x * (size_t)W.gscratch_len;
  const uint32_t tsize = hash ? max(64u, min(kWingLoad * psize, cap)) : 0u;
  uint32_t* vals = keys + cap;
  // hits[slot]: butterflies found through a probe-set edge, charged to it in one decrement once
  // the intersections are done.
  uint32_t* hits = vals + cap;
  // The slice's positions are numbered t = 0 .. fn - 1: rows of `width` of every nchunks positions.
  const uint32_t width = chunk_end - chunk, rows = d1 / nchunks, rest = d1 - rows * nchunks;
  const uint32_t fn = rows * width + (rest > chunk ? min(rest - chunk, width) : 0u);
  auto pos_of = [&](uint32_t t) {
    const uint32_t row = width == 1 ? t : t / width;
    return b1 + row * nchunks + chunk + (t - row * width);
  };
  // The chunk's first-level edge of this thread (number t0 + rank).
  uint32_t f_edge = 0, f_st = ES_GONE, f_len = 0, f_beg = 0;
  uint32_t* accp = kLevel == LV_WARP ? S.acc + (threadIdx.x & ~31u) : S.acc;
  // Each (first-level vertex y, probe set) intersection runs in one of two directions: scan
  // N(y) and probe the probe-set table, or (when the probe set is much shorter than N(y))
  // walk the probe set and binary-search N(y), which is sorted.  The direction rides in the
  // top bit of the second-level position.
  uint32_t t_chunk = 0;
  auto load_first = [&](uint32_t y, uint32_t e) {
    f_edge = e;
    const uint32_t b2 = offA[y], d2 = offA[y + 1] - b2;
    f_st = edge_status(W, e, e1);
    f_len = 0;
    if (y == a || f_st == ES_GONE) return;
    if (reverse_cheaper(psize, d2)) { f_beg = pb | kRevFlag; f_len = psize; }
    else { f_beg = b2; f_len = d2; }
  };
  // The first probe-set entry and the first chunk's first-level entry of this thread are loaded
  // together, before the table is built: one chain of round trips instead of two.
  uint32_t key0 = 0, e0 = 0, st0 = ES_GONE, y0 = 0, g0 = 0;
  if (pb + rank < pe) {
    key0 = edgA[pb + rank];
    e0 = eidA[pb + rank];
  }
  if (rank < fn) {
    const uint32_t j = pos_of(rank);
    y0 = edgB[j];
    g0 = eidB[j];
  }
  for (uint32_t s = rank; s < tsize; s += gsize) {
    keys[s] = kEmpty;
    hits[s] = 0;
  }
  if (pb + rank < pe) st0 = edge_status(W, e0, e1);
  if (rank < fn) load_first(y0, g0);
  const bool few = kLevel == LV_BLOCK && hash && fn <= 32;  // a light round's slice
  if (few && rank < fn) {
    S.len[rank] = f_len;
    S.sb[rank] = f_beg;
  }
  accp[rank] = 0;
  sync();
  auto put = [&](uint32_t key, uint32_t e, uint32_t es) {
    if (es == ES_GONE) return;
    const uint32_t val = es == ES_KEEP ? (e | kKeepBit) : e;
    if (hash) t_put(keys, vals, tsize, key, val, ctl);
    else mark[key] = val + 1;
  };
  put(key0, e0, st0);
  for (uint32_t p = pb + rank + gsize; p < pe; p += gsize) {
    const uint32_t key = edgA[p], e = eidA[p];
    put(key, e, edge_status(W, e, e1));
  }
  sync();
  auto first = [&](uint32_t t, bool valid, uint32_t& L, uint32_t& sb) {
    t_chunk = t - rank;
    if (t_chunk) {
      accp[rank] = 0;
      f_st = ES_GONE;
      f_len = 0;
      if (valid) {
        const uint32_t j = pos_of(t);
        load_first(edgB[j], eidB[j]);
      }
    }
    L = f_len;
    sb = f_beg;
  };
  // One butterfly found through second-level entry q: its edge loses 1 now; the probe-set edge
  // loses 1 through its hit counter when it has a table slot; the first-level edge through the
  // chunk's accumulator.
  auto charge = [&](unsigned long long x) {
    const uint32_t q = (uint32_t)(x >> 32), slot = (uint32_t)x & kNoSlot, lo = ((uint32_t)x >> 14) & 511u;
    const uint32_t e3 = eidA[q];
    const uint32_t es = edge_status(W, e3, e1);
    if (es == ES_GONE) return;
    if (es == ES_CHARGE) dec_known(W, ctl, A, e3, 1);
    if (slot != kNoSlot) {
      atomicAdd(&hits[slot], 1u);
    } else {
      const uint32_t val = mark[edgA[q]] - 1u;
      if (!(val & kKeepBit)) dec_known(W, ctl, A, val, 1);
    }
    atomicAdd(&accp[lo], 1u);
  };
  unsigned my_work = 0, my_rev = 0;
  auto pair = [&](bool valid, uint32_t lo, uint32_t q, uint32_t z) {
    bool hit = false;
    unsigned long long ent = 0;
    if (valid) ++my_work;
    if (valid && z != b) {
      if (q & kRevFlag) {  // walk N(a), binary-search N(y)
        ++my_rev;
        const uint32_t e4 = eidA[q & ~kRevFlag];
        const uint32_t s4 = edge_status(W, e4, e1);
        if (s4 != ES_GONE) {
          const uint32_t y = edgB[pos_of(t_chunk + lo)];
          const uint32_t end = offA[y + 1];
          const uint32_t at = lower_bound_u32(edgA, offA[y], end, z);
          if (at != end && edgA[at] == z) {
            const uint32_t e3 = eidA[at];
            const uint32_t s3 = edge_status(W, e3, e1);
            if (s3 != ES_GONE) {
              if (s3 == ES_CHARGE) dec_known(W, ctl, A, e3, 1);
              if (s4 == ES_CHARGE) dec_known(W, ctl, A, e4, 1);
              atomicAdd(&accp[lo], 1u);
            }
          }
        }
      } else if (hash) {
        const uint32_t slot = t_slot(keys, tsize, z);
        hit = slot != kEmpty;
        ent = ((unsigned long long)q << 32) | (lo << 14) | (slot & kNoSlot);
      } else {
        hit = mark[z] != 0;
        ent = ((unsigned long long)q << 32) | (lo << 14) | kNoSlot;
      }
    }
    Q.push(hit, ent, charge);
  };
  // Summed decrements of one edge: (edge, amount).
  auto charge_sum = [&](unsigned long long x) { dec_known(W, ctl, A, (uint32_t)x, (int64_t)(x >> 32)); };
  // The first-level edges' decrements; those of the last chunk wait in the queue and are charged
  // together with the probe set's.
  auto done = [&] {
    Q.flush(charge);
    sync();
    const uint32_t got = f_st == ES_CHARGE ? accp[rank] : 0u;
    Q.push(got != 0, ((unsigned long long)got << 32) | f_edge, charge_sum);
    if (t_chunk + gsize < fn) Q.flush(charge_sum);
  };
  if (kLevel == LV_WARP) {
    warp_iter(0, fn, edgA, first, pair, done);
  } else if (hash) {
    auto piece = [&](uint32_t lo, uint32_t k, uint32_t q, uint32_t n, const uint32_t* x) {
      if (q & kRevFlag) {
#pragma unroll 1
        for (uint32_t r = 0; r < kPiece / 32; ++r)
          if ((k & ~31u) + 32 * r < n) pair(k + 32 * r < n, lo, q + 32 * r, r == 0 ? x[0] : r == 1 ? x[1] : r == 2 ? x[2] : x[3]);
        return;
      }
      // The four first probes of a lane are made together; only collisions go on one by one.
      uint32_t slot[kPiece / 32], key[kPiece / 32];
#pragma unroll
      for (uint32_t r = 0; r < kPiece / 32; ++r) {
        slot[r] = hslot(x[r], tsize);
        key[r] = keys[slot[r]];
      }
#pragma unroll
      for (uint32_t r = 0; r < kPiece / 32; ++r) {
        const bool valid = x[r] != kEmpty && x[r] != b;
        my_work += x[r] != kEmpty;
        if (!valid || key[r] == kEmpty) slot[r] = kEmpty;
        else if (key[r] != x[r]) slot[r] = t_slot_next(keys, tsize, x[r], slot[r]);
        Q.push(slot[r] != kEmpty, ((unsigned long long)(q + 32 * r) << 32) | (lo << 14) | (slot[r] & kNoSlot), charge);
      }
    };
    if (few) {
      few_pieces(fn, S.len, S.sb, edgA, piece);
      done();
    } else {
      block_pieces(0, fn, S, edgA, first, piece, done);
    }
  } else {
    block_iter(0, fn, S, edgA, first, pair, done);
  }
  // The probe-set edges' decrements, one per edge.
  for (uint32_t s0 = 0; s0 < tsize; s0 += gsize) {
    const uint32_t s = s0 + rank;
    const uint32_t h = s < tsize ? hits[s] : 0u;
    const uint32_t val = h ? vals[s] : kKeepBit;
    Q.push(!(val & kKeepBit), ((unsigned long long)h << 32) | val, charge_sum);
  }
  Q.flush(charge_sum);
  if (!hash) {  // clear the dense markers
    for (uint32_t p = pb + rank; p < pe; p += gsize) mark[edgA[p]] = 0;
  }
  A.work += my_work;
  if (s_trace) {
    const int mode = kLevel == LV_WARP ? 0 : (hash ? 1 : 2);
    const unsigned w = __reduce_add_sync(0xffffffffu, my_work);
    const unsigned rw = __reduce_add_sync(0xffffffffu, my_rev);
    if (lane_id() == 0) {
      if (w) atomicAdd(&s_st.mode_work[mode], (unsigned long long)w);
      if (rw) atomicAdd(&s_st.rev_work, (unsigned long long)rw);
    }
    if (rank == 0) atomicAdd(&s_st.mode_items[mode], 1ull);
  }
  sync();
}

// ---- the persistent kernel ------------------------------------------------------------------
// Wing items run on one warp when their work is small and their probe set fits a warp table.
struct Classify {
  int64_t small_work;
  int64_t huge_work;   // tip items above this run on the whole grid
  int64_t chunk_work;  // target probes per work unit of a CTA-level wing item
  int64_t units_per_cta;  // work units per CTA a round's CTA-level wing work is cut into
  int64_t warp_units;     // wing: every item with a warp-sized probe set runs as warp units

  __device__ __forceinline__ bool tip_small(const Work& W, int64_t wk, uint32_t deg) const {
    return wk <= (int64_t)(tip_one_word(W, deg) ? kTipWarpSlots : kTipWarpSlots / 2) && wk <= small_work;
  }
  // Estimated probes from each side: the two-hop list sizes, capped by deg(u)*deg(v) times a
  // binary-search factor (the reverse-direction intersections).
  __device__ __forceinline__ int64_t cost_v(const Lists& G, uint32_t v, uint32_t u) const {
    const int64_t du = G.offK[u + 1] - G.offK[u], dv = G.offC[v + 1] - G.offC[v];
    return min(G.S[G.nK + v], du * dv * 16);
  }
  __device__ __forceinline__ int64_t cost_u(const Lists& G, uint32_t v, uint32_t u) const {
    const int64_t du = G.offK[u + 1] - G.offK[u], dv = G.offC[v + 1] - G.offC[v];
    return min(G.S[u], du * dv * 16);
  }
};

// Estimated work of peeling item x (plus one, so that items without work still count): the
// cheaper side's two-hop probes of a wing item, the two-hop wedges of a tip item.
template <bool kWing>
__device__ __forceinline__ unsigned long long item_weight(const Lists& G, const Classify& cls, uint32_t x) {
  if (kWing) {
    const uint32_t v = G.center_of[x], u = G.u_of[x];
    const int64_t c = min(cls.cost_v(G, v, u), cls.cost_u(G, v, u));
    return 1ull + (unsigned long long)(c > 0 ? c : 0);
  }
  return 1ull + (unsigned long long)(G.wk[x] > 0 ? G.wk[x] : 0);
}

// The peel instances of one launch.  n == 1: the whole grid runs instance 0.  Otherwise CTA b
// runs instances cta_beg[b] .. cta_end[b] - 1 one after another; instance i spans the ncta[i]
// CTAs from first[i] (heavy graphs get many CTAs, light graphs share one CTA in turn).
struct Instances {
  const Work* W;
  const uint32_t* first;
  const uint32_t* ncta;
  const uint32_t* cta_beg;
  const uint32_t* cta_end;
  uint32_t n;
};

// Adds the CTA's statistics to the control block (CTA 0 also its rounds and phase times).
__device__ void flush_stats(Ctl* ctl) {
  __syncthreads();
  if (threadIdx.x < 3) {
    if (s_st.mode_items[threadIdx.x]) atomicAdd(&ctl->mode_items[threadIdx.x], s_st.mode_items[threadIdx.x]);
    if (s_st.mode_work[threadIdx.x]) atomicAdd(&ctl->mode_work[threadIdx.x], s_st.mode_work[threadIdx.x]);
  }
  if (threadIdx.x == 3 && s_st.rev_work) atomicAdd(&ctl->rev_work, s_st.rev_work);
  if (vblock() != 0) return;
  if (threadIdx.x < 42) {
    ctl->pbin_ns[threadIdx.x] += s_st.pbin_ns[threadIdx.x];
    ctl->pbin_rounds[threadIdx.x] += s_st.pbin_rounds[threadIdx.x];
    ctl->pbin_est[threadIdx.x] += s_st.pbin_est[threadIdx.x];
  }
  if (threadIdx.x < 3) ctl->phase_ns[threadIdx.x] += s_st.phase_ns[threadIdx.x];
  if (threadIdx.x == 0) {
    ctl->rounds += s_st.rounds;
    ctl->scanned += s_st.scanned;
    ctl->n_small += s_st.n_small;
    ctl->n_big += s_st.n_big;
    ctl->n_huge += s_st.n_huge;
    ctl->advances += s_st.advances;
  }
}

// All rounds of one peel instance, run by its CTAs; false when a bounded wait ran out or an
// invariant broke (recorded in ctl->err).
template <bool kWing>
__device__ bool peel_instance(const Lists& G, const Work& W, Ctl* ctl, const Classify& cls) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Shared& S = *reinterpret_cast<Shared*>(smem_raw);
  uint32_t* pool = reinterpret_cast<uint32_t*>(smem_raw + ((sizeof(Shared) + 15) & ~size_t(15)));
  const unsigned warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint32_t* kept = pool + kPoolWords - 4 * kPT;  // beyond the tip tables and the advance's bins
  uint32_t* wkeys = pool + warp * (kWing ? 3 * kWingWarpSlots : 2 * kTipWarpSlots);
  const unsigned gtid = vblock() * kPT + threadIdx.x;
  const unsigned gthreads = vgrid() * kPT;
  const bool cta0 = vblock() == 0;
  WarpQueue Q{S.queue[warp], 0u};
  for (unsigned i = threadIdx.x; i < sizeof(Stats) / 8; i += kPT) reinterpret_cast<unsigned long long*>(&s_st)[i] = 0;
  if (threadIdx.x == 0) {
    s_bar_target = *(volatile unsigned long long*)&ctl->bar_base;
    s_bar_timeout = ctl->barrier_timeout_ns;
    s_skip_arrival = vblock() == 0 ? ctl->test_skip_arrival : 0u;
    s_err = 0;
    s_trace = ctl->trace;
    S.flat_steps = 0;
  }
  unsigned alist_cur = *(volatile unsigned*)&ctl->alist_cur;
  const bool range = *(volatile unsigned*)&ctl->range_mode != 0;
  const bool trace = cta0 && ctl->trace != 0;
  unsigned part_idx = *(volatile unsigned*)&ctl->npart;  // partitions opened (range mode)
  unsigned alive = *(volatile unsigned*)&ctl->alive;     // kept per CTA: every CTA sees the frontier sizes
  unsigned near_done = *(volatile unsigned*)&ctl->near_done;
  const unsigned at_compact = *(volatile unsigned*)&ctl->alive_at_compact;
  const unsigned min_gain = *(volatile unsigned*)&ctl->min_gain;
  // Near items a window opens with: near_min, but no more than four per thread (a round scans the
  // near list once, so on few CTAs a long list costs more than the advances it saves).
  const unsigned near_min = min(ctl->near_min, 4u * gthreads);
  const unsigned near_div = max(1u, ctl->near_div);
  unsigned long long work = 0;
  __syncthreads();
  if (!*(volatile unsigned*)&ctl->started) {
    for (int64_t x = gtid; x < W.N; x += gthreads)
      W.alist[0][x] = W.items ? W.items[W.item0 + x] : W.item0 + (uint32_t)x;
    if (!grid_barrier(ctl)) return false;
    if (cta0 && threadIdx.x == 0) ctl->started = 1;
  }
  const bool trace_est = ctl->trace != 0;
  // What the last barrier of a round hands to the next one: the next minimum and the near list's
  // length; the window bound changes only in an advance; the frontier sizes of the last round.
  const unsigned long long r0 = *(volatile unsigned long long*)&ctl->round;
  unsigned long long next_k = *(volatile unsigned long long*)&ctl->nm[r0 & 1ull];
  unsigned near_len = (unsigned)*(volatile unsigned long long*)&ctl->near_len;
  unsigned long long win_hi = *(volatile unsigned long long*)&ctl->win_hi;
  unsigned ps = (unsigned)(*(volatile unsigned long long*)&ctl->fsmall[(r0 & 1ull) ^ 1ull] >> 32);
  unsigned pg = (unsigned)(*(volatile unsigned long long*)&ctl->fbig[(r0 & 1ull) ^ 1ull] >> 32);
  unsigned ph = (unsigned)(*(volatile unsigned long long*)&ctl->fhuge[(r0 & 1ull) ^ 1ull] >> 32);
  // Tip: flat items of the previous round whose counters are still to be cleared.
  unsigned clear_n = 0, clear_nh = 0, clear_nb = 0;
  bool clear_lists = false;  // by tip_items_lists

  for (unsigned long long r = r0;; ++r) {
    const unsigned par = (unsigned)(r & 1ull), npar = par ^ 1u;
    // Pause at a round boundary once enough items have been peeled since the lists were last
    // compacted; the host compacts them and relaunches (all CTAs hold the same values here).
    const bool pause = alive != 0 && 2u * alive < at_compact && at_compact - alive >= min_gain;
    if (alive == 0 || pause) {
      if (!kWing && clear_n) {
        Acc none{kInf, 0};
        const TipWave V{W.fhuge[npar], W.front[npar], W.N - 1, clear_nh, clear_nb, clear_n};
        if (clear_lists) tip_items_lists(G, W, ctl, V, true, S, kept, none);
        else tip_items_flat(G, W, ctl, V, true, S, kept, none);
      }
      if (cta0 && threadIdx.x == 0) {
        ctl->round = r;
        ctl->alist_cur = alist_cur;
        ctl->alive = alive;
        ctl->near_done = near_done;
        ctl->bar_base = s_bar_target;
        ctl->part_done += s_st.part_done;
      }
      break;
    }
    unsigned long long k = next_k;
    if (k == kInf) {
      unsigned long long part_target_next = 0, part_ratio_next = 0;  // range mode
      // ---- window advance (no unpeeled item left in the near list): compact the alive list
      // and take its minimum; a log2 histogram of distances to the minimum picks the window
      // bound; the near list is rebuilt from the alive list.  Unpeeled items lie above the old
      // bound here: their bucket is their count.
      const unsigned na = alist_cur ^ 1u;
      const unsigned alen = *(volatile unsigned*)&ctl->alen[alist_cur];
      unsigned long long mn = kInf;
      for (unsigned q0 = gtid - lane; q0 < alen; q0 += gthreads) {  // whole warps: one add per warp
        const unsigned q = q0 + lane;
        const uint32_t x = q < alen ? W.alist[alist_cur][q] : kEmpty;
        const bool live = x != kEmpty && W.state[x] == ALIVE;
        const unsigned at = warp_append(&ctl->alen[na], live);
        if (!live) continue;
        W.alist[na][at] = x;
        const int64_t c = W.cnt[x];
        if (range) W.D[x] = c;
        mn = min(mn, (unsigned long long)c);
      }
      __syncwarp();
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) mn = min(mn, __shfl_xor_sync(0xffffffffu, mn, o));
      if (lane == 0 && mn != kInf) atomicMin(&ctl->k_lo, mn);
      if (threadIdx.x < 66) S.hist[threadIdx.x] = 0;
      if (cta0) {
        // The previous advance's histograms were last read before two barriers ago.
        if (threadIdx.x < 66) {
          ctl->hist[threadIdx.x] = 0;
          ctl->whist[threadIdx.x] = 0;
        }
        if (range && threadIdx.x < 256) ctl->wsub[threadIdx.x] = 0;
        if (threadIdx.x == 0) {
          ctl->near_len = 0;
          if (range) {
            ctl->part_done += s_st.part_done;
            s_st.part_done = 0;
          }
        }
      }
      if (!grid_barrier(ctl)) return false;
      near_done = 0;
      if (range) {
        ++part_idx;  // the window opened here is partition part_idx - 1
        if (cta0 && threadIdx.x == 0) ctl->npart = part_idx;
      }
      const unsigned long long klo = *(volatile unsigned long long*)&ctl->k_lo;
      const unsigned alen2 = *(volatile unsigned*)&ctl->alen[na];
      unsigned long long hi = kInf;
      if (!range) {
        for (unsigned q = gtid; q < alen2; q += gthreads) {
          const unsigned long long d = (unsigned long long)W.cnt[W.alist[na][q]] - klo;
          atomicAdd(&S.hist[d ? 64 - __clzll(d) : 0], 1u);
        }
        __syncthreads();
        if (threadIdx.x < 66 && S.hist[threadIdx.x]) atomicAdd(&ctl->hist[threadIdx.x], S.hist[threadIdx.x]);
        if (!grid_barrier(ctl)) return false;
        // Every CTA derives the same bound: the smallest B with >= target items at distance < 2^B.
        const unsigned target = max(near_min, alen2 / near_div);
        unsigned long long cum = 0;
        const int B = (int)find_bin(ctl->hist, 65, target, cum);
        if (B < 63) {
          const unsigned long long span = 1ull << B;
          if (klo <= kInf - span) hi = klo + span;
        }
      } else {
        // Partition bound: about part_target of estimated work below it.  A log2 histogram of
        // distances to the minimum (weighted by work) picks the octave, a 256-bin linear
        // histogram inside it the bound.  The bins live in the (idle) table pool.
        unsigned long long* wh = reinterpret_cast<unsigned long long*>(pool);
        if (threadIdx.x < 66) wh[threadIdx.x] = 0;
        __syncthreads();
        for (unsigned q0 = gtid - lane; q0 < alen2; q0 += gthreads) {
          const unsigned q = q0 + lane;
          int bin = -1;
          uint32_t w = 0;
          if (q < alen2) {
            const uint32_t x = W.alist[na][q];
            const unsigned long long d = (unsigned long long)W.cnt[x] - klo;
            bin = d ? 64 - __clzll(d) : 0;
            w = W.wgt[x];
          }
          warp_bin_add(wh, bin, w);
        }
        __syncthreads();
        if (threadIdx.x < 66 && wh[threadIdx.x]) atomicAdd(&ctl->whist[threadIdx.x], wh[threadIdx.x]);
        if (!grid_barrier(ctl)) return false;
        const unsigned long long base = *(volatile unsigned long long*)&ctl->part_target;
        const unsigned long long done = *(volatile unsigned long long*)&ctl->part_done;
        const unsigned long long used = *(volatile unsigned long long*)&ctl->part_used;
        unsigned long long ratio_q = *(volatile unsigned long long*)&ctl->part_ratio_q;
        if (used > 0 && done > 0) {
          const unsigned long long rq = min(done * 256ull / used, 256ull * 4096ull);
          ratio_q = ratio_q ? (ratio_q + rq) / 2 : rq;
        }
        const unsigned long long target = max(1ull, ratio_q > 256 ? base * 256ull / ratio_q : base);
        part_target_next = target;
        part_ratio_next = ratio_q;
        unsigned long long cum = 0;
        const int B = (int)find_bin(ctl->whist, 65, target, cum);
        if (B == 0) {
          hi = klo + 1;
        } else if (B < 63) {
          const unsigned long long lo_d = 1ull << (B - 1), width = lo_d;  // distances [2^(B-1), 2^B)
          __syncthreads();
          if (threadIdx.x < 256) wh[threadIdx.x] = 0;
          __syncthreads();
          for (unsigned q0 = gtid - lane; q0 < alen2; q0 += gthreads) {
            const unsigned q = q0 + lane;
            int bin = -1;
            uint32_t w = 0;
            if (q < alen2) {
              const uint32_t x = W.alist[na][q];
              const unsigned long long d = (unsigned long long)W.cnt[x] - klo;
              if (d >= lo_d && d < lo_d + width) {
                bin = (int)((d - lo_d) * 256ull / width);
                w = W.wgt[x];
              }
            }
            warp_bin_add(wh, bin, w);
          }
          __syncthreads();
          if (threadIdx.x < 256 && wh[threadIdx.x]) atomicAdd(&ctl->wsub[threadIdx.x], wh[threadIdx.x]);
          if (!grid_barrier(ctl)) return false;
          const unsigned j = find_bin(ctl->wsub, 255, target, cum);
          // Bin j covers distances [lo_d + ceil(j w / 256), lo_d + ceil((j + 1) w / 256)).
          const unsigned long long end_d = lo_d + ((unsigned long long)(j + 1) * width + 255ull) / 256ull;
          if (klo <= kInf - end_d) hi = klo + end_d;
        }
      }
      for (unsigned q0 = gtid - lane; q0 < alen2; q0 += gthreads) {
        const unsigned q = q0 + lane;
        const uint32_t x = q < alen2 ? W.alist[na][q] : kEmpty;
        const bool in = x != kEmpty && (hi == kInf || (unsigned long long)W.cnt[x] < hi);
        const unsigned at = (unsigned)warp_append(&ctl->near_len, in);
        if (in) W.near[at] = x;
      }
      if (cta0 && threadIdx.x == 0) {
        ctl->win_hi = hi;
        ctl->alen[alist_cur] = 0;  // read by every CTA before the first barrier
        ctl->k_lo = kInf;          // read by every CTA right after the first barrier
        s_st.advances += 1;
      }
      alist_cur = na;
      if (!grid_barrier(ctl, &ctl->near_len)) return false;
      near_len = (unsigned)s_words[0];
      win_hi = hi;
      phase_mark(trace, 0);
      if (range && cta0 && threadIdx.x == 0) {  // every CTA read the previous values before this barrier
        ctl->part_used = part_target_next;
        ctl->part_ratio_q = part_ratio_next;
        ctl->part_done = 0;
      }
      k = klo;
    }
    const unsigned char act = (unsigned char)(1u + par);
    if (threadIdx.x == 0) {
      s_win_hi = win_hi;
      s_k = (long long)k;
      s_act = act;
    }
    // ---- phase F: the frontier is every near item in bucket k (range mode: every near item not
    // taken yet); the minimum of the other near items is the first part of the next round's
    // minimum.  Four items per thread are loaded at a time.
    {
      const unsigned nl = near_len;
      // The previous round's frontier (ps, pg, ph items) becomes PEELED.
      unsigned long long mn = kInf;
      unsigned long long est = 0;
      for (unsigned q0 = near_done + gtid; q0 < nl; q0 += 4 * gthreads) {
        uint32_t xs[4];
        uint8_t st[4];
        long long cs[4];
#pragma unroll
        for (unsigned i = 0; i < 4; ++i) {
          const unsigned q = q0 + i * gthreads;
          xs[i] = q < nl ? W.near[q] : kEmpty;
        }
#pragma unroll
        for (unsigned i = 0; i < 4; ++i) {
          st[i] = PEELED;
          cs[i] = 0;
          if (xs[i] != kEmpty) {
            st[i] = W.state[xs[i]];
            cs[i] = W.cnt[xs[i]];
          }
        }
#pragma unroll 1
        for (unsigned i = 0; i < 4 && q0 + i * gthreads < nl; ++i) {
          const uint32_t x = xs[0];
          const uint8_t sx = st[0];
          const long long c = cs[0];
          xs[0] = xs[1]; xs[1] = xs[2]; xs[2] = xs[3];
          st[0] = st[1]; st[1] = st[2]; st[2] = st[3];
          cs[0] = cs[1]; cs[1] = cs[2]; cs[2] = cs[3];
          if (sx != ALIVE) continue;
          if (!range && c > (long long)k) {
            mn = min(mn, (unsigned long long)c);
            continue;
          }
          W.state[x] = act;
          if (range) W.part_out[x] = part_idx - 1;
          else W.D[x] = (int64_t)k;
          // An item without live butterflies gets no units: nothing is left to remove.
          if (kWing) {
            const uint32_t inf = G.info[x], v = G.center_of[x], u = G.u_of[x];
            const bool fv = (inf & kInfoFromV) != 0;
            const unsigned long long add = (1ull << 32) | (c != 0 ? inf & kInfoUnits : 0u);
            const bool small = (inf & kInfoSmall) != 0;
            const unsigned long long at = atomicAdd(small ? &ctl->fsmall[par] : &ctl->fbig[par], add);
            const uint32_t pos = (uint32_t)(at >> 32);
            W.front[par][small ? (int64_t)pos : W.N - 1 - pos] =
                make_uint4(x, (fv ? u : v) | (inf & kInfoFromV), fv ? v : u, (uint32_t)at);
            if (range || trace_est) est += item_weight<kWing>(G, cls, x) - 1ull;
          } else {
            const int64_t wk = G.wk[x];
            const uint32_t b = G.offK[x], d = G.offK[x + 1] - b;
            const unsigned long long pairs = c != 0 ? (unsigned long long)wk + d : 0ull;
            const uint4 it = make_uint4(x, b, d, (uint32_t)min(pairs, 0xFFFFFFFFull));
            const unsigned long long add = (1ull << 32) | 1ull;
            if (cls.tip_small(W, wk, d)) {
              W.front[par][atomicAdd(&ctl->fsmall[par], add) >> 32] = it;
            } else if (wk > cls.huge_work && W.gshared != nullptr) {
              atomicAdd(&ctl->huge_sum[par], pairs);
              atomicMax(&ctl->huge_max[par], pairs);
              W.fhuge[par][atomicAdd(&ctl->fhuge[par], add) >> 32] = it;
            } else {
              W.front[par][W.N - 1 - (int64_t)(atomicAdd(&ctl->fbig[par], add) >> 32)] = it;
            }
            est += (unsigned long long)(wk > 0 ? wk : 0);
          }
        }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) mn = min(mn, __shfl_xor_sync(0xffffffffu, mn, o));
      if (lane == 0 && mn != kInf) atomicMin(&ctl->nm[npar], mn);
      if ((range || trace_est) && __any_sync(0xffffffffu, est != 0)) {
        est = warp_sum(est);
        if (lane == 0) atomicAdd(&ctl->round_est[par], est);
      }
      // (from the other end of the grid: the threads at this end had near items to look at)
      for (unsigned q = gthreads - 1u - gtid; q < ps + pg + ph; q += gthreads) {
        const uint32_t x = q < ps ? W.front[npar][q].x
                                  : (q < ps + pg ? W.front[npar][W.N - 1 - (q - ps)].x : W.fhuge[npar][q - ps - pg].x);
        W.state[x] = PEELED;
      }
      if (!kWing && clear_n) {
        Acc none{kInf, 0};
        const TipWave V{W.fhuge[npar], W.front[npar], W.N - 1, clear_nh, clear_nb, clear_n};
        if (clear_lists) tip_items_lists(G, W, ctl, V, true, S, kept, none);
        else tip_items_flat(G, W, ctl, V, true, S, kept, none);
        clear_n = 0;
      }
      if (cta0 && threadIdx.x == 0) s_st.scanned += nl - near_done;
      if (range) near_done = nl;
    }
    if (!grid_barrier(ctl, &ctl->fsmall[par], &ctl->fbig[par], &ctl->fhuge[par])) return false;
    phase_mark(trace, 1);
    // ---- phase P: process the frontier (small items per warp, then heavy items per CTA).
    Acc A{kInf, 0};
    const unsigned ns = (unsigned)(s_words[0] >> 32), nwu = (unsigned)s_words[0];
    const unsigned nb = (unsigned)(s_words[1] >> 32), nu = (unsigned)s_words[1];
    const unsigned nh = kWing ? 0u : (unsigned)(s_words[2] >> 32);
    ps = ns;
    pg = nb;
    ph = nh;
    unsigned long long round_est = 0;
    if (cta0 && threadIdx.x == 0) {
      if (range || trace) round_est = *(volatile unsigned long long*)&ctl->round_est[par];
      ctl->nm[par] = kInf;  // every CTA has read it
      // Slots of the previous round: last read in phase F.
      ctl->fsmall[npar] = 0;
      ctl->fbig[npar] = 0;
      ctl->fhuge[npar] = 0;
      ctl->round_est[npar] = 0;
      ctl->cur_small[npar] = 0;
      ctl->cur_big[npar] = 0;
      ctl->cur_huge[npar] = 0;
      ctl->huge_sum[npar] = 0;
      ctl->huge_max[npar] = 0;
      s_st.rounds += 1;
      s_st.n_small += ns;
      s_st.n_big += nb;
      s_st.n_huge += nh;
      s_st.part_done += round_est;
    }
    alive -= ns + nb + nh;
    {
      // Tip items: the huge ones run over the whole grid, in waves of up to ngroups; when the round
      // has so few items that one wave holds them all, they all run there (one warp or CTA per item
      // leaves the rest of the grid idle).
      const unsigned ng = kWing ? 0u : (W.gshared ? min(W.ngroups, kMaxGroups) : 0u);
      const unsigned items = ns + nb + nh;
      const bool flat_all = !kWing && vgrid() >= 8 && items > 0 && items <= min(ng, kFlatAll);
      // Warp-level items: warps claim runs of consecutive units and process an item's units of a
      // run as one first-level slice, independently of the other warps (tip: an item is one
      // unit).  The first run of a warp is its own number; the cursor hands out the later ones.
      const unsigned gwarps = vgrid() * kPW;
      const unsigned Kw = kWing ? max(1u, nwu / (4u * gwarps)) : 1u;
      const uint4* const fsm = W.front[par];
      for (unsigned u = (vblock() * kPW + warp) * Kw; u < nwu && !flat_all;) {
        const unsigned uend = min(u + Kw, nwu);
        if (kWing) {
          uint32_t lo = 0, hi = ns;  // the last item whose first unit <= u, 32-way search
          while (hi - lo > 1) {
            const uint32_t step = (hi - lo + 31) / 32;
            const uint32_t idx = lo + lane * step;
            const bool le = idx < hi && fsm[idx].w <= u;
            const unsigned bal = __ballot_sync(0xffffffffu, le);
            lo = lo + (31 - __clz(bal)) * step;  // lane 0 always qualifies
            hi = min(lo + step, hi);
          }
          for (unsigned uu = u, q = lo; uu < uend; ++q) {  // uniform across the warp
            const uint4 it = fsm[q];
            const uint32_t next = q + 1 < ns ? fsm[q + 1].w : nwu;
            const uint32_t c1 = min(uend, next);
            if (c1 > uu) wing_item<LV_WARP>(G, W, ctl, it, wkeys, S, Q, A, uu - it.w, next - it.w, c1 - it.w);
            uu = max(uu, c1);
          }
        } else {
          const uint4 it = fsm[u];
          if (it.w) tip_item_warp(G, W, ctl, it, wkeys, Q, A);
        }
        if (gwarps * Kw >= nwu) break;
        unsigned c = 0;
        if (lane == 0) c = atomicAdd(&ctl->cur_small[par], Kw);
        u = gwarps * Kw + __shfl_sync(0xffffffffu, c, 0);
      }
      if (ns) __syncthreads();  // warp tables and the CTA table share memory
      if (nu && !flat_all) {
        const uint4* const fbg = W.front[par] + (W.N - 1);  // item q: fbg[-q]
        if (kWing && nb <= kOneSlice && 2 * nb <= vgrid()) {
          // Light rounds: K units make a slice such that every CTA gets at most one slice (of one
          // item).  Each warp derives the layout from the items' unit counts by itself.
          const unsigned K = (nu + vgrid() - nb - 1) / (vgrid() - nb);
          unsigned carry = 0;
          for (unsigned q0 = 0; q0 < nb; q0 += 32) {
            const unsigned q = q0 + lane;
            uint4 it = make_uint4(0, 0, 0, nu);
            if (q < nb) it = fbg[-(int64_t)q];
            unsigned next = __shfl_down_sync(0xffffffffu, it.w, 1);
            if (lane == 31) next = q + 1 < nb ? fbg[-(int64_t)(q + 1)].w : nu;
            const unsigned units = q < nb ? next - it.w : 0u, slices = (units + K - 1) / K;
            const unsigned end = carry + warp_inclusive_scan(slices);
            const unsigned m = __ballot_sync(0xffffffffu, slices && vblock() >= end - slices && vblock() < end);
            if (m) {  // this CTA's slice: units sl, sl + n, ... of the item of lane l, as one of n slices
              const int l = __ffs(m) - 1;
              it.x = __shfl_sync(0xffffffffu, it.x, l);
              it.y = __shfl_sync(0xffffffffu, it.y, l);
              it.z = __shfl_sync(0xffffffffu, it.z, l);
              const unsigned n = __shfl_sync(0xffffffffu, slices, l);
              const unsigned sl = vblock() - (__shfl_sync(0xffffffffu, end, l) - n);
              wing_item<LV_BLOCK>(G, W, ctl, it, pool, S, Q, A, sl, n, sl + 1);
              break;
            }
            carry = __shfl_sync(0xffffffffu, end, 31);
          }
        } else {
          // CTAs claim runs of K consecutive units (wing: a units_per_cta-th of a CTA's share; tip:
          // one unit, which is one item); the units of one item inside a run are processed as one
          // slice, so the item's probe table is built once per run, not once per unit.  The first
          // run of a CTA is its own number; the cursor hands out the later ones.
          const unsigned K = kWing ? max(1u, nu / ((unsigned)cls.units_per_cta * vgrid())) : 1u;
          const bool more = vgrid() * K < nu;  // some run is left for the cursor
          for (unsigned u0 = vblock() * K; u0 < nu;) {
            const unsigned uend = min(u0 + K, nu);
            if (more && threadIdx.x == 0) S.item = atomicAdd(&ctl->cur_big[par], K);
            if (kWing) {
              uint32_t lo = 0, hi = nb;  // the last item whose first unit <= u0, 32-way search by every warp
              while (hi - lo > 1) {
                const uint32_t step = (hi - lo + 31) / 32;
                const uint32_t idx = lo + lane * step;
                const bool le = idx < hi && fbg[-(int64_t)idx].w <= u0;
                const unsigned bal = __ballot_sync(0xffffffffu, le);
                lo = lo + (31 - __clz(bal)) * step;  // lane 0 always qualifies
                hi = min(lo + step, hi);
              }
              for (unsigned uu = u0, q = lo; uu < uend; ++q) {  // uniform across the CTA
                const uint4 it = fbg[-(int64_t)q];
                const uint32_t next = q + 1 < nb ? fbg[-(int64_t)(q + 1)].w : nu;
                const uint32_t c1 = min(uend, next);
                if (c1 > uu) wing_item<LV_BLOCK>(G, W, ctl, it, pool, S, Q, A, uu - it.w, next - it.w, c1 - it.w);
                uu = max(uu, c1);
              }
            } else {
              const uint4 it = fbg[-(int64_t)u0];
              if (it.w) tip_item_block(G, W, ctl, it.x, pool, S, Q, A);
            }
            if (!more) break;
            __syncthreads();
            u0 = vgrid() * K + S.item;
            __syncthreads();
          }
        }
      }
      if constexpr (!kWing) {
        bool waves = nh || flat_all;
        // More huge items than a wave holds: one CTA each, unless the longest would outlast the rest
        // (every wave costs three barriers; 472 items in waves of one took 22 ms on 44 CTAs, one CTA each 5).
        if (nh > ng && !flat_all) {
          const unsigned long long sum = *(volatile unsigned long long*)&ctl->huge_sum[par];
          const unsigned long long longest = *(volatile unsigned long long*)&ctl->huge_max[par];
          if (longest <= 4 * (sum / vgrid()) + 4096ull * (nh / ng)) {
            waves = false;
            for (unsigned u0 = vblock(); u0 < nh;) {
              if (threadIdx.x == 0) S.item = atomicAdd(&ctl->cur_huge[par], 1u);
              const uint4 it = W.fhuge[par][u0];
              if (it.w) tip_item_block(G, W, ctl, it.x, pool, S, Q, A);
              __syncthreads();
              u0 = vgrid() + S.item;
              __syncthreads();
            }
          }
        }
        if (waves) {
          const unsigned total = flat_all ? items : nh;
          for (unsigned w0 = 0; w0 < total; w0 += ng) {
            const unsigned n = min(ng, total - w0);
            const TipWave V{W.fhuge[par] + w0, W.front[par], W.N - 1, nh > w0 ? min(n, nh - w0) : 0u, nb, n};
            clear_lists = total <= ng && tip_items_lists(G, W, ctl, V, false, S, kept, A);
            if (!clear_lists) tip_items_flat(G, W, ctl, V, false, S, kept, A);
            if (total > ng) {  // the slices are reused by the next wave or round
              if (!grid_barrier(ctl)) return false;
              tip_items_flat(G, W, ctl, V, true, S, kept, A);
              if (w0 + ng < total && !grid_barrier(ctl)) return false;
            } else {  // cleared by the next round
              clear_n = n;
              clear_nh = V.nh;
              clear_nb = nb;
            }
          }
        }
      }
    }
    {
      unsigned long long mn = A.mn;
      if (__any_sync(0xffffffffu, mn != kInf)) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mn = min(mn, __shfl_xor_sync(0xffffffffu, mn, o));
        if (lane == 0) atomicMin(&ctl->nm[npar], mn);
      }
      work += A.work;
    }
    if (!grid_barrier(ctl, &ctl->nm[npar], &ctl->near_len)) return false;
    next_k = s_words[0];
    near_len = (unsigned)s_words[1];
    phase_mark(trace, 2, round_est);
  }
  work = warp_sum(work);
  if (lane == 0 && work) atomicAdd(&ctl->work, work);
  flush_stats(ctl);
  return true;
}

// kMinBlocks: CTAs per SM the register allocation must allow.  2 caps a thread at 64 registers
// (some spill); 1 leaves 128 and no spills, at half the resident warps.  The single-
// instance tip peel runs faster on the latter (light rounds: fewer CTAs also shorten its grid
// barriers), and so does the wing peel while its rounds are light; with more edges the rounds are
// heavy and the intersections need the warps.  Wing peel of R-MAT graphs, one against two CTAs:
// 2^18 edges 186 / 213 ms, 2^20 566 / 643, 2^21 1040 / 1147, 2^22 2032 / 2122, 2^23 4167 / 4128,
// 2^24 9248 / 8514.
// Fewer edges take two as well where rounds are heavy, since edges alike are peeled together: the dearest edge
// is within four times the mean of the estimated work, and the mean is not small; and where most work lies with
// probe sets too long for shared memory, since probes wait for device memory.  One against two CTAs (in brackets
// dearest / mean, mean, share of long sets):
//   K_{60,3000} 118 / 81 ms (1, 180,000, 0), uniform 2000 x 2000 with 4e5 edges 61 / 47 (1.3, 35,000, 0),
//   1500 x 1500 with 1e5 9.4 / 8.8 (1.4, 4,086, 0), 3000 x 3000 with 6e4 1.01 / 1.13 (2, 386, 0);
//   four hubs of 20,000 39.7 / 26.4 (2.2, 35,600, 1.0), two 17.8 / 14.1 (10, 4,115, 0.9);
//   Zipf with 3e5 edges 139 / 168 (20, 7,800, 0.05), R-MAT as above (12 to 24, 10,800 to 30,000, at most 0.01).
// Asking takes a wait of the host, which is left out where edges are few or, by their degrees, cheap.
// Batches keep two (more graphs at a time).
constexpr int64_t kWingOneCta = int64_t(6) << 20;
constexpr int64_t kWingAskSpread = int64_t(1) << 15;
constexpr int64_t kWingHeavyMean = 2048;
template <bool kWing, int kMinBlocks>
__global__ void __launch_bounds__(kPT, kMinBlocks) peel_kernel(Lists G, const Lists* levels, Instances I, Ctl* ctls,
                                                               Classify cls) {
  // levels: the live-list versions of a two-phase fine pass (an instance reads
  // levels[W.level]); null: every instance reads G.
  __shared__ Work sW;
  __shared__ Lists sG;
  const unsigned ib = I.n > 1 ? I.cta_beg[blockIdx.x] : 0u, ie = I.n > 1 ? I.cta_end[blockIdx.x] : 1u;
  for (unsigned inst = ib; inst < ie; ++inst) {
    if (threadIdx.x == 0) {
      s_vb = I.n > 1 ? blockIdx.x - I.first[inst] : blockIdx.x;
      s_vg = I.n > 1 ? I.ncta[inst] : gridDim.x;
      sW = I.W[inst];
      sG = levels ? levels[sW.level] : G;
    }
    __syncthreads();
    if (!peel_instance<kWing>(sG, sW, ctls + inst, cls)) return;
    __syncthreads();
  }
}

// ---- set-up kernels -------------------------------------------------------------------------
__global__ void peel_init_kernel(const int64_t* __restrict__ counts, int64_t N, int64_t* D, int64_t* cnt,
                                 uint8_t* state) {
  for (int64_t x = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; x < N; x += (int64_t)gridDim.x * blockDim.x) {
    const int64_t c = counts[x];
    D[x] = c;
    cnt[x] = c;
    state[x] = ALIVE;
  }
}

// wk[u] = sum over v in N(u) of (deg(v) - 1): the two-hop wedges of a count-side vertex.
__global__ void tip_work_kernel(const uint32_t* __restrict__ offK, const uint32_t* __restrict__ edgK,
                                const uint32_t* __restrict__ offC, int64_t nK, int64_t* wk) {
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const unsigned lane = threadIdx.x & 31u;
  for (int64_t u = warp; u < nK; u += nwarps) {
    int64_t s = 0;
    for (uint32_t j = offK[u] + lane; j < offK[u + 1]; j += 32) {
      const uint32_t v = edgK[j];
      s += (int64_t)(offC[v + 1] - offC[v]) - 1;
    }
    s = warp_sum(s);
    if (lane == 0) wk[u] = s;
  }
}

// S[x] = sum over neighbours y of deg(y), for both sides (count side first).
__global__ void nbr_degree_sum_kernel(const uint32_t* __restrict__ off, const uint32_t* __restrict__ edg,
                                      const uint32_t* __restrict__ off_other, int64_t n, int64_t* S) {
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const unsigned lane = threadIdx.x & 31u;
  for (int64_t x = warp; x < n; x += nwarps) {
    int64_t s = 0;
    for (uint32_t j = off[x] + lane; j < off[x + 1]; j += 32) {
      const uint32_t y = edg[j];
      s += (int64_t)(off_other[y + 1] - off_other[y]);
    }
    s = warp_sum(s);
    if (lane == 0) S[x] = s;
  }
}

__global__ void center_of_kernel(const uint32_t* __restrict__ offC, int64_t nC, uint32_t* center_of) {
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const unsigned lane = threadIdx.x & 31u;
  for (int64_t v = warp; v < nC; v += nwarps)
    for (uint32_t j = offC[v] + lane; j < offC[v + 1]; j += 32) center_of[j] = (uint32_t)v;
}

// out[0] = the maximum of a, out[1] = how many entries lie above `above`.
__global__ void max_i64_kernel(const int64_t* __restrict__ a, int64_t n, int64_t above, unsigned long long* out) {
  unsigned long long m = 0, c = 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    m = max(m, (unsigned long long)a[i]);
    c += a[i] > above;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
  c = warp_sum(c);
  if ((threadIdx.x & 31) == 0) {
    atomicMax(out, m);
    if (c) atomicAdd(out + 1, c);
  }
}

// Live-entry count per vertex.  kByEdge: an entry is live when its edge is not peeled
// (wing); otherwise when its neighbour (a count-side vertex) is not peeled (tip, centre lists).
template <bool kByEdge>
__global__ void live_degree_kernel(const uint32_t* __restrict__ off, const uint32_t* __restrict__ nbr,
                                   const uint32_t* __restrict__ eid, int64_t n, const uint8_t* __restrict__ state,
                                   uint32_t* deg) {
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const unsigned lane = threadIdx.x & 31u;
  for (int64_t x = warp; x < n; x += nwarps) {
    uint32_t c = 0;
    for (uint32_t p = off[x] + lane; p < off[x + 1]; p += 32)
      c += state[kByEdge ? eid[p] : nbr[p]] == ALIVE;
    c = warp_sum(c);
    if (lane == 0) deg[x] = c;
  }
}

// Stable filter of every list to its live entries (order kept, so lists stay ascending).
template <bool kByEdge>
__global__ void compact_lists_kernel(const uint32_t* __restrict__ off, const uint32_t* __restrict__ nbr,
                                     const uint32_t* __restrict__ eid, int64_t n, const uint8_t* __restrict__ state,
                                     const uint32_t* __restrict__ noff, uint32_t* nnbr, uint32_t* neid) {
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const unsigned lane = threadIdx.x & 31u;
  for (int64_t x = warp; x < n; x += nwarps) {
    uint32_t dst = noff[x];
    const uint32_t e = off[x + 1];
    for (uint32_t p0 = off[x]; p0 < e; p0 += 32) {
      const uint32_t p = p0 + lane;
      bool live = false;
      uint32_t y = 0, id = 0;
      if (p < e) {
        y = nbr[p];
        id = eid ? eid[p] : 0u;
        live = state[kByEdge ? id : y] == ALIVE;
      }
      const unsigned bal = __ballot_sync(0xffffffffu, live);
      if (live) {
        const uint32_t at = dst + __popc(bal & ((1u << lane) - 1u));
        nnbr[at] = y;
        if (neid) neid[at] = id;
      }
      dst += __popc(bal);
    }
  }
}

__global__ void iota_kernel(uint32_t* a, int64_t n) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    a[i] = (uint32_t)i;
}

int grid_for(int64_t n, int per_block = 256) { return std::max(1, std::min(ceil_div(n, per_block), sm_count() * 16)); }

// One version of one side's live lists.
struct ListVersion {
  DevBuf<uint32_t> off, nbr, eid;
};

// One side's live lists: every compaction makes a new version from the current one.  With
// keep_all (two-phase peel) every version stays: the fine pass reads, for each partition, the
// newest version that still holds all of its items.  Otherwise only the newest stays.
struct LiveSide {
  std::vector<std::unique_ptr<ListVersion>> ver;
  int64_t n = 0;
  bool keep_all = false;
};

template <bool kByEdge>
void compact_side(LiveSide& L, const uint32_t* off, const uint32_t* nbr, const uint32_t* eid, const uint8_t* state,
                  bool with_eid, cudaStream_t s) {
  auto nv = std::make_unique<ListVersion>();
  DevBuf<uint32_t> deg(L.n > 0 ? L.n : 1, s);
  if (L.n) PB_LAUNCH(live_degree_kernel<kByEdge>, grid_for(L.n * 32), 256, 0, s, off, nbr, eid, L.n, state, deg.get());
  nv->off.alloc(L.n + 1, s);
  exclusive_scan_u32(deg.get(), nv->off.get(), L.n, s);
  uint32_t live = 0;
  PB_CUDA_TRY(cudaMemcpyAsync(&live, nv->off.get() + L.n, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
  PB_CUDA_TRY(cudaStreamSynchronize(s));
  nv->nbr.alloc(live + 1, s);
  if (with_eid) nv->eid.alloc(live + 1, s);
  if (L.n)
    PB_LAUNCH(compact_lists_kernel<kByEdge>, grid_for(L.n * 32), 256, 0, s, off, nbr, with_eid ? eid : nullptr, L.n,
              state, nv->off.get(), nv->nbr.get(), with_eid ? nv->eid.get() : nullptr);
  if (!L.keep_all) L.ver.clear();  // stream-ordered frees, after the compaction has read them
  L.ver.push_back(std::move(nv));
}

// {error bits OR-ed, unpeeled items summed} over the control blocks of one launch.
__global__ void ctl_status_kernel(const Ctl* __restrict__ ctls, unsigned n, unsigned* out) {
  unsigned err = 0, alive = 0;
  for (unsigned i = threadIdx.x; i < n; i += blockDim.x) {
    err |= ctls[i].err;
    alive += ctls[i].alive;
  }
  err = __reduce_or_sync(0xffffffffu, err);
  alive = __reduce_add_sync(0xffffffffu, alive);
  if (threadIdx.x == 0) {
    out[0] = err;
    out[1] = alive;
  }
}

// Per partition of the coarse pass: items and summed estimated work (the fine pass's CTA
// shares); with part null, the totals over all items (partition 0).
template <bool kWing>
__global__ void part_stats_kernel(Lists G, Classify cls, const uint32_t* __restrict__ part, int64_t N,
                                  bool with_fixed, unsigned* cnt, unsigned long long* work) {
  for (int64_t x = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; x < N; x += (int64_t)gridDim.x * blockDim.x) {
    const uint32_t p = part ? part[x] : 0u;
    atomicAdd(&cnt[p], 1u);
    const unsigned long long w = item_weight<kWing>(G, cls, (uint32_t)x);
    // An item's fixed cost in its own units: a tip item takes a CTA about 5 us and 3.5 ns a wedge (a
    // partition of 2967 items of 800 wedges ran 20 ms on its one CTA, one of 18 items with three
    // quarters of the wedges 2.4 ms).
    const unsigned long long fixed = kWing ? 256ull : (w <= kTipWarpSlots ? 128ull : 1400ull);
    atomicAdd(&work[p], w + (with_fixed ? fixed : 0ull));
  }
}

template <bool kWing>
__global__ void item_weight_kernel(Lists G, Classify cls, int64_t N, uint32_t* wgt) {
  for (int64_t x = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; x < N; x += (int64_t)gridDim.x * blockDim.x) {
    const unsigned long long w = item_weight<kWing>(G, cls, (uint32_t)x);
    wgt[x] = (uint32_t)min(w, 0xFFFFFFFFull);
  }
}

// info[e]: how the item of edge e is peeled, from the current lists (the live lists shrink between
// launches).  Units are slices of about `chunk` estimated probes, never below twice the probe set
// (each unit rebuilds the probe table), at most one per first-level entry and 4096 in all;
// chunk grows with the summed cost (*total) so that a frontier of all items stays below 2^32 units.
// Warp-unit setting: every item whose probe set fits a warp table runs on warps, cut into units;
// otherwise only items of at most small_work probes run on warps, whole.
__global__ void wing_info_kernel(Lists G, Classify cls, int64_t N, const unsigned long long* __restrict__ total,
                                 uint32_t* info) {
  const int64_t chunk = max((int64_t)cls.chunk_work, (int64_t)(*total >> 30));
  for (int64_t x = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; x < N; x += (int64_t)gridDim.x * blockDim.x) {
    const uint32_t v = G.center_of[x], u = G.u_of[x];
    const int64_t cv = cls.cost_v(G, v, u), cu = cls.cost_u(G, v, u);
    const bool fv = cv <= cu;
    const int64_t cost = fv ? cv : cu;
    const int64_t du = G.offK[u + 1] - G.offK[u], dv = G.offC[v + 1] - G.offC[v];
    const int64_t psize = fv ? du : dv, d1 = fv ? dv : du;
    const bool small = psize <= (int64_t)kWingWarpSet && (cls.warp_units || cost <= cls.small_work);
    const int64_t unit = small ? chunk : max(chunk, kUnitSets * psize / 2);
    int64_t units = small && !cls.warp_units ? 1 : (cost + unit - 1) / unit;
    units = max((int64_t)1, min(units, min(d1, (int64_t)4096)));
    info[x] = (uint32_t)units | (small ? kInfoSmall : 0u) | (fv ? kInfoFromV : 0u);
  }
}

template <bool kWing>
__global__ void total_weight_kernel(Lists G, Classify cls, int64_t N, unsigned long long* total) {
  unsigned long long s = 0;
  for (int64_t x = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; x < N; x += (int64_t)gridDim.x * blockDim.x)
    s += item_weight<kWing>(G, cls, (uint32_t)x);
  s = warp_sum(s);
  if ((threadIdx.x & 31) == 0 && s) atomicAdd(total, s);
}

// out: summed estimated work of all edges, of those with a probe set above kWingSet, and the largest.
__global__ void wing_spread_kernel(Lists G, Classify cls, int64_t N, unsigned long long* out) {
  unsigned long long all = 0, wide = 0, most = 0;
  for (int64_t x = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; x < N; x += (int64_t)gridDim.x * blockDim.x) {
    const uint32_t v = G.center_of[x], u = G.u_of[x];
    const int64_t cv = cls.cost_v(G, v, u), cu = cls.cost_u(G, v, u);
    const int64_t psize = cv <= cu ? G.offK[u + 1] - G.offK[u] : G.offC[v + 1] - G.offC[v];
    const unsigned long long w = item_weight<true>(G, cls, (uint32_t)x);
    all += w;
    if (psize > (int64_t)kWingSet) wide += w;
    most = max(most, w);
  }
  all = warp_sum(all);
  wide = warp_sum(wide);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) most = max(most, __shfl_xor_sync(0xffffffffu, most, o));
  if ((threadIdx.x & 31) == 0 && all) {
    atomicAdd(out, all);
    if (wide) atomicAdd(out + 1, wide);
    atomicMax(out + 2, most);
  }
}

// gid[x] = i for the items x in [base[i], base[i + 1]) (one CTA per range).
__global__ void range_ids_kernel(const uint32_t* __restrict__ base, uint32_t n, const uint32_t* unused, uint32_t* gid) {
  const uint32_t i = blockIdx.x;
  if (i >= n) return;
  for (uint32_t x = base[i] + threadIdx.x; x < base[i + 1]; x += blockDim.x) gid[x] = i;
}

// key[x] = pbase[gid[x]] + part[x]: graph-major global partition ids of a batch.
__global__ void global_part_kernel(const uint32_t* __restrict__ gid, const uint32_t* __restrict__ part,
                                   const uint32_t* __restrict__ pbase, int64_t N, uint32_t* key) {
  for (int64_t x = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; x < N; x += (int64_t)gridDim.x * blockDim.x)
    key[x] = pbase[gid[x]] + part[x];
}

// Splits `grid` CTAs among instances by weight: an instance whose share is at least one CTA
// gets a CTA range of its own (its barriers span only that range); the light ones are packed,
// longest first onto the least-loaded CTA, into the CTAs left over, where they run one after
// another.  Fills the launch order (slot -> instance), each slot's first CTA and CTA count,
// and each CTA's slot range.
void assign_ctas(const std::vector<double>& pweight, int grid, std::vector<int>& inst_of, std::vector<uint32_t>& first,
                 std::vector<uint32_t>& cnt, std::vector<uint32_t>& cbeg, std::vector<uint32_t>& cend) {
  const int ninst = (int)pweight.size();
  std::vector<int> ord(ninst);
  for (int i = 0; i < ninst; ++i) ord[i] = i;
  std::sort(ord.begin(), ord.end(), [&](int a, int b) { return pweight[a] > pweight[b]; });
  double wsum = 0;
  for (double w : pweight) wsum += w;
  int nheavy = 0;
  while (nheavy < ninst && pweight[ord[nheavy]] / wsum * grid >= 1.0) ++nheavy;
  double lw = 0;
  for (int j = nheavy; j < ninst; ++j) lw += pweight[ord[j]];
  int light_ctas = 0;
  if (nheavy < ninst) light_ctas = std::min(ninst - nheavy, std::max(1, (int)std::ceil(lw / wsum * grid)));
  // Heavy instances share the rest; demote the lightest ones while they outnumber it.
  while (nheavy > grid - light_ctas) {
    --nheavy;
    if (!light_ctas) light_ctas = 1;
  }
  if (!nheavy) light_ctas = std::min(grid, ninst);
  const int hbudget = grid - light_ctas;
  std::vector<int> ncta(ninst, 0);
  if (nheavy) {
    double hw = 0;
    for (int j = 0; j < nheavy; ++j) hw += pweight[ord[j]];
    int total = 0;
    for (int j = 0; j < nheavy; ++j) {
      ncta[ord[j]] = std::max(1, (int)(pweight[ord[j]] / hw * hbudget));
      total += ncta[ord[j]];
    }
    for (int j = 0; total < hbudget; j = (j + 1) % nheavy, ++total) ++ncta[ord[j]];
    while (total > hbudget) {  // some instance has more than one CTA here (hbudget >= nheavy)
      int k = ord[0];
      for (int j = 1; j < nheavy; ++j)
        if (ncta[ord[j]] > ncta[k]) k = ord[j];
      --ncta[k];
      --total;
    }
  }
  inst_of.clear();
  first.clear();
  cnt.clear();
  cbeg.assign(grid, 0);
  cend.assign(grid, 0);
  uint32_t cta = 0;
  for (int j = 0; j < nheavy; ++j) {
    const int i = ord[j];
    for (int c = 0; c < ncta[i]; ++c) {
      cbeg[cta + c] = (uint32_t)inst_of.size();
      cend[cta + c] = (uint32_t)inst_of.size() + 1;
    }
    inst_of.push_back(i);
    first.push_back(cta);
    cnt.push_back((uint32_t)ncta[i]);
    cta += (uint32_t)ncta[i];
  }
  if (nheavy < ninst) {
    std::vector<std::vector<int>> bins(light_ctas);
    std::vector<double> load(light_ctas, 0.0);
    for (int j = nheavy; j < ninst; ++j) {
      const int b = (int)(std::min_element(load.begin(), load.end()) - load.begin());
      bins[b].push_back(ord[j]);
      load[b] += pweight[ord[j]];
    }
    for (int b = 0; b < light_ctas; ++b, ++cta) {
      cbeg[cta] = (uint32_t)inst_of.size();
      for (int i : bins[b]) {
        inst_of.push_back(i);
        first.push_back(cta);
        cnt.push_back(1u);
      }
      cend[cta] = (uint32_t)inst_of.size();
    }
  }
}

template <bool kWing>
PeelResult run_peel(const pb_graph& g, int use_v, const int64_t* counts, int64_t* out, cudaStream_t s,
                    const PeelTuning& tune, const PeelParts* parts) {
  PeelResult res;
  Lists G{};
  const uint32_t* offK0 = use_v ? g.offU.get() : g.offV.get();
  const uint32_t* edgK0 = use_v ? g.edgU.get() : g.edgV.get();
  const uint32_t* offC0 = use_v ? g.offV.get() : g.offU.get();
  const uint32_t* edgC0 = use_v ? g.edgV.get() : g.edgU.get();
  G.nK = use_v ? g.nu : g.nv;
  G.nC = use_v ? g.nv : g.nu;
  const int64_t N = kWing ? g.m : G.nK;
  if (N == 0) return res;
  PB_REQUIRE(N < (int64_t)UINT32_MAX, PB_ETOOBIG, "too many items to peel");
  G.offK = offK0;
  G.edgK = edgK0;
  G.offC = offC0;
  G.edgC = edgC0;
  const bool batch = parts && parts->base.size() > 1;
  // Two-phase peel (a schedule of the same rounds, never a different result): a coarse pass
  // cuts the items into partitions of about equal estimated work by ranges of their final
  // numbers, then every partition runs its exact rounds as an independent instance.
  bool two_phase_req = tune.two_phase;
  double parts_per_cta = tune.parts_per_cta;
  int64_t parts_total = tune.parts_total;
  if (const char* e = getenv("PB_PEEL_TWO_PHASE")) {  // diagnostic hook: partitions per CTA, 0 = off
    parts_per_cta = atof(e);
    parts_total = 0;
    two_phase_req = parts_per_cta > 0;
  }
  const bool two_phase = !batch && two_phase_req && g_recorder == nullptr;
  const bool two_phase_batch = batch && two_phase_req && g_recorder == nullptr;

  DevBuf<int64_t> cnt(N, s);
  DevBuf<uint32_t> eti, iota, center_of, alist0(N, s), alist1(N, s), nearl(N, s);
  DevBuf<uint4> fr0(N, s), fr1(N, s), fh0, fh1;
  // Independent instances (the graphs of a batch) or the whole input as one.
  std::vector<int64_t> pbase{0}, psize{N};
  std::vector<double> pweight{1.0};
  if (batch) {
    pbase.clear();
    psize.clear();
    pweight.clear();
    for (size_t i = 0; i < parts->base.size(); ++i) {
      if (parts->size[i] <= 0) continue;
      pbase.push_back(parts->base[i]);
      psize.push_back(parts->size[i]);
      pweight.push_back(std::max(parts->weight[i], 1.0));
    }
    if (pbase.empty()) return res;
  }
  // Grid-shared dense counters: tip peeling keeps one slice per heavy item of a wave (they run
  // concurrently), up to kMaxGroups slices within kGsharedBudget.  A slice is indexed by the peeled
  // side, whose vertices also bound the items of a wave (sized by the longer side, the slices of a
  // peel of 40 vertices against 400,000 were 205 MB to clear: 0.94 ms, now 0.80).  Slices share no line of
  // memory, nor neighbouring ones: their adds would wait for one another (tip peel of K_{8,50000} with slices
  // of 9 words 0.84 ms, of 64 words or more 0.51).
  const int64_t gstride = (G.nK + 64) / 32 * 32;
  const unsigned ngroups = (unsigned)std::max<int64_t>(
      1, std::min<int64_t>(std::min<int64_t>(kMaxGroups, G.nK), kGsharedBudget / (4 * gstride)));
  DevBuf<uint32_t> gshared;
  if (!kWing) {
    gshared.alloc((size_t)gstride * ngroups, s);
    PB_CUDA_TRY(cudaMemsetAsync(gshared.get(), 0, gshared.bytes(), s));
  }
  DevBuf<uint8_t> state(N, s);
  LiveSide liveK, liveC;
  liveK.n = G.nK;
  liveC.n = G.nC;
  liveK.keep_all = liveC.keep_all = two_phase;
  DevBuf<int64_t> snap;  // two-phase: every item's count when its partition opens
  DevBuf<uint32_t> part;
  if (two_phase || two_phase_batch) {
    snap.alloc(N, s);
    part.alloc(N, s);
  }
  PB_LAUNCH(peel_init_kernel, grid_for(N), 256, 0, s, counts, N, (two_phase || two_phase_batch) ? snap.get() : out,
            cnt.get(), state.get());
  Classify cls{tune.small_work, tune.huge_work, tune.chunk_work, std::max<int64_t>(1, tune.units_per_cta),
               tune.warp_units ? 1 : 0};
  if (const char* e = getenv("PB_PEEL_WARP_UNITS")) cls.warp_units = atoi(e) != 0;  // diagnostic hook
  // Thresholds may be lowered through the environment (tests use this to drive small graphs
  // through the CTA- and grid-level paths).
  if (const char* e = getenv("PB_PEEL_SMALL_WORK")) cls.small_work = atoll(e);
  if (const char* e = getenv("PB_PEEL_HUGE_WORK")) cls.huge_work = atoll(e);
  if (const char* e = getenv("PB_PEEL_CHUNK_WORK")) cls.chunk_work = atoll(e);
  // Work estimates of the lists a version holds: neighbour-degree sums (wing) or two-hop wedges
  // (tip).
  std::vector<std::unique_ptr<DevBuf<int64_t>>> work_bufs;
  std::vector<std::unique_ptr<DevBuf<uint32_t>>> info_bufs;
  auto refresh_work = [&](Lists& L) {
    if (!two_phase) {  // stream-ordered: whoever reads the old ones has been launched
      work_bufs.clear();
      info_bufs.clear();
    }
    auto buf = std::make_unique<DevBuf<int64_t>>(kWing ? L.nK + L.nC : L.nK, s);
    if (kWing) {
      if (L.nK) PB_LAUNCH(nbr_degree_sum_kernel, grid_for(L.nK * 32), 256, 0, s, L.offK, L.edgK, L.offC, L.nK, buf->get());
      if (L.nC)
        PB_LAUNCH(nbr_degree_sum_kernel, grid_for(L.nC * 32), 256, 0, s, L.offC, L.edgC, L.offK, L.nC, buf->get() + L.nK);
      L.S = buf->get();
      auto info = std::make_unique<DevBuf<uint32_t>>(N, s);
      DevBuf<unsigned long long> total(1, s);
      PB_CUDA_TRY(cudaMemsetAsync(total.get(), 0, sizeof(unsigned long long), s));
      PB_LAUNCH(total_weight_kernel<kWing>, grid_for(N), 256, 0, s, L, cls, N, total.get());
      PB_LAUNCH(wing_info_kernel, grid_for(N), 256, 0, s, L, cls, N, total.get(), info->get());
      L.info = info->get();
      info_bufs.push_back(std::move(info));
    } else {
      PB_LAUNCH(tip_work_kernel, grid_for(L.nK * 32), 256, 0, s, L.offK, L.edgK, L.offC, L.nK, buf->get());
      L.wk = buf->get();
    }
    work_bufs.push_back(std::move(buf));
  };
  bool need_scratch = false;
  int64_t scratch_len = 0;
  int64_t n_huge = 0;  // tip items that may run over the whole grid (the lists only shrink)
  if (kWing) {
    eti.alloc(g.m, s);
    iota.alloc(g.m, s);
    center_of.alloc(g.m, s);
    edge_to_idxs(g, use_v, eti.get(), s);
    PB_LAUNCH(iota_kernel, grid_for(g.m), 256, 0, s, iota.get(), g.m);
    PB_LAUNCH(center_of_kernel, grid_for(G.nC * 32), 256, 0, s, G.offC, G.nC, center_of.get());
    G.eidK = eti.get();
    G.eidC = iota.get();
    G.center_of = center_of.get();
    G.u_of = edgC0;  // edge ids are positions in the centre side's original lists
    refresh_work(G);
    need_scratch = g.max_deg > kWingSet;
    scratch_len = std::max(G.nK, G.nC);
  } else {
    refresh_work(G);
    DevBuf<unsigned long long> mx(2, s);
    PB_CUDA_TRY(cudaMemsetAsync(mx.get(), 0, 2 * sizeof(unsigned long long), s));
    PB_LAUNCH(max_i64_kernel, grid_for(G.nK), 256, 0, s, G.wk, G.nK, cls.huge_work, mx.get());
    unsigned long long hmx[2];
    readback(hmx, mx.get(), sizeof(hmx), s);
    need_scratch = 2ull * hmx[0] > (uint64_t)kTipSlots;
    scratch_len = G.nK;
    // One list for all heavy items of a round; the graphs of a batch have a stretch of N each.
    n_huge = (int64_t)hmx[1];
    fh0.alloc(batch ? N : n_huge + 1, s);
    fh1.alloc(batch ? N : n_huge + 1, s);
  }
  const Lists G0 = G;  // the full lists (version 0)

  const size_t smem = ((sizeof(Shared) + 15) & ~size_t(15)) + (size_t)kPoolWords * sizeof(uint32_t);
  void (*kern)(Lists, const Lists*, Instances, Ctl*, Classify) = peel_kernel<kWing, 2>;
  if constexpr (!kWing) {
    if (!batch) kern = peel_kernel<false, 1>;
  } else {
    bool one = !two_phase && g.m <= kWingOneCta;
    // Two CTAs per SM double the markers of long probe sets; above 4 GiB that is not worth it.
    const bool room = !need_scratch || 2 * (int64_t)sm_count() * scratch_len * 4 <= int64_t(4) << 30;
    if (one && room && g.m > kWingAskSpread && (int64_t)g.max_deg * g.max_deg >= kWingHeavyMean) {
      DevBuf<unsigned long long> spread(3, s);
      PB_CUDA_TRY(cudaMemsetAsync(spread.get(), 0, spread.bytes(), s));
      PB_LAUNCH(wing_spread_kernel, std::min(grid_for(N), 2 * sm_count()), 256, 0, s, G, cls, N, spread.get());
      unsigned long long h[3];
      readback(h, spread.get(), sizeof(h), s);
      const double mean = (double)h[0] / (double)N;
      one = h[1] <= h[0] / 2 && (mean < (double)kWingHeavyMean || (double)h[2] > 4.0 * mean);
    }
    if (one) kern = peel_kernel<true, 1>;
  }
  PB_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int per_sm = 0;
  PB_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kPT, smem));
  PB_REQUIRE(per_sm >= 1, PB_ECUDA, "peeling kernel does not fit on an SM");
  int grid = sm_count() * per_sm;
  // A single instance may run on fewer CTAs: its barriers and grid-stride phases then span
  // fewer CTAs, which shortens light rounds.
  int64_t cap = batch ? 0 : tune.max_ctas;
  if (const char* e = getenv("PB_PEEL_CTAS")) cap = atoll(e);  // diagnostic hook
  if (cap > 0) grid = (int)std::max<int64_t>(1, std::min<int64_t>(grid, cap));

  // The fine pass of a two-phase tip peel runs many small instances: two CTAs per SM give each of
  // them a CTA of its own (R-MAT 2^22 edges, 296 partitions asked for: 64.2 ms against 66.3).
  auto fine_kern = kern;
  int fine_grid = grid;
  if (!kWing && two_phase && cap <= 0) {
    fine_kern = peel_kernel<kWing, 2>;
    PB_CUDA_TRY(cudaFuncSetAttribute(fine_kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    PB_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fine_kern, kPT, smem));
    fine_grid = sm_count() * std::max(1, per_sm);
    // ... unless their dense counters would take more than half of what is left of the device (the
    // fine pass's lists are still to come).  Below 4 GiB there is nothing to ask.
    const size_t scratch = need_scratch ? (size_t)fine_grid * (size_t)scratch_len * sizeof(uint32_t) : 0;
    if (fine_grid > grid && scratch > size_t(4) << 30 && scratch > device_bytes_left() / 2) {
      fine_kern = kern;
      fine_grid = grid;
    }
  }

  DevBuf<uint32_t> gscratch;
  if (need_scratch) {
    gscratch.alloc((size_t)std::max(grid, fine_grid) * (size_t)scratch_len, s);
    PB_CUDA_TRY(cudaMemsetAsync(gscratch.get(), 0, gscratch.bytes(), s));
  }
  Work W{};
  W.D = (two_phase || two_phase_batch) ? snap.get() : out;
  W.cnt = cnt.get();
  W.state = state.get();
  W.alist[0] = alist0.get();
  W.alist[1] = alist1.get();
  W.near = nearl.get();
  W.front[0] = fr0.get();
  W.front[1] = fr1.get();
  W.fhuge[0] = fh0.get();
  W.fhuge[1] = fh1.get();
  W.gshared = gshared.get();
  W.gshared_stride = gstride;
  W.ngroups = ngroups;
  W.gscratch = gscratch.get();
  W.gscratch_len = scratch_len;
  W.tip_cb = 31;
  while (W.tip_cb > 1 && ((uint64_t)(G.nK - 1) >> (32 - W.tip_cb)) != 0) --W.tip_cb;
  W.N = N;
  W.item0 = 0;
  W.part_out = two_phase ? part.get() : nullptr;

  Ctl hctl;
  std::memset(&hctl, 0, sizeof(hctl));
  hctl.nm[0] = kInf;
  hctl.nm[1] = kInf;
  hctl.k_lo = kInf;
  hctl.alive = (unsigned)N;
  hctl.alen[0] = (unsigned)N;
  hctl.alive_at_compact = (unsigned)N;
  hctl.min_gain = (unsigned)std::max<int64_t>(1 << 16, N / 64);
  // A recorded / captured pipeline runs the peel as one launch without list compaction (the
  // host cannot step in between launches of a CUDA graph); so do per-graph instances.
  if (g_recorder != nullptr || batch) hctl.min_gain = 0xFFFFFFFFu;
  hctl.barrier_timeout_ns = kBarrierTimeoutNs;
  const bool trace = [] {
    const char* tr = getenv("PB_TRACE");
    return tr && *tr && *tr != '0';
  }();
  hctl.trace = trace ? 1u : 0u;
  hctl.near_min = (unsigned)tune.near_min;
  hctl.near_div = (unsigned)tune.near_div;
  // Diagnostic hooks for the window size.
  if (const char* e = getenv("PB_PEEL_NEAR_MIN")) hctl.near_min = (unsigned)strtoul(e, nullptr, 10);
  if (const char* e = getenv("PB_PEEL_NEAR_DIV")) hctl.near_div = (unsigned)strtoul(e, nullptr, 10);
  if (const char* e = getenv("PB_PEEL_BARRIER_TIMEOUT_MS")) hctl.barrier_timeout_ns = 1000000ull * strtoull(e, nullptr, 10);
  // Test hook: CTA 0 skips its arrivals, so the first grid barrier cannot complete and every
  // wait runs out; checks that a timeout comes back as PB_ETIMEOUT with the context usable.
  if (const char* e = getenv("PB_PEEL_TEST_STUCK_BARRIER"))
    if (*e && *e != '0') hctl.test_skip_arrival = 1;
  DevBuf<unsigned> status(2, s);
  DevBuf<uint32_t> wgt;  // coarse passes: static per-item work estimates
  if (two_phase || two_phase_batch) {
    wgt.alloc(N, s);
    PB_LAUNCH(item_weight_kernel<kWing>, grid_for(N), 256, 0, s, G0, cls, N, wgt.get());
    W.wgt = wgt.get();
  }

  // One cooperative launch of independent instances with CTA shares by weight (no compaction
  // pauses: every instance runs to its end).  per_slot may adjust each launch slot's Work.
  auto launch_instances = [&](const std::vector<Work>& wproto, const std::vector<Ctl>& cproto,
                              const std::vector<double>& weights, const Lists* levels_dev,
                              const std::function<void(Work&, uint32_t)>& per_slot,
                              std::vector<Ctl>* inst_out = nullptr, bool fine = false) {
    const auto lkern = fine ? fine_kern : kern;
    const int lgrid = fine ? fine_grid : grid;
    std::vector<int> inst_of;
    std::vector<uint32_t> first, ncta, cbeg, cend;
    assign_ctas(weights, lgrid, inst_of, first, ncta, cbeg, cend);
    const int n_slots = (int)inst_of.size();
    std::vector<Work> ws(n_slots);
    std::vector<Ctl> hctls(n_slots);
    for (int q = 0; q < n_slots; ++q) {
      ws[q] = wproto[inst_of[q]];
      hctls[q] = cproto[inst_of[q]];
      if (per_slot) per_slot(ws[q], ncta[q]);
    }
    DevBuf<Ctl> ctls(n_slots, s);
    DevBuf<Work> dws(n_slots, s);
    DevBuf<uint32_t> meta(2 * (size_t)n_slots + 2 * (size_t)lgrid, s);
    std::vector<uint32_t> hmeta;
    hmeta.insert(hmeta.end(), first.begin(), first.end());
    hmeta.insert(hmeta.end(), ncta.begin(), ncta.end());
    hmeta.insert(hmeta.end(), cbeg.begin(), cbeg.end());
    hmeta.insert(hmeta.end(), cend.begin(), cend.end());
    const void* src_c = hctls.data();
    const void* src_w = ws.data();
    const void* src_m = hmeta.data();
    if (capturing()) {  // the graph copies from host memory that outlives it
      void* pc = g_recorder->pinned_alloc(sizeof(Ctl) * n_slots);
      void* pw = g_recorder->pinned_alloc(sizeof(Work) * n_slots);
      void* pm = g_recorder->pinned_alloc(sizeof(uint32_t) * hmeta.size());
      std::memcpy(pc, src_c, sizeof(Ctl) * n_slots);
      std::memcpy(pw, src_w, sizeof(Work) * n_slots);
      std::memcpy(pm, src_m, sizeof(uint32_t) * hmeta.size());
      src_c = pc;
      src_w = pw;
      src_m = pm;
    }
    PB_CUDA_TRY(cudaMemcpyAsync(ctls.get(), src_c, sizeof(Ctl) * n_slots, cudaMemcpyHostToDevice, s));
    PB_CUDA_TRY(cudaMemcpyAsync(dws.get(), src_w, sizeof(Work) * n_slots, cudaMemcpyHostToDevice, s));
    PB_CUDA_TRY(cudaMemcpyAsync(meta.get(), src_m, sizeof(uint32_t) * hmeta.size(), cudaMemcpyHostToDevice, s));
    Instances I{dws.get(), meta.get(), meta.get() + n_slots, meta.get() + 2 * n_slots,
                meta.get() + 2 * n_slots + lgrid, (uint32_t)n_slots};
    Ctl* cp = ctls.get();
    Lists Gk = G0;
    const Lists* lv = levels_dev;
    void* args[] = {&Gk, &lv, &I, &cp, &cls};
    PB_CUDA_TRY(cudaLaunchCooperativeKernel((const void*)lkern, dim3(lgrid), dim3(kPT), args, smem, s));
    if (g_launch_counter) ++*g_launch_counter;
    PB_LAUNCH(ctl_status_kernel, 1, 32, 0, s, cp, (unsigned)n_slots, status.get());
    if (capturing()) {
      PB_CUDA_TRY(cudaMemcpyAsync(g_recorder->status, status.get(), 2 * sizeof(unsigned), cudaMemcpyDeviceToHost, s));
      return;
    }
    PB_CUDA_TRY(cudaMemcpyAsync(hctls.data(), cp, sizeof(Ctl) * n_slots, cudaMemcpyDeviceToHost, s));
    PB_CUDA_TRY(cudaStreamSynchronize(s));
    if (inst_out) inst_out->assign(wproto.size(), Ctl{});
    for (int q = 0; q < n_slots; ++q) {
      const Ctl& c = hctls[q];
      PB_REQUIRE(!(c.err & ERR_TIMEOUT), PB_ETIMEOUT, "peeling: a grid barrier wait ran out of time");
      PB_REQUIRE(c.err == 0, PB_ECUDA, "peeling: a table invariant was violated");
      PB_REQUIRE(c.alive == 0, PB_ECUDA, "peeling: an instance stopped with unpeeled items");
      res.rounds += (int64_t)c.rounds;
      res.fine_rounds_max = std::max<int64_t>(res.fine_rounds_max, (int64_t)c.rounds);
      res.work += (int64_t)c.work;
      if (inst_out) (*inst_out)[inst_of[q]] = c;
    }
  };

  // Fine passes: grid-shared counters, and the lists of the items that run on them, must be per instance,
  // since partitions share item ids.  Instances with a CTA range of their own get one slice each
  // while kGsharedBudget lasts; the others never take the grid-level path.
  const int64_t slices = std::max<int64_t>(1, kGsharedBudget / (4 * gstride));
  std::vector<DevBuf<uint32_t>> slice_bufs;
  std::vector<DevBuf<uint4>> heavy_bufs;
  auto heavy_lists = [&](Work& x, uint32_t ncta) {
    x.gshared = nullptr;
    x.fhuge[0] = x.fhuge[1] = nullptr;
    x.ngroups = 1;
    if (!kWing && ncta >= 2 && (int64_t)slice_bufs.size() < slices) {
      slice_bufs.emplace_back((size_t)gstride, s);
      PB_CUDA_TRY(cudaMemsetAsync(slice_bufs.back().get(), 0, slice_bufs.back().bytes(), s));
      x.gshared = slice_bufs.back().get();
      for (auto& f : x.fhuge) {
        heavy_bufs.emplace_back((size_t)std::min(x.N, n_huge), s);
        f = heavy_bufs.back().get();
      }
    }
  };

  auto release_coarse = [&] {  // what the coarse pass alone used
    gshared.release();
    fh0.release();
    fh1.release();
    wgt.release();
  };

  if (batch) {
    const int ninst = (int)pbase.size();
    std::vector<Work> ws(ninst, W);
    std::vector<Ctl> cs(ninst, hctl);
    for (int i = 0; i < ninst; ++i) {
      const int64_t b = pbase[i], n = psize[i];
      Work& x = ws[i];
      x.alist[0] = alist0.get() + b;
      x.alist[1] = alist1.get() + b;
      x.near = nearl.get() + b;
      x.front[0] = fr0.get() + b;
      x.front[1] = fr1.get() + b;
      x.fhuge[0] = kWing ? nullptr : fh0.get() + b;
      x.fhuge[1] = kWing ? nullptr : fh1.get() + b;
      x.N = n;
      x.item0 = (uint32_t)b;
      Ctl& c = cs[i];
      c.alive = (unsigned)n;
      c.alen[0] = (unsigned)n;
      c.alive_at_compact = (unsigned)n;
    }
    if (!two_phase_batch) {
      launch_instances(ws, cs, pweight, nullptr, nullptr);
      res.rounds = res.fine_rounds_max;  // a batch reports the rounds of its longest graph
      res.fine_rounds_max = 0;
      return res;
    }
    // Two-phase schedule per graph: a coarse pass with one range-mode instance per graph (about
    // parts_per_cta partitions per CTA, split by the graphs' work), then one fine instance per
    // (graph, partition).  Partition ids are local to a graph: items of different graphs never
    // meet in a list.
    DevBuf<uint32_t> gid(N, s);
    DevBuf<uint32_t> dbase(ninst + 1, s);
    std::vector<uint32_t> hb(ninst + 1);
    for (int i = 0; i < ninst; ++i) hb[i] = (uint32_t)pbase[i];
    hb[ninst] = (uint32_t)(pbase[ninst - 1] + psize[ninst - 1]);
    PB_CUDA_TRY(cudaMemcpyAsync(dbase.get(), hb.data(), sizeof(uint32_t) * (ninst + 1), cudaMemcpyHostToDevice, s));
    PB_LAUNCH(range_ids_kernel, ninst, 256, 0, s, dbase.get(), (uint32_t)ninst, (const uint32_t*)nullptr, gid.get());
    DevBuf<unsigned> icnt(ninst, s);
    DevBuf<unsigned long long> iwork(ninst, s);
    PB_CUDA_TRY(cudaMemsetAsync(icnt.get(), 0, sizeof(unsigned) * ninst, s));
    PB_CUDA_TRY(cudaMemsetAsync(iwork.get(), 0, sizeof(unsigned long long) * ninst, s));
    PB_LAUNCH(part_stats_kernel<kWing>, grid_for(N), 256, 0, s, G, cls, (const uint32_t*)gid.get(), N, false, icnt.get(),
              iwork.get());
    std::vector<unsigned long long> hiw(ninst);
    PB_CUDA_TRY(cudaMemcpyAsync(hiw.data(), iwork.get(), sizeof(unsigned long long) * ninst, cudaMemcpyDeviceToHost, s));
    PB_CUDA_TRY(cudaStreamSynchronize(s));
    double wsum = 0;
    for (unsigned long long w : hiw) wsum += (double)w;
    const double want = std::max(1.0, parts_total > 0 ? (double)parts_total : parts_per_cta * grid);
    for (int i = 0; i < ninst; ++i) {
      const double parts_i = std::max(1.0, std::round(want * (double)hiw[i] / std::max(1.0, wsum)));
      cs[i].range_mode = 1;
      cs[i].part_target = std::max<unsigned long long>(1, (unsigned long long)((double)hiw[i] / parts_i));
      ws[i].part_out = part.get();
    }
    std::vector<Ctl> coarse;
    launch_instances(ws, cs, pweight, nullptr, nullptr, &coarse);
    res.coarse_rounds = res.fine_rounds_max;
    res.rounds = 0;
    res.fine_rounds_max = 0;
    release_coarse();
    // Global partition keys (graph-major) and the fine instances in that order.
    std::vector<uint32_t> pb0(ninst + 1, 0);
    for (int i = 0; i < ninst; ++i) pb0[i + 1] = pb0[i] + std::max(1u, coarse[i].npart);
    const uint32_t ntot = pb0[ninst];
    DevBuf<uint32_t> dpb(ninst + 1, s), key(N, s);
    PB_CUDA_TRY(cudaMemcpyAsync(dpb.get(), pb0.data(), sizeof(uint32_t) * (ninst + 1), cudaMemcpyHostToDevice, s));
    PB_LAUNCH(global_part_kernel, grid_for(N), 256, 0, s, (const uint32_t*)gid.get(), (const uint32_t*)part.get(),
              (const uint32_t*)dpb.get(), N, key.get());
    int bits = 1;
    while (bits < 32 && (1ull << bits) < ntot) ++bits;
    DevBuf<uint32_t> key2(N, s), perm(N, s), perm2(N, s);
    PB_LAUNCH(iota_kernel, grid_for(N), 256, 0, s, perm.get(), N);
    const bool alt = radix_sort_pairs_u32(key.get(), perm.get(), key2.get(), perm2.get(), N, 0, bits, s);
    const uint32_t* items = alt ? perm2.get() : perm.get();
    // key still holds each item's global partition (radix_sort_pairs_u32 sorts into key / key2).
    PB_LAUNCH(global_part_kernel, grid_for(N), 256, 0, s, (const uint32_t*)gid.get(), (const uint32_t*)part.get(),
              (const uint32_t*)dpb.get(), N, key2.get());
    DevBuf<unsigned> pcnt(ntot, s);
    DevBuf<unsigned long long> pwork(ntot, s);
    PB_CUDA_TRY(cudaMemsetAsync(pcnt.get(), 0, sizeof(unsigned) * ntot, s));
    PB_CUDA_TRY(cudaMemsetAsync(pwork.get(), 0, sizeof(unsigned long long) * ntot, s));
    PB_LAUNCH(part_stats_kernel<kWing>, grid_for(N), 256, 0, s, G, cls, (const uint32_t*)key2.get(), N, true, pcnt.get(),
              pwork.get());
    std::vector<unsigned> hcnt(ntot);
    std::vector<unsigned long long> hwork(ntot);
    PB_CUDA_TRY(cudaMemcpyAsync(hcnt.data(), pcnt.get(), sizeof(unsigned) * ntot, cudaMemcpyDeviceToHost, s));
    PB_CUDA_TRY(cudaMemcpyAsync(hwork.data(), pwork.get(), sizeof(unsigned long long) * ntot, cudaMemcpyDeviceToHost, s));
    PB_CUDA_TRY(cudaStreamSynchronize(s));
    PB_LAUNCH(peel_init_kernel, grid_for(N), 256, 0, s, (const int64_t*)snap.get(), N, out, cnt.get(), state.get());
    std::vector<Work> fws;
    std::vector<Ctl> fcs;
    std::vector<double> fw;
    std::vector<int> graph_of;
    int64_t b = 0;
    for (int i = 0; i < ninst; ++i) {
      for (uint32_t p = 0; p + pb0[i] < pb0[i + 1]; ++p) {
        const int64_t n = hcnt[pb0[i] + p];
        if (n == 0) continue;
        Work x = ws[i];
        x.D = out;
        x.part_out = nullptr;
        x.items = items;
        x.part = part.get();
        x.my_part = p;
        x.alist[0] = alist0.get() + b;
        x.alist[1] = alist1.get() + b;
        x.near = nearl.get() + b;
        x.front[0] = fr0.get() + b;
        x.front[1] = fr1.get() + b;
        x.N = n;
        x.item0 = (uint32_t)b;
        fws.push_back(x);
        Ctl c = hctl;
        c.alive = (unsigned)n;
        c.alen[0] = (unsigned)n;
        c.alive_at_compact = (unsigned)n;
        fcs.push_back(c);
        fw.push_back(std::max(1.0, (double)hwork[pb0[i] + p]));
        graph_of.push_back(i);
        b += n;
      }
    }
    PB_REQUIRE(b == N, PB_ECUDA, "two-phase peel: partition sizes do not add up");
    std::vector<Ctl> fine;
    const int64_t coarse_work = res.work;
    res.work = 0;
    launch_instances(fws, fcs, fw, nullptr, heavy_lists, &fine);
    std::vector<int64_t> per_graph(ninst, 0);
    for (size_t q = 0; q < fine.size(); ++q) per_graph[graph_of[q]] += (int64_t)fine[q].rounds;
    res.rounds = *std::max_element(per_graph.begin(), per_graph.end());  // the longest graph, as above
    res.work += coarse_work;
    res.parts = (int64_t)fws.size();
    return res;
  }

  if (two_phase) {
    // Coarse pass: partitions of equal estimated work, about parts_per_cta per CTA (or
    // parts_total in all).
    DevBuf<unsigned long long> wtot(1, s);
    DevBuf<unsigned> ctot(1, s);
    PB_CUDA_TRY(cudaMemsetAsync(wtot.get(), 0, sizeof(unsigned long long), s));
    PB_CUDA_TRY(cudaMemsetAsync(ctot.get(), 0, sizeof(unsigned), s));
    PB_LAUNCH(part_stats_kernel<kWing>, grid_for(N), 256, 0, s, G, cls, (const uint32_t*)nullptr, N, false, ctot.get(),
              wtot.get());
    unsigned long long total_w = 0;
    readback(&total_w, wtot.get(), sizeof(total_w), s);
    const double nparts_target = std::max(1.0, parts_total > 0 ? (double)parts_total : parts_per_cta * grid);
    hctl.range_mode = 1;
    hctl.part_target = std::max<unsigned long long>(1, (unsigned long long)((double)total_w / nparts_target));
  }

  // Single instance over the whole grid: launch, and between launches compact the lists to
  // their live entries (every version is kept for the fine pass of a two-phase peel).
  std::vector<Lists> levels{G0};
  std::vector<unsigned> level_from{0};  // version j holds every item of partitions >= level_from[j]
  DevBuf<Work> dW(1, s);
  DevBuf<Ctl> ctl(1, s);
  if (capturing()) {
    // The graph copies from host memory that outlives it; the status words come back to a
    // pinned buffer the caller checks after every replay.
    Ctl* h0 = (Ctl*)g_recorder->pinned_alloc(sizeof(Ctl));
    std::memcpy(h0, &hctl, sizeof(Ctl));
    Work* w0 = (Work*)g_recorder->pinned_alloc(sizeof(Work));
    std::memcpy(w0, &W, sizeof(Work));
    PB_CUDA_TRY(cudaMemcpyAsync(ctl.get(), h0, sizeof(Ctl), cudaMemcpyHostToDevice, s));
    PB_CUDA_TRY(cudaMemcpyAsync(dW.get(), w0, sizeof(Work), cudaMemcpyHostToDevice, s));
  } else {
    PB_CUDA_TRY(cudaMemcpyAsync(ctl.get(), &hctl, sizeof(Ctl), cudaMemcpyHostToDevice, s));
    PB_CUDA_TRY(cudaMemcpyAsync(dW.get(), &W, sizeof(Work), cudaMemcpyHostToDevice, s));
  }
  Instances I1{dW.get(), nullptr, nullptr, nullptr, nullptr, 1u};
  Ctl* ctl_ptr = ctl.get();
  const Lists* no_levels = nullptr;
  int launches = 0;
  if (capturing()) {
    void* args[] = {&G, &no_levels, &I1, &ctl_ptr, &cls};
    PB_CUDA_TRY(cudaLaunchCooperativeKernel((const void*)kern, dim3(grid), dim3(kPT), args, smem, s));
    if (g_launch_counter) ++*g_launch_counter;
    // {err, alive} of the control block into the recorder's status slot (pinned).
    PB_LAUNCH(ctl_status_kernel, 1, 32, 0, s, ctl_ptr, 1u, status.get());
    PB_CUDA_TRY(cudaMemcpyAsync(g_recorder->status, status.get(), 2 * sizeof(unsigned), cudaMemcpyDeviceToHost, s));
    return res;
  }
  while (true) {
    void* args[] = {&G, &no_levels, &I1, &ctl_ptr, &cls};
    PB_CUDA_TRY(cudaLaunchCooperativeKernel((const void*)kern, dim3(grid), dim3(kPT), args, smem, s));
    if (g_launch_counter) ++*g_launch_counter;
    ++launches;
    PB_CUDA_TRY(cudaMemcpyAsync(&hctl, ctl.get(), sizeof(Ctl), cudaMemcpyDeviceToHost, s));
    PB_CUDA_TRY(cudaStreamSynchronize(s));
    PB_REQUIRE(!(hctl.err & ERR_TIMEOUT), PB_ETIMEOUT, "peeling: a grid barrier wait ran out of time");
    PB_REQUIRE(hctl.err == 0, PB_ECUDA, "peeling: a table invariant was violated");
    if (hctl.alive == 0) break;
    PB_REQUIRE(launches < 4096, PB_ECUDA, "peeling: too many relaunches");
    // Compact the lists to their live entries and resume.
    if (kWing) {
      compact_side<true>(liveK, G.offK, G.edgK, G.eidK, state.get(), true, s);
      compact_side<true>(liveC, G.offC, G.edgC, G.eidC, state.get(), true, s);
      G.offK = liveK.ver.back()->off.get();
      G.edgK = liveK.ver.back()->nbr.get();
      G.eidK = liveK.ver.back()->eid.get();
      G.offC = liveC.ver.back()->off.get();
      G.edgC = liveC.ver.back()->nbr.get();
      G.eidC = liveC.ver.back()->eid.get();
    } else {
      compact_side<false>(liveC, G.offC, G.edgC, nullptr, state.get(), false, s);
      G.offC = liveC.ver.back()->off.get();
      G.edgC = liveC.ver.back()->nbr.get();
    }
    refresh_work(G);
    if (two_phase) {
      // Partitions not opened yet (npart and later) have all their items in the new version.
      levels.push_back(G);
      level_from.push_back(hctl.npart);
    }
    const unsigned alive = hctl.alive;
    PB_CUDA_TRY(cudaMemcpyAsync(&ctl.get()->alive_at_compact, &alive, sizeof(unsigned), cudaMemcpyHostToDevice, s));
  }
  res.rounds = (int64_t)hctl.rounds;
  res.work = (int64_t)hctl.work;
  if (trace) {
    fprintf(stderr,
            "[pb] peel %s%s: rounds %llu launches %d advances %llu | ms advance %.1f F %.1f P %.1f | "
            "near scanned %llu items small %llu big %llu huge %llu work %llu\n",
            kWing ? "wing" : "tip", two_phase ? " (coarse pass)" : "", hctl.rounds, launches, hctl.advances,
            hctl.phase_ns[0] / 1e6, hctl.phase_ns[1] / 1e6, hctl.phase_ns[2] / 1e6, hctl.scanned, hctl.n_small,
            hctl.n_big, hctl.n_huge, hctl.work);
    if (kWing)
      fprintf(stderr,
              "[pb]   wing items / probes: warp %llu / %llu, CTA table %llu / %llu, dense markers %llu / %llu, "
              "reverse-direction probes %llu\n",
              hctl.mode_items[0], hctl.mode_work[0], hctl.mode_items[1], hctl.mode_work[1], hctl.mode_items[2],
              hctl.mode_work[2], hctl.rev_work);
    for (int b = 0; b < 42; ++b)
      if (hctl.pbin_rounds[b])
        fprintf(stderr, "[pb]   P rounds with est work in [2^%d, 2^%d): %llu rounds, %.1f ms, est %.3g (%.3g/s)\n",
                b ? b - 1 : 0, b, hctl.pbin_rounds[b], hctl.pbin_ns[b] / 1e6, (double)hctl.pbin_est[b],
                hctl.pbin_ns[b] ? hctl.pbin_est[b] / (hctl.pbin_ns[b] / 1e9) : 0.0);
  }
  if (!two_phase) return res;

  // ---- fine pass: one instance per partition, all in one launch ----------------------------
  release_coarse();
  res.coarse_rounds = res.rounds;
  const unsigned nparts = hctl.npart;
  PB_REQUIRE(nparts >= 1, PB_ECUDA, "two-phase peel: the coarse pass opened no partition");
  // Items sorted by partition (stable: ascending ids inside a partition).
  int bits = 1;
  while (bits < 32 && (1ull << bits) < nparts) ++bits;
  DevBuf<uint32_t> pkeys(N, s), pkeys2(N, s), perm(N, s), perm2(N, s);
  PB_CUDA_TRY(cudaMemcpyAsync(pkeys.get(), part.get(), sizeof(uint32_t) * N, cudaMemcpyDeviceToDevice, s));
  PB_LAUNCH(iota_kernel, grid_for(N), 256, 0, s, perm.get(), N);
  const bool alt = radix_sort_pairs_u32(pkeys.get(), perm.get(), pkeys2.get(), perm2.get(), N, 0, bits, s);
  const uint32_t* items = alt ? perm2.get() : perm.get();
  DevBuf<unsigned> pcnt(nparts, s);
  DevBuf<unsigned long long> pwork(nparts, s);
  PB_CUDA_TRY(cudaMemsetAsync(pcnt.get(), 0, sizeof(unsigned) * nparts, s));
  PB_CUDA_TRY(cudaMemsetAsync(pwork.get(), 0, sizeof(unsigned long long) * nparts, s));
  PB_LAUNCH(part_stats_kernel<kWing>, grid_for(N), 256, 0, s, G0, cls, (const uint32_t*)part.get(), N, true, pcnt.get(),
            pwork.get());
  std::vector<unsigned> hcnt(nparts);
  std::vector<unsigned long long> hwork(nparts);
  PB_CUDA_TRY(cudaMemcpyAsync(hcnt.data(), pcnt.get(), sizeof(unsigned) * nparts, cudaMemcpyDeviceToHost, s));
  PB_CUDA_TRY(cudaMemcpyAsync(hwork.data(), pwork.get(), sizeof(unsigned long long) * nparts, cudaMemcpyDeviceToHost, s));
  PB_CUDA_TRY(cudaStreamSynchronize(s));
  // Fresh per-item state: every partition starts from the counts its items had when it opened.
  PB_LAUNCH(peel_init_kernel, grid_for(N), 256, 0, s, (const int64_t*)snap.get(), N, out, cnt.get(), state.get());
  DevBuf<Lists> dlevels(levels.size(), s);
  PB_CUDA_TRY(cudaMemcpyAsync(dlevels.get(), levels.data(), sizeof(Lists) * levels.size(), cudaMemcpyHostToDevice, s));
  Ctl c0;
  std::memset(&c0, 0, sizeof(c0));
  c0.nm[0] = c0.nm[1] = kInf;
  c0.k_lo = kInf;
  c0.min_gain = 0xFFFFFFFFu;
  c0.barrier_timeout_ns = hctl.barrier_timeout_ns;
  c0.near_min = hctl.near_min;
  c0.near_div = hctl.near_div;
  std::vector<Work> ws;
  std::vector<Ctl> cs;
  std::vector<double> weights;
  int64_t b = 0;
  for (unsigned p = 0; p < nparts; ++p) {
    const int64_t n = hcnt[p];
    if (n == 0) continue;
    Work x = W;
    x.D = out;
    x.part_out = nullptr;
    x.items = items;
    x.part = part.get();
    x.my_part = p;
    unsigned lv = 0;
    for (unsigned j = 0; j < level_from.size(); ++j)
      if (level_from[j] <= p) lv = j;
    x.level = lv;
    x.alist[0] = alist0.get() + b;
    x.alist[1] = alist1.get() + b;
    x.near = nearl.get() + b;
    x.front[0] = fr0.get() + b;
    x.front[1] = fr1.get() + b;
    x.N = n;
    x.item0 = (uint32_t)b;
    ws.push_back(x);
    Ctl c = c0;
    c.alive = (unsigned)n;
    c.alen[0] = (unsigned)n;
    c.alive_at_compact = (unsigned)n;
    cs.push_back(c);
    weights.push_back(std::max(1.0, (double)hwork[p]));
    b += n;
  }
  PB_REQUIRE(b == N, PB_ECUDA, "two-phase peel: partition sizes do not add up");
  const int64_t coarse_work = res.work;
  res.rounds = 0;
  res.work = 0;
  launch_instances(ws, cs, weights, dlevels.get(), heavy_lists, nullptr, true);
  res.work += coarse_work;
  res.parts = (int64_t)ws.size();
  if (trace)
    fprintf(stderr, "[pb] peel %s fine pass: %zu partitions, %d list versions, %lld rounds, longest %lld\n",
            kWing ? "wing" : "tip", ws.size(), (int)levels.size(), (long long)res.rounds,
            (long long)res.fine_rounds_max);
  return res;
}

}  // namespace

PeelResult peel_vertices(const pb_graph& g, int use_v, const int64_t* counts_dev, int64_t* tip_dev, cudaStream_t s,
                         const PeelTuning& tune, const PeelParts* parts) {
  return run_peel<false>(g, use_v, counts_dev, tip_dev, s, tune, parts);
}

PeelResult peel_edges(const pb_graph& g, int use_v, const int64_t* ecounts_dev, int64_t* wing_dev, cudaStream_t s,
                      const PeelTuning& tune) {
  return run_peel<true>(g, use_v, ecounts_dev, wing_dev, s, tune, nullptr);
}

}  // namespace pb
