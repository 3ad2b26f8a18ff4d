// Wedge aggregation and butterfly accumulation on the ranked CSR.
//
// Semantics (CountWorkEfficientParallel, butterfly_count.h:1218-1320; the per-edge and total
// variants butterfly_ecount.h:1334-1429 and butterfly_count_total.h:662-749): for every
// endpoint i, the wedges are (i, v, u2) with v in N(i), u2 in N(v), u2 < min(i, v); w(u2) is
// the number of wedges of i that end in u2.  Then
//   VERT : tagged endpoints i and u2 gain C(w,2); tagged centres v gain w-1 per wedge;
//   EDGE : edges (i,v) and (v,u2) gain w-1 per wedge;
//   TOTAL: the sum of C(w,2).
// Endpoint and centre are on opposite sides, so for one endpoint either the centre credits or
// the endpoint credits matter, never both.
//
// Aggregators (the multiplicity table w), by the wedges W_i of the endpoint:
//   warp : W_i <= small_w and a short row; one warp, an open-addressing table in shared memory.
//   mid  : W_i <= mid_w and a row and a table that suit a CTA of 128 threads; many such CTAs share an SM, since
//          an endpoint of this size is a chain of a few round trips, not a throughput problem.
//   block: larger endpoints, one CTA of 512 threads per endpoint taken from a global work counter.
// The CTA kernels choose among dense counters over [0, i) (BATCHS-style; 16 bits wide when the
// degree allows), a hash table, dense counters for the low ranks with a hash table for the rest,
// and a per-CTA dense array in global scratch memory when none of them holds the endpoint.
// Hash entries are one 32-bit word (key and count) whenever the count fits beside the key, so an
// insertion is one shared-memory atomic.
// The wedge list of an endpoint is cut into pieces of neighbour lists, each walked by a warp, so
// consecutive lanes read consecutive entries of N(v) (coalesced).
// Per-edge credits are gathered per slot of the ranked CSR, where the wedges of a piece lie next to
// each other (one 128-byte atomic request per 32 wedges instead of 32 scattered ones), and moved to
// output edge order once at the end.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <vector>

#include "pb_engine.cuh"
#include "pb_mlp.cuh"
#include "pb_prims.cuh"
#include "pb_walk.cuh"

namespace pb {

namespace {

constexpr uint32_t kEmpty = 0xFFFFFFFFu;
constexpr int kWarpTable = 1024;  // slots per warp
constexpr int kWarpsPerBlockSmall = 8;
constexpr int64_t kListRange = int64_t(1) << 26;  // endpoints that the item lists hold at a time
constexpr size_t kAskBytes = size_t(256) << 20;  // per-slot counts above this ask what is left of the device
constexpr uint32_t kHotRanks = 256;   // count_warp_kernel: vertex counts gathered per CTA
// A row is walked by the threads that own its endpoint, however few wedges it has, so long rows move
// up a class: beyond kWarpRow slots to a CTA of 128 threads, beyond kMidRow to one of 512.  Limits of
// (1024, 16384) left the 128-thread class of 2^18 R-MAT edges waiting for its longest rows: aggregation
// 0.43 ms, (512, 1024) 0.34, (128, 512) 0.32, (256, 1024) 0.30; 2^24 edges take 18.7 ms with each.
constexpr uint32_t kWarpRow = 256;
constexpr uint32_t kMidRow = 1024;

enum Per { VERT = 0, EDGE = 1, TOTAL = 2 };

struct Params {
  const uint32_t* __restrict__ off;
  const uint32_t* __restrict__ adj;
  const uint32_t* __restrict__ pref;
  const int64_t* __restrict__ wsum;
  int64_t n;
  int per;
  int64_t* out;
  int64_t out_len;  // entries of out
  int64_t m2;       // slots of the ranked CSR
  uint32_t* err;    // record of the first bounds violation {code, index lo, index hi, aux}
  uint32_t* sacc32;             // per-edge counts per slot: 32 bits wide when every count fits,
  unsigned long long* sacc64;   // else 64; both null: credits go to out at once, through eout
  const uint32_t* __restrict__ eout;
  unsigned long long* mstats;  // per mode (dense, hash, global, hybrid): endpoints, wedges
  // Block aggregator (null for the mid kernel):
  const uint8_t* modes;        // modes[q]: aggregation mode of item q
  uint8_t* mode_out;           // mode_out[q]: mode item q ran with (scheduler hooks)
  unsigned long long* cycles;  // cycles[q]: SM cycles item q took (clock64, thread 0)
};

// Records the first bounds violation.
__device__ __noinline__ void record_violation(uint32_t* err, uint32_t code, uint64_t idx, uint32_t aux) {
  if (atomicCAS(&err[0], 0u, code) == 0u) {
    err[1] = (uint32_t)idx;
    err[2] = (uint32_t)(idx >> 32);
    err[3] = aux;
  }
}

// out[idx] += v.  Indices derived from memory are bounds-checked; a violation is recorded
// (and reported as an error by the host) instead of being accessed.
__device__ __forceinline__ void credit(const Params& P, uint64_t idx, int64_t v, uint32_t code) {
  if (idx >= (uint64_t)P.out_len) { record_violation(P.err, code, idx, 0); return; }
  atomic_add_i64(&P.out[idx], v);
}

__device__ __forceinline__ bool slot_ok(const Params& P, uint64_t slot, uint32_t code) {
  if (slot >= (uint64_t)P.m2) { record_violation(P.err, code, slot, 0); return false; }
  return true;
}

// Per-edge credit of a slot (checked by the caller).
__device__ __forceinline__ void credit_slot(const Params& P, uint32_t slot, uint32_t v) {
  if (P.sacc32) atomicAdd(&P.sacc32[slot], v);
  else if (P.sacc64) atomicAdd(&P.sacc64[slot], (unsigned long long)v);
  else credit(P, P.eout[slot], v, 12);
}

// Fibonacci hashing: the high bits of key * 2^32/phi, folded into the table size (any size).
__device__ __forceinline__ uint32_t hash_slot(uint32_t key, uint32_t size) { return __umulhi(key * 0x9E3779B1u, size); }

// Tables.  kOne: one word per slot, key << cb | count (cb count bits; the caller guarantees counts
// of at most 2^cb - 2, so no entry equals kEmpty).  Otherwise keys and counts in two arrays of
// `size` words (cb is 0).  Insert-or-increment; tables hold at most 3/4 of their slots, so a probe
// sequence never exceeds the table size; the bound turns a broken invariant into a recorded error
// instead of an endless loop.
template <bool kOne>
__device__ __forceinline__ bool table_insert(uint32_t* tab, uint32_t size, int cb, uint32_t key) {
  uint32_t h = hash_slot(key, size);
  for (uint32_t probes = 0; probes < size; ++probes) {
    uint32_t k = tab[h];
    if (k == kEmpty) {
      k = atomicCAS(&tab[h], kEmpty, kOne ? (key << cb) | 1u : key);
      if (k == kEmpty) {
        if (!kOne) atomicAdd(&tab[size + h], 1u);
        return true;
      }
    }
    if ((kOne ? k >> cb : k) == key) {
      atomicAdd(&tab[kOne ? h : size + h], 1u);
      return true;
    }
    h = h + 1 == size ? 0u : h + 1;
  }
  return false;
}

template <bool kOne>
__device__ __forceinline__ uint32_t table_find(const uint32_t* tab, uint32_t size, int cb, uint32_t key) {
  uint32_t h = hash_slot(key, size);
  for (uint32_t probes = 0; probes < size; ++probes) {
    const uint32_t k = tab[h];
    if ((kOne ? k >> cb : k) == key) return kOne ? k & ((1u << cb) - 1u) : tab[size + h];
    if (k == kEmpty) return 0;  // unreachable for keys that were inserted
    h = h + 1 == size ? 0u : h + 1;
  }
  return 0;
}

// Entry of slot s: its key and count (count 0 when empty).
__device__ __forceinline__ uint32_t table_entry(const uint32_t* tab, uint32_t size, int cb, uint32_t s, uint32_t& key) {
  const uint32_t k = tab[s];
  key = k >> cb;
  return k == kEmpty ? 0u : (cb ? k & ((1u << cb) - 1u) : tab[size + s]);
}

// Endpoint lists: {endpoint, first slot, end slot, wedges (saturated)}.
__device__ __forceinline__ unsigned list_at(uint32_t* counter, bool have) {
  const unsigned bal = __ballot_sync(0xffffffffu, have);
  unsigned base = 0;
  if (bal && lane_id() == (unsigned)(__ffs(bal) - 1)) base = atomicAdd(counter, (uint32_t)__popc(bal));
  base = __shfl_sync(0xffffffffu, base, bal ? __ffs(bal) - 1 : 0);
  return base + __popc(bal & ((1u << lane_id()) - 1u));
}

// One slot of an endpoint's row, as a lane holds it: the wedges of the slot, the tagged neighbour
// and where the neighbour's row begins.
struct SlotRow {
  uint32_t L, vt, vs;
};

__device__ __forceinline__ SlotRow load_slot(uint32_t j, bool valid, const Params& P) {
  SlotRow r{0, kEmpty, 0};
  if (valid) {
    r.L = P.pref[j];
    r.vt = P.adj[j];
    if ((r.vt >> 1) < P.n) r.vs = P.off[r.vt >> 1];
    else { record_violation(P.err, 28, r.vt, j); r.L = 0; }
  }
  return r;
}

// Iterates every wedge of an endpoint (slots [b, e) of the ranked CSR) with one warp, 32 slots and
// then four steps of 32 wedges at a time (their loads are issued together).  `row` holds the first
// group's slots.  slots(): all lanes, once per group; f(lo, slot2, u2): lo = lane of the wedge's
// slot; group_end(j, vt): all lanes, with this lane's slot (vt = kEmpty beyond the end).
template <class Slots, class F, class End>
__device__ __forceinline__ void warp_wedges(uint32_t b, uint32_t e, SlotRow row, const Params& P, Slots&& slots, F&& f,
                                            End&& group_end) {
  const unsigned lane = lane_id();
  walk_groups(b, e - b, 32, lane, [&](uint32_t j, bool valid) {
    if (j != b + lane) row = load_slot(j, valid, P);
    slots();
    const uint32_t incl = warp_inclusive_scan(row.L);
    const uint32_t from = row.vs - (incl - row.L);  // slot2 = from + t
    const uint32_t T = __shfl_sync(0xffffffffu, incl, 31);
    for (uint32_t t0 = 0; t0 < T; t0 += 128) {
      uint32_t at[4], s2[4], x[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const uint32_t t = t0 + 32 * r + lane;
        uint32_t lo = 0;
#pragma unroll
        for (uint32_t step = 16; step > 0; step >>= 1) {
          const uint32_t y = __shfl_sync(0xffffffffu, incl, lo + step - 1);
          if (y <= t) lo += step;
        }
        at[r] = lo;
        s2[r] = __shfl_sync(0xffffffffu, from, lo) + t;
        x[r] = kEmpty;
        if (t < T && slot_ok(P, s2[r], 20)) x[r] = P.adj[s2[r]];
      }
#pragma unroll
      for (int r = 0; r < 4; ++r)
        if (x[r] != kEmpty) f(at[r], s2[r], x[r] >> 1);
    }
    __syncwarp();
    group_end(j, row.vt);
  });
}

// ---------------------------------------------------------------------------------------------
// Small endpoints: a warp each.  Bound by latency: an endpoint is a chain of round trips for a few
// dozen to 512 wedges, so what counts is the number of warps (48 per SM with one-word tables of
// 4 KiB; 24 with two-array tables) and that the next endpoint's list entry and first slots are
// loaded while this one is counted.
// The vertices of the lowest ranks share wedges with most endpoints: their counts are gathered per
// CTA (1e6 endpoints adding to one address took 5.2 ms on the power-law graph of 1e7 edges, the
// aggregation as a whole 12.2 ms; 6.5 ms with this).
// kOneWord false: two-array tables (more than 2^22 vertices leave no room for a count of 512).
template <bool kOneWord>
__global__ void __launch_bounds__(256, kOneWord ? 6 : 3) count_warp_kernel(Params P, const uint4* __restrict__ items,
                                                                         const uint32_t* __restrict__ n_items_dev,
                                                                         int count_bits) {
  extern __shared__ __align__(16) uint32_t smem_w[];
  const unsigned lane = lane_id();
  const int wib = threadIdx.x >> 5;
  const int cb = kOneWord ? count_bits : 0;
  uint32_t* hot = smem_w;  // low and high words of the lowest ranks' counts
  for (uint32_t s = threadIdx.x; s < 2 * kHotRanks; s += blockDim.x) hot[s] = 0;
  __syncthreads();
  uint32_t* tab = smem_w + 2 * kHotRanks + wib * ((kOneWord ? 1 : 2) * kWarpTable + 32);
  uint32_t* acc = tab + (kOneWord ? 1 : 2) * kWarpTable;  // credits of the group's 32 slots
  const uint32_t n_items = *n_items_dev;
  const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
  int64_t total = 0;
  uint32_t q = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  // Two list entries ahead, one row ahead.
  uint4 next = q < n_items ? items[q] : make_uint4(0, 0, 0, 0);
  uint4 after = q + nwarps < n_items ? items[q + nwarps] : make_uint4(0, 0, 0, 0);
  SlotRow next_row = load_slot(next.y + lane, lane < next.z - next.y, P);
  for (; q < n_items; q += nwarps) {
    const uint4 it = next;
    const SlotRow row = next_row;
    const uint32_t i = it.x, b = it.y, e = it.z;
    next = after;
    after = q + 2 * nwarps < n_items ? items[q + 2 * nwarps] : make_uint4(0, 0, 0, 0);
    // The next endpoint's first slots: issued here, their row starts (a dependent load) below.
    next_row = SlotRow{0, kEmpty, 0};
    if (lane < next.z - next.y) {
      next_row.L = P.pref[next.y + lane];
      next_row.vt = P.adj[next.y + lane];
    }
    const bool tag_i = !(__shfl_sync(0xffffffffu, row.vt, 0) & 1u);
    const bool need_center = P.per == EDGE || (P.per == VERT && !tag_i);
    const uint32_t tsize = max(64u, (2u * it.w + 3u) & ~3u);
    const uint32_t words = kOneWord ? tsize : 2 * tsize;
    for (uint32_t s = lane * 4; s < words; s += 128) {
      const uint32_t x = s < tsize ? kEmpty : 0u;
      *reinterpret_cast<uint4*>(tab + s) = make_uint4(x, x, x, x);
    }
    __syncwarp();
    warp_wedges(b, e, row, P, [] {}, [&](uint32_t, uint32_t, uint32_t u2) {
      if (!table_insert<kOneWord>(tab, tsize, cb, u2)) record_violation(P.err, 25, u2, i);
    }, [](uint32_t, uint32_t) {});
    __syncwarp();
    if (next_row.vt != kEmpty) {
      if ((next_row.vt >> 1) < P.n) next_row.vs = P.off[next_row.vt >> 1];
      else { record_violation(P.err, 28, next_row.vt, next.y + lane); next_row.L = 0; }
    }
    if (need_center) {
      warp_wedges(b, e, row, P,
                  [&] {
                    acc[lane] = 0;
                    __syncwarp();
                  },
                  [&](uint32_t lo, uint32_t slot2, uint32_t u2) {
                    const uint32_t w = table_find<kOneWord>(tab, tsize, cb, u2);
                    if (w > 1) {
                      if (P.per == EDGE) credit_slot(P, slot2, w - 1);
                      atomicAdd(&acc[lo], w - 1);
                    }
                  },
                  [&](uint32_t j, uint32_t vt) {
                    const uint32_t a = acc[lane];
                    if (a && vt != kEmpty) {
                      if (P.per == EDGE) credit_slot(P, j, a);
                      else credit(P, vt >> 1, a, 11);
                    }
                    __syncwarp();
                  });
    } else {
      int64_t mine = 0;
      for (uint32_t s = lane; s < tsize; s += 32) {
        uint32_t k;
        const int64_t w = table_entry(tab, tsize, cb, s, k);
        if (w < 2) continue;
        const int64_t bf = w * (w - 1) / 2;
        mine += bf;
        if (P.per == VERT) {
          if (k < kHotRanks) {
            const uint32_t old = atomicAdd(&hot[k], (uint32_t)bf);
            if (old + (uint32_t)bf < old) atomicAdd(&hot[kHotRanks + k], 1u);
          } else {
            credit(P, k, bf, 14);
          }
        }
      }
      if (P.per == VERT) {
        mine = warp_sum(mine);
        if (lane == 0 && mine) credit(P, i, mine, 15);
      } else {
        total += mine;
      }
    }
    __syncwarp();
  }
  if (P.per == TOTAL) {
    total = warp_sum(total);
    if (lane == 0 && total) atomic_add_i64(P.out, total);
  } else if (P.per == VERT) {
    __syncthreads();
    for (uint32_t s = threadIdx.x; s < kHotRanks; s += blockDim.x) {
      const int64_t v = ((int64_t)hot[kHotRanks + s] << 32) | hot[s];
      if (v) credit(P, s, v, 17);
    }
  }
}

// ---------------------------------------------------------------------------------------------
constexpr int kBlock = 512;    // threads of the block aggregator
constexpr int kBlockPerSm = 3; // with 72 KiB of shared memory each (pb_engine.cuh): aggregation of
                               // the R-MAT graph of 2^24 edges, per edge: 18.6 ms (18.0 with today's
                               // mid class); 512 threads x 2 per SM 22.0, 256 x 4 21.5, 256 x 6 21.7,
                               // 1024 x 1 27.2
constexpr int kMidBlock = 128; // threads of the mid aggregator

template <int NT>
struct BlockShared {
  uint32_t vs[NT];
  uint32_t vt[NT];
  uint32_t len[NT];
  uint16_t list[NT];
  int64_t red[32];
  uint32_t item, long_above;
  uint32_t n_short[2], n_long[2], turn;  // block_wedges: list counters of the chunks in turn
};
template <int NT>
constexpr size_t shared_fixed() { return (sizeof(BlockShared<NT>) + 15) & ~size_t(15); }

__device__ __forceinline__ int64_t block_sum_i64(int64_t x, int64_t* smem) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  x = warp_sum(x);
  __syncthreads();
  if (lane == 0) smem[warp] = x;
  __syncthreads();
  int64_t t = 0;
  if (warp == 0) {
    t = lane < nwarps ? smem[lane] : 0;
    t = warp_sum(t);
  }
  return t;  // valid in thread 0
}

// Iterates every wedge of an endpoint with the whole CTA, NT neighbours at a time.  Neighbours with
// prefixes N(v)[0, L) of up to S.long_above wedges go to the warps in turn, longer ones are walked by all
// warps together.  Lane t of a walk takes entries t, t + 32, ... with four loads in flight, so loads
// and atomics on the entries' slots are coalesced.  f(slot2, u2) per wedge; part_end(j, vt): all
// lanes of a warp, after its part of neighbour slot j.  Ends with a barrier, so a walk may follow
// another at once and read what its f wrote.
// A list that all warps walk costs each of them a turn however short its part is, so it must be long
// beside a warp's share of the chunk: above a quarter of it, and above kLong.
constexpr uint32_t kLong = 512;
template <int NT>
__device__ __forceinline__ uint32_t long_above(int64_t W, uint32_t deg) {
  if (NT == kMidBlock) return kLong;  // at most kMidWedges wedges
  const float chunk = (float)W * fminf(1.f, (float)NT / (float)deg);
  return max(kLong, (uint32_t)fminf(chunk / (float)(4 * (NT / 32)), 1e9f));
}

template <int kStride, class F>
__device__ __forceinline__ void walk_prefix(const uint32_t* __restrict__ adj, uint32_t beg, uint32_t len, uint32_t first,
                                            F&& f) {
  walk_turns<kStride>(beg, len, first, [&](uint32_t s0, int32_t left) {
    uint32_t x[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) x[r] = left > r * kStride ? __ldg(adj + (s0 + r * kStride)) : kEmpty;
#pragma unroll
    for (int r = 0; r < 4; ++r)
      if (x[r] != kEmpty) f(s0 + r * kStride, x[r] >> 1);
  });
}

template <int NT, class F, class End>
__device__ __forceinline__ void block_wedges(uint32_t b, uint32_t e, const Params& P, BlockShared<NT>& S, F&& f,
                                             End&& part_end) {
  const uint32_t tid = threadIdx.x, lane = tid & 31u;
  walk_groups(b, e - b, NT, tid, [&](uint32_t j, bool valid) {
    const uint32_t j0 = j - tid;
    uint32_t L = 0, vt = 0, vs = 0;
    if (valid) {
      L = P.pref[j];
      vt = P.adj[j];
      if ((vt >> 1) < P.n) vs = P.off[vt >> 1];
      else { record_violation(P.err, 29, vt, j); L = 0; }
      if (L && !slot_ok(P, (uint64_t)vs + L - 1, 21)) L = 0;
    }
    S.vs[tid] = vs;
    S.vt[tid] = vt;
    S.len[tid] = L;
    // Neighbours without wedges are left out: slots k of the chunk, in any order.
    const uint32_t limit = S.long_above, turn = S.turn;
    const unsigned some = __ballot_sync(0xffffffffu, L > 0 && L <= limit);
    unsigned at = 0;
    if (lane == 0 && some) at = atomicAdd(&S.n_short[turn], (uint32_t)__popc(some));
    at = __shfl_sync(0xffffffffu, at, 0) + __popc(some & ((1u << lane) - 1u));
    if (L > 0 && L <= limit) S.list[at] = (uint16_t)tid;
    if (L > limit) S.list[NT - 1 - atomicAdd(&S.n_long[turn], 1u)] = (uint16_t)tid;
    __syncthreads();
    const uint32_t ns = S.n_short[turn], nl = S.n_long[turn];
    // Every thread has taken its turn by now, and the next chunk (of this walk or of the caller's next
    // one) adds to the other counters only behind the barrier below, so they are cleared in between.
    if (tid == 0) {
      S.turn = turn ^ 1u;
      S.n_short[turn ^ 1u] = S.n_long[turn ^ 1u] = 0;
    }
    for (uint32_t p = tid >> 5; p < ns; p += NT / 32) {
      const uint32_t k = S.list[p], beg = S.vs[k];
      walk_prefix<32>(P.adj, beg, S.len[k], lane, f);
      __syncwarp();
      part_end(j0 + k, S.vt[k]);
    }
    for (uint32_t p = 0; p < nl; ++p) {
      const uint32_t k = S.list[NT - 1 - p], beg = S.vs[k];
      walk_prefix<NT>(P.adj, beg, S.len[k], tid, f);
      __syncwarp();
      part_end(j0 + k, S.vt[k]);
    }
    __syncthreads();
  });
}

// The mid aggregator: CTAs of 128 threads with a table of about 19.5 KiB, ten to an SM.  An SM has
// 228 KiB, of which every resident CTA takes one for the system: with 22 KiB each, nine fit and the
// tenth of the grid starts when the others are through (aggregation of the R-MAT graph with 2^24 edges
// per edge 18.46 ms; a grid of nine per SM 18.43, ten of 21.5 KiB 18.15).
constexpr int kMidSmem = 43 << 9;
constexpr int kMidPerSm = 10;
constexpr int kSmBytes = 228 << 10, kCtaReserved = 1 << 10;
static_assert(kMidPerSm * (kMidSmem + kCtaReserved) <= kSmBytes, "the mid CTAs of an SM must be resident together");
static_assert(kBlockPerSm * (CountConfig{}.smem_bytes + kCtaReserved) <= kSmBytes,
              "the block CTAs of an SM must be resident together");
constexpr int64_t kMidWedges = 2047;

enum Mode : uint32_t { MODE_DENSE = 0, MODE_HASH = 1, MODE_GLOBAL = 2, MODE_HYBRID = 3 };
// Items with fewer wedges are left to the plain rule when the learned scheduler runs.
constexpr int64_t kSchedMinWedges = 2048;

// What a CTA's table area of tw words can hold.  Counts of an endpoint are at most its degree.
struct Geom {
  uint32_t tw;      // words of the table area
  uint32_t hy_words;  // hybrid: words of the dense counters (16 bits each); the hash takes the rest
  int cb;           // count bits of a one-word hash entry

  __device__ __forceinline__ int bits(uint32_t deg) const { return deg < (1u << cb) - 1u ? cb : 0; }
  __device__ __forceinline__ bool wide(uint32_t deg) const { return deg > 0xFFFFu; }
  __device__ __forceinline__ bool dense_ok(uint32_t i, uint32_t deg) const { return i <= (wide(deg) ? tw : 2 * tw); }
  __device__ __forceinline__ bool hash_ok(uint64_t W, uint32_t deg) const { return W * (bits(deg) ? 2 : 4) <= tw; }
  __device__ __forceinline__ uint32_t hy_dense() const { return 2 * hy_words; }
  __device__ __forceinline__ uint32_t hy_slots(uint32_t deg) const { return (tw - hy_words) / (bits(deg) ? 1 : 2); }
  __device__ __forceinline__ bool hybrid_ok(uint64_t hi, uint32_t deg) const {
    return !wide(deg) && 4 * hi <= 3ull * hy_slots(deg);
  }
  // The plain rule.  Dense counters when clearing and scanning them costs less than the wedges do;
  // else a hash table; dense counters again; low ranks dense and the rest hashed; global scratch.
  __device__ __forceinline__ Mode rule(uint32_t i, uint64_t W, uint32_t deg, uint64_t hi) const {
    if (dense_ok(i, deg) && (uint64_t)i <= 4 * W) return MODE_DENSE;
    if (hash_ok(W, deg)) return MODE_HASH;
    if (dense_ok(i, deg)) return MODE_DENSE;
    return hybrid_ok(hi, deg) ? MODE_HYBRID : MODE_GLOBAL;
  }
};

// Wedges of an endpoint that end at or above rank d, counted by one warp (valid in lane 0): per
// neighbour, the prefix length minus the entries below d (one binary search each).
__device__ __forceinline__ uint64_t warp_high_wedges(const Params& P, const uint4& it, int64_t W, uint32_t d) {
  unsigned long long lo_w = 0;
  for (uint32_t t = lane_id(); t < it.z - it.y; t += 32) {
    const uint32_t j = it.y + t, v = P.adj[j] >> 1;
    if (v >= P.n) continue;
    const uint32_t vb = P.off[v];
    lo_w += min(lower_bound_u32(P.adj, vb, P.off[v + 1], d << 1) - vb, P.pref[j]);
  }
  return (uint64_t)(W - (int64_t)warp_sum(lo_w));
}

// The plain rule's mode of every block-aggregator item (one warp each); *n_global counts those
// that need global scratch.
__global__ void plain_modes_kernel(Params P, const uint4* __restrict__ items, const uint32_t* __restrict__ n_items_dev,
                                   Geom G, uint8_t* modes, uint32_t* n_global) {
  const uint32_t n_items = *n_items_dev;
  const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t q = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; q < n_items; q += nwarps) {
    const uint4 it = items[q];
    const int64_t W = P.wsum[it.x + 1] - P.wsum[it.x];
    const uint32_t deg = it.z - it.y;
    uint64_t hi = 0;
    if (!G.dense_ok(it.x, deg) && !G.hash_ok(W, deg)) hi = warp_high_wedges(P, it, W, G.hy_dense());
    if (lane_id() == 0) {
      const Mode m = G.rule(it.x, W, deg, hi);
      modes[q] = (uint8_t)m;
      if (m == MODE_GLOBAL) atomicAdd(n_global, 1u);
    }
  }
}

// One CTA of NT threads per endpoint.  Bound by its instructions and barriers: on the R-MAT graph with 2^24
// edges (12.4 ms with 512 threads, 3.6 with 128) the schedulers issue in 69% (62%) of the cycles while
// the shared-memory pipe is busy for 45%, L2 for 12% and DRAM for 4%; the largest stalls are the
// barriers between chunks.  The two table walks read 4 bytes a wedge each, mostly from L2.
template <int NT, int kMinBlocks>
__global__ void __launch_bounds__(NT, kMinBlocks) count_block_kernel(Params P, const uint4* __restrict__ items,
                                                                     const uint32_t* __restrict__ n_items_dev,
                                                                     uint32_t* cursor, uint32_t* gscratch, Geom G) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  BlockShared<NT>& S = *reinterpret_cast<BlockShared<NT>*>(smem_raw);
  uint32_t* table = reinterpret_cast<uint32_t*>(smem_raw + shared_fixed<NT>());
  uint32_t* gcnt = gscratch ? gscratch + (size_t)blockIdx.x * (size_t)P.n : nullptr;
  const uint32_t n_items = *n_items_dev;
  const unsigned lane = lane_id();
  int64_t total = 0;
  if (threadIdx.x == 0) S.turn = S.n_short[0] = S.n_long[0] = 0;
  // The first item of a CTA is its own number; the cursor hands out the later ones.
  for (uint32_t q = blockIdx.x; q < n_items;) {
    if (threadIdx.x == 0) S.item = gridDim.x + atomicAdd(cursor, 1u);
    const long long t_item = clock64();
    const uint4 it = items[q];
    const uint32_t i = it.x, b = it.y, e = it.z, deg = e - b;
    const int64_t W = NT == kMidBlock ? (int64_t)it.w : P.wsum[i + 1] - P.wsum[i];
    const bool tag_i = !(P.adj[b] & 1u);
    const bool need_center = P.per == EDGE || (P.per == VERT && !tag_i);
    Mode mode;
    if (NT == kMidBlock) mode = G.rule(i, W, deg, 0);
    else mode = (Mode)(P.modes[q] & 3u);
    if (threadIdx.x == 0) S.long_above = long_above<NT>(W, deg);
    if (threadIdx.x == 0 && P.mstats) {
      atomicAdd(&P.mstats[mode], 1ull);
      atomicAdd(&P.mstats[4 + mode], (unsigned long long)W);
    }
    const bool wide = G.wide(deg);
    const int cb = G.bits(deg);
    // Dense counters (dense, hybrid): u2 below dlim; hash table (hash, hybrid) of tsize slots.
    const uint32_t dlim = mode == MODE_DENSE ? i : (mode == MODE_HYBRID ? G.hy_dense() : 0u);
    uint32_t* tab = mode == MODE_HYBRID ? table + G.hy_words : table;
    const uint32_t tsize = mode == MODE_HASH ? max(64u, 2u * (uint32_t)W) : (mode == MODE_HYBRID ? G.hy_slots(deg) : 0u);
    const uint32_t dwords = mode == MODE_HYBRID ? G.hy_words : (wide ? dlim : (dlim + 1) / 2);
    for (uint32_t s = threadIdx.x; s < dwords; s += NT) table[s] = 0;
    for (uint32_t s = threadIdx.x; s < tsize; s += NT) {
      tab[s] = kEmpty;
      if (!cb) tab[tsize + s] = 0;
    }
    __syncthreads();
    // Phase 1: multiplicities.  The two common modes have loops of their own.
    const auto nothing = [](uint32_t, uint32_t) {};
    if (mode == MODE_DENSE && !wide) {
      block_wedges<NT>(b, e, P, S, [&](uint32_t, uint32_t u2) {
        if (u2 < dlim) atomicAdd(&table[u2 >> 1], 1u << (16 * (u2 & 1u)));
        else record_violation(P.err, 22, u2, i);
      }, nothing);
    } else if (mode == MODE_HASH && cb) {
      block_wedges<NT>(b, e, P, S, [&](uint32_t, uint32_t u2) {
        if (!table_insert<true>(tab, tsize, cb, u2)) record_violation(P.err, 26, u2, i);
      }, nothing);
    } else {
      block_wedges<NT>(b, e, P, S, [&](uint32_t, uint32_t u2) {
        if (u2 < dlim) {
          if (wide) atomicAdd(&table[u2], 1u);
          else atomicAdd(&table[u2 >> 1], 1u << (16 * (u2 & 1u)));
        } else if (tsize) {
          if (!(cb ? table_insert<true>(tab, tsize, cb, u2) : table_insert<false>(tab, tsize, 0, u2)))
            record_violation(P.err, 35, u2, i);
        } else if (mode == MODE_GLOBAL && u2 < P.n) {
          atomicAdd(&gcnt[u2], 1u);
        } else {
          record_violation(P.err, 23, u2, i);
        }
      }, nothing);
    }
    if (need_center) {
      // Phase 2: centre / edge credits.  A part's sum fits 32 bits: the w(i, u2) of distinct u2 add
      // up to at most the edges of the graph, fewer than 2^31 (lists are strictly ascending).
      uint32_t mine = 0;
      auto charge = [&](uint32_t slot2, uint32_t w) {
        if (w > 1) {
          if (P.per == EDGE) credit_slot(P, slot2, w - 1);
          mine += w - 1;
        }
      };
      auto part_end = [&](uint32_t j, uint32_t vt) {
        const uint32_t s = __reduce_add_sync(0xffffffffu, mine);
        mine = 0;
        if (lane == 0 && s) {
          if (P.per == EDGE) credit_slot(P, j, s);
          else credit(P, vt >> 1, s, 11);
        }
      };
      if (mode == MODE_DENSE && !wide) {
        block_wedges<NT>(b, e, P, S, [&](uint32_t slot2, uint32_t u2) {
          if (u2 < dlim) charge(slot2, (table[u2 >> 1] >> (16 * (u2 & 1u))) & 0xFFFFu);
        }, part_end);
      } else if (mode == MODE_HASH && cb) {
        block_wedges<NT>(b, e, P, S, [&](uint32_t slot2, uint32_t u2) {
          charge(slot2, table_find<true>(tab, tsize, cb, u2));
        }, part_end);
      } else {
        block_wedges<NT>(b, e, P, S, [&](uint32_t slot2, uint32_t u2) {
          uint32_t w = 0;
          if (u2 < dlim) w = wide ? table[u2] : (table[u2 >> 1] >> (16 * (u2 & 1u))) & 0xFFFFu;
          else if (tsize) w = cb ? table_find<true>(tab, tsize, cb, u2) : table_find<false>(tab, tsize, 0, u2);
          else if (mode == MODE_GLOBAL && u2 < P.n) w = gcnt[u2];
          charge(slot2, w);
        }, part_end);
      }
      if (mode == MODE_GLOBAL) {  // restore the zero invariant of the scratch array
        block_wedges<NT>(b, e, P, S, [&](uint32_t, uint32_t u2) {
          if (u2 < P.n) gcnt[u2] = 0;
        }, nothing);
      }
    } else {
      // Phase 3: endpoint credits, once per distinct u2.
      int64_t mine = 0;
      auto pair = [&](uint32_t u2, int64_t w) {
        if (w < 2) return;
        const int64_t bf = w * (w - 1) / 2;
        mine += bf;
        if (P.per == VERT) credit(P, u2, bf, 16);
      };
      for (uint32_t s = threadIdx.x; s < dwords; s += NT) {
        const uint32_t x = table[s];
        if (wide) {
          pair(s, x);
        } else if (x) {
          pair(2 * s, x & 0xFFFFu);
          pair(2 * s + 1, x >> 16);
        }
      }
      for (uint32_t s = threadIdx.x; s < tsize; s += NT) {
        uint32_t k;
        const uint32_t w = table_entry(tab, tsize, cb, s, k);
        pair(k, w);
      }
      if (mode == MODE_GLOBAL)
        block_wedges<NT>(b, e, P, S, [&](uint32_t, uint32_t u2) {
          if (u2 >= P.n) { record_violation(P.err, 27, u2, i); return; }
          pair(u2, atomicExch(&gcnt[u2], 0u));
        }, nothing);
      if (P.per == VERT) {
        const int64_t s = block_sum_i64(mine, S.red);
        if (threadIdx.x == 0 && s) credit(P, i, s, 19);
      } else {
        total += mine;
      }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      if (P.mode_out) P.mode_out[q] = (uint8_t)mode;
      if (P.cycles) P.cycles[q] = (unsigned long long)(clock64() - t_item);
    }
    q = S.item;
    __syncthreads();
  }
  if (P.per == TOTAL) {
    const int64_t s = block_sum_i64(total, S.red);
    if (threadIdx.x == 0 && s) atomic_add_i64(P.out, s);
  }
}

// Per-edge results: the credits of an edge's two slots, added at its output index.
__global__ void edge_gather_kernel(Params P) {
  for (int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; s < P.m2; s += (int64_t)gridDim.x * blockDim.x) {
    const unsigned long long v = P.sacc32 ? (unsigned long long)P.sacc32[s] : P.sacc64[s];
    if (v) credit(P, P.eout[s], (int64_t)v, 12);
  }
}

// Splits the endpoints [i0, n) with wedges into the warp, mid and block lists.
// counts: [0] block, [1] global scratch, [2] block cursor, [3] warp, [4] mid, [5] mid cursor.
__global__ void classify_endpoints_kernel(const int64_t* __restrict__ wsum, const uint32_t* __restrict__ off,
                                          int64_t i0, int64_t n, int small_w, int64_t mid_w, Geom mid,
                                          uint4* small_items, uint4* mid_items, uint4* items, uint32_t* counts,
                                          uint32_t* err) {
  const int64_t step = (int64_t)gridDim.x * blockDim.x;
  const int64_t rounds = (n - i0 + step - 1) / step;
  for (int64_t r = 0; r < rounds; ++r) {
    const int64_t i = i0 + r * step + (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    int64_t W = 0;
    uint4 it = make_uint4(0, 0, 0, 0);
    if (i < n) {
      W = wsum[i + 1] - wsum[i];
      if (W < 0) record_violation(err, 34, (uint64_t)i, 0);
      it = make_uint4((uint32_t)i, off[i], off[i + 1], (uint32_t)min(W, (int64_t)0xFFFFFFFFll));
    }
    const uint32_t deg = it.z - it.y;
    // A long row takes a CTA however few wedges it has: a warp would walk its slots alone.
    const bool small = W > 0 && W <= small_w && deg <= kWarpRow;
    const bool fits = W > 0 && !small && W <= mid_w && deg <= kMidRow && (mid.dense_ok(it.x, deg) || mid.hash_ok(W, deg));
    const bool big = W > 0 && !small && !fits;
    const unsigned a = list_at(&counts[3], small), c = list_at(&counts[4], fits), d = list_at(&counts[0], big);
    if (small) small_items[a] = it;
    else if (fits) mid_items[c] = it;
    else if (big) items[d] = it;
  }
}

// ---- scheduler support ---------------------------------------------------------------------
constexpr int kItemFeatures = 12;  // features per item; 4 one-hot mode slots follow

// One warp per block-aggregator item: cost-model features and the valid modes (bit m set when
// mode m can hold the item's multiplicity table; the global mode always can).
__global__ void item_features_kernel(Params P, const uint4* __restrict__ items, uint32_t n_items, Geom G, float* F,
                                     uint8_t* valid) {
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const unsigned lane = threadIdx.x & 31u;
  for (int64_t q = warp; q < n_items; q += nwarps) {
    const uint32_t i = items[q].x, b = items[q].y, e = items[q].z;
    const int64_t W = P.wsum[i + 1] - P.wsum[i];
    const uint32_t hy_dense = G.hy_dense();
    unsigned long long lo_w = 0, sumdeg = 0;
    for (uint32_t t = lane; t < e - b; t += 32) {
      const uint32_t j = b + t, v = P.adj[j] >> 1;
      if (v >= P.n) continue;
      const uint32_t vb = P.off[v], ve = P.off[v + 1];
      sumdeg += ve - vb;
      const uint32_t below = lower_bound_u32(P.adj, vb, ve, hy_dense << 1) - vb;
      lo_w += min(below, P.pref[j]);
    }
    lo_w = warp_sum(lo_w);
    sumdeg = warp_sum(sumdeg);
    if (lane == 0) {
      const int64_t hi = W - (int64_t)lo_w;
      const uint64_t hi_c = hi > 0x7fffffff ? 0x7fffffffull : (uint64_t)(hi > 0 ? hi : 0);
      const bool tag_i = !(P.adj[b] & 1u);
      const bool need_center = P.per == EDGE || (P.per == VERT && !tag_i);
      const uint32_t deg = e - b;
      float* f = F + q * kMlpIn;
      f[0] = log2f(1.f + (float)W);
      f[1] = log2f(1.f + (float)i);
      f[2] = log2f(1.f + (float)deg);
      f[3] = log2f(1.f + (float)hi_c);
      f[4] = log2f(1.f + (float)lo_w);
      f[5] = log2f(1.f + (float)sumdeg);
      f[6] = need_center ? 1.f : 0.f;
      f[7] = P.per == EDGE ? 1.f : 0.f;
      f[8] = log2f(1.f + (float)P.n);
      f[9] = f[1] - f[0];
      f[10] = P.sacc32 ? 1.f : 0.f;
      f[11] = log2f(1.f + (float)W / (float)(deg ? deg : 1u));
      for (int k = kItemFeatures; k < kMlpIn; ++k) f[k] = 0.f;
      const bool dense_ok = G.dense_ok(i, deg), hash_ok = G.hash_ok(W, deg), hybrid_ok = G.hybrid_ok(hi_c, deg);
      // The plain rule's choice rides in the top bits.
      const uint32_t rule = G.rule(i, W, deg, hi_c);
      valid[q] = (uint8_t)((dense_ok ? 1u : 0u) | (hash_ok ? 2u : 0u) | 4u | (hybrid_ok ? 8u : 0u) | (rule << 4));
    }
  }
}

// Candidate modes of the learned choice: the shared-memory modes (the global-scratch mode is
// the fallback of items no shared-memory mode can hold; it is never cheaper).
__constant__ int kCandMode[3] = {MODE_DENSE, MODE_HASH, MODE_HYBRID};

// Cost-model rows: item q with candidate c is row 3q + c (features, then the one-hot mode).
__global__ void sched_candidates_kernel(const float* __restrict__ F, uint32_t n_items, float* X) {
  const int64_t total = (int64_t)n_items * 3 * kMlpIn;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = e / kMlpIn;
    const int f = (int)(e - r * kMlpIn);
    const int64_t q = r / 3;
    const int m = kCandMode[r - 3 * q];
    X[e] = f < kItemFeatures ? F[q * kMlpIn + f] : (f - kItemFeatures == m ? 1.f : 0.f);
  }
}

// The valid shared-memory mode with the least predicted log2 cycles; the plain rule's mode is
// kept unless another one is predicted at least kSchedMargin (log2 units, 10%) cheaper.  Items
// no shared-memory mode can hold take the global mode.
constexpr float kSchedMargin = 0.1375f;
__global__ void sched_choose_kernel(const float* __restrict__ y, const uint8_t* __restrict__ valid, uint32_t n_items,
                                    uint8_t* modes, float* pred, uint32_t* n_global) {
  for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < n_items; q += (int64_t)gridDim.x * blockDim.x) {
    const uint32_t vq = valid[q], rule = vq >> 4;
    int best = MODE_GLOBAL;
    float by = 1e30f, ry = 1e30f;
    for (int c = 0; c < 3; ++c) {
      const int m = kCandMode[c];
      if (!(vq & (1u << m))) continue;
      const float v = y[q * 3 + c];
      if (v < by) { by = v; best = m; }
      if ((uint32_t)m == rule) ry = v;
    }
    if (rule != MODE_GLOBAL && ry - by < kSchedMargin) {
      best = (int)rule;
      by = ry;
    }
    modes[q] = (uint8_t)best;
    pred[q] = best == MODE_GLOBAL ? -1.f : by;  // no prediction for the fallback
    if (best == MODE_GLOBAL) atomicAdd(n_global, 1u);
  }
}

// sub[k]: the positions q of block-aggregator items with at least min_w wedges.
__global__ void heavy_items_kernel(const uint4* __restrict__ items, uint32_t n_items,
                                   const int64_t* __restrict__ wsum, int64_t min_w, uint32_t* sub, uint32_t* n_sub) {
  for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < n_items; q += (int64_t)gridDim.x * blockDim.x) {
    const uint32_t i = items[q].x;
    if (wsum[i + 1] - wsum[i] >= min_w) sub[atomicAdd(n_sub, 1u)] = (uint32_t)q;
  }
}

__global__ void gather_items_kernel(const uint4* __restrict__ src, const uint32_t* __restrict__ idx, uint32_t n,
                                    uint4* dst) {
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x)
    dst[k] = src[idx[k]];
}

// Scatters the scored items' modes, predictions and features back to their positions.
__global__ void scatter_scored_kernel(const uint32_t* __restrict__ sub, uint32_t n, const uint8_t* __restrict__ msub,
                                      const float* __restrict__ psub, const float* __restrict__ fsub, uint8_t* modes,
                                      float* pred, float* F) {
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x) {
    const uint32_t q = sub[k];
    modes[q] = msub[k];
    pred[q] = psub[k];
    for (int f = 0; f < kMlpIn; ++f) F[(size_t)q * kMlpIn + f] = fsub[(size_t)k * kMlpIn + f];
  }
}

__device__ __forceinline__ uint64_t mix64(uint64_t z) {
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

// A seeded random valid mode per item (exploration for trace collection).
__global__ void sched_explore_kernel(const uint8_t* __restrict__ valid, uint32_t n_items, uint64_t seed,
                                     uint8_t* modes, uint32_t* n_global) {
  for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < n_items; q += (int64_t)gridDim.x * blockDim.x) {
    const uint32_t vm = valid[q] & 15u;
    const uint32_t c = __popc(vm);
    uint32_t k = (uint32_t)(mix64(seed + 0x9E3779B97F4A7C15ull * (uint64_t)(q + 1)) % c);
    int m = 0;
    for (; m < 4; ++m)
      if (vm & (1u << m)) {
        if (k == 0) break;
        --k;
      }
    modes[q] = (uint8_t)m;
    if (m == MODE_GLOBAL) atomicAdd(n_global, 1u);
  }
}

// What the scheduled items of one list ran with, read back when the call's kernels are through.
struct SchedRecord {
  uint32_t items;
  DevBuf<float> F, pred;
  DevBuf<uint8_t> used;
  DevBuf<unsigned long long> cycles;
};

uint32_t table_words(size_t smem_bytes, size_t fixed) { return (uint32_t)((smem_bytes - fixed) / 4) & ~31u; }

}  // namespace

int64_t count_table_ranks(int smem_bytes) { return 2 * (int64_t)table_words(smem_bytes, shared_fixed<kBlock>()); }

CountResult count_ranked(const Ranked& R, int per, int64_t* out, const CountConfig& cfg, cudaStream_t s) {
  CountResult res;
  const int64_t n = R.n;
  const int64_t out_len = per == VERT ? n : (per == EDGE ? R.m2 / 2 : 1);
  if (out_len > 0) PB_CUDA_TRY(cudaMemsetAsync(out, 0, sizeof(int64_t) * out_len, s));
  if (n == 0 || R.w_rank == 0) return res;
  Params P{};
  P.off = R.off.get();
  P.adj = R.adj.get();
  P.pref = R.pref.get();
  P.wsum = R.wsum.get();
  P.n = n;
  P.per = per;
  P.out = out;
  P.out_len = out_len;
  P.m2 = R.m2;
  DevBuf<CountTail> own_tail;
  CountTail* tail = cfg.tail;
  if (!tail) {
    own_tail.alloc(1, s);
    tail = own_tail.get();
    PB_CUDA_TRY(cudaMemsetAsync(tail, 0, sizeof(CountTail), s));
  }
  P.err = cfg.err ? cfg.err : tail->err;
  P.mstats = tail->mstats;
  uint32_t* const counts = tail->counts;
  const int sms = sm_count();
  int small_w = std::min(cfg.small_w, kWarpTable / 2);
  int smem_bytes = cfg.smem_bytes;
  // Test hooks: shrink the CTA table / the warp threshold so small graphs reach every CTA mode.
  const char* hook_smem = getenv("PB_COUNT_SMEM");
  if (hook_smem) smem_bytes = std::max(16384, std::min(atoi(hook_smem), cfg.smem_bytes));
  if (const char* ev = getenv("PB_COUNT_SMALL_W")) small_w = std::max(0, std::min(atoi(ev), small_w));
  int blocks_per_sm = cfg.blocks_per_sm;
  if (const char* ev = getenv("PB_COUNT_BPS")) blocks_per_sm = std::max(1, std::min(atoi(ev), kBlockPerSm));
  int64_t sched_min_w = kSchedMinWedges;
  if (const char* ev = getenv("PB_SCHED_MIN_WEDGES")) sched_min_w = atoll(ev);  // test hook: score light items too

  // Table geometry of the CTA aggregators.
  int key_bits = 0;
  while (((uint64_t)(n - 1) >> key_bits) != 0) ++key_bits;
  const int count_bits = 32 - std::max(1, key_bits);
  auto geom_of = [&](size_t bytes, size_t fixed) {
    Geom g;
    g.tw = table_words(bytes, fixed);
    g.hy_words = (g.tw / 4 * 3) & ~31u;
    g.cb = count_bits;
    return g;
  };
  const Geom G = geom_of(smem_bytes, shared_fixed<kBlock>());
  const Geom Gm = geom_of(kMidSmem, shared_fixed<kMidBlock>());
  // Endpoints of up to mid_w wedges take the mid aggregator.  Tracing covers every item, the learned
  // scheduler those from sched_min_w on: they see the block aggregator only.
  SchedHooks* sh = cfg.sched;
  int64_t mid_w = kMidWedges;
  if (hook_smem || (sh && sh->trace_X)) mid_w = 0;
  else if (sh && sh->model) mid_w = std::min(mid_w, sched_min_w - 1);
  // Under graph capture nothing is timed or read back here (the recording run checked).
  const bool cap = capturing();
  cudaEvent_t ev[2] = {nullptr, nullptr};
  if (!cap && !cfg.ev)
    for (auto& e : ev) PB_CUDA_TRY(cudaEventCreate(&e));
  else if (!cap)
    std::copy(cfg.ev, cfg.ev + 2, ev);
  // The lists hold kListRange endpoints at a time, so that they take 3.2 GB at most (48 bytes an endpoint,
  // where the other arrays of a call take 40 to 48).
  const int64_t nl = std::min(n, kListRange);
  DevBuf<uint4> lists((size_t)nl * 3, s);  // warp, mid and block lists
  uint4 *small_items = lists.get(), *mid_items = small_items + nl, *items = mid_items + nl;
  DevBuf<uint8_t> modes(nl, s);
  // Per-edge counts are gathered per slot, in 32 bits when they fit: (max degree - 1)^2 < 2^32.  The
  // slots' counts take 8 or 16 bytes an edge, so above kAskBytes they must find room: where they would
  // take more than half of what is left of the device (global scratch is still to come), every
  // credit goes to its edge at once, which takes no memory.
  DevBuf<uint32_t> sacc32;
  DevBuf<unsigned long long> sacc64;
  const uint64_t md = R.max_deg > 0 ? R.max_deg - 1 : 0;
  const char* acc64 = getenv("PB_EDGE_ACC64");  // test hook: force 64-bit per-edge accumulation
  const bool wide_acc = md * md >= (1ull << 32) || (acc64 && *acc64 == '1');
  if (per == EDGE) {
    P.eout = R.eout.get();
    const size_t bytes = (size_t)R.m2 * (wide_acc ? 8 : 4);
    const bool direct = bytes > kAskBytes && bytes > device_bytes_left() / 2;
    if (!direct && !wide_acc) {
      sacc32.alloc(R.m2, s);
      PB_CUDA_TRY(cudaMemsetAsync(sacc32.get(), 0, sacc32.bytes(), s));
      P.sacc32 = sacc32.get();
    } else if (!direct) {
      sacc64.alloc(R.m2, s);
      PB_CUDA_TRY(cudaMemsetAsync(sacc64.get(), 0, sacc64.bytes(), s));
      P.sacc64 = sacc64.get();
    }
  }
  DevBuf<uint32_t> gscratch;
  std::vector<SchedRecord> records;
  for (int64_t i0 = 0; i0 < n; i0 += kListRange) {
    const int64_t i1 = std::min(n, i0 + kListRange);
    if (i0 > 0) PB_CUDA_TRY(cudaMemsetAsync(counts, 0, sizeof(tail->counts), s));
    PB_LAUNCH(classify_endpoints_kernel, std::max(1, std::min(ceil_div(i1 - i0, 256), sms * 8)), 256, 0, s, R.wsum.get(),
              R.off.get(), i0, i1, small_w, mid_w, Gm, small_items, mid_items, items, counts, P.err);
    uint32_t hc[5];
    readback(hc, counts, sizeof(hc), s);
    const uint32_t n_block = hc[0], n_small = hc[3], n_mid = hc[4];
    if (n_block > 0) {
      PB_LAUNCH(plain_modes_kernel, (int)std::min<int64_t>(ceil_div(n_block, 8), sms * 8), 256, 0, s, P, items,
                counts, G, modes.get(), counts + 1);
      readback(&hc[1], counts + 1, sizeof(uint32_t), s);
    }
    res.n_big += (int)(n_block + n_mid);
    if (!cap && i0 == 0) PB_CUDA_TRY(cudaEventRecord(ev[0], s));
    // Scheduler: per-item modes (learned or exploring) and the record of what each item ran
    // with and how long it took.
    const bool sched_on = sh && n_block > 0 && (sh->model || sh->explore || sh->trace_X);
    DevBuf<float> sF, sPred;
    DevBuf<uint8_t> sValid, sUsed;
    DevBuf<uint32_t> sNG;
    DevBuf<unsigned long long> sCyc;
    bool need_global = hc[1] > 0;
    if (sched_on) {
      const uint32_t ni = n_block;
      cudaEvent_t a0, a1;
      PB_CUDA_TRY(cudaEventCreate(&a0));
      PB_CUDA_TRY(cudaEventCreate(&a1));
      PB_CUDA_TRY(cudaEventRecord(a0, s));
      sF.alloc((size_t)ni * kMlpIn, s);
      sValid.alloc(ni, s);
      sUsed.alloc(ni, s);
      sCyc.alloc(ni, s);
      sNG.alloc(1, s);
      PB_CUDA_TRY(cudaMemsetAsync(sNG.get(), 0, sizeof(uint32_t), s));
      const int g1 = std::max(1, std::min(ceil_div(ni, 256), sms * 8));
      // Learned choices score only the items heavy enough for the mode to matter (the rest keep
      // the plain rule, so the scheduler's own cost stays small); tracing covers every item.
      if (sh->model && !sh->trace_X) {
        DevBuf<uint32_t> sub(ni, s), nsub(1, s);
        PB_CUDA_TRY(cudaMemsetAsync(nsub.get(), 0, sizeof(uint32_t), s));
        PB_LAUNCH(heavy_items_kernel, g1, 256, 0, s, items, ni, R.wsum.get(), sched_min_w, sub.get(), nsub.get());
        uint32_t nh = 0;
        readback(&nh, nsub.get(), sizeof(nh), s);
        sPred.alloc(ni, s);
        PB_CUDA_TRY(cudaMemsetAsync(sPred.get(), 0xFF, sizeof(float) * ni, s));  // NaN: no prediction
        PB_CUDA_TRY(cudaMemsetAsync(sF.get(), 0, sF.bytes(), s));
        if (nh > 0) {
          DevBuf<uint4> hitems(nh, s);
          DevBuf<float> hF((size_t)nh * kMlpIn, s), hPr(nh, s);
          DevBuf<uint8_t> hValid(nh, s), hModes(nh, s);
          const int gh = std::max(1, std::min(ceil_div(nh, 256), sms * 8));
          PB_LAUNCH(gather_items_kernel, gh, 256, 0, s, items, sub.get(), nh, hitems.get());
          PB_LAUNCH(item_features_kernel, std::max(1, std::min(ceil_div((int64_t)nh * 32, 256), sms * 8)), 256, 0, s, P,
                    hitems.get(), nh, G, hF.get(), hValid.get());
          DevBuf<float> X((size_t)nh * 3 * kMlpIn, s), y((size_t)nh * 3, s);
          PB_LAUNCH(sched_candidates_kernel, std::max(1, std::min(ceil_div((int64_t)nh * 3 * kMlpIn, 256), sms * 8)), 256,
                    0, s, hF.get(), nh, X.get());
          sh->model->predict_dev(X.get(), (int64_t)nh * 3, y.get(), s);
          PB_LAUNCH(sched_choose_kernel, gh, 256, 0, s, y.get(), hValid.get(), nh, hModes.get(), hPr.get(), sNG.get());
          PB_LAUNCH(scatter_scored_kernel, gh, 256, 0, s, sub.get(), nh, hModes.get(), hPr.get(), hF.get(), modes.get(),
                    sPred.get(), sF.get());
        }
      } else {
        PB_LAUNCH(item_features_kernel, std::max(1, std::min(ceil_div((int64_t)ni * 32, 256), sms * 8)), 256, 0, s, P,
                  items, ni, G, sF.get(), sValid.get());
      }
      if (sh->model && sh->trace_X) {
        DevBuf<float> X((size_t)ni * 3 * kMlpIn, s), y((size_t)ni * 3, s);
        PB_LAUNCH(sched_candidates_kernel, std::max(1, std::min(ceil_div((int64_t)ni * 3 * kMlpIn, 256), sms * 8)), 256,
                  0, s, sF.get(), ni, X.get());
        sh->model->predict_dev(X.get(), (int64_t)ni * 3, y.get(), s);
        sPred.alloc(ni, s);
        PB_LAUNCH(sched_choose_kernel, g1, 256, 0, s, y.get(), sValid.get(), ni, modes.get(), sPred.get(), sNG.get());
      } else if (sh->explore) {
        PB_LAUNCH(sched_explore_kernel, g1, 256, 0, s, sValid.get(), ni, sh->seed, modes.get(), sNG.get());
      }
      P.mode_out = sUsed.get();
      P.cycles = sCyc.get();
      uint32_t ng = 0;
      PB_CUDA_TRY(cudaMemcpyAsync(&ng, sNG.get(), sizeof(ng), cudaMemcpyDeviceToHost, s));
      PB_CUDA_TRY(cudaEventRecord(a1, s));
      PB_CUDA_TRY(cudaEventSynchronize(a1));
      need_global = ng > 0 || hc[1] > 0;  // unscored items follow the plain rule
      float ms = 0;
      PB_CUDA_TRY(cudaEventElapsedTime(&ms, a0, a1));
      sh->ms += ms;
      cudaEventDestroy(a0);
      cudaEventDestroy(a1);
    }
    if (n_block > 0) {
      int grid = (int)std::min<int64_t>(n_block, (int64_t)sms * blocks_per_sm);
      if (need_global) {
        // One dense counter array of n entries per CTA: at very large n (the 1e9-edge R-MAT) the
        // CTA count is capped so the arrays stay within half of the free device memory (64 GB at
        // most).
        if (!gscratch.get()) {
          size_t free_b = 0, total_b = 0;
          PB_CUDA_TRY(cudaMemGetInfo(&free_b, &total_b));
          const size_t budget = std::min<size_t>(free_b / 2, size_t(64) << 30);
          const size_t per_cta = (size_t)n * sizeof(uint32_t);
          const int want = i1 < n ? sms * blocks_per_sm : grid;  // later lists may be longer
          const int ctas = (int)std::max<int64_t>(1, std::min<int64_t>(want, (int64_t)(budget / per_cta)));
          gscratch.alloc((size_t)ctas * (size_t)n, s);
          PB_CUDA_TRY(cudaMemsetAsync(gscratch.get(), 0, gscratch.bytes(), s));
        }
        grid = (int)std::min<int64_t>(grid, (int64_t)(gscratch.n / (size_t)n));
      }
      P.modes = modes.get();
      auto kern = count_block_kernel<kBlock, kBlockPerSm>;
      // The limit belongs to the kernel, not to the call: other threads launch it with other geometries.
      PB_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmBytes - kCtaReserved));
      PB_LAUNCH(kern, grid, kBlock, smem_bytes, s, P, items, counts, counts + 2, gscratch.get(), G);
    }
    P.modes = nullptr;
    P.mode_out = nullptr;
    P.cycles = nullptr;
    if (n_mid > 0) {
      auto kern = count_block_kernel<kMidBlock, kMidPerSm>;
      PB_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kMidSmem));
      PB_LAUNCH(kern, (int)std::min<int64_t>(n_mid, (int64_t)sms * kMidPerSm), kMidBlock, kMidSmem, s, P, mid_items,
                counts + 4, counts + 5, (uint32_t*)nullptr, Gm);
    }
    if (n_small > 0) {
      const bool one_word = (uint32_t)small_w <= (1u << count_bits) - 2u;
      auto kern = one_word ? count_warp_kernel<true> : count_warp_kernel<false>;
      const int smem =
          (2 * (int)kHotRanks + kWarpsPerBlockSmall * ((one_word ? 1 : 2) * kWarpTable + 32)) * (int)sizeof(uint32_t);
      PB_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
      PB_LAUNCH(kern, (int)std::min<int64_t>(ceil_div(n_small, kWarpsPerBlockSmall), (int64_t)sms * (one_word ? 6 : 3)),
                kWarpsPerBlockSmall * 32, smem, s, P, small_items, counts + 3, count_bits);
    }
    if (sched_on) records.push_back({n_block, std::move(sF), std::move(sPred), std::move(sUsed), std::move(sCyc)});
  }
  if (P.sacc32 || P.sacc64)
    PB_LAUNCH(edge_gather_kernel, std::max(1, std::min(ceil_div(R.m2, 256), sms * 8)), 256, 0, s, P);
  if (cap) return res;
  PB_CUDA_TRY(cudaEventRecord(ev[1], s));
  if (cfg.tail && cfg.ev && records.empty()) {
    res.pending = true;
    return res;
  }
  CountTail h;
  PB_CUDA_TRY(cudaMemcpyAsync(&h, tail, sizeof(h), cudaMemcpyDeviceToHost, s));
  PB_CUDA_TRY(cudaStreamSynchronize(s));
  finish_count(res, h, ev);
  double mae_sum = 0;
  int64_t npred = 0;
  for (const SchedRecord& r : records) {
    const uint32_t ni = r.items;
    std::vector<float> hF((size_t)ni * kMlpIn), hPred;
    std::vector<uint8_t> hUsed(ni);
    std::vector<unsigned long long> hCyc(ni);
    PB_CUDA_TRY(cudaMemcpy(hF.data(), r.F.get(), r.F.bytes(), cudaMemcpyDeviceToHost));
    PB_CUDA_TRY(cudaMemcpy(hUsed.data(), r.used.get(), r.used.bytes(), cudaMemcpyDeviceToHost));
    PB_CUDA_TRY(cudaMemcpy(hCyc.data(), r.cycles.get(), r.cycles.bytes(), cudaMemcpyDeviceToHost));
    if (sh->model) {
      hPred.resize(ni);
      PB_CUDA_TRY(cudaMemcpy(hPred.data(), r.pred.get(), r.pred.bytes(), cudaMemcpyDeviceToHost));
    }
    for (uint32_t q = 0; q < ni; ++q) {
      const double cyc = (double)std::max<unsigned long long>(hCyc[q], 1ull);
      const double lc = std::log2(cyc);
      if (sh->trace_X) {
        for (int f = 0; f < kMlpIn; ++f)
          sh->trace_X->push_back(f < kItemFeatures ? hF[(size_t)q * kMlpIn + f]
                                                   : (f - kItemFeatures == (int)hUsed[q] ? 1.f : 0.f));
        sh->trace_y->push_back((float)lc);
      }
      if (sh->model && hPred[q] >= 0.f) {  // items the model predicted (not the fallback)
        sh->meas_cycles += cyc;
        sh->pred_cycles += std::exp2((double)hPred[q]);
        mae_sum += std::fabs((double)hPred[q] - lc);
        ++npred;
      }
    }
    sh->items += ni;
  }
  if (!records.empty()) sh->mae_log2 = npred ? mae_sum / npred : 0.0;
  if (!cfg.ev)
    for (auto& e : ev) cudaEventDestroy(e);
  return res;
}

void finish_count(CountResult& res, const CountTail& tail, const cudaEvent_t* ev) {
  for (int k = 0; k < 4; ++k) {
    res.mode_items[k] = tail.mstats[k];
    res.mode_wedges[k] = tail.mstats[4 + k];
  }
  res.pending = false;
  float ms = 0;
  PB_CUDA_TRY(cudaEventElapsedTime(&ms, ev[0], ev[1]));
  res.agg_ms = ms;
  const uint32_t* e = tail.err;
  PB_REQUIRE(e[0] == 0, PB_ECUDA,
             "aggregation: bounds violation code " + std::to_string(e[0]) + " index " +
                 std::to_string(((uint64_t)e[2] << 32) | e[1]) + " aux " + std::to_string(e[3]));
}

}  // namespace pb
