// Ranking stage: degrees, count-side choice, vertex orders (SIDE/DEG/ADEG/COCORE/ACOCORE),
// the ranked CSR with tag bits, and the per-endpoint wedge scan.
#include <algorithm>
#include <cstdlib>

#include "pb_engine.cuh"
#include "pb_prims.cuh"
#include "pb_walk.cuh"

namespace pb {

namespace {

// Neighbour list of combined id x (V ids first, then nv + U id).  `shift` converts a list
// entry to a combined id.
struct Lists {
  const uint32_t* offV;
  const uint32_t* edgV;
  const uint32_t* offU;
  const uint32_t* edgU;
  int64_t nv;
  __device__ __forceinline__ void get(int64_t x, uint32_t& b, uint32_t& e, const uint32_t*& a, int64_t& shift) const {
    if (x < nv) { b = offV[x]; e = offV[x + 1]; a = edgV; shift = nv; }
    else { b = offU[x - nv]; e = offU[x - nv + 1]; a = edgU; shift = 0; }
  }
};

__device__ __forceinline__ uint32_t degree_of(const Lists& L, int64_t x) {
  uint32_t b, e; const uint32_t* a; int64_t sh;
  L.get(x, b, e, a, sh);
  return e - b;
}

// wedgeF (butterfly_utils.h:1061-1070): (v_deg * (v_deg - 1)) / 2 in 32-bit unsigned
// arithmetic, summed per side in 64 bits (cmpWedgeCounts, :1080-1086).
// Both sides in one launch (blockIdx.y: 0 V, 1 U).
__global__ void side_wedges_kernel(const uint32_t* __restrict__ offV, int64_t nv, const uint32_t* __restrict__ offU,
                                   int64_t nu, unsigned long long* acc) {
  const uint32_t* off = blockIdx.y ? offU : offV;
  const int64_t n = blockIdx.y ? nu : nv;
  unsigned long long s = 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    uint32_t d = off[i + 1] - off[i];
    s += (unsigned long long)((uint32_t)(d * (d - 1u)) / 2u);
  }
  s = warp_sum(s);
  if ((threadIdx.x & 31) == 0 && s) atomicAdd(&acc[blockIdx.y], s);
}

// Sort key (ascending = earlier rank) for the degree-based orders.
__global__ void order_keys_kernel(Lists L, int64_t n, int rank_type, int use_v, uint32_t kmax, uint32_t* keys,
                                  uint32_t* ids) {
  for (int64_t x = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; x < n; x += (int64_t)gridDim.x * blockDim.x) {
    uint32_t k;
    if (rank_type == PB_SIDE) {
      bool on_count = use_v ? (x >= L.nv) : (x < L.nv);
      k = on_count ? 0u : 1u;
    } else if (rank_type == PB_DEG) {
      k = kmax - degree_of(L, x);
    } else {  // PB_ADEG
      k = kmax - log_key(degree_of(L, x));
    }
    keys[x] = k;
    ids[x] = (uint32_t)x;
  }
}

// The bucket rounds of getCoCoreRanks / getApproxCoCoreRanks (butterfly_utils.h:448-559), all in
// one cooperative launch: every undone vertex whose key equals the current maximum k is finished;
// each neighbour with key < k (undone, outside the bucket) loses one degree per finished neighbour
// and its key becomes f(new degree) (min with k is implied, since f(new) <= key < k).  Keys only
// decrease, so atomicMin of f over all decrements leaves f(final degree).
// Two barriers a round: the scan that collects bucket k also takes the maximum of the other keys;
// the updates that follow can only lower them, so the next round's k is that maximum or the round
// is empty.  A finished vertex's list is cut into units of kCoUnit entries, so that the hubs of the
// first rounds are not one warp's work.  One launch pair and a host readback per round with one warp
// per vertex took 5.2 ms (R-MAT 2^24 edges, 15 rounds) and 1.8 ms (46 rounds of a uniform graph with
// 1e6 edges); this takes 0.97 ms and 0.45 ms.
struct CoCtl {
  unsigned long long bar;
  uint32_t err, kmax[2], len[2];
};
// Bound of every barrier wait, and the arrivals that complete a barrier: the CTAs (test hook: one more, so
// that every wait runs out).
struct CoWait {
  unsigned long long timeout_ns;
  unsigned arrivals;
};
constexpr uint32_t kCoDone = 0x80000000u;  // finished (keys are degrees or their logarithms, below 2^23)
constexpr uint32_t kCoUnit = 256;
constexpr int kCoThreads = 1024;
// The grid has a thread per vertex, and where rows are long a warp per four units of all lists: the two
// CTAs of K_{1000,1000}'s vertices took 480 us over its 8,000 units.  ACOCORE ranking with one / two / four / eight
// units a warp: K_{1000,1000} 66 / 68 / 76 / 89 us, 3000 x 3000 with 1.4e6 edges 90 / 89 / 95 / 102 (203 by
// vertices); the 46 COCORE rounds of a uniform graph with 1e6 edges 519 / 509 / 460 / 461, since a round's
// barriers grow with the CTAs.
constexpr int64_t kCoUnitsPerWarp = 4;
constexpr unsigned long long kCoTimeoutNs = 60ull * 1000000000ull;

// Grid barrier of a cooperative launch: arrivals are counted in a word that is never reset.
// Bounded: on expiry sets err and returns false in every CTA.
__device__ bool co_barrier(CoCtl* c, unsigned long long target, unsigned long long timeout_ns) {
  __syncthreads();
  int bad = 0;
  if (threadIdx.x == 0) {
    asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(&c->bar), "l"(1ull) : "memory");
    unsigned long long seen, t0 = 0;
    for (unsigned polls = 0;;) {
      asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(seen) : "l"(&c->bar) : "memory");
      if (seen >= target) break;
      if ((++polls & 63u) == 0) {
        unsigned long long now;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
        if (!t0) t0 = now;
        else if (now - t0 > timeout_ns) {
          atomicExch(&c->err, 1u);
          atomicOr(&c->bar, 1ull << 63);
        }
      }
    }
    bad = (seen >> 63) != 0;
  }
  return __syncthreads_or(bad) == 0;
}

__global__ void __launch_bounds__(kCoThreads, 1) cocore_kernel(Lists L, int64_t n, int approx, uint32_t* key, uint32_t* dact,
                                                              uint2* units, CoCtl* ctl, CoWait wait) {
  __shared__ uint32_t s_k, s_len;
  const unsigned lane = threadIdx.x & 31u;
  const int64_t gtid = (int64_t)blockIdx.x * kCoThreads + threadIdx.x, gthreads = (int64_t)gridDim.x * kCoThreads;
  unsigned long long target = 0;
  auto post_max = [&](uint32_t m, uint32_t* to) {
    m = __reduce_max_sync(0xffffffffu, m);
    if (lane == 0 && m) atomicMax(to, m);
  };
  {
    uint32_t m = 0;
    for (int64_t x = gtid; x < n; x += gthreads) {
      uint32_t b, e; const uint32_t* a; int64_t sh;
      L.get(x, b, e, a, sh);
      const uint32_t k = approx ? log_key(e - b) : e - b;
      dact[x] = e - b;
      key[x] = k;
      m = max(m, k + 1u);
    }
    post_max(m, &ctl->kmax[0]);
  }
  if (!co_barrier(ctl, target += wait.arrivals, wait.timeout_ns)) return;
  for (unsigned par = 0;; par ^= 1u) {
    if (threadIdx.x == 0) s_k = *(volatile uint32_t*)&ctl->kmax[par];
    __syncthreads();
    if (s_k == 0) break;
    const uint32_t k = s_k - 1u;
    uint32_t m = 0;
    for (int64_t x0 = gtid - lane; x0 < n; x0 += gthreads) {  // whole warps
      const int64_t x = x0 + lane;
      const uint32_t kx = x < n ? key[x] : kCoDone;
      const bool mine = kx == k;
      if (kx < k) m = max(m, kx + 1u);
      if (!__any_sync(0xffffffffu, mine)) continue;
      uint32_t nu = 0;
      if (mine) {
        key[x] = k | kCoDone;
        uint32_t b, e; const uint32_t* a; int64_t sh;
        L.get(x, b, e, a, sh);
        nu = (e - b + kCoUnit - 1) / kCoUnit;
      }
      const uint32_t incl = warp_inclusive_scan(nu);
      uint32_t at = 0;
      if (lane == 31 && incl) at = atomicAdd(&ctl->len[par], incl);
      at = __shfl_sync(0xffffffffu, at, 31) + incl - nu;
      for (uint32_t c = 0; c < nu; ++c) units[at + c] = make_uint2((uint32_t)x, c);
    }
    post_max(m, &ctl->kmax[par ^ 1u]);
    if (!co_barrier(ctl, target += wait.arrivals, wait.timeout_ns)) return;
    if (threadIdx.x == 0) s_len = *(volatile uint32_t*)&ctl->len[par];
    __syncthreads();
    if (blockIdx.x == 0 && threadIdx.x == 0) {  // every CTA has read kmax[par]; len[par ^ 1] is the last round's
      ctl->kmax[par] = 0;
      ctl->len[par ^ 1u] = 0;
    }
    const uint32_t len = s_len;
    for (uint32_t q = (uint32_t)(gtid >> 5); q < len; q += (uint32_t)(gthreads >> 5)) {
      const uint2 u = units[q];
      uint32_t b, e; const uint32_t* a; int64_t sh;
      L.get(u.x, b, e, a, sh);
      b += u.y * kCoUnit;
      e = min(e, b + kCoUnit);
      for (uint32_t j = b + lane; j < e; j += 32) {
        const int64_t y = (int64_t)a[j] + sh;
        if (key[y] < k) {
          const uint32_t nd = atomicSub(&dact[y], 1u) - 1u;
          atomicMin(&key[y], approx ? log_key(nd) : nd);
        }
      }
    }
    if (!co_barrier(ctl, target += wait.arrivals, wait.timeout_ns)) return;
  }
}

__global__ void cocore_keys_kernel(const uint32_t* __restrict__ key, int64_t n, uint32_t kmax, uint32_t* skeys,
                                   uint32_t* ids) {
  for (int64_t x = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; x < n; x += (int64_t)gridDim.x * blockDim.x) {
    skeys[x] = kmax - (key[x] & ~kCoDone);
    ids[x] = (uint32_t)x;
  }
}

// rank[order[r]] = r and the degrees in rank order.
__global__ void invert_order_kernel(Lists L, const uint32_t* __restrict__ order, int64_t n, uint32_t* rank,
                                    uint32_t* rdeg) {
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n; r += (int64_t)gridDim.x * blockDim.x) {
    const uint32_t x = order[r];
    rank[x] = (uint32_t)r;
    rdeg[r] = degree_of(L, x);
  }
}

// Calls f(valid, slot, row) for every slot of [s0, s0 + len) of a CSR (row: the slot's row), 32 slots of
// one warp at a time: work is cut by slots, not rows, since rows are as uneven as degrees (one
// warp per row left the last hubs running alone: the wedge scan of the power-law graph with 1e7 edges
// took 4.4 ms, in chunks of slots 0.29; its fill 1.2 and 0.14).  The rows of a group's slots are found in the
// next kRowWindows windows of 32 rows, beyond them by a search: vertices without edges may lie millions
// of rows deep between two slots (2^24 vertices, 20,000 edges, SIDE order: walked through, a count took
// 286 ms, searched over 1.8).
constexpr int kRowWindows = 4;
template <class F>
__device__ __forceinline__ void warp_slots(const uint32_t* __restrict__ off, int64_t n, uint32_t s0, uint32_t len, F&& f) {
  const unsigned lane = threadIdx.x & 31u;
  int64_t lo = 0, hi = n;  // the last row with off[row] <= s0, 32-way search
  while (hi - lo > 1) {
    const int64_t step = (hi - lo + 31) / 32, idx = lo + lane * step;
    const unsigned le = __ballot_sync(0xffffffffu, idx < hi && off[idx] <= s0);
    lo += (31 - __clz(le)) * step;  // lane 0 always qualifies
    hi = min(lo + step, hi);
  }
  uint32_t r = (uint32_t)lo;
  walk_groups(s0, len, 32, lane, [&](uint32_t slot, bool valid) {
    uint32_t row = r;
    int windows = 0;
    for (uint32_t base = r;; base += 32) {
      // Starts of rows base + 1 .. base + 32 (off[n] lies above every slot).
      const uint32_t bnd = off[min((int64_t)base + 1 + lane, n)];
      uint32_t c = 0;  // how many of them are at or before this lane's slot
#pragma unroll
      for (uint32_t step = 16; step > 0; step >>= 1)
        if (__shfl_sync(0xffffffffu, bnd, c + step - 1) <= slot) c += step;
      if (__shfl_sync(0xffffffffu, bnd, c) <= slot) ++c;
      if (valid && row == base) row = base + c;
      if (!__any_sync(0xffffffffu, valid && row == base + 32)) break;
      if (++windows < kRowWindows) continue;
      // Many empty rows: the lanes that are left search, in steps that double.
      if (valid && row == base + 32) {
        int64_t first = row, step = 32;
        while (first + step < n && off[first + step] <= slot) {
          first += step;
          step *= 2;
        }
        int64_t end = min(first + step, n);  // off[first] <= slot < off[end]
        while (end - first > 1) {
          const int64_t mid = (first + end) >> 1;
          if (off[mid] <= slot) first = mid;
          else end = mid;
        }
        row = (uint32_t)first;
      }
      __syncwarp();
      break;
    }
    f(valid, slot, row);
    r = __shfl_sync(0xffffffffu, row, 31);
  });
}
// Slots a warp takes at a time: 256 share the search for the first row, 32 while that many warps are
// all resident (small graphs are bound by one warp's chain).
constexpr uint32_t kSlotChunk = 256;

// The neighbours of the ranked graph, slot by slot in rank order (rankGraph,
// butterfly_utils.h:579-623): row r is the vertex x = order[r], y its neighbour of the slot.
// With eout, also the output edge index of the slot (CountERank's conversion,
// butterfly_ecount.h:1728-1738): slots whose neighbour is on the count side index the centre side's
// lists directly; the others hold the index of the same edge in the neighbour's (centre side) list,
// found by binary search (edgeToIdxs, butterfly_utils.h:2034-2062).
// Large graphs (dest != null): dest = rank(y), adj = (r << 1 | on_count_side(x)), to be sorted by dest
// into the rows of y; otherwise adj = (rank(y) << 1 | on_count_side(y)), to be sorted within the row.
__global__ void ranked_fill_kernel(Lists L, const uint32_t* __restrict__ order, const uint32_t* __restrict__ rank,
                                   const uint32_t* __restrict__ roff, int64_t n, int64_t m2, uint32_t chunk, int use_v, uint32_t* dest,
                                   uint32_t* adj, uint32_t* eout) {
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t c = warp * chunk; c < m2; c += nwarps * chunk) {
    warp_slots(roff, n, (uint32_t)c, (uint32_t)min((int64_t)chunk, m2 - c), [&](bool valid, uint32_t s, uint32_t r) {
      if (!valid) return;
      const int64_t x = order[r];
      uint32_t b, e; const uint32_t* a; int64_t sh;
      L.get(x, b, e, a, sh);
      const uint32_t j = b + (s - roff[r]);
      const uint32_t yl = a[j];
      const int64_t y = (int64_t)yl + sh;
      const bool y_v = y < L.nv;
      const uint32_t tag = use_v ? (y_v ? 0u : 1u) : (y_v ? 1u : 0u);
      if (dest) {
        dest[s] = rank[y];
        adj[s] = (r << 1) | (tag ^ 1u);
      } else {
        adj[s] = (rank[y] << 1) | tag;
      }
      if (eout) {
        uint32_t o = j;
        if (!tag) {
          const uint32_t* yo = y_v ? L.offV : L.offU;
          const uint32_t* ya = y_v ? L.edgV : L.edgU;
          o = lower_bound_u32(ya, yo[yl], yo[yl + 1], (uint32_t)(x < L.nv ? x : x - L.nv));
        }
        eout[s] = o;
      }
    });
  }
}

// below[v] = #{u2 in N(v) : u2 < v} in the ranked CSR.
__global__ void below_self_kernel(const uint32_t* __restrict__ off, const uint32_t* __restrict__ adj, int64_t n,
                                  uint32_t* below) {
  for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x) {
    uint32_t b = off[v];
    below[v] = lower_bound_u32(adj, b, off[v + 1], (uint32_t)v << 1) - b;
  }
}

// countWedgesScan on the ranked graph (butterfly_utils.h:1192-1239, INVERSE direction): for
// slot (i, v) the wedges are the u2 in N(v) with u2 < min(i, v).  Lists are ascending, so that
// prefix length is a binary search for i in N(v) (when i < v) or the per-vertex below[v].
__global__ void wedge_scan_kernel(const uint32_t* __restrict__ off, const uint32_t* __restrict__ adj,
                                  const uint32_t* __restrict__ below, int64_t n, int64_t m2, uint32_t chunk, uint32_t* pref,
                                  int64_t* wcount, uint32_t* rowid) {
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const unsigned lane = threadIdx.x & 31u;
  for (int64_t c = warp * chunk; c < m2; c += nwarps * chunk) {
    warp_slots(off, n, (uint32_t)c, (uint32_t)min((int64_t)chunk, m2 - c), [&](bool valid, uint32_t j, uint32_t i) {
      uint32_t L = 0;
      if (valid) {
        const uint32_t v = adj[j] >> 1;
        if (i < v) {
          const uint32_t vb = off[v];
          L = lower_bound_u32(adj, vb, off[v + 1], i << 1) - vb;
        } else {
          const uint32_t vb = below ? 0u : off[v];
          L = below ? below[v] : lower_bound_u32(adj, vb, off[v + 1], v << 1) - vb;
        }
        pref[j] = L;
        if (rowid) rowid[j] = i;
      }
      // One add per row and group of 32 slots (a row's slots are neighbouring lanes).
      const int64_t incl = warp_inclusive_scan((int64_t)L);
      const uint32_t row = valid ? i : 0xFFFFFFFFu;
      const uint32_t prev = __shfl_up_sync(0xffffffffu, row, 1);
      const unsigned heads = __ballot_sync(0xffffffffu, lane == 0 || row != prev);
      const int first = 31 - __clz(heads & (0xffffffffu >> (31 - lane)));
      const int64_t before = __shfl_sync(0xffffffffu, incl, first > 0 ? first - 1 : 0);
      const uint32_t next = __shfl_down_sync(0xffffffffu, row, 1);
      const int64_t sum = incl - (first > 0 ? before : 0);
      if (valid && (lane == 31 || next != row) && sum) atomic_add_i64(&wcount[i], sum);
    });
  }
}

// eti for the orientation of use_v (edgeToIdxs, butterfly_utils.h:2034-2062).
__global__ void eti_kernel(const uint32_t* __restrict__ offC, const uint32_t* __restrict__ edgC,
                           const uint32_t* __restrict__ offK, const uint32_t* __restrict__ edgK, int64_t nk,
                           uint32_t* eti) {
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const unsigned lane = threadIdx.x & 31u;
  for (int64_t i = warp; i < nk; i += nwarps) {
    for (uint32_t e = offK[i] + lane; e < offK[i + 1]; e += 32) {
      uint32_t v = edgK[e];
      eti[e] = lower_bound_u32(edgC, offC[v], offC[v + 1], (uint32_t)i);
    }
  }
}

// Checked mode: rows strictly ascending, values < 2n, output edge indices < m and each
// output edge index used by exactly two slots (one per direction).
__global__ void validate_ranked_kernel(const uint32_t* __restrict__ off, const uint32_t* __restrict__ adj,
                                       const uint32_t* __restrict__ eout, int64_t n, int64_t m, uint32_t* uses,
                                       uint32_t* err) {
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n; r += (int64_t)gridDim.x * blockDim.x) {
    const uint32_t b = off[r], e = off[r + 1];
    if (e < b || (int64_t)e > 2 * m) { if (atomicCAS(&err[0], 0u, 30u) == 0u) { err[1] = (uint32_t)r; err[3] = e; } continue; }
    for (uint32_t k = b; k < e; ++k) {
      const uint32_t t = adj[k];
      if ((int64_t)t >= 2 * n || (k > b && t <= adj[k - 1])) {
        if (atomicCAS(&err[0], 0u, 31u) == 0u) { err[1] = k; err[3] = t; }
        break;
      }
      if (eout) {
        const uint32_t o = eout[k];
        if ((int64_t)o >= m) {
          if (atomicCAS(&err[0], 0u, 32u) == 0u) { err[1] = k; err[3] = o; }
          break;
        }
        atomicAdd(&uses[o], 1u);
      }
    }
  }
}

__global__ void validate_uses_kernel(const uint32_t* __restrict__ uses, int64_t m, uint32_t* err) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m; i += (int64_t)gridDim.x * blockDim.x)
    if (uses[i] != 2u && atomicCAS(&err[0], 0u, 33u) == 0u) { err[1] = (uint32_t)i; err[3] = uses[i]; }
}

// Slots from which the ranked rows are built by one radix sort of (row, neighbour) pairs over the
// whole CSR instead of a sort within each row.  Relabel of R-MAT graphs, per vertex, radix against row
// sort: 2^18 slots 0.115 / 0.098 ms, 2^19 0.119 / 0.121, 2^20 0.125 / 0.190, 2^23 0.449 / 1.033.
// The radix sort holds every array twice (12 bytes a slot more, 16 with output edges, and its counters); where
// that does not fit what is left of the device, rows are sorted in place whatever the size.
constexpr int64_t kRankSort = int64_t(1) << 19;
bool radix_fits(int64_t m2, bool with_eout) {
  const size_t bytes = (size_t)m2 * (with_eout ? 16 : 12) + (size_t)m2 / 4;
  // A recorded pipeline must take the same way when it is captured, so it does not ask.
  return bytes <= size_t(1) << 30 || g_recorder != nullptr || bytes <= device_bytes_left();
}

int bits_for(uint64_t x) {
  int b = 0;
  while (b < 64 && (x >> b) != 0) ++b;
  return b;
}

Lists lists_of(const pb_graph& g) {
  return Lists{g.offV.get(), g.edgV.get(), g.offU.get(), g.edgU.get(), g.nv};
}

// Wedge scan stage of R-MAT graphs with the below[] kernel against without: 2^14 slots 39 / 35 us,
// 2^18 54 / 50, 2^20 78 / 77, 2^21 85 / 93.
constexpr int64_t kSmallSlots = int64_t(1) << 18;

uint32_t slot_chunk(int64_t m2) { return m2 <= (int64_t)sm_count() * 64 * 32 ? 32u : kSlotChunk; }

int grid_for(int64_t n, int per_block = 256) { return std::max(1, std::min(ceil_div(n, per_block), sm_count() * 16)); }

}  // namespace

void side_wedge_sums(const pb_graph& g, unsigned long long* sums, cudaStream_t s) {
  PB_CUDA_TRY(cudaMemsetAsync(sums, 0, 2 * sizeof(unsigned long long), s));
  if (g.nv + g.nu)
    PB_LAUNCH(side_wedges_kernel, dim3(grid_for(std::max(g.nv, g.nu)), 2), 256, 0, s, g.offV.get(), g.nv, g.offU.get(), g.nu,
              sums);
}

void cmp_wedge_counts(const pb_graph& g, int* use_v, int64_t* w_min, int64_t* wv, int64_t* wu, cudaStream_t s) {
  DevBuf<unsigned long long> acc(2, s);
  side_wedge_sums(g, acc.get(), s);
  unsigned long long h[2];
  readback(h, acc.get(), sizeof(h), s);
  *wv = (int64_t)h[0];
  *wu = (int64_t)h[1];
  *use_v = *wv <= *wu;
  *w_min = *wv <= *wu ? *wv : *wu;
}

void vertex_order(const pb_graph& g, int rank_type, int use_v, Ranked& R, cudaStream_t s) {
  const int64_t n = g.nv + g.nu;
  R.n = n;
  R.use_v = use_v;
  R.order.alloc(n, s);
  R.rank.alloc(n, s);
  if (n == 0) return;
  DevBuf<uint32_t> keys(n, s), keys2(n, s), ids2(n, s);
  uint32_t kmax = 0;
  int nbits = 0;
  uint32_t* ids = R.order.get();
  if (rank_type == PB_COCORE || rank_type == PB_ACOCORE) {
    const int approx = rank_type == PB_ACOCORE;
    DevBuf<uint32_t> key(n, s), dact(n, s);
    DevBuf<uint2> units((size_t)(n + 2 * g.m / kCoUnit + 1), s);
    R.co.alloc(sizeof(CoCtl), s);
    CoCtl* ctl = reinterpret_cast<CoCtl*>(R.co.get());
    PB_CUDA_TRY(cudaMemsetAsync(ctl, 0, sizeof(CoCtl), s));
    kmax = approx ? (g.max_deg ? 32u - (uint32_t)__builtin_clz(g.max_deg) : 0u) : g.max_deg;
    Lists lists = lists_of(g);
    int64_t nn = n;
    int ap = approx;
    uint32_t *kp = key.get(), *dp = dact.get();
    uint2* up = units.get();
    CoWait wait{kCoTimeoutNs, 0};
    if (const char* e = getenv("PB_RANK_BARRIER_TIMEOUT_MS")) wait.timeout_ns = 1000000ull * strtoull(e, nullptr, 10);
    void* args[] = {&lists, &nn, &ap, &kp, &dp, &up, &ctl, &wait};
    const int64_t unit_ctas = 2 * g.m / (kCoUnitsPerWarp * kCoUnit * (kCoThreads / 32));
    const int grid = (int)std::max<int64_t>(1, std::min<int64_t>(sm_count(), std::max<int64_t>(ceil_div(n, kCoThreads), unit_ctas)));
    wait.arrivals = (unsigned)grid;
    // Test hook: no barrier completes, with 1 in any ranking, with 2 in captured graphs.
    if (const char* e = getenv("PB_RANK_TEST_STUCK_BARRIER")) wait.arrivals += *e == '1' || (*e == '2' && capturing());
    PB_CUDA_TRY(cudaLaunchCooperativeKernel((const void*)cocore_kernel, dim3(grid), dim3(kCoThreads), args, 0, s));
    if (g_launch_counter) ++*g_launch_counter;
    PB_LAUNCH(cocore_keys_kernel, grid_for(n), 256, 0, s, key.get(), n, kmax, keys.get(), ids);
    nbits = bits_for(kmax);
  } else {
    if (rank_type == PB_DEG) kmax = g.max_deg;
    else if (rank_type == PB_ADEG) kmax = g.max_deg ? 32u - (uint32_t)__builtin_clz(g.max_deg) : 0u;
    else kmax = 1;
    PB_LAUNCH(order_keys_kernel, grid_for(n), 256, 0, s, lists_of(g), n, rank_type, use_v, kmax, keys.get(), ids);
    nbits = bits_for(kmax);
  }
  // Stable sort by key: ties keep combined-id order.
  bool alt = radix_sort_pairs_u32(keys.get(), ids, keys2.get(), ids2.get(), n, 0, nbits, s);
  if (alt) std::swap(R.order.p, ids2.p);
  R.rdeg.alloc(n, s);
  PB_LAUNCH(invert_order_kernel, grid_for(n), 256, 0, s, lists_of(g), R.order.get(), n, R.rank.get(), R.rdeg.get());
}

void build_ranked_csr(const pb_graph& g, Ranked& R, bool with_eout, cudaStream_t s) {
  const int64_t n = R.n;
  R.m2 = 2 * g.m;
  R.off.alloc(n + 1, s);
  R.adj.alloc(R.m2 > 0 ? R.m2 : 1, s);
  if (with_eout) R.eout.alloc(R.m2 > 0 ? R.m2 : 1, s);
  R.max_deg = g.max_deg;
  if (n == 0) {
    PB_CUDA_TRY(cudaMemsetAsync(R.off.get(), 0, sizeof(uint32_t), s));
    return;
  }
  exclusive_scan_u32(R.rdeg.get(), R.off.get(), n, s);
  R.rdeg.release();
  if (R.m2 == 0) return;
  const uint32_t chunk = slot_chunk(R.m2);
  const int grid = grid_for((R.m2 + chunk - 1) / chunk * 32);
  if (R.m2 < kRankSort || !radix_fits(R.m2, with_eout)) {
    PB_LAUNCH(ranked_fill_kernel, grid, 256, 0, s, lists_of(g), R.order.get(), R.rank.get(), R.off.get(), n, R.m2, chunk, R.use_v,
              (uint32_t*)nullptr, R.adj.get(), with_eout ? R.eout.get() : nullptr);
    segmented_sort_rows(R.off.get(), n, R.adj.get(), with_eout ? R.eout.get() : nullptr, bits_for((uint64_t)(2 * n)),
                        g.max_deg, s);
    return;
  }
  DevBuf<uint32_t> dest(R.m2, s), dest2(R.m2, s), adj2(R.m2, s), eout2;
  if (with_eout) eout2.alloc(R.m2, s);
  PB_LAUNCH(ranked_fill_kernel, grid, 256, 0, s, lists_of(g), R.order.get(), R.rank.get(), R.off.get(), n, R.m2, chunk, R.use_v,
            dest.get(), R.adj.get(), with_eout ? R.eout.get() : nullptr);
  if (radix_sort_pairs_u32(dest.get(), R.adj.get(), dest2.get(), adj2.get(), R.m2, 0, bits_for((uint64_t)(n - 1)), s,
                           R.eout.get(), eout2.get())) {
    std::swap(R.adj.p, adj2.p);
    std::swap(R.eout.p, eout2.p);
  }
}

void wedge_scan(Ranked& R, cudaStream_t s, bool with_rows) {
  const int64_t n = R.n;
  R.wsum.alloc(n + 1, s);
  R.pref.alloc(R.m2 > 0 ? R.m2 : 1, s);
  if (with_rows) R.rowid.alloc(R.m2 > 0 ? R.m2 : 1, s);
  if (n == 0) {
    PB_CUDA_TRY(cudaMemsetAsync(R.wsum.get(), 0, sizeof(int64_t), s));
    R.w_rank = 0;
    return;
  }
  // Small graphs look below[v] up slot by slot: the second search costs less than a launch.
  const bool with_below = R.m2 > kSmallSlots;
  DevBuf<uint32_t> below;
  DevBuf<int64_t> wc(n, s);
  PB_CUDA_TRY(cudaMemsetAsync(wc.get(), 0, wc.bytes(), s));
  if (with_below) {
    below.alloc(n, s);
    PB_LAUNCH(below_self_kernel, grid_for(n), 256, 0, s, R.off.get(), R.adj.get(), n, below.get());
  }
  const uint32_t chunk = slot_chunk(R.m2);
  if (R.m2 > 0)
    PB_LAUNCH(wedge_scan_kernel, grid_for((R.m2 + chunk - 1) / chunk * 32), 256, 0, s, R.off.get(), R.adj.get(),
              below.get(), n, R.m2, chunk, R.pref.get(), wc.get(), R.rowid.get());
  exclusive_scan_i64(wc.get(), R.wsum.get(), n, s);
  readback(&R.w_rank, R.wsum.get() + n, sizeof(int64_t), s);
  if (R.co.get()) {
    uint32_t err = 0;
    const uint32_t* word = &reinterpret_cast<CoCtl*>(R.co.get())->err;
    // A captured graph hands the word of every replay to the recorder's status.
    if (capturing())
      PB_CUDA_TRY(cudaMemcpyAsync(g_recorder->status + 2, word, sizeof(err), cudaMemcpyDeviceToHost, s));
    readback(&err, word, sizeof(err), s);
    PB_REQUIRE(err == 0, PB_ETIMEOUT, "ranking: a grid barrier wait ran out of time");
  }
}

bool check_mode() {
  static int on = -1;
  if (on < 0) {
    const char* e = getenv("PB_CHECK");
    on = (e && *e && *e != '0') ? 1 : 0;
  }
  return on == 1;
}

void validate_ranked(const Ranked& R, int64_t m, uint32_t* err, cudaStream_t s) {
  if (R.n == 0) return;
  DevBuf<uint32_t> uses;
  if (R.eout.get()) {
    uses.alloc(m > 0 ? m : 1, s);
    PB_CUDA_TRY(cudaMemsetAsync(uses.get(), 0, uses.bytes(), s));
  }
  PB_LAUNCH(validate_ranked_kernel, grid_for(R.n), 256, 0, s, R.off.get(), R.adj.get(), R.eout.get(), R.n, m,
            uses.get(), err);
  if (R.eout.get() && m > 0) PB_LAUNCH(validate_uses_kernel, grid_for(m), 256, 0, s, uses.get(), m, err);
}

void edge_to_idxs(const pb_graph& g, int use_v, uint32_t* eti, cudaStream_t s) {
  const int64_t nk = use_v ? g.nu : g.nv;
  if (nk == 0 || g.m == 0) return;
  const uint32_t* offC = use_v ? g.offV.get() : g.offU.get();
  const uint32_t* edgC = use_v ? g.edgV.get() : g.edgU.get();
  const uint32_t* offK = use_v ? g.offU.get() : g.offV.get();
  const uint32_t* edgK = use_v ? g.edgU.get() : g.edgV.get();
  PB_LAUNCH(eti_kernel, grid_for(nk * 32), 256, 0, s, offC, edgC, offK, edgK, nk, eti);
}

}  // namespace pb
