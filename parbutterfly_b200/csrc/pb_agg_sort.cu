// SORT and HIST wedge aggregation (count types SORT/ASORT and HIST/AHIST).
//
// Reference: CountSort / CountSortCE (butterfly_count.h:43-313) materialise the wedges of a batch
// of endpoints, sort them by endpoint pair and read multiplicities off the runs; CountHist /
// CountHistCE (:572-893) reduce the wedge keys with a semisort histogram
// (pbbsa::sparse_histogram, lib/histogram.h:252-345).  Batches hold at most max_wedges wedges
// (the -m option, getNextWedgeIdx, butterfly_utils.h:1700-1714).
//
// Device version.  A batch of endpoints [i0, i1) is flattened: wedge t of the batch lives at
// position t, with key ((i - i0) << bits of u2) | u2 (32-bit keys when they fit), the slot j of
// (i, v) and the slot of (v, u2) in side arrays.  Warps materialise chunks of consecutive wedges,
// 32 slots at a time.
//   SORT: stable LSD radix sort of (key, position) pairs; run boundaries give w.
//   HIST: one radix pass on the top bits of a key hash groups each key's wedges into one
//         bucket; one CTA per bucket builds the bucket's histogram in a shared-memory table,
//         with __match_any_sync combining equal keys of a warp into one atomic; a bucket whose
//         distinct keys overflow the table is redone against a global-memory table.
// Credits then follow the ranked semantics: C(w,2) per distinct pair to tagged endpoints (and to
// the total), w-1 per wedge to tagged centres (VERT) or to both wedge edges (EDGE).
#include <algorithm>
#include <type_traits>

#include "pb_engine.cuh"
#include "pb_prims.cuh"

namespace pb {

namespace {

enum Per { VERT = 0, EDGE = 1, TOTAL = 2 };
constexpr uint32_t kChunk = 512;  // wedges per materialising warp

// The last index s in [lo, hi) with a[s] <= t (a ascending, a[lo] <= t): 32-way search by a warp.
__device__ __forceinline__ int64_t warp_last_le(const int64_t* __restrict__ a, int64_t lo, int64_t hi, int64_t t) {
  while (hi - lo > 1) {
    const int64_t step = (hi - lo + 31) / 32;
    const int64_t idx = lo + lane_id() * step;
    const unsigned le = __ballot_sync(0xffffffffu, idx < hi && a[idx] <= t);
    lo += (31 - __clz(le)) * step;  // lane 0 always qualifies
    hi = min(lo + step, hi);
  }
  return lo;
}

// Materialises wedges [t_begin, t_end) (global flattened indices) at positions t - t_begin.
// Bound by its writes (20 bytes a wedge).  A warp takes kChunk wedges and walks their slots 32 at
// a time: lanes load 32 slots at once, every wedge finds its slot by a search over the lanes'
// prefixes, so neighbouring lanes write neighbouring positions.  Where a group of 32 slots holds no
// wedge, every lane searches the prefix for a wedge of its own: most slots of the low ranks hold
// none, and a wedge may lie thousands of slots behind the one before it.  (1e7 wedges of a uniform
// graph with 1e6 edges: empty slots walked one by one 129 ms, searched over for one wedge at a time
// 1.9, for 32 0.23.)
template <class K>
__global__ void materialize_kernel(const uint32_t* __restrict__ off, const uint32_t* __restrict__ adj,
                                   const uint32_t* __restrict__ pref, const int64_t* __restrict__ spre,
                                   const uint32_t* __restrict__ rowid, int64_t m2, int64_t t_begin, int64_t t_end,
                                   uint32_t i0, int ubits, K* keys, uint32_t* vals, uint32_t* jarr, uint32_t* s2arr) {
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const unsigned lane = threadIdx.x & 31u;
  for (int64_t c0 = t_begin + warp * (int64_t)kChunk; c0 < t_end; c0 += nwarps * (int64_t)kChunk) {
    const int64_t c1 = min(c0 + (int64_t)kChunk, t_end);
    int64_t s = warp_last_le(spre, 0, m2, c0), t = c0;
    while (t < c1) {
      const int64_t j = s + lane;
      int64_t base = c1, end = c1;  // lanes beyond the last slot hold nothing
      uint32_t vs = 0, row = 0;
      if (j < m2) {
        base = spre[j];
        end = base + pref[j];
        vs = off[adj[j] >> 1];
        row = rowid[j];
      }
      const int64_t gend = min(c1, __shfl_sync(0xffffffffu, end, 31));
      for (int64_t t0 = t; t0 < gend; t0 += 32) {
        const int64_t x = t0 + lane;
        uint32_t lo = 0;  // the last lane whose slot begins at or before x (it holds x)
#pragma unroll
        for (uint32_t step = 16; step > 0; step >>= 1)
          if (__shfl_sync(0xffffffffu, base, lo + step) <= x) lo += step;
        const int64_t b = __shfl_sync(0xffffffffu, base, lo);
        const uint32_t v0 = __shfl_sync(0xffffffffu, vs, lo), r = __shfl_sync(0xffffffffu, row, lo);
        if (x < gend) {
          const uint32_t slot2 = v0 + (uint32_t)(x - b);
          const int64_t pos = x - t_begin;
          keys[pos] = ((K)(r - i0) << ubits) | (K)(adj[slot2] >> 1);
          vals[pos] = (uint32_t)pos;
          jarr[pos] = (uint32_t)(s + lo);
          s2arr[pos] = slot2;
        }
      }
      if (gend > t) {
        t = gend;
        s += 32;
      } else {
        const int64_t x = t + lane;
        int64_t lo = s, hi = m2;  // the last slot with spre[slot] <= x
        while (hi - lo > 1) {
          const int64_t mid = (lo + hi) >> 1;
          if (spre[mid] <= x) lo = mid;
          else hi = mid;
        }
        if (x < c1) {
          const uint32_t slot2 = off[adj[lo] >> 1] + (uint32_t)(x - spre[lo]);
          const int64_t pos = x - t_begin;
          keys[pos] = ((K)(rowid[lo] - i0) << ubits) | (K)(adj[slot2] >> 1);
          vals[pos] = (uint32_t)pos;
          jarr[pos] = (uint32_t)lo;
          s2arr[pos] = slot2;
        }
        const int last = (int)min((int64_t)31, c1 - t - 1);
        s = __shfl_sync(0xffffffffu, lo, last);
        t += last + 1;
      }
    }
  }
}

struct Credit {
  const uint32_t* off;
  const uint32_t* adj;
  const uint32_t* eout;
  int per;
  uint32_t i0;
  int ubits;  // key = (endpoint - i0) << ubits | u2
  int64_t* out;
  uint32_t* out32;
  unsigned long long* total;
  __device__ __forceinline__ void add(uint64_t idx, int64_t v) const {
    if (out32) atomicAdd(&out32[idx], (uint32_t)v);
    else atomic_add_i64(&out[idx], v);
  }
  __device__ __forceinline__ uint32_t endpoint(uint64_t key) const { return i0 + (uint32_t)(key >> ubits); }
  __device__ __forceinline__ uint32_t end2(uint64_t key) const { return (uint32_t)(key & ((1ull << ubits) - 1ull)); }
  // One wedge of multiplicity w: centre / edge credits.
  __device__ __forceinline__ void wedge(uint32_t i, uint32_t j, uint32_t slot2, int64_t w) const {
    if (w < 2) return;
    if (per == EDGE) {
      add(eout[j], w - 1);
      add(eout[slot2], w - 1);
    } else if (per == VERT) {
      const uint32_t vt = adj[j];
      if (vt & 1u) add(vt >> 1, w - 1);
    }
  }
  // One distinct (i, u2) of multiplicity w: endpoint credits.  i is on the count side when
  // its neighbours are not (tag bit of any entry of its row).
  __device__ __forceinline__ void pair(uint32_t i, uint32_t u2, int64_t w) const {
    if (w < 2) return;
    const int64_t b = w * (w - 1) / 2;
    if (per == TOTAL) atomicAdd(total, (unsigned long long)b);
    else if (per == VERT && !(adj[off[i]] & 1u)) {
      add(i, b);
      add(u2, b);
    }
  }
};

// SORT: sorted keys -> run heads.
template <class K>
__global__ void run_heads_kernel(const K* __restrict__ keys, int64_t n, uint32_t* head) {
  for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += (int64_t)gridDim.x * blockDim.x)
    head[p] = (p == 0 || keys[p] != keys[p - 1]) ? 1u : 0u;
}

// start[r]: first position of run r; start[number of runs] = n.
__global__ void run_starts_kernel(const uint32_t* __restrict__ head, const uint32_t* __restrict__ rid, int64_t n,
                                  uint32_t* start) {
  for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += (int64_t)gridDim.x * blockDim.x)
    if (head[p]) start[rid[p]] = (uint32_t)p;
  if (blockIdx.x == 0 && threadIdx.x == 0) start[rid[n]] = (uint32_t)n;
}

// Runs lie in endpoint order, so neighbouring lanes mostly credit one endpoint i: their credits are
// added up in the warp first; those of the lowest ranks (which share wedges with most endpoints) in
// shared memory (3.8e6 wedges of a Zipf graph: 178 us with every credit on its own, 145 so).
constexpr uint32_t kHotRanks = 256;

template <class K>
__global__ void __launch_bounds__(256) sort_credit_kernel(const K* __restrict__ keys, const uint32_t* __restrict__ vals,
                                   const uint32_t* __restrict__ jarr, const uint32_t* __restrict__ s2arr,
                                   const uint32_t* __restrict__ head, const uint32_t* __restrict__ rid,
                                   const uint32_t* __restrict__ start, int64_t n, Credit C) {
  __shared__ uint32_t hot[2 * kHotRanks];  // low and high words
  for (uint32_t s = threadIdx.x; s < 2 * kHotRanks; s += blockDim.x) hot[s] = 0;
  __syncthreads();
  const unsigned lane = threadIdx.x & 31u;
  auto credit = [&](uint32_t x, unsigned long long v) {
    if (x < kHotRanks) {
      const uint32_t lo = (uint32_t)v, old = atomicAdd(&hot[x], lo);
      const uint32_t hi = (uint32_t)(v >> 32) + (old + lo < old ? 1u : 0u);
      if (hi) atomicAdd(&hot[kHotRanks + x], hi);
    } else {
      C.add(x, (int64_t)v);
    }
  };
  unsigned long long total = 0;
  const int64_t step = (int64_t)gridDim.x * blockDim.x;
  for (int64_t p0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x - lane; p0 < n; p0 += step) {  // whole warps
    const int64_t p = p0 + lane;
    unsigned long long mine = 0;  // butterflies of the run that begins here
    uint32_t i = 0xFFFFFFFFu;
    if (p < n) {
      const uint32_t h = head[p], r = rid[p] - (h ? 0u : 1u);  // rid = heads strictly before p
      const int64_t w = (int64_t)start[r + 1] - start[r];
      const uint64_t key = keys[p];
      i = C.endpoint(key);
      if (w >= 2) {
        if (C.per == EDGE || (C.per == VERT && (C.adj[C.off[i]] & 1u))) {
          const uint32_t pos = vals[p];
          C.wedge(i, jarr[pos], s2arr[pos], w);
        } else if (h) {
          mine = (unsigned long long)(w * (w - 1) / 2);
          if (C.per == VERT) credit(C.end2(key), mine);
        }
      }
    }
    if (C.per == VERT) {
      if (!__any_sync(0xffffffffu, mine != 0)) continue;
      const unsigned long long incl = warp_inclusive_scan(mine);
      const uint32_t next = __shfl_down_sync(0xffffffffu, i, 1), prev = __shfl_up_sync(0xffffffffu, i, 1);
      const unsigned heads = __ballot_sync(0xffffffffu, lane == 0 || i != prev);
      const int first = 31 - __clz(heads & (0xffffffffu >> (31 - lane)));
      const unsigned long long before = __shfl_sync(0xffffffffu, incl, first > 0 ? first - 1 : 0);
      const unsigned long long sum = incl - (first > 0 ? before : 0ull);
      if (sum && (lane == 31 || next != i)) credit(i, sum);
    } else {
      total += mine;
    }
  }
  if (C.per == TOTAL) {
    total = warp_sum(total);
    if (lane == 0 && total) atomicAdd(C.total, total);
  } else if (C.per == VERT) {
    __syncthreads();
    for (uint32_t s = threadIdx.x; s < kHotRanks; s += blockDim.x) {
      const unsigned long long v = ((unsigned long long)hot[kHotRanks + s] << 32) | hot[s];
      if (v) C.add(s, (int64_t)v);
    }
  }
}

// HIST: bucket of a key (top bits of a 64-bit mix), the radix digit of the semisort pass.
__device__ __forceinline__ uint32_t key_bucket(uint64_t k, int bits) {
  k ^= k >> 33;
  k *= 0xff51afd7ed558ccdull;
  k ^= k >> 33;
  return (uint32_t)(k >> (64 - bits));
}

__global__ void bucket_keys_kernel(const uint64_t* __restrict__ keys, int64_t n, int bits, uint32_t* bkey) {
  for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += (int64_t)gridDim.x * blockDim.x)
    bkey[p] = key_bucket(keys[p], bits);
}

__global__ void bucket_bounds_kernel(const uint32_t* __restrict__ bkey_sorted, int64_t n, uint32_t nb, uint32_t* bstart) {
  for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += (int64_t)gridDim.x * blockDim.x) {
    const uint32_t b = bkey_sorted[p];
    const uint32_t prev = p ? bkey_sorted[p - 1] : 0xFFFFFFFFu;
    if (b != prev)
      for (uint32_t q = (prev == 0xFFFFFFFFu ? 0u : prev + 1u); q <= b; ++q) bstart[q] = (uint32_t)p;
    if (p == n - 1)
      for (uint32_t q = b + 1; q <= nb; ++q) bstart[q] = (uint32_t)n;
  }
}

constexpr int kHistThreads = 256;
constexpr uint32_t kHistSlots = 2048;  // 64-bit keys + 32-bit counts: 24 KiB
constexpr unsigned long long kNoKey = ~0ull;

__device__ __forceinline__ uint32_t hslot64(uint64_t k, uint32_t mask) {
  return (uint32_t)((k * 0x9E3779B97F4A7C15ull) >> 40) & mask;
}

// Insert-or-add with a bounded probe; false when the table is full.
__device__ __forceinline__ bool h64_add(unsigned long long* keys, uint32_t* cnt, uint32_t mask, uint64_t k, uint32_t c) {
  uint32_t h = hslot64(k, mask);
  for (uint32_t probes = 0; probes <= mask; ++probes) {
    unsigned long long cur = keys[h];
    if (cur == k) { atomicAdd(&cnt[h], c); return true; }
    if (cur == kNoKey) {
      unsigned long long prev = atomicCAS(&keys[h], kNoKey, (unsigned long long)k);
      if (prev == kNoKey || prev == k) { atomicAdd(&cnt[h], c); return true; }
    }
    h = (h + 1) & mask;
  }
  return false;
}

__device__ __forceinline__ uint32_t h64_get(const unsigned long long* keys, const uint32_t* cnt, uint32_t mask, uint64_t k) {
  uint32_t h = hslot64(k, mask);
  for (uint32_t probes = 0; probes <= mask; ++probes) {
    const unsigned long long cur = keys[h];
    if (cur == k) return cnt[h];
    if (cur == kNoKey) return 0;
    h = (h + 1) & mask;
  }
  return 0;
}

// One CTA per bucket.  Equal keys of a warp are combined with __match_any_sync before the
// shared-memory insert.  Overflowing buckets are flagged and redone by hist_global_kernel.
__global__ void __launch_bounds__(kHistThreads) hist_bucket_kernel(const uint64_t* __restrict__ keys,
                                                                   const uint32_t* __restrict__ vals,
                                                                   const uint32_t* __restrict__ jarr,
                                                                   const uint32_t* __restrict__ s2arr,
                                                                   const uint32_t* __restrict__ bstart, uint32_t nb,
                                                                   Credit C, uint32_t* overflow) {
  __shared__ unsigned long long tk[kHistSlots];
  __shared__ uint32_t tc[kHistSlots];
  __shared__ int failed;
  const unsigned lane = threadIdx.x & 31u;
  for (uint32_t b = blockIdx.x; b < nb; b += gridDim.x) {
    const uint32_t p0 = bstart[b], p1 = bstart[b + 1];
    if (p0 == p1) continue;
    for (uint32_t s = threadIdx.x; s < kHistSlots; s += kHistThreads) { tk[s] = kNoKey; tc[s] = 0; }
    if (threadIdx.x == 0) failed = 0;
    __syncthreads();
    for (uint32_t q0 = p0; q0 < p1; q0 += kHistThreads) {
      const uint32_t q = q0 + threadIdx.x;
      const bool valid = q < p1;
      const uint64_t k = valid ? keys[q] : kNoKey;
      const unsigned peers = __match_any_sync(0xffffffffu, k);
      if (valid && lane == (unsigned)(__ffs(peers) - 1))
        if (!h64_add(tk, tc, kHistSlots - 1, k, (uint32_t)__popc(peers))) failed = 1;
    }
    __syncthreads();
    if (failed) {
      if (threadIdx.x == 0) overflow[atomicAdd(&overflow[0], 1u) + 1] = b;
      __syncthreads();
      continue;
    }
    for (uint32_t q = p0 + threadIdx.x; q < p1; q += kHistThreads) {
      const uint64_t k = keys[q];
      const int64_t w = h64_get(tk, tc, kHistSlots - 1, k);
      const uint32_t pos = vals[q];
      C.wedge(C.endpoint(k), jarr[pos], s2arr[pos], w);
    }
    for (uint32_t s = threadIdx.x; s < kHistSlots; s += kHistThreads) {
      const unsigned long long k = tk[s];
      if (k == kNoKey) continue;
      C.pair(C.endpoint(k), C.end2(k), tc[s]);
    }
    __syncthreads();
  }
}

// Redo of overflowing buckets against a global open-addressing table (one bucket per CTA,
// regions of the table carved by bucket start).
__global__ void hist_global_kernel(const uint64_t* __restrict__ keys, const uint32_t* __restrict__ vals,
                                   const uint32_t* __restrict__ jarr, const uint32_t* __restrict__ s2arr,
                                   const uint32_t* __restrict__ bstart, const uint32_t* __restrict__ overflow,
                                   unsigned long long* gk, uint32_t* gc, Credit C) {
  const uint32_t nover = overflow[0];
  for (uint32_t o = blockIdx.x; o < nover; o += gridDim.x) {
    const uint32_t b = overflow[o + 1];
    const uint32_t p0 = bstart[b], p1 = bstart[b + 1];
    // Region of 4 x bucket length; the table is the largest power of two inside it (load <= 1/2).
    unsigned long long* tk = gk + 4ull * p0;
    uint32_t* tc = gc + 4ull * p0;
    const uint32_t cap = 4 * (p1 - p0);
    uint32_t mask = 1;
    while (mask * 2 <= cap) mask *= 2;
    mask -= 1;
    for (uint32_t s = threadIdx.x; s <= mask; s += blockDim.x) { tk[s] = kNoKey; tc[s] = 0; }
    __syncthreads();
    for (uint32_t q = p0 + threadIdx.x; q < p1; q += blockDim.x) h64_add(tk, tc, mask, keys[q], 1u);
    __syncthreads();
    for (uint32_t q = p0 + threadIdx.x; q < p1; q += blockDim.x) {
      const uint64_t k = keys[q];
      const uint32_t pos = vals[q];
      C.wedge(C.endpoint(k), jarr[pos], s2arr[pos], h64_get(tk, tc, mask, k));
    }
    for (uint32_t s = threadIdx.x; s <= mask; s += blockDim.x)
      if (tk[s] != kNoKey) C.pair(C.endpoint(tk[s]), C.end2(tk[s]), tc[s]);
    __syncthreads();
  }
}

__global__ void gather_keys_kernel(const uint64_t* __restrict__ keys, const uint32_t* __restrict__ perm, int64_t n,
                                   uint64_t* out) {
  for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x)
    out[q] = keys[perm[q]];
}

__global__ void widen_kernel(const uint32_t* __restrict__ in, int64_t n, int64_t* out) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    out[i] = (int64_t)in[i];
}

// One warp per chunk of wedges, all of them resident at most eight times over.
int materialize_grid(int64_t cnt) {
  return std::max(1, std::min(ceil_div(cnt, (int64_t)kChunk * 8), sm_count() * 32));
}

int grid_for(int64_t n) { return std::max(1, std::min(ceil_div(n, 256), sm_count() * 16)); }

int bits_for(uint64_t x) {
  int b = 0;
  while (b < 64 && (x >> b) != 0) ++b;
  return b;
}

}  // namespace

CountResult count_ranked_materialized(const Ranked& R, int per, int64_t* out, bool hist, int64_t max_wedges,
                                      cudaStream_t s) {
  CountResult res;
  const int64_t n = R.n, m2 = R.m2;
  const int64_t out_len = per == VERT ? n : (per == EDGE ? m2 / 2 : 1);
  if (out_len > 0) PB_CUDA_TRY(cudaMemsetAsync(out, 0, sizeof(int64_t) * out_len, s));
  if (n == 0 || R.w_rank == 0) return res;
  cudaEvent_t e0, e1;
  PB_CUDA_TRY(cudaEventCreate(&e0));
  PB_CUDA_TRY(cudaEventCreate(&e1));
  PB_CUDA_TRY(cudaEventRecord(e0, s));
  // Per-slot exclusive wedge prefix (the flattened wedge index of each slot's first wedge).
  DevBuf<int64_t> spre(m2 + 1, s);
  const uint32_t* rowid = R.rowid.get();
  exclusive_scan_u32_i64(R.pref.get(), spre.get(), m2, s);
  // Batch budget: -m, capped so that one batch's arrays stay within a few GiB.
  const int64_t cap = std::min<int64_t>(max_wedges > 0 ? max_wedges : (int64_t)1 << 27, (int64_t)1 << 27);
  // Endpoint wedge prefix on the host, to cut batches at endpoint boundaries (one batch: its ends).
  const bool one_batch = R.w_rank <= cap;
  std::vector<int64_t> wsum;
  if (!one_batch) {
    wsum.resize(n + 1);
    PB_CUDA_TRY(cudaMemcpyAsync(wsum.data(), R.wsum.get(), sizeof(int64_t) * (n + 1), cudaMemcpyDeviceToHost, s));
    PB_CUDA_TRY(cudaStreamSynchronize(s));
  }
  const int ubits = std::max(1, bits_for((uint64_t)(n - 1)));
  const uint64_t md = R.max_deg > 0 ? R.max_deg - 1 : 0;
  DevBuf<uint32_t> out32;
  if (per == EDGE && md * md < (1ull << 32)) {
    out32.alloc(out_len, s);
    PB_CUDA_TRY(cudaMemsetAsync(out32.get(), 0, out32.bytes(), s));
  }
  DevBuf<unsigned long long> total(1, s);
  PB_CUDA_TRY(cudaMemsetAsync(total.get(), 0, sizeof(unsigned long long), s));
  // SORT on keys of one width: sorted runs give the multiplicities.
  auto sort_batch = [&](auto* keys, auto* keys2, int64_t cnt, int64_t tb, int key_bits, const Credit& C) {
    using K = std::remove_pointer_t<decltype(keys)>;
    DevBuf<uint32_t> vals(cnt, s), vals2(cnt, s), jarr(cnt, s), s2arr(cnt, s);
    PB_LAUNCH(materialize_kernel<K>, materialize_grid(cnt), 256, 0, s, R.off.get(), R.adj.get(), R.pref.get(),
              spre.get(), rowid, m2, tb, tb + cnt, C.i0, ubits, keys, vals.get(), jarr.get(), s2arr.get());
    bool alt;
    if constexpr (sizeof(K) == 4) alt = radix_sort_pairs_u32(keys, vals.get(), keys2, vals2.get(), cnt, 0, key_bits, s);
    else alt = radix_sort_pairs_u64(keys, vals.get(), keys2, vals2.get(), cnt, 0, key_bits, s);
    K* k = alt ? keys2 : keys;
    uint32_t* v = alt ? vals2.get() : vals.get();
    DevBuf<uint32_t> head(cnt, s), rid(cnt + 1, s), start(cnt + 1, s);
    PB_LAUNCH(run_heads_kernel<K>, grid_for(cnt), 256, 0, s, k, cnt, head.get());
    exclusive_scan_u32(head.get(), rid.get(), cnt, s);
    PB_LAUNCH(run_starts_kernel, grid_for(cnt), 256, 0, s, head.get(), rid.get(), cnt, start.get());
    PB_LAUNCH(sort_credit_kernel<K>, grid_for(cnt), 256, 0, s, k, v, jarr.get(), s2arr.get(), head.get(), rid.get(),
              start.get(), cnt, C);
  };
  int64_t i0 = 0;
  while (i0 < n) {
    // Largest i1 with wsum[i1] - wsum[i0] <= cap (at least one endpoint).
    int64_t i1 = n;
    if (!one_batch) {
      i1 = std::upper_bound(wsum.begin() + i0 + 1, wsum.end(), wsum[i0] + cap) - wsum.begin() - 1;
      if (i1 <= i0) i1 = i0 + 1;
    }
    const int64_t tb = one_batch ? 0 : wsum[i0], te = one_batch ? R.w_rank : wsum[i1], cnt = te - tb;
    PB_REQUIRE(cnt < (int64_t)UINT32_MAX, PB_ETOOBIG, "a single endpoint's wedges exceed 2^32");
    if (cnt > 0) {
      Credit C{R.off.get(), R.adj.get(), R.eout.get(), per, (uint32_t)i0, ubits, out, out32.get(), total.get()};
      const int key_bits = ubits + bits_for((uint64_t)(i1 - i0 - 1));
      if (!hist && key_bits <= 32) {
        DevBuf<uint32_t> keys(cnt, s), keys2(cnt, s);
        sort_batch(keys.get(), keys2.get(), cnt, tb, key_bits, C);
      } else if (!hist) {
        DevBuf<uint64_t> keys(cnt, s), keys2(cnt, s);
        sort_batch(keys.get(), keys2.get(), cnt, tb, key_bits, C);
      } else {
        DevBuf<uint64_t> keys(cnt, s), keys2(cnt, s);
        DevBuf<uint32_t> vals(cnt, s), jarr(cnt, s), s2arr(cnt, s);
        PB_LAUNCH(materialize_kernel<uint64_t>, materialize_grid(cnt), 256, 0, s, R.off.get(), R.adj.get(),
                  R.pref.get(), spre.get(), rowid, m2, tb, te, (uint32_t)i0, ubits, keys.get(), vals.get(),
                  jarr.get(), s2arr.get());
        // Semisort: bucket keys by hash (about 1024 wedges per bucket), one stable radix pass.
        int bits = bits_for((uint64_t)std::max<int64_t>(1, cnt / 1024));
        bits = std::max(1, std::min(bits, 24));
        const uint32_t nb = 1u << bits;
        DevBuf<uint32_t> bkey(cnt, s), bkey2(cnt, s), perm2(cnt, s);
        PB_LAUNCH(bucket_keys_kernel, grid_for(cnt), 256, 0, s, keys.get(), cnt, bits, bkey.get());
        // sort (bucket, original position) pairs; positions double as the permutation
        const bool alt = radix_sort_pairs_u32(bkey.get(), vals.get(), bkey2.get(), perm2.get(), cnt, 0, bits, s);
        uint32_t* bs = alt ? bkey2.get() : bkey.get();
        uint32_t* pm = alt ? perm2.get() : vals.get();
        DevBuf<uint32_t> bstart(nb + 1, s);
        PB_LAUNCH(bucket_bounds_kernel, grid_for(cnt), 256, 0, s, bs, cnt, nb, bstart.get());
        // gather keys into bucket order
        DevBuf<uint32_t> overflow(nb + 1, s);
        PB_CUDA_TRY(cudaMemsetAsync(overflow.get(), 0, sizeof(uint32_t), s));
        PB_LAUNCH(gather_keys_kernel, grid_for(cnt), 256, 0, s, keys.get(), pm, cnt, keys2.get());
        PB_LAUNCH(hist_bucket_kernel, std::min<int>(nb, sm_count() * 8), kHistThreads, 0, s, keys2.get(), pm,
                  jarr.get(), s2arr.get(), bstart.get(), nb, C, overflow.get());
        uint32_t nover = 0;
        PB_CUDA_TRY(cudaMemcpyAsync(&nover, overflow.get(), sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
        PB_CUDA_TRY(cudaStreamSynchronize(s));
        if (nover) {
          DevBuf<unsigned long long> gk(4 * cnt + 64, s);
          DevBuf<uint32_t> gc(4 * cnt + 64, s);
          PB_LAUNCH(hist_global_kernel, std::min<int>(nover, sm_count() * 4), 512, 0, s, keys2.get(), pm, jarr.get(),
                    s2arr.get(), bstart.get(), overflow.get(), gk.get(), gc.get(), C);
        }
        PB_CUDA_TRY(cudaStreamSynchronize(s));
      }
    }
    i0 = i1;
  }
  if (per == TOTAL)
    PB_CUDA_TRY(cudaMemcpyAsync(out, total.get(), sizeof(int64_t), cudaMemcpyDeviceToDevice, s));
  if (out32.get()) PB_LAUNCH(widen_kernel, grid_for(out_len), 256, 0, s, out32.get(), out_len, out);
  PB_CUDA_TRY(cudaEventRecord(e1, s));
  PB_CUDA_TRY(cudaEventSynchronize(e1));
  float ms = 0;
  PB_CUDA_TRY(cudaEventElapsedTime(&ms, e0, e1));
  res.agg_ms = ms;
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  return res;
}

}  // namespace pb
