// Group-by and aggregation operators for sm_100a.
//
// Reference: code/group/test_group_option.cpp — vector_group (:44-60) adds
// m1[i] + m2[i] into group_vector[vecInx[i] - 1] (1-based group ids, int
// counters) and returns the int64 sum of the groups; hashtable_group (:71-88)
// does the same through std::unordered_map<int, int> keyed by vecInx[i] - 1.  Here
// sums and counts are int64.  code/aggregation/test_aggregation_option.cpp — aggalgo_*
// (:28-107) sums price*qty*tax + price*qty in double; here the same expression
// in int64 fixed point (tax in hundredths: sum of price*qty*(100 + tax),
// exactly 100x the decimal value) and, for parity with the double code, a
// deterministic double variant.
//
// Dense group-by accumulates per block in shared memory when the group vector
// fits (exact 64-bit sums from 32-bit shared atomics), else in L2 with 64-bit
// atomics.  Hash group-by aggregates in shared-memory tables: per block when
// every distinct key fits one table, else per partition of the key hash
// (see the plans below).
#include <algorithm>
#include <cstring>
#include <type_traits>

#include "compact.cuh"

namespace olap {

constexpr int kGroupThreads = 512;
constexpr int32_t kEmptyKey = INT32_MIN;

__host__ __device__ __forceinline__ uint32_t mix32(uint32_t x) {
  x ^= x >> 16;
  x *= 0x7feb352du;
  x ^= x >> 15;
  x *= 0x846ca68bu;
  x ^= x >> 16;
  return x;
}

// Dense: group_vector[vecInx[i] - 1] += m1[i] + m2[i]; counts optional.
template <bool SMEM>
__global__ void __launch_bounds__(kGroupThreads) group_vector_kernel(
    int64_t n, const int32_t* __restrict__ idx, const int32_t* __restrict__ m1, const int32_t* __restrict__ m2,
    int64_t G, unsigned long long* __restrict__ sums, unsigned long long* __restrict__ counts,
    unsigned long long* total, unsigned long long* range_err) {
  extern __shared__ unsigned long long sacc[];  // [G] sums, then [G] counts
  const int tid = threadIdx.x;
  const bool want_counts = counts != nullptr;
  if (SMEM) {
    for (int64_t i = tid; i < G * (want_counts ? 2 : 1); i += blockDim.x) sacc[i] = 0;
    __syncthreads();
  }
  const uint64_t pol = policy_evict_first();
  int64_t tot = 0;
  unsigned int bad = 0;
  auto add = [&](int32_t gi, int32_t a, int32_t b) {
    const int64_t g = static_cast<int64_t>(gi) - 1;
    if (g < 0 || g >= G) {
      ++bad;
      return;
    }
    const int64_t v = static_cast<int64_t>(a) + b;
    tot += v;
    if (SMEM) {
      smem_add_u64(&sacc[g], static_cast<uint64_t>(v));
      if (want_counts) atomicAdd(reinterpret_cast<unsigned int*>(&sacc[G + g]), 1u);
    } else {
      atomicAdd(&sums[g], static_cast<unsigned long long>(v));
      if (want_counts) atomicAdd(&counts[g], 1ull);
    }
  };
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  const int64_t t0 = static_cast<int64_t>(blockIdx.x) * blockDim.x + tid;
  const bool vec = ((reinterpret_cast<uintptr_t>(idx) | reinterpret_cast<uintptr_t>(m1) |
                     reinterpret_cast<uintptr_t>(m2)) & 15) == 0;
  const int64_t n4 = vec ? n >> 2 : 0;
  for (int64_t i = t0; i < n4; i += stride) {
    const int4 g = ld_stream_v4(idx + 4 * i, pol), a = ld_stream_v4(m1 + 4 * i, pol), b = ld_stream_v4(m2 + 4 * i, pol);
    add(g.x, a.x, b.x);
    add(g.y, a.y, b.y);
    add(g.z, a.z, b.z);
    add(g.w, a.w, b.w);
  }
  for (int64_t r = 4 * n4 + t0; r < n; r += stride) add(idx[r], m1[r], m2[r]);
  tot = warp_sum_i64(tot);
  const unsigned int wbad = __reduce_add_sync(0xffffffffu, bad);
  if ((tid & 31) == 0) {
    if (tot) atomicAdd(total, static_cast<unsigned long long>(tot));
    if (wbad) atomicAdd(range_err, static_cast<unsigned long long>(wbad));
  }
  if (SMEM) {
    __syncthreads();
    for (int64_t i = tid; i < G; i += blockDim.x) {
      if (sacc[i]) atomicAdd(&sums[i], sacc[i]);
      if (want_counts) {
        const unsigned int c = static_cast<unsigned int>(sacc[G + i]);
        if (c) atomicAdd(&counts[i], static_cast<unsigned long long>(c));
      }
    }
  }
}

// Global hash table of the hash group-by: keys[cap] (kEmptyKey = free),
// sums[cap], counts[cap].
struct HashAgg {
  int32_t* keys;
  unsigned long long* sums;
  unsigned long long* counts;
  uint64_t mask;
  unsigned long long* overflow;
};

__device__ __forceinline__ void global_add(const HashAgg& t, int32_t k, uint64_t s, uint64_t c) {
  uint64_t h = mix32(static_cast<uint32_t>(k)) & t.mask;
  for (uint64_t step = 0; step <= t.mask; ++step) {
    const int32_t prev = atomicCAS(t.keys + h, kEmptyKey, k);
    if (prev == kEmptyKey || prev == k) {
      if (s) atomicAdd(t.sums + h, static_cast<unsigned long long>(s));
      atomicAdd(t.counts + h, static_cast<unsigned long long>(c));
      return;
    }
    h = (h + 1) & t.mask;
  }
  atomicAdd(t.overflow, 1ull);
}

// ---- hash group-by --------------------------------------------------------
//
// Two plans, chosen by the capacity (a power of two >= 2 x the distinct keys):
//  * capacity <= kAggSlots: every block keeps a shared-memory table of at
//    least `capacity` slots, so each distinct key stays in shared memory; blocks
//    flush their tables into the global table once, and the occupied slots
//    are compacted into the outputs.  One read of the columns.
//  * larger: the rows are partitioned by the key hash into P partitions, whole
//    waves of one block per SM, with so few distinct keys each that they fill
//    at most about a quarter of a shared table (a histogram pass, a scan of
//    the partition offsets, a scatter pass); then one block per partition
//    aggregates it in a shared table of 8,192 or 14,336 slots and writes its
//    groups straight to the outputs.
// Optionally (OLAP_TUNE_GROUP_COMBINE) a warp first combines its rows that
// share a key (match_any plus two 32-bit reductions of the split values), so
// each distinct key of a warp costs one shared-table update.

constexpr int kAggThreads = 1024;
constexpr int kAggSlots = 8192;  // 16 B per slot: 128 KB of shared memory
constexpr int kAggMaxSlots = 14336;  // 224 KB: the partitions' tables of many groups
static_assert(kAggSlots % kAggThreads == 0 && kAggMaxSlots % kAggThreads == 0, "whole merge blocks");

struct SmemAgg {
  int32_t* key;
  unsigned int* cnt;
  uint32_t* lo;     // low words of the 64-bit sums (signed); the high words follow at lo + slots
  uint32_t slots;   // a multiple of 4
  uint32_t nb;      // buckets of 4 slots (any count, so a table can fill the shared memory)

  // Home bucket of key k: the low 16 hash bits scaled to [0, nb) (plan 2's
  // partitions take the high bits); probing wraps after the last bucket.
  __device__ __forceinline__ uint32_t home(int32_t k) const {
    return __umulhi(mix32(static_cast<uint32_t>(k)) << 16, nb);
  }
  __device__ __forceinline__ uint32_t next(uint32_t b) const { return b + 1 == nb ? 0u : b + 1; }
  __device__ __forceinline__ uint64_t sum(uint32_t i) const {
    return (static_cast<uint64_t>(lo[slots + i]) << 32) + static_cast<uint64_t>(static_cast<int64_t>(static_cast<int32_t>(lo[i])));
  }
};

// What adding v to a slot's signed low word adds to its high word: v's own
// high part, and one for a signed overflow of the low word (rare, so values of
// both signs seldom touch the high word).
__device__ __forceinline__ int32_t agg_high(uint32_t old, int32_t v) {
  const int32_t o = static_cast<int32_t>(old), r = static_cast<int32_t>(old + static_cast<uint32_t>(v));
  return ((o ^ r) & (v ^ r)) < 0 ? (v < 0 ? -1 : 1) : 0;
}
__device__ __forceinline__ int32_t agg_high(uint32_t old, int64_t v) {
  const int32_t l = static_cast<int32_t>(v);
  return static_cast<int32_t>((v - l) >> 32) + agg_high(old, l);
}

__device__ __forceinline__ SmemAgg smem_agg(unsigned char* base, uint32_t slots) {
  SmemAgg t;
  t.lo = reinterpret_cast<uint32_t*>(base);
  t.key = reinterpret_cast<int32_t*>(t.lo + 2 * slots);
  t.cnt = reinterpret_cast<unsigned int*>(t.key + slots);
  t.slots = slots;
  t.nb = slots >> 2;
  return t;
}

__device__ __forceinline__ void smem_agg_clear(const SmemAgg& t) {
  for (uint32_t i = threadIdx.x; i < t.slots; i += blockDim.x) {
    t.key[i] = kEmptyKey;
    t.cnt[i] = 0;
    t.lo[i] = 0;
    t.lo[t.slots + i] = 0;
  }
}

__device__ __forceinline__ int4 lds_volatile_v4(const int32_t* p) {
  int4 v;
  const unsigned a = static_cast<unsigned>(__cvta_generic_to_shared(p));
  asm volatile("ld.volatile.shared.v4.s32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
  return v;
}

// Adds (s, c) to key k's slot; false when the table has no room for k.
// Buckets of 4 slots, probed linearly: one 16-byte read finds k or the first
// free slot of a bucket, which keeps the probe loops of a warp short at low
// load.  Keys are never removed, so a key lives in the first bucket that had
// a free slot when it was inserted, and a thread that loses a slot's CAS to
// the same key uses that slot.  Returns k's slot from the bucket run starting
// at b, inserting k when absent (volatile reads: other threads insert
// concurrently); -1 when the table has no room for k.
__device__ __forceinline__ int smem_find_insert(const SmemAgg& t, int32_t k, uint32_t b) {
  for (uint32_t step = 0; step < t.nb; ++step) {
    const int4 q = lds_volatile_v4(t.key + 4 * b);
    int slot = q.x == k ? 0 : q.y == k ? 1 : q.z == k ? 2 : q.w == k ? 3 : -1;
    if (slot < 0 && (q.x == kEmptyKey || q.y == kEmptyKey || q.z == kEmptyKey || q.w == kEmptyKey)) {
      // k is new to this bucket and it has room: claim the first free slot,
      // starting at another slot every 8 buckets.  Most buckets hold one or
      // two keys; with all of those in their first slots the sums and counts
      // of a warp's rows fell on 8 to 16 of the 32 banks (5.3 passes per
      // atomic instead of 3.5).
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int j = i ^ static_cast<int>((b >> 3) & 3u);
        const int32_t cur = j == 0 ? q.x : j == 1 ? q.y : j == 2 ? q.z : q.w;
        if (slot < 0 && cur == kEmptyKey) {
          const int32_t prev = atomicCAS(t.key + 4 * b + j, kEmptyKey, k);
          if (prev == kEmptyKey || prev == k) slot = j;
        }
      }
    }
    if (slot >= 0) return static_cast<int>(4 * b) + slot;
    b = t.next(b);
  }
  return -1;
}

// Adds (s, c) to key k's slot; false when the table has no room for k.
__device__ __forceinline__ bool smem_agg_add(const SmemAgg& t, int32_t k, uint64_t s, uint32_t c) {
  const int i = smem_find_insert(t, k, t.home(k));
  if (i < 0) return false;
  const uint32_t old = atomicAdd(t.lo + i, static_cast<uint32_t>(s));
  const int32_t h = agg_high(old, static_cast<int64_t>(s));
  if (h) atomicAdd(t.lo + t.slots + i, static_cast<uint32_t>(h));
  atomicAdd(t.cnt + i, c);
  return true;
}

// Warp combine of the rows that share a key: returns true on the lane that
// carries its key's (sum, count) for this warp step.  v lies in [-2^32, 2^32):
// v + 2^32 splits into 24 low and 9 high bits, whose 32-bit sums over at most
// 32 lanes cannot overflow.
__device__ __forceinline__ bool warp_combine(bool valid, int32_t k, int64_t v, int64_t* gs, uint32_t* gc) {
  const int lane = threadIdx.x & 31;
  const unsigned long long tag = valid ? static_cast<unsigned long long>(static_cast<uint32_t>(k))
                                       : (0x100000000ull | static_cast<unsigned long long>(lane));
  const unsigned int m = __match_any_sync(0xffffffffu, tag);
  if (__all_sync(0xffffffffu, (m & (m - 1)) == 0)) {  // no key repeats in this warp step
    *gs = v;
    *gc = 1;
    return valid;
  }
  if (!valid) return false;
  const uint64_t u = static_cast<uint64_t>(v + (int64_t(1) << 32));
  const uint32_t lo = __reduce_add_sync(m, static_cast<uint32_t>(u & 0xffffffu));
  const uint32_t hi = __reduce_add_sync(m, static_cast<uint32_t>(u >> 24));
  const uint32_t c = __popc(m);
  *gs = (static_cast<int64_t>(hi) << 24) + static_cast<int64_t>(lo) - (static_cast<int64_t>(c) << 32);
  *gc = c;
  return lane == __ffs(m) - 1;
}

__device__ __forceinline__ int32_t agg_key(int32_t key, int32_t key_offset) {
  return static_cast<int32_t>(static_cast<uint32_t>(key) + static_cast<uint32_t>(key_offset));
}

// Rows [b, e) of the columns, 4 per thread per step (16-byte loads when
// aligned), handed to f(valid, row, key, value) by every lane of the warp.
template <class F>
__device__ __forceinline__ void agg_rows(int64_t b, int64_t e, int64_t t0, int64_t stride, const int32_t* keys,
                                         const int32_t* vals, const int32_t* vals2, bool vec, F&& f) {
  const uint64_t pol = policy_evict_first();
  const int32_t* v2 = vals2 ? vals2 : vals;  // a valid address even where the guarded load is hoisted
  const int64_t b4 = vec ? (b + 3) & ~int64_t(3) : e;  // first aligned row
  const int64_t head = b4 < e ? b4 : e;
  // head rows one by one (at most 3), then groups of 4, then the tail
  for (int64_t base = b; base < head; base += stride) {
    const int64_t r = base + t0;
    const bool ok = r < head;
    f(ok, ok ? keys[r] : 0, ok ? static_cast<int64_t>(vals[r]) + (vals2 ? vals2[r] : 0) : 0);
  }
  const int64_t n4 = (e - head) >> 2;
  for (int64_t base = 0; base < n4; base += 2 * stride) {
    // two groups of 4 rows per thread in flight before either is used
    int4 k[2], v[2], w[2];
    bool ok[2];
#pragma unroll
    for (int g = 0; g < 2; ++g) {
      const int64_t i = base + g * stride + t0;
      ok[g] = i < n4;
      k[g] = make_int4(0, 0, 0, 0);
      v[g] = k[g];
      w[g] = k[g];
      if (ok[g]) {
        k[g] = ld_stream_v4(keys + head + 4 * i, pol);
        v[g] = ld_stream_v4(vals + head + 4 * i, pol);
        if (vals2) w[g] = ld_stream_v4(v2 + head + 4 * i, pol);
      }
    }
#pragma unroll
    for (int g = 0; g < 2; ++g) {
      f(ok[g], k[g].x, static_cast<int64_t>(v[g].x) + w[g].x);
      f(ok[g], k[g].y, static_cast<int64_t>(v[g].y) + w[g].y);
      f(ok[g], k[g].z, static_cast<int64_t>(v[g].z) + w[g].z);
      f(ok[g], k[g].w, static_cast<int64_t>(v[g].w) + w[g].w);
    }
  }
  for (int64_t base = head + 4 * n4; base < e; base += stride) {
    const int64_t r = base + t0;
    const bool ok = r < e;
    f(ok, ok ? keys[r] : 0, ok ? static_cast<int64_t>(vals[r]) + (vals2 ? vals2[r] : 0) : 0);
  }
}

// Plan 1: shared tables of `slots` = capacity slots per block, flushed into
// the global table.
__global__ void __launch_bounds__(kAggThreads) group_hash_smem_kernel(int64_t n, const int32_t* __restrict__ keys,
                                                                      int32_t key_offset,
                                                                      const int32_t* __restrict__ vals,
                                                                      const int32_t* __restrict__ vals2,
                                                                      uint32_t slots, int combine, HashAgg t,
                                                                      unsigned long long* range_err) {
  extern __shared__ __align__(16) unsigned char agg_smem[];
  const SmemAgg st = smem_agg(agg_smem, slots);
  smem_agg_clear(st);
  __syncthreads();
  const bool vec = ((reinterpret_cast<uintptr_t>(keys) | reinterpret_cast<uintptr_t>(vals) |
                     reinterpret_cast<uintptr_t>(vals2)) & 15) == 0;
  // each block takes a contiguous share of the rows
  const int64_t per = ((n + gridDim.x - 1) / gridDim.x + 3) & ~int64_t(3);
  const int64_t b = static_cast<int64_t>(blockIdx.x) * per;
  const int64_t e = b + per < n ? b + per : n;
  unsigned int bad = 0;
  if (b < e)
    agg_rows(b, e, threadIdx.x, blockDim.x, keys, vals, vals2, vec, [&](bool ok, int32_t key, int64_t v) {
      const int32_t k = agg_key(key, key_offset);
      if (ok && k == kEmptyKey) {  // reserved as the empty marker
        ++bad;
        ok = false;
      }
      int64_t gs = v;
      uint32_t gc = 1;
      if (combine ? warp_combine(ok, k, v, &gs, &gc) : ok)
        if (!smem_agg_add(st, k, static_cast<uint64_t>(gs), gc)) global_add(t, k, static_cast<uint64_t>(gs), gc);
    });
  const unsigned int wbad = __reduce_add_sync(0xffffffffu, bad);
  if ((threadIdx.x & 31) == 0 && wbad) atomicAdd(range_err, static_cast<unsigned long long>(wbad));
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < slots; i += blockDim.x)
    if (st.key[i] != kEmptyKey) global_add(t, st.key[i], st.sum(i), st.cnt[i]);
}

// ---- batched shared-table updates -------------------------------------------
// R rows (count 1 each) into the shared table, with every step of the R rows
// issued together: the R home buckets are read first (plain loads: a stale
// read can only miss a key, since keys are never removed, and a miss takes
// the volatile insert path), then the R low-word adds whose old values tell
// an overflow, the R count adds, and the high words where one is needed.  Only
// 32-bit shared atomics: on B200 a 64-bit shared atomicAdd runs several times
// slower than a 32-bit one.  V: int32_t, or int64_t for values of 33 bits.
// kAll: every row is valid.  `sync`: the lanes of the warp that call together
// (0 when the callers are not warp-uniform); they are brought back together
// after the insert path, whose probe loop ends at a different step on each
// lane (left diverged, the warp would run all later steps once per lane
// group).  Returns the mask of the rows that found no room (the caller adds
// them elsewhere).
template <int R, bool kAll, class V>
__device__ __forceinline__ uint32_t smem_agg_rows(const SmemAgg& t, const int32_t (&k)[R], const V (&v)[R],
                                                  uint32_t valid, uint32_t sync) {
  uint32_t b[R];
  int4 q[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    b[r] = 4 * t.home(k[r]);
    q[r] = *reinterpret_cast<const int4*>(t.key + b[r]);
  }
  int s[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    s[r] = -1;
    if (q[r].x == k[r]) s[r] = b[r];
    if (q[r].y == k[r]) s[r] = b[r] + 1;
    if (q[r].z == k[r]) s[r] = b[r] + 2;
    if (q[r].w == k[r]) s[r] = b[r] + 3;
    if (!kAll && !((valid >> r) & 1u)) s[r] = -2;
  }
  uint32_t lost = 0;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    if (s[r] == -1) {
      s[r] = smem_find_insert(t, k[r], b[r] >> 2);
      if (s[r] < 0) lost |= 1u << r;
    }
  }
  if (sync) __syncwarp(sync);
  uint32_t old[R];
#pragma unroll
  for (int r = 0; r < R; ++r)
    old[r] = s[r] >= 0 ? atomicAdd(t.lo + s[r], static_cast<uint32_t>(v[r])) : 0u;
#pragma unroll
  for (int r = 0; r < R; ++r)
    if (s[r] >= 0) atomicAdd(t.cnt + s[r], 1u);
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int32_t h = agg_high(old[r], v[r]);
    if (h && s[r] >= 0) atomicAdd(t.lo + t.slots + s[r], static_cast<uint32_t>(h));
  }
  return lost;
}

constexpr int kRowsThreads = 1024;

// Plan 1 with batched updates: each block aggregates a contiguous share of
// the rows in a `slots`-slot shared table, 4 rows per thread step with the
// next step's columns already loading (software pipelined), then adds its
// slots to the global table; a row whose key finds no room goes to the
// global table directly.
template <bool HAS2>
__global__ void __launch_bounds__(kRowsThreads) group_hash_rows_kernel(int64_t n, const int32_t* __restrict__ keys,
                                                                       int32_t key_offset,
                                                                       const int32_t* __restrict__ vals,
                                                                       const int32_t* __restrict__ vals2,
                                                                       uint32_t slots, HashAgg g,
                                                                       unsigned long long* range_err) {
  extern __shared__ __align__(16) unsigned char agg_smem[];
  const SmemAgg t = smem_agg(agg_smem, slots);
  smem_agg_clear(t);
  __syncthreads();
  const bool vec = ((reinterpret_cast<uintptr_t>(keys) | reinterpret_cast<uintptr_t>(vals) |
                     (HAS2 ? reinterpret_cast<uintptr_t>(vals2) : 0)) & 15) == 0;
  const int64_t per = ((n + gridDim.x - 1) / gridDim.x + 3) & ~int64_t(3);
  const int64_t b = static_cast<int64_t>(blockIdx.x) * per;
  const int64_t e = b + per < n ? b + per : n;
  const uint64_t pol = policy_evict_first();
  unsigned int bad = 0;
  using V = std::conditional_t<HAS2, int64_t, int32_t>;
  auto rows = [&](auto all, const int4 kk, const int4 a, const int4 c, uint32_t valid, uint32_t sync) {
    const int32_t kr[4] = {kk.x, kk.y, kk.z, kk.w}, ar[4] = {a.x, a.y, a.z, a.w}, cr[4] = {c.x, c.y, c.z, c.w};
    int32_t k[4];
    V v[4];
    bool none = false;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      k[u] = agg_key(kr[u], key_offset);
      v[u] = static_cast<V>(ar[u]) + (HAS2 ? cr[u] : 0);
      none |= k[u] == kEmptyKey;
    }
    // reserved as the empty marker (rare): not valid rows
    if (none) {
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (((valid >> u) & 1u) && k[u] == kEmptyKey) {
          ++bad;
          valid &= ~(1u << u);
        }
      }
    }
    const uint32_t lost = (decltype(all)::value && __all_sync(0xffffffffu, valid == 0xFu))
                              ? smem_agg_rows<4, true>(t, k, v, 0xFu, sync)
                              : smem_agg_rows<4, false>(t, k, v, valid, sync);
    if (lost) {  // rare: keys that found no room in the table
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if ((lost >> u) & 1u) global_add(g, k[u], static_cast<uint64_t>(static_cast<int64_t>(v[u])), 1);
    }
  };
  auto one = [&](int64_t r) {
    rows(std::false_type{}, make_int4(keys[r], 0, 0, 0), make_int4(vals[r], 0, 0, 0),
         make_int4(HAS2 ? vals2[r] : 0, 0, 0, 0), 1u, 0u);
  };
  if (b < e) {
    const int64_t b4 = (b + 3) & ~int64_t(3);
    const int64_t head = vec ? (b4 < e ? b4 : e) : e;
    const int64_t n4 = (e - head) >> 2;
    // rows before the first aligned one, and all rows when unaligned: one at a time
    for (int64_t r = b + threadIdx.x; r < head; r += blockDim.x) one(r);
    const int32_t* kp = keys + head;
    const int32_t* ap = vals + head;
    const int32_t* cp = HAS2 ? vals2 + head : vals + head;
    // Every lane of a warp runs the same steps (a lane past the end has no
    // rows in its last one), so the table updates can bring the warp back
    // together.
    const int64_t lane = threadIdx.x & 31;
    const int64_t w0 = static_cast<int64_t>(threadIdx.x) - lane;
    int4 kk = make_int4(0, 0, 0, 0), a = kk, c = kk;
    if (w0 + lane < n4) {
      kk = ld_stream_v4(kp + 4 * (w0 + lane), pol);
      a = ld_stream_v4(ap + 4 * (w0 + lane), pol);
      if (HAS2) c = ld_stream_v4(cp + 4 * (w0 + lane), pol);
    }
    for (int64_t i0 = w0; i0 < n4; i0 += blockDim.x) {
      // the next step's columns load while this step's rows update the table
      const int64_t i = i0 + lane, nx = i + blockDim.x;
      int4 kn = make_int4(0, 0, 0, 0), an = kn, cn = kn;
      if (nx < n4) {
        kn = ld_stream_v4(kp + 4 * nx, pol);
        an = ld_stream_v4(ap + 4 * nx, pol);
        if (HAS2) cn = ld_stream_v4(cp + 4 * nx, pol);
      }
      rows(std::true_type{}, kk, a, c, i < n4 ? 0xFu : 0u, 0xffffffffu);
      kk = kn;
      a = an;
      c = cn;
    }
    for (int64_t r = head + 4 * n4 + threadIdx.x; r < e; r += blockDim.x) one(r);
  }
  const unsigned int wbad = __reduce_add_sync(0xffffffffu, bad);
  if ((threadIdx.x & 31) == 0 && wbad) atomicAdd(range_err, static_cast<unsigned long long>(wbad));
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < slots; i += blockDim.x)
    if (t.key[i] != kEmptyKey && t.cnt[i]) global_add(g, t.key[i], t.sum(i), t.cnt[i]);
}

// Plan 2.  Partition of a key: its hash scaled onto the partitions (the shared
// tables index with the low bits).
__device__ __forceinline__ uint32_t agg_part(int32_t k, int n_parts) {
  return __umulhi(mix32(static_cast<uint32_t>(k)), static_cast<uint32_t>(n_parts));
}

struct PartPlan {
  int64_t n;
  int64_t per;        // rows per block of the histogram and scatter passes (multiple of 4)
  int32_t n_blocks;   // blocks of those passes
  int32_t n_parts;    // P
  uint32_t slots;     // slots of a partition's shared table
  int32_t key_offset;
};

// Per block and partition: rows of the block's share in the partition,
// hist[b * P + p]; the partition totals are summed into ptot[p].
__global__ void __launch_bounds__(1024) group_part_hist_kernel(PartPlan pp, const int32_t* __restrict__ keys,
                                                               unsigned int* __restrict__ hist,
                                                               unsigned long long* __restrict__ ptot,
                                                               unsigned long long* range_err) {
  extern __shared__ unsigned int s_hist[];
  for (int p = threadIdx.x; p < pp.n_parts; p += blockDim.x) s_hist[p] = 0;
  __syncthreads();
  const int64_t b = static_cast<int64_t>(blockIdx.x) * pp.per;
  const int64_t e = b + pp.per < pp.n ? b + pp.per : pp.n;
  const uint64_t pol = policy_evict_first();
  const bool vec = (reinterpret_cast<uintptr_t>(keys) & 15) == 0;
  unsigned int bad = 0;
  auto one = [&](int32_t key) {
    const int32_t k = agg_key(key, pp.key_offset);
    if (k == kEmptyKey) {
      ++bad;
      return;
    }
    atomicAdd(&s_hist[agg_part(k, pp.n_parts)], 1u);
  };
  int64_t done = b;  // four 16-byte loads per thread in flight
  if (vec) {
    const int64_t step = 16 * static_cast<int64_t>(blockDim.x);
    for (; done + step <= e; done += step) {
      int4 k[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) k[u] = ld_stream_v4_ordered(keys + done + 4 * (threadIdx.x + u * static_cast<int64_t>(blockDim.x)), pol);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        one(k[u].x);
        one(k[u].y);
        one(k[u].z);
        one(k[u].w);
      }
    }
  }
  for (int64_t r = done + threadIdx.x; r < e; r += blockDim.x) one(keys[r]);
  const unsigned int wbad = __reduce_add_sync(0xffffffffu, bad);
  if ((threadIdx.x & 31) == 0 && wbad) atomicAdd(range_err, static_cast<unsigned long long>(wbad));
  __syncthreads();
  for (int p = threadIdx.x; p < pp.n_parts; p += blockDim.x) {
    const unsigned int c = s_hist[p];
    hist[static_cast<int64_t>(blockIdx.x) * pp.n_parts + p] = c;
    if (c) atomicAdd(&ptot[p], static_cast<unsigned long long>(c));
  }
}

// A slice of a partition too large for one block: its table is written whole
// to the partial table of the slice's number, and group_part_merge_kernel adds
// the tables of a partition's slices up.
constexpr int kMaxPartials = 256;  // slices, and partial tables
struct AggSlice {
  long long begin, end;
};
struct AggUnits {
  int2 merge[kMaxPartials];       // per split partition: its first slice and their number
  AggSlice slice[kMaxPartials];
  long long limit;                // rows of a partition up to which one block takes it whole
  int n_slices, n_merges;
};

// Exclusive scan over the block's 1,024 threads; *total gets the sum.
__device__ __forceinline__ long long block_scan_1024(long long v, long long* s_run, long long* total) {
  s_run[threadIdx.x] = v;
  __syncthreads();
  for (int o = 1; o < 1024; o <<= 1) {
    const long long y = threadIdx.x >= o ? s_run[threadIdx.x - o] : 0;
    __syncthreads();
    s_run[threadIdx.x] += y;
    __syncthreads();
  }
  const long long x = s_run[threadIdx.x] - v;
  *total = s_run[1023];
  __syncthreads();
  return x;
}

// Partition starts: part_begin[p] = rows of the partitions before p
// (part_begin[P] = all rows); cursor[p] starts at part_begin[p].  One block.
// The partition sizes also decide the work of the aggregation's blocks here,
// on the device, so that the host need not wait for them: a partition far
// above the average (skewed keys) is split into slices of at most `limit`
// rows, so no single block gets it all.
__global__ void __launch_bounds__(1024) group_part_scan_kernel(PartPlan pp, const unsigned long long* __restrict__ ptot,
                                                               long long* __restrict__ part_begin,
                                                               unsigned long long* __restrict__ cursor,
                                                               AggUnits* __restrict__ units) {
  __shared__ long long s_run[1024];
  const int per = (pp.n_parts + blockDim.x - 1) / blockDim.x;
  const int b = threadIdx.x * per;
  const int e = b + per < pp.n_parts ? b + per : pp.n_parts;
  long long s = 0;
  for (int i = b; i < e; ++i) s += static_cast<long long>(ptot[i]);
  long long all;
  long long run = block_scan_1024(s, s_run, &all);
  const long long first = run;
  for (int i = b; i < e; ++i) {
    part_begin[i] = run;
    cursor[i] = static_cast<unsigned long long>(run);
    run += static_cast<long long>(ptot[i]);
  }
  if (threadIdx.x == 0) part_begin[pp.n_parts] = all;
  // slices of `limit` rows, twice as long until there are at most kMaxPartials
  const long long avg = (pp.n + pp.n_parts - 1) / pp.n_parts;
  long long limit = 2 * avg > 65536 ? 2 * avg : 65536;
  long long n_slices, mine, slices;
  for (;; limit *= 2) {
    mine = 0;
    for (int i = b; i < e; ++i) {
      const long long sz = static_cast<long long>(ptot[i]);
      if (sz > limit) mine += (sz + limit - 1) / limit;
    }
    slices = block_scan_1024(mine, s_run, &n_slices);
    if (n_slices <= kMaxPartials) break;
  }
  if (threadIdx.x == 0) {
    units->limit = limit;
    units->n_slices = static_cast<int>(n_slices);
    units->n_merges = 0;
  }
  if (n_slices == 0) return;
  long long big = 0, n_merges;
  for (int i = b; i < e; ++i) big += static_cast<long long>(ptot[i]) > limit;
  big = block_scan_1024(big, s_run, &n_merges);
  if (threadIdx.x == 0) units->n_merges = static_cast<int>(n_merges);
  run = first;
  for (int i = b; i < e; ++i) {
    const long long sz = static_cast<long long>(ptot[i]);
    if (sz > limit) {
      const int k = static_cast<int>((sz + limit - 1) / limit);
      units->merge[big++] = make_int2(static_cast<int>(slices), k);
      for (int q = 0; q < k; ++q) {
        const long long lo = run + q * limit;
        units->slice[slices++] = AggSlice{lo, lo + limit < run + sz ? lo + limit : run + sz};
      }
    }
    run += sz;
  }
}

// A partitioned row: {key, value} (8 bytes) or, with a second value
// column, {key, pad, value as int64} (16 bytes): one store per row.
template <bool HAS2>
struct PartRow;
template <>
struct PartRow<false> {
  using T = int2;
  __device__ static T make(int32_t k, int32_t a, int32_t) { return make_int2(k, a); }
  __device__ static int32_t key(const T& r) { return r.x; }
  __device__ static int64_t val(const T& r) { return r.y; }
};
template <>
struct PartRow<true> {
  using T = longlong2;
  __device__ static T make(int32_t k, int32_t a, int32_t c) {
    return make_longlong2(static_cast<long long>(static_cast<uint32_t>(k)), static_cast<long long>(a) + c);
  }
  __device__ static int32_t key(const T& r) { return static_cast<int32_t>(static_cast<uint32_t>(r.x)); }
  __device__ static int64_t val(const T& r) { return r.y; }
};

template <bool HAS2>
__global__ void __launch_bounds__(1024) group_part_scatter_kernel(PartPlan pp, const int32_t* __restrict__ keys,
                                                                  const int32_t* __restrict__ vals,
                                                                  const int32_t* __restrict__ vals2,
                                                                  const unsigned int* __restrict__ hist,
                                                                  unsigned long long* __restrict__ cursor,
                                                                  typename PartRow<HAS2>::T* __restrict__ rows) {
  extern __shared__ unsigned int s_cur[];
  // this block's run in each partition (order inside a partition is free)
  for (int p = threadIdx.x; p < pp.n_parts; p += blockDim.x) {
    const unsigned int c = hist[static_cast<int64_t>(blockIdx.x) * pp.n_parts + p];
    s_cur[p] = c ? static_cast<unsigned int>(atomicAdd(&cursor[p], static_cast<unsigned long long>(c))) : 0u;
  }
  __syncthreads();
  const int64_t b = static_cast<int64_t>(blockIdx.x) * pp.per;
  const int64_t e = b + pp.per < pp.n ? b + pp.per : pp.n;
  const uint64_t pol = policy_evict_first();
  const bool vec = ((reinterpret_cast<uintptr_t>(keys) | reinterpret_cast<uintptr_t>(vals) |
                     reinterpret_cast<uintptr_t>(vals2)) & 15) == 0;
  auto one = [&](int32_t key, int32_t a, int32_t c) {
    const int32_t k = agg_key(key, pp.key_offset);
    if (k == kEmptyKey) return;
    const unsigned int pos = atomicAdd(&s_cur[agg_part(k, pp.n_parts)], 1u);
    rows[pos] = PartRow<HAS2>::make(k, a, c);
  };
  if (vec) {
    for (int64_t r = b + 4 * threadIdx.x; r < e; r += 4 * blockDim.x) {
      if (r + 4 <= e) {
        const int4 kk = ld_stream_v4(keys + r, pol), a = ld_stream_v4(vals + r, pol);
        const int4 c = HAS2 ? ld_stream_v4(vals2 + r, pol) : make_int4(0, 0, 0, 0);
        // the four cursor updates are independent: issue them together
        const int32_t k[4] = {agg_key(kk.x, pp.key_offset), agg_key(kk.y, pp.key_offset),
                              agg_key(kk.z, pp.key_offset), agg_key(kk.w, pp.key_offset)};
        unsigned int pos[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
          pos[u] = k[u] != kEmptyKey ? atomicAdd(&s_cur[agg_part(k[u], pp.n_parts)], 1u) : 0u;
        const int32_t av[4] = {a.x, a.y, a.z, a.w}, cv[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (k[u] != kEmptyKey) rows[pos[u]] = PartRow<HAS2>::make(k[u], av[u], cv[u]);
      } else {
        for (int64_t q = r; q < e; ++q) one(keys[q], vals[q], HAS2 ? vals2[q] : 0);
      }
    }
  } else {
    for (int64_t r = b + threadIdx.x; r < e; r += blockDim.x) one(keys[r], vals[r], HAS2 ? vals2[r] : 0);
  }
}

// The same scatter with coalesced writes: each tile of 8,192 rows (16 per
// thread) is counting-sorted by partition in shared
// memory, then written out so that consecutive threads write consecutive rows
// of a partition's run.  A run ends at a whole 32-byte sector; the rows past
// it (at most kCarry per partition) are carried into the next tile, because a
// sector written in two pieces costs L2 a read-modify-write when it is evicted
// in between (writing every row at once took 778 us for 2^27 rows in 444
// partitions, the same rows in input order 519 us, no rows 472 us).  The rest
// is the shared-memory pipe and the tile's chain of dependent phases: so two
// blocks fit an SM, the next tile's keys load while the current tile is
// written out and are ranked right after (one phase between barriers), and a
// sorted row's partition is hashed again instead of kept beside it.  Shared
// memory: the sorted rows, the carried rows, then per partition the tile
// count, the tile offset of the new rows, the block's cursor, the destination
// base, the tile index its write ends at, and the carried count.
constexpr int kScatterThreads = 512;
constexpr int kScatterBlocks = 2;

template <bool HAS2>
constexpr int scatter_carry() {  // rows a sector holds, less one
  return 32 / static_cast<int>(sizeof(typename PartRow<HAS2>::T)) - 1;
}
// G: 16-byte loads of a column per thread and tile (4, or 2 where the
// partitions leave no room for the longer tile).
template <bool HAS2, int G>
constexpr size_t scatter_smem(int64_t parts) {
  return sizeof(typename PartRow<HAS2>::T) * (4 * G * kScatterThreads + 2 * scatter_carry<HAS2>() * parts) + 6 * 4 * parts;
}

template <bool HAS2, int G>
__global__ void __launch_bounds__(kScatterThreads, kScatterBlocks) group_part_scatter_tiled_kernel(
    PartPlan pp, const int32_t* __restrict__ keys, const int32_t* __restrict__ vals,
    const int32_t* __restrict__ vals2, const unsigned int* __restrict__ hist, unsigned long long* __restrict__ cursor,
    typename PartRow<HAS2>::T* __restrict__ rows) {
  using Row = typename PartRow<HAS2>::T;
  constexpr int W = kScatterThreads / 32;
  constexpr int R = 4 * G;
  constexpr int kTile = R * kScatterThreads;
  constexpr int C = scatter_carry<HAS2>();
  extern __shared__ __align__(16) unsigned char sc_smem[];
  const int P = pp.n_parts;
  Row* s_rows = reinterpret_cast<Row*>(sc_smem);
  Row* s_carry = s_rows + kTile + C * P;
  unsigned int* s_cnt = reinterpret_cast<unsigned int*>(s_carry + C * P);
  unsigned int* s_off = s_cnt + P;
  unsigned int* s_cur = s_off + P;
  unsigned int* s_dst = s_cur + P;
  unsigned int* s_end = s_dst + P;
  unsigned int* s_left = s_end + P;
  __shared__ unsigned int s_warp[W];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t b = static_cast<int64_t>(blockIdx.x) * pp.per;
  const int64_t e = b + pp.per < pp.n ? b + pp.per : pp.n;
  if (b >= e) return;
  for (int p = tid; p < P; p += kScatterThreads) {
    const unsigned int c = hist[static_cast<int64_t>(blockIdx.x) * P + p];
    s_cur[p] = c ? static_cast<unsigned int>(atomicAdd(&cursor[p], static_cast<unsigned long long>(c))) : 0u;
    s_cnt[p] = 0;
    s_left[p] = 0;
  }
  const uint64_t pol = policy_evict_first();
  const bool vec = ((reinterpret_cast<uintptr_t>(keys) | reinterpret_cast<uintptr_t>(vals) |
                     reinterpret_cast<uintptr_t>(vals2)) & 15) == 0;
  const int per_thread = (P + kScatterThreads - 1) / kScatterThreads;  // partitions per thread in the scan
  auto prefetch_tile = [&](int64_t t0) {  // the tile's columns into L2, ahead of its loads
    if (tid != 0 || t0 >= e) return;
    const int64_t m = e - t0 < kTile ? e - t0 : kTile;
    prefetch_l2_range(keys + t0, 4 * m);
    prefetch_l2_range(vals + t0, 4 * m);
    if (HAS2) prefetch_l2_range(vals2 + t0, 4 * m);
  };
  // this thread's 16 rows of a tile: 4 at t0 + 4 (tid + 512 h) for each h
  auto row0 = [&](int64_t t0, int h) { return t0 + 4 * (tid + h * static_cast<int64_t>(kScatterThreads)); };
  int32_t k[R];
  uint32_t slot[R];  // partition << 13 | rank, or ~0u for no row
  // what the key column would hold for the reserved key: no row
  const int32_t no_key = static_cast<int32_t>(static_cast<uint32_t>(kEmptyKey) - static_cast<uint32_t>(pp.key_offset));
  auto load_keys = [&](int64_t t0) {
#pragma unroll
    for (int h = 0; h < G; ++h) {
      const int64_t r0 = row0(t0, h);
      if (vec && r0 + 4 <= e) {
        const int4 kk = ld_stream_v4_ordered(keys + r0, pol);
        k[4 * h] = kk.x; k[4 * h + 1] = kk.y; k[4 * h + 2] = kk.z; k[4 * h + 3] = kk.w;
      } else {
#pragma unroll
        for (int u = 0; u < 4; ++u) k[4 * h + u] = r0 + u < e ? keys[r0 + u] : no_key;
      }
    }
  };
  auto rank_keys = [&]() {
#pragma unroll
    for (int q = 0; q < R; ++q) {
      k[q] = agg_key(k[q], pp.key_offset);
      slot[q] = ~0u;
      if (k[q] != kEmptyKey) {
        const uint32_t part = agg_part(k[q], P);
        slot[q] = (part << 13) | atomicAdd(&s_cnt[part], 1u);
      }
    }
  };
  prefetch_tile(b + kTile);
  load_keys(b);
  __syncthreads();  // the counts are zero
  rank_keys();
  for (int64_t t0 = b; t0 < e; t0 += kTile) {
    const bool more = t0 + kTile < e;
    prefetch_tile(t0 + 2 * kTile);
    __syncthreads();
    // exclusive scan of the tile's rows per partition, carried ones first
    // (each thread a run of partitions)
    unsigned int run = 0;
    for (int j = 0; j < per_thread; ++j) {
      const int p = tid * per_thread + j;
      if (p < P) run += s_cnt[p] + s_left[p];
    }
    unsigned int inc = run;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned int y = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += y;
    }
    if (lane == 31) s_warp[warp] = inc;
    __syncthreads();
    unsigned int off = inc - run, n_valid = 0;
#pragma unroll
    for (int w = 0; w < W; ++w) {
      const unsigned int x = s_warp[w];
      if (w < warp) off += x;
      n_valid += x;
    }
    for (int j = 0; j < per_thread; ++j) {
      const int p = tid * per_thread + j;
      if (p < P) {
        const unsigned int old = s_left[p], all = s_cnt[p] + old, cur = s_cur[p];
        // written up to the last whole sector, all of it at the end
        const unsigned int left = more ? min(all, (cur + all) & static_cast<unsigned int>(C)) : 0u;
        for (unsigned int c = 0; c < old; ++c) s_rows[off + c] = s_carry[C * p + c];
        s_off[p] = off + old;
        s_dst[p] = cur - off;
        s_end[p] = off + all - left;
        s_cur[p] = cur + all - left;
        s_left[p] = left;
        s_cnt[p] = 0;
        off += all;
      }
    }
    __syncthreads();
    // rows into their sorted places (the values are read only now: 16 of them
    // beside the keys would not fit a thread's registers)
#pragma unroll
    for (int h = 0; h < G; ++h) {
      const int64_t r0 = row0(t0, h);
      int32_t a[4], c[4];
      if (vec && r0 + 4 <= e) {
        const int4 av = ld_stream_v4(vals + r0, pol);
        const int4 cv = HAS2 ? ld_stream_v4(vals2 + r0, pol) : make_int4(0, 0, 0, 0);
        a[0] = av.x; a[1] = av.y; a[2] = av.z; a[3] = av.w;
        c[0] = cv.x; c[1] = cv.y; c[2] = cv.z; c[3] = cv.w;
      } else {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          a[u] = r0 + u < e ? vals[r0 + u] : 0;
          c[u] = HAS2 && r0 + u < e ? vals2[r0 + u] : 0;
        }
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const uint32_t sl = slot[4 * h + u];
        if (sl != ~0u) s_rows[s_off[sl >> 13] + (sl & 8191u)] = PartRow<HAS2>::make(k[4 * h + u], a[u], c[u]);
      }
    }
    __syncthreads();
    // coalesced writes (sorted row i goes to its partition's run, or is
    // carried), while the next tile's keys load
    if (more) load_keys(t0 + kTile);
    for (unsigned int i = tid; i < n_valid; i += kScatterThreads) {
      const Row x = s_rows[i];
      const uint32_t p = agg_part(PartRow<HAS2>::key(x), P);
      const unsigned int end = s_end[p];
      if (i < end) rows[s_dst[p] + i] = x;
      else s_carry[C * p + (i - end)] = x;
    }
    if (more) rank_keys();
  }
}

// Appends the occupied slots of a block's shared table to the outputs
// (positions from one global counter per block).  Every thread of the block
// calls it (it synchronises the block).
__device__ __forceinline__ void append_groups(const SmemAgg& st, int64_t capacity, int32_t* __restrict__ out_keys,
                                              int64_t* __restrict__ out_sums, int64_t* __restrict__ out_counts,
                                              unsigned long long* d_groups, unsigned long long* overflow) {
  __shared__ unsigned int s_n;
  __shared__ unsigned long long s_base;
  if (threadIdx.x == 0) s_n = 0;
  __syncthreads();
  constexpr int kPer = kAggMaxSlots / kAggThreads;
  unsigned int pos[kPer];
#pragma unroll
  for (int j = 0; j < kPer; ++j) {
    const uint32_t i = j * kAggThreads + threadIdx.x;
    pos[j] = i < st.slots && st.key[i] != kEmptyKey ? atomicAdd(&s_n, 1u) : ~0u;
  }
  __syncthreads();
  if (threadIdx.x == 0) s_base = s_n ? atomicAdd(d_groups, static_cast<unsigned long long>(s_n)) : 0ull;
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kPer; ++j) {
    if (pos[j] == ~0u) continue;
    const uint32_t i = j * kAggThreads + threadIdx.x;
    const unsigned long long o = s_base + pos[j];
    if (o >= static_cast<unsigned long long>(capacity)) {  // more groups than the outputs hold
      atomicAdd(overflow, 1ull);
      continue;
    }
    out_keys[o] = st.key[i];
    out_sums[o] = static_cast<int64_t>(st.sum(i));
    if (out_counts) out_counts[o] = static_cast<int64_t>(st.cnt[i]);
  }
}

// Blocks [0, kMaxPartials): the slices of split partitions (none in the usual
// case: they return at once), each to its partial table.  The others: one
// partition each, aggregated in a shared table, its groups appended to the
// outputs; a split one is left to its slices.
template <bool HAS2>
__global__ void __launch_bounds__(kAggThreads) group_part_agg_kernel(
    const long long* __restrict__ part_begin, const AggUnits* __restrict__ units,
    const typename PartRow<HAS2>::T* __restrict__ rows, uint32_t slots, int combine, int64_t capacity,
    int32_t* __restrict__ out_keys, int64_t* __restrict__ out_sums, int64_t* __restrict__ out_counts,
    unsigned long long* d_groups, unsigned long long* overflow, int4* __restrict__ partials) {
  extern __shared__ __align__(16) unsigned char agg_smem[];
  using V = std::conditional_t<HAS2, int64_t, int32_t>;
  using Row = typename PartRow<HAS2>::T;
  int64_t b, e;
  int partial = -1;
  if (blockIdx.x < kMaxPartials) {
    partial = blockIdx.x;
    if (partial >= units->n_slices) return;
    b = units->slice[partial].begin;
    e = units->slice[partial].end;
  } else {
    b = part_begin[blockIdx.x - kMaxPartials];
    e = part_begin[blockIdx.x - kMaxPartials + 1];
    if (e - b > units->limit || b == e) return;
  }
  const SmemAgg st = smem_agg(agg_smem, slots);
  smem_agg_clear(st);
  __syncthreads();
  unsigned int lost = 0;
  const Row* p = rows + b + threadIdx.x;
  int64_t left = e - b;
  // whole steps of 8 rows per thread, in two batches; the step after next is
  // on its way into L2
  constexpr int64_t kStep = 8 * kAggThreads;
  if (!combine) {
    for (; left >= kStep; left -= kStep, p += kStep) {
      if (threadIdx.x == 0 && left >= 3 * kStep) prefetch_l2_range(p + 2 * kStep, kStep * sizeof(Row));
      Row x[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) x[u] = p[u * kAggThreads];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        int32_t k[4];
        V v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          k[u] = PartRow<HAS2>::key(x[4 * h + u]);
          v[u] = static_cast<V>(PartRow<HAS2>::val(x[4 * h + u]));
        }
        lost += __popc(smem_agg_rows<4, true>(st, k, v, 0xFu, 0xffffffffu));  // the loop is block-uniform
      }
    }
  }
  for (; left > 0; left -= 4 * kAggThreads, p += 4 * kAggThreads) {
    int32_t k[4];
    V v[4];
    uint32_t valid = 0;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const bool ok = u * kAggThreads + static_cast<int64_t>(threadIdx.x) < left;
      Row x{};
      if (ok) x = p[u * kAggThreads];
      k[u] = ok ? PartRow<HAS2>::key(x) : 0;
      v[u] = ok ? static_cast<V>(PartRow<HAS2>::val(x)) : 0;
      valid |= static_cast<uint32_t>(ok) << u;
    }
    if (!combine) {
      lost += __popc(smem_agg_rows<4, false>(st, k, v, valid, 0xffffffffu));
      continue;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      int64_t gs = v[u];
      uint32_t gc = 1;
      if (warp_combine((valid >> u) & 1u, k[u], gs, &gs, &gc))
        if (!smem_agg_add(st, k[u], static_cast<uint64_t>(gs), gc)) ++lost;
    }
  }
  if (lost) atomicAdd(overflow, static_cast<unsigned long long>(lost));
  __syncthreads();
  if (partial >= 0) {  // the whole table, as laid out in shared memory (16 bytes per slot)
    const int4* src = reinterpret_cast<const int4*>(agg_smem);
    int4* dst = partials + static_cast<int64_t>(partial) * slots;
    for (uint32_t i = threadIdx.x; i < slots; i += blockDim.x) dst[i] = src[i];
    return;
  }
  append_groups(st, capacity, out_keys, out_sums, out_counts, d_groups, overflow);
}

// Adds up the tables of a split partition's slices and appends the groups.  A
// block takes the keys of kMergeSlots slots' home buckets, so that a partition
// is merged by slots / kMergeSlots blocks (one block for all of it took 886 us
// for the 111 tables of a key that half of 2^26 rows have, 81 us so): in
// each table those keys lie in these slots and in the full buckets that follow
// (a run ends at a bucket with a free slot, and the tables have the same layout
// and hash).
constexpr uint32_t kMergeSlots = kAggThreads;
__global__ void __launch_bounds__(kAggThreads) group_part_merge_kernel(
    const AggUnits* __restrict__ units, const int4* __restrict__ partials, uint32_t slots, int64_t capacity,
    int32_t* __restrict__ out_keys, int64_t* __restrict__ out_sums, int64_t* __restrict__ out_counts,
    unsigned long long* d_groups, unsigned long long* overflow, const unsigned long long* timeouts) {
  if (blockIdx.x == 0 && threadIdx.x == 0) overflow[1] = *timeouts;  // beside the overflow count, for the caller's one copy
  extern __shared__ __align__(16) unsigned char agg_smem[];
  const SmemAgg st = smem_agg(agg_smem, slots);
  const int shares = static_cast<int>(slots / kMergeSlots), work = units->n_merges * shares;
  for (int w = blockIdx.x; w < work; w += gridDim.x) {  // (usually none)
    const int2 m = units->merge[w / shares];
    smem_agg_clear(st);
    __syncthreads();
    const uint32_t first = static_cast<uint32_t>(w % shares) * kMergeSlots;  // slots [first, first + kMergeSlots)
    auto table = [&](int q) {
      return smem_agg(reinterpret_cast<unsigned char*>(const_cast<int4*>(partials) +
                                                       static_cast<int64_t>(m.x + q) * slots),
                      slots);
    };
    auto mine = [&](int32_t k) {
      return k != kEmptyKey && 4 * st.home(k) - first < kMergeSlots;  // its home bucket lies in this block's slots
    };
    unsigned int lost = 0;
    auto add = [&](int32_t k, uint32_t lo, uint32_t hi, uint32_t c) {
      const int at = smem_find_insert(st, k, st.home(k));
      if (at < 0) {
        ++lost;
        return;
      }
      const uint32_t old = atomicAdd(st.lo + at, lo);
      const uint32_t h = hi + static_cast<uint32_t>(agg_high(old, static_cast<int32_t>(lo)));
      if (h) atomicAdd(st.lo + slots + at, h);
      atomicAdd(st.cnt + at, c);
    };
    // this block's slots, a thread each, four tables in flight
    const uint32_t i = first + threadIdx.x;
    for (int q0 = 0; q0 < m.y; q0 += 4) {
      int32_t k[4];
      uint32_t lo[4], hi[4], c[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const bool in = q0 + u < m.y;
        const SmemAgg t = table(in ? q0 + u : q0);
        k[u] = in ? t.key[i] : kEmptyKey;
        lo[u] = t.lo[i];
        hi[u] = t.lo[slots + i];
        c[u] = t.cnt[i];
      }
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (mine(k[u])) add(k[u], lo[u], hi[u], c[u]);
    }
    // the full buckets behind them, a warp on a table, a lane per slot
    const uint32_t lane = threadIdx.x & 31u;
    for (int q = threadIdx.x >> 5; q < m.y; q += kAggThreads / 32) {
      const SmemAgg t = table(q);
      uint32_t b = (first + kMergeSlots) / 4 - 1;  // the last of its own buckets
      for (uint32_t step = 0; step < t.nb; ++step) {
        const int4 x = *reinterpret_cast<const int4*>(t.key + 4 * b);
        if (x.x == kEmptyKey || x.y == kEmptyKey || x.z == kEmptyKey || x.w == kEmptyKey) break;
        b = t.next(b);
        if (b == first / 4) break;  // all the way round
        if (lane < 4 && mine(t.key[4 * b + lane]))
          add(t.key[4 * b + lane], t.lo[4 * b + lane], t.lo[slots + 4 * b + lane], t.cnt[4 * b + lane]);
        __syncwarp();
      }
    }
    if (lost) atomicAdd(overflow, static_cast<unsigned long long>(lost));
    __syncthreads();
    append_groups(st, capacity, out_keys, out_sums, out_counts, d_groups, overflow);
    __syncthreads();  // the table is cleared next
  }
}

// The global table of plan 1 empty, and the counters zero (one launch).
__global__ void group_table_init_kernel(HashAgg t, int64_t capacity, unsigned long long* d_groups) {
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < capacity; i += stride) {
    t.keys[i] = kEmptyKey;
    t.sums[i] = 0;
    t.counts[i] = 0;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    *d_groups = 0;
    *t.overflow = 0;
  }
}

// Its occupied slots to the outputs, in no particular order (a block claims
// its positions with one atomic).
__global__ void __launch_bounds__(256) group_table_append_kernel(HashAgg t, int64_t capacity, int32_t* __restrict__ out_keys,
                                                                 int64_t* __restrict__ out_sums,
                                                                 int64_t* __restrict__ out_counts,
                                                                 unsigned long long* d_groups,
                                                                 const unsigned long long* timeouts) {
  __shared__ unsigned int s_n;
  __shared__ unsigned long long s_base;
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (threadIdx.x == 0) s_n = 0;
  if (i == 0) t.overflow[1] = *timeouts;  // beside the overflow count, for the caller's one copy
  __syncthreads();
  const int32_t k = i < capacity ? t.keys[i] : kEmptyKey;
  const unsigned int at = k != kEmptyKey ? atomicAdd(&s_n, 1u) : 0u;
  __syncthreads();
  if (threadIdx.x == 0) s_base = s_n ? atomicAdd(d_groups, static_cast<unsigned long long>(s_n)) : 0ull;
  __syncthreads();
  if (k == kEmptyKey) return;
  const unsigned long long o = s_base + at;  // at most `capacity` slots are occupied
  out_keys[o] = k;
  out_sums[o] = static_cast<int64_t>(t.sums[i]);
  if (out_counts) out_counts[o] = static_cast<int64_t>(t.counts[i]);
}

// SUM(price * qty * (100 + tax)) in int64 (exact modulo 2^64).
__global__ void __launch_bounds__(512) agg_fixed_kernel(int64_t n, const int32_t* __restrict__ price,
                                                        const int32_t* __restrict__ qty,
                                                        const int32_t* __restrict__ tax,
                                                        unsigned long long* sum) {
  __shared__ long long s_red[16];
  const uint64_t pol = policy_evict_first();
  uint64_t s = 0;
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  const int64_t t0 = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  auto term = [](int32_t p, int32_t q, int32_t t) {
    return static_cast<uint64_t>(static_cast<int64_t>(p) * q) * static_cast<uint64_t>(static_cast<int64_t>(100) + t);
  };
  const bool vec = ((reinterpret_cast<uintptr_t>(price) | reinterpret_cast<uintptr_t>(qty) |
                     reinterpret_cast<uintptr_t>(tax)) & 15) == 0;
  const int64_t n4 = vec ? n >> 2 : 0;
  for (int64_t i = t0; i < n4; i += stride) {
    const int4 p = ld_stream_v4(price + 4 * i, pol), q = ld_stream_v4(qty + 4 * i, pol), t = ld_stream_v4(tax + 4 * i, pol);
    s += term(p.x, q.x, t.x) + term(p.y, q.y, t.y) + term(p.z, q.z, t.z) + term(p.w, q.w, t.w);
  }
  for (int64_t r = 4 * n4 + t0; r < n; r += stride) s += term(price[r], qty[r], tax[r]);
  int64_t v = warp_sum_i64(static_cast<int64_t>(s));
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) s_red[warp] = v;
  __syncthreads();
  if (warp == 0) {
    long long x = lane < static_cast<int>(blockDim.x >> 5) ? s_red[lane] : 0;
    x = warp_sum_i64(x);
    if (lane == 0) atomicAdd(sum, static_cast<unsigned long long>(x));
  }
}

// Double variant, deterministic: fixed per-block partial sums (each block a
// fixed contiguous range, reduced in a fixed tree order), then one block sums
// the partials in a fixed tree order.
constexpr int kAggF64Blocks = 1024;
__global__ void __launch_bounds__(256) agg_f64_partial_kernel(int64_t n, const double* __restrict__ tax,
                                                              const double* __restrict__ qty,
                                                              const double* __restrict__ price,
                                                              double* __restrict__ partial) {
  __shared__ double s[256];
  const int64_t per = (n + gridDim.x - 1) / gridDim.x;
  const int64_t b = static_cast<int64_t>(blockIdx.x) * per;
  const int64_t e = b + per < n ? b + per : n;
  double acc = 0.0;
  for (int64_t r = b + threadIdx.x; r < e; r += blockDim.x) {
    const double netto = price[r] * qty[r];
    acc += netto * tax[r] + netto;
  }
  s[threadIdx.x] = acc;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (threadIdx.x < o) s[threadIdx.x] += s[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) partial[blockIdx.x] = s[0];
}

// The partials by a tree in a fixed order, one thread each (one thread adding
// them up one after another took 28 us).
__global__ void __launch_bounds__(kAggF64Blocks) agg_f64_final_kernel(const double* __restrict__ partial, double* out) {
  __shared__ double s[kAggF64Blocks];
  s[threadIdx.x] = partial[threadIdx.x];
  for (int o = kAggF64Blocks / 2; o > 0; o >>= 1) {
    __syncthreads();
    if (threadIdx.x < o) s[threadIdx.x] += s[threadIdx.x + o];
  }
  if (threadIdx.x == 0) *out = s[0];
}

// The context's grow-only buffer (declared in olap_internal.cuh).
char* big_scratch(olap_ctx* ctx, size_t bytes) {
  if (bytes <= ctx->big_bytes) return ctx->big;
  if (cudaStreamSynchronize(ctx->stream) != cudaSuccess) return nullptr;
  if (ctx->big) cudaFree(ctx->big);
  ctx->big = nullptr;
  ctx->big_bytes = 0;
  const size_t want = bytes + bytes / 4;
  if (cudaMalloc(reinterpret_cast<void**>(&ctx->big), want) != cudaSuccess) {
    cudaGetLastError();
    return nullptr;
  }
  ctx->big_bytes = want;
  return ctx->big;
}

static unsigned grid_of(const olap_ctx* ctx, int64_t items, int threads, int per_sm) {
  int64_t g = (items + threads - 1) / threads;
  const int64_t cap = static_cast<int64_t>(ctx->sm_count) * per_sm;
  if (g > cap) g = cap;
  return static_cast<unsigned>(g < 1 ? 1 : g);
}

}  // namespace olap

extern "C" {

int olap_group_vector(olap_ctx* ctx, int64_t n, const int32_t* vecInx, const int32_t* m1,
                      const int32_t* m2, int64_t group_num, int64_t* group_vector, int64_t* counts,
                      int64_t* d_total) {
  if (!ctx) return OLAP_ERR_INVALID;
  std::lock_guard<std::mutex> lk(ctx->mu);
  OLAP_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  OLAP_REQUIRE(ctx, n >= 0 && group_num >= 1 && group_vector && d_total, "bad arguments");
  OLAP_REQUIRE(ctx, n == 0 || (vecInx && m1 && m2), "null column");
  OLAP_CUDA_TRY(ctx, cudaMemsetAsync(group_vector, 0, sizeof(int64_t) * group_num, ctx->stream));
  if (counts) OLAP_CUDA_TRY(ctx, cudaMemsetAsync(counts, 0, sizeof(int64_t) * group_num, ctx->stream));
  OLAP_CUDA_TRY(ctx, cudaMemsetAsync(d_total, 0, sizeof(int64_t), ctx->stream));
  if (n == 0) return OLAP_OK;
  const int64_t smem = group_num * 8 * (counts ? 2 : 1);
  const bool use_smem = smem <= 96 * 1024;
  auto sums = reinterpret_cast<unsigned long long*>(group_vector);
  auto cnts = reinterpret_cast<unsigned long long*>(counts);
  auto tot = reinterpret_cast<unsigned long long*>(d_total);
  if (use_smem) {
    OLAP_CUDA_TRY(ctx, cudaFuncSetAttribute(olap::group_vector_kernel<true>,
                                            cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024));
    const int per_sm = smem > 48 * 1024 ? 2 : 4;
    olap::group_vector_kernel<true><<<olap::grid_of(ctx, (n + 3) / 4, olap::kGroupThreads, per_sm),
                                      olap::kGroupThreads, static_cast<size_t>(smem), ctx->stream>>>(
        n, vecInx, m1, m2, group_num, sums, cnts, tot, &ctx->counters->range_errors);
  } else {
    olap::group_vector_kernel<false><<<olap::grid_of(ctx, (n + 3) / 4, olap::kGroupThreads, 4),
                                       olap::kGroupThreads, 0, ctx->stream>>>(
        n, vecInx, m1, m2, group_num, sums, cnts, tot, &ctx->counters->range_errors);
  }
  OLAP_CUDA_TRY(ctx, cudaGetLastError());
  return OLAP_OK;
}

int64_t olap_group_hash_capacity(int64_t max_groups) {
  int64_t cap = 1024;
  while (cap < 2 * max_groups) cap <<= 1;
  return cap;
}

int olap_group_hash(olap_ctx* ctx, int64_t n, const int32_t* keys, int32_t key_offset,
                    const int32_t* vals, const int32_t* vals2, int64_t capacity, int32_t* out_keys,
                    int64_t* out_sums, int64_t* out_counts, int64_t* d_groups) {
  if (!ctx) return OLAP_ERR_INVALID;
  std::lock_guard<std::mutex> lk(ctx->mu);
  OLAP_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  OLAP_REQUIRE(ctx, n >= 0 && capacity >= 1024 && (capacity & (capacity - 1)) == 0,
               "capacity must be a power of two >= 1024 (see olap_group_hash_capacity)");
  OLAP_REQUIRE(ctx, n < (int64_t(1) << 32), "at most 2^32 - 1 rows per call");
  OLAP_REQUIRE(ctx, out_keys && out_sums && d_groups, "null output");
  OLAP_REQUIRE(ctx, n == 0 || (keys && vals), "null column");
  olap::Arena ar(ctx);
  unsigned long long* overflow = ar.take<unsigned long long>(2);  // overflows, wait timeouts so far
  if (!overflow) return olap::set_error(ctx, OLAP_ERR_CAPACITY, "scratch arena exhausted");
  int st = OLAP_OK;
  char* mem = nullptr;
  cudaError_t e = cudaSuccess;
  // Warp combining of equal keys (match_any + reductions) costs more than the
  // same-address shared atomics it saves on uniform and mildly skewed keys
  // (measured on B200), so it is off unless the tuning knob asks for it.
  const int combine = ctx->tune[olap::TUNE_GROUP_COMBINE] == 1 ? 1 : 0;
  const int64_t plan_knob = ctx->tune[olap::TUNE_GROUP_PLAN];
  // Knob: 1 plan 1 where it fits (batched table updates), 2 plan 2 always,
  // 3 plan 1 with one row's table update after another; 0 the default (1).
  const bool plan1 = plan_knob == 2 ? false : capacity <= olap::kAggSlots;
  const bool batched = plan_knob != 3 && combine == 0;
  if (plan1) {
    // Plan 1: per-block shared tables of `capacity` slots, then the global
    // table (in the context's grow-only buffer) and its compaction.
    const size_t bytes = static_cast<size_t>(capacity) * (4 + 8 + 8);
    mem = olap::big_scratch(ctx, bytes);
    if (!mem) return olap::set_error(ctx, OLAP_ERR_NOMEM, "device memory for the group table");
    olap::HashAgg t;
    t.sums = reinterpret_cast<unsigned long long*>(mem);
    t.counts = t.sums + capacity;
    t.keys = reinterpret_cast<int32_t*>(t.counts + capacity);
    t.mask = static_cast<uint64_t>(capacity - 1);
    t.overflow = overflow;
    auto* d_groups_u = reinterpret_cast<unsigned long long*>(d_groups);
    olap::group_table_init_kernel<<<olap::grid_of(ctx, capacity, 256, 8), 256, 0, ctx->stream>>>(t, capacity,
                                                                                                d_groups_u);
    const uint32_t slots = static_cast<uint32_t>(capacity);  // per-block table
    if (n && e == cudaSuccess && batched) {
      // The block tables fill the shared memory once the keys are many: at
      // lower load fewer keys overflow their home bucket, and the lanes of a
      // warp take the insert path less often.
      uint32_t tslots = slots;
      if (capacity >= 2048)
        tslots = std::max<uint32_t>(slots, static_cast<uint32_t>(ctx->smem_optin / 16) & ~3u);
      const size_t smem = static_cast<size_t>(tslots) * 16;
      auto launch = [&](auto kern) {
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
        int bps = 1;
        if (e == cudaSuccess)
          e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, kern, olap::kRowsThreads, smem);
        int64_t grid = static_cast<int64_t>(ctx->sm_count) * (bps < 1 ? 1 : bps);
        grid = std::min<int64_t>(grid, (n + 4 * olap::kRowsThreads - 1) / (4 * olap::kRowsThreads));
        if (e == cudaSuccess)
          kern<<<static_cast<unsigned>(grid < 1 ? 1 : grid), olap::kRowsThreads, smem, ctx->stream>>>(
              n, keys, key_offset, vals, vals2, tslots, t, &ctx->counters->range_errors);
      };
      if (vals2)
        launch(olap::group_hash_rows_kernel<true>);
      else
        launch(olap::group_hash_rows_kernel<false>);
    } else if (n && e == cudaSuccess) {
      const size_t smem = static_cast<size_t>(slots) * 16;
      e = cudaFuncSetAttribute(olap::group_hash_smem_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               static_cast<int>(smem));
      int bps = 1;
      if (e == cudaSuccess)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, olap::group_hash_smem_kernel, olap::kAggThreads,
                                                          smem);
      int64_t grid = static_cast<int64_t>(ctx->sm_count) * (bps < 1 ? 1 : bps);
      grid = std::min<int64_t>(grid, (n + 4 * olap::kAggThreads - 1) / (4 * olap::kAggThreads));
      if (e == cudaSuccess)
        olap::group_hash_smem_kernel<<<static_cast<unsigned>(grid < 1 ? 1 : grid), olap::kAggThreads, smem,
                                       ctx->stream>>>(n, keys, key_offset, vals, vals2,
                                                      slots, combine, t,
                                                      &ctx->counters->range_errors);
    }
    if (e == cudaSuccess)
      olap::group_table_append_kernel<<<static_cast<unsigned>((capacity + 255) / 256), 256, 0, ctx->stream>>>(
          t, capacity, out_keys, out_sums, out_counts, d_groups_u, &ctx->counters->wait_timeouts);
  } else {
    // Plan 2: partition, then one block per partition.
    olap::PartPlan pp;
    pp.n = n;
    pp.key_offset = key_offset;
    if (capacity > (int64_t(1) << 27))
      return olap::set_error(ctx, OLAP_ERR_UNSUPPORTED, "hash group-by capacity above 2^27 slots");
    // Partitions: whole waves of one block per SM (no half-empty last wave),
    // as few as keep the buckets of a partition's table at about a key on
    // average (a key outside its home bucket leaves the batched path: 0.1 % of
    // them at 0.7 keys a bucket, 0.4 % at one), since the scatter's runs get
    // shorter with every partition: three waves of 14,336-slot tables for 2^20
    // groups, eight for 2^22.  Few groups take 8,192-slot tables, which are
    // cleared and emptied faster.
    const int64_t keys_max = capacity / 2, sms = ctx->sm_count;
    auto need = [&](int64_t slots, int64_t per4) {  // waves at per4 / 4 keys per bucket
      return (4 * keys_max + per4 * sms * (slots / 4) - 1) / (per4 * sms * (slots / 4));
    };
    pp.slots = olap::kAggSlots;
    int64_t waves = need(olap::kAggSlots, 3);
    if (waves > 2) {
      pp.slots = olap::kAggMaxSlots;
      // at least three: 2^27 rows, scatter and aggregation, 2^20 groups in two
      // waves 593 + 596 us and in three 613 + 457, 2^19 groups in one wave 573 +
      // 620 us and in three 612 + 394
      waves = std::max<int64_t>(3, need(olap::kAggMaxSlots, 4));
    }
    // The tiled scatter keeps some words per partition in shared memory: with
    // more partitions than fit, fewer, as long as `capacity` distinct keys
    // still fit their tables (13,600 of 14,336 slots), then the shorter tile,
    // then the scatter without tiles.
    const size_t room = static_cast<size_t>(ctx->smem_optin) - 1024;
    auto tile_smem = [&](int64_t w, int g) {
      const int64_t p = w * sms;
      return g == 4 ? (vals2 ? olap::scatter_smem<true, 4>(p) : olap::scatter_smem<false, 4>(p))
                    : (vals2 ? olap::scatter_smem<true, 2>(p) : olap::scatter_smem<false, 2>(p));
    };
    int tile_g = 0;
    for (int g : {4, 2}) {
      int64_t w = waves;
      while (w > 1 && tile_smem(w, g) > room) --w;
      if (w == waves || w * sms * 13600 >= capacity) {
        waves = w;
        tile_g = g;
        break;
      }
    }
    if (!tile_g) {
      // The scatter keeps a cursor per partition only, and so many partitions
      // have few rows each: clearing and emptying a table is what one costs.  As
      // few as hold `capacity` distinct keys, then (20M rows of 20M keys, scatter
      // and aggregation: 9,472 partitions 520 + 722 us, 5,032 486 + 476).
      waves = (capacity + 13600 * sms - 1) / (13600 * sms);
    }
    pp.n_parts = static_cast<int32_t>(waves * sms);
    pp.n_blocks = ctx->sm_count * 2;
    pp.per = ((n + pp.n_blocks - 1) / pp.n_blocks + 3) & ~int64_t(3);
    if (pp.per < 4) pp.per = 4;
    const size_t hist_bytes = sizeof(unsigned int) * static_cast<size_t>(pp.n_parts) * pp.n_blocks;
    // part_begin[P + 1], then ptot[P] and cursor[P] (zeroed together)
    const size_t begin_bytes = sizeof(long long) * (3 * static_cast<size_t>(pp.n_parts) + 1);
    const size_t row_bytes = vals2 ? 16 : 8;
    // after the rows: the slices, the merge list and the partial tables
    // of partitions too large for one block (at most kMaxPartials of them)
    const size_t rows_off = (begin_bytes + hist_bytes + 255) & ~size_t(255);
    const size_t units_off = (rows_off + static_cast<size_t>(n > 0 ? n : 1) * row_bytes + 255) & ~size_t(255);
    const size_t part_off = (units_off + sizeof(olap::AggUnits) + 255) & ~size_t(255);
    const size_t bytes = part_off + static_cast<size_t>(olap::kMaxPartials) * pp.slots * 16;
    mem = olap::big_scratch(ctx, bytes);
    if (!mem) return olap::set_error(ctx, OLAP_ERR_NOMEM, "device memory for the group partitions");
    long long* part_begin = reinterpret_cast<long long*>(mem);
    auto* ptot = reinterpret_cast<unsigned long long*>(part_begin + pp.n_parts + 1);
    auto* cursor = ptot + pp.n_parts;
    unsigned int* hist = reinterpret_cast<unsigned int*>(mem + begin_bytes);
    char* rowbuf = mem + rows_off;
    auto* d_units = reinterpret_cast<olap::AggUnits*>(mem + units_off);
    auto* d_partials = reinterpret_cast<int4*>(mem + part_off);
    e = cudaMemsetAsync(d_groups, 0, sizeof(int64_t), ctx->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(overflow, 0, sizeof(unsigned long long), ctx->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(ptot, 0, sizeof(unsigned long long) * pp.n_parts, ctx->stream);
    const size_t psmem = sizeof(unsigned int) * pp.n_parts;
    if (e == cudaSuccess && psmem > 48 * 1024) {
      e = cudaFuncSetAttribute(olap::group_part_hist_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               static_cast<int>(psmem));
      if (e == cudaSuccess)
        e = cudaFuncSetAttribute(olap::group_part_scatter_kernel<true>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(psmem));
      if (e == cudaSuccess)
        e = cudaFuncSetAttribute(olap::group_part_scatter_kernel<false>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(psmem));
    }
    const size_t asmem = static_cast<size_t>(pp.slots) * 16;
    const size_t tsmem = tile_g ? tile_smem(waves, tile_g) : 0;
    auto scatter_tiled = [&](auto* rows, auto kern) {
      e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(tsmem));
      if (e == cudaSuccess)
        kern<<<pp.n_blocks, olap::kScatterThreads, tsmem, ctx->stream>>>(pp, keys, vals, vals2, hist, cursor, rows);
    };
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(olap::group_part_agg_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               static_cast<int>(asmem));
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(olap::group_part_agg_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               static_cast<int>(asmem));
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(olap::group_part_merge_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               static_cast<int>(asmem));
    if (e == cudaSuccess) {
      olap::group_part_hist_kernel<<<pp.n_blocks, 1024, psmem, ctx->stream>>>(pp, keys, hist, ptot,
                                                                              &ctx->counters->range_errors);
      olap::group_part_scan_kernel<<<1, 1024, 0, ctx->stream>>>(pp, ptot, part_begin, cursor, d_units);
      auto* d_groups_u = reinterpret_cast<unsigned long long*>(d_groups);
      const unsigned agg_grid = static_cast<unsigned>(pp.n_parts + olap::kMaxPartials);
      if (vals2) {
        auto* rows = reinterpret_cast<longlong2*>(rowbuf);
        if (e == cudaSuccess && tile_g == 4) scatter_tiled(rows, olap::group_part_scatter_tiled_kernel<true, 4>);
        else if (e == cudaSuccess && tile_g == 2) scatter_tiled(rows, olap::group_part_scatter_tiled_kernel<true, 2>);
        else if (e == cudaSuccess)
          olap::group_part_scatter_kernel<true><<<pp.n_blocks, 1024, psmem, ctx->stream>>>(pp, keys, vals, vals2,
                                                                                          hist, cursor, rows);
        if (e == cudaSuccess)
          olap::group_part_agg_kernel<true><<<agg_grid, olap::kAggThreads, asmem, ctx->stream>>>(
              part_begin, d_units, rows, pp.slots, combine, capacity, out_keys, out_sums, out_counts, d_groups_u, overflow,
              d_partials);
      } else {
        auto* rows = reinterpret_cast<int2*>(rowbuf);
        if (e == cudaSuccess && tile_g == 4) scatter_tiled(rows, olap::group_part_scatter_tiled_kernel<false, 4>);
        else if (e == cudaSuccess && tile_g == 2) scatter_tiled(rows, olap::group_part_scatter_tiled_kernel<false, 2>);
        else if (e == cudaSuccess)
          olap::group_part_scatter_kernel<false><<<pp.n_blocks, 1024, psmem, ctx->stream>>>(pp, keys, vals,
                                                                                           nullptr, hist, cursor,
                                                                                           rows);
        if (e == cudaSuccess)
          olap::group_part_agg_kernel<false><<<agg_grid, olap::kAggThreads, asmem, ctx->stream>>>(
              part_begin, d_units, rows, pp.slots, combine, capacity, out_keys, out_sums, out_counts, d_groups_u, overflow,
              d_partials);
      }
      // a split partition has at least two slices
      if (e == cudaSuccess)
        olap::group_part_merge_kernel<<<ctx->sm_count, olap::kAggThreads, asmem, ctx->stream>>>(
            d_units, d_partials, pp.slots, capacity, out_keys, out_sums, out_counts, d_groups_u, overflow,
            &ctx->counters->wait_timeouts);
      if (e == cudaSuccess) e = cudaGetLastError();
    }
  }
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e != cudaSuccess && st == OLAP_OK) st = olap::check_cuda(ctx, e, "group_hash");
  unsigned long long ov[2] = {0, 0};
  if (st == OLAP_OK) cudaMemcpyAsync(ov, overflow, sizeof(ov), cudaMemcpyDeviceToHost, ctx->stream);
  OLAP_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
  if (st == OLAP_OK && ov[0]) return olap::set_error(ctx, OLAP_ERR_CAPACITY, "group hash table full");
  if (st == OLAP_OK && ov[1]) st = olap::check_timeouts(ctx, ctx->stream);
  return st;
}

int olap_agg_fixed(olap_ctx* ctx, int64_t n, const int32_t* price, const int32_t* qty,
                   const int32_t* tax_pct, int64_t* d_sum) {
  if (!ctx) return OLAP_ERR_INVALID;
  std::lock_guard<std::mutex> lk(ctx->mu);
  OLAP_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  OLAP_REQUIRE(ctx, n >= 0 && d_sum, "bad arguments");
  OLAP_REQUIRE(ctx, n == 0 || (price && qty && tax_pct), "null column");
  OLAP_CUDA_TRY(ctx, cudaMemsetAsync(d_sum, 0, sizeof(int64_t), ctx->stream));
  if (n == 0) return OLAP_OK;
  olap::agg_fixed_kernel<<<olap::grid_of(ctx, (n + 3) / 4, 512, 4), 512, 0, ctx->stream>>>(
      n, price, qty, tax_pct, reinterpret_cast<unsigned long long*>(d_sum));
  OLAP_CUDA_TRY(ctx, cudaGetLastError());
  return OLAP_OK;
}

int olap_agg_f64(olap_ctx* ctx, int64_t n, const double* tax, const double* qty, const double* price,
                 double* d_sum) {
  if (!ctx) return OLAP_ERR_INVALID;
  std::lock_guard<std::mutex> lk(ctx->mu);
  OLAP_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  OLAP_REQUIRE(ctx, n >= 0 && d_sum, "bad arguments");
  OLAP_REQUIRE(ctx, n == 0 || (tax && qty && price), "null column");
  olap::Arena ar(ctx);
  double* partial = ar.take<double>(olap::kAggF64Blocks);
  if (!partial) return olap::set_error(ctx, OLAP_ERR_CAPACITY, "scratch arena exhausted");
  olap::agg_f64_partial_kernel<<<olap::kAggF64Blocks, 256, 0, ctx->stream>>>(n, tax, qty, price, partial);
  olap::agg_f64_final_kernel<<<1, olap::kAggF64Blocks, 0, ctx->stream>>>(partial, d_sum);
  OLAP_CUDA_TRY(ctx, cudaGetLastError());
  return OLAP_OK;
}

}  // extern "C"
