// Dimension-vector builder and the batched multi-query star-join.
//
// The reference bakes each query's dimension vectors in its generator
// (include/gendata_util.hpp:449-542): entry k of table t is a group code when
// the dimension row passes the query's filter, else DIM_NULL.  Here dimension
// tables keep their attributes instead — an int32 filter attribute and an
// int32 group attribute per dimension row — and a query's predicate on a
// table is a range [lo, hi) on the filter attribute; its group code is the
// group attribute (or 0 when the table is not a group dimension).
//
// olap_build_dimvec materialises one query's int8 dimension vector from those
// attributes (the input of the plain star-join).
//
// The batched path runs up to 64 such queries in one persistent pass over
// the shared fact table:
//  * a table's filter attribute falls into one of at most 129 intervals between
//    the queries' range ends, and all rows of an interval pass the same
//    queries; so a batch gives each dimension row a 16-bit record, its interval
//    and its group attribute (9.2 MB for the four headline tables), and keeps
//    the query mask of each interval in shared memory;
//  * over the fact rows: each row's record is probed once per table (only
//    while some live query still uses the table), the intervals' masks are
//    ANDed with the mask of the queries whose fact range covers the row, and
//    only the queries left in the mask do per-query work (group id, one int64
//    atomic).
// Per query the result is bit-identical to the plain star-join over the
// dimension vectors that olap_build_dimvec builds for it.
#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <type_traits>
#include <vector>

#include "olap_internal.cuh"

namespace olap {

// Packed dimension attribute record: filter attribute (low word) and group
// attribute (high word).
__global__ void pack_dim_attrs_kernel(const int32_t* __restrict__ filt, const int32_t* __restrict__ grp,
                                      int64_t n, int2* __restrict__ out) {
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride)
    out[i] = make_int2(filt[i], grp ? grp[i] : 0);
}

__global__ void build_dimvec_kernel(const int32_t* __restrict__ filt, const int32_t* __restrict__ grp, int64_t n,
                                    int32_t lo, int32_t hi, int use_group, int8_t* __restrict__ out,
                                    unsigned long long* range_err) {
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  unsigned int bad = 0;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride) {
    const int32_t f = filt[i];
    int8_t v = static_cast<int8_t>(OLAP_DIM_NULL);
    if (f >= lo && f < hi) {
      const int32_t g = use_group ? grp[i] : 0;
      if (g < 0 || g >= OLAP_DIM_NULL) ++bad;  // not representable as a code
      else v = static_cast<int8_t>(g);
    }
    out[i] = v;
  }
  if (bad) atomicAdd(range_err, static_cast<unsigned long long>(bad));
}

// Device-side query descriptor of the batched kernel (one per query).
struct BatchQuery {
  int64_t row_begin, row_end;
  int32_t lo[OLAP_MAX_DIMS];      // filter range [lo, hi) per table
  int32_t hi[OLAP_MAX_DIMS];
  int32_t factor[OLAP_MAX_DIMS];  // group weight per table (0: not a group dimension)
  int32_t uses;                   // bit t: table t participates
  int32_t grouped;                // bit t: table t contributes its group attribute
  int64_t group_nums;
  int64_t out_offset;             // first slot of this query in the shared output
  int32_t smem_off;               // first slot of its per-block accumulators, or -1
  int32_t pad;
};

constexpr int kMaxBatchQueries = 64;
constexpr int kBatchSmemSlots = 4096;  // default per-block int64 accumulators (32 KiB); tunable
constexpr int kMaxSegments = 2 * kMaxBatchQueries + 2;

// Everything a batch uploads (one pinned staging copy per slot).
struct BatchDesc {
  BatchQuery q[kMaxBatchQueries];
  int64_t seg_begin[kMaxSegments];             // sorted; segment s = [seg_begin[s], seg_begin[s+1])
  unsigned long long seg_mask[kMaxSegments];   // queries whose fact range covers segment s
  unsigned long long uses_mask[OLAP_MAX_DIMS]; // queries using table t
  unsigned long long* out;                     // concatenated group vectors
  unsigned long long* totals;                  // [n_queries]
  int64_t out_total;                           // slots of out in use
  int32_t n_queries;
  int32_t n_seg;
};

// Intervals of a table's filter attribute: interval 0 lies below every query's
// range end, interval i from cut[i - 1] on.  mask[i]: the queries whose range
// on the table holds interval i (a query that does not use the table passes
// every row); mask[kIntervals + i]: the same without the queries that group by
// the table, for rows whose group attribute is no int8 code (DIM_NULL in the
// dimension vector the plain path builds).
constexpr int kMaxCuts = 2 * kMaxBatchQueries;
constexpr int kIntervals = kMaxCuts + 1;
struct BatchCuts {
  int32_t cut[OLAP_MAX_DIMS][kMaxCuts];  // ascending, INT32_MAX after the last
  int32_t n[OLAP_MAX_DIMS];
  int32_t pad[OLAP_MAX_DIMS];
  unsigned long long mask[OLAP_MAX_DIMS][2 * kIntervals];
};

// A dimension row: its interval (plus kIntervals without a group code) in the
// low 9 bits, its group code above.
constexpr int kRecordGroupShift = 9;
constexpr int kBatchStagedRows = 4096;  // records of the smallest table kept in shared memory up to this many

struct BatchParams {
  const int2* attrs[OLAP_MAX_DIMS];   // packed attribute records per table
  uint16_t* rec[OLAP_MAX_DIMS];       // per-batch records per table
  BatchCuts* cuts;
  uint32_t dim_len[OLAP_MAX_DIMS];
  const int32_t* fk[OLAP_MAX_DIMS];
  const int32_t* m1;
  const int32_t* m2;
  int64_t n_rows;
  const BatchDesc* desc;
  int32_t tables_used;                // union of the queries' `uses`
  int32_t probe_order;                // 4 x 2-bit table ids, smallest table first
  int32_t agg;                        // OLAP_AGG_* of every query (one aggregate)
  int32_t smem_slots;                 // per-block shared accumulators (dynamic shared memory)
  int32_t packed;                     // every factor fits 16 bits, every output offset 31
  int32_t vec;                        // the fact columns read start on 16-byte boundaries
  int32_t block;                      // threads per block of the scan (part of a recorded graph)
  unsigned long long* range_err;
};

constexpr int kBatchThreads = 512;     // default block size; tunable (128..1024)
constexpr int kBatchMaxThreads = 1024;
constexpr int kBatchMaxSmemSlots = 24576;  // 192 KiB

__device__ __forceinline__ int64_t batch_value(int agg, int32_t x, int32_t y) {
  switch (agg) {
    case OLAP_AGG_M1_PLUS_M2: return static_cast<int64_t>(x) + y;
    case OLAP_AGG_M1: return x;
    case OLAP_AGG_M2: return y;
    case OLAP_AGG_M1_TIMES_M2: return static_cast<int64_t>(x) * y;
    default: return 1;
  }
}

// The rows' records, table blockIdx.y: the interval by binary search among the
// cuts (64 range tests per row took 291 us for the four headline tables).
__global__ void __launch_bounds__(256) batch_records_kernel(const BatchParams p) {
  __shared__ int32_t s_cut[kMaxCuts];
  const int t = blockIdx.y;
  if (!((p.tables_used >> t) & 1)) return;
  const int64_t n = p.dim_len[t];
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  int64_t k = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (static_cast<int64_t>(blockIdx.x) * blockDim.x >= n) return;
  for (int i = threadIdx.x; i < kMaxCuts; i += blockDim.x) s_cut[i] = p.cuts->cut[t][i];
  const int nc = p.cuts->n[t];
  __syncthreads();
  for (; k < n; k += stride) {
    const int2 a = p.attrs[t][k];
    int at = 0;  // cuts <= the attribute
#pragma unroll
    for (int w = kMaxCuts / 2; w > 0; w >>= 1)
      if (s_cut[at + w - 1] <= a.x) at += w;
    at += s_cut[at] <= a.x;
    at = min(at, nc);
    const bool code_ok = static_cast<uint32_t>(a.y) < static_cast<uint32_t>(OLAP_DIM_NULL);
    p.rec[t][k] = static_cast<uint16_t>(code_ok ? at | a.y << kRecordGroupShift : at + kIntervals);
  }
}

// The fact pass: persistent, 4 rows per thread per step (128-bit loads).
// A random read costs L1 a cycle per lane whatever its size, so the smallest
// table's records are kept in shared memory when they are few; the others'
// share L2 with little else.  PAR = false: the tables are probed one after
// another, smallest first, each only for the rows that still have a live query
// using it (up to four dependent round trips per step).  PAR = true: every used
// table's record is read in one round trip (the union of a batch's predicates
// passes nearly every row, so the skipped probes save little); more registers,
// so at most 512 threads per block.
//
// Per surviving (row, query) one emission.  The row's group codes are the bytes
// of one word in probe order, so with factors of 16 bits (PACK) the group id
// is two dot products, and everything an emission needs of its query is one
// 16-byte shared read.  A lane's rows are ascending, so its fact-range segment
// only ever moves forward and its mask stays in registers.  For one or two
// queries (`few`, a loop of its own) a warp whose rows are in none of them makes
// no list: one query over 60M rows 588 us with the empty lists, 472 us without.
// With four queries the vote costs what it saves, with 64 it costs 1 %.
template <bool PAR, bool PACK>
__global__ void __launch_bounds__(PAR ? 512 : kBatchMaxThreads, 1) batch_scan_kernel(const BatchParams p) {
  __shared__ int64_t sseg[kMaxSegments];
  __shared__ unsigned long long smask[kMaxSegments];
  extern __shared__ unsigned long long sacc[];  // p.smem_slots per-block accumulators
  // Per query: its group factor at each probe position (0: not grouped; PACK:
  // four 16-bit ones in two words), its groups, and where they are: a shared
  // slot, or -1 - the offset in `out` (PACK), or {smem_off, offset} (!PACK).
  __shared__ int4 s_qf[kMaxBatchQueries];
  __shared__ int4 s_qi[PACK ? 1 : kMaxBatchQueries];
  constexpr int kQueue = 224;  // per warp; with the largest accumulators the block still fits an SM
  __shared__ uint16_t s_queue[PAR ? 16 : kBatchMaxThreads / 32][kQueue];
  __shared__ unsigned int s_bad;
  __shared__ unsigned long long s_int[OLAP_MAX_DIMS][2 * kIntervals];  // by probe position: interval -> query mask
  __shared__ uint16_t s_rec[kBatchStagedRows];                        // the first table's records
  const BatchDesc& D = *p.desc;
  unsigned long long* const out = D.out;
  const int tid = threadIdx.x;
  const int nq = D.n_queries, nseg = D.n_seg;
  // The used tables in probe order (smallest first).
  int tab[OLAP_MAX_DIMS] = {0, 0, 0, 0};
  uint32_t tlen[OLAP_MAX_DIMS] = {0, 0, 0, 0};
  unsigned long long tuses[OLAP_MAX_DIMS] = {0, 0, 0, 0};
  int ntab = 0;
#pragma unroll
  for (int o = 0; o < OLAP_MAX_DIMS; ++o) {
    const int t = (p.probe_order >> (2 * o)) & 3;
    if ((p.tables_used >> t) & 1) {
#pragma unroll
      for (int w = 0; w < OLAP_MAX_DIMS; ++w)
        if (w == ntab) {
          tab[w] = t;
          tlen[w] = p.dim_len[t];
          tuses[w] = D.uses_mask[t];
        }
      ++ntab;
    }
  }
  for (int i = tid; i < nq; i += blockDim.x) {
    const BatchQuery& Q = D.q[i];
    int32_t f[OLAP_MAX_DIMS] = {0, 0, 0, 0};
#pragma unroll
    for (int o = 0; o < OLAP_MAX_DIMS; ++o)
      if (o < ntab && ((Q.grouped >> tab[o]) & 1)) f[o] = Q.factor[tab[o]];
    if (PACK) {
      s_qf[i] = make_int4(f[0] | f[1] << 16, f[2] | f[3] << 16, static_cast<int32_t>(Q.group_nums),
                          Q.smem_off >= 0 ? Q.smem_off : -1 - static_cast<int32_t>(Q.out_offset));
    } else {
      s_qf[i] = make_int4(f[0], f[1], f[2], f[3]);
      s_qi[i] = make_int4(static_cast<int32_t>(Q.group_nums), Q.smem_off, static_cast<int32_t>(Q.out_offset),
                          static_cast<int32_t>(Q.out_offset >> 32));
    }
  }
  for (int i = tid; i < p.smem_slots; i += blockDim.x) sacc[i] = 0ull;
  for (int i = tid; i < nseg; i += blockDim.x) {
    sseg[i] = D.seg_begin[i];
    smask[i] = D.seg_mask[i];
  }
  if (tid == 0) s_bad = 0;
#pragma unroll
  for (int o = 0; o < OLAP_MAX_DIMS; ++o)
    for (int i = tid; o < ntab && i < 2 * kIntervals; i += blockDim.x) s_int[o][i] = p.cuts->mask[tab[o]][i];
  const bool staged = ntab > 0 && tlen[0] <= kBatchStagedRows;
  for (uint32_t i = tid; staged && i < tlen[0]; i += blockDim.x) s_rec[i] = p.rec[tab[0]][i];
  __syncthreads();
  const uint64_t pol_stream = policy_evict_first();
  const int agg = p.agg;
  const bool need_m1 = agg == OLAP_AGG_M1_PLUS_M2 || agg == OLAP_AGG_M1 || agg == OLAP_AGG_M1_TIMES_M2;
  const bool need_m2 = agg == OLAP_AGG_M1_PLUS_M2 || agg == OLAP_AGG_M2 || agg == OLAP_AGG_M1_TIMES_M2;
  unsigned int bad = 0;
  // one (row, query) pair: the row's packed codes c4 and value v
  auto emit = [&](int q, uint32_t c4, int64_t v) {
    const int4 f = s_qf[q];
    if (PACK) {
      const uint32_t g = __dp2a_hi(static_cast<uint32_t>(f.y), c4, __dp2a_lo(static_cast<uint32_t>(f.x), c4, 0u));
      if (g >= static_cast<uint32_t>(f.z)) {
        ++bad;
      } else if (f.w >= 0) {
        smem_add_split(reinterpret_cast<uint32_t*>(sacc), p.smem_slots, f.w + g, static_cast<uint64_t>(v));
      } else {
        atomicAdd(&out[static_cast<int64_t>(-1 - f.w) + g], static_cast<unsigned long long>(v));
      }
    } else {
      const int4 qi = s_qi[q];
      const int32_t g = static_cast<int32_t>(c4 & 255u) * f.x + static_cast<int32_t>((c4 >> 8) & 255u) * f.y +
                        static_cast<int32_t>((c4 >> 16) & 255u) * f.z + static_cast<int32_t>(c4 >> 24) * f.w;
      if (static_cast<uint32_t>(g) >= static_cast<uint32_t>(qi.x)) {
        ++bad;
      } else if (qi.y >= 0) {
        smem_add_split(reinterpret_cast<uint32_t*>(sacc), p.smem_slots, qi.y + g, static_cast<uint64_t>(v));
      } else {
        const int64_t base = (static_cast<int64_t>(qi.w) << 32) | static_cast<uint32_t>(qi.z);
        atomicAdd(&out[base + g], static_cast<unsigned long long>(v));
      }
    }
  };
  // The warp's 32 rows of one register slot: (row, query) pairs listed in
  // shared memory, then emitted 32 at a time with every lane busy.  (Each lane
  // emitting its own row's queries left 3 lanes busy on average: a row has
  // about one query, but some row of the 32 has four.)
  const int lane = tid & 31;
  uint16_t* queue = s_queue[tid >> 5];
  auto emit_rows = [&](auto few, unsigned long long mk, uint32_t c4, int32_t x, int32_t y) {
    if (decltype(few)::value && !__any_sync(0xffffffffu, mk != 0ull)) return;
    uint32_t lo = static_cast<uint32_t>(mk), hi = static_cast<uint32_t>(mk >> 32);
    const int cnt = __popc(lo) + __popc(hi);
    int inc = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int z = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += z;
    }
    const int all = __shfl_sync(0xffffffffu, inc, 31);
    if (all > kQueue) {  // more than the list holds
      const int64_t v = batch_value(agg, x, y);
      for (; lo; lo &= lo - 1) emit(__ffs(lo) - 1, c4, v);
      for (; hi; hi &= hi - 1) emit(__ffs(hi) + 31, c4, v);
      __syncwarp();
      return;
    }
    uint16_t* at = queue + (inc - cnt);
    for (; lo; lo &= lo - 1) *at++ = static_cast<uint16_t>(lane << 6 | (__ffs(lo) - 1));
    for (; hi; hi &= hi - 1) *at++ = static_cast<uint16_t>(lane << 6 | (__ffs(hi) + 31));
    __syncwarp();
    for (int b = 0; b < all; b += 32) {
      const uint32_t e = b + lane < all ? queue[b + lane] : 0u;
      const uint32_t c = __shfl_sync(0xffffffffu, c4, e >> 6);
      const int32_t xs = __shfl_sync(0xffffffffu, x, e >> 6), ys = __shfl_sync(0xffffffffu, y, e >> 6);
      if (b + lane < all) emit(static_cast<int>(e & 63u), c, batch_value(agg, xs, ys));
    }
    __syncwarp();
  };
  const int64_t n4 = (p.n_rows + 3) >> 2;
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  int seg = 0;                                           // segment of the step's first row
  int64_t seg_end = nseg > 1 ? sseg[1] : INT64_MAX;      // where it ends
  unsigned long long seg_mask = smask[0];
  // every lane of a warp runs the same steps (one past the end has no rows)
  auto scan_rows = [&](auto few) {
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + tid; i - lane < n4; i += stride) {
      const int64_t r0 = 4 * i;
      const int nv = r0 + 4 <= p.n_rows ? 4 : r0 < p.n_rows ? static_cast<int>(p.n_rows - r0) : 0;
      const bool full = nv == 4, vec = full && p.vec;  // vec: 16-byte loads, which must stay inside that guard
      // Arrays are indexed by probe position o (table t = tab[o]), so that
      // every index is a compile-time constant.
      int32_t key[OLAP_MAX_DIMS][4];
      int32_t x[4] = {0, 0, 0, 0}, y[4] = {0, 0, 0, 0};
#pragma unroll
      for (int o = 0; o < OLAP_MAX_DIMS; ++o) {
        if (o >= ntab) continue;
        const int32_t* f = p.fk[tab[o]];
        if (vec) {
          const int4 v = ld_stream_v4_ordered(f + r0, pol_stream);
          key[o][0] = v.x; key[o][1] = v.y; key[o][2] = v.z; key[o][3] = v.w;
        } else {
          for (int k = 0; k < 4; ++k) key[o][k] = k < nv ? f[r0 + k] : 0;
        }
      }
      if (need_m1) {
        if (vec) {
          const int4 v = ld_stream_v4_ordered(p.m1 + r0, pol_stream);
          x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w;
        } else {
#pragma unroll
          for (int k = 0; k < 4; ++k) x[k] = k < nv ? p.m1[r0 + k] : 0;
        }
      }
      if (need_m2) {
        if (vec) {
          const int4 v = ld_stream_v4_ordered(p.m2 + r0, pol_stream);
          y[0] = v.x; y[1] = v.y; y[2] = v.z; y[3] = v.w;
        } else {
#pragma unroll
          for (int k = 0; k < 4; ++k) y[k] = k < nv ? p.m2[r0 + k] : 0;
        }
      }
      // Queries whose fact range covers each row.
      while (seg_end <= r0) {
        ++seg;
        seg_end = seg + 1 < nseg ? sseg[seg + 1] : INT64_MAX;
        seg_mask = smask[seg];
      }
      unsigned long long m[4] = {seg_mask, seg_mask, seg_mask, seg_mask};
      if (!full || seg_end < r0 + 4) {
        int s = seg;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          while (s + 1 < nseg && sseg[s + 1] <= r0 + k) ++s;
          m[k] = k < nv ? smask[s] : 0ull;
        }
      }
      // A key out of range drops the row for the queries that use the table;
      // the table is not probed for it, and the row counts once per such query
      // when every other table the query uses passes it (as the plain path
      // counts: no in-range key of the query meets its filter's null).
      uint32_t inr = 0;  // bit 4*o + k: key[o][k] in range
#pragma unroll
      for (int k = 0; k < 4; ++k) {
#pragma unroll
        for (int o = 0; o < OLAP_MAX_DIMS; ++o) {
          if (o >= ntab) continue;
          if (static_cast<uint32_t>(key[o][k]) < tlen[o]) inr |= 1u << (4 * o + k);
        }
      }
      // queries that use a table whose key of row k is out of range
      auto oob_queries = [&](int k) -> unsigned long long {
        unsigned long long q = 0;
#pragma unroll
        for (int o = 0; o < OLAP_MAX_DIMS; ++o)
          if (o < ntab && !((inr >> (4 * o + k)) & 1u)) q |= tuses[o];
        return q;
      };
      uint32_t codes[4] = {0u, 0u, 0u, 0u};  // the row's group codes, a byte per probe position
      // the record of row k in table o, read while `want` (and its key is in range)
      auto record = [&](int o, int k, bool want) -> uint32_t {
        const bool in = want && ((inr >> (4 * o + k)) & 1u);
        if (o == 0 && staged) return s_rec[in ? key[0][k] : 0];
        return in ? __ldg(p.rec[tab[o]] + key[o][k]) : 0u;
      };
      // its interval's queries stay (all of them where the record was not wanted)
      auto apply = [&](int o, int k, uint32_t r, bool want) {
        const bool in = want && ((inr >> (4 * o + k)) & 1u);
        m[k] &= in ? s_int[o][r & ((1u << kRecordGroupShift) - 1u)] : ~0ull;
        codes[k] |= (r >> kRecordGroupShift) << (8 * o);
      };
      if (PAR) {
        uint32_t rec[OLAP_MAX_DIMS][4];
#pragma unroll
        for (int o = 0; o < OLAP_MAX_DIMS; ++o) {
          if (o >= ntab) continue;
#pragma unroll
          for (int k = 0; k < 4; ++k) rec[o][k] = record(o, k, m[k] != 0ull);
        }
#pragma unroll
        for (int o = 0; o < OLAP_MAX_DIMS; ++o) {
          if (o >= ntab) continue;
#pragma unroll
          for (int k = 0; k < 4; ++k) apply(o, k, rec[o][k], m[k] != 0ull);
        }
      } else {
        // breadth-first across the 4 rows; a table is probed for a row only
        // while a live query of the row uses it
#pragma unroll
        for (int o = 0; o < OLAP_MAX_DIMS; ++o) {
          if (o >= ntab) continue;
          const unsigned long long ut = tuses[o];
          uint32_t rec[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) rec[k] = record(o, k, (m[k] & ut) != 0ull);
#pragma unroll
          for (int k = 0; k < 4; ++k) apply(o, k, rec[k], (m[k] & ut) != 0ull);
        }
      }
      if (inr != (1u << (4 * ntab)) - 1u) {  // rare: some key out of range
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const unsigned long long oq = k < nv ? oob_queries(k) : 0ull;
          bad += __popcll(m[k] & oq);
          m[k] &= ~oq;
        }
      }
      // Per-query work only for the queries left in each row's mask.
      __syncwarp();
      emit_rows(few, m[0], codes[0], x[0], y[0]);
      emit_rows(few, m[1], codes[1], x[1], y[1]);
      emit_rows(few, m[2], codes[2], x[2], y[2]);
      emit_rows(few, m[3], codes[3], x[3], y[3]);
    }
  };
  if (nq <= 2) scan_rows(std::true_type{});
  else scan_rows(std::false_type{});
  const unsigned int wbad = __reduce_add_sync(0xffffffffu, bad);
  if ((tid & 31) == 0 && wbad) atomicAdd(&s_bad, wbad);
  __syncthreads();
  for (int q = 0; q < nq; ++q) {
    const BatchQuery& Q = D.q[q];
    if (Q.smem_off < 0) continue;
    for (int64_t g = tid; g < Q.group_nums; g += blockDim.x) {
      const unsigned long long v = smem_split_get(reinterpret_cast<const uint32_t*>(sacc), p.smem_slots,
                                                  Q.smem_off + g);
      if (v) atomicAdd(&out[Q.out_offset + g], v);
    }
  }
  if (tid == 0 && s_bad) atomicAdd(p.range_err, static_cast<unsigned long long>(s_bad));
}

// Intervals of table t (one block): the queries' range ends sorted by counting
// the smaller ones, then each interval's queries.
__device__ __forceinline__ void batch_cuts(const BatchParams& p, int t) {
  __shared__ int32_t s_lo[kMaxBatchQueries], s_hi[kMaxBatchQueries], s_cut[kMaxCuts];
  __shared__ unsigned long long s_uses, s_grouped;
  const BatchDesc& D = *p.desc;
  const int nq = D.n_queries;
  if (threadIdx.x == 0) s_uses = s_grouped = 0;
  for (int i = threadIdx.x; i < kMaxCuts; i += blockDim.x) s_cut[i] = INT32_MAX;
  __syncthreads();
  for (int q = threadIdx.x; q < nq; q += blockDim.x) {
    s_lo[q] = D.q[q].lo[t];
    s_hi[q] = D.q[q].hi[t];
    if ((D.q[q].uses >> t) & 1) atomicOr(&s_uses, 1ull << q);
    if ((D.q[q].grouped >> t) & 1) atomicOr(&s_grouped, 1ull << q);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 2 * nq; i += blockDim.x) {
    const int32_t v = i < nq ? s_lo[i] : s_hi[i - nq];
    int at = 0;
    for (int c = 0; c < 2 * nq; ++c) {
      const int32_t w = c < nq ? s_lo[c] : s_hi[c - nq];
      at += w < v || (w == v && c < i);
    }
    s_cut[at] = v;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < kMaxCuts; i += blockDim.x) p.cuts->cut[t][i] = s_cut[i];
  if (threadIdx.x == 0) p.cuts->n[t] = 2 * nq;
  const unsigned long long all = nq == 64 ? ~0ull : ((1ull << nq) - 1);
  for (int i = threadIdx.x; i <= 2 * nq; i += blockDim.x) {
    unsigned long long m = 0;
    if (i > 0) {
      const int32_t v = s_cut[i - 1];  // the interval's first value, when it holds any
      for (int q = 0; q < nq; ++q) m |= static_cast<unsigned long long>(s_lo[q] <= v && v < s_hi[q]) << q;
    }
    m = (m & s_uses) | (all & ~s_uses);
    p.cuts->mask[t][i] = m;
    p.cuts->mask[t][kIntervals + i] = m & ~(s_grouped & s_uses);
  }
}

// The tables' intervals (one block each), and zeroes in the batch's outputs
// (their location and size come with the descriptor, so a recorded graph
// serves any output buffer and query count).
__global__ void batch_zero_kernel(const BatchParams p) {
  if (blockIdx.x < OLAP_MAX_DIMS && ((p.tables_used >> blockIdx.x) & 1)) batch_cuts(p, blockIdx.x);
  const BatchDesc& D = *p.desc;
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  const int64_t t0 = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  for (int64_t i = t0; i < D.out_total; i += stride) D.out[i] = 0ull;
  for (int64_t i = t0; i < D.n_queries; i += stride) D.totals[i] = 0ull;
}

// totals[q] = sum of query q's group vector (one block per query).  Launched
// with max_queries blocks; blocks past the batch's count return.
__global__ void batch_totals_kernel(const BatchParams p) {
  __shared__ long long red[32];
  const BatchDesc& D = *p.desc;
  if (static_cast<int>(blockIdx.x) >= D.n_queries) return;
  const BatchQuery& Q = D.q[blockIdx.x];
  int64_t s = 0;
  for (int64_t g = threadIdx.x; g < Q.group_nums; g += blockDim.x) s += static_cast<int64_t>(D.out[Q.out_offset + g]);
  s = warp_sum_i64(s);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    long long v = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0;
    v = warp_sum_i64(v);
    if (threadIdx.x == 0) D.totals[blockIdx.x] = static_cast<unsigned long long>(v);
  }
}

static unsigned grid_n(const olap_ctx* ctx, int64_t n, int threads) {
  int64_t g = (n + threads - 1) / threads;
  const int64_t cap = static_cast<int64_t>(ctx->sm_count) * (2048 / threads);
  if (g > cap) g = cap;
  return static_cast<unsigned>(g < 1 ? 1 : g);
}

}  // namespace olap

// Batch handle: two staging slots (pinned host and device descriptors, one
// recorded graph each) so that one batch can be prepared while the previous
// one runs; packed attributes and 16-bit records per table.
struct olap_batch {
  olap_ctx* ctx = nullptr;
  int max_queries = 0;
  olap::BatchDesc* d_desc[2] = {};      // device
  olap::BatchDesc* h_desc[2] = {};      // pinned host staging
  cudaEvent_t done[2] = {};             // recorded after each slot's batch
  bool pending[2] = {false, false};
  cudaGraph_t graph[2] = {};
  cudaGraphExec_t exec[2] = {};
  olap::BatchParams params[2];
  bool have_params[2] = {false, false};
  int64_t runs = 0;
  int64_t captures = 0;                 // graphs recorded so far
  int2* attrs[OLAP_MAX_DIMS] = {};
  uint16_t* rec[OLAP_MAX_DIMS] = {};
  olap::BatchCuts* d_cuts[2] = {};      // device, per staging slot
  int64_t attr_len[OLAP_MAX_DIMS] = {};
  int block = olap::kBatchThreads;        // scan kernel block size (olap_batch_tune / _autotune)
  int smem_slots = olap::kBatchSmemSlots; // per-block shared accumulators
  int parallel_probe = 0;                 // 1: every table's record in one round trip (block <= 512)
};

extern "C" {

int olap_build_dimvec(olap_ctx* ctx, const int32_t* filter_attr, const int32_t* group_attr, int64_t n,
                      int32_t lo, int32_t hi, int use_group, int8_t* dimvec) {
  if (!ctx) return OLAP_ERR_INVALID;
  std::lock_guard<std::mutex> lk(ctx->mu);
  OLAP_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  OLAP_REQUIRE(ctx, n >= 0, "n must be >= 0");
  OLAP_REQUIRE(ctx, n == 0 || (filter_attr && dimvec && (!use_group || group_attr)), "null argument");
  if (n == 0) return OLAP_OK;
  olap::build_dimvec_kernel<<<olap::grid_n(ctx, n, 256), 256, 0, ctx->stream>>>(
      filter_attr, group_attr, n, lo, hi, use_group, dimvec, &ctx->counters->range_errors);
  OLAP_CUDA_TRY(ctx, cudaGetLastError());
  return OLAP_OK;
}

int olap_batch_create(olap_ctx* ctx, int max_queries, olap_batch** out) {
  if (!ctx || !out || max_queries < 1 || max_queries > olap::kMaxBatchQueries) return OLAP_ERR_INVALID;
  std::lock_guard<std::mutex> lk(ctx->mu);
  OLAP_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  olap_batch* b = new (std::nothrow) olap_batch();
  if (!b) return OLAP_ERR_NOMEM;
  b->ctx = ctx;
  b->max_queries = max_queries;
  bool ok = true;
  for (int s = 0; s < 2 && ok; ++s) {
    ok &= cudaMalloc(&b->d_desc[s], sizeof(olap::BatchDesc)) == cudaSuccess;
    ok &= cudaMallocHost(&b->h_desc[s], sizeof(olap::BatchDesc)) == cudaSuccess;
    ok &= cudaMalloc(&b->d_cuts[s], sizeof(olap::BatchCuts)) == cudaSuccess;
    ok &= cudaEventCreateWithFlags(&b->done[s], cudaEventDisableTiming) == cudaSuccess;
  }
  if (!ok) {
    cudaGetLastError();
    for (int s = 0; s < 2; ++s) {
      if (b->d_desc[s]) cudaFree(b->d_desc[s]);
      if (b->d_cuts[s]) cudaFree(b->d_cuts[s]);
      if (b->h_desc[s]) cudaFreeHost(b->h_desc[s]);
      if (b->done[s]) cudaEventDestroy(b->done[s]);
    }
    delete b;
    return OLAP_ERR_NOMEM;
  }
  *out = b;
  return OLAP_OK;
}

int olap_batch_destroy(olap_batch* b) {
  if (!b) return OLAP_ERR_INVALID;
  cudaSetDevice(b->ctx->device);
  for (int s = 0; s < 2; ++s) {
    if (b->pending[s]) cudaEventSynchronize(b->done[s]);
    if (b->exec[s]) cudaGraphExecDestroy(b->exec[s]);
    if (b->graph[s]) cudaGraphDestroy(b->graph[s]);
    cudaFree(b->d_desc[s]);
    cudaFree(b->d_cuts[s]);
    cudaFreeHost(b->h_desc[s]);
    cudaEventDestroy(b->done[s]);
  }
  for (int t = 0; t < OLAP_MAX_DIMS; ++t) {
    if (b->attrs[t]) cudaFree(b->attrs[t]);
    if (b->rec[t]) cudaFree(b->rec[t]);
  }
  delete b;
  return OLAP_OK;
}

int olap_batch_set_dimension(olap_batch* b, int table, const int32_t* filter_attr, const int32_t* group_attr,
                             int64_t n) {
  if (!b || table < 0 || table >= OLAP_MAX_DIMS || n < 1 || n > INT32_MAX || !filter_attr)
    return OLAP_ERR_INVALID;
  olap_ctx* ctx = b->ctx;
  std::lock_guard<std::mutex> lk(ctx->mu);
  OLAP_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  if (b->attr_len[table] != n) {
    for (int s = 0; s < 2; ++s)
      if (b->pending[s]) cudaEventSynchronize(b->done[s]);
    cudaStreamSynchronize(ctx->stream);
    if (b->attrs[table]) cudaFree(b->attrs[table]);
    if (b->rec[table]) cudaFree(b->rec[table]);
    b->attrs[table] = nullptr;
    b->rec[table] = nullptr;
    b->attr_len[table] = 0;
    OLAP_CUDA_TRY(ctx, cudaMalloc(&b->attrs[table], sizeof(int2) * n));
    OLAP_CUDA_TRY(ctx, cudaMalloc(&b->rec[table], sizeof(uint16_t) * n));
    b->attr_len[table] = n;
  }
  olap::pack_dim_attrs_kernel<<<olap::grid_n(ctx, n, 256), 256, 0, ctx->stream>>>(filter_attr, group_attr, n,
                                                                                 b->attrs[table]);
  OLAP_CUDA_TRY(ctx, cudaGetLastError());
  b->have_params[0] = b->have_params[1] = false;  // recorded graphs refer to the old buffers
  return OLAP_OK;
}

int olap_batch_graph_captures(olap_batch* b, int64_t* captures) {
  if (!b || !captures) return OLAP_ERR_INVALID;
  std::lock_guard<std::mutex> lk(b->ctx->mu);
  *captures = b->captures;
  return OLAP_OK;
}

int olap_batch_run(olap_batch* b, const olap_batch_query* queries, int n_queries, const int32_t* const* fk,
                   const int32_t* m1, const int32_t* m2, int64_t n_rows, int agg, int64_t* out,
                   int64_t out_slots, int64_t* totals, int use_graph) {
  if (!b) return OLAP_ERR_INVALID;
  olap_ctx* ctx = b->ctx;
  std::lock_guard<std::mutex> lk(ctx->mu);
  OLAP_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  OLAP_REQUIRE(ctx, n_queries >= 1 && n_queries <= b->max_queries && queries, "1..max_queries queries");
  OLAP_REQUIRE(ctx, n_rows >= 0 && out && totals && fk, "bad arguments");
  OLAP_REQUIRE(ctx, agg >= OLAP_AGG_M1_PLUS_M2 && agg <= OLAP_AGG_COUNT, "unknown aggregate");
  // The staging slot of this run; its previous batch must have finished
  // reading the pinned descriptors before they are overwritten.
  const int slot = static_cast<int>(b->runs & 1);
  if (b->pending[slot]) {
    OLAP_CUDA_TRY(ctx, cudaEventSynchronize(b->done[slot]));
    b->pending[slot] = false;
  }
  olap::BatchDesc& D = *b->h_desc[slot];
  std::memset(&D, 0, sizeof(D));
  int tables = 0;
  int64_t off = 0;
  std::vector<int64_t> cuts = {0, n_rows};
  for (int q = 0; q < n_queries; ++q) {
    const olap_batch_query& in = queries[q];
    olap::BatchQuery& d = D.q[q];
    OLAP_REQUIRE(ctx, in.row_begin >= 0 && in.row_end >= in.row_begin && in.row_end <= n_rows,
                 "query fact range outside the table");
    OLAP_REQUIRE(ctx, in.group_nums >= 1 && in.group_nums <= INT32_MAX, "group_nums must be in [1, 2^31)");
    d.row_begin = in.row_begin;
    d.row_end = in.row_end;
    d.group_nums = in.group_nums;
    d.out_offset = off;
    int64_t gbound = 0;
    for (int t = 0; t < OLAP_MAX_DIMS; ++t) {
      d.lo[t] = in.lo[t];
      d.hi[t] = in.hi[t];
      d.factor[t] = in.factor[t];
      if (in.uses & (1 << t)) {
        OLAP_REQUIRE(ctx, b->attrs[t] && fk[t], "query uses a table without attributes or fk column");
        d.uses |= 1 << t;
        D.uses_mask[t] |= 1ull << q;
        if (in.grouped & (1 << t)) {
          d.grouped |= 1 << t;
          gbound += 128 * std::llabs(static_cast<long long>(in.factor[t]));
        }
      }
    }
    OLAP_REQUIRE(ctx, gbound <= INT32_MAX, "group factors too large");
    tables |= d.uses;
    off += in.group_nums;
    cuts.push_back(in.row_begin);
    cuts.push_back(in.row_end);
  }
  OLAP_REQUIRE(ctx, off <= out_slots, "out holds fewer slots than the queries' groups");
  // Per-block shared accumulators for the queries with the fewest groups
  // (they see the most same-address atomics), as long as they fit.
  {
    std::vector<int> byg(n_queries);
    for (int q = 0; q < n_queries; ++q) byg[q] = q;
    std::stable_sort(byg.begin(), byg.end(), [&](int x, int y) { return D.q[x].group_nums < D.q[y].group_nums; });
    int64_t used = 0;
    for (int q : byg) {
      D.q[q].smem_off = -1;
      if (used + D.q[q].group_nums <= b->smem_slots) {
        D.q[q].smem_off = static_cast<int32_t>(used);
        used += D.q[q].group_nums;
      }
    }
  }
  // Fact-range segments: between consecutive cut points the set of queries
  // whose range covers a row is constant.
  std::sort(cuts.begin(), cuts.end());
  cuts.erase(std::unique(cuts.begin(), cuts.end()), cuts.end());
  int nseg = 0;
  for (size_t c = 0; c + 1 < cuts.size(); ++c) {
    unsigned long long m = 0;
    for (int q = 0; q < n_queries; ++q)
      if (D.q[q].row_begin <= cuts[c] && cuts[c + 1] <= D.q[q].row_end) m |= 1ull << q;
    D.seg_begin[nseg] = cuts[c];
    D.seg_mask[nseg] = m;
    ++nseg;
  }
  if (nseg == 0) {  // empty table
    D.seg_begin[0] = 0;
    D.seg_mask[0] = 0;
    nseg = 1;
  }
  D.n_queries = n_queries;
  D.n_seg = nseg;
  D.out = reinterpret_cast<unsigned long long*>(out);
  D.totals = reinterpret_cast<unsigned long long*>(totals);
  D.out_total = off;
  olap::BatchParams p;
  std::memset(&p, 0, sizeof(p));
  int order[OLAP_MAX_DIMS] = {0, 1, 2, 3};
  std::stable_sort(order, order + OLAP_MAX_DIMS, [&](int x, int y) { return b->attr_len[x] < b->attr_len[y]; });
  for (int o = 0; o < OLAP_MAX_DIMS; ++o) p.probe_order |= order[o] << (2 * o);
  for (int t = 0; t < OLAP_MAX_DIMS; ++t) {
    p.attrs[t] = b->attrs[t];
    p.rec[t] = b->rec[t];
    p.dim_len[t] = static_cast<uint32_t>(b->attr_len[t]);
    p.fk[t] = fk[t];
  }
  p.m1 = m1;
  p.m2 = m2;
  p.n_rows = n_rows;
  p.desc = b->d_desc[slot];
  p.cuts = b->d_cuts[slot];
  p.tables_used = tables;
  p.agg = agg;
  p.smem_slots = b->smem_slots;
  p.block = b->block;
  p.range_err = &ctx->counters->range_errors;
  const bool need_m1 = agg == OLAP_AGG_M1_PLUS_M2 || agg == OLAP_AGG_M1 || agg == OLAP_AGG_M1_TIMES_M2;
  const bool need_m2 = agg == OLAP_AGG_M1_PLUS_M2 || agg == OLAP_AGG_M2 || agg == OLAP_AGG_M1_TIMES_M2;
  OLAP_REQUIRE(ctx, n_rows == 0 || ((!need_m1 || m1) && (!need_m2 || m2)), "measure columns required");
  uintptr_t starts = (need_m1 ? reinterpret_cast<uintptr_t>(m1) : 0) | (need_m2 ? reinterpret_cast<uintptr_t>(m2) : 0);
  for (int t = 0; t < OLAP_MAX_DIMS; ++t)
    if ((tables >> t) & 1) starts |= reinterpret_cast<uintptr_t>(fk[t]);
  p.vec = (starts & 15) == 0;
  const size_t scan_smem = sizeof(unsigned long long) * static_cast<size_t>(b->smem_slots);
  const bool par = b->parallel_probe != 0 && b->block <= 512;
  // 16-bit factors and 31-bit output offsets (every batch but extreme ones)
  bool packed = off <= INT32_MAX;
  for (int q = 0; q < n_queries; ++q)
    for (int t = 0; t < OLAP_MAX_DIMS; ++t)
      if ((D.q[q].grouped >> t) & 1) packed &= D.q[q].factor[t] >= 0 && D.q[q].factor[t] <= UINT16_MAX;
  p.packed = packed;  // a recorded graph launches one kind of scan
  void (*scan)(const olap::BatchParams) =
      packed ? (par ? olap::batch_scan_kernel<true, true> : olap::batch_scan_kernel<false, true>)
             : (par ? olap::batch_scan_kernel<true, false> : olap::batch_scan_kernel<false, false>);
  OLAP_CUDA_TRY(ctx, cudaFuncSetAttribute(scan, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          static_cast<int>(scan_smem)));
  int bps = 1;
  OLAP_CUDA_TRY(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, scan, b->block, scan_smem));
  const unsigned grid = static_cast<unsigned>(ctx->sm_count) * static_cast<unsigned>(bps < 1 ? 1 : bps);
  // The work of one batch: descriptors H2D, zero outputs, query masks of the
  // used tables, one persistent pass over the fact table.
  auto enqueue = [&](cudaStream_t st) -> cudaError_t {
    cudaError_t e = cudaMemcpyAsync(b->d_desc[slot], b->h_desc[slot], sizeof(olap::BatchDesc),
                                    cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) {
      olap::batch_zero_kernel<<<static_cast<unsigned>(ctx->sm_count) * 2, 512, 0, st>>>(p);
      e = cudaGetLastError();
    }
    int64_t longest = 0;
    for (int t = 0; t < OLAP_MAX_DIMS; ++t)
      if ((tables >> t) & 1) longest = std::max(longest, b->attr_len[t]);
    if (e == cudaSuccess && longest) {
      olap::batch_records_kernel<<<dim3(olap::grid_n(ctx, longest, 256), OLAP_MAX_DIMS), 256, 0, st>>>(p);
      e = cudaGetLastError();
    }
    if (e == cudaSuccess && n_rows > 0) {
      scan<<<grid, b->block, scan_smem, st>>>(p);
      e = cudaGetLastError();
    }
    if (e == cudaSuccess) {
      olap::batch_totals_kernel<<<b->max_queries, 256, 0, st>>>(p);
      e = cudaGetLastError();
    }
    return e;
  };
  if (!use_graph) {
    OLAP_CUDA_TRY(ctx, enqueue(ctx->stream));
  } else {
    // Graph of this slot: re-captured when the launch parameters (tables,
    // fact columns, aggregate) change, replayed otherwise.  Queries, output
    // buffers and their sizes travel in the descriptor its copy node reads
    // from the slot's pinned staging.
    const bool same = b->have_params[slot] && b->exec[slot] && std::memcmp(&b->params[slot], &p, sizeof(p)) == 0;
    if (!same) {
      if (b->exec[slot]) cudaGraphExecDestroy(b->exec[slot]);
      if (b->graph[slot]) cudaGraphDestroy(b->graph[slot]);
      b->exec[slot] = nullptr;
      b->graph[slot] = nullptr;
      b->have_params[slot] = false;
      cudaStream_t cs;
      OLAP_CUDA_TRY(ctx, cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking));
      cudaError_t e = cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal);
      if (e == cudaSuccess) {
        cudaError_t e2 = enqueue(cs);
        e = cudaStreamEndCapture(cs, &b->graph[slot]);
        if (e == cudaSuccess) e = e2;
      }
      if (e == cudaSuccess) e = cudaGraphInstantiate(&b->exec[slot], b->graph[slot], 0);
      cudaStreamDestroy(cs);
      if (e != cudaSuccess) return olap::check_cuda(ctx, e, "batch graph capture");
      b->params[slot] = p;
      b->have_params[slot] = true;
      ++b->captures;
    }
    OLAP_CUDA_TRY(ctx, cudaGraphLaunch(b->exec[slot], ctx->stream));
  }
  OLAP_CUDA_TRY(ctx, cudaEventRecord(b->done[slot], ctx->stream));
  b->pending[slot] = true;
  ++b->runs;
  return OLAP_OK;
}

int olap_batch_tune(olap_batch* b, int block, int smem_slots) {
  if (!b) return OLAP_ERR_INVALID;
  olap_ctx* ctx = b->ctx;
  std::lock_guard<std::mutex> lk(ctx->mu);
  OLAP_REQUIRE(ctx, block >= 128 && block <= olap::kBatchMaxThreads && block % 32 == 0,
               "block must be a multiple of 32 in [128, 1024]");
  OLAP_REQUIRE(ctx, smem_slots >= 0 && smem_slots <= olap::kBatchMaxSmemSlots,
               "smem_slots must be in [0, 24576]");
  b->block = block;
  b->smem_slots = smem_slots;
  return OLAP_OK;
}

int olap_batch_set_probe(olap_batch* b, int parallel_probe) {
  if (!b || (parallel_probe != 0 && parallel_probe != 1)) return OLAP_ERR_INVALID;
  std::lock_guard<std::mutex> lk(b->ctx->mu);
  b->parallel_probe = parallel_probe;
  return OLAP_OK;
}

int olap_batch_get_tuning(olap_batch* b, int* block, int* smem_slots, int* parallel_probe) {
  if (!b) return OLAP_ERR_INVALID;
  std::lock_guard<std::mutex> lk(b->ctx->mu);
  if (block) *block = b->block;
  if (smem_slots) *smem_slots = b->smem_slots;
  if (parallel_probe) *parallel_probe = (b->parallel_probe && b->block <= 512) ? 1 : 0;
  return OLAP_OK;
}

int olap_batch_autotune(olap_batch* b, const olap_batch_query* queries, int n_queries,
                        const int32_t* const* fk, const int32_t* m1, const int32_t* m2, int64_t n_rows,
                        int agg, int64_t* out, int64_t out_slots, int64_t* totals, int64_t sample_rows,
                        int* best_block, int* best_slots, double* best_ms) {
  if (!b || !queries || n_queries < 1 || n_queries > b->max_queries) return OLAP_ERR_INVALID;
  olap_ctx* ctx = b->ctx;
  if (sample_rows <= 0) sample_rows = int64_t(64) << 20;
  const int64_t rows = std::min(n_rows, sample_rows);
  // The queries' fact ranges scaled onto the sample's rows [0, rows), so the
  // sample sees the same mix of live queries per row as the whole table (a
  // prefix cut would drop the queries whose ranges start past it, and the
  // shape that wins on fewer queries is not the one that wins on all).
  std::vector<olap_batch_query> qs(queries, queries + n_queries);
  const double scale = n_rows > rows ? static_cast<double>(rows) / static_cast<double>(n_rows) : 1.0;
  for (auto& q : qs) {
    const int64_t lo = std::min<int64_t>(rows, static_cast<int64_t>(static_cast<double>(q.row_begin) * scale));
    const int64_t hi = std::min<int64_t>(rows, static_cast<int64_t>(static_cast<double>(q.row_end) * scale));
    q.row_begin = std::max<int64_t>(0, lo);
    q.row_end = std::max<int64_t>(q.row_begin, hi);
  }
  cudaEvent_t e0, e1;
  {
    std::lock_guard<std::mutex> lk(ctx->mu);
    OLAP_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
    OLAP_CUDA_TRY(ctx, cudaEventCreate(&e0));
    OLAP_CUDA_TRY(ctx, cudaEventCreate(&e1));
  }
  unsigned long long errs_before = 0;
  cudaMemcpyAsync(&errs_before, &ctx->counters->range_errors, sizeof(errs_before), cudaMemcpyDeviceToHost,
                  ctx->stream);
  cudaStreamSynchronize(ctx->stream);
  const int saved_block = b->block, saved_slots = b->smem_slots, saved_probe = b->parallel_probe;
  double best = 1e30;
  int bb = saved_block, bs = saved_slots, bp = saved_probe;
  for (int probe : {0, 1})
  for (int block : {256, 512, 1024}) {
    if (probe && block > 512) continue;
    for (int slots : {0, 2048, 4096, 8192, 16384}) {
      b->block = block;
      b->smem_slots = slots;
      b->parallel_probe = probe;
      float ms = 0.f, best_c = 1e30f;
      bool ok = true;
      for (int rep = 0; rep < 3 && ok; ++rep) {
        cudaEventRecord(e0, ctx->stream);
        const int st = olap_batch_run(b, qs.data(), n_queries, fk, m1, m2, rows, agg, out, out_slots, totals, 0);
        cudaEventRecord(e1, ctx->stream);
        if (st != OLAP_OK || cudaEventSynchronize(e1) != cudaSuccess) {
          cudaGetLastError();
          ok = false;
          break;
        }
        cudaEventElapsedTime(&ms, e0, e1);
        if (rep > 0) best_c = std::min(best_c, ms);  // the first run warms caches
      }
      if (ok && best_c < best) {
        best = best_c;
        bb = block;
        bs = slots;
        bp = probe;
      }
    }
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  // Rows the timed runs dropped were counted; restore the earlier count.
  cudaMemcpyAsync(&ctx->counters->range_errors, &errs_before, sizeof(errs_before), cudaMemcpyHostToDevice,
                  ctx->stream);
  cudaStreamSynchronize(ctx->stream);
  if (best >= 1e29) {
    b->block = saved_block;
    b->smem_slots = saved_slots;
    b->parallel_probe = saved_probe;
    return olap::set_error(ctx, OLAP_ERR_CUDA, "no batch autotune candidate ran");
  }
  b->block = bb;
  b->smem_slots = bs;
  b->parallel_probe = bp;
  if (best_block) *best_block = bb;
  if (best_slots) *best_slots = bs;
  if (best_ms) *best_ms = best;
  return OLAP_OK;
}

}  // extern "C"
