// Select, project and gather operators for sm_100a.
//
// Reference: code/select/test_select_option.cpp (predicate `col <= val` in
// every sel_lt_T_* primitive, :28-440; the 3-predicate driver selalgo_rowwise
// :450-467) and code/project/test_project_option.cpp (pairs (Ra, Rc) of the
// rows where Ra <= c and Rc <= c, :34-864).  Selection vectors are int32 row
// ids in ascending order, produced from a bitmap by the mark and expansion
// kernels of compact.cuh; bitmaps hold bit i of row i at byte i/8, bit
// i%8 (the storage order of a little-endian std::vector<bool>).
#include <algorithm>
#include <cstring>

#include "compact.cuh"

namespace olap {

// cmp(col, val) as col <= val: col < val is col <= val - 1, and nothing is
// below INT32_MIN.
struct LePred {
  int32_t val;
  int none;
  LePred(int32_t v, int cmp) : val(cmp == OLAP_CMP_LT && v != INT32_MIN ? v - 1 : v), none(cmp == OLAP_CMP_LT && v == INT32_MIN) {}
};

__device__ __forceinline__ int32_t lane4(const int4& v, int k) {
  return k == 0 ? v.x : k == 1 ? v.y : k == 2 ? v.z : v.w;
}

// Marks of cmp(col[r], val) over the column; a warp takes whole tiles.  Bound by
// the column read: full tiles of an aligned column (kVec) take four 16-byte
// loads per lane at a time, and two lanes' 4-bit results make one byte of the
// bitmap (row order, no ballots).  An unaligned column takes 128 rows at a
// time, lane l the rows 32 u + l, so that a ballot is a word and four loads are
// in flight (2^27 rows to a bitmap: 460 us with one row per lane and step,
// 154 us so).  The predicate is col <= val (the caller turns < into it), none
// when `none`.  counts may be null (the bitmap alone).
template <bool kVec>
__global__ void __launch_bounds__(512) select_mark_kernel(const int32_t* __restrict__ col, int64_t n, int32_t val,
                                                          int none, uint32_t* __restrict__ bits,
                                                          uint32_t* __restrict__ counts, int32_t tile,
                                                          int64_t n_tiles) {
  const int lane = threadIdx.x & 31;
  const int64_t n_warps = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
  const uint64_t pol = policy_evict_first();
  const uint32_t keep = none ? 0u : 15u;
  for (int64_t t = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5; t < n_tiles; t += n_warps) {
    const int64_t first = t * tile;
    const int64_t end = first + tile < n ? first + tile : n;
    uint32_t c = 0;
    if (kVec && first + tile <= n) {
      const int32_t* src = col + first + 4 * lane;
      unsigned char* dst = reinterpret_cast<unsigned char*>(bits) + (first >> 3) + (lane >> 1);
      auto put = [&](const int4 v, int at) {
        uint32_t m = static_cast<uint32_t>(v.x <= val) | static_cast<uint32_t>(v.y <= val) << 1 |
                     static_cast<uint32_t>(v.z <= val) << 2 | static_cast<uint32_t>(v.w <= val) << 3;
        m &= keep;
        c += __popc(m);
        m |= __shfl_down_sync(0xffffffffu, m, 1) << 4;
        if (!(lane & 1)) dst[at >> 3] = static_cast<unsigned char>(m);
      };
      int at = 0;
      for (; at + 512 <= tile; at += 512) {
        int4 v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) v[u] = ld_stream_v4_ordered(src + at + 128 * u, pol);
#pragma unroll
        for (int u = 0; u < 4; ++u) put(v[u], at + 128 * u);
      }
      for (; at < tile; at += 128) put(ld_stream_v4_ordered(src + at, pol), at);
    } else {
      constexpr int G = kVec ? 1 : 4;  // words at a time (kVec: only the last tile comes here)
      for (int64_t r0 = first; r0 < end; r0 += 32 * G) {
        int32_t v[G];
#pragma unroll
        for (int u = 0; u < G; ++u)
          v[u] = ld_stream_s32_if(r0 + 32 * u + lane < end, col + r0 + 32 * u + lane, pol, 0);
#pragma unroll
        for (int u = 0; u < G; ++u) {
          const uint32_t word = __ballot_sync(0xffffffffu, v[u] <= val && !none && r0 + 32 * u + lane < end);
          if (lane == 0 && r0 + 32 * u < end) {
            bits[(r0 >> 5) + u] = word;
            c += __popc(word);
          }
        }
      }
    }
    if (counts) {
      c = __reduce_add_sync(0xffffffffu, c);
      if (lane == 0) counts[t] = c;
    }
  }
}

// Selected rows: their ids.
struct RowEmit {
  static constexpr bool kVals = false;
  int32_t* out;
  __device__ __forceinline__ void emit(int64_t pos, int64_t item, int64_t) const { out[pos] = static_cast<int32_t>(item); }
};

// Refinement of a selection vector: the passing entries of each tile go to
// `vals` (those of tile t from element t * tile on), from where they are
// copied to the output once their positions are known (run_copy_kernel).  By
// then no block reads the vector any more, so the output may be the vector
// itself.  Lane l takes the entries 32 u + l of a step, whose rows are close
// when the vector is dense.  Bound by the latency of the two dependent reads:
// the next step's entries load while this one's rows are looked up (2^27
// entries, all rows in order, 30 % pass, with the copy: 500 us in one pass with
// look-back, 644 us with one entry per lane and step, 356 us so; every tenth
// row: 174, 174 and 150 us a call).
__global__ void __launch_bounds__(512, 3) select_refine_kernel(const int32_t* __restrict__ col, uint32_t col_len,
                                                               const int32_t* __restrict__ in_rowids, int32_t val,
                                                               int none, const Marks mk,
                                                               unsigned long long* range_err) {
  const int lane = threadIdx.x & 31;
  const uint32_t lt = (1u << lane) - 1u;
  const int n_warps = static_cast<int>((gridDim.x * blockDim.x) >> 5);
  const uint64_t pol = policy_evict_first();
  const uint32_t keep = none ? 0u : 15u;
  const int32_t* const at = col_len ? col : in_rowids;  // an entry outside the column looks up its first word
  unsigned int bad = 0;
  for (int t = static_cast<int>((blockIdx.x * blockDim.x + threadIdx.x) >> 5); t < mk.n_tiles; t += n_warps) {
    const int64_t first = static_cast<int64_t>(t) * mk.tile;
    const int len = static_cast<int>(first + mk.tile < mk.n ? mk.tile : mk.n - first);
    const int whole = len & ~127;  // entries in full steps: all but the chunk's last
    const int32_t* src = in_rowids + first + lane;
    int32_t* vals = static_cast<int32_t*>(mk.vals) + first;
    uint32_t c = 0;
    int32_t next[4];
    auto load_next = [&](int r) {
      if (r < whole) {
#pragma unroll
        for (int u = 0; u < 4; ++u) next[u] = ld_stream_s32(src + r + 32 * u, pol);
      } else {
#pragma unroll
        for (int u = 0; u < 4; ++u) next[u] = ld_stream_s32_if(r + 32 * u + lane < len, src + r + 32 * u, pol, 0);
      }
    };
    load_next(0);
    for (int r = 0; r < len; r += 128) {
      uint32_t has = 15u;
      if (r >= whole) {
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (r + 32 * u + lane >= len) has &= ~(1u << u);
      }
      int32_t row[4], v[4];
      uint32_t in = 0;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        row[u] = next[u];
        in |= static_cast<uint32_t>(static_cast<uint32_t>(row[u]) < col_len) << u;
      }
      in &= has;
      bad += __popc(has ^ in);  // not rows of col: dropped and counted
#pragma unroll
      for (int u = 0; u < 4; ++u) v[u] = __ldg(at + ((in >> u) & 1u ? row[u] : 0));
      if (r + 128 < len) load_next(r + 128);
      in &= keep;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const bool pass = ((in >> u) & 1u) && v[u] <= val;
        const uint32_t w = __ballot_sync(0xffffffffu, pass);
        if (pass) vals[c + __popc(w & lt)] = row[u];
        c += __popc(w);
      }
    }
    if (lane == 0) mk.counts[t] = c;
  }
  if (bad) atomicAdd(range_err, static_cast<unsigned long long>(bad));
}

// Rows where Ra <= c and Rc <= c; writes the pair (Ra, Rc).
struct ProjectOp {
  static constexpr int kGroups = kCompactGroups;
  const int32_t* ra;
  const int32_t* rc;
  int32_t* out_a;
  int32_t* out_c;
  int32_t cond;
  int32_t vec;
  int4 a[kCompactGroups], c[kCompactGroups];

  __device__ __forceinline__ bool vec_ok() const { return vec != 0; }
  __device__ __forceinline__ void prefetch(int u, int64_t first) {
    a[u] = ld_stream_v4(ra + first, policy_evict_first());
    c[u] = ld_stream_v4(rc + first, policy_evict_first());
  }
  template <bool kFull>
  __device__ __forceinline__ uint32_t flags(int u, int64_t first, int nv) {
    const uint64_t pol = policy_evict_first();
    if (kFull) {
      // a[u], c[u] loaded by prefetch()
    } else if (vec && nv == 4) {
      a[u] = ld_stream_v4(ra + first, pol);
      c[u] = ld_stream_v4(rc + first, pol);
    } else {
      int32_t x[4] = {0, 0, 0, 0}, y[4] = {0, 0, 0, 0};
      for (int k = 0; k < nv; ++k) {
        x[k] = ra[first + k];
        y[k] = rc[first + k];
      }
      a[u] = make_int4(x[0], x[1], x[2], x[3]);
      c[u] = make_int4(y[0], y[1], y[2], y[3]);
    }
    uint32_t m = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (k < nv) m |= static_cast<uint32_t>(lane4(a[u], k) <= cond && lane4(c[u], k) <= cond) << k;
    return m;
  }
  __device__ __forceinline__ void emit(int u, int k, int64_t, int64_t pos) {
    out_a[pos] = lane4(a[u], k);
    out_c[pos] = lane4(c[u], k);
  }
};

// Rows of a row store (an array of structs, row_bytes apart): the pair (Ra,
// Rc) read as int32 at byte offsets off_a and off_c of each row, for the rows
// where both are <= c (proalgo_rowwise over row_store_min / row_store_max,
// project/test_project_option.cpp:34-147).  Rows are not 16-byte vectors, so
// every group takes the per-row loads.
struct ProjectRowsOp {
  static constexpr int kGroups = kCompactGroups;
  const unsigned char* rows;
  int64_t row_bytes;
  int32_t off_a, off_c;
  int32_t* out_a;
  int32_t* out_c;
  int32_t cond;
  int4 a[kCompactGroups], c[kCompactGroups];

  __device__ __forceinline__ bool vec_ok() const { return false; }
  __device__ __forceinline__ void prefetch(int, int64_t) {}
  template <bool kFull>
  __device__ __forceinline__ uint32_t flags(int u, int64_t first, int nv) {
    int32_t x[4] = {0, 0, 0, 0}, y[4] = {0, 0, 0, 0};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (k >= nv) continue;
      const unsigned char* r = rows + (first + k) * row_bytes;
      x[k] = __ldg(reinterpret_cast<const int32_t*>(r + off_a));
      y[k] = __ldg(reinterpret_cast<const int32_t*>(r + off_c));
    }
    a[u] = make_int4(x[0], x[1], x[2], x[3]);
    c[u] = make_int4(y[0], y[1], y[2], y[3]);
    uint32_t m = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (k < nv) m |= static_cast<uint32_t>(x[k] <= cond && y[k] <= cond) << k;
    return m;
  }
  __device__ __forceinline__ void emit(int u, int k, int64_t, int64_t pos) {
    out_a[pos] = lane4(a[u], k);
    out_c[pos] = lane4(c[u], k);
  }
};

// SUM(Rd) and COUNT over rows with Ra, Rb, Rc all <= condition.
__global__ void __launch_bounds__(512) selalgo_kernel(int32_t cond, int64_t n, const int32_t* __restrict__ ra,
                                                      const int32_t* __restrict__ rb, const int32_t* __restrict__ rc,
                                                      const int32_t* __restrict__ rd, int vec,
                                                      unsigned long long* sum, unsigned long long* count) {
  __shared__ long long s_red[16][2];
  const uint64_t pol = policy_evict_first();
  int64_t s = 0, c = 0;
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  const int64_t tid = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  const int64_t n4 = vec ? n >> 2 : 0;
  for (int64_t i = tid; i < n4; i += stride) {
    const int4 a = ld_stream_v4(ra + 4 * i, pol), b = ld_stream_v4(rb + 4 * i, pol);
    const int4 cc = ld_stream_v4(rc + 4 * i, pol), d = ld_stream_v4(rd + 4 * i, pol);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const bool p = lane4(a, k) <= cond && lane4(b, k) <= cond && lane4(cc, k) <= cond;
      s += p ? lane4(d, k) : 0;
      c += p;
    }
  }
  for (int64_t r = 4 * n4 + tid; r < n; r += stride) {
    const bool p = ra[r] <= cond && rb[r] <= cond && rc[r] <= cond;
    s += p ? rd[r] : 0;
    c += p;
  }
  s = warp_sum_i64(s);
  c = warp_sum_i64(c);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) {
    s_red[warp][0] = s;
    s_red[warp][1] = c;
  }
  __syncthreads();
  if (warp == 0) {
    long long x = lane < static_cast<int>(blockDim.x >> 5) ? s_red[lane][0] : 0;
    long long y = lane < static_cast<int>(blockDim.x >> 5) ? s_red[lane][1] : 0;
    x = warp_sum_i64(x);
    y = warp_sum_i64(y);
    if (lane == 0) {
      if (x) atomicAdd(sum, static_cast<unsigned long long>(x));
      if (y) atomicAdd(count, static_cast<unsigned long long>(y));
    }
  }
}

constexpr int kMaxGatherCols = 8;
struct GatherParams {
  const int32_t* cols[kMaxGatherCols];
  int32_t* outs[kMaxGatherCols];
  unsigned long long* range_err;
  int64_t col_len;
  int ncols;
};

// outs[c][i] = cols[c][rowids[i]]; a row id outside [0, col_len) yields 0 and
// is counted.  Row ids close together: four neighbours per thread, 16-byte
// loads of the ids and stores of the values.  Bound by DRAM (nearly every
// line of the columns is read).
__global__ void gather_dense_kernel(const int32_t* __restrict__ rowids, int64_t k, const GatherParams gp, int vec) {
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  const int64_t tid = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  const uint64_t pol = policy_evict_first();
  const int64_t k4 = vec ? k >> 2 : 0;
  unsigned int bad = 0;
  auto ok = [&](int32_t r) { return r >= 0 && r < gp.col_len; };
  for (int64_t i = tid; i < k4; i += stride) {
    const int4 r = ld_stream_v4(rowids + 4 * i, pol);
    const bool ox = ok(r.x), oy = ok(r.y), oz = ok(r.z), ow = ok(r.w);
    bad += !ox + !oy + !oz + !ow;
    for (int c = 0; c < gp.ncols; ++c) {
      const int32_t* col = gp.cols[c];
      int4 v;
      v.x = ox ? __ldg(col + r.x) : 0;
      v.y = oy ? __ldg(col + r.y) : 0;
      v.z = oz ? __ldg(col + r.z) : 0;
      v.w = ow ? __ldg(col + r.w) : 0;
      reinterpret_cast<int4*>(gp.outs[c])[i] = v;
    }
  }
  for (int64_t j = 4 * k4 + tid; j < k; j += stride) {
    const int32_t r = rowids[j];
    const bool o = ok(r);
    bad += !o;
    for (int c = 0; c < gp.ncols; ++c) gp.outs[c][j] = o ? __ldg(gp.cols[c] + r) : 0;
  }
  if (bad) atomicAdd(gp.range_err, static_cast<unsigned long long>(bad));
}

// Row ids far apart: a lane per row id, so that the values of a warp's 32
// neighbours lie in as few lines as their rows do (a load costs L1 a cycle
// per line; four neighbours per lane spread every load over 32 lines), four
// row ids per thread in flight, and a 64-byte fetch on an L2 miss (the rest of
// a larger one is rarely used).
// 2^28-row columns, 4 of them, before (four neighbours per lane, 64-byte
// fetches only above 16 rows apart) and now: 439 and 286 us at 3 % of the
// rows, 704 and 623 us at 10 %.
__global__ void __launch_bounds__(256) gather_sparse_kernel(const int32_t* __restrict__ rowids, int64_t k,
                                                            const GatherParams gp) {
  const int64_t step = 4 * static_cast<int64_t>(blockDim.x);
  const uint64_t pol = policy_evict_first();
  unsigned int bad = 0;
  for (int64_t b = static_cast<int64_t>(blockIdx.x) * step + threadIdx.x; b < k; b += gridDim.x * step) {
    int32_t r[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int64_t i = b + u * static_cast<int64_t>(blockDim.x);
      r[u] = ld_stream_s32_if(i < k, rowids + i, pol, 0);
      if (i < k && (r[u] < 0 || r[u] >= gp.col_len)) {
        ++bad;
        r[u] = -1;
      }
    }
    for (int c = 0; c < gp.ncols; ++c) {
      const int32_t* col = gp.cols[c];
      int32_t v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int64_t i = b + u * static_cast<int64_t>(blockDim.x);
        v[u] = i < k && r[u] >= 0 ? ld_gather_64(col + r[u]) : 0;
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int64_t i = b + u * static_cast<int64_t>(blockDim.x);
        if (i < k) gp.outs[c][i] = v[u];
      }
    }
  }
  if (bad) atomicAdd(gp.range_err, static_cast<unsigned long long>(bad));
}

static bool al16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

template <class Op>
static int run_compaction(olap_ctx* ctx, const Op& op, int64_t n_items, int64_t* d_count) {
  Arena ar(ctx);
  ScanTiles st;
  unsigned long long* total = d_count ? reinterpret_cast<unsigned long long*>(d_count)
                                      : ar.take<unsigned long long>(1);
  if (!total) return set_error(ctx, OLAP_ERR_CAPACITY, "scratch arena exhausted");
  int rc = make_scan_tiles(ctx, ar, n_items, total, ctx->stream, &st, compact_tile_items<Op>());
  if (rc != OLAP_OK) return rc;
  compact_kernel<Op><<<compact_grid(ctx, st.n_tiles), kCompactThreads, 0, ctx->stream>>>(op, n_items, st);
  OLAP_CUDA_TRY(ctx, cudaGetLastError());
  return OLAP_OK;
}

// Look-back of tile 1 while tile 0's status is never published: the wait
// runs out after spin_limit polls (the failure path of every compaction).
__global__ void lookback_timeout_kernel(ScanTiles st, uint32_t spin_limit, long long* out) {
  const int64_t b = lookback(st, 1, 1, spin_limit);
  if (threadIdx.x == 0) *out = b;
}

static unsigned stream_grid(const olap_ctx* ctx, int64_t items, int threads) {
  int64_t g = (items + threads - 1) / threads;
  const int64_t cap = static_cast<int64_t>(ctx->sm_count) * (2048 / threads);
  if (g > cap) g = cap;
  return static_cast<unsigned>(g < 1 ? 1 : g);
}

}  // namespace olap

extern "C" {

int olap_select_rowids(olap_ctx* ctx, const int32_t* col, int64_t col_len, int32_t val, int cmp,
                       const int32_t* in_rowids, int64_t n_in, int32_t* out_rowids, int64_t* d_count) {
  if (!ctx) return OLAP_ERR_INVALID;
  std::lock_guard<std::mutex> lk(ctx->mu);
  OLAP_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  const int64_t n = in_rowids ? n_in : col_len;
  OLAP_REQUIRE(ctx, col_len >= 0 && col_len <= INT32_MAX && n >= 0 && n <= INT32_MAX,
               "lengths must be in [0, 2^31)");
  OLAP_REQUIRE(ctx, cmp == OLAP_CMP_LE || cmp == OLAP_CMP_LT, "cmp must be OLAP_CMP_LE or OLAP_CMP_LT");
  OLAP_REQUIRE(ctx, n == 0 || (col && out_rowids), "null column or output");
  olap::Arena ar(ctx);
  unsigned long long* total = d_count ? reinterpret_cast<unsigned long long*>(d_count)
                                      : ar.take<unsigned long long>(1);
  if (!total) return olap::set_error(ctx, OLAP_ERR_CAPACITY, "scratch arena exhausted");
  const olap::LePred le(val, cmp);
  if (in_rowids)
    return olap::mark_and_expand(
        ctx, ar, n, sizeof(int32_t), ctx->sm_count * int64_t(48), olap::RunCopy{out_rowids}, total,
        [&](const olap::Marks& mk, int64_t first, const olap::RunCopy&) {
          unsigned grid, block;
          olap::mark_grid(ctx, mk.n_tiles, 512, 3, &grid, &block);
          olap::select_refine_kernel<<<grid, block, 0, ctx->stream>>>(col, static_cast<uint32_t>(col_len), in_rowids + first, le.val, le.none,
                                                                      mk, &ctx->counters->range_errors);
          OLAP_CUDA_TRY(ctx, cudaGetLastError());
          return OLAP_OK;
        });
  auto* const kernel = olap::al16(col) ? olap::select_mark_kernel<true> : olap::select_mark_kernel<false>;
  return olap::mark_and_expand(
      ctx, ar, n, 0, ctx->sm_count * int64_t(64), olap::RowEmit{out_rowids}, total,
      [&](const olap::Marks& mk, int64_t first, const olap::RowEmit&) {
        unsigned grid, block;
        olap::mark_grid(ctx, mk.n_tiles, 512, 4, &grid, &block);
        kernel<<<grid, block, 0, ctx->stream>>>(col + first, mk.n, le.val, le.none, mk.bits, mk.counts, mk.tile,
                                                mk.n_tiles);
        OLAP_CUDA_TRY(ctx, cudaGetLastError());
        return OLAP_OK;
      });
}

int olap_debug_wait_timeout(olap_ctx* ctx, uint32_t spin_limit) {
  if (!ctx || spin_limit < 1) return OLAP_ERR_INVALID;
  std::lock_guard<std::mutex> lk(ctx->mu);
  OLAP_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  olap::Arena ar(ctx);
  olap::ScanTiles st;
  unsigned long long* total = ar.take<unsigned long long>(1);
  long long* out = ar.take<long long>(1);
  if (!total || !out) return olap::set_error(ctx, OLAP_ERR_CAPACITY, "scratch arena exhausted");
  int rc = olap::make_scan_tiles(ctx, ar, 2, total, ctx->stream, &st, 1);  // two one-item tiles
  if (rc != OLAP_OK) return rc;
  olap::lookback_timeout_kernel<<<1, 32, 0, ctx->stream>>>(st, spin_limit, out);
  OLAP_CUDA_TRY(ctx, cudaGetLastError());
  return olap::check_timeouts(ctx, ctx->stream);
}

int olap_select_bitmap(olap_ctx* ctx, const int32_t* col, int64_t n, int32_t val, int cmp,
                       uint32_t* bitmap) {
  if (!ctx) return OLAP_ERR_INVALID;
  std::lock_guard<std::mutex> lk(ctx->mu);
  OLAP_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  OLAP_REQUIRE(ctx, n >= 0, "n must be >= 0");
  OLAP_REQUIRE(ctx, cmp == OLAP_CMP_LE || cmp == OLAP_CMP_LT, "cmp must be OLAP_CMP_LE or OLAP_CMP_LT");
  if (n == 0) return OLAP_OK;
  OLAP_REQUIRE(ctx, col && bitmap, "null column or bitmap");
  const olap::LePred le(val, cmp);
  // a bitmap has no tile counts to add up: short tiles, balanced over the warps
  const int64_t tile = std::min<int64_t>(olap::mark_tile(n, ctx->sm_count * int64_t(64)), 1 << 20);
  const int64_t n_tiles = (n + tile - 1) / tile;
  unsigned grid, block;
  olap::mark_grid(ctx, n_tiles, 512, 4, &grid, &block);
  auto* const kernel = olap::al16(col) ? olap::select_mark_kernel<true> : olap::select_mark_kernel<false>;
  kernel<<<grid, block, 0, ctx->stream>>>(col, n, le.val, le.none, bitmap, nullptr, static_cast<int32_t>(tile),
                                          n_tiles);
  OLAP_CUDA_TRY(ctx, cudaGetLastError());
  return OLAP_OK;
}

int olap_selalgo(olap_ctx* ctx, int32_t condition, int64_t n, const int32_t* Ra, const int32_t* Rb,
                 const int32_t* Rc, const int32_t* Rd, int64_t* d_sum, int64_t* d_count) {
  if (!ctx) return OLAP_ERR_INVALID;
  std::lock_guard<std::mutex> lk(ctx->mu);
  OLAP_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  OLAP_REQUIRE(ctx, n >= 0 && d_sum, "n must be >= 0 and d_sum given");
  OLAP_REQUIRE(ctx, n == 0 || (Ra && Rb && Rc && Rd), "null column");
  olap::Arena ar(ctx);
  int64_t* cnt = d_count ? d_count : ar.take<int64_t>(1);
  if (!cnt) return olap::set_error(ctx, OLAP_ERR_CAPACITY, "scratch arena exhausted");
  OLAP_CUDA_TRY(ctx, cudaMemsetAsync(d_sum, 0, sizeof(int64_t), ctx->stream));
  OLAP_CUDA_TRY(ctx, cudaMemsetAsync(cnt, 0, sizeof(int64_t), ctx->stream));
  if (n == 0) return OLAP_OK;
  const int vec = olap::al16(Ra) && olap::al16(Rb) && olap::al16(Rc) && olap::al16(Rd);
  olap::selalgo_kernel<<<olap::stream_grid(ctx, (n + 3) / 4, 512), 512, 0, ctx->stream>>>(
      condition, n, Ra, Rb, Rc, Rd, vec, reinterpret_cast<unsigned long long*>(d_sum),
      reinterpret_cast<unsigned long long*>(cnt));
  OLAP_CUDA_TRY(ctx, cudaGetLastError());
  return OLAP_OK;
}

int olap_project_pairs(olap_ctx* ctx, int32_t condition, int64_t n, const int32_t* Ra,
                       const int32_t* Rc, int32_t* out_a, int32_t* out_c, int64_t* d_count) {
  if (!ctx) return OLAP_ERR_INVALID;
  std::lock_guard<std::mutex> lk(ctx->mu);
  OLAP_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  OLAP_REQUIRE(ctx, n >= 0 && n <= INT32_MAX, "n must be in [0, 2^31)");
  OLAP_REQUIRE(ctx, n == 0 || (Ra && Rc && out_a && out_c), "null column or output");
  olap::ProjectOp op;
  std::memset(&op, 0, sizeof(op));
  op.ra = Ra;
  op.rc = Rc;
  op.out_a = out_a;
  op.out_c = out_c;
  op.cond = condition;
  op.vec = olap::al16(Ra) && olap::al16(Rc);
  return olap::run_compaction(ctx, op, n, d_count);
}

int olap_project_pairs_rows(olap_ctx* ctx, int32_t condition, int64_t n, const void* rows, int64_t row_bytes,
                            int64_t off_a, int64_t off_c, int32_t* out_a, int32_t* out_c, int64_t* d_count) {
  if (!ctx) return OLAP_ERR_INVALID;
  std::lock_guard<std::mutex> lk(ctx->mu);
  OLAP_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  OLAP_REQUIRE(ctx, n >= 0 && n <= INT32_MAX, "n must be in [0, 2^31)");
  OLAP_REQUIRE(ctx, n == 0 || (rows && out_a && out_c), "null rows or output");
  OLAP_REQUIRE(ctx, row_bytes >= 4 && row_bytes % 4 == 0, "row_bytes must be a positive multiple of 4");
  OLAP_REQUIRE(ctx, off_a >= 0 && off_c >= 0 && off_a % 4 == 0 && off_c % 4 == 0 && off_a + 4 <= row_bytes &&
                        off_c + 4 <= row_bytes,
               "field offsets must be 4-byte aligned and inside the row");
  OLAP_REQUIRE(ctx, (reinterpret_cast<uintptr_t>(rows) & 3) == 0, "rows must be 4-byte aligned");
  olap::ProjectRowsOp op;
  std::memset(&op, 0, sizeof(op));
  op.rows = static_cast<const unsigned char*>(rows);
  op.row_bytes = row_bytes;
  op.off_a = static_cast<int32_t>(off_a);
  op.off_c = static_cast<int32_t>(off_c);
  op.out_a = out_a;
  op.out_c = out_c;
  op.cond = condition;
  return olap::run_compaction(ctx, op, n, d_count);
}

int olap_gather_i32(olap_ctx* ctx, const int32_t* rowids, int64_t k, int ncols,
                    const int32_t* const* cols, int64_t col_len, int32_t* const* outs) {
  if (!ctx) return OLAP_ERR_INVALID;
  std::lock_guard<std::mutex> lk(ctx->mu);
  OLAP_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  OLAP_REQUIRE(ctx, k >= 0 && ncols >= 1 && ncols <= olap::kMaxGatherCols, "1..8 columns");
  if (k == 0) return OLAP_OK;
  OLAP_REQUIRE(ctx, rowids && cols && outs, "null argument");
  olap::GatherParams gp;
  std::memset(&gp, 0, sizeof(gp));
  gp.ncols = ncols;
  gp.col_len = col_len;
  gp.range_err = &ctx->counters->range_errors;
  bool vec = olap::al16(rowids);
  for (int c = 0; c < ncols; ++c) {
    OLAP_REQUIRE(ctx, cols[c] && outs[c], "null column or output");
    gp.cols[c] = cols[c];
    gp.outs[c] = outs[c];
    vec &= olap::al16(outs[c]);
  }
  // more than 6 rows apart on average (measured on 2^28-row columns: 4 rows
  // apart 876 us dense and 896 sparse, 10 apart 704 and 623)
  const unsigned grid = olap::stream_grid(ctx, (k + 3) / 4, 256);
  if (col_len > 6 * k)
    olap::gather_sparse_kernel<<<grid, 256, 0, ctx->stream>>>(rowids, k, gp);
  else
    olap::gather_dense_kernel<<<grid, 256, 0, ctx->stream>>>(rowids, k, gp, vec);
  OLAP_CUDA_TRY(ctx, cudaGetLastError());
  return OLAP_OK;
}

}  // extern "C"
