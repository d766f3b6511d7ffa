// Order-preserving stream compaction for sm_100a.
//
// Selection vectors in the reference are row ids in ascending order
// (select/test_select_option.cpp:391-423), and the column-wise OLAP core keeps
// its OID lists in row order (OLAPcore/test_multi_compute_operator.cpp
// :240-283).  Both ways here produce exactly that order.
//
// Marks and expansion (select, hash-probe pairs, column-wise lists): the
// operator's own kernel writes one bit per item, a count per tile and what it
// read of the marked items; expand_kernel adds up the counts before its tiles
// and writes the items out.  No block waits for another, so the first kernel
// runs at its loads' pace (2^28 rows: select 362 us in one pass with look-back,
// 172 + 69 us this way).
//
// One pass (the project operators): each block claims tiles in increasing
// order through an atomic counter, ranks its selected items with warp ballots
// and a scan of the warp counts, and finds the tile's output offset with a
// decoupled look-back over the status words of the preceding tiles (a warp
// inspects 32 predecessors at a time).
//
// Every tile a block waits for was claimed earlier by a block that is already
// running, so the waits end; they are bounded anyway: after kSpinLimit polls a
// block records a timeout in the context's counters and stops, and the host
// call reports OLAP_ERR_TIMEOUT.
#pragma once

#include <algorithm>
#include <type_traits>

#include "olap_internal.cuh"

namespace olap {

constexpr int kCompactThreads = 256;
constexpr int kCompactGroups = 4;  // default int4 loads per thread and tile (ops set Op::kGroups)
constexpr uint32_t kSpinLimit = 1u << 22;

// Status word of a tile: flag in bits 62-63 (0 none, 1 aggregate, 2
// inclusive prefix), value in bits 0-61.
constexpr uint64_t kFlagAgg = 1ull << 62;
constexpr uint64_t kFlagInc = 2ull << 62;
constexpr uint64_t kValMask = (1ull << 62) - 1;

struct ScanTiles {
  unsigned long long* status;   // [n_tiles], zeroed before the launch
  unsigned int* next_tile;      // claim counter, zeroed before the launch
  unsigned long long* timeouts; // context counter
  unsigned long long* total;    // selected items in all tiles (written by the last tile)
  int64_t n_tiles;
};

__device__ __forceinline__ uint64_t ld_relaxed_u64(const unsigned long long* p) {
  uint64_t v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_relaxed_u64(unsigned long long* p, uint64_t v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// Claims the next tile for this block (all threads get the same id).
__device__ __forceinline__ int64_t claim_tile(const ScanTiles& st, unsigned int* s_tile) {
  if (threadIdx.x == 0) *s_tile = atomicAdd(st.next_tile, 1u);
  __syncthreads();
  const int64_t t = *s_tile;
  __syncthreads();
  return t;
}

// Exclusive prefix of this tile's count over all earlier tiles; run by one
// full warp (warp 0).  Returns -1 on timeout.
__device__ __forceinline__ int64_t lookback(const ScanTiles& st, int64_t tile, uint64_t count,
                                           uint32_t spin_limit = kSpinLimit) {
  const int lane = threadIdx.x & 31;
  if (tile == 0) {
    if (lane == 0) st_relaxed_u64(&st.status[0], kFlagInc | count);
    return 0;
  }
  if (lane == 0) st_relaxed_u64(&st.status[tile], kFlagAgg | count);
  uint64_t excl = 0;
  int64_t t = tile - 1;
  uint32_t spins = 0;
  while (true) {
    const int64_t idx = t - lane;
    uint64_t w = idx >= 0 ? ld_relaxed_u64(&st.status[idx]) : kFlagInc;
    while (__any_sync(0xffffffffu, (w >> 62) == 0)) {
      if (++spins > spin_limit) {
        if (lane == 0) atomicAdd(st.timeouts, 1ull);
        return -1;
      }
      __nanosleep(64);
      if ((w >> 62) == 0) w = ld_relaxed_u64(&st.status[idx]);
    }
    const uint32_t inc = __ballot_sync(0xffffffffu, (w >> 62) == 2);
    uint64_t v = w & kValMask;
    if (inc) {
      const int k = __ffs(inc) - 1;  // closest predecessor with an inclusive prefix
      if (lane > k) v = 0;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      excl += v;
      break;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    excl += v;
    t -= 32;
  }
  if (lane == 0) st_relaxed_u64(&st.status[tile], kFlagInc | (excl + count));
  return static_cast<int64_t>(excl);
}

// Compaction kernel.  Items are numbered 0 .. n_items-1.  A tile holds
// kCompactThreads x 4 x G items (G = Op::kGroups); in group u, lane l of
// warp w owns the 4 consecutive items tile_first + u*1024 + w*128 + 4l + k,
// so each group is one coalesced 16-byte load per thread and row order is
// (u, w, l, k).  A thread ranks its selected items inside its warp with four
// ballots, the block ranks the (u, w) warp counts with one warp scan, and the
// tile's output base comes from the look-back.  The Op is called per group
// and per selected item:
//   template <bool kFull> uint32_t op.flags(int u, int64_t first, int nv)
//       -> 4-bit mask of the selected items among first .. first+3 (only the
//       first nv exist); kFull: nv == 4 and op.vec_ok() (16-byte loads are
//       allowed), and op.prefetch(u, first) ran for every group first; the
//       op may cache what it loaded for group u;
//   void op.emit(int u, int k, int64_t item, int64_t pos)  -> write selected
//       item `item` (= first + k of group u) at output position `pos`.
// A larger G keeps more bytes in flight per block for ops that cache little.
template <class Op>
constexpr int64_t compact_tile_items() {
  return static_cast<int64_t>(kCompactThreads) * 4 * Op::kGroups;
}

template <class Op>
__global__ void __launch_bounds__(kCompactThreads) compact_kernel(const Op op_in, int64_t n_items, ScanTiles st) {
  constexpr int G = Op::kGroups;
  constexpr int W = kCompactThreads / 32;
  constexpr int E = G * W;  // warp counts per tile
  static_assert(G <= 16 && E % 32 == 0, "groups per thread: a multiple of 4, at most 16");
  constexpr int PER = E / 32;
  Op op = op_in;  // per-thread copy: ops cache the loaded items between flags() and emit()
  __shared__ unsigned int s_tile;
  __shared__ uint32_t s_cnt[E];  // warp counts of (u, w), then their exclusive prefixes in the tile
  __shared__ long long s_base;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t lt = (1u << lane) - 1u;
  for (;;) {
    const int64_t tile = claim_tile(st, &s_tile);
    if (tile >= st.n_tiles) return;
    const int64_t tile_first = tile * compact_tile_items<Op>();
    const bool full = op.vec_ok() && tile_first + compact_tile_items<Op>() <= n_items;
    uint64_t mk = 0;  // 4 bits per group
    if (full) {
      // full tile, aligned columns: every group's loads are issued before
      // the first is used, so G x 16 bytes per thread are in flight
#pragma unroll
      for (int u = 0; u < G; ++u)
        op.prefetch(u, tile_first + static_cast<int64_t>(u) * kCompactThreads * 4 + 4 * threadIdx.x);
#pragma unroll
      for (int u = 0; u < G; ++u) {
        const int64_t first = tile_first + static_cast<int64_t>(u) * kCompactThreads * 4 + 4 * threadIdx.x;
        mk |= static_cast<uint64_t>(op.template flags<true>(u, first, 4)) << (4 * u);
      }
    } else {
#pragma unroll
      for (int u = 0; u < G; ++u) {
        const int64_t first = tile_first + static_cast<int64_t>(u) * kCompactThreads * 4 + 4 * threadIdx.x;
        const int64_t left = n_items - first;
        const int nv = left >= 4 ? 4 : (left > 0 ? static_cast<int>(left) : 0);
        const uint32_t m = nv > 0 ? op.template flags<false>(u, first, nv) : 0u;
        mk |= static_cast<uint64_t>(m) << (4 * u);
      }
    }
#pragma unroll
    for (int u = 0; u < G; ++u) {
      const uint32_t c = __reduce_add_sync(0xffffffffu, __popc(static_cast<uint32_t>(mk >> (4 * u)) & 15u));
      if (lane == 0) s_cnt[u * W + warp] = c;
    }
    __syncthreads();
    if (warp == 0) {
      uint32_t v[PER];
      uint32_t sum = 0;
#pragma unroll
      for (int i = 0; i < PER; ++i) {
        v[i] = s_cnt[lane * PER + i];
        sum += v[i];
      }
      uint32_t inc = sum;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
      }
      uint32_t run = inc - sum;
#pragma unroll
      for (int i = 0; i < PER; ++i) {
        s_cnt[lane * PER + i] = run;
        run += v[i];
      }
      const uint64_t tile_count = __shfl_sync(0xffffffffu, inc, 31);
      const int64_t b = lookback(st, tile, tile_count);
      if (lane == 0) {
        s_base = b;
        if (tile == st.n_tiles - 1 && b >= 0) *st.total = static_cast<unsigned long long>(b) + tile_count;
      }
    }
    __syncthreads();
    const long long base = s_base;
    if (base < 0) return;  // timed out: the host reports it
#pragma unroll
    for (int u = 0; u < G; ++u) {
      const uint32_t m = static_cast<uint32_t>(mk >> (4 * u)) & 15u;
      uint32_t before = 0;
#pragma unroll
      for (int k = 0; k < 4; ++k) before += __popc(__ballot_sync(0xffffffffu, (m >> k) & 1u) & lt);
      if (!m) continue;
      int64_t pos = base + s_cnt[u * W + warp] + before;
      const int64_t first = tile_first + static_cast<int64_t>(u) * kCompactThreads * 4 + 4 * threadIdx.x;
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if ((m >> k) & 1u) op.emit(u, k, first + k, pos++);
    }
  }
}

// ---- compaction in two kernels: marks, then expansion ------------------------
// An op whose evaluation is long or latency-bound (probes), or that streams at
// full DRAM rate (select), does not wait for its output offsets: a mark kernel
// writes one bit per item, the selected items' values packed at the start of
// their mark tile, and each tile's count; expand_kernel then turns the marks
// into positions.  No look-back, so no block waits for another, and a warp
// works alone on its tile, so that tiles are sized to give every warp of the
// device the same number of them (and a short input reaches every SM).  The
// marks stay in L2 between the two kernels; an input whose marks do not fit
// the arena runs in chunks, the running total kept on the device.
constexpr int kExpandThreads = 1024;
constexpr int kExpandDirect = 8;  // selected items per word of a step up to which the lanes write their own
constexpr int kExpandStaged = 24;  // ... up to which they go through shared memory
constexpr int kMarkRounds = 4;  // tiles per warp of a mark kernel on a long input
constexpr int64_t kMarkScratch = int64_t(64) << 20;  // as the default arena
constexpr int64_t kFewChunks = 2;

constexpr size_t kExpandSmem = kExpandThreads * kExpandStaged * sizeof(uint16_t);  // a step's items, per warp

struct Marks {
  uint32_t* bits;    // bit i % 32 of word i / 32: item i of the chunk is selected
  uint32_t* counts;  // selected items per mark tile
  void* vals;        // their values: those of tile t from element t * tile on
  int64_t n;         // items of the chunk
  int32_t tile;      // items per mark tile, a multiple of 128
  int32_t n_tiles;
};

// First position of each warp's run of `per` whole tiles (warp w of block b takes
// them from tile (b W + w) per on): *run_in and every tile before its own.  All
// threads of a block of kThreads call it.
template <int kThreads>
__device__ __forceinline__ int64_t expand_base(const Marks& mk, int per, const unsigned long long* __restrict__ run_in) {
  constexpr int W = kThreads / 32;
  __shared__ unsigned long long s_sum[W];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int b0 = min(static_cast<int>(blockIdx.x) * W * per, mk.n_tiles);
  unsigned long long s = 0;
  for (int i = tid; i < (b0 >> 2); i += kThreads) {
    const uint4 c = __ldg(reinterpret_cast<const uint4*>(mk.counts) + i);
    s += static_cast<unsigned long long>(c.x) + c.y + c.z + c.w;
  }
  if (tid < (b0 & 3)) s += __ldg(mk.counts + (b0 & ~3) + tid);
  const int t0 = min(b0 + warp * per, mk.n_tiles);
  s = static_cast<unsigned long long>(warp_sum_i64(static_cast<int64_t>(s)));
  if (lane == 0) s_sum[warp] = s;
  __syncthreads();
  s = (lane < W ? s_sum[lane] : 0ull) + (run_in && lane == 0 ? *run_in : 0ull);
  for (int t = b0 + lane; t < t0; t += 32) s += __ldg(mk.counts + t);
  return warp_sum_i64(static_cast<int64_t>(s));
}

// Emit: constexpr bool kVals; void emit(int64_t pos, int64_t item, int64_t v)
// writes item `item` (of the whole input) at output position pos; v is the
// index of its value in Marks::vals.  A warp takes a run of whole tiles, up to
// 1,024 items (a word per lane) at a step: several short tiles, or a part of
// a long one.  Only the first sum over the tiles before a block's needs the
// whole block.  Bound by instructions: where few items of a step are
// selected, each lane writes its own word's (neighbouring lanes write
// neighbouring positions, so a store still covers few lines), through shared
// memory when there are no values to fetch (2^28 rows at 10 %: 85 -> 69 us; with
// values 54 -> 56 us for 120M rows at 5 %, so those write directly); where many
// are, the warp takes the words one after another, a lane per item.
template <class Emit>
__global__ void __launch_bounds__(kExpandThreads, 2) expand_kernel(const Emit em, const Marks mk, int64_t first_item,
                                                                   const unsigned long long* __restrict__ run_in,
                                                                   unsigned long long* __restrict__ run_out,
                                                                   unsigned long long* __restrict__ total) {
  constexpr int W = kExpandThreads / 32;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t lt = (1u << lane) - 1u;
  extern __shared__ uint16_t s_items[];
  uint16_t* const s_at = s_items + warp * 32 * kExpandStaged;  // items of a step, in order
  const int per = (mk.n_tiles + gridDim.x * W - 1) / (gridDim.x * W);  // tiles per warp
  int64_t base = expand_base<kExpandThreads>(mk, per, run_in);
  const int t0 = min((static_cast<int>(blockIdx.x) * W + warp) * per, mk.n_tiles), t1 = min(t0 + per, mk.n_tiles);
  const int wpt = mk.tile >> 5;                      // words per tile
  const int tps = wpt <= 32 ? 32 / wpt : 1;          // tiles per step, one when a tile takes several steps
  const int head = wpt <= 32 ? lane / wpt * wpt : 0; // lane of the first word of this lane's tile
  for (int t = t0; t < t1; t += tps) {
    const int64_t tb = static_cast<int64_t>(t) * mk.tile;
    const int64_t span = static_cast<int64_t>(min(tps, t1 - t)) * mk.tile;
    const int len = static_cast<int>(tb + span < mk.n ? span : mk.n - tb);
    int64_t v = tb + 32 * head;  // next value of this lane's tile
    for (int r = 0; r < len; r += 1024) {
      uint32_t word = r + 32 * lane < len ? __ldg(mk.bits + ((tb + r) >> 5) + lane) : 0u;
      const uint32_t c = __popc(word);
      uint32_t inc = c;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
      }
      const uint32_t before = inc - c;
      const uint32_t in_tile = Emit::kVals ? before - __shfl_sync(0xffffffffu, before, head) : 0u;
      const int all = static_cast<int>(__shfl_sync(0xffffffffu, inc, 31));
      const int64_t item = first_item + tb + r;
      const int words = (min(len - r, 1024) + 31) >> 5;
      if (Emit::kVals && all <= kExpandDirect * words) {
        int64_t pos = base + before, vi = v + in_tile;
        while (word) {
          em.emit(pos++, item + 32 * lane + __ffs(word) - 1, vi++);
          word &= word - 1;
        }
      } else if (all <= kExpandStaged * words) {
        for (int k = before; word; ++k) {
          s_at[k] = static_cast<uint16_t>(32 * lane + __ffs(word) - 1);
          word &= word - 1;
        }
        __syncwarp();
        const int64_t ahead = Emit::kVals ? v + in_tile - before : 0;  // value index less position, by lane
        for (int k0 = 0; k0 < all; k0 += 32) {  // same trips in every lane: 69 us; a loop per lane 80
          const int k = k0 + lane;
          const int off = k < all ? s_at[k] : 0;
          const int64_t vi = Emit::kVals ? __shfl_sync(0xffffffffu, ahead, off >> 5) + k : 0;
          if (k < all) em.emit(base + k, item + off, vi);
        }
        __syncwarp();
      } else {
#pragma unroll 4
        for (int w = 0; w < words; ++w) {
          const uint32_t x = __shfl_sync(0xffffffffu, word, w);
          const uint32_t at = __popc(x & lt);
          const int64_t pos = base + __shfl_sync(0xffffffffu, before, w) + at;
          const int64_t vi = Emit::kVals ? __shfl_sync(0xffffffffu, v + in_tile, w) + at : 0;
          if ((x >> lane) & 1u) em.emit(pos, item + 32 * w + lane, vi);
        }
      }
      base += all;
      v += all;
    }
  }
  if (t1 == mk.n_tiles && t0 < t1 && lane == 0) {
    if (run_out) *run_out = static_cast<unsigned long long>(base);
    if (total) *total = static_cast<unsigned long long>(base);
  }
}

// Where the values are all that is wanted (no items, so no marks): each tile's
// run of values to its place in `out`.  Bound by the latency of the runs, which
// are short: four loads per lane in flight.
constexpr int kRunThreads = 512;
constexpr int kRunBlocks = 3;  // per SM
struct RunCopy {
  int32_t* out;
};
template <class Copy>
__global__ void __launch_bounds__(kRunThreads, kRunBlocks) run_copy_kernel(
    const Copy rc, const Marks mk, int64_t, const unsigned long long* __restrict__ run_in,
    unsigned long long* __restrict__ run_out, unsigned long long* __restrict__ total) {
  constexpr int W = kRunThreads / 32;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int per = (mk.n_tiles + gridDim.x * W - 1) / (gridDim.x * W);
  int64_t base = expand_base<kRunThreads>(mk, per, run_in);
  const int t0 = min((static_cast<int>(blockIdx.x) * W + warp) * per, mk.n_tiles), t1 = min(t0 + per, mk.n_tiles);
  const uint64_t pol = policy_evict_first();
  for (int t = t0; t < t1; ++t) {
    const int32_t* src = static_cast<const int32_t*>(mk.vals) + static_cast<int64_t>(t) * mk.tile + lane;
    const int c = static_cast<int>(__ldg(mk.counts + t));
    int32_t* dst = rc.out + base + lane;
    for (int k = 0; k < c; k += 128) {
      int32_t v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) v[u] = ld_stream_s32_if(k + 32 * u + lane < c, src + k + 32 * u, pol, 0);
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (k + 32 * u + lane < c) dst[k + 32 * u] = v[u];
    }
    base += c;
  }
  if (t1 == mk.n_tiles && t0 < t1 && lane == 0) {
    if (run_out) *run_out = static_cast<unsigned long long>(base);
    if (total) *total = static_cast<unsigned long long>(base);
  }
}

// Items per warp tile for n items on `warps` resident warps: kMarkRounds
// tiles per warp, the same number for each, down to one step of 128 items.
inline int64_t mark_tile(int64_t n, int64_t warps) {
  const int64_t t = (n + kMarkRounds * warps - 1) / (kMarkRounds * warps);
  return (t + 127) & ~int64_t(127);
}

// Grid and block of a mark kernel whose warps take tiles in turn: blocks of
// `threads` while the tiles fill every SM, smaller ones for a short input.
inline void mark_grid(const olap_ctx* ctx, int64_t n_tiles, int threads, int blocks_per_sm, unsigned* grid,
                      unsigned* block) {
  const int64_t cap = static_cast<int64_t>(ctx->sm_count) * blocks_per_sm;
  int t = threads;
  while (t > 64 && n_tiles < cap * (t / 32)) t >>= 1;
  const int64_t g = (n_tiles + t / 32 - 1) / (t / 32);
  *grid = static_cast<unsigned>(g < cap ? g : cap);
  *block = static_cast<unsigned>(t);
}

// Runs mark(marks, first_item, emit) and the expansion over n items with
// val_bytes per value, in chunks whose marks fit the arena; *total gets the
// count.  `warps`: resident warps of the mark kernel.
template <class Emit, class Mark>
int mark_and_expand(olap_ctx* ctx, Arena& ar, int64_t n, size_t val_bytes, int64_t warps, Emit em,
                    unsigned long long* total, Mark&& mark) {
  if (n == 0) {
    OLAP_CUDA_TRY(ctx, cudaMemsetAsync(total, 0, sizeof(unsigned long long), ctx->stream));
    return OLAP_OK;
  }
  const char* small = "scratch arena too small for the compaction state";
  unsigned long long* run = ar.take<unsigned long long>(2);
  uint32_t* counts = ar.take<uint32_t>(static_cast<size_t>(kMarkRounds * warps));
  if (!run || !counts) return set_error(ctx, OLAP_ERR_CAPACITY, small);
  // items per chunk: 1/8 byte of marks and val_bytes of values each
  const int64_t left = static_cast<int64_t>(ar.cap - ar.off) - 1024;
  int64_t chunk = left > 0 ? left * 8 / (1 + 8 * static_cast<int64_t>(val_bytes)) & ~int64_t(127) : 0;
  if (chunk < 128) return set_error(ctx, OLAP_ERR_CAPACITY, small);
  // An arena with room for a small part only: up to kMarkScratch bytes of the
  // context's growing buffer instead (2^25 probe rows to pairs in a 1 MB arena:
  // 2.4 ms in 146 chunks, 0.35 ms in three).  Not for a graph, which would hold
  // on to a buffer that a later call may replace.
  char* big = nullptr;
  const int64_t per128 = 16 + 128 * static_cast<int64_t>(val_bytes);  // bytes of marks and values
  if (n > kFewChunks * chunk && !capturing(ctx->stream)) {
    const int64_t rows = std::min((n + 127) & ~int64_t(127), (kMarkScratch - 1024) / per128 * 128);
    if (rows > kFewChunks * chunk && (big = big_scratch(ctx, static_cast<size_t>(rows / 128 * per128 + 1024)))) chunk = rows;
  }
  // equal chunks, and tiles addressed by 32 bits
  const int64_t n_chunks = (n + chunk - 1) / chunk;
  chunk = ((n + n_chunks - 1) / n_chunks + 127) & ~int64_t(127);
  Marks mk;
  if (big) {
    mk.bits = reinterpret_cast<uint32_t*>(big);
    mk.vals = val_bytes ? big + ((chunk / 8 + 255) & ~int64_t(255)) : nullptr;
  } else {
    mk.bits = ar.take<uint32_t>(static_cast<size_t>(chunk / 32));
    mk.vals = val_bytes ? ar.take<char>(static_cast<size_t>(chunk) * val_bytes) : nullptr;
  }
  mk.counts = counts;
  if (!mk.bits || (val_bytes && !mk.vals)) return set_error(ctx, OLAP_ERR_CAPACITY, small);
  mk.tile = static_cast<int32_t>(mark_tile(chunk, warps));
  constexpr bool kRuns = std::is_same_v<Emit, RunCopy>;
  void (*out_kernel)(const Emit, const Marks, int64_t, const unsigned long long*, unsigned long long*, unsigned long long*);
  if constexpr (kRuns) out_kernel = run_copy_kernel<Emit>;
  else out_kernel = expand_kernel<Emit>;
  constexpr size_t out_smem = kRuns ? 0 : kExpandSmem;
  constexpr int out_threads = kRuns ? kRunThreads : kExpandThreads;
  if (!kRuns)
    OLAP_CUDA_TRY(ctx, cudaFuncSetAttribute(out_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            static_cast<int>(kExpandSmem)));
  int which = 0;
  for (int64_t first = 0; first < n; first += chunk, which ^= 1) {
    mk.n = chunk < n - first ? chunk : n - first;
    mk.n_tiles = static_cast<int32_t>((mk.n + mk.tile - 1) / mk.tile);
    const int rc = mark(mk, first, em);
    if (rc != OLAP_OK) return rc;
    const int64_t blocks = (mk.n_tiles + out_threads / 32 - 1) / (out_threads / 32);
    const int64_t cap = static_cast<int64_t>(ctx->sm_count) * (kRuns ? kRunBlocks : 2);
    out_kernel<<<static_cast<unsigned>(blocks < cap ? blocks : cap), out_threads, out_smem, ctx->stream>>>(
        em, mk, first, first ? run + which : nullptr, run + (which ^ 1), first + mk.n == n ? total : nullptr);
    OLAP_CUDA_TRY(ctx, cudaGetLastError());
  }
  return OLAP_OK;
}

// Host helper: scan-tile state for n_items in tiles of tile_items
// (compact_tile_items<Op>()) from the arena; zeroes it on the stream.
inline int make_scan_tiles(olap_ctx* ctx, Arena& ar, int64_t n_items, unsigned long long* total,
                           cudaStream_t stream, ScanTiles* st, int64_t tile_items) {
  st->n_tiles = (n_items + tile_items - 1) / tile_items;
  if (st->n_tiles < 1) st->n_tiles = 1;
  st->status = ar.take<unsigned long long>(static_cast<size_t>(st->n_tiles));
  st->next_tile = ar.take<unsigned int>(1);
  st->timeouts = &ctx->counters->wait_timeouts;
  st->total = total;
  if (!st->status || !st->next_tile)
    return set_error(ctx, OLAP_ERR_CAPACITY, "scratch arena too small for the compaction state");
  OLAP_CUDA_TRY(ctx, cudaMemsetAsync(st->status, 0, sizeof(unsigned long long) * st->n_tiles, stream));
  OLAP_CUDA_TRY(ctx, cudaMemsetAsync(st->next_tile, 0, sizeof(unsigned int), stream));
  if (total) OLAP_CUDA_TRY(ctx, cudaMemsetAsync(total, 0, sizeof(unsigned long long), stream));
  return OLAP_OK;
}

inline unsigned compact_grid(const olap_ctx* ctx, int64_t n_tiles) {
  int64_t g = static_cast<int64_t>(ctx->sm_count) * 8;  // 8 x 256 threads per SM
  if (g > n_tiles) g = n_tiles;
  return static_cast<unsigned>(g < 1 ? 1 : g);
}

// Checks the wait-timeout counter after a synchronising call.
inline int check_timeouts(olap_ctx* ctx, cudaStream_t stream) {
  unsigned long long t = 0;
  OLAP_CUDA_TRY(ctx, cudaMemcpyAsync(&t, &ctx->counters->wait_timeouts, sizeof(t),
                                     cudaMemcpyDeviceToHost, stream));
  OLAP_CUDA_TRY(ctx, cudaStreamSynchronize(stream));
  if (t) {
    OLAP_CUDA_TRY(ctx, cudaMemsetAsync(&ctx->counters->wait_timeouts, 0, sizeof(t), stream));
    return set_error(ctx, OLAP_ERR_TIMEOUT, "a bounded device wait expired in a compaction");
  }
  return OLAP_OK;
}

}  // namespace olap
