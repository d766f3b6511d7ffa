// Column-wise OLAP core and the star-join operator for sm_100a.
//
// Column-wise model (code/OLAPcore/test_multi_compute_operator.cpp):
//  * join_cwm_sv (:908-958, thread body :290-322) builds the static vector
//    int16 groupID[N] (GROUP_NULL when a dimension misses) one dimension per
//    pass; here all dimensions in one pass, same vector;
//  * agg_cwm_sv (:764-827, :662-673) sums M1+M2 by groupID;
//  * join_cwm_dv (:840-894, :240-283) keeps the surviving rows as (OID,
//    groupID) lists in row order; here one order-preserving compaction;
//  * agg_cwm_dv (:685-752, :645-655) sums M1[OID]+M2[OID] by groupID.
// Group ids are int16 there, so these entry points accept group_nums up to
// 32766 (GROUP_NULL is 32767).
//
// Star-join operator (code/starjoin/test_starjoin_option.cpp): the count of
// rows surviving four dimension probes (starjoinalgo_rowwise :37-50), the
// static vector of 4-bit packed group ids (starjoinalgo_cwm_sv :66-121:
// c<<12 + s<<8 + p<<4 + d, GROUP_NULL otherwise, count of entries that are
// not GROUP_NULL) and the compacted (position, group) pairs
// (starjoinalgo_cwm_dv :137-189).
#include <algorithm>
#include <cstring>
#include <type_traits>

#include "compact.cuh"

namespace olap {

struct DimSet {
  const int8_t* vec[OLAP_MAX_DIMS];
  const int32_t* fk[OLAP_MAX_DIMS];
  uint32_t len[OLAP_MAX_DIMS];
  int32_t mul[OLAP_MAX_DIMS];  // factor, or 1 << shift for the packed ids
  int32_t off[OLAP_MAX_DIMS];  // staged copy's byte offset in shared memory, or -1
  int32_t nib[OLAP_MAX_DIMS];  // staged as 4-bit codes
  int32_t nd;
  int32_t smem;                // staged bytes (multiple of 16)
};

// What a probe kernel does with the rows' group ids.
enum {
  CWM_SV16 = 0,   // join_cwm_sv: int16 per row, GROUP_NULL where a dimension misses
  CWM_SV32 = 1,   // starjoin_cwm_sv: int32 per row, and the count of the others
  CWM_MARK16 = 2, // the *_dv lists: marks of the surviving rows, int16 or int32 ids
  CWM_MARK32 = 3,
};

// Copies the staged vectors of this block into shared memory; bit j of the
// result: dimension j is probed there.  *late: the first of them keeps more
// than 3/4 of its entries.  4-bit codes (two per byte, low first, 15 = DIM_NULL) are
// packed here from the int8 vector; one with any other code than DIM_NULL and
// 0..14 is probed through L2 instead.
__device__ __forceinline__ uint32_t stage_dims(const DimSet& d, unsigned char* sdim, bool* late) {
  uint32_t staged = 0;
  __shared__ uint32_t s_null[OLAP_MAX_DIMS];
  if (threadIdx.x < OLAP_MAX_DIMS) s_null[threadIdx.x] = 0;
  __syncthreads();
#pragma unroll
  for (int j = 0; j < OLAP_MAX_DIMS; ++j) {
    if (j >= d.nd || d.off[j] < 0) continue;
    const int8_t* src = d.vec[j];
    unsigned char* dst = sdim + d.off[j];
    const uint32_t n16 = (reinterpret_cast<uintptr_t>(src) & 15) == 0 ? d.len[j] >> 4 : 0u;
    uint32_t bad = 0, null8 = 0;  // entries that are DIM_NULL, eight per count
    auto nulls = [&](uint32_t w) {
      const uint32_t m = __vcmpeq4(w, 0x7F7F7F7Fu);
      null8 += __popc(m);
      return m;
    };
    auto pack4 = [&](uint32_t w) -> uint32_t {  // 4 codes to 16 bits
      bad |= ~(nulls(w) | __vcmpltu4(w, 0x0F0F0F0Fu));
      const uint32_t x = w & 0x0F0F0F0Fu, y = x | (x >> 4);
      return (y & 0xFFu) | ((y >> 8) & 0xFF00u);
    };
    if (!d.nib[j]) {
      for (uint32_t i = threadIdx.x; i < n16; i += blockDim.x) {
        const int4 v = __ldg(reinterpret_cast<const int4*>(src) + i);
        nulls(v.x); nulls(v.y); nulls(v.z); nulls(v.w);
        reinterpret_cast<int4*>(dst)[i] = v;
      }
      for (uint32_t i = (n16 << 4) + threadIdx.x; i < d.len[j]; i += blockDim.x) {
        null8 += src[i] == OLAP_DIM_NULL ? 8 : 0;
        dst[i] = src[i];
      }
    } else {
      for (uint32_t i = threadIdx.x; i < n16; i += blockDim.x) {
        const int4 v = __ldg(reinterpret_cast<const int4*>(src) + i);
        reinterpret_cast<uint2*>(dst)[i] = make_uint2(pack4(v.x) | pack4(v.y) << 16, pack4(v.z) | pack4(v.w) << 16);
      }
      for (uint32_t i = 2 * ((n16 << 3) + threadIdx.x); i < d.len[j]; i += 2 * blockDim.x) {
        const uint32_t lo = static_cast<uint8_t>(src[i]), hi = i + 1 < d.len[j] ? static_cast<uint8_t>(src[i + 1]) : 127u;
        dst[i >> 1] = static_cast<unsigned char>(pack4(lo | hi << 8));
      }
    }
    null8 = __reduce_add_sync(0xffffffffu, null8);
    if ((threadIdx.x & 31) == 0 && null8) atomicAdd(&s_null[j], null8 >> 3);
    if (__syncthreads_or(bad != 0)) continue;
    staged |= 1u << j;
    if (j == 0) *late = s_null[0] < d.len[0] >> 2;
  }
  __syncthreads();
  return staged;
}

// All dimensions of the rows in one pass, a warp on a tile of rows at a time,
// 128 rows at a step: lane l the rows 4 l .. 4 l + 3 by 16-byte key loads (VEC),
// or where a column is not aligned the rows 32 u + l, so that the loads of a
// warp are still runs (60M rows to the vector: 788 us with four neighbours per
// lane there, 252 us so).  Every key is range-checked first (a row with one out
// of range is dropped and counted), then the dimensions are probed: those
// staged in shared memory, smallest first, then the rest through L2; with LATE
// the first of them last (a dimension that keeps nearly everything filters
// nothing before the L2 probes).  Bound by instructions, so a row is dropped
// without a branch or a predicate: its largest code stays DIM_NULL, and from
// then on it reads entry 0 of the vectors in L2, one line for all such rows.
template <int MODE, bool LATE, bool VEC>
__device__ __forceinline__ void cwm_probe_rows(const DimSet& d, const unsigned char* sdim, uint32_t staged, int64_t n,
                                               int32_t tile, int64_t n_tiles, void* __restrict__ out, const Marks& mk,
                                               int64_t* tot, unsigned int* bad) {
  const int lane = threadIdx.x & 31;
  const uint32_t lt = (1u << lane) - 1u;
  auto off = [lane](int u) { return VEC ? 4 * lane + u : 32 * u + lane; };  // a step's row of register slot u
  const uint64_t pol = policy_evict_first();
  const int64_t n_warps = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
  for (int64_t t = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5; t < n_tiles; t += n_warps) {
    const int64_t first = t * tile;
    const int len = static_cast<int>(first + tile < n ? tile : n - first);
    uint32_t c = 0;
    for (int r0 = 0; r0 < len; r0 += 128) {
      const int64_t r = first + r0;
      uint32_t k[OLAP_MAX_DIMS][4];
      int32_t top[4];  // largest code of the row so far: DIM_NULL once a dimension misses
      const bool full = r0 + 128 <= len;
      if (full) {
#pragma unroll
        for (int j = 0; j < OLAP_MAX_DIMS; ++j) {
          if (j >= d.nd) continue;
          if (VEC) {
            const int4 v = ld_stream_v4(d.fk[j] + r + 4 * lane, pol);
            k[j][0] = v.x; k[j][1] = v.y; k[j][2] = v.z; k[j][3] = v.w;
          } else {
#pragma unroll
            for (int u = 0; u < 4; ++u) k[j][u] = static_cast<uint32_t>(ld_stream_s32(d.fk[j] + r + off(u), pol));
          }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) top[u] = INT8_MIN;
      } else {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const bool in = r0 + off(u) < len;
          top[u] = in ? INT8_MIN : OLAP_DIM_NULL;
#pragma unroll
          for (int j = 0; j < OLAP_MAX_DIMS; ++j)
            if (j < d.nd) k[j][u] = static_cast<uint32_t>(ld_stream_s32_if(in, d.fk[j] + r + off(u), pol, 0));
        }
      }
      uint32_t out_of_range = 0;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        bool ok = true;
#pragma unroll
        for (int j = 0; j < OLAP_MAX_DIMS; ++j) ok &= j >= d.nd || k[j][u] < d.len[j];
        if (!ok) out_of_range |= 1u << u;
      }
      if (out_of_range) {  // rare: those rows count, and their keys become 0, so that no probe leaves its vector
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          if (!((out_of_range >> u) & 1u)) continue;
          *bad += top[u] != OLAP_DIM_NULL;
          top[u] = OLAP_DIM_NULL;
#pragma unroll
          for (int j = 0; j < OLAP_MAX_DIMS; ++j) k[j][u] = 0;
        }
      }
      int32_t g[4] = {0, 0, 0, 0};
#pragma unroll
      for (int q = 0; q < OLAP_MAX_DIMS; ++q) {
        const int j = LATE ? (q + 1) & (OLAP_MAX_DIMS - 1) : q;
        if (j >= d.nd) continue;
        int32_t v[4];
        if (!((staged >> j) & 1u)) {  // through L2; the dropped rows all read entry 0
#pragma unroll
          for (int u = 0; u < 4; ++u) v[u] = __ldg(d.vec[j] + (top[u] == OLAP_DIM_NULL ? 0u : k[j][u]));
        } else if (d.nib[j]) {  // code 15 is DIM_NULL
          const uint32_t* codes = reinterpret_cast<const uint32_t*>(sdim + d.off[j]);
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            v[u] = static_cast<int32_t>(codes[k[j][u] >> 3] >> ((k[j][u] << 2) & 31u)) & 15;
            top[u] = max(top[u], v[u] + (OLAP_DIM_NULL - 15));
          }
        } else {
          const int8_t* codes = reinterpret_cast<const int8_t*>(sdim + d.off[j]);
#pragma unroll
          for (int u = 0; u < 4; ++u) v[u] = codes[k[j][u]];
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          top[u] = max(top[u], v[u]);
          g[u] += v[u] * d.mul[j];
        }
      }
      bool live[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) live[u] = top[u] != OLAP_DIM_NULL;
      __syncwarp();
      if (MODE == CWM_SV16 || MODE == CWM_SV32) {
        int32_t v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) v[u] = live[u] ? g[u] : OLAP_GROUP_NULL;
        if (VEC && full) {
          if (MODE == CWM_SV16)
            *reinterpret_cast<short4*>(static_cast<int16_t*>(out) + r + 4 * lane) =
                make_short4(static_cast<int16_t>(v[0]), static_cast<int16_t>(v[1]), static_cast<int16_t>(v[2]),
                            static_cast<int16_t>(v[3]));
          else
            *reinterpret_cast<int4*>(static_cast<int32_t*>(out) + r + 4 * lane) = make_int4(v[0], v[1], v[2], v[3]);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          if (MODE == CWM_SV32) *tot += v[u] != OLAP_GROUP_NULL;
          if ((VEC && full) || r0 + off(u) >= len) continue;
          if (MODE == CWM_SV16) static_cast<int16_t*>(out)[r + off(u)] = static_cast<int16_t>(v[u]);
          else static_cast<int32_t*>(out)[r + off(u)] = v[u];
        }
      } else if (!VEC) {
        // a ballot is a word of the bitmap; the ids of a step go out as one run
        uint32_t w[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          w[u] = __ballot_sync(0xffffffffu, live[u]);
          const int64_t at = first + c + __popc(w[u] & lt);
          if (live[u] && MODE == CWM_MARK16) static_cast<int16_t*>(mk.vals)[at] = static_cast<int16_t>(g[u]);
          if (live[u] && MODE == CWM_MARK32) static_cast<int32_t*>(mk.vals)[at] = g[u];
          c += __popc(w[u]);
        }
        if (lane == 0) reinterpret_cast<uint4*>(mk.bits)[r >> 7] = make_uint4(w[0], w[1], w[2], w[3]);
      } else {
        // two lanes' 4 rows make a byte of the bitmap (the chunk's holds
        // whole 128-item steps); the ids in row order
        const uint32_t alive = static_cast<uint32_t>(live[0]) | static_cast<uint32_t>(live[1]) << 1 |
                               static_cast<uint32_t>(live[2]) << 2 | static_cast<uint32_t>(live[3]) << 3;
        const uint32_t hi = __shfl_down_sync(0xffffffffu, alive, 1);
        if (!(lane & 1))
          reinterpret_cast<unsigned char*>(mk.bits)[((first + r0) >> 3) + (lane >> 1)] = static_cast<unsigned char>(alive | hi << 4);
        if (__any_sync(0xffffffffu, alive)) {
          const uint32_t mine = __popc(alive);
          uint32_t inc = mine;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += y;
          }
          int64_t at = first + c + inc - mine;
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            if (!live[u]) continue;
            if (MODE == CWM_MARK16) static_cast<int16_t*>(mk.vals)[at++] = static_cast<int16_t>(g[u]);
            else static_cast<int32_t*>(mk.vals)[at++] = g[u];
          }
          c += __shfl_sync(0xffffffffu, inc, 31);
        }
      }
    }
    if ((MODE == CWM_MARK16 || MODE == CWM_MARK32) && lane == 0) mk.counts[t] = c;
  }
}

template <int MODE, bool VEC>
__global__ void __launch_bounds__(1024, 1) cwm_probe_kernel(const DimSet d, int64_t n, int32_t tile, int64_t n_tiles,
                                                            void* __restrict__ out, const Marks mk,
                                                            unsigned long long* count, unsigned long long* range_err) {
  extern __shared__ __align__(16) unsigned char sdim[];
  bool late = false;
  const uint32_t staged = stage_dims(d, sdim, &late);
  unsigned int bad = 0;
  int64_t tot = 0;
  if (late) cwm_probe_rows<MODE, true, VEC>(d, sdim, staged, n, tile, n_tiles, out, mk, &tot, &bad);
  else cwm_probe_rows<MODE, false, VEC>(d, sdim, staged, n, tile, n_tiles, out, mk, &tot, &bad);
  const unsigned int wbad = __reduce_add_sync(0xffffffffu, bad);
  if (MODE == CWM_SV32) tot = warp_sum_i64(tot);
  if ((threadIdx.x & 31) == 0) {
    if (wbad) atomicAdd(range_err, static_cast<unsigned long long>(wbad));
    if (MODE == CWM_SV32 && tot) atomicAdd(count, static_cast<unsigned long long>(tot));
  }
}

// The *_sv vectors of few rows: a thread per row and nothing staged, so a short
// kernel.  Four dimensions, 10,000 rows: 3.0 us, cwm_probe_kernel 5.4; 500,000
// rows 7.3 and 8.7 us, 1M rows 10.9 and 10.4, 2M rows 17.9 and 14.1.
constexpr int64_t kFewRows = 1 << 20;
template <int MODE>
__global__ void __launch_bounds__(256) cwm_few_rows_kernel(const DimSet d, int64_t n, void* __restrict__ out,
                                                           unsigned long long* count, unsigned long long* range_err) {
  const int64_t r = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  uint32_t k[OLAP_MAX_DIMS];
  bool ok = true, live = r < n;
#pragma unroll
  for (int j = 0; j < OLAP_MAX_DIMS; ++j) {
    if (j >= d.nd) continue;
    k[j] = live ? static_cast<uint32_t>(d.fk[j][r]) : 0u;
    ok &= k[j] < d.len[j];
  }
  const bool bad = live && !ok;
  live &= ok;
  int32_t g = 0;
#pragma unroll
  for (int j = 0; j < OLAP_MAX_DIMS; ++j) {
    if (j >= d.nd || !live) continue;
    const int32_t c = __ldg(d.vec[j] + k[j]);
    live = c != OLAP_DIM_NULL;
    g += c * d.mul[j];
  }
  const int32_t v = live ? g : OLAP_GROUP_NULL;
  if (r < n) {
    if (MODE == CWM_SV16) static_cast<int16_t*>(out)[r] = static_cast<int16_t>(v);
    else static_cast<int32_t*>(out)[r] = v;
  }
  const uint32_t wbad = __popc(__ballot_sync(0xffffffffu, bad));
  const uint32_t some = MODE == CWM_SV32 ? __popc(__ballot_sync(0xffffffffu, v != OLAP_GROUP_NULL)) : 0u;
  if ((threadIdx.x & 31) == 0) {
    if (wbad) atomicAdd(range_err, static_cast<unsigned long long>(wbad));
    if (some) atomicAdd(count, static_cast<unsigned long long>(some));
  }
}

// The surviving rows of join_cwm_dv (int64 OID, int16 group) ...
struct OidEmit {
  static constexpr bool kVals = true;
  const int16_t* vals;
  int64_t* oid;
  int16_t* gid;
  __device__ __forceinline__ void emit(int64_t pos, int64_t item, int64_t v) const {
    oid[pos] = item;
    gid[pos] = __ldg(vals + v);
  }
};
// ... and of starjoinalgo_cwm_dv (int32 position, int32 packed group).
struct PosEmit {
  static constexpr bool kVals = true;
  const int32_t* vals;
  int32_t* pos32;
  int32_t* grp32;
  __device__ __forceinline__ void emit(int64_t pos, int64_t item, int64_t v) const {
    pos32[pos] = static_cast<int32_t>(item);
    grp32[pos] = __ldg(vals + v);
  }
};

// group_vector[g] += v in a block's shared accumulators (low words, then high
// words) or, where they do not fit, in L2.
__device__ __forceinline__ void agg_cwm_add(uint32_t* sacc, bool smem, int64_t G, unsigned long long* gv, int32_t g,
                                            int64_t v, int64_t* tot) {
  *tot += v;
  if (smem) smem_add_split(sacc, G, g, static_cast<uint64_t>(v));
  else atomicAdd(&gv[g], static_cast<unsigned long long>(v));
}

// agg_cwm_sv / agg_cwm_dv: group_vector[g] += M1[row] + M2[row].  Bound by the
// latency of the measures' reads.  The list (oid): lane = consecutive entries,
// whose rows ascend and share lines, four per thread in flight.  The vector:
// two 16-byte loads of eight ids per thread, the next two already loading, and
// 16-byte loads of the measures of four rows where any of them survives.
__global__ void __launch_bounds__(512, 2) agg_cwm_kernel(const int16_t* __restrict__ gid,
                                                         const int64_t* __restrict__ oid, int64_t n,
                                                         const int32_t* __restrict__ m1,
                                                         const int32_t* __restrict__ m2, int64_t rows, int64_t G,
                                                         int vec, unsigned long long* __restrict__ gv,
                                                         unsigned long long* total, unsigned long long* range_err) {
  extern __shared__ uint32_t sacc[];
  const bool smem = G * 8 <= 64 * 1024;
  for (int64_t i = threadIdx.x; smem && i < 2 * G; i += blockDim.x) sacc[i] = 0;
  __syncthreads();
  const uint64_t pol = policy_evict_first();
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  const int64_t t0 = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  int64_t tot = 0;
  unsigned int bad = 0;
  int64_t done = 0;  // entries of the vectorised part
  if (oid) {
    done = n;
    const bool far = rows > 6 * n;  // few of a line's rows survive: fetch half of it
    for (int64_t i = t0; i < n; i += 4 * stride) {
      int32_t g[4], x[4], y[4];
      int64_t row[4];
      uint32_t live = 0;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int64_t e = i + u * stride;
        g[u] = e < n ? __ldg(gid + e) : OLAP_GROUP_NULL;
        row[u] = e < n ? __ldg(reinterpret_cast<const long long*>(oid) + e) : 0;
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const bool some = g[u] != OLAP_GROUP_NULL;
        const bool ok = some && g[u] >= 0 && g[u] < G && row[u] >= 0 && row[u] < rows;
        bad += some && !ok;
        live |= static_cast<uint32_t>(ok) << u;
        x[u] = ok ? (far ? ld_gather_64(m1 + row[u]) : __ldg(m1 + row[u])) : 0;
        y[u] = ok ? (far ? ld_gather_64(m2 + row[u]) : __ldg(m2 + row[u])) : 0;
      }
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if ((live >> u) & 1u) agg_cwm_add(sacc, smem, G, gv, g[u], static_cast<int64_t>(x[u]) + y[u], &tot);
    }
  } else if (vec) {
    const int64_t n8 = n >> 3;
    done = 8 * n8;
    const int4* g8 = reinterpret_cast<const int4*>(gid);
    constexpr int32_t kNull2 = OLAP_GROUP_NULL << 16 | OLAP_GROUP_NULL;
    const int4 none = make_int4(kNull2, kNull2, kNull2, kNull2);
    int4 next[2] = {t0 < n8 ? __ldg(g8 + t0) : none, t0 + stride < n8 ? __ldg(g8 + t0 + stride) : none};
    for (int64_t i = t0; i < n8; i += 2 * stride) {
      int32_t w[8];  // 16 ids
      int4 a[4], b[4];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int4 q = next[h];
        const int64_t e = i + h * stride;
        next[h] = e + 2 * stride < n8 ? __ldg(g8 + e + 2 * stride) : none;
        w[4 * h] = q.x; w[4 * h + 1] = q.y; w[4 * h + 2] = q.z; w[4 * h + 3] = q.w;
#pragma unroll
        for (int p = 0; p < 2; ++p) {
          const bool any = w[4 * h + 2 * p] != kNull2 || w[4 * h + 2 * p + 1] != kNull2;
          a[2 * h + p] = ld_stream_v4_if(any, m1 + 8 * e + 4 * p, pol);
          b[2 * h + p] = ld_stream_v4_if(any, m2 + 8 * e + 4 * p, pol);
        }
      }
#pragma unroll
      for (int p = 0; p < 4; ++p) {
        const int32_t x[4] = {a[p].x, a[p].y, a[p].z, a[p].w}, y[4] = {b[p].x, b[p].y, b[p].z, b[p].w};
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int32_t g = u & 1 ? w[2 * p + (u >> 1)] >> 16 : static_cast<int16_t>(w[2 * p + (u >> 1)]);
          if (g == OLAP_GROUP_NULL) continue;
          if (g < 0 || g >= G) ++bad;
          else agg_cwm_add(sacc, smem, G, gv, g, static_cast<int64_t>(x[u]) + y[u], &tot);
        }
      }
    }
  }
  for (int64_t i = done + t0; i < n; i += stride) {  // the vector, row by row
    const int32_t g = gid[i];
    if (g == OLAP_GROUP_NULL) continue;
    if (g < 0 || g >= G || i >= rows) ++bad;
    else agg_cwm_add(sacc, smem, G, gv, g, static_cast<int64_t>(m1[i]) + m2[i], &tot);
  }
  tot = warp_sum_i64(tot);
  const unsigned int wbad = __reduce_add_sync(0xffffffffu, bad);
  if ((threadIdx.x & 31) == 0) {
    if (tot) atomicAdd(total, static_cast<unsigned long long>(tot));
    if (wbad) atomicAdd(range_err, static_cast<unsigned long long>(wbad));
  }
  __syncthreads();
  for (int64_t i = threadIdx.x; smem && i < G; i += blockDim.x) {
    const unsigned long long v = smem_split_get(sacc, G, i);
    if (v) atomicAdd(&gv[i], v);
  }
}

static bool aligned_to(const void* p, uintptr_t a) { return (reinterpret_cast<uintptr_t>(p) & (a - 1)) == 0; }

// Dimensions in probe order from the reference's table-indexed arrays.
static int make_dims(olap_ctx* ctx, int8_t* const* dimvec_array, const int64_t* dimvec_len,
                     int32_t* const* fk_array, const int* orders, int dimvec_nums, const int* factor,
                     bool empty, DimSet* d) {
  std::memset(d, 0, sizeof(*d));
  OLAP_REQUIRE(ctx, dimvec_nums >= 0 && dimvec_nums <= OLAP_MAX_DIMS, "dimvec_nums must be in [0, 4]");
  OLAP_REQUIRE(ctx, dimvec_nums == 0 || (dimvec_array && fk_array && orders && factor && dimvec_len),
               "null plan arrays");
  d->nd = dimvec_nums;
  for (int j = 0; j < dimvec_nums; ++j) {
    const int t = orders[j];
    OLAP_REQUIRE(ctx, t >= 0 && t < OLAP_MAX_DIMS, "orders[] entry must name table 0..3");
    OLAP_REQUIRE(ctx, dimvec_array[t] && (empty || fk_array[t]), "null dimension vector or fk column");
    OLAP_REQUIRE(ctx, dimvec_len[t] >= 1 && dimvec_len[t] <= INT32_MAX, "dimvec_len must be in [1, 2^31)");
    d->vec[j] = dimvec_array[t];
    d->fk[j] = fk_array[t];
    d->len[j] = static_cast<uint32_t>(dimvec_len[t]);
    d->mul[j] = factor[j];
  }
  return OLAP_OK;
}

constexpr int kStageBytes = 112 * 1024;

// Probe order and staging for n rows: smallest dimension first (the order
// does not change the ids); a vector goes to shared memory whole up to 32 KB,
// as 4-bit codes above (half the bytes, which leaves L1 the room that the
// loads in flight need), while all of it stays within 112 KB and the rows a
// block probes repay its copy.
static void stage_plan(DimSet* d, int64_t n) {
  int idx[OLAP_MAX_DIMS] = {0, 1, 2, 3};
  const DimSet in = *d;
  std::stable_sort(idx, idx + d->nd, [&](int a, int b) { return in.len[a] < in.len[b]; });
  d->smem = 0;
  for (int j = 0; j < d->nd; ++j) {
    const int s = idx[j];
    d->vec[j] = in.vec[s];
    d->fk[j] = in.fk[s];
    d->len[j] = in.len[s];
    d->mul[j] = in.mul[s];
    d->nib[j] = in.len[s] > 32 * 1024;
    const int64_t bytes = ((d->nib[j] ? (static_cast<int64_t>(in.len[s]) + 1) / 2 : in.len[s]) + 15) & ~int64_t(15);
    d->off[j] = -1;
    if (d->smem + bytes <= kStageBytes && n >= 16 * static_cast<int64_t>(in.len[s])) {
      d->off[j] = d->smem;
      d->smem += static_cast<int32_t>(bytes);
    }
  }
}

template <int MODE>
static int launch_probe(olap_ctx* ctx, const DimSet& d, int64_t n, int32_t tile, void* out, const Marks& mk,
                        unsigned long long* count) {
  unsigned grid, block;
  const int64_t n_tiles = (n + tile - 1) / tile;
  mark_grid(ctx, n_tiles, 1024, 1, &grid, &block);
  bool vec = aligned_to(out, MODE == CWM_SV16 ? 8 : 16);
  for (int j = 0; j < d.nd; ++j) vec &= aligned_to(d.fk[j], 16);
  auto* const kernel = vec ? cwm_probe_kernel<MODE, true> : cwm_probe_kernel<MODE, false>;
  OLAP_CUDA_TRY(ctx, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kStageBytes));
  kernel<<<grid, block, static_cast<size_t>(d.smem), ctx->stream>>>(d, n, tile, n_tiles, out, mk, count,
                                                                  &ctx->counters->range_errors);
  OLAP_CUDA_TRY(ctx, cudaGetLastError());
  return OLAP_OK;
}

// One value per row (the *_sv vectors).
template <int MODE>
static int row_vector(olap_ctx* ctx, DimSet d, int64_t n, void* out, unsigned long long* count) {
  if (n <= kFewRows) {
    cwm_few_rows_kernel<MODE><<<static_cast<unsigned>((n + 255) / 256), 256, 0, ctx->stream>>>(
        d, n, out, count, &ctx->counters->range_errors);
    OLAP_CUDA_TRY(ctx, cudaGetLastError());
    return OLAP_OK;
  }
  stage_plan(&d, n);
  const int64_t tile = std::min<int64_t>(mark_tile(n, ctx->sm_count * int64_t(32)), 1 << 20);
  return launch_probe<MODE>(ctx, d, n, static_cast<int32_t>(tile), out, Marks{}, count);
}

// The surviving rows in row order: marks of each chunk, then their expansion.
template <int MODE, class Emit>
static int survivors(olap_ctx* ctx, DimSet d, int64_t n, Emit em, int64_t* d_count) {
  stage_plan(&d, n);
  Arena ar(ctx);
  using V = std::remove_const_t<std::remove_pointer_t<decltype(em.vals)>>;
  return mark_and_expand(ctx, ar, n, sizeof(V), ctx->sm_count * int64_t(32), em,
                         reinterpret_cast<unsigned long long*>(d_count),
                         [&](const Marks& mk, int64_t first, Emit& e) {
                           e.vals = static_cast<const V*>(mk.vals);
                           DimSet c = d;
                           for (int j = 0; j < d.nd; ++j) c.fk[j] = d.fk[j] + first;
                           return launch_probe<MODE>(ctx, c, mk.n, mk.tile, nullptr, mk, nullptr);
                         });
}

}  // namespace olap

extern "C" {

int olap_join_cwm_sv(olap_ctx* ctx, int8_t* const* dimvec_array, const int64_t* dimvec_len,
                     int32_t* const* fk_array, const int* orders, int dimvec_nums, int16_t* groupID,
                     const int* factor, int64_t size_lineorder) {
  if (!ctx) return OLAP_ERR_INVALID;
  std::lock_guard<std::mutex> lk(ctx->mu);
  OLAP_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  OLAP_REQUIRE(ctx, size_lineorder >= 0 && (size_lineorder == 0 || groupID), "bad output");
  olap::DimSet d;
  int st = olap::make_dims(ctx, dimvec_array, dimvec_len, fk_array, orders, dimvec_nums, factor,
                           size_lineorder == 0, &d);
  if (st != OLAP_OK || size_lineorder == 0) return st;
  return olap::row_vector<olap::CWM_SV16>(ctx, d, size_lineorder, groupID, nullptr);
}

int olap_agg_cwm_sv(olap_ctx* ctx, const int16_t* groupID, int64_t size_lineorder, const int32_t* M1,
                    const int32_t* M2, int64_t group_nums, int64_t* group_vector, int64_t* d_count) {
  if (!ctx) return OLAP_ERR_INVALID;
  std::lock_guard<std::mutex> lk(ctx->mu);
  OLAP_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  OLAP_REQUIRE(ctx, group_nums >= 1 && group_nums <= 32766, "group_nums must be in [1, 32766] (int16 ids)");
  OLAP_REQUIRE(ctx, size_lineorder >= 0 && group_vector && d_count, "bad arguments");
  OLAP_REQUIRE(ctx, size_lineorder == 0 || (groupID && M1 && M2), "null column");
  OLAP_CUDA_TRY(ctx, cudaMemsetAsync(group_vector, 0, sizeof(int64_t) * group_nums, ctx->stream));
  OLAP_CUDA_TRY(ctx, cudaMemsetAsync(d_count, 0, sizeof(int64_t), ctx->stream));
  if (size_lineorder == 0) return OLAP_OK;
  const size_t smem = group_nums * 8 <= 64 * 1024 ? static_cast<size_t>(group_nums * 8) : 0;
  OLAP_CUDA_TRY(ctx, cudaFuncSetAttribute(olap::agg_cwm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          64 * 1024));
  const int vec = olap::aligned_to(groupID, 16) && olap::aligned_to(M1, 16) && olap::aligned_to(M2, 16);
  const int64_t blocks = std::min<int64_t>(ctx->sm_count * int64_t(2), (size_lineorder + 2047) / 2048);
  olap::agg_cwm_kernel<<<static_cast<unsigned>(blocks), 512, smem, ctx->stream>>>(
      groupID, nullptr, size_lineorder, M1, M2, size_lineorder, group_nums, vec,
      reinterpret_cast<unsigned long long*>(group_vector), reinterpret_cast<unsigned long long*>(d_count),
      &ctx->counters->range_errors);
  OLAP_CUDA_TRY(ctx, cudaGetLastError());
  return OLAP_OK;
}

int olap_join_cwm_dv(olap_ctx* ctx, int8_t* const* dimvec_array, const int64_t* dimvec_len,
                     int32_t* const* fk_array, const int* orders, int dimvec_nums, int64_t* OID,
                     int16_t* groupID, const int* factor, int64_t* d_index, int64_t size_lineorder) {
  if (!ctx) return OLAP_ERR_INVALID;
  std::lock_guard<std::mutex> lk(ctx->mu);
  OLAP_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  OLAP_REQUIRE(ctx, size_lineorder >= 0 && d_index && (size_lineorder == 0 || (OID && groupID)), "bad output");
  olap::DimSet d;
  int st = olap::make_dims(ctx, dimvec_array, dimvec_len, fk_array, orders, dimvec_nums, factor,
                           size_lineorder == 0, &d);
  if (st != OLAP_OK) return st;
  return olap::survivors<olap::CWM_MARK16>(ctx, d, size_lineorder, olap::OidEmit{nullptr, OID, groupID}, d_index);
}

int olap_agg_cwm_dv(olap_ctx* ctx, const int64_t* OID, const int16_t* groupID, int64_t index,
                    const int32_t* M1, const int32_t* M2, int64_t size_lineorder, int64_t group_nums,
                    int64_t* group_vector, int64_t* d_count) {
  if (!ctx) return OLAP_ERR_INVALID;
  std::lock_guard<std::mutex> lk(ctx->mu);
  OLAP_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  OLAP_REQUIRE(ctx, group_nums >= 1 && group_nums <= 32766, "group_nums must be in [1, 32766] (int16 ids)");
  OLAP_REQUIRE(ctx, index >= 0 && group_vector && d_count, "bad arguments");
  OLAP_REQUIRE(ctx, index == 0 || (OID && groupID && M1 && M2), "null column");
  OLAP_CUDA_TRY(ctx, cudaMemsetAsync(group_vector, 0, sizeof(int64_t) * group_nums, ctx->stream));
  OLAP_CUDA_TRY(ctx, cudaMemsetAsync(d_count, 0, sizeof(int64_t), ctx->stream));
  if (index == 0) return OLAP_OK;
  const size_t smem = group_nums * 8 <= 64 * 1024 ? static_cast<size_t>(group_nums * 8) : 0;
  OLAP_CUDA_TRY(ctx, cudaFuncSetAttribute(olap::agg_cwm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          64 * 1024));
  const int64_t blocks = std::min<int64_t>(ctx->sm_count * int64_t(2), (index + 2047) / 2048);
  olap::agg_cwm_kernel<<<static_cast<unsigned>(blocks), 512, smem, ctx->stream>>>(
      groupID, OID, index, M1, M2, size_lineorder, group_nums, 0,
      reinterpret_cast<unsigned long long*>(group_vector), reinterpret_cast<unsigned long long*>(d_count),
      &ctx->counters->range_errors);
  OLAP_CUDA_TRY(ctx, cudaGetLastError());
  return OLAP_OK;
}

int olap_starjoin_count(olap_ctx* ctx, int64_t size_lineorder, int8_t* const* dimvec, const int64_t* dimvec_len,
                        int32_t* const* fk, int64_t* d_count) {
  if (!ctx) return OLAP_ERR_INVALID;
  std::lock_guard<std::mutex> lk(ctx->mu);
  OLAP_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  OLAP_REQUIRE(ctx, dimvec && dimvec_len && fk && d_count, "null argument");
  olap_starjoin_query q;
  std::memset(&q, 0, sizeof(q));
  q.dimvec_nums = OLAP_MAX_DIMS;
  q.n_aggs = 1;
  q.agg[0] = OLAP_AGG_COUNT;
  for (int j = 0; j < OLAP_MAX_DIMS; ++j) {
    q.dimvec[j] = dimvec[j];
    q.dimvec_len[j] = dimvec_len[j];
    q.fk[j] = fk[j];
    q.factor[j] = 0;
  }
  q.row_begin = 0;
  q.row_end = size_lineorder;
  q.group_nums = 1;
  olap::Arena ar(ctx);
  return olap::starjoin_device(ctx, &q, nullptr, d_count, false, ctx->stream, ar);
}

int olap_starjoin_cwm_sv(olap_ctx* ctx, int64_t size_lineorder, int8_t* const* dimvec,
                         const int64_t* dimvec_len, int32_t* const* fk, int32_t* result, int64_t* d_count) {
  if (!ctx) return OLAP_ERR_INVALID;
  std::lock_guard<std::mutex> lk(ctx->mu);
  OLAP_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  OLAP_REQUIRE(ctx, dimvec && dimvec_len && fk && d_count && size_lineorder >= 0, "null argument");
  OLAP_REQUIRE(ctx, size_lineorder == 0 || result, "null result");
  const int orders[4] = {0, 1, 2, 3};
  const int shifts[4] = {1 << 12, 1 << 8, 1 << 4, 1};  // GROUP_BITS_TABLE = 4 (metadata.h:76)
  olap::DimSet d;
  int st = olap::make_dims(ctx, dimvec, dimvec_len, fk, orders, 4, shifts, size_lineorder == 0, &d);
  if (st != OLAP_OK) return st;
  OLAP_CUDA_TRY(ctx, cudaMemsetAsync(d_count, 0, sizeof(int64_t), ctx->stream));
  if (size_lineorder == 0) return OLAP_OK;
  return olap::row_vector<olap::CWM_SV32>(ctx, d, size_lineorder, result, reinterpret_cast<unsigned long long*>(d_count));
}

int olap_starjoin_cwm_dv(olap_ctx* ctx, int64_t size_lineorder, int8_t* const* dimvec,
                         const int64_t* dimvec_len, int32_t* const* fk, int32_t* out_pos,
                         int32_t* out_group, int64_t* d_count) {
  if (!ctx) return OLAP_ERR_INVALID;
  std::lock_guard<std::mutex> lk(ctx->mu);
  OLAP_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  OLAP_REQUIRE(ctx, dimvec && dimvec_len && fk && d_count && size_lineorder >= 0 && size_lineorder <= INT32_MAX,
               "bad argument");
  OLAP_REQUIRE(ctx, size_lineorder == 0 || (out_pos && out_group), "null output");
  const int orders[4] = {0, 1, 2, 3};
  const int shifts[4] = {1 << 12, 1 << 8, 1 << 4, 1};
  olap::DimSet d;
  int st = olap::make_dims(ctx, dimvec, dimvec_len, fk, orders, 4, shifts, size_lineorder == 0, &d);
  if (st != OLAP_OK) return st;
  return olap::survivors<olap::CWM_MARK32>(ctx, d, size_lineorder, olap::PosEmit{nullptr, out_pos, out_group}, d_count);
}

}  // extern "C"
