// INNER probe fused with the payload gather for the sm_100a equi-join. Replaces
// hash_join::inner_join / distinct_hash_join::inner_join / cudf::inner_join
// (src/op/sirius_physical_hash_join.cpp:1671, :1688, :1872) and the two cudf::gather calls of
// gather_join_output (:1299-1359): the output row (probe rid, build rid, probe payloads, build
// payloads) is written once, by the kernel that found the match.
//
// DISTINCT tables (one slot per build row, unique keys) take a single pass, the unit probe
// (sj_probe_units.cu) where it serves the output, else the staged kernel here:
//   - every thread owns KPT = 4 consecutive probe rows and reads their keys with 128-bit
//     streaming loads (ld.global.cs: the probe stream must not evict the table from L2);
//   - keys outside [key_min, key_max] or NULL are rejected without touching the table;
//   - the thread issues the KPT bucket loads (32 B = one sector each) back to back, so a warp
//     keeps 128 independent sector reads in flight;
//   - matches are compacted warp-aggregated: __shfl_up prefix of the per-lane hit counts and one
//     atomicAdd per warp reserves the warp's output range;
//   - payloads are gathered straight into the reserved positions (build columns by row id).
// GROUPED tables (duplicated keys, or NULLs equal) take match -> scan -> expand:
//   - match_units (sj_probe_units.cu) finds each probe row's group and appends {probe row, group start} and
//     the group size to a compacted match list, summing the output size M;
//   - an exclusive scan turns group sizes into output offsets;
//   - the expand kernel gives every warp tiles of 256 consecutive outputs and finds each output's entry, so
//     a probe key matching 10^6 build rows is spread over the whole GPU instead of one thread.
#include <algorithm>
#include <type_traits>

#include "sj_device.cuh"
#include "sj_internal.h"
#include "sj_partition.cuh"
#include "sj_probe_direct.h"
#include "sj_probe_units.h"
#include "sj_scan.cuh"
#include "sj_units.cuh"

namespace sj {

TableDev table_dev(const sj_table* t);

constexpr int KPT = 4;  // probe rows per thread per tile

template <typename K>
__device__ __forceinline__ void load_keys(const K* __restrict__ keys, int64_t row0, int64_t n, bool vec,
                                          K (&k)[KPT]) {
  if (vec && row0 + KPT <= n) {
    if (sizeof(K) == 4) {
      const int4 x = __ldcs(reinterpret_cast<const int4*>(keys + row0));
      k[0] = (K)x.x;
      k[1] = (K)x.y;
      k[2] = (K)x.z;
      k[3] = (K)x.w;
    } else {
      const longlong2* p = reinterpret_cast<const longlong2*>(keys + row0);
      const longlong2 x = __ldcs(p), y = __ldcs(p + 1);
      k[0] = (K)x.x;
      k[1] = (K)x.y;
      k[2] = (K)y.x;
      k[3] = (K)y.y;
    }
  } else {
#pragma unroll
    for (int j = 0; j < KPT; ++j) k[j] = row0 + j < n ? __ldcs(keys + row0 + j) : (K)0;
  }
}

__device__ __forceinline__ uint64_t load_elem_cs(const void* base, int64_t i, int w) {
  switch (w) {
    case 8: return __ldcs(reinterpret_cast<const unsigned long long*>(base) + i);
    case 4: return __ldcs(reinterpret_cast<const unsigned int*>(base) + i);
    case 2: return __ldcs(reinterpret_cast<const unsigned short*>(base) + i);
    default: return __ldg(reinterpret_cast<const unsigned char*>(base) + i);
  }
}

// Rows of a probe tile that can match: in range, valid. Bit j = row0 + j.
template <typename K>
__device__ __forceinline__ uint32_t live_rows(const TableDev& t, const K (&k)[KPT], int64_t row0, int64_t n,
                                              const uint32_t* kv, int64_t kvoff) {
  uint32_t act = 0;
#pragma unroll
  for (int j = 0; j < KPT; ++j) {
    const int64_t r = row0 + j;
    if (r < n && bit_valid(kv, kvoff, r) && in_range(t, k[j])) act |= 1u << j;
  }
  return act;
}

// ------------------------------------------------------------------------------------------------
// Warp write-out. A warp stages its matches (probe row, build row id) in shared memory in
// compacted order, reserves one output range with a single atomicAdd, and then writes every
// output column with consecutive lanes on consecutive positions: full 32-byte sectors reach L2
// instead of lane-strided partial ones, and the probe payload is read in near-sequential order.
// ------------------------------------------------------------------------------------------------
constexpr int kProbeThreads = 256;
constexpr int kWarpsPerCta = kProbeThreads / 32;
constexpr int kStage = 32 * KPT;  // matches one warp can stage per tile

template <bool STREAM>
__device__ __forceinline__ void emit_column(const PayloadIn& in, const PayloadOut& o, const int32_t* s_idx,
                                            uint32_t tot, int64_t base, int64_t cap) {
  const int lane = threadIdx.x & 31;
  uint64_t v[KPT];
#pragma unroll
  for (int u = 0; u < KPT; ++u) {
    const uint32_t i = lane + 32u * u;
    v[u] = 0;
    if (i < tot) v[u] = STREAM && in.stride == in.width ? load_elem_cs(in.data, s_idx[i], in.width) : pl_load(in, s_idx[i]);
  }
#pragma unroll
  for (int u = 0; u < KPT; ++u) {
    const uint32_t i = lane + 32u * u;
    const int64_t p = base + i;
    const bool live = i < tot && p < cap;
    if (live) store_elem(o.data, p, in.width, v[u]);
    if (has_validity(in)) {
      const unsigned bits = __ballot_sync(kFullMask, live && payload_valid(in, s_idx[i]));
      if (lane == 0 && bits) {
        const int64_t p0 = base + 32u * u;
        const int sh = (int)(p0 & 31);
        atomicOr(o.valid + (p0 >> 5), bits << sh);
        if (sh && (bits >> (32 - sh))) atomicOr(o.valid + (p0 >> 5) + 1, bits >> (32 - sh));
      }
    }
  }
}

// s_row: probe array indices (row ids unless the probe was partitioned: prid_map).
// s_rid: table positions (build row ids unless the table maps them: brid_map); rewritten in
// place to build row ids after the position-ordered attached payloads have been gathered.
// Row-store write-out: one record load per match gives the build row id and all attached fields.
__device__ __forceinline__ void write_records(const Record (&r)[KPT / 2], int half, uint32_t tot, int64_t base,
                                              const GatherArgs& g) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int h = 0; h < KPT / 2; ++h) {
    const uint32_t i = lane + 32u * (half * (KPT / 2) + h);
    const int64_t p = base + i;
    const bool live = i < tot && p < g.capacity;
    if (live && g.out_brid) g.out_brid[p] = (int32_t)r[h].w[0];
    for (int c = 0; c < g.n_bin; ++c) {
      const int w = g.bin[c].width;
      if (live) store_elem(g.bout[c].data, p, w, record_field(r[h], g.rec_off[c], w));
      if (g.rec_voff[c] >= 0) {
        const unsigned bits = __ballot_sync(kFullMask, live && record_field(r[h], g.rec_voff[c], 1) != 0);
        if (lane == 0 && bits) {
          const int64_t p0 = base + 32u * (half * (KPT / 2) + h);
          const int sh = (int)(p0 & 31);
          atomicOr(g.bout[c].valid + (p0 >> 5), bits << sh);
          if (sh && (bits >> (32 - sh))) atomicOr(g.bout[c].valid + (p0 >> 5) + 1, bits >> (32 - sh));
        }
      }
    }
  }
}

__device__ __forceinline__ void load_records(Record (&r)[KPT / 2], int half, const int32_t* s_rid, uint32_t tot,
                                             const GatherArgs& g) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int h = 0; h < KPT / 2; ++h) {
    const uint32_t i = lane + 32u * (half * (KPT / 2) + h);
    if (i < tot)
      r[h] = load_record(static_cast<const char*>(g.rec) + (int64_t)s_rid[i] * g.rec_stride, g.rec_stride);
  }
}

// s_row: probe array indices (row ids unless the probe was partitioned: prid_map).
// s_rid: table positions (build row ids unless the table maps them: brid_map); rewritten in
// place to build row ids after the position-ordered attached payloads have been gathered.
// base: the warp's first output position; when `deferred` it is lane 0's still-pending atomicAdd
// result, broadcast only after this warp's gather loads are in flight.
__device__ __forceinline__ void warp_write_out(const int32_t* s_row, int32_t* s_rid, uint32_t tot,
                                               unsigned long long base_in, bool deferred, const GatherArgs& g) {
  const int lane = threadIdx.x & 31;
  if (g.rec) {
    const int64_t base = (int64_t)(deferred ? __shfl_sync(kFullMask, base_in, 0) : base_in);
    if (g.out_prid) {
      for (uint32_t i = lane; i < tot; i += 32) {
        const int64_t p = base + i;
        if (p < g.capacity) g.out_prid[p] = g.prid_map ? __ldg(g.prid_map + s_row[i]) : s_row[i];
      }
    }
    Record r[KPT / 2];
    load_records(r, 0, s_rid, tot, g);
    write_records(r, 0, tot, base, g);
    load_records(r, 1, s_rid, tot, g);
    write_records(r, 1, tot, base, g);
    for (int c = 0; c < g.n_pin; ++c) emit_column<true>(g.pin[c], g.pout[c], s_row, tot, base, g.capacity);
    return;
  }
  const int64_t base = (int64_t)(deferred ? __shfl_sync(kFullMask, base_in, 0) : base_in);
  if (g.out_prid) {
    for (uint32_t i = lane; i < tot; i += 32) {
      const int64_t p = base + i;
      if (p < g.capacity) g.out_prid[p] = g.prid_map ? __ldg(g.prid_map + s_row[i]) : s_row[i];
    }
  }
  if (g.bin_by_pos)
    for (int c = 0; c < g.n_bin; ++c) emit_column<false>(g.bin[c], g.bout[c], s_rid, tot, base, g.capacity);
  if (g.brid_map) {
    for (uint32_t i = lane; i < tot; i += 32) s_rid[i] = brid_of(g, s_rid[i]);
    __syncwarp();
  }
  if (g.out_brid) {
    for (uint32_t i = lane; i < tot; i += 32) {
      const int64_t p = base + i;
      if (p < g.capacity) g.out_brid[p] = s_rid[i];
    }
  }
  if (!g.bin_by_pos)
    for (int c = 0; c < g.n_bin; ++c) emit_column<false>(g.bin[c], g.bout[c], s_rid, tot, base, g.capacity);
  for (int c = 0; c < g.n_pin; ++c) emit_column<true>(g.pin[c], g.pout[c], s_row, tot, base, g.capacity);
}

// ------------------------------------------------------------------------------------------------
// DISTINCT: probe + gather in one pass
// ------------------------------------------------------------------------------------------------
// CTA_AGG: the CTA sums its warps' match counts and reserves the whole tile's output range with
// one atomicAdd (instead of one per warp), which matters when a probe of tens of millions of rows
// would otherwise queue ~10^5-10^6 atomics on the single output counter.
template <typename K, bool WIDE, bool VEC, bool COUNT_ONLY, bool CTA_AGG>
__global__ void __launch_bounds__(kProbeThreads, 4) probe_distinct_kernel(TableDev t, const K* __restrict__ keys,
                                                                           const uint32_t* __restrict__ kv,
                                                                           int64_t kvoff, int64_t n_host,
                                                                           const int64_t* d_n, GatherArgs g) {
  using Ops = SlotOps<WIDE>;
  __shared__ int32_t s_row[kWarpsPerCta][kStage];
  __shared__ int32_t s_rid[kWarpsPerCta][kStage];
  __shared__ unsigned s_wtot[kWarpsPerCta], s_wbase[kWarpsPerCta];
  __shared__ unsigned long long s_cta_base;
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int64_t n = d_n ? *d_n : n_host;
  const int64_t per_cta = (int64_t)blockDim.x * KPT;
  const int64_t tiles = (n + per_cta - 1) / per_cta;
  unsigned long long counted = 0;
  for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const int64_t row0 = tile * per_cta + (int64_t)threadIdx.x * KPT;
    K k[KPT];
    load_keys<K>(keys, row0, n, VEC, k);
    uint32_t act = live_rows<K>(t, k, row0, n, kv, kvoff);
    uint32_t b[KPT];
    uint64_t ks[KPT];
    const uint64_t kmask = ~((1ull << t.rbits) - 1);
#pragma unroll
    for (int j = 0; j < KPT; ++j) {
      const uint64_t kb = key_u64<K>(k[j]);
      b[j] = home_bucket(t, kb);
      ks[j] = Ops::probe_key((uint64_t)(long long)k[j] - (uint64_t)t.kmin, kb, t.rbits);
    }
    int32_t rid[KPT] = {0, 0, 0, 0};
    uint32_t hit = 0;
    for (uint32_t step = 0; act && step <= t.segmask; ++step) {
      Bucket bk[KPT];
#pragma unroll
      for (int j = 0; j < KPT; ++j)
        if (act >> j & 1u) bk[j] = load_bucket<true>(t.slots, b[j]);
#pragma unroll
      for (int j = 0; j < KPT; ++j) {
        if (!(act >> j & 1u)) continue;
        bool done = false;
#pragma unroll
        for (int q = 0; q < Ops::kSlots; ++q) {
          if (!done && Ops::match_s(bk[j], q, ks[j], kmask)) {
            rid[j] = Ops::rid(bk[j], q, t.rbits);
            hit |= 1u << j;
            done = true;
          }
          done |= Ops::empty(bk[j], q);
        }
        if (done) act &= ~(1u << j);
        else b[j] = next_bucket(b[j], t.segmask);
      }
    }
    const uint32_t cnt = __popc(hit);
    if (COUNT_ONLY) {
      counted += cnt;
      continue;
    }
    const uint32_t incl = warp_inclusive_sum(cnt);
    const uint32_t tot = __shfl_sync(kFullMask, incl, 31);
    if (!CTA_AGG && tot == 0) continue;
    uint32_t sp = incl - cnt;
#pragma unroll
    for (int j = 0; j < KPT; ++j) {
      if (hit >> j & 1u) {
        s_row[warp][sp] = (int32_t)(row0 + j);
        s_rid[warp][sp] = rid[j];
        ++sp;
      }
    }
    unsigned long long base = 0;
    bool deferred = false;
    if (CTA_AGG) {
      if (lane == 0) s_wtot[warp] = tot;
      __syncthreads();
      if (threadIdx.x == 0) {
        unsigned run = 0;
#pragma unroll
        for (int w = 0; w < kWarpsPerCta; ++w) {
          s_wbase[w] = run;
          run += s_wtot[w];
        }
        s_cta_base = run ? atomicAdd(g.d_count, (unsigned long long)run) : 0ull;
      }
      __syncthreads();
      base = s_cta_base + s_wbase[warp];
    } else {
      if (lane == 0) base = atomicAdd(g.d_count, (unsigned long long)tot);
      deferred = true;  // broadcast from lane 0 inside the write-out
      __syncwarp();
    }
    if (tot) warp_write_out(s_row[warp], s_rid[warp], tot, base, deferred, g);
    __syncwarp();
  }
  if (COUNT_ONLY) {
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) counted += __shfl_down_sync(kFullMask, counted, d);
    if (lane == 0 && counted) atomicAdd(g.d_count, counted);
  }
}

// ------------------------------------------------------------------------------------------------
// GROUPED expand: output position j -> (entry e with m_off[e] <= j < m_off[e+1]) -> one row.
//
// Every warp works alone (no CTA barrier): it owns a contiguous range of 256-output tiles and, per tile,
// stages the entries the tile touches (at most 256, 32 at a time until one starts behind the tile) as one
// 8-byte word each — probe row, and what to add to an output's place in the tile to get its group member —
// and one bit per output where an entry starts. An output's entry is then the number of starts up to it:
// one word, one popc, one 8-byte load from shared memory, whatever the groups' sizes. Lane l handles outputs
// j0 + 32m + l (m < 8), so each store is one coalesced warp access. A warp's first entry comes from a 32-ary
// search of m_off (5 steps for 32M entries); every later tile starts at the entry the previous tile ended in,
// and its first entries are loaded while the tile before is written. 32M Zipf probe rows into 8M, 1.1e8 outputs
// of 12 bytes: 427 us (511 before: 257 entries of 16 bytes staged for every 256 outputs, 92 instructions per
// output, now about 48). It waits for records and entries (8 loads per lane in flight, 32 warps per SM); fewer
// loads and more warps took 479 (4, 40 warps) and 551 us (2, 48 warps).
// ------------------------------------------------------------------------------------------------
constexpr int kExpandThreads = 256;
constexpr int kExpandWarps = kExpandThreads / 32;
constexpr int kExpandItems = 8;
constexpr int kExpandOut = 32 * kExpandItems;  // outputs per warp tile
constexpr int kExpandRun = 8;                  // consecutive tiles of a warp, fewer when there are not enough

// Largest e in [0, n) with off[e] <= j (off[0] <= j assumed), found by the whole warp: each step
// compares 32 evenly spaced candidates and keeps the gap between the last one at or below j and
// the next.
__device__ __forceinline__ int64_t warp_upper_index(const int64_t* off, int64_t n, int64_t j) {
  const int lane = threadIdx.x & 31;
  int64_t lo = 0, hi = n - 1;  // off[lo] <= j; the answer is in [lo, hi]
  while (lo < hi) {
    const int64_t span = hi - lo;
    const int64_t cand = lo + 1 + (span * lane) / 32;  // 32 candidates in (lo, hi]
    const bool le = cand <= hi && __ldg(off + cand) <= j;
    const unsigned m = __ballot_sync(kFullMask, le);
    if (m == 0) {
      hi = lo;  // every candidate (the first is lo + 1) is above j: the answer is lo
    } else {
      const int top = 31 - __clz(m);
      const int64_t c_top = lo + 1 + (span * top) / 32;
      const int64_t c_next = top < 31 ? lo + 1 + (span * (top + 1)) / 32 : hi + 1;
      lo = c_top;
      hi = c_next - 1;
    }
  }
  return lo;
}

// RS > 0: a compile-time output shape — row-store records of RS bytes holding the build row id and
// one payload of RS / 2 bytes at offset RS / 2 (no validity), no probe payloads; one load per row.
// RS = 0: the shape is read from `g` at run time.
template <int RS>
__global__ void __launch_bounds__(kExpandThreads, RS == 16 ? 3 : 4) expand_kernel(const int2* __restrict__ m_ent,
                                                                const int64_t* __restrict__ m_off,
                                                                const unsigned long long* d_nent,
                                                                const int32_t* __restrict__ grp_rid,
                                                                GatherArgs g) {
  __shared__ int2 s_ent_all[kExpandWarps][kExpandOut + 32];  // {probe row, group start - offset in the tile}
  __shared__ uint32_t s_start_all[kExpandWarps][kExpandItems];  // bit l of word m: an entry starts at 32 m + l > 0
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  int2* s_ent = s_ent_all[warp];
  uint32_t* s_starts = s_start_all[warp];
  const int64_t nent = (int64_t)*d_nent;
  if (nent == 0) return;
  const int64_t M = __ldg(m_off + nent);
  const int64_t cap = M < g.capacity ? M : g.capacity;
  const uint32_t ntile = (uint32_t)((cap + kExpandOut - 1) / kExpandOut);  // some output is written: it fits the device
  const uint32_t nwarps = gridDim.x * kExpandWarps;
  // every warp gets tiles first (1.2M outputs: 69 us with 8 tiles for each of 600 warps, 16 with one or two each)
  const uint32_t run = ntile >= nwarps * kExpandRun ? kExpandRun : 1 + ntile / nwarps;
  for (uint32_t t_lo = (blockIdx.x * kExpandWarps + warp) * run; t_lo < ntile; t_lo += nwarps * run) {
    const uint32_t t_hi = min(t_lo + run, ntile);
    int64_t e0 = warp_upper_index(m_off, nent, (int64_t)t_lo * kExpandOut);
    // the tile's first 32 entries, loaded while the tile before is written
    int64_t off = 0;
    int2 ent = make_int2(0, 0);
    auto fetch = [&]() {
      const bool in = e0 + lane < nent;
      off = in ? __ldg(m_off + e0 + lane) : INT64_MAX;
      if (in) ent = __ldg(m_ent + e0 + lane);
    };
    if (RS > 0) fetch();
    for (uint32_t tile = t_lo; tile < t_hi; ++tile) {
      if (RS == 0) fetch();  // this shape has no registers left to hold them
      const int64_t j0 = (int64_t)tile * kExpandOut;
      const int64_t j1 = j0 + kExpandOut < cap ? j0 + kExpandOut : cap;
      if (lane < kExpandItems) s_starts[lane] = 0;
      __syncwarp();
      auto stage = [&](int i) {
        const bool in = off < j1;
        const int rel = in ? (int)(off - j0) : 1;  // a group has at most 2^31 rows
        if (in) {
          s_ent[i + lane] = make_int2(ent.x, ent.y - rel);
          if (rel > 0) atomicOr(&s_starts[rel >> 5], 1u << (rel & 31));
        }
        return rel;
      };
      // one or two entries start at or before the tile
      int eb = __popc(__ballot_sync(kFullMask, stage(0) <= 0)) - 1;
      for (int i = 32; i < kExpandOut + 32 && __all_sync(kFullMask, off < j1); i += 32) {
        const int64_t e = e0 + i + lane;
        off = e < nent ? __ldg(m_off + e) : INT64_MAX;
        if (e < nent) ent = __ldg(m_ent + e);
        stage(i);
      }
      __syncwarp();
      // 1. entries: the starts up to each output, counted from the tile's first entry
      const unsigned upto = kFullMask >> (31 - lane);
      if constexpr (RS > 0) {
        // one record load per output, and stores at fixed distances from the tile's first output
        using V = std::conditional_t<RS == 8, uint2, uint4>;
        const int n_out = (int)(j1 - j0);
        int32_t row[kExpandItems];
        V v[kExpandItems];
#pragma unroll
        for (int m = 0; m < kExpandItems; ++m) {
          const uint32_t starts = s_starts[m];
          const int r = 32 * m + lane;
          if (r < n_out) {
            const int2 x = s_ent[eb + __popc(starts & upto)];
            row[m] = x.x;
            v[m] = __ldg(static_cast<const V*>(g.rec) + (uint32_t)(x.y + r));
          }
          eb += __popc(starts);
        }
        e0 += eb;  // the entry of the tile's last output
        if (tile + 1 < t_hi) fetch();
        int32_t* op = g.out_prid ? g.out_prid + j0 + lane : nullptr;
        int32_t* ob = g.out_brid ? g.out_brid + j0 + lane : nullptr;
        using P = std::conditional_t<RS == 8, unsigned int, unsigned long long>;
        P* oc = static_cast<P*>(g.bout[0].data) + j0 + lane;
#pragma unroll
        for (int m = 0; m < kExpandItems; ++m) {
          if (32 * m + lane >= n_out) continue;
          if (op) __stcs(op + 32 * m, row[m]);
          if (ob) __stcs(ob + 32 * m, (int32_t)v[m].x);
          if constexpr (RS == 8) __stcs(oc + 32 * m, v[m].y);
          else __stcs(oc + 32 * m, (unsigned long long)v[m].w << 32 | v[m].z);
        }
      } else {
        int32_t row[kExpandItems], gi[kExpandItems];
#pragma unroll
        for (int m = 0; m < kExpandItems; ++m) {
          const uint32_t starts = s_starts[m];
          const int r = 32 * m + lane;
          row[m] = 0;
          gi[m] = -1;
          if (j0 + r < j1) {
            const int2 x = s_ent[eb + __popc(starts & upto)];
            row[m] = x.x;
            gi[m] = x.y + r;
          }
          eb += __popc(starts);
        }
        e0 += eb;
        // 2. group members (table positions)
        int32_t pos[kExpandItems];
#pragma unroll
        for (int m = 0; m < kExpandItems; ++m) pos[m] = gi[m] < 0 ? 0 : grp_rid ? __ldg(grp_rid + gi[m]) : gi[m];
        // 3. build side: one row-store record per item, or row id (+ payloads by row id / position)
        if (g.rec) {
          constexpr int kHalf = kExpandItems / 2;  // 4 records (up to 32 registers) in flight at a time
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            Record r[kHalf];
#pragma unroll
            for (int q = 0; q < kHalf; ++q) {
              const int m = h * kHalf + q;
              if (gi[m] >= 0)
                r[q] = load_record(static_cast<const char*>(g.rec) + (int64_t)pos[m] * g.rec_stride, g.rec_stride);
            }
#pragma unroll
            for (int q = 0; q < kHalf; ++q) {
              const int m = h * kHalf + q;
              const int64_t j = j0 + 32 * m + lane;
              const bool live = gi[m] >= 0;
              if (live && g.out_prid) __stcs(g.out_prid + j, row[m]);
              if (live && g.out_brid) __stcs(g.out_brid + j, (int32_t)r[q].w[0]);
              for (int c = 0; c < g.n_bin; ++c) {
                const int w = g.bin[c].width;
                if (live) store_elem_cs(g.bout[c].data, j, w, record_field(r[q], g.rec_off[c], w));
                if (g.rec_voff[c] >= 0) {
                  const unsigned word = __ballot_sync(kFullMask, live && record_field(r[q], g.rec_voff[c], 1) != 0);
                  if (lane == 0 && j - lane < j1) g.bout[c].valid[(j - lane) >> 5] = word;
                }
              }
            }
          }
        } else {
          int32_t rid[kExpandItems];
#pragma unroll
          for (int m = 0; m < kExpandItems; ++m) rid[m] = gi[m] >= 0 ? brid_of(g, pos[m]) : 0;
#pragma unroll
          for (int m = 0; m < kExpandItems; ++m) {
            const int64_t j = j0 + 32 * m + lane;
            const bool live = gi[m] >= 0;
            if (live && g.out_prid) __stcs(g.out_prid + j, row[m]);
            if (live && g.out_brid) __stcs(g.out_brid + j, rid[m]);
            for (int c = 0; c < g.n_bin; ++c) {
              const PayloadIn in = g.bin[c];
              const int32_t idx = g.bin_by_pos ? pos[m] : rid[m];
              bool v = false;
              if (live) {
                store_elem_cs(g.bout[c].data, j, in.width, pl_load(in, idx));
                v = payload_valid(in, idx);
              }
              if (has_validity(in)) {
                const unsigned word = __ballot_sync(kFullMask, v);
                if (lane == 0 && j - lane < j1) g.bout[c].valid[(j - lane) >> 5] = word;
              }
            }
          }
        }
        // 4. probe payloads (by probe row)
        for (int c = 0; c < g.n_pin; ++c) {
          const PayloadIn in = g.pin[c];
          uint64_t v[kExpandItems];
#pragma unroll
          for (int m = 0; m < kExpandItems; ++m) v[m] = gi[m] >= 0 ? pl_load(in, row[m]) : 0;
#pragma unroll
          for (int m = 0; m < kExpandItems; ++m) {
            const int64_t j = j0 + 32 * m + lane;
            const bool live = gi[m] >= 0;
            if (live) store_elem_cs(g.pout[c].data, j, in.width, v[m]);
            if (has_validity(in)) {
              const unsigned word = __ballot_sync(kFullMask, live && payload_valid(in, row[m]));
              if (lane == 0 && j - lane < j1) g.pout[c].valid[(j - lane) >> 5] = word;
            }
          }
        }
      }
      __syncwarp();  // every lane is done with this tile's staged entries
    }
  }
}

// ------------------------------------------------------------------------------------------------
// host side
// ------------------------------------------------------------------------------------------------
static bool aligned16(const void* p) { return ((uintptr_t)p & 15u) == 0; }

static int probe_grid(const sj_table* t, int64_t n, int block) {
  const int64_t tiles = (n + (int64_t)block * KPT - 1) / ((int64_t)block * KPT);
  const int64_t cap = (int64_t)sm_count(t->device) * std::max(1, t->params.ctas_per_sm);
  return (int)std::max<int64_t>(1, std::min(tiles, cap));
}

template <typename K, bool WIDE, bool VEC, bool COUNT_ONLY>
static void launch_distinct(const sj_table* t, const sj_column& p, const int64_t* d_n, const GatherArgs& g,
                            cudaStream_t s) {
  const int block = kProbeThreads;
  const int grid = probe_grid(t, p.num_rows, block);
  // output reservation: per CTA tile for large probes (or when asked), per warp otherwise
  const int agg = t->params.aggregation;
  const bool cta = agg == SJ_AGG_CTA || (agg == SJ_AGG_AUTO && p.num_rows >= (1 << 20));
  KernelTimer timer(COUNT_ONLY ? "probe_distinct_count" : "probe_distinct", s);
  if (cta && !COUNT_ONLY)
    probe_distinct_kernel<K, WIDE, VEC, COUNT_ONLY, true><<<grid, block, 0, s>>>(
        table_dev(t), static_cast<const K*>(p.data), p.validity, p.validity_offset, p.num_rows, d_n, g);
  else
    probe_distinct_kernel<K, WIDE, VEC, COUNT_ONLY, false><<<grid, block, 0, s>>>(
        table_dev(t), static_cast<const K*>(p.data), p.validity, p.validity_offset, p.num_rows, d_n, g);
}

// d_n: optional device-resident row count (a partitioned probe's valid rows); p.num_rows bounds it.
template <bool COUNT_ONLY>
static void dispatch_distinct(const sj_table* t, const sj_column& p, const int64_t* d_n, const GatherArgs& g,
                              cudaStream_t s) {
  const bool wide = t->slot_kind == SJ_SLOT_WIDE128;
  const bool vec = aligned16(p.data);
#define SJ_D(K, W, V) launch_distinct<K, W, V, COUNT_ONLY>(t, p, d_n, g, s)
  if (t->key_type == SJ_INT32) {
    if (wide) { if (vec) SJ_D(int32_t, true, true); else SJ_D(int32_t, true, false); }
    else { if (vec) SJ_D(int32_t, false, true); else SJ_D(int32_t, false, false); }
  } else {
    if (wide) { if (vec) SJ_D(int64_t, true, true); else SJ_D(int64_t, true, false); }
    else { if (vec) SJ_D(int64_t, false, true); else SJ_D(int64_t, false, false); }
  }
#undef SJ_D
}

static sj_status check_probe(const sj_table* t, const sj_column& p) {
  SJ_TRY(validate_column(&p, "probe key", true));
  if (p.type != t->key_type) return set_error(SJ_ERR_INVALID, "probe key type differs from the build key type");
  if (p.num_rows > INT32_MAX) return set_error(SJ_ERR_INVALID, "probe side exceeds the int32 row-id range");
  return SJ_OK;
}

sj_status probe_count(const sj_table* t, const sj_column& p, const Allocator& alloc, cudaStream_t s,
                      int64_t* d_count) {
  SJ_TRY(check_probe(t, p));
  (void)alloc;
  SJ_CUDA_TRY(cudaMemsetAsync(d_count, 0, sizeof(int64_t), s));
  if (p.num_rows == 0) return SJ_OK;
  unsigned long long* dc = reinterpret_cast<unsigned long long*>(d_count);
  if (t->layout == SJ_LAYOUT_DISTINCT) {
    GatherArgs g{};
    g.d_count = dc;
    dispatch_distinct<true>(t, p, nullptr, g, s);
  } else {
    match_units(t, p, nullptr, nullptr, nullptr, dc, s);
  }
  SJ_CUDA_TRY(cudaGetLastError());
  return SJ_OK;
}

static sj_status fill_gather(const sj_table* t, const sj_column& p, const GatherSpec& gs, GatherArgs& g) {
  if (gs.n_probe_payload < 0 || gs.n_probe_payload > kMaxPayload || gs.n_build_payload < 0 ||
      gs.n_build_payload > kMaxPayload)
    return set_error(SJ_ERR_INVALID, "at most 8 payload columns per side");
  if (gs.capacity < 0) return set_error(SJ_ERR_INVALID, "capacity must be >= 0");
  if ((gs.n_probe_payload && (!gs.probe_payload || !gs.out_probe_payload)) ||
      (gs.n_build_payload && !gs.out_build_payload))
    return set_error(SJ_ERR_INVALID, "payload column arrays must not be NULL");
  const bool attached = gs.n_build_payload > 0 && gs.build_payload == nullptr;
  if (attached && gs.n_build_payload != t->n_attached)
    return set_error(SJ_ERR_INVALID, "build_payload is NULL (use the attached columns) but num_build_payload "
                                     "differs from the number of columns attached at build");
  g.n_pin = gs.n_probe_payload;
  g.n_bin = gs.n_build_payload;
  auto fill = [&](const sj_column& in, const sj_mut_column& out, int64_t rows, PayloadIn& pi, PayloadOut& po,
                  const char* side) -> sj_status {
    SJ_TRY(validate_column(&in, side, false));
    if (in.num_rows != rows)
      return set_error(SJ_ERR_INVALID, std::string(side) + " payload row count differs from its key column");
    if (out.type != in.type) return set_error(SJ_ERR_INVALID, std::string(side) + " output type differs");
    if (gs.capacity > 0 && !out.data) return set_error(SJ_ERR_INVALID, std::string(side) + " output data is NULL");
    if (in.validity && gs.capacity > 0 && !out.validity)
      return set_error(SJ_ERR_INVALID, std::string(side) + " payload has NULLs but its output has no validity");
    pi = column_payload(in.data, in.validity, in.validity_offset, type_width(in.type));
    po.data = out.data;
    po.valid = in.validity ? out.validity : nullptr;
    return SJ_OK;
  };
  for (int c = 0; c < g.n_pin; ++c)
    SJ_TRY(fill(gs.probe_payload[c], gs.out_probe_payload[c], p.num_rows, g.pin[c], g.pout[c], "probe"));
  if (attached) {
    for (int c = 0; c < g.n_bin; ++c) {
      const sj_mut_column& out = gs.out_build_payload[c];
      if (out.type != t->apay_type[c]) return set_error(SJ_ERR_INVALID, "attached build output type differs");
      if (gs.capacity > 0 && !out.data) return set_error(SJ_ERR_INVALID, "build output data is NULL");
      if (t->apay_valid[c] && gs.capacity > 0 && !out.validity)
        return set_error(SJ_ERR_INVALID, "attached build payload has NULLs but its output has no validity");
      g.bin[c] = PayloadIn{t->apay[c], nullptr, t->apay_valid[c], 0, type_width(t->apay_type[c]), t->apay_stride[c],
                           t->apay_vstride[c], 0};
      g.bout[c] = PayloadOut{out.data, t->apay_valid[c] ? out.validity : nullptr};
      if (t->arow) {
        g.rec_off[c] = (int16_t)(static_cast<const char*>(t->apay[c]) - static_cast<const char*>(t->arow));
        g.rec_voff[c] = t->apay_valid[c] ? (int16_t)(reinterpret_cast<const char*>(t->apay_valid[c]) -
                                                     static_cast<const char*>(t->arow))
                                         : (int16_t)-1;
      }
    }
    g.bin_by_pos = 1;
    if (t->arow && t->arow_stride <= 32) {
      g.rec = t->arow;
      g.rec_stride = t->arow_stride;
    }
  } else {
    for (int c = 0; c < g.n_bin; ++c)
      SJ_TRY(fill(gs.build_payload[c], gs.out_build_payload[c], t->build_rows, g.bin[c], g.bout[c], "build"));
  }
  g.brid_map = t->pos_rid;
  g.brid_stride = t->pos_stride;
  g.out_prid = gs.out_probe_rid;
  g.out_brid = gs.out_build_rid;
  g.capacity = gs.capacity;
  return SJ_OK;
}

static size_t align256(size_t b) { return (b + 255) & ~(size_t)255; }

// Partitioned probe of a DISTINCT table: radix-scatter the probe rows (key, row id, payloads) by
// the table's partition bits, then stream the partitioned arrays through the probe kernel, so
// each partition's probes hit its L2-resident table segment and attached payload rows.
// Probe-side radix bits: the coarsest prefix of the table's partition bits whose share of the
// table footprint (slots + position map + attached payloads) stays under 48 MB of L2 (or the
// table's probe_partition_mb). A coarse
// probe partition covers 2^(table bits - probe bits) contiguous table segments, and fewer
// partitions mean longer contiguous runs in the scatter (16M-row table, 768 MB: 12 MB shares made
// the probe 2 % faster and the scatter 15 % slower than 48 MB shares; 24 MB was in between).
static int probe_partition_bits(const sj_table* t) {
  size_t fp = t->slots_bytes + t->arow_bytes;
  const size_t share = (size_t)(t->params.probe_partition_mb > 0 ? t->params.probe_partition_mb : 48) << 20;
  int b = 1;
  while (b < t->pbits && (fp >> b) > share) ++b;
  return std::min(b, t->pbits);
}

// Tile-local partition (one pass, no histogram) + the probe of its runs, when the unit probe serves the
// output shape and the probe payloads are plain 4/8-byte columns without NULLs.
static bool partition_is_local(const sj_table* t, const GatherArgs& g) {
  bool local = probe_runs_ok(t, g) && g.n_pin <= 2;
  for (int c = 0; c < g.n_pin; ++c)
    local = local && !g.pin[c].valid && !g.pin[c].valid8 && (g.pin[c].width == 4 || g.pin[c].width == 8) &&
            g.pin[c].stride == g.pin[c].width;
  return local;
}

static sj_status probe_partitioned(const sj_table* t, const sj_column& p, GatherArgs g, const Allocator& alloc,
                                   cudaStream_t s) {
  const int64_t n = p.num_rows;
  const int pbits = probe_partition_bits(t);
  const int kw = t->key_type == SJ_INT32 ? 4 : 8;
  const bool local = partition_is_local(t, g);
  const int64_t n_tiles = (n + kPartTileRows - 1) / kPartTileRows;
  const size_t run_bytes = (size_t)n_tiles * ((size_t)1 << pbits) * sizeof(int32_t);
  size_t bytes = align256((size_t)n * kw) + align256((size_t)n * 4) + 256 +
                 (local ? 2 * align256(run_bytes) : partition_scratch_bytes(pbits, t->device));
  for (int c = 0; c < g.n_pin; ++c)
    bytes += align256((size_t)n * g.pin[c].width) + (g.pin[c].valid ? align256((size_t)n) : 0);
  Scratch sc;
  SJ_TRY(sc.get(alloc, bytes, s));
  // 256-byte boundaries whatever the allocator returns: the partitioned columns are written in 16-byte pieces
  char* cur = reinterpret_cast<char*>(align256(reinterpret_cast<size_t>(sc.ptr)));
  auto carve = [&](size_t b) {
    char* r = cur;
    cur += align256(b);
    return r;
  };
  PartSrc ps{};
  PartDst pd{};
  ps.keys = p.data;
  ps.kvalid = p.validity;
  ps.kvoff = p.validity_offset;
  ps.n = n;
  ps.n_pay = g.n_pin;
  pd.keys = carve((size_t)n * kw);
  pd.rid = reinterpret_cast<int32_t*>(carve((size_t)n * 4));
  for (int c = 0; c < g.n_pin; ++c) {
    ps.pay[c] = g.pin[c];
    pd.pay[c] = carve((size_t)n * g.pin[c].width);
    pd.valid8[c] = g.pin[c].valid ? reinterpret_cast<uint8_t*>(carve((size_t)n)) : nullptr;
  }
  if (local) {
    const TableDev range = table_dev(t);
    int32_t* run_off = reinterpret_cast<int32_t*>(carve(run_bytes));
    int32_t* run_cnt = reinterpret_cast<int32_t*>(carve(run_bytes));
    SJ_TRY(local_partition(ps, t->key_type, pbits, range.kmin, range.kmax, pd, LocalRuns{run_off, run_cnt}, t->device, s));
    g.prid_map = pd.rid;
    for (int c = 0; c < g.n_pin; ++c) g.pin[c] = column_payload(pd.pay[c], nullptr, 0, g.pin[c].width);
    const RunArgs ra{run_off, run_cnt, (uint32_t)n_tiles, 1u << pbits, 0, 0};
    probe_runs(t, pd.keys, n, ra, g, s);
    SJ_CUDA_TRY(cudaGetLastError());
    return SJ_OK;
  }
  void* pscratch = carve(partition_scratch_bytes(pbits, t->device));
  const int64_t *d_total, *d_offs;
  int G;
  SJ_TRY(radix_partition(ps, t->key_type, pbits, pd, pscratch, t->device, s, &d_total, &d_offs, &G));
  g.prid_map = pd.rid;
  for (int c = 0; c < g.n_pin; ++c)
    g.pin[c] = PayloadIn{pd.pay[c], nullptr, pd.valid8[c], 0, g.pin[c].width, g.pin[c].width, 1, 0};
  const sj_column pk{pd.keys, nullptr, 0, n, t->key_type, 0};
  if (!probe_direct(t, pk, d_total, g, s)) dispatch_distinct<false>(t, pk, d_total, g, s);
  SJ_CUDA_TRY(cudaGetLastError());
  return SJ_OK;
}

// How many of kSampleRows evenly spaced probe rows have a key in the build's range.
template <typename K>
__global__ void __launch_bounds__(256) sample_range_kernel(TableDev t, const K* __restrict__ keys, const uint32_t* kv,
                                                           int64_t kvoff, int64_t n, uint32_t* in_range_rows) {
  const int64_t i = (int64_t)(blockIdx.x * blockDim.x + threadIdx.x) * n / kSampleRows;
  const int in = __syncthreads_count(in_range(t, __ldg(keys + i)) && bit_valid(kv, kvoff, i));
  if (threadIdx.x == 0 && in) atomicAdd(in_range_rows, (uint32_t)in);
}

// Which probe rows have a match, as one bit per row (SEMI, ANTI, MARK), in partition order. Against the lookup in
// place (kind_units_kernel), us for SEMI of int64 keys, 70 % of the rows with a match and the others in the range:
//   slots      16M rows        64M rows      64M, half of them out of range
//   128 MB   223 / 328       732 / 1,022       535 / 775       (in place / in partition order)
//   256 MB   311 / 336     1,093 / 1,026       643 / 788
//   512 MB   374 / 370     1,349 / 1,061       737 / 804
//   1 GB                   1,484 / 1,115       805 / 839
// In place after the choice takes about 40 us more on 64M rows: the kernels of the other way return at once, and the
// blocks of its CTAs follow one another. So: slots of 256 MB or more, 32M rows or more that touch each sector about
// once or more, and a key in the build's range for 5/8 of the rows (1/2 from 512 MB on). The last only the device
// knows: a sample decides there. In place, too, when the scratch is refused, and in a capture, whose graph would go
// on to use memory that the caller's allocator has got back.
sj_status find_in_order(const sj_table* t, const sj_column& p, const Allocator& alloc, cudaStream_t s, Scratch& bits,
                        const uint32_t** words, RangeGate* gate) {
  SJ_TRY(check_probe(t, p));
  const int64_t n = p.num_rows;
  constexpr int64_t kLeast = (int64_t)256 << 20;
  const int64_t slots = (int64_t)t->slots_bytes, sectors = n * kBucketBytes;
  if (t->pbits == 0 || slots < kLeast || sectors < std::max(slots, 4 * kLeast)) return SJ_OK;
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(s, &capture) != cudaSuccess) {
    cudaGetLastError();
    return SJ_OK;
  }
  if (capture != cudaStreamCaptureStatusNone) return SJ_OK;
  int pbits = 1;
  const size_t share = (size_t)(t->params.probe_partition_mb > 0 ? t->params.probe_partition_mb : 48) << 20;
  while (pbits < t->pbits && (t->slots_bytes >> pbits) > share) ++pbits;
  const int kw = t->key_type == SJ_INT32 ? 4 : 8;
  const int64_t n_tiles = (n + kPartTileRows - 1) / kPartTileRows;
  const size_t run_bytes = (size_t)n_tiles * ((size_t)1 << pbits) * sizeof(int32_t);
  const size_t bit_bytes = 16 + (size_t)((n + 31) / 32) * sizeof(uint32_t);
  Scratch sc;
  if (bits.get(alloc, bit_bytes, s) != SJ_OK ||
      sc.get(alloc, align256((size_t)n * kw) + align256((size_t)n * 4) + 2 * align256(run_bytes) + 256, s) != SJ_OK) {
    clear_error();
    return SJ_OK;
  }
  uint32_t* count = bits.as<uint32_t>();
  SJ_CUDA_TRY(cudaMemsetAsync(count, 0, sizeof(uint32_t), s));
  uint32_t* set = count + 4;
  const TableDev d = table_dev(t);
  {
    KernelTimer timer("sample_range", s);
    if (t->key_type == SJ_INT32)
      sample_range_kernel<int32_t><<<kSampleRows / 256, 256, 0, s>>>(d, static_cast<const int32_t*>(p.data), p.validity,
                                                                     p.validity_offset, n, count);
    else
      sample_range_kernel<int64_t><<<kSampleRows / 256, 256, 0, s>>>(d, static_cast<const int64_t*>(p.data), p.validity,
                                                                     p.validity_offset, n, count);
  }
  char* cur = reinterpret_cast<char*>(align256(reinterpret_cast<size_t>(sc.ptr)));
  PartSrc ps{};
  PartDst pd{};
  ps.keys = p.data;
  ps.kvalid = p.validity;
  ps.kvoff = p.validity_offset;
  ps.n = n;
  pd.keys = cur;
  pd.rid = reinterpret_cast<int32_t*>(cur + align256((size_t)n * kw));
  int32_t* run_off = reinterpret_cast<int32_t*>(cur + align256((size_t)n * kw) + align256((size_t)n * 4));
  int32_t* run_cnt = run_off + align256(run_bytes) / sizeof(int32_t);
  *gate = RangeGate{count, slots < 2 * kLeast ? kSampleRows / 8 * 5 : kSampleRows / 2};
  SJ_TRY(local_partition(ps, t->key_type, pbits, d.kmin, d.kmax, pd, LocalRuns{run_off, run_cnt, set, *gate}, t->device, s));
  const RunArgs ra{run_off, run_cnt, (uint32_t)n_tiles, 1u << pbits, 0, 0};
  find_units(t, pd.keys, n, ra, pd.rid, set, *gate, s);
  SJ_CUDA_TRY(cudaGetLastError());
  *words = set;
  return SJ_OK;
}

sj_status probe_gather(const sj_table* t, const sj_column& p, const GatherSpec& gs, const Allocator& alloc,
                       cudaStream_t s, int64_t* d_count) {
  SJ_TRY(check_probe(t, p));
  GatherArgs g{};
  SJ_TRY(fill_gather(t, p, gs, g));
  g.d_count = reinterpret_cast<unsigned long long*>(d_count);
  SJ_CUDA_TRY(cudaMemsetAsync(d_count, 0, sizeof(int64_t), s));
  const size_t vbytes = (size_t)((gs.capacity + 31) / 32) * sizeof(uint32_t);
  for (int c = 0; c < g.n_pin; ++c)
    if (g.pout[c].valid && vbytes) SJ_CUDA_TRY(cudaMemsetAsync(g.pout[c].valid, 0, vbytes, s));
  for (int c = 0; c < g.n_bin; ++c)
    if (g.bout[c].valid && vbytes) SJ_CUDA_TRY(cudaMemsetAsync(g.bout[c].valid, 0, vbytes, s));
  if (p.num_rows == 0) return SJ_OK;

  if (t->layout == SJ_LAYOUT_DISTINCT) {
    // the unit probe sets the matched bits: wherever it serves the gather and, when partitioned, walks runs
    if (gs.matched && t->params.probe_kernel != SJ_PROBE_KERNEL_DIRECT_TMA && probe_runs_ok(t, g)) {
      const bool split = t->pbits > 0 && p.num_rows >= kMinPartitionedProbe;
      if (!split || partition_is_local(t, g)) {
        g.matched = gs.matched;
        *gs.matched_set = true;
      }
    }
    if (t->pbits > 0 && p.num_rows >= kMinPartitionedProbe) return probe_partitioned(t, p, g, alloc, s);
    if (!probe_direct(t, p, nullptr, g, s)) dispatch_distinct<false>(t, p, nullptr, g, s);
    SJ_CUDA_TRY(cudaGetLastError());
    return SJ_OK;
  }
  if (!g.out_prid && !g.out_brid && g.n_pin == 0 && g.n_bin == 0) {
    // nothing to write: the count alone. The expand numbers tiles in 32 bits, enough for outputs that are in
    // memory; without any, the matches up to `capacity` may be 2^40 and more.
    match_units(t, p, nullptr, nullptr, nullptr, g.d_count, s);
    SJ_CUDA_TRY(cudaGetLastError());
    return SJ_OK;
  }
  const int64_t n = p.num_rows;
  Scratch sc;
  const size_t b_row = ((size_t)n * 4 + 255) & ~(size_t)255;
  const size_t b_off = ((size_t)(n + 1) * 8 + 255) & ~(size_t)255;
  const size_t b_tmp = kScanBlocks * sizeof(int64_t);
  SJ_TRY(sc.get(alloc, 3 * b_row + b_off + b_tmp + 256, s));
  char* base = sc.as<char>();
  int2* m_ent = reinterpret_cast<int2*>(base);  // {probe row, group start}
  int32_t* m_cnt = reinterpret_cast<int32_t*>(base + 2 * b_row);
  int64_t* m_off = reinterpret_cast<int64_t*>(base + 3 * b_row);
  int64_t* tmp = reinterpret_cast<int64_t*>(base + 3 * b_row + b_off);
  unsigned long long* d_nent = reinterpret_cast<unsigned long long*>(base + 3 * b_row + b_off + b_tmp);
  SJ_CUDA_TRY(cudaMemsetAsync(d_nent, 0, sizeof(unsigned long long), s));
  match_units(t, p, m_ent, m_cnt, d_nent, g.d_count, s);
  {
    KernelTimer timer("scan", s);
    device_exclusive_scan<int32_t, int64_t>(m_cnt, m_off, d_nent, 0, tmp, s);
  }
  // every block resident at once: a warp's tile range is fixed, so a second wave would be a tail
  // the compile-time shape: records [row id | one 4- or 8-byte payload], nothing else gathered
  int rs = 0;
  if (g.rec && g.n_pin == 0 && g.n_bin == 1 && g.rec_voff[0] < 0 && !g.bout[0].valid &&
      (g.rec_stride == 8 || g.rec_stride == 16) && g.bin[0].width * 2 == g.rec_stride &&
      g.rec_off[0] * 2 == g.rec_stride)
    rs = g.rec_stride;
  auto kernel = rs == 8 ? expand_kernel<8> : rs == 16 ? expand_kernel<16> : expand_kernel<0>;
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kExpandThreads, 0);
  const int grid = sm_count(t->device) * std::max(1, per_sm);
  KernelTimer timer("expand", s);
  kernel<<<grid, kExpandThreads, 0, s>>>(m_ent, m_off, d_nent, t->grp_rid, g);
  SJ_CUDA_TRY(cudaGetLastError());
  return SJ_OK;
}

}  // namespace sj
