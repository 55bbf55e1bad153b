// Units: the rows that a warp looks up together, and their lookup. A unit is 32 * S consecutive probe rows, or a
// piece of a partition's run of a tile, or short runs of several tiles (tile-local partition); a CTA takes kUnitWarps consecutive ones. Shared by
// the INNER probe, the lookups of GROUPED tables (sj_probe_units.cu) and the other join types (sj_probe_kinds.cu).
#pragma once

#include "sj_partition.cuh"
#include "sj_probe_core.cuh"
#include "sj_probe_direct.h"

namespace sj {

constexpr int kUnitThreads = 256;
constexpr int kUnitWarps = kUnitThreads / 32;

constexpr uint32_t kNoPos = 0xffffffffu;

// INNER probes of at most this many rows take units of 32 rows: a row has a thread of its own and the chain of
// dependent loads is all there is. Units of 32 against units of 128 rows, keys and payloads of 4 bytes: 10K rows
// 4.0 / 6.9 us, 200K 5.4 / 7.6, 400K 8.4 / 8.5, 600K 11.8 / 10.6, 2M 30.2 / 28.6 (two warps of 64 rows with a
// reservation each, before: 6.5, 8.5, 12.8, 17.7, 50.5); of 8 bytes: 200K 5.5 / 7.9, 400K 8.5 / 9.1, 600K 12.0 / 11.3;
// 128-bit slots: 200K 5.9 / 8.5, 400K 9.4 / 9.8, 600K 14.0 / 12.3.
constexpr int64_t kFewRows = 400000;

constexpr uint32_t kSampleRows = 1 << 15;

__device__ __forceinline__ bool gate_open(const RangeGate& g) { return g.rows == nullptr || *g.rows >= g.need; }

struct Units {
  uint32_t part, first;  // RUNS: the CTA's partition; its first unit (piece of a run)
};

__device__ __forceinline__ uint32_t run_ctas(const RunArgs& ra) {  // of a partition
  const uint32_t units = ra.log2_join ? (ra.n_tiles + (1u << ra.log2_join) - 1u) >> ra.log2_join : ra.n_tiles << ra.log2_pieces;
  return (units + kUnitWarps - 1) / kUnitWarps;
}

template <bool RUNS>
__device__ __forceinline__ Units cta_units(const RunArgs& ra, uint32_t cta) {
  Units u{0, cta * kUnitWarps};
  if constexpr (RUNS) {
    const uint32_t ctas = run_ctas(ra);
    u.part = cta / ctas;
    u.first = (cta - u.part * ctas) * kUnitWarps;
  }
  return u;
}

// The warp's unit: its rows, numbered from 0, and where they are in the probe arrays.
struct UnitRows {
  uint32_t first, rows;
  __device__ __forceinline__ uint32_t row(uint32_t v) const { return first + v; }
};

// Runs of up to 32 consecutive tiles, lane l's from the unit's row `before` on, at before + shift of the arrays.
struct JoinedRows {
  uint32_t rows, before, shift, log2_join;
  // Called by the whole warp; v >= rows gives no row.
  __device__ __forceinline__ uint32_t row(uint32_t v) const {
    uint32_t tile = 0;  // the last one whose rows start at or before v
    for (uint32_t step = 1u << log2_join >> 1; step; step >>= 1)
      if (__shfl_sync(kFullMask, before, tile + step) <= v) tile += step;
    return v + __shfl_sync(kFullMask, shift, tile);
  }
};

template <bool RUNS, int S>
__device__ __forceinline__ UnitRows unit_rows(const RunArgs& ra, const Units& u, uint32_t n) {
  const uint32_t unit = u.first + (threadIdx.x >> 5);
  if constexpr (RUNS) {
    const uint32_t tile = unit >> ra.log2_pieces, piece = unit & ((1u << ra.log2_pieces) - 1u);
    if (tile >= ra.n_tiles) return {0, 0};
    const size_t at = (size_t)u.part * ra.n_tiles + tile;
    const uint32_t cnt = (uint32_t)__ldg(ra.run_cnt + at), lo = cnt * piece >> ra.log2_pieces;
    return {(uint32_t)__ldg(ra.run_off + at) + lo, (cnt * (piece + 1) >> ra.log2_pieces) - lo};
  } else {
    const uint32_t first = unit * (32 * S);
    return {first, first < n ? min(32u * S, n - first) : 0};
  }
}

__device__ __forceinline__ JoinedRows joined_rows(const RunArgs& ra, const Units& u) {
  const int lane = threadIdx.x & 31;
  const uint32_t tile = ((u.first + (threadIdx.x >> 5)) << ra.log2_join) + lane;
  const bool mine = (uint32_t)lane >> ra.log2_join == 0 && tile < ra.n_tiles;
  const size_t at = (size_t)u.part * ra.n_tiles + tile;
  const uint32_t cnt = mine ? (uint32_t)__ldg(ra.run_cnt + at) : 0;
  const uint32_t incl = warp_inclusive_sum(cnt);
  return {__shfl_sync(kFullMask, incl, 31), incl - cnt, (mine ? (uint32_t)__ldg(ra.run_off + at) : 0u) - (incl - cnt), ra.log2_join};
}

template <bool RUNS, int S, bool JOIN>
__device__ __forceinline__ auto rows_of_unit(const RunArgs& ra, const Units& u, uint32_t n) {
  if constexpr (JOIN) return joined_rows(ra, u);
  else return unit_rows<RUNS, S>(ra, u, n);
}

// A warp's rows that go on past their home bucket.
template <int S>
struct WaitRows {
  SectorKey key[32 * S];
  uint32_t bucket[32 * S];  // then the row's position
};

// Table positions (SLOT: slots) of rows first + v0 + 32 j + lane (keys k[j]) of the warp's unit, kNoPos where
// there is none. RUNS: the partition has dropped NULL keys and those outside the build's key range.
template <typename K, bool WIDE, bool RUNS, int S, bool SLOT = false>
__device__ __forceinline__ void unit_lookup(const TableDev& t, const K (&k)[S], const uint32_t* __restrict__ kv, int64_t kvoff,
                                            uint32_t first, uint32_t v0, uint32_t rows, WaitRows<S>& wait, uint32_t (&pos)[S]) {
  using Ops = SectorOps<WIDE>;
  const int lane = threadIdx.x & 31;
  const unsigned below = (1u << lane) - 1u;
  const uint32_t rid_mask = (1u << t.rbits) - 1u;
  uint32_t n_wait = 0;
  uint32_t waits = 0;  // byte j: 1 + place in the list of the lane's row j, or 0
#pragma unroll
  for (int j = 0; j < S; ++j) {
    const uint32_t v = v0 + 32 * j + lane;
    SectorKey key;
    uint32_t b = home_bucket(t, key_u64<K>(k[j])), q = 0;
    pos[j] = kNoPos;
    bool cont = false;
    const bool in = sector_key<K, WIDE>(t, k[j], key);
    if (v < rows && (RUNS || (in && bit_valid(kv, kvoff, first + v)))) {
      const Sector s = load_sector(t.slots, b);
      uint32_t p;
      if (SLOT ? Ops::find_slot(s, key, rid_mask, q) : Ops::find(s, key, rid_mask, p, q)) pos[j] = SLOT ? b * Ops::kSlots + q : p;
      else cont = t.segmask != 0 && !Ops::open(s);
    }
    const unsigned bal = __ballot_sync(kFullMask, cont);
    if (bal) {
      if (cont) {
        const uint32_t e = n_wait + __popc(bal & below);
        wait.key[e] = key;
        wait.bucket[e] = next_bucket(b, t.segmask);
        waits |= (e + 1) << (8 * j);
      }
      n_wait += __popc(bal);
    }
  }
  if (n_wait) {
    __syncwarp();
    for (uint32_t e0 = 0; e0 < n_wait; e0 += 32) {
      const uint32_t e = e0 + lane;
      bool act = e < n_wait;
      SectorKey key{};
      uint32_t b = 0, res = kNoPos;
      if (act) {
        key = wait.key[e];
        b = wait.bucket[e];
      }
      for (uint32_t step = 0; step < t.segmask && __any_sync(kFullMask, act); ++step) {
        if (act) {
          const Sector s = load_sector(t.slots, b);
          uint32_t q = 0, p;
          const bool f = SLOT ? Ops::find_slot(s, key, rid_mask, q) : Ops::find(s, key, rid_mask, p, q);
          if (f) res = SLOT ? b * Ops::kSlots + q : p;
          act = !f && !Ops::open(s);
          b = next_bucket(b, t.segmask);
        }
      }
      if (e < n_wait) wait.bucket[e] = res;
    }
    __syncwarp();
#pragma unroll
    for (int j = 0; j < S; ++j)
      if (waits >> (8 * j) & 0xffu) pos[j] = wait.bucket[(waits >> (8 * j) & 0xffu) - 1];
  }
}

}  // namespace sj
