// INNER probe and gather of a DISTINCT table in units. A unit is one warp's rows: 32 * S consecutive ones,
// or a piece of partition p's run of a tile (tile-local partition). A CTA takes 8 consecutive units (of one partition),
// 32 * S rows of each at a time: the keys of all S row groups in flight, their home buckets, one walk for the
// rows that go on, the probe side's row ids and payload, one reservation for the CTA (its atomicAdd returns
// behind the first records' loads), records, stores. Row group j's matches go to consecutive positions, so
// each column is stored in contiguous runs. Positions stay in registers and no row is staged.
//
// What bounds it: a random 32-byte load costs an SM one L1 tag cycle (275 G/s on the whole GPU, any width,
// from 1024 threads per SM on), and a match needs two (bucket, record or payload); instructions, half of
// them at half rate, cost about as much. So the code per row is short (the rows that go on are walked once
// per 128 rows, one per lane, not once more with every row group), CTAs are small, many (6 per SM, 48 warps)
// and start in order: partition after partition is swept without a work counter, and one CTA's barriers and
// its reservation (same-address atomics return one per 0.67 ns on the whole GPU) are covered by the others.
// Shared memory is kept small too: what it takes from L1 limits the loads in flight (a 32 KB list per CTA
// made the lookups 60 % slower).
#include <algorithm>
#include <type_traits>

#include "sj_internal.h"
#include "sj_partition.cuh"
#include "sj_probe_units.h"
#include "sj_units.cuh"

namespace sj {

TableDev table_dev(const sj_table* t);

__device__ __forceinline__ uint64_t ld_col(const void* base, uint32_t i, int w) {
  return w == 8 ? (uint64_t)__ldcs(static_cast<const unsigned long long*>(base) + i)
                : (uint64_t)__ldcs(static_cast<const unsigned int*>(base) + i);
}
__device__ __forceinline__ uint64_t ld_at(const void* a, int w) {
  return w == 8 ? (uint64_t)__ldg(static_cast<const unsigned long long*>(a))
                : (uint64_t)__ldg(static_cast<const unsigned int*>(a));
}
__device__ __forceinline__ void st_col(void* base, uint32_t i, int w, uint64_t v) {
  if (w == 8) __stcs(static_cast<unsigned long long*>(base) + i, (unsigned long long)v);
  else __stcs(static_cast<unsigned int*>(base) + i, (unsigned int)v);
}

// SP, SB >= 0: a compile-time output shape: both row ids, SP probe payloads and SB build payloads out of
// row-store records, 8 bytes each. -1: the shape is read from `a`. -2: so too, and the rows' match bits are set
// (apart: with the bits in every shape the -1 shape spilled and 32M row-id-only rows took 500 us, not 437).
template <int SP, int SB>
struct Shape {
  static constexpr bool kFixed = SP >= 0, kMatched = SP == -2;
  __device__ __forceinline__ static int n_pin(const DirectArgs& a) { return kFixed ? SP : a.n_pin; }
  __device__ __forceinline__ static int pin_w(const DirectArgs& a, int c) { return kFixed ? 8 : a.pin_w[c]; }
  __device__ __forceinline__ static bool rec(const DirectArgs& a) { return kFixed ? SB > 0 : a.rec != nullptr; }
  __device__ __forceinline__ static int stride(const DirectArgs& a) { return kFixed ? (SB == 1 ? 16 : 32) : a.rec_stride; }
  __device__ __forceinline__ static int n_bin(const DirectArgs& a) { return kFixed ? SB : a.n_bin; }
  __device__ __forceinline__ static bool prid(const DirectArgs& a) { return kFixed || a.out_prid; }
  __device__ __forceinline__ static bool brid(const DirectArgs& a) { return kFixed || a.out_brid; }
};

// Row id and first payload of probe row `row` (index into the probe arrays).
template <typename Sh>
__device__ __forceinline__ void load_probe_side(const DirectArgs& a, uint32_t row, bool live, int32_t& prid, uint64_t& v) {
  prid = a.prid_map && live ? __ldcs(a.prid_map + row) : (int32_t)row;
  v = Sh::n_pin(a) > 0 && live ? ld_col(a.pin[0], row, Sh::pin_w(a, 0)) : 0;
}

// Writes a match: probe row `row` (index into the probe arrays) and table position `pos` to output position
// p if live, with the row id prid and the first probe payload v; `ready()`, called by the whole warp between
// the first loads and the first store, gives p and may clear live.
template <typename Sh, typename Ready>
__device__ __forceinline__ void emit_match(const DirectArgs& a, uint32_t row, int32_t prid, uint64_t v, uint32_t pos,
                                           bool live, Ready&& ready) {
  uint32_t w[8];
  int32_t brid = (int32_t)pos;
  if (Sh::rec(a)) {
    if (live) {
      const char* rp = static_cast<const char*>(a.rec) + (size_t)pos * Sh::stride(a);
      if (Sh::stride(a) == 32) {
        asm("ld.global.nc.v8.u32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
            : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]), "=r"(w[4]), "=r"(w[5]), "=r"(w[6]), "=r"(w[7])
            : "l"(rp));
      } else if (Sh::stride(a) == 16) {
        const uint4 x = __ldg(reinterpret_cast<const uint4*>(rp));
        w[0] = x.x; w[1] = x.y; w[2] = x.z; w[3] = x.w;
      } else {
        const uint2 x = __ldg(reinterpret_cast<const uint2*>(rp));
        w[0] = x.x; w[1] = x.y;
      }
      brid = (int32_t)w[0];
    }
  } else if (a.brid_map && live) {
    brid = __ldg(reinterpret_cast<const int32_t*>(reinterpret_cast<const char*>(a.brid_map) + (size_t)pos * a.brid_stride));
  }
  uint32_t p;
  ready(p, live);
  if (!live) return;
  if (Sh::prid(a)) __stcs(a.out_prid + p, prid);
  if (Sh::n_pin(a) > 0) st_col(a.pout[0], p, Sh::pin_w(a, 0), v);
  if (Sh::n_pin(a) > 1) st_col(a.pout[1], p, Sh::pin_w(a, 1), ld_col(a.pin[1], row, Sh::pin_w(a, 1)));
  if (Sh::brid(a)) __stcs(a.out_brid + p, brid);
  if (Sh::rec(a)) {
    if (Sh::stride(a) == 8) {  // one 4-byte field
      __stcs(static_cast<unsigned int*>(a.bout[0]) + p, w[1]);
    } else {
#pragma unroll
      for (int c = 0; c < kDirectMaxBuildPayload; ++c)
        if (c < Sh::n_bin(a))
          __stcs(static_cast<unsigned long long*>(a.bout[c]) + p, ((unsigned long long)w[3 + 2 * c] << 32) | w[2 + 2 * c]);
    }
    return;
  }
  for (int c = 0; c < Sh::n_bin(a); ++c)
    st_col(a.bout[c], p, a.bin_w[c],
           ld_at(static_cast<const char*>(a.bin[c]) + (int64_t)(a.bin_by_pos ? (int32_t)pos : brid) * a.bin_stride[c], a.bin_w[c]));
}

constexpr int kUnitCtasPerSm = 6;  // 40 registers

// Sets the bits of the lanes' rows that `found` names: a whole word when the rows are in their own order (lane 0's is
// the word's first), else one bit for each partitioned row's row id. (Collected per tile in shared memory and flushed in
// lines, the bits of 64M rows took 605-770 us with the lookup against 570: what shared memory takes from L1 and from the
// warps per SM costs more than the atomics.)
template <bool RUNS>
__device__ __forceinline__ void mark_found(uint32_t* words, const int32_t* prid_map, uint32_t row, bool any, unsigned found) {
  const int lane = threadIdx.x & 31;
  if constexpr (RUNS) {
    if (found >> lane & 1u) {
      const uint32_t r = (uint32_t)__ldg(prid_map + row);
      atomicOr(words + (r >> 5), 1u << (r & 31));
    }
  } else {
    if (lane == 0 && any) words[row >> 5] = found;
  }
}

// The lookup alone, in partition order: bit i of `words` = probe row i has a match. A CTA takes kFindBlocks blocks of
// units, one after the other in the order of the partitions: a launch whose gate is closed is that much cheaper (64K
// CTAs that return at once take 37 us). With a grid-stride loop instead the sweep lost its order, 1,457 us for 1,164,
// and with four blocks 64M rows into 64M keys took 1,214 us instead of 1,157.
constexpr int kFindBlocks = 2;

template <typename K, bool WIDE, bool JOIN>
__global__ void __launch_bounds__(kUnitThreads, 8) find_units_kernel(TableDev t, const K* __restrict__ keys, uint32_t n,
                                                                     RunArgs ra, const int32_t* __restrict__ prid_map,
                                                                     uint32_t* words, RangeGate gate) {
  constexpr int S = 4;
  __shared__ WaitRows<S> s_wait[kUnitWarps];
  if (!gate_open(gate)) return;
  const int lane = threadIdx.x & 31;
  const uint32_t end = min(ra.P * run_ctas(ra), (blockIdx.x + 1) * kFindBlocks);
  for (uint32_t cta = blockIdx.x * kFindBlocks; cta < end; ++cta) {
    const auto u = rows_of_unit<true, S, JOIN>(ra, cta_units<true>(ra, cta), n);
    for (uint32_t v0 = 0; v0 < u.rows; v0 += 32 * S) {
      K k[S];
      uint32_t row[S];
#pragma unroll
      for (int j = 0; j < S; ++j) {
        const uint32_t v = v0 + 32 * j + lane;
        row[j] = u.row(v);
        k[j] = v < u.rows ? __ldcs(keys + row[j]) : (K)0;
      }
      uint32_t pos[S];
      unit_lookup<K, WIDE, true, S>(t, k, nullptr, 0, 0, v0, u.rows, s_wait[threadIdx.x >> 5], pos);
#pragma unroll
      for (int j = 0; j < S; ++j)
        mark_found<true>(words, prid_map, row[j], v0 + 32 * j < u.rows, __ballot_sync(kFullMask, pos[j] != kNoPos));
    }
  }
}

template <typename K, bool WIDE, bool RUNS, int S, int SP, int SB, bool JOIN = false>
__global__ void __launch_bounds__(kUnitThreads, kUnitCtasPerSm) probe_units_kernel(TableDev t, const K* __restrict__ keys,
                                                                      const uint32_t* __restrict__ kv, int64_t kvoff,
                                                                      uint32_t n, const int64_t* d_n, RunArgs ra,
                                                                      DirectArgs a) {
  using Sh = Shape<SP, SB>;
  if (!RUNS && d_n) n = min(n, (uint32_t)*d_n);
  __shared__ WaitRows<S> s_wait[kUnitWarps];
  __shared__ uint32_t s_cnt[kUnitWarps];
  __shared__ uint32_t s_base;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned below = (1u << lane) - 1u;
  WaitRows<S>& wait = s_wait[warp];
  const uint32_t cap = (uint32_t)(a.capacity < (int64_t)0x7fffffff ? a.capacity : (int64_t)0x7fffffff);
  const auto u = rows_of_unit<RUNS, S, JOIN>(ra, cta_units<RUNS>(ra, blockIdx.x), n);
  uint32_t first = 0;
  if constexpr (!JOIN) first = u.first;
  for (uint32_t v0 = 0; __syncthreads_or(v0 < u.rows); v0 += 32 * S) {
    K k[S];
    uint32_t row[S];
#pragma unroll
    for (int j = 0; j < S; ++j) {
      const uint32_t v = v0 + 32 * j + lane;
      row[j] = u.row(v);
      k[j] = v < u.rows ? __ldcs(keys + row[j]) : (K)0;
    }
    uint32_t pos[S];
    unit_lookup<K, WIDE, RUNS, S>(t, k, kv, kvoff, first, v0, u.rows, wait, pos);
    uint32_t cnt = 0;
#pragma unroll
    for (int j = 0; j < S; ++j) {
      const unsigned bal = __ballot_sync(kFullMask, pos[j] != kNoPos);
      cnt += __popc(bal);
      if constexpr (Sh::kMatched) mark_found<RUNS>(a.matched, a.prid_map, row[j], v0 + 32 * j < u.rows, bal);
    }
    if (lane == 0) s_cnt[warp] = cnt;
    int32_t prid[S];
    uint64_t pv[S];
#pragma unroll
    for (int j = 0; j < S; ++j) load_probe_side<Sh>(a, row[j], pos[j] != kNoPos, prid[j], pv[j]);
    __syncthreads();
    const uint32_t c = lane < kUnitWarps ? s_cnt[lane] : 0;
    const uint32_t incl = warp_inclusive_sum(c);
    uint32_t run = __shfl_sync(kFullMask, incl - c, warp);
    if (warp == 0 && lane == kUnitWarps - 1) s_base = incl ? (uint32_t)atomicAdd(a.d_count, (unsigned long long)incl) : 0;
#pragma unroll
    for (int j = 0; j < S; ++j) {
      const bool hit = pos[j] != kNoPos;
      const unsigned bal = __ballot_sync(kFullMask, hit);
      emit_match<Sh>(a, row[j], prid[j], pv[j], pos[j], hit, [&](uint32_t& p, bool& live) {
        if (j == 0) {  // the reservation is back
          __syncthreads();
          run += s_base;
        }
        p = run + __popc(bal & below);
        run += __popc(bal);
        live = live && p < cap;
      });
    }
  }
}

// GROUPED tables: each probe row's group. COMPACT: appends (row, group start, group size) of the rows with
// matches; always: adds the matches up. One reservation per CTA (1024 rows): with one per warp of 128 rows the
// entry counter alone took 176 us of a 32M-row probe (one same-address atomic per 0.67 ns).
template <typename K, bool WIDE, bool COMPACT>
__global__ void __launch_bounds__(kUnitThreads, 6) match_units_kernel(TableDev t, const K* __restrict__ keys,
                                                                      const uint32_t* __restrict__ kv, int64_t kvoff,
                                                                      uint32_t n, int2* m_ent, int32_t* m_cnt,
                                                                      unsigned long long* d_nent,
                                                                      unsigned long long* d_total) {
  constexpr int S = 4;
  __shared__ WaitRows<S> s_wait[kUnitWarps];
  __shared__ uint32_t s_ent[kUnitWarps];
  __shared__ unsigned long long s_sum[kUnitWarps], s_base;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned below = (1u << lane) - 1u;
  const auto [first, rows] = unit_rows<false, S>(RunArgs{}, cta_units<false>(RunArgs{}, blockIdx.x), n);
  K k[S];
#pragma unroll
  for (int j = 0; j < S; ++j) {
    const uint32_t v = 32 * j + lane;
    k[j] = v < rows ? __ldcs(keys + first + v) : (K)0;
  }
  uint32_t slot[S];
  unit_lookup<K, WIDE, false, S, true>(t, k, kv, kvoff, first, 0, rows, s_wait[warp], slot);
  int32_t start[S], cnt[S];
  unsigned long long sum = 0;
  uint32_t ents = 0;
#pragma unroll
  for (int j = 0; j < S; ++j) {
    const uint32_t v = 32 * j + lane;
    if (t.null_group >= 0 && v < rows && !bit_valid(kv, kvoff, first + v)) slot[j] = (uint32_t)t.null_group;
    start[j] = cnt[j] = 0;
    if (slot[j] != kNoPos) {
      start[j] = __ldg(t.grp_off + slot[j]);
      cnt[j] = __ldg(t.grp_off + slot[j] + 1) - start[j];
    }
  }
#pragma unroll
  for (int j = 0; j < S; ++j) {
    sum += (unsigned long long)cnt[j];
    ents += __popc(__ballot_sync(kFullMask, cnt[j] > 0));
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) sum += __shfl_down_sync(kFullMask, sum, d);
  if (lane == 0) {
    s_ent[warp] = ents;
    s_sum[warp] = sum;
  }
  __syncthreads();
  const uint32_t c = lane < kUnitWarps ? s_ent[lane] : 0;
  const uint32_t incl = warp_inclusive_sum(c);
  if (warp == 0) {
    unsigned long long all = lane < kUnitWarps ? s_sum[lane] : 0;
#pragma unroll
    for (int d = kUnitWarps / 2; d > 0; d >>= 1) all += __shfl_down_sync(kFullMask, all, d);
    if (lane == 0 && all) atomicAdd(d_total, all);
    if (COMPACT && lane == kUnitWarps - 1) s_base = incl ? atomicAdd(d_nent, (unsigned long long)incl) : 0ull;
  }
  if constexpr (COMPACT) {
    uint32_t run = __shfl_sync(kFullMask, incl - c, warp);
    __syncthreads();
    run += (uint32_t)s_base;
#pragma unroll
    for (int j = 0; j < S; ++j) {
      const unsigned bal = __ballot_sync(kFullMask, cnt[j] > 0);
      const uint32_t e = run + __popc(bal & below);
      run += __popc(bal);
      if (cnt[j] <= 0) continue;
      m_ent[e] = make_int2((int32_t)(first + 32 * j + lane), start[j]);
      m_cnt[e] = cnt[j];
    }
  }
}

// Records are held in registers when they are [row id | one 4-byte field] or [row id | - | 8-byte
// fields]; the fields of other records are gathered from the row store one by one.
static DirectArgs plain_records(DirectArgs a) {
  if (a.rec && !a.rec_std && !(a.n_bin == 1 && a.rec_stride == 8 && a.rec_off[0] == 4)) {
    a.brid_map = static_cast<const int32_t*>(a.rec);
    a.brid_stride = a.rec_stride;
    a.bin_by_pos = 1;
    for (int c = 0; c < a.n_bin; ++c) {
      a.bin[c] = static_cast<const char*>(a.rec) + a.rec_off[c];
      a.bin_stride[c] = a.rec_stride;
    }
    a.rec = nullptr;
  }
  return a;
}

// Units of about 128 rows: a run holds kPartTileRows / P rows. Longer ones are cut into pieces: with whole runs of 1024
// rows a warp's chain was eight times as long and the few warps of a 1M-row probe took 100 us instead of 63. Short ones,
// of `joined` partitions or more, are joined with those of neighbouring tiles: they lie side by side in the run tables,
// and a row is found by a search of log2(tiles) shuffles. Unjoined, a unit of 256 partitions has 16 rows for its 128
// places: 33.5M int64 rows into 4M keys, one payload, 1,271 us and 866 joined; into 100M keys, 128 partitions, 64M rows
// with three payloads 2,615 and 2,186; their bits (SEMI, 256 partitions) 1,298 and 643. With 64 partitions a unit is
// half full: bits 658 and 603, but 64M rows with three payloads 1,727 and 1,799.
static RunArgs run_units(RunArgs ra, uint32_t joined) {
  ra.log2_pieces = ra.log2_join = 0;
  while (((uint64_t)ra.P * 128 << ra.log2_pieces) < kPartTileRows) ++ra.log2_pieces;
  if (ra.P < joined) return ra;
  while (ra.log2_join < 5 && (uint64_t)kPartTileRows << ra.log2_join < (uint64_t)ra.P * 128) ++ra.log2_join;
  return ra;
}

static int unit_grid(int64_t n, int unit, const RunArgs* ra) {
  auto ctas = [](int64_t units) { return (units + kUnitWarps - 1) / kUnitWarps; };
  if (!ra) return (int)ctas((n + unit - 1) / unit);
  const int64_t tiles = ra->n_tiles;
  return (int)(ra->P * ctas(ra->log2_join ? (tiles + (1 << ra->log2_join) - 1) >> ra->log2_join : tiles << ra->log2_pieces));
}

void probe_units(const sj_table* t, const void* keys, const uint32_t* kv, int64_t kvoff, int64_t n, const int64_t* d_n,
                 const RunArgs* runs, const DirectArgs& a_in, cudaStream_t s) {
  if (n == 0) return;
  const DirectArgs a = plain_records(a_in);
  const RunArgs ra = runs ? run_units(*runs, 128) : RunArgs{};
  const bool few = !runs && n <= kFewRows;
  const int grid = unit_grid(n, few ? 32 : 128, runs ? &ra : nullptr);
  const TableDev d = table_dev(t);
  KernelTimer timer("probe_units", s);
  using std::integral_constant;
  auto shape = [&](auto k, auto w, auto sp, auto sb) {
    using K = decltype(k);
    constexpr bool W = decltype(w)::value;
    constexpr int SP = decltype(sp)::value, SB = decltype(sb)::value;
    // joined runs, of very large tables, in the general shapes and the widest: a first call loads every variant
    constexpr int JP = SP < 0 || SP == 1 ? SP : -1, JB = SP < 0 || SP == 1 ? SB : -1;
    auto kernel = runs && ra.log2_join ? probe_units_kernel<K, W, true, 4, JP, JB, true>
                  : runs ? probe_units_kernel<K, W, true, 4, SP, SB>
                  : few ? probe_units_kernel<K, W, false, 1, SP, SB> : probe_units_kernel<K, W, false, 4, SP, SB>;
    kernel<<<grid, kUnitThreads, 0, s>>>(d, static_cast<const K*>(keys), kv, kvoff, (uint32_t)n, d_n, ra, a);
  };
  auto go = [&](auto k, auto w) {
    const bool ids = a.out_prid && a.out_brid, rec = ids && a.rec && a.rec_stride != 8;
    if (a.matched) shape(k, w, integral_constant<int, -2>{}, integral_constant<int, -2>{});
    else if (rec && a.n_pin == 1 && a.pin_w[0] == 8 && a.n_bin == 2) shape(k, w, integral_constant<int, 1>{}, integral_constant<int, 2>{});
    else if (rec && a.n_pin == 0 && a.n_bin == 1) shape(k, w, integral_constant<int, 0>{}, integral_constant<int, 1>{});
    else if (ids && a.n_pin == 0 && a.n_bin == 0) shape(k, w, integral_constant<int, 0>{}, integral_constant<int, 0>{});
    else shape(k, w, integral_constant<int, -1>{}, integral_constant<int, -1>{});
  };
  const bool wide = t->slot_kind == SJ_SLOT_WIDE128;
  if (t->key_type == SJ_INT32) {
    if (wide) go(int32_t{}, std::true_type{});
    else go(int32_t{}, std::false_type{});
  } else {
    if (wide) go(int64_t{}, std::true_type{});
    else go(int64_t{}, std::false_type{});
  }
}

void find_units(const sj_table* t, const void* keys, int64_t n, const RunArgs& runs, const int32_t* prid_map,
                uint32_t* words, const RangeGate& gate, cudaStream_t s) {
  if (n == 0) return;
  const RunArgs ra = run_units(runs, 64);
  const int grid = (unit_grid(n, 128, &ra) + kFindBlocks - 1) / kFindBlocks;
  const TableDev d = table_dev(t);
  KernelTimer timer("find_units", s);
  auto go = [&](auto k, auto w) {
    using K = decltype(k);
    constexpr bool W = decltype(w)::value;
    auto kernel = ra.log2_join ? find_units_kernel<K, W, true> : find_units_kernel<K, W, false>;
    kernel<<<grid, kUnitThreads, 0, s>>>(d, static_cast<const K*>(keys), (uint32_t)n, ra, prid_map, words, gate);
  };
  const bool wide = t->slot_kind == SJ_SLOT_WIDE128;
  if (t->key_type == SJ_INT32) {
    if (wide) go(int32_t{}, std::true_type{});
    else go(int32_t{}, std::false_type{});
  } else {
    if (wide) go(int64_t{}, std::true_type{});
    else go(int64_t{}, std::false_type{});
  }
}

void match_units(const sj_table* t, const sj_column& p, int2* m_ent, int32_t* m_cnt, unsigned long long* d_nent,
                 unsigned long long* d_total, cudaStream_t s) {
  if (p.num_rows == 0) return;
  const bool compact = m_ent != nullptr;
  const int grid = unit_grid(p.num_rows, 128, nullptr);
  const TableDev d = table_dev(t);
  KernelTimer timer(compact ? "grouped_match" : "grouped_count", s);
  auto go = [&](auto k, auto w) {
    using K = decltype(k);
    constexpr bool W = decltype(w)::value;
    auto kernel = compact ? match_units_kernel<K, W, true> : match_units_kernel<K, W, false>;
    kernel<<<grid, kUnitThreads, 0, s>>>(d, static_cast<const K*>(p.data), p.validity, p.validity_offset,
                                         (uint32_t)p.num_rows, m_ent, m_cnt, d_nent, d_total);
  };
  const bool wide = t->slot_kind == SJ_SLOT_WIDE128;
  if (t->key_type == SJ_INT32) {
    if (wide) go(int32_t{}, std::true_type{});
    else go(int32_t{}, std::false_type{});
  } else {
    if (wide) go(int64_t{}, std::true_type{});
    else go(int64_t{}, std::false_type{});
  }
}

}  // namespace sj
