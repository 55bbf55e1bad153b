// LEFT, SEMI, ANTI, MARK and FULL joins on a built table: the other join types of the operator's
// BUILD_PROBE path (src/op/sirius_physical_hash_join.cpp:1640-1700 — filtered_join::semi_join /
// anti_join, hash_join::left_join / full_join, distinct_hash_join::left_join — and the MARK result of
// resolve_mark_join_result, :1461-1525).
//
//   SEMI / ANTI  one pass over the probe rows: a lookup in place, and the selected rows compacted with their probe
//                payloads (kind_units_kernel; a NULL key finds nothing unless NULLs compare equal and the build
//                has NULL keys). No scratch. Where slots of 256 MB and more meet enough rows, the lookup runs in
//                partition order instead (find_in_order, sj_probe.cu) and leaves one bit per probe row, and the
//                rows are selected by them; that takes scratch, and without it the one pass remains.
//   MARK         the same lookups: mark byte and validity bit of every probe row. Unmatched rows are
//                NULL when their key is NULL, or all of them when the build has a NULL key.
//   LEFT         the INNER probe + gather (probe_gather, any table layout), then the unmatched probe
//                rows appended after the INNER rows on the same counter with build row id
//                SJ_NO_ROW: the rows whose bit is clear in a mask that the unit probe sets as it looks
//                the rows up, or that is set from the INNER rows' probe row ids (or, when those are not
//                written or overflowed the capacity, the ANTI lookup); validity of the NULL-padded build
//                payloads is set by range.
//   FULL         LEFT, then the unmatched build rows: the build rows whose bit is clear in a mask
//                set from the INNER rows' build row ids (NULL-key rows included). When no build row
//                ids are written or the INNER rows overflowed the capacity: a pass that flags every
//                table slot (group) some probe row matched, then a DISTINCT table walks its slots, a
//                GROUPED table its group-ordered members (group of member i = the last group starting
//                at or before i), and the NULL-key build rows come from the table's NULL-row list.
#include <algorithm>

#include "sj_device.cuh"
#include "sj_internal.h"
#include "sj_probe_units.h"
#include "sj_units.cuh"

namespace sj {

TableDev table_dev(const sj_table* t);

constexpr int kKindThreads = 256;
constexpr int kKindStage = 256;  // staged row ids per warp (SEMI / ANTI rows, FULL's unmatched build rows)
constexpr int32_t kNoRow = (int32_t)0x80000000;

enum KindMode { kSemi = 0, kAnti = 1, kMark = 2, kFlags = 3 };

struct KindArgs {
  int32_t* out_prid;
  int32_t* out_brid;  // LEFT/FULL append: written with kNoRow
  int32_t n_pin;
  PayloadIn pin[kMaxPayload];
  PayloadOut pout[kMaxPayload];
  int64_t capacity;
  unsigned long long* d_count;
  uint8_t* mark;
  uint32_t* mark_valid;
  int32_t build_has_null;
  uint8_t* flags;  // kFlags: one byte per slot (+ the NULL group)
  const unsigned long long* inner_rows;  // kAnti, kFlags, select_rows: INNER rows that the match bits
                                         // were set from; past `capacity` the bits are incomplete and the
                                         // rows are looked up instead. NULL: the bits are complete
  RangeGate gate;  // closed: looked up in place
};

// Rows written by the warps of a CTA to consecutive output positions: one reservation for all of them. `cnt`: the
// warp's rows; `part`, in shared memory, keeps the warps' counts. Returns the warp's first position.
__device__ __forceinline__ unsigned long long cta_reserve(uint32_t cnt, uint32_t (&part)[kUnitWarps],
                                                          unsigned long long& base, unsigned long long* d_count) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) part[warp] = cnt;
  __syncthreads();
  const uint32_t c = lane < kUnitWarps ? part[lane] : 0;
  const uint32_t incl = warp_inclusive_sum(c);
  const uint32_t mine = __shfl_sync(kFullMask, incl - c, warp);
  if (warp == 0 && lane == kUnitWarps - 1) base = incl ? atomicAdd(d_count, (unsigned long long)incl) : 0ull;
  __syncthreads();
  return base + mine;
}

// Rows that fit behind position `base`.
__device__ __forceinline__ uint32_t rows_left(int64_t capacity, int64_t base) {
  const int64_t left = capacity - base;
  return left <= 0 ? 0u : left > 0x7fffffff ? 0x7fffffffu : (uint32_t)left;
}

// Validity bits of the lanes with `on`, whose rows went to consecutive positions. Called by the whole warp.
__device__ __forceinline__ void set_out_bits(uint32_t* valid, uint32_t pos, bool on, bool bit) {
  const unsigned any = __ballot_sync(kFullMask, on);
  if (!any) return;
  const uint32_t word0 = __shfl_sync(kFullMask, pos, __ffs(any) - 1) >> 5;
  const bool low = (pos >> 5) == word0;
  const uint32_t b = on && bit ? 1u << (pos & 31) : 0u;
  const uint32_t w0 = __reduce_or_sync(kFullMask, low ? b : 0u), w1 = __reduce_or_sync(kFullMask, low ? 0u : b);
  if ((threadIdx.x & 31) == 0) {
    if (w0) atomicOr(valid + word0, w0);
    if (w1) atomicOr(valid + word0 + 1, w1);
  }
}

// Payload values of N probe rows of the lane, and their stores: all loads of a column are in flight together.
template <int N>
__device__ __forceinline__ void load_rows(const PayloadIn& in, const uint32_t (&row)[N], uint32_t sel, uint64_t (&v)[N]) {
  auto go = [&](auto x) {
    using T = decltype(x);
#pragma unroll
    for (int j = 0; j < N; ++j) v[j] = (sel >> j & 1u) ? (uint64_t)__ldcs(static_cast<const T*>(in.data) + row[j]) : 0ull;
  };
  switch (in.width) {
    case 8: return go((unsigned long long)0);
    case 4: return go((unsigned int)0);
    case 2: return go((unsigned short)0);
    default: return go((unsigned char)0);
  }
}
template <int N>
__device__ __forceinline__ void store_rows(void* out, int width, int64_t base, const uint32_t (&at)[N], uint32_t sel,
                                           const uint64_t (&v)[N]) {
  auto go = [&](auto x) {
    using T = decltype(x);
#pragma unroll
    for (int j = 0; j < N; ++j)
      if (sel >> j & 1u) __stcs(static_cast<T*>(out) + base + at[j], (T)v[j]);
  };
  switch (width) {
    case 8: return go((unsigned long long)0);
    case 4: return go((unsigned int)0);
    case 2: return go((unsigned short)0);
    default: return go((unsigned char)0);
  }
}

// Writes the lane's rows row[j] (bit j of `sel`) to the positions base + at[j]: row ids and probe payloads. The j-th
// rows of a warp go to consecutive positions.
template <int N>
__device__ __forceinline__ void emit_rows(const KindArgs& a, const uint32_t (&row)[N], int64_t base, const uint32_t (&at)[N],
                                          uint32_t sel) {
#pragma unroll
  for (int j = 0; j < N; ++j) {
    if (!(sel >> j & 1u)) continue;
    if (a.out_prid) __stcs(a.out_prid + base + at[j], (int32_t)row[j]);
    if (a.out_brid) __stcs(a.out_brid + base + at[j], kNoRow);
  }
  for (int c = 0; c < a.n_pin; ++c) {
    uint64_t v[N];
    load_rows<N>(a.pin[c], row, sel, v);
    store_rows<N>(a.pout[c].data, a.pin[c].width, base, at, sel, v);
    if (!a.pout[c].valid) continue;
#pragma unroll
    for (int j = 0; j < N; ++j) {
      const bool on = sel >> j & 1u;
      set_out_bits(a.pout[c].valid + (base >> 5), (uint32_t)(base & 31) + at[j], on, on && payload_valid(a.pin[c], row[j]));
    }
  }
}

// Mark bytes of 32 * S rows from `row0` on, word j of `found` for 32 of them: four bytes per lane where the rows are
// whole and the bytes aligned.
template <int S>
__device__ __forceinline__ void mark_bytes(uint8_t* mark, const unsigned (&found)[S], uint32_t rows) {
  const int lane = threadIdx.x & 31;
  if (rows == 32u * S && ((uintptr_t)mark & 3) == 0) {
    unsigned w = found[0];
#pragma unroll
    for (int j = 1; j < S; ++j) w = lane >> 3 == j ? found[j] : w;
    const uint32_t x = w >> (4 * (lane & 7)) & 0xfu;
    if (lane < 8 * S) reinterpret_cast<uint32_t*>(mark)[lane] = (x & 1u) | (x & 2u) << 7 | (x & 4u) << 14 | (x & 8u) << 21;
  } else {
#pragma unroll
    for (int j = 0; j < S; ++j)
      if (32u * j + lane < rows) mark[32 * j + lane] = found[j] >> lane & 1u;
  }
}

// SEMI, ANTI (and the unmatched probe rows of LEFT and FULL), MARK, and FULL's flags of matched slots in one pass, the
// table looked up in place, in units of 32 * S rows: no scratch and no bits. A CTA reserves once for its rows and
// writes them in order, payload column after payload column.
// It is bound by instructions while the table is in L2, so 64 warps per SM and short code: us for 64M int64 keys into
// 4M / 16M keys, 80 % in the build: SEMI with an 8-byte payload 653 / 1,277, MARK 452 / 1,130 (one 64-bit lookup per
// lane and 32-row step, matches staged per warp: 901 / 1,390 and 727 / 1,261; match bits, then a pass over them: 686
// and 477 / -). With 48 warps: 706 / 1,250 and 512 / 1,069. NULLS: the probe keys have NULLs (apart, since the test for
// the bitmask alone took 38 of 387 us of a MARK). Where all of a unit lies outside the build's range nothing is looked
// up (64M rows, SEMI 277 -> 127 us); MARK, for which it cost 4 %, does not ask. BLOCKS: consecutive blocks of units per
// CTA, for a launch that may have nothing to do (64K CTAs that return at once take 37 us). Not every form has a variant
// of its own: the first call of a process loads them all (64 take 5.3 ms).
template <typename K, bool WIDE, int MODE, int S, bool NULLS, int BLOCKS>
__global__ void __launch_bounds__(kUnitThreads, 8) kind_units_kernel(TableDev t, const K* __restrict__ keys,
                                                                     const uint32_t* __restrict__ kv_in, int64_t kvoff,
                                                                     uint32_t n, KindArgs a) {
  __shared__ WaitRows<S> s_wait[kUnitWarps];
  __shared__ uint32_t s_cnt[kUnitWarps];
  __shared__ unsigned long long s_base;
  // the match bits are complete: the rows are emitted, the build rows found by them
  if ((MODE == kAnti || MODE == kFlags) && a.inner_rows && (int64_t)*a.inner_rows <= a.capacity) return;
  if (BLOCKS > 1 && a.gate.rows && gate_open(a.gate)) return;  // looked up in partition order
  const uint32_t* kv = NULLS ? kv_in : nullptr;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool null_found = NULLS && t.null_group >= 0 && __ldg(t.grp_off + t.null_group + 1) > __ldg(t.grp_off + t.null_group);
  for (uint32_t block = 0; block < BLOCKS; ++block) {
    const auto [first, rows] = unit_rows<false, S>(RunArgs{}, Units{0, (blockIdx.x * BLOCKS + block) * kUnitWarps}, n);
    K k[S];
#pragma unroll
    for (int j = 0; j < S; ++j) k[j] = 32 * j + lane < rows ? __ldcs(keys + first + 32 * j + lane) : (K)0;
    uint32_t pos[S];
    bool any = true;
    if constexpr (MODE == kSemi || MODE == kAnti) {  // where the whole unit lies outside the build's range, that is all there is to do
      any = false;
#pragma unroll
      for (int j = 0; j < S; ++j) {
        SectorKey key;
        any |= sector_key<K, WIDE>(t, k[j], key);
        pos[j] = kNoPos;
      }
      any = __any_sync(kFullMask, any);
    }
    if (any) unit_lookup<K, WIDE, false, S, MODE == kFlags>(t, k, kv, kvoff, first, 0, rows, s_wait[warp], pos);
    unsigned found[S], known[S];
#pragma unroll
    for (int j = 0; j < S; ++j) {
      const uint32_t v = 32 * j + lane;
      const bool null = NULLS && v < rows && (null_found || MODE == kMark) && !bit_valid(kv, kvoff, first + v);
      if (MODE == kFlags) {
        if (null) pos[j] = (uint32_t)t.null_group;
        if (pos[j] != kNoPos) a.flags[pos[j]] = 1;
        continue;
      }
      found[j] = __ballot_sync(kFullMask, pos[j] != kNoPos || (null && null_found));
      if (MODE == kMark) known[j] = NULLS ? ~__ballot_sync(kFullMask, null) : kFullMask;
      if (MODE == kAnti) found[j] = __ballot_sync(kFullMask, v < rows) & ~found[j];
    }
    if (MODE == kMark && rows > 0) {
      mark_bytes<S>(a.mark + first, found, rows);
      if (a.mark_valid && 32u * lane < rows) {
        unsigned w = 0;
#pragma unroll
        for (int j = 0; j < S; ++j) w = lane == j ? found[j] | (a.build_has_null ? 0u : known[j]) : w;
        const uint32_t left = rows - 32 * lane;
        a.mark_valid[(first >> 5) + lane] = left >= 32 ? w : w & ((1u << left) - 1u);
      }
    }
    if constexpr (MODE == kSemi || MODE == kAnti) {
      uint32_t cnt = 0;
#pragma unroll
      for (int j = 0; j < S; ++j) cnt += __popc(found[j]);
      const int64_t base = (int64_t)cta_reserve(cnt, s_cnt, s_base, a.d_count);
      if (cnt == 0) continue;
      const uint32_t room = rows_left(a.capacity, base);
      uint32_t row[S], at[S], run = 0, sel = 0;
#pragma unroll
      for (int j = 0; j < S; ++j) {
        row[j] = first + 32 * j + lane;
        at[j] = run + __popc(found[j] & ((1u << lane) - 1u));
        run += __popc(found[j]);
        if ((found[j] >> lane & 1u) && at[j] < room) sel |= 1u << j;
      }
      emit_rows<S>(a, row, base, at, sel);
    }
  }
}

// Emits the probe rows whose bit in `words` is set (WANT) or clear, with their probe payloads. A warp takes 1024
// rows, one word per lane; a CTA reserves once for its 8192 rows, and the words' rows go to consecutive
// positions, so rows, payload loads and stores stay in order. 64M rows, 70 % of them with an 8-byte payload:
// 190 us (5.7 TB/s), 254 with one word at a time.
template <bool WANT>
__global__ void __launch_bounds__(kUnitThreads) select_rows_kernel(const uint32_t* __restrict__ words, uint32_t n, KindArgs a) {
  __shared__ uint32_t s_cnt[kUnitWarps];
  __shared__ unsigned long long s_base;
  if (a.inner_rows && (int64_t)*a.inner_rows > a.capacity) return;  // the bits are incomplete
  if (!gate_open(a.gate)) return;                                   // not set: looked up in place
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned below = (1u << lane) - 1u;
  const uint32_t word0 = (blockIdx.x * kUnitWarps + warp) * 32;
  const uint32_t row0 = (word0 + lane) * 32;
  uint32_t w = 0;
  if (row0 < n) {
    w = __ldg(words + word0 + lane);
    if (!WANT) w = ~w;
    if (n - row0 < 32) w &= (1u << (n - row0)) - 1u;
  }
  const uint32_t incl = warp_inclusive_sum(__popc(w));
  const int64_t base = (int64_t)cta_reserve(__shfl_sync(kFullMask, incl, 31), s_cnt, s_base, a.d_count);
  const uint32_t mine = incl - __popc(w);
  const uint32_t room = rows_left(a.capacity, base);
  constexpr int B = 8;  // words at a time
  for (int q0 = 0; q0 < 32; q0 += B) {
    uint32_t row[B], at[B], sel = 0;
#pragma unroll
    for (int h = 0; h < B; ++h) {
      const uint32_t wq = __shfl_sync(kFullMask, w, q0 + h);
      row[h] = (word0 + q0 + h) * 32 + lane;
      at[h] = __shfl_sync(kFullMask, mine, q0 + h) + __popc(wq & below);
      if ((wq >> lane & 1u) && at[h] < room) sel |= 1u << h;
    }
    if (__any_sync(kFullMask, sel != 0)) emit_rows<B>(a, row, base, at, sel);
  }
}

// MARK from the match bits: one byte per row, and the validity words (a row without a match is NULL when its
// key is, or when the build has a NULL key). One thread per word.
__global__ void __launch_bounds__(kKindThreads) mark_rows_kernel(const uint32_t* __restrict__ words, const uint32_t* __restrict__ kv,
                                                                 int64_t kvoff, int64_t n, KindArgs a) {
  const int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, row0 = q * 32;
  if (row0 >= n || !gate_open(a.gate)) return;
  const uint32_t w = __ldg(words + q);
  const int rows = (int)(n - row0 < 32 ? n - row0 : 32);
  uint8_t* out = a.mark + row0;
  if (rows == 32 && ((uintptr_t)out & 15) == 0) {
    uint32_t b[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const uint32_t x = w >> (4 * i) & 0xfu;
      b[i] = (x & 1u) | (x & 2u) << 7 | (x & 4u) << 14 | (x & 8u) << 21;
    }
    reinterpret_cast<uint4*>(out)[0] = make_uint4(b[0], b[1], b[2], b[3]);
    reinterpret_cast<uint4*>(out)[1] = make_uint4(b[4], b[5], b[6], b[7]);
  } else {
    for (int i = 0; i < rows; ++i) out[i] = w >> i & 1u;
  }
  if (!a.mark_valid) return;
  uint32_t valid = w;
  if (!a.build_has_null) {
    uint32_t known = kFullMask;
    if (kv) {
      known = 0;
      for (int i = 0; i < rows; ++i) known |= (uint32_t)bit_valid(kv, kvoff, row0 + i) << i;
    }
    valid |= known;
  }
  a.mark_valid[q] = rows == 32 ? valid : valid & ((1u << rows) - 1u);
}

struct BuildEmitArgs {
  int32_t* out_prid;
  int32_t* out_brid;
  int32_t n_bin;
  PayloadIn bin[kMaxPayload];
  PayloadOut bout[kMaxPayload];
  const int32_t* pos_rid;  // table position -> build row id (NULL: positions are row ids)
  int32_t pos_stride;
  int64_t capacity;
  unsigned long long* d_count;
  const uint8_t* flags;
  // FULL by build-row bits: when set and the INNER rows fit the capacity, the unmatched build rows
  // are the rows whose bit in `matched` is clear (unmatched_build_rows_kernel); the slot / member /
  // NULL-row walks then do nothing
  const unsigned long long* inner_rows;
  const uint32_t* matched;
};

__device__ __forceinline__ bool full_by_bits(const BuildEmitArgs& a) {
  return a.inner_rows != nullptr && (int64_t)*a.inner_rows <= a.capacity;
}

// Unmatched build rows of a FULL join, staged per warp like the SEMI / ANTI rows: build row ids
// collect in the warp's shared-memory area, and a flush reserves their output range with one
// atomicAdd and writes them (probe row id SJ_NO_ROW, build row id, build payloads) in order.
struct BuildEmitter {
  const BuildEmitArgs& a;
  int32_t* st;        // this warp's kKindStage staged build row ids
  uint32_t fill = 0;  // warp-uniform
  __device__ BuildEmitter(const BuildEmitArgs& args, int32_t* stage) : a(args), st(stage) {}
  __device__ void add(bool sel, int32_t brid) {
    const int lane = threadIdx.x & 31;
    const unsigned bal = __ballot_sync(kFullMask, sel);
    if (!bal) return;
    if (sel) st[fill + __popc(bal & ((1u << lane) - 1u))] = brid;
    fill += __popc(bal);
    if (fill > (uint32_t)(kKindStage - 32)) flush();
  }
  __device__ void flush() {
    const int lane = threadIdx.x & 31;
    __syncwarp();
    unsigned long long base = 0;
    if (lane == 0 && fill) base = atomicAdd(a.d_count, (unsigned long long)fill);
    base = __shfl_sync(kFullMask, base, 0);
    for (uint32_t e = lane; e < fill; e += 32) {
      const int64_t p = (int64_t)base + e;
      if (p >= a.capacity) break;
      const int32_t brid = st[e];
      if (a.out_prid) a.out_prid[p] = kNoRow;
      if (a.out_brid) a.out_brid[p] = brid;
      for (int c = 0; c < a.n_bin; ++c) {
        store_elem(a.bout[c].data, p, a.bin[c].width, pl_load(a.bin[c], brid));
        if (a.bout[c].valid && payload_valid(a.bin[c], brid)) set_out_bit(a.bout[c].valid, p);
      }
    }
    __syncwarp();
    fill = 0;
  }
};

__device__ __forceinline__ int32_t rid_of_pos(const BuildEmitArgs& a, int64_t pos) {
  return a.pos_rid ? __ldg(reinterpret_cast<const int32_t*>(reinterpret_cast<const char*>(a.pos_rid) +
                                                             pos * a.pos_stride))
                   : (int32_t)pos;
}

// FULL, DISTINCT table: every live slot nobody matched.
template <bool WIDE>
__global__ void __launch_bounds__(kKindThreads) unmatched_slots_kernel(TableDev t, int64_t n_slots, BuildEmitArgs a) {
  using Ops = SlotOps<WIDE>;
  const int lane = threadIdx.x & 31;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  __shared__ int32_t s_stage[kKindThreads / 32][kKindStage];
  BuildEmitter em(a, s_stage[threadIdx.x >> 5]);
  if (full_by_bits(a)) return;  // unmatched_build_rows_kernel emits them
  for (int64_t i0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) & ~31ll; i0 < n_slots; i0 += stride) {
    const int64_t i = i0 + lane;
    bool sel = false;
    int32_t brid = 0;
    if (i < n_slots) {
      const Bucket bk = load_bucket<true>(t.slots, (uint32_t)(i / Ops::kSlots));
      const int q = (int)(i % Ops::kSlots);
      if (!Ops::empty(bk, q) && !a.flags[i]) {
        sel = true;
        brid = rid_of_pos(a, Ops::rid(bk, q, t.rbits));
      }
    }
    em.add(sel, brid);
  }
  em.flush();
}

// FULL, GROUPED table: member i (group order) belongs to the last group s with grp_off[s] <= i.
__global__ void __launch_bounds__(kKindThreads) unmatched_members_kernel(TableDev t, int64_t n_members,
                                                                         int64_t n_groups, BuildEmitArgs a) {
  const int lane = threadIdx.x & 31;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  __shared__ int32_t s_stage[kKindThreads / 32][kKindStage];
  BuildEmitter em(a, s_stage[threadIdx.x >> 5]);
  if (full_by_bits(a)) return;  // unmatched_build_rows_kernel emits them
  for (int64_t i0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) & ~31ll; i0 < n_members; i0 += stride) {
    const int64_t i = i0 + lane;
    bool sel = false;
    int32_t brid = 0;
    if (i < n_members) {
      int64_t lo = 0, hi = n_groups - 1;  // largest s with grp_off[s] <= i
      while (lo < hi) {
        const int64_t mid = (lo + hi + 1) >> 1;
        if (__ldg(t.grp_off + mid) <= i) lo = mid;
        else hi = mid - 1;
      }
      if (!a.flags[lo]) {
        sel = true;
        brid = rid_of_pos(a, t.grp_rid ? (int64_t)__ldg(t.grp_rid + i) : i);
      }
    }
    em.add(sel, brid);
  }
  em.flush();
}

// FULL: the NULL-key build rows (not in the table when NULLs never match).
__global__ void __launch_bounds__(kKindThreads) null_build_rows_kernel(const int32_t* __restrict__ null_rid,
                                                                       int64_t n_null, BuildEmitArgs a) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  __shared__ int32_t s_stage[kKindThreads / 32][kKindStage];
  BuildEmitter em(a, s_stage[threadIdx.x >> 5]);
  if (full_by_bits(a)) return;  // unmatched_build_rows_kernel emits them
  for (int64_t i0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) & ~31ll; i0 < n_null; i0 += stride) {
    const int64_t i = i0 + (threadIdx.x & 31);
    em.add(i < n_null, i < n_null ? __ldg(null_rid + i) : 0);
  }
  em.flush();
}

// FULL by build-row bits: every build row (NULL keys included) whose bit is clear.
__global__ void __launch_bounds__(kKindThreads) unmatched_build_rows_kernel(const uint32_t* __restrict__ matched,
                                                                            int64_t nb, BuildEmitArgs a) {
  if (!full_by_bits(a)) return;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  __shared__ int32_t s_stage[kKindThreads / 32][kKindStage];
  BuildEmitter em(a, s_stage[threadIdx.x >> 5]);
  for (int64_t i0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) & ~31ll; i0 < nb; i0 += stride) {
    const int64_t i = i0 + (threadIdx.x & 31);
    em.add(i < nb && !(__ldg(matched + (i >> 5)) >> (i & 31) & 1u), (int32_t)i);
  }
  em.flush();
}

// Sets validity bits [lo, hi) (bounds read from the device, clamped to cap; lo_p NULL = 0).
__global__ void set_valid_range_kernel(uint32_t* words, const unsigned long long* lo_p, const unsigned long long* hi_p,
                                       int64_t cap) {
  const int64_t lo = lo_p ? std::min<int64_t>((int64_t)*lo_p, cap) : 0;
  const int64_t hi = std::min<int64_t>((int64_t)*hi_p, cap);
  if (hi <= lo) return;
  for (int64_t w = (lo >> 5) + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; w <= ((hi - 1) >> 5);
       w += (int64_t)gridDim.x * blockDim.x) {
    const int64_t a = std::max<int64_t>(lo, w * 32) - w * 32;
    const int64_t b = std::min<int64_t>(hi, w * 32 + 32) - w * 32;
    const unsigned mask = (b - a == 32) ? kFullMask : (((1u << (b - a)) - 1u) << a);
    atomicOr(words + w, mask);
  }
}

__global__ void set_count_kernel(int64_t* d_count, int64_t v) { *d_count = v; }

// ------------------------------------------------------------------------------------------------
// host side
// ------------------------------------------------------------------------------------------------
// LEFT / FULL: bit r of `bits` for every probe row r among the first min(*d_n, cap) INNER rows.
__global__ void __launch_bounds__(256) matched_bits_kernel(const int32_t* __restrict__ prid,
                                                           const unsigned long long* d_n, int64_t cap, uint32_t* bits) {
  const int64_t n = (int64_t)*d_n < cap ? (int64_t)*d_n : cap;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const uint32_t r = (uint32_t)__ldg(prid + i);
    atomicOr(bits + (r >> 5), 1u << (r & 31));
  }
}

static int kind_grid(const sj_table* t, int64_t n) {
  const int64_t need = (n + kKindThreads - 1) / kKindThreads;
  return (int)std::max<int64_t>(1, std::min<int64_t>(need, (int64_t)sm_count(t->device) * 8));
}

// Probes of at most this many rows take units of 32 rows. Units of 32 against units of 128, int64 keys, SEMI with a
// payload / MARK: 10K rows 3.8 / 2.9 against 5.1 / 3.6 us, 200K 4.9 / 3.8 against 5.6 / 4.2, 300K 6.6 / 5.3 against
// 6.3 / 5.0, 400K 7.3 / 5.4 against 6.3 / 4.8.
constexpr int64_t kFewKindRows = 1 << 18;

template <int MODE>
static void launch_kind(const sj_table* t, const sj_column& p, const KindArgs& a, cudaStream_t s) {
  // 64M rows, SEMI with two / four blocks: 539 / 563 us in place after the choice (70 % out of range), 1,034 / 1,023 in
  // partition order; MARK 487 / 485 and 958 / 952
  constexpr int kBlocks = MODE == kSemi || MODE == kAnti ? 2 : 4;
  const bool idle = MODE == kFlags || a.gate.rows || a.inner_rows;  // may have nothing to do
  const bool few = !idle && p.num_rows <= kFewKindRows;
  const int64_t per_cta = (few ? 32 : 128) * kUnitWarps * (idle ? kBlocks : 1);
  const int grid = (int)((p.num_rows + per_cta - 1) / per_cta);
  const bool wide = t->slot_kind == SJ_SLOT_WIDE128;
  const TableDev d = table_dev(t);
  KernelTimer timer(MODE == kMark ? "mark" : MODE == kFlags ? "match_flags" : MODE == kSemi ? "semi"
                    : a.inner_rows ? "unmatched_probe" : "anti", s);
  auto go = [&](auto k, auto w) {
    using K = decltype(k);
    constexpr bool W = decltype(w)::value;
    auto launch = [&](auto kernel) {
      kernel<<<grid, kUnitThreads, 0, s>>>(d, static_cast<const K*>(p.data), p.validity, p.validity_offset,
                                           (uint32_t)p.num_rows, a);
    };
    if constexpr (MODE == kFlags) {
      launch(kind_units_kernel<K, W, MODE, 4, true, kBlocks>);
    } else {
      if (idle) launch(p.validity ? kind_units_kernel<K, W, MODE, 4, true, kBlocks> : kind_units_kernel<K, W, MODE, 4, false, kBlocks>);
      else if (few) launch(kind_units_kernel<K, W, MODE, 1, true, 1>);
      else launch(p.validity ? kind_units_kernel<K, W, MODE, 4, true, 1> : kind_units_kernel<K, W, MODE, 4, false, 1>);
    }
  };
  if (t->key_type == SJ_INT32) {
    if (wide) go(int32_t{}, std::true_type{});
    else go(int32_t{}, std::false_type{});
  } else {
    if (wide) go(int64_t{}, std::true_type{});
    else go(int64_t{}, std::false_type{});
  }
}

template <bool WANT>
static void launch_select(const uint32_t* words, int64_t n, const KindArgs& a, cudaStream_t s) {
  KernelTimer timer("select_rows", s);
  const int64_t per_cta = (int64_t)kUnitWarps * 1024;
  select_rows_kernel<WANT><<<(int)((n + per_cta - 1) / per_cta), kUnitThreads, 0, s>>>(words, (uint32_t)n, a);
}

static sj_status probe_payloads(const sj_column& p, const GatherSpec& gs, KindArgs& a) {
  if (gs.n_probe_payload < 0 || gs.n_probe_payload > kMaxPayload)
    return set_error(SJ_ERR_INVALID, "at most 8 payload columns per side");
  if (gs.n_probe_payload && (!gs.probe_payload || !gs.out_probe_payload))
    return set_error(SJ_ERR_INVALID, "payload column arrays must not be NULL");
  a.n_pin = gs.n_probe_payload;
  for (int c = 0; c < a.n_pin; ++c) {
    const sj_column& in = gs.probe_payload[c];
    const sj_mut_column& out = gs.out_probe_payload[c];
    SJ_TRY(validate_column(&in, "probe payload", false));
    if (in.num_rows != p.num_rows) return set_error(SJ_ERR_INVALID, "probe payload row count differs from its key column");
    if (out.type != in.type) return set_error(SJ_ERR_INVALID, "probe output type differs");
    if (gs.capacity > 0 && !out.data) return set_error(SJ_ERR_INVALID, "probe output data is NULL");
    if (in.validity && gs.capacity > 0 && !out.validity)
      return set_error(SJ_ERR_INVALID, "probe payload has NULLs but its output has no validity");
    a.pin[c] = column_payload(in.data, in.validity, in.validity_offset, type_width(in.type));
    a.pout[c] = PayloadOut{out.data, in.validity ? out.validity : nullptr};
  }
  return SJ_OK;
}

static sj_status zero_validity(const sj_mut_column* outs, int n, int64_t capacity, cudaStream_t s) {
  const size_t bytes = (size_t)((capacity + 31) / 32) * sizeof(uint32_t);
  for (int c = 0; c < n; ++c)
    if (outs[c].validity && bytes) SJ_CUDA_TRY(cudaMemsetAsync(outs[c].validity, 0, bytes, s));
  return SJ_OK;
}

sj_status probe_join(const sj_table* t, int32_t kind, const sj_column& p, const GatherSpec& gs, uint8_t* out_mark,
                     uint32_t* out_mark_valid, const Allocator& alloc, cudaStream_t s, int64_t* d_count) {
  if (kind == SJ_JOIN_INNER) return probe_gather(t, p, gs, alloc, s, d_count);
  if (kind < SJ_JOIN_INNER || kind > SJ_JOIN_FULL) return set_error(SJ_ERR_INVALID, "unknown join kind");
  SJ_TRY(validate_column(&p, "probe key", true));
  if (p.type != t->key_type) return set_error(SJ_ERR_INVALID, "probe key type differs from the build key type");
  if (p.num_rows > INT32_MAX) return set_error(SJ_ERR_INVALID, "probe side exceeds the int32 row-id range");
  if (gs.capacity < 0) return set_error(SJ_ERR_INVALID, "capacity must be >= 0");
  unsigned long long* dc = reinterpret_cast<unsigned long long*>(d_count);
  KindArgs a{};
  a.capacity = gs.capacity;
  a.d_count = dc;

  if (kind == SJ_JOIN_MARK) {
    if (t->null_eq == SJ_NULLS_EQUAL) return set_error(SJ_ERR_INVALID, "MARK joins compare NULLs as unequal");
    if (p.num_rows > 0 && !out_mark) return set_error(SJ_ERR_INVALID, "MARK needs out_mark");
    a.mark = out_mark;
    a.mark_valid = out_mark_valid;
    a.build_has_null = t->null_rows > 0;
    set_count_kernel<<<1, 1, 0, s>>>(d_count, p.num_rows);
    Scratch bits;
    const uint32_t* words = nullptr;
    SJ_TRY(find_in_order(t, p, alloc, s, bits, &words, &a.gate));
    if (words) {
      const int64_t n_words = (p.num_rows + 31) / 32;
      KernelTimer timer("mark_rows", s);
      mark_rows_kernel<<<(int)((n_words + kKindThreads - 1) / kKindThreads), kKindThreads, 0, s>>>(
          words, p.validity, p.validity_offset, p.num_rows, a);
    }
    if (p.num_rows > 0) launch_kind<kMark>(t, p, a, s);
    SJ_CUDA_TRY(cudaGetLastError());
    return SJ_OK;
  }
  if (kind == SJ_JOIN_SEMI || kind == SJ_JOIN_ANTI) {
    SJ_TRY(probe_payloads(p, gs, a));
    a.out_prid = gs.out_probe_rid;
    SJ_CUDA_TRY(cudaMemsetAsync(d_count, 0, sizeof(int64_t), s));
    SJ_TRY(zero_validity(gs.out_probe_payload, gs.n_probe_payload, gs.capacity, s));
    Scratch bits;
    const uint32_t* words = nullptr;
    SJ_TRY(find_in_order(t, p, alloc, s, bits, &words, &a.gate));
    if (words) {
      if (kind == SJ_JOIN_SEMI) launch_select<true>(words, p.num_rows, a, s);
      else launch_select<false>(words, p.num_rows, a, s);
    }
    if (p.num_rows > 0) {
      if (kind == SJ_JOIN_SEMI) launch_kind<kSemi>(t, p, a, s);
      else launch_kind<kAnti>(t, p, a, s);
    }
    SJ_CUDA_TRY(cudaGetLastError());
    return SJ_OK;
  }

  // LEFT / FULL
  const bool full = kind == SJ_JOIN_FULL;
  const bool attached = gs.n_build_payload > 0 && gs.build_payload == nullptr;
  if (full && attached)
    return set_error(SJ_ERR_INVALID, "FULL joins gather build payloads from caller columns (build_payload != NULL)");
  for (int c = 0; c < gs.n_build_payload; ++c)
    if (gs.capacity > 0 && (!gs.out_build_payload || !gs.out_build_payload[c].validity))
      return set_error(SJ_ERR_INVALID, "LEFT/FULL build payload outputs need validity (NULL padding)");
  for (int c = 0; full && c < gs.n_probe_payload; ++c)
    if (gs.capacity > 0 && (!gs.out_probe_payload || !gs.out_probe_payload[c].validity))
      return set_error(SJ_ERR_INVALID, "FULL probe payload outputs need validity (NULL padding)");
  SJ_TRY(probe_payloads(p, gs, a));
  if (gs.n_build_payload > 0 && !gs.out_build_payload)
    return set_error(SJ_ERR_INVALID, "payload column arrays must not be NULL");
  SJ_TRY(zero_validity(gs.out_build_payload, gs.n_build_payload, gs.capacity, s));
  if (full) SJ_TRY(zero_validity(gs.out_probe_payload, gs.n_probe_payload, gs.capacity, s));
  Scratch marks;  // [0] = INNER rows, [1] = LEFT rows
  SJ_TRY(marks.get(alloc, 2 * sizeof(unsigned long long), s));
  unsigned long long* m = marks.as<unsigned long long>();

  // 1. INNER rows, and where the unit probe serves them, one bit per probe row with a match
  Scratch mbits;
  const size_t mbytes = (size_t)((p.num_rows + 31) / 32) * sizeof(uint32_t);
  bool by_probe = false;
  GatherSpec inner = gs;
  // The bits are optional here, and the INNER probe's own scratch, taken after them and given back before the
  // next step, has the better claim: a budget that holds either but not both must do.
  auto get_bits = [&]() -> sj_status {
    SJ_TRY(mbits.get(alloc, mbytes, s));
    SJ_CUDA_TRY(cudaMemsetAsync(mbits.ptr, 0, mbytes, s));
    return SJ_OK;
  };
  if (p.num_rows > 0) {
    if (sj_status e = get_bits(); e == SJ_OK) {
      inner.matched = mbits.as<uint32_t>();
      inner.matched_set = &by_probe;
    } else if (e != SJ_ERR_OOM) {
      return e;
    }
  }
  sj_status probed = probe_gather(t, p, inner, alloc, s, d_count);
  if (probed == SJ_ERR_OOM && mbits.ptr) {
    mbits.drop();
    by_probe = false;
    probed = probe_gather(t, p, gs, alloc, s, d_count);
  }
  SJ_TRY(probed);
  clear_error();  // of an allocation that was refused and then done without
  SJ_CUDA_TRY(cudaMemcpyAsync(m, d_count, sizeof(int64_t), cudaMemcpyDeviceToDevice, s));
  // 2. unmatched probe rows, appended: the rows whose bit is clear. Where the probe did not set the bits they
  // are set from the INNER rows' probe row ids; if those overflowed the capacity (known on the device) or are
  // not written, the rows are looked up again
  a.out_prid = gs.out_probe_rid;
  a.out_brid = gs.out_build_rid;
  if (p.num_rows > 0) {
    if (by_probe) {
      launch_select<false>(mbits.as<uint32_t>(), p.num_rows, a, s);
    } else if (gs.out_probe_rid && gs.capacity > 0) {
      if (!mbits.ptr) SJ_TRY(get_bits());
      {
        KernelTimer timer("matched_bits", s);
        matched_bits_kernel<<<kind_grid(t, std::min<int64_t>(gs.capacity, p.num_rows)), 256, 0, s>>>(
            gs.out_probe_rid, m, gs.capacity, mbits.as<uint32_t>());
      }
      a.inner_rows = m;
      launch_select<false>(mbits.as<uint32_t>(), p.num_rows, a, s);
      launch_kind<kAnti>(t, p, a, s);
    } else {
      launch_kind<kAnti>(t, p, a, s);
    }
  }
  mbits.drop();
  SJ_CUDA_TRY(cudaMemcpyAsync(m + 1, d_count, sizeof(int64_t), cudaMemcpyDeviceToDevice, s));

  // 3. FULL: unmatched build rows. With build row ids written: the build rows no INNER row names
  // (one bit per build row, set from the INNER rows' build row ids), else — or when the INNER rows
  // overflowed the capacity, decided on the device — the slots (groups) no probe row matched
  Scratch flags, bbits;
  if (full) {
    const int64_t ns = t->num_slots();
    const int64_t nflags = ns + 1;  // + the NULL group
    SJ_TRY(flags.get(alloc, (size_t)nflags, s));
    SJ_CUDA_TRY(cudaMemsetAsync(flags.ptr, 0, (size_t)nflags, s));
    const bool bits_ok = gs.out_build_rid != nullptr && gs.capacity > 0 && t->build_rows > 0;
    if (bits_ok) {
      const size_t words = (size_t)((t->build_rows + 31) / 32);
      SJ_TRY(bbits.get(alloc, words * sizeof(uint32_t), s));
      SJ_CUDA_TRY(cudaMemsetAsync(bbits.ptr, 0, words * sizeof(uint32_t), s));
      KernelTimer timer("matched_build_bits", s);
      matched_bits_kernel<<<kind_grid(t, std::min<int64_t>(gs.capacity, p.num_rows)), 256, 0, s>>>(
          gs.out_build_rid, m, gs.capacity, bbits.as<uint32_t>());
    }
    KindArgs fa{};
    fa.flags = flags.as<uint8_t>();
    fa.capacity = gs.capacity;
    fa.inner_rows = bits_ok ? m : nullptr;  // the flags pass returns at once when the bits apply
    if (p.num_rows > 0) launch_kind<kFlags>(t, p, fa, s);
    BuildEmitArgs e{};
    e.out_prid = gs.out_probe_rid;
    e.out_brid = gs.out_build_rid;
    e.n_bin = gs.n_build_payload;
    for (int c = 0; c < e.n_bin; ++c) {
      const sj_column& in = gs.build_payload[c];
      SJ_TRY(validate_column(&in, "build payload", false));
      if (in.num_rows != t->build_rows) return set_error(SJ_ERR_INVALID, "build payload row count differs from its key column");
      if (gs.out_build_payload[c].type != in.type) return set_error(SJ_ERR_INVALID, "build output type differs");
      e.bin[c] = column_payload(in.data, in.validity, in.validity_offset, type_width(in.type));
      e.bout[c] = PayloadOut{gs.out_build_payload[c].data, in.validity ? gs.out_build_payload[c].validity : nullptr};
    }
    e.pos_rid = t->pos_rid;
    e.pos_stride = t->pos_stride;
    e.capacity = gs.capacity;
    e.d_count = dc;
    e.flags = fa.flags;
    e.inner_rows = bits_ok ? m : nullptr;
    e.matched = bits_ok ? bbits.as<uint32_t>() : nullptr;
    const TableDev d = table_dev(t);
    KernelTimer timer("unmatched_build", s);
    if (bits_ok)
      unmatched_build_rows_kernel<<<kind_grid(t, t->build_rows), kKindThreads, 0, s>>>(e.matched, t->build_rows, e);
    if (t->layout == SJ_LAYOUT_DISTINCT) {
      if (ns > 0) {
        if (t->slot_kind == SJ_SLOT_WIDE128) unmatched_slots_kernel<true><<<kind_grid(t, ns), kKindThreads, 0, s>>>(d, ns, e);
        else unmatched_slots_kernel<false><<<kind_grid(t, ns), kKindThreads, 0, s>>>(d, ns, e);
      }
    } else {
      const int64_t members = t->valid_rows + (d.null_group >= 0 ? t->null_rows : 0);
      if (members > 0)
        unmatched_members_kernel<<<kind_grid(t, members), kKindThreads, 0, s>>>(d, members, ns + 1, e);
    }
    if (t->null_rid && t->null_rows > 0)
      null_build_rows_kernel<<<kind_grid(t, t->null_rows), kKindThreads, 0, s>>>(t->null_rid, t->null_rows, e);
  }

  // 4. validity of payload columns whose inputs have no NULLs (NULL padding by row range)
  const unsigned long long* total = dc;
  auto range = [&](uint32_t* words, const unsigned long long* lo, const unsigned long long* hi) {
    if (!words || gs.capacity == 0) return;
    const int64_t nw = (gs.capacity + 31) / 32;
    const int g = (int)std::max<int64_t>(1, std::min<int64_t>((nw + 255) / 256, (int64_t)sm_count(t->device) * 4));
    set_valid_range_kernel<<<g, 256, 0, s>>>(words, lo, hi, gs.capacity);
  };
  for (int c = 0; c < gs.n_build_payload; ++c) {
    const bool nullable = attached ? t->apay_valid[c] != nullptr : gs.build_payload[c].validity != nullptr;
    if (nullable) continue;
    range(gs.out_build_payload[c].validity, nullptr, m);      // INNER rows
    if (full) range(gs.out_build_payload[c].validity, m + 1, total);  // unmatched build rows
  }
  for (int c = 0; full && c < gs.n_probe_payload; ++c) {
    if (gs.probe_payload[c].validity) continue;
    range(gs.out_probe_payload[c].validity, nullptr, m + 1);  // INNER + unmatched probe rows
  }
  SJ_CUDA_TRY(cudaGetLastError());
  return SJ_OK;
}

}  // namespace sj
