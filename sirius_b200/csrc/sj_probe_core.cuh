// What a lookup compares: a bucket as the eight 32-bit words of its sector, and the key in the form its slots
// hold. Everything is 32-bit and one bucket test is short, since the lookups are bound by instructions about
// as much as by the random loads.
#pragma once

#include "sj_device.cuh"

namespace sj {

// What a key is compared with in a bucket: PACKED64 the slot's key field ((key - key_min) << rid_bits,
// the row-id bits masked out), WIDE128 the whole key.
struct SectorKey {
  uint32_t lo, hi;
};

struct Sector {
  uint32_t w[8];
};

__device__ __forceinline__ Sector load_sector(const void* slots, uint32_t b) {
  Sector s;
  asm("ld.global.nc.v8.u32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=r"(s.w[0]), "=r"(s.w[1]), "=r"(s.w[2]), "=r"(s.w[3]), "=r"(s.w[4]), "=r"(s.w[5]), "=r"(s.w[6]), "=r"(s.w[7])
      : "l"(static_cast<const char*>(slots) + (size_t)b * kBucketBytes));
  return s;
}

template <bool WIDE>
struct SectorOps;

template <>
struct SectorOps<false> {
  // rid_bits <= 31, so the key field holds the whole high word. Of each slot, low word ^ key's low word is
  // the row id where the key field matches and more than any row id elsewhere, so the smallest of the four
  // tells both. EMPTY never matches: its key field is all ones and a live one never is.
  __device__ __forceinline__ static bool find(const Sector& s, SectorKey k, uint32_t rid_mask, uint32_t& pos, uint32_t&) {
    uint32_t x[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) x[i] = s.w[2 * i + 1] == k.hi ? s.w[2 * i] ^ k.lo : 0xffffffffu;
    pos = min(min(x[0], x[1]), min(x[2], x[3]));
    return pos <= rid_mask;
  }
  __device__ __forceinline__ static bool find_slot(const Sector& s, SectorKey k, uint32_t rid_mask, uint32_t& q) {
    bool any = false;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const bool m = s.w[2 * i + 1] == k.hi && (s.w[2 * i] ^ k.lo) <= rid_mask;
      q = m ? (uint32_t)i : q;
      any |= m;
    }
    return any;
  }
  __device__ __forceinline__ static bool open(const Sector& s) { return (s.w[6] & s.w[7]) == 0xffffffffu; }
  static constexpr uint32_t kSlots = 4;
};

template <>
struct SectorOps<true> {
  // a live slot's row-id word has high half 0, EMPTY's is all ones
  __device__ __forceinline__ static bool find(const Sector& s, SectorKey k, uint32_t, uint32_t& pos, uint32_t& q) {
    const bool m0 = ((s.w[0] ^ k.lo) | (s.w[1] ^ k.hi) | s.w[3]) == 0;
    const bool m1 = ((s.w[4] ^ k.lo) | (s.w[5] ^ k.hi) | s.w[7]) == 0;
    pos = m0 ? s.w[2] : s.w[6];
    q = m0 ? 0u : 1u;
    return m0 | m1;
  }
  __device__ __forceinline__ static bool find_slot(const Sector& s, SectorKey k, uint32_t rid_mask, uint32_t& q) {
    uint32_t pos;
    return find(s, k, rid_mask, pos, q);
  }
  __device__ __forceinline__ static bool open(const Sector& s) { return s.w[7] != 0; }
  static constexpr uint32_t kSlots = 2;
};

// Key of a probe row; false when it lies outside the build's key range.
template <typename K, bool WIDE>
__device__ __forceinline__ bool sector_key(const TableDev& t, K k, SectorKey& out) {
  const uint64_t kb = key_u64<K>(k);
  bool in;
  uint64_t kn;
  if constexpr (sizeof(K) == 4) {
    const uint32_t n32 = (uint32_t)k - (uint32_t)t.kmin;
    in = n32 <= (uint32_t)t.kmax - (uint32_t)t.kmin;
    kn = n32;
  } else {
    kn = kb - (uint64_t)t.kmin;
    in = kn <= (uint64_t)t.kmax - (uint64_t)t.kmin;
  }
  const uint64_t c = WIDE ? kb : kn << t.rbits;
  out.lo = (uint32_t)c;
  out.hi = (uint32_t)(c >> 32);
  return in;
}

}  // namespace sj
