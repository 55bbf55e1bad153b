// Radix partitioning for the partitioned join variant (tables larger than L2).
//
// Rows are split by the top `pbits` bits of mix64(key) — the same bits that select a key's
// segment of the partitioned hash table — so after partitioning, partition p's probe rows only
// touch table segment p and the build payload rows stored with it. Processing partitions in order
// keeps one segment (a few MB) resident in the 126 MB L2 while its probes stream through, which
// turns the probe's random DRAM accesses (~40 G/s on B200) into L2 hits.
//
// Two passes over the input, both with a fixed grid of G CTAs where CTA c owns the contiguous row
// range [c*chunk, (c+1)*chunk):
//   1. histogram: per-CTA counts of the valid rows of each partition (shared-memory atomics,
//      warp-aggregated with __match_any_sync), stored partition-major as hist[p * G + c];
//   2. an exclusive scan of hist gives every (partition, CTA) its output offset; the scatter pass
//      re-reads the rows tile by tile, counting-sorts each tile by partition in shared memory and
//      writes key, row id and payloads (validity as one byte per row) as contiguous runs.
//      NULL-key rows are dropped (they never match).
// The outputs are partition-major: partition p occupies [off[p*G], off[(p+1)*G]).
#include <algorithm>
#include <type_traits>

#include "sj_partition.cuh"
#include "sj_scan.cuh"
#include "sj_units.cuh"

namespace sj {

constexpr int kPartThreads = 256;
constexpr int kMaxPartBits = kMaxPartitionBits;

__device__ __forceinline__ int partition_of(uint64_t kb, int pbits) {
  return pbits ? (int)(mix64_high(kb) >> (32 - pbits)) : 0;
}

template <typename K>
__device__ __forceinline__ void hist_load4(const K* keys, int64_t i0, int64_t hi, bool vec, K (&k)[4]) {
  if (vec && i0 + 4 <= hi) {
    if (sizeof(K) == 4) {
      const int4 x = __ldcs(reinterpret_cast<const int4*>(keys + i0));
      k[0] = (K)x.x; k[1] = (K)x.y; k[2] = (K)x.z; k[3] = (K)x.w;
    } else {
      const longlong2 x = __ldcs(reinterpret_cast<const longlong2*>(keys + i0));
      const longlong2 y = __ldcs(reinterpret_cast<const longlong2*>(keys + i0) + 1);
      k[0] = (K)x.x; k[1] = (K)x.y; k[2] = (K)y.x; k[3] = (K)y.y;
    }
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j) k[j] = i0 + j < hi ? __ldcs(keys + i0 + j) : (K)0;
  }
}

// Histogram pass: each thread loads 4 groups of 4 consecutive keys (16-byte loads) per step, all
// before counting them, so 8 (int64) or 4 (int32) vector loads per thread are in flight. Whole steps
// of columns without NULLs are counted without a check per row. 64M int64 keys, 64 partitions, two
// CTAs of 1024 threads per SM: 97 us (5.5 TB/s); with a check of every row and the whole 64-bit hash
// 116 us. Eight counters per partition, chosen by lane, changed nothing: not the atomics' conflicts.
template <typename K, int THREADS = kPartThreads>
__global__ void __launch_bounds__(THREADS) part_hist_kernel(PartSrc s, int pbits, int64_t chunk, bool vec,
                                                            int32_t* hist) {
  extern __shared__ int32_t h[];
  constexpr int kGroups = 4;
  constexpr uint32_t kStep = THREADS * 4;
  const int P = 1 << pbits;
  for (int p = threadIdx.x; p < P; p += THREADS) h[p] = 0;
  __syncthreads();
  const int64_t lo = (int64_t)blockIdx.x * chunk;
  const int64_t hi = lo + chunk < s.n ? lo + chunk : s.n;
  const K* keys = static_cast<const K*>(s.keys);
  const bool plain = s.kvalid == nullptr && vec;
  for (int64_t base = lo; base < hi; base += kStep * kGroups) {
    K k[kGroups][4];
    const K* mine = keys + base + threadIdx.x * 4;
    if (plain && base + kStep * kGroups <= hi) {
#pragma unroll
      for (int g = 0; g < kGroups; ++g) hist_load4<K>(mine, g * kStep, (int64_t)kStep * kGroups, true, k[g]);
#pragma unroll
      for (int g = 0; g < kGroups; ++g)
#pragma unroll
        for (int j = 0; j < 4; ++j) atomicAdd(&h[partition_of(key_u64<K>(k[g][j]), pbits)], 1);
      continue;
    }
#pragma unroll
    for (int g = 0; g < kGroups; ++g) hist_load4<K>(keys, base + g * kStep + threadIdx.x * 4, hi, vec, k[g]);
#pragma unroll
    for (int g = 0; g < kGroups; ++g) {
      const int64_t i0 = base + g * kStep + threadIdx.x * 4;
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (i0 + j < hi && bit_valid(s.kvalid, s.kvoff, i0 + j))
          atomicAdd(&h[partition_of(key_u64<K>(k[g][j]), pbits)], 1);
    }
  }
  __syncthreads();
  for (int p = threadIdx.x; p < P; p += THREADS) hist[(int64_t)p * gridDim.x + blockIdx.x] = h[p];
}

// Scatter pass, staged through shared memory one tile of kTile rows at a time: the tile's rows
// are counted per partition, sorted by partition in shared memory (counting sort), and every
// partition's run is then written to its output range with consecutive threads on consecutive
// positions, so each write front advances in whole sectors instead of one row per warp store.
constexpr int kTileRowsPerThread = 8;
constexpr int kTile = kPartThreads * kTileRowsPerThread;

struct ScatterSmem {
  // offsets into the dynamic shared-memory block; payloads stay in the tile's natural row order
  // (loaded together with the keys) and are reached from a sorted slot through `nat`
  size_t cur, tcnt, toff, key, rid, part, nat, pay[kMaxPayload], val[kMaxPayload], total;
};

static ScatterSmem scatter_smem(int pbits, int kw, const PartSrc& s) {
  const size_t P = (size_t)1 << pbits;
  ScatterSmem m{};
  size_t o = 0;
  auto take = [&](size_t b) {
    size_t r = o;
    o += (b + 15) & ~(size_t)15;
    return r;
  };
  m.cur = take(P * 8);
  m.tcnt = take(P * 4);
  m.toff = take(P * 4);
  m.key = take((size_t)kTile * kw);
  m.rid = take((size_t)kTile * 4);
  m.part = take((size_t)kTile * 2);
  m.nat = take((size_t)kTile * 2);
  for (int c = 0; c < s.n_pay; ++c) {
    m.pay[c] = take((size_t)kTile * s.pay[c].width);
    m.val[c] = s.pay[c].valid ? take(kTile) : 0;
  }
  m.total = o;
  return m;
}

// The dynamic shared memory limit of a kernel is one value for the whole process, so each kernel gets the most that
// any call asks of it: with the call's own size, a thread that partitions into fewer parts lowered the limit
// between another thread's set and its launch.
static sj_status allow_smem(const void* kernel, size_t most) {
  SJ_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most));
  return SJ_OK;
}

static size_t most_scatter_smem() {
  PartSrc s{};
  s.n_pay = kMaxPayload;
  static const uint32_t some = 0;
  for (int c = 0; c < kMaxPayload; ++c) s.pay[c] = column_payload(nullptr, &some, 0, 8);
  return scatter_smem(kMaxPartBits, 8, s).total;
}

template <typename K>
__global__ void __launch_bounds__(kPartThreads) part_scatter_kernel(PartSrc s, int pbits, int64_t chunk,
                                                                    const int64_t* __restrict__ off, PartDst d,
                                                                    ScatterSmem m) {
  extern __shared__ __align__(16) unsigned char sm[];
  unsigned long long* cur = reinterpret_cast<unsigned long long*>(sm + m.cur);
  unsigned int* tcnt = reinterpret_cast<unsigned int*>(sm + m.tcnt);
  unsigned int* toff = reinterpret_cast<unsigned int*>(sm + m.toff);
  K* skey = reinterpret_cast<K*>(sm + m.key);
  int32_t* srid = reinterpret_cast<int32_t*>(sm + m.rid);
  uint16_t* spart = reinterpret_cast<uint16_t*>(sm + m.part);
  uint16_t* snat = reinterpret_cast<uint16_t*>(sm + m.nat);
  __shared__ unsigned int s_wsum[kPartThreads / 32];
  const int P = 1 << pbits;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  for (int p = tid; p < P; p += kPartThreads) cur[p] = (unsigned long long)off[(int64_t)p * gridDim.x + blockIdx.x];
  const int64_t lo = (int64_t)blockIdx.x * chunk;
  const int64_t hi = lo + chunk < s.n ? lo + chunk : s.n;
  const K* keys = static_cast<const K*>(s.keys);
  K* okeys = static_cast<K*>(d.keys);
  for (int64_t t0 = lo; t0 < hi; t0 += kTile) {
    for (int p = tid; p < P; p += kPartThreads) tcnt[p] = 0;
    __syncthreads();
    // 1. load rows, partition, rank within the tile's partition
    int pr[kTileRowsPerThread];
    unsigned rank[kTileRowsPerThread];
    K kk[kTileRowsPerThread];
#pragma unroll
    for (int j = 0; j < kTileRowsPerThread; ++j) {
      const int64_t i = t0 + j * kPartThreads + tid;
      pr[j] = -1;
      kk[j] = 0;
      if (i < hi && bit_valid(s.kvalid, s.kvoff, i)) {
        kk[j] = __ldcs(keys + i);
        pr[j] = partition_of(key_u64<K>(kk[j]), pbits);
        const int nat = j * kPartThreads + tid;
        for (int c = 0; c < s.n_pay; ++c) {
          const PayloadIn& in = s.pay[c];
          store_elem(sm + m.pay[c], nat, in.width, load_elem(in.data, i, in.width));
          if (in.valid) sm[m.val[c] + nat] = bit_valid(in.valid, in.voff, i) ? 1 : 0;
        }
      }
      const unsigned peers = __match_any_sync(kFullMask, pr[j]);
      const int leader = __ffs(peers) - 1;
      unsigned base = 0;
      if (pr[j] >= 0 && lane == leader) base = atomicAdd(&tcnt[pr[j]], (unsigned)__popc(peers));
      base = __shfl_sync(kFullMask, base, leader);
      rank[j] = base + __popc(peers & ((1u << lane) - 1));
    }
    __syncthreads();
    // 2. exclusive scan of the tile histogram (P <= 1024 bins, 4 per thread at most)
    constexpr int kBinsPerThread = (1 << kMaxPartitionBits) / kPartThreads;
    unsigned v[kBinsPerThread], acc = 0;
#pragma unroll
    for (int q = 0; q < kBinsPerThread; ++q) {
      const int p = tid * kBinsPerThread + q;
      v[q] = p < P ? tcnt[p] : 0;
      acc += v[q];
    }
    unsigned incl = acc;
#pragma unroll
    for (int dd = 1; dd < 32; dd <<= 1) {
      const unsigned o = __shfl_up_sync(kFullMask, incl, dd);
      if (lane >= dd) incl += o;
    }
    if (lane == 31) s_wsum[wid] = incl;
    __syncthreads();
    unsigned wbase = 0;
    for (int w = 0; w < wid; ++w) wbase += s_wsum[w];
    unsigned run = wbase + incl - acc;
#pragma unroll
    for (int q = 0; q < kBinsPerThread; ++q) {
      const int p = tid * kBinsPerThread + q;
      if (p < P) toff[p] = run;
      run += v[q];
    }
    unsigned tile_valid = 0;
    for (int w = 0; w < kPartThreads / 32; ++w) tile_valid += s_wsum[w];
    __syncthreads();
    // 3. counting-sort the tile into shared memory
#pragma unroll
    for (int j = 0; j < kTileRowsPerThread; ++j) {
      if (pr[j] < 0) continue;
      const int64_t i = t0 + j * kPartThreads + tid;
      const unsigned slot = toff[pr[j]] + rank[j];
      skey[slot] = kk[j];
      srid[slot] = (int32_t)i;
      spart[slot] = (uint16_t)pr[j];
      snat[slot] = (uint16_t)(j * kPartThreads + tid);
    }
    __syncthreads();
    // 4. write the partition runs: consecutive slots of one partition go to consecutive positions
    for (unsigned slot = tid; slot < tile_valid; slot += kPartThreads) {
      const int p = spart[slot];
      const int64_t pos = (int64_t)cur[p] + (slot - toff[p]);
      okeys[pos] = skey[slot];
      *reinterpret_cast<int32_t*>(reinterpret_cast<char*>(d.rid) + pos * (d.stride ? d.stride : 4)) = srid[slot];
      const int nat = snat[slot];
      for (int c = 0; c < s.n_pay; ++c) {
        const int w = s.pay[c].width;
        store_elem(static_cast<char*>(d.pay[c]) + pos * (d.stride ? d.stride : w), 0, w,
                   load_elem_smem(sm + m.pay[c], nat, w));
        if (d.valid8[c]) d.valid8[c][pos * (d.stride ? d.stride : 1)] = sm[m.val[c] + nat];
      }
    }
    __syncthreads();
    for (int p = tid; p < P; p += kPartThreads) cur[p] += tcnt[p];
    __syncthreads();
  }
}

// Scatter pass for plain outputs (no row store) with at most 2 payload columns of 4 or 8 bytes
// without NULLs — the probe side's shape. Each thread holds its 8 rows of a tile (key, payloads)
// in registers, so all 8-24 loads are in flight at once; the tile is ranked and counting-sorted in
// shared memory as above (payloads placed directly at their sorted slot), and the loads of the
// NEXT tile are issued before this tile's runs are written out, so DRAM reads overlap the writes.
constexpr int kFastMaxPay = 2;

struct FastSmem {
  size_t cur, tcnt, toff, key, rid, dst, pay[kFastMaxPay], total;
};

static FastSmem fast_smem(int pbits, int kw, int n_pay) {
  const size_t P = (size_t)1 << pbits;
  FastSmem m{};
  size_t o = 0;
  auto take = [&](size_t b) {
    size_t r = o;
    o += (b + 15) & ~(size_t)15;
    return r;
  };
  m.cur = take(P * 8);
  m.tcnt = take(P * 4);
  m.toff = take(P * 4);
  m.key = take((size_t)kTile * kw);
  m.rid = take((size_t)kTile * 4);
  m.dst = take((size_t)kTile * 4);
  for (int c = 0; c < n_pay; ++c) m.pay[c] = take((size_t)kTile * 8);
  m.total = o;
  return m;
}

bool partition_plain_shape(const PartSrc& s, const PartDst& d);
static bool fast_scatter_ok(const PartSrc& s, const PartDst& d) { return partition_plain_shape(s, d); }
bool partition_plain_shape(const PartSrc& s, const PartDst& d) {
  if (d.stride != 0 || s.n_pay > kFastMaxPay) return false;
  for (int c = 0; c < s.n_pay; ++c)
    if (s.pay[c].valid || s.pay[c].valid8 || (s.pay[c].width != 4 && s.pay[c].width != 8) ||
        s.pay[c].stride != s.pay[c].width || d.valid8[c])
      return false;
  return true;
}

// Row of a tile held by thread t as its j-th row: threads hold consecutive row pairs, so a pair is
// one 16-byte (int64) or 8-byte (int32) vector load when the columns are aligned for it.
__device__ __forceinline__ int64_t fast_row(int64_t t0, int j, int t) {
  return t0 + (int64_t)(j >> 1) * 2 * kPartThreads + 2 * t + (j & 1);
}

template <typename T, typename U>
__device__ __forceinline__ void ld_pair_cs(const T* p, U& a, U& b) {
  if constexpr (sizeof(T) == 8) {
    const ulonglong2 x = __ldcs(reinterpret_cast<const ulonglong2*>(p));
    a = (U)x.x;
    b = (U)x.y;
  } else {
    const uint2 x = __ldcs(reinterpret_cast<const uint2*>(p));
    a = (U)x.x;
    b = (U)x.y;
  }
}

// VEC: the key and payload columns start on a multiple of twice their element width (t0 is even)
template <typename K, int NP, bool VEC>
__device__ __forceinline__ void fast_load_tile(const PartSrc& s, int64_t t0, int64_t hi,
                                               K (&kk)[kTileRowsPerThread],
                                               uint64_t (&pv)[kFastMaxPay][kTileRowsPerThread], uint32_t& live) {
  const K* keys = static_cast<const K*>(s.keys);
  live = 0;
#pragma unroll
  for (int j = 0; j < kTileRowsPerThread; j += 2) {
    const int64_t i = fast_row(t0, j, threadIdx.x);
    kk[j] = kk[j + 1] = 0;
#pragma unroll
    for (int c = 0; c < kFastMaxPay; ++c) pv[c][j] = pv[c][j + 1] = 0;
    if (VEC && i + 1 < hi) {
      ld_pair_cs(keys + i, kk[j], kk[j + 1]);
#pragma unroll
      for (int c = 0; c < NP; ++c) {
        if (s.pay[c].width == 8) {
          ld_pair_cs(static_cast<const unsigned long long*>(s.pay[c].data) + i, pv[c][j], pv[c][j + 1]);
        } else {
          unsigned a, b;
          ld_pair_cs(static_cast<const unsigned int*>(s.pay[c].data) + i, a, b);
          pv[c][j] = a;
          pv[c][j + 1] = b;
        }
      }
    } else {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        if (i + h >= hi) continue;
        kk[j + h] = __ldcs(keys + i + h);
#pragma unroll
        for (int c = 0; c < NP; ++c)
          pv[c][j + h] = s.pay[c].width == 8
                             ? __ldcs(static_cast<const unsigned long long*>(s.pay[c].data) + i + h)
                             : (uint64_t)__ldcs(static_cast<const unsigned int*>(s.pay[c].data) + i + h);
      }
    }
    if (i < hi && bit_valid(s.kvalid, s.kvoff, i)) live |= 1u << j;
    if (i + 1 < hi && bit_valid(s.kvalid, s.kvoff, i + 1)) live |= 1u << (j + 1);
  }
}

// VEC: the source columns take pair loads (fast_load_tile).
template <typename K, int NP, bool VEC = false>
__global__ void __launch_bounds__(kPartThreads, 3) part_scatter_fast_kernel(PartSrc s, int pbits, int64_t chunk,
                                                                         const int64_t* __restrict__ off, PartDst d,
                                                                         FastSmem m) {
  extern __shared__ __align__(16) unsigned char sm[];
  unsigned long long* cur = reinterpret_cast<unsigned long long*>(sm + m.cur);
  unsigned int* tcnt = reinterpret_cast<unsigned int*>(sm + m.tcnt);
  unsigned int* toff = reinterpret_cast<unsigned int*>(sm + m.toff);
  K* skey = reinterpret_cast<K*>(sm + m.key);
  int32_t* srid = reinterpret_cast<int32_t*>(sm + m.rid);
  uint32_t* sdst = reinterpret_cast<uint32_t*>(sm + m.dst);
  __shared__ unsigned int s_wsum[kPartThreads / 32];
  const int P = 1 << pbits;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  for (int p = tid; p < P; p += kPartThreads) cur[p] = (unsigned long long)off[(int64_t)p * gridDim.x + blockIdx.x];
  const int64_t lo = (int64_t)blockIdx.x * chunk;
  const int64_t hi = lo + chunk < s.n ? lo + chunk : s.n;
  K* okeys = static_cast<K*>(d.keys);
  K kk[kTileRowsPerThread];
  uint64_t pv[kFastMaxPay][kTileRowsPerThread];
  uint32_t live = 0;
  if (lo < hi) fast_load_tile<K, NP, VEC>(s, lo, hi, kk, pv, live);
  for (int64_t t0 = lo; t0 < hi; t0 += kTile) {
    for (int p = tid; p < P; p += kPartThreads) tcnt[p] = 0;
    __syncthreads();
    // 1. partition and rank within the tile's partition
    int pr[kTileRowsPerThread];
    unsigned rank[kTileRowsPerThread];
#pragma unroll
    for (int j = 0; j < kTileRowsPerThread; ++j) {
      pr[j] = (live >> j & 1u) ? partition_of(key_u64<K>(kk[j]), pbits) : -1;
      const unsigned peers = __match_any_sync(kFullMask, pr[j]);
      const int leader = __ffs(peers) - 1;
      unsigned base = 0;
      if (pr[j] >= 0 && lane == leader) base = atomicAdd(&tcnt[pr[j]], (unsigned)__popc(peers));
      base = __shfl_sync(kFullMask, base, leader);
      rank[j] = base + __popc(peers & ((1u << lane) - 1));
    }
    __syncthreads();
    // 2. exclusive scan of the tile histogram
    constexpr int kBinsPerThread = (1 << kMaxPartitionBits) / kPartThreads;
    unsigned v[kBinsPerThread], acc = 0;
#pragma unroll
    for (int q = 0; q < kBinsPerThread; ++q) {
      const int p = tid * kBinsPerThread + q;
      v[q] = p < P ? tcnt[p] : 0;
      acc += v[q];
    }
    unsigned incl = acc;
#pragma unroll
    for (int dd = 1; dd < 32; dd <<= 1) {
      const unsigned o = __shfl_up_sync(kFullMask, incl, dd);
      if (lane >= dd) incl += o;
    }
    if (lane == 31) s_wsum[wid] = incl;
    __syncthreads();
    unsigned wbase = 0;
    for (int w = 0; w < wid; ++w) wbase += s_wsum[w];
    unsigned run = wbase + incl - acc;
#pragma unroll
    for (int q = 0; q < kBinsPerThread; ++q) {
      const int p = tid * kBinsPerThread + q;
      if (p < P) toff[p] = run;
      run += v[q];
    }
    unsigned tile_valid = 0;
    for (int w = 0; w < kPartThreads / 32; ++w) tile_valid += s_wsum[w];
    __syncthreads();
    // 3. counting-sort the tile into shared memory (payloads straight to their sorted slot, with
    //    each row's output position, so the write-out reads nothing per partition)
#pragma unroll
    for (int j = 0; j < kTileRowsPerThread; ++j) {
      if (pr[j] < 0) continue;
      const unsigned slot = toff[pr[j]] + rank[j];
      skey[slot] = kk[j];
      srid[slot] = (int32_t)fast_row(t0, j, tid);
      sdst[slot] = (uint32_t)cur[pr[j]] + rank[j];
#pragma unroll
      for (int c = 0; c < NP; ++c) reinterpret_cast<uint64_t*>(sm + m.pay[c])[slot] = pv[c][j];
    }
    __syncthreads();
    // 4. loads of the next tile go out before this tile's write-out
    if (t0 + kTile < hi) fast_load_tile<K, NP, VEC>(s, t0 + kTile, hi, kk, pv, live);
    for (unsigned slot = tid; slot < tile_valid; slot += kPartThreads) {
      const uint32_t pos = sdst[slot];
      okeys[pos] = skey[slot];
      d.rid[pos] = srid[slot];
#pragma unroll
      for (int c = 0; c < NP; ++c) {
        const uint64_t x = reinterpret_cast<const uint64_t*>(sm + m.pay[c])[slot];
        if (s.pay[c].width == 8) static_cast<unsigned long long*>(d.pay[c])[pos] = x;
        else static_cast<unsigned int*>(d.pay[c])[pos] = (unsigned int)x;
      }
    }
    __syncthreads();
    for (int p = tid; p < P; p += kPartThreads) cur[p] += tcnt[p];
    __syncthreads();
  }
}

// The source key and payload columns start on a multiple of twice their element width, so the
// row pairs of fast_load_tile are aligned vector loads (chunks and tiles start on even rows).
static bool pair_aligned_src(const PartSrc& src, int kw) {
  bool ok = ((uintptr_t)src.keys % (2 * kw)) == 0;
  for (int c = 0; c < src.n_pay; ++c) ok = ok && ((uintptr_t)src.pay[c].data % (2 * src.pay[c].width)) == 0;
  return ok;
}

template <typename K>
static sj_status launch_fast_scatter(const PartSrc& src, int pbits, int64_t chunk, const int64_t* offs,
                                     const PartDst& dst, int G, cudaStream_t s) {
  const FastSmem m = fast_smem(pbits, sizeof(K), src.n_pay);
  auto go = [&](auto kernel) -> sj_status {
    SJ_TRY(allow_smem((const void*)kernel, fast_smem(kMaxPartBits, 8, kFastMaxPay).total));
    KernelTimer timer("partition_scatter", s);
    kernel<<<G, kPartThreads, m.total, s>>>(src, pbits, chunk, offs, dst, m);
    return SJ_OK;
  };
  if (pair_aligned_src(src, sizeof(K))) {
    if (src.n_pay == 0) return go(part_scatter_fast_kernel<K, 0, true>);
    if (src.n_pay == 1) return go(part_scatter_fast_kernel<K, 1, true>);
    return go(part_scatter_fast_kernel<K, 2, true>);
  }
  if (src.n_pay == 0) return go(part_scatter_fast_kernel<K, 0>);
  if (src.n_pay == 1) return go(part_scatter_fast_kernel<K, 1>);
  return go(part_scatter_fast_kernel<K, 2>);
}

// Upper bound of the partition grid (scratch sizing); the grid used is never larger.
static int part_grid(int device) { return sm_count(device) * 4; }

static int scatter_per_sm(const PartSrc& src, int key_type, int pbits, bool fast) {
  int r = 0;
  if (fast) {
    const FastSmem m = fast_smem(pbits, key_type == SJ_INT32 ? 4 : 8, src.n_pay);
    const void* k = nullptr;
    if (key_type == SJ_INT32)
      k = src.n_pay == 0 ? (const void*)part_scatter_fast_kernel<int32_t, 0>
          : src.n_pay == 1 ? (const void*)part_scatter_fast_kernel<int32_t, 1>
                           : (const void*)part_scatter_fast_kernel<int32_t, 2>;
    else
      k = src.n_pay == 0 ? (const void*)part_scatter_fast_kernel<int64_t, 0>
          : src.n_pay == 1 ? (const void*)part_scatter_fast_kernel<int64_t, 1>
                           : (const void*)part_scatter_fast_kernel<int64_t, 2>;
    allow_smem(k, fast_smem(kMaxPartBits, 8, kFastMaxPay).total);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&r, k, kPartThreads, m.total);
  } else {
    const ScatterSmem m = scatter_smem(pbits, key_type == SJ_INT32 ? 4 : 8, src);
    const void* k = key_type == SJ_INT32 ? (const void*)part_scatter_kernel<int32_t>
                                         : (const void*)part_scatter_kernel<int64_t>;
    allow_smem(k, most_scatter_smem());
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&r, k, kPartThreads, m.total);
  }
  cudaGetLastError();
  return std::max(1, std::min(4, r));
}

size_t partition_scratch_bytes(int pbits, int device) {
  const size_t PG = ((size_t)1 << pbits) * part_grid(device);
  return ((PG * 4 + 255) & ~(size_t)255) + (((PG + 1) * 8 + 255) & ~(size_t)255) + kScanBlocks * 8 + 256;
}

// Partition `src` into `dst` (arrays of src.n entries each). `scratch` must hold
// partition_scratch_bytes(pbits). On return (stream-ordered), *d_total_out points at the device
// int64 count of rows written and *d_part_off at the partition-major offsets (p * G entries).
sj_status radix_partition(const PartSrc& src, int key_type, int pbits, const PartDst& dst, void* scratch,
                          int device, cudaStream_t s, const int64_t** d_total_out, const int64_t** d_offs_out,
                          int* grid_out) {
  if (pbits < 0 || pbits > kMaxPartBits) return set_error(SJ_ERR_INVALID, "partition bits out of range");
  // Every CTA owns one chunk (no grid-stride loop), so the grid must be resident in one wave:
  // G = SMs x (the scatter kernel's resident CTAs per SM, at most 4).
  const bool fast = fast_scatter_ok(src, dst);
  const int G = sm_count(device) * scatter_per_sm(src, key_type, pbits, fast);
  const int P = 1 << pbits;
  const size_t PG = (size_t)P * G;
  char* base = static_cast<char*>(scratch);
  int32_t* hist = reinterpret_cast<int32_t*>(base);
  int64_t* offs = reinterpret_cast<int64_t*>(base + ((PG * 4 + 255) & ~(size_t)255));
  int64_t* tmp = reinterpret_cast<int64_t*>(base + ((PG * 4 + 255) & ~(size_t)255) + (((PG + 1) * 8 + 255) & ~(size_t)255));
  // chunks start on 4-row boundaries so the histogram can use 16-byte key loads
  const int64_t chunk = std::max<int64_t>(4, ((src.n + G - 1) / G + 3) / 4 * 4);
  const bool vec = ((uintptr_t)src.keys & 15u) == 0;
  {
    KernelTimer timer("partition_hist", s);
    if (key_type == SJ_INT32)
      part_hist_kernel<int32_t><<<G, kPartThreads, P * sizeof(int32_t), s>>>(src, pbits, chunk, vec, hist);
    else
      part_hist_kernel<int64_t><<<G, kPartThreads, P * sizeof(int32_t), s>>>(src, pbits, chunk, vec, hist);
  }
  {
    KernelTimer timer("partition_scan", s);
    device_exclusive_scan<int32_t, int64_t>(hist, offs, nullptr, (int64_t)PG, tmp, s);
  }
  if (fast) {
    SJ_TRY(key_type == SJ_INT32 ? launch_fast_scatter<int32_t>(src, pbits, chunk, offs, dst, G, s)
                                : launch_fast_scatter<int64_t>(src, pbits, chunk, offs, dst, G, s));
    SJ_CUDA_TRY(cudaGetLastError());
    *d_total_out = offs + PG;
    *d_offs_out = offs;
    *grid_out = G;
    return SJ_OK;
  }
  const ScatterSmem m = scatter_smem(pbits, key_type == SJ_INT32 ? 4 : 8, src);
  if (key_type == SJ_INT32) {
    SJ_TRY(allow_smem((const void*)part_scatter_kernel<int32_t>, most_scatter_smem()));
    KernelTimer timer("partition_scatter", s);
    part_scatter_kernel<int32_t><<<G, kPartThreads, m.total, s>>>(src, pbits, chunk, offs, dst, m);
  } else {
    SJ_TRY(allow_smem((const void*)part_scatter_kernel<int64_t>, most_scatter_smem()));
    KernelTimer timer("partition_scatter", s);
    part_scatter_kernel<int64_t><<<G, kPartThreads, m.total, s>>>(src, pbits, chunk, offs, dst, m);
  }
  SJ_CUDA_TRY(cudaGetLastError());
  *d_total_out = offs + PG;
  *d_offs_out = offs;
  *grid_out = G;
  return SJ_OK;
}

// ------------------------------------------------------------------------------------------------
// Column scatter of the partition operator: no row ids and no copy of the partition key are written,
// only the caller's columns (1..8 bytes wide, any number). A tile of kColTile rows is ranked by
// partition once (shared-memory atomics) and its output positions are kept sorted in shared memory;
// each column then goes through one staging buffer: placed at the rows' sorted slots, written out in
// partition runs with consecutive threads on consecutive positions. The loads of the next column (or
// of the next tile's keys) are in registers before a column is written, so reads overlap writes. The
// key column, when the caller wants it reordered too, is staged from the registers it was hashed in.
// 4096-row tiles: a run holds 4096 / P rows, twice the length of the 2048-row tiles above. 64M int64 keys
// and one int64 column into 64 partitions: 1,114 us with row ids and a key copy written by
// part_scatter_fast_kernel, 502 us here (4.3 TB/s of 2.1 GB). While it took 514 us, other shapes of threads
// x rows x CTAs per SM took 542 (256x8x4), 541 (512x4x3), 524 (256x16x2) and 526 us (1024x4x2). It is bound
// by its write fronts, P per CTA, that advance by one run of a tile at a time.
// ------------------------------------------------------------------------------------------------
constexpr int kColThreads = 512;
constexpr int kColRows = 8;      // rows per thread
constexpr int kColCtasPerSm = 2;
constexpr int kColHistThreads = 1024;
constexpr int kColTile = kColThreads * kColRows;

// Row of a tile that thread t holds as its j-th: consecutive row pairs, as fast_row.
__device__ __forceinline__ int col_row(int j, int t) { return (j >> 1) * 2 * kColThreads + 2 * t + (j & 1); }

template <typename T>
__device__ __forceinline__ void col_load_t(const T* src, bool pairs, uint32_t t0, uint32_t hi, uint64_t (&v)[kColRows]) {
#pragma unroll
  for (int j = 0; j < kColRows; j += 2) {
    const uint32_t i = t0 + col_row(j, threadIdx.x);
    v[j] = v[j + 1] = 0;
    if constexpr (sizeof(T) >= 4) {
      if (pairs && i + 1 < hi) {
        ld_pair_cs(src + i, v[j], v[j + 1]);
        continue;
      }
    }
    if (i < hi) v[j] = (uint64_t)__ldcs(src + i);
    if (i + 1 < hi) v[j + 1] = (uint64_t)__ldcs(src + i + 1);
  }
}

__device__ __forceinline__ void col_load(const PartColumn& c, uint32_t t0, uint32_t hi, uint64_t (&v)[kColRows]) {
  if (c.bits) {
#pragma unroll
    for (int j = 0; j < kColRows; ++j) {
      const uint32_t i = t0 + col_row(j, threadIdx.x);
      v[j] = i < hi && bit_valid(c.bits, c.voff, i) ? 1 : 0;
    }
    return;
  }
  switch (c.width) {
    case 8: return col_load_t(static_cast<const unsigned long long*>(c.src), c.pairs, t0, hi, v);
    case 4: return col_load_t(static_cast<const unsigned int*>(c.src), c.pairs, t0, hi, v);
    case 2: return col_load_t(static_cast<const unsigned short*>(c.src), false, t0, hi, v);
    default: return col_load_t(static_cast<const unsigned char*>(c.src), false, t0, hi, v);
  }
}

template <typename T>
__device__ __forceinline__ void col_stage(void* stage, int tile_n, const uint16_t (&slot)[kColRows],
                                          const uint64_t (&v)[kColRows]) {
#pragma unroll
  for (int j = 0; j < kColRows; ++j)
    if (col_row(j, threadIdx.x) < tile_n) static_cast<T*>(stage)[slot[j]] = (T)v[j];
}

template <typename T>
__device__ __forceinline__ void col_write(const void* stage, const uint32_t* sdst, void* dst, int tile_n) {
#pragma unroll
  for (int q = 0; q < kColRows; ++q) {
    const int s = q * kColThreads + threadIdx.x;
    if (s < tile_n) static_cast<T*>(dst)[sdst[s]] = static_cast<const T*>(stage)[s];
  }
}

// At least one column.
template <typename K>
__global__ void __launch_bounds__(kColThreads, kColCtasPerSm) part_columns_kernel(const K* __restrict__ keys, bool key_pairs,
                                                                      uint32_t n, int pbits, uint32_t chunk,
                                                                      const int64_t* __restrict__ off, PartColumns cols) {
  using U = std::conditional_t<sizeof(K) == 8, unsigned long long, unsigned int>;
  __shared__ __align__(16) unsigned char stage[kColTile * 8];
  __shared__ unsigned int s_wsum[kColThreads / 32];
  extern __shared__ uint32_t s_col[];
  const int P = 1 << pbits;
  uint32_t* sdst = s_col;              // output position of each sorted slot
  uint32_t* cur = sdst + kColTile;     // next output position of each partition
  uint32_t* gbase = cur + P;           // output position of a row = gbase[its partition] + its sorted slot
  uint32_t* tcnt = gbase + P;          // the tile's rows of each partition
  uint32_t* tbase = tcnt + P;          // their first sorted slot
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  for (int p = tid; p < P; p += kColThreads) {
    cur[p] = (uint32_t)off[(int64_t)p * gridDim.x + blockIdx.x];
    tcnt[p] = 0;
  }
  const uint32_t lo = min(n, blockIdx.x * chunk), hi = min(n, lo + chunk);
  uint64_t v[kColRows];
  const U* ukeys = reinterpret_cast<const U*>(keys);
  if (lo < hi) col_load_t(ukeys, key_pairs, lo, hi, v);
  __syncthreads();
  for (uint32_t t0 = lo; t0 < hi; t0 += kColTile) {
    const int tile_n = (int)(hi - t0 < kColTile ? hi - t0 : kColTile);
    // 1. rank every row within its partition
    uint32_t pr[kColRows];  // partition << 16 | rank
#pragma unroll
    for (int j = 0; j < kColRows; ++j) {
      if (col_row(j, tid) >= tile_n) continue;
      const uint32_t p = (uint32_t)partition_of(key_u64<K>((K)v[j]), pbits);
      pr[j] = p << 16 | atomicAdd(&tcnt[p], 1u);
    }
    __syncthreads();
    // 2. exclusive scan of the tile's counts
    constexpr int kBins = (1 << kMaxPartBits) / kColThreads;
    uint32_t c[kBins], acc = 0;
#pragma unroll
    for (int q = 0; q < kBins; ++q) {
      const int p = tid * kBins + q;
      c[q] = p < P ? tcnt[p] : 0;
      acc += c[q];
    }
    uint32_t incl = warp_inclusive_sum(acc);
    if (lane == 31) s_wsum[wid] = incl;
    __syncthreads();
    uint32_t run = incl - acc;
    for (int w = 0; w < wid; ++w) run += s_wsum[w];
#pragma unroll
    for (int q = 0; q < kBins; ++q) {
      const int p = tid * kBins + q;
      if (p < P) {
        tbase[p] = run;
        tcnt[p] = 0;
        gbase[p] = cur[p] - run;
        cur[p] += c[q];
      }
      run += c[q];
    }
    __syncthreads();
    // 3. the rows' sorted slots and the slots' output positions
    uint16_t slot[kColRows];
#pragma unroll
    for (int j = 0; j < kColRows; ++j) {
      slot[j] = 0;
      if (col_row(j, tid) >= tile_n) continue;
      const uint32_t p = pr[j] >> 16;
      slot[j] = (uint16_t)(tbase[p] + (pr[j] & 0xffffu));
      sdst[slot[j]] = gbase[p] + slot[j];
    }
    __syncthreads();
    // 4. column by column (the key column, if wanted, comes first and is already in registers)
    const uint32_t t1 = t0 + kColTile;
    if (!cols.c[0].is_key) col_load(cols.c[0], t0, hi, v);
    for (int q = 0; q < cols.n; ++q) {
      const PartColumn& col = cols.c[q];
      switch (col.width) {
        case 8: col_stage<unsigned long long>(stage, tile_n, slot, v); break;
        case 4: col_stage<unsigned int>(stage, tile_n, slot, v); break;
        case 2: col_stage<unsigned short>(stage, tile_n, slot, v); break;
        default: col_stage<unsigned char>(stage, tile_n, slot, v); break;
      }
      __syncthreads();
      if (q + 1 < cols.n) col_load(cols.c[q + 1], t0, hi, v);
      else if (t1 < hi) col_load_t(ukeys, key_pairs, t1, hi, v);
      switch (col.width) {
        case 8: col_write<unsigned long long>(stage, sdst, col.dst, tile_n); break;
        case 4: col_write<unsigned int>(stage, sdst, col.dst, tile_n); break;
        case 2: col_write<unsigned short>(stage, sdst, col.dst, tile_n); break;
        default: col_write<unsigned char>(stage, sdst, col.dst, tile_n); break;
      }
      __syncthreads();
    }
  }
}

static size_t columns_smem(int pbits) {
  return ((size_t)kColTile + 4 * ((size_t)1 << pbits)) * sizeof(uint32_t);
}

sj_status partition_columns(const void* keys, int key_type, int64_t n, int pbits, const PartColumns& cols, void* scratch,
                            int device, cudaStream_t s, const int64_t** d_total_out, const int64_t** d_offs_out,
                            int* grid_out) {
  if (pbits < 0 || pbits > kMaxPartBits) return set_error(SJ_ERR_INVALID, "partition bits out of range");
  // one chunk per CTA, all resident, and none for less than a tile (25K rows: 7 CTAs, not 296)
  const int G = (int)std::max<int64_t>(1, std::min<int64_t>((n + kColTile - 1) / kColTile, (int64_t)sm_count(device) * kColCtasPerSm));
  const int P = 1 << pbits;
  const size_t PG = (size_t)P * G;
  char* base = static_cast<char*>(scratch);
  int32_t* hist = reinterpret_cast<int32_t*>(base);
  int64_t* offs = reinterpret_cast<int64_t*>(base + ((PG * 4 + 255) & ~(size_t)255));
  int64_t* tmp = reinterpret_cast<int64_t*>(base + ((PG * 4 + 255) & ~(size_t)255) + (((PG + 1) * 8 + 255) & ~(size_t)255));
  const int64_t chunk = std::max<int64_t>(4, ((n + G - 1) / G + 3) / 4 * 4);
  const int kw = key_type == SJ_INT32 ? 4 : 8;
  const bool vec = ((uintptr_t)keys & 15u) == 0, key_pairs = ((uintptr_t)keys % (2 * kw)) == 0;
  PartSrc src{};
  src.keys = keys;
  src.n = n;
  {
    KernelTimer timer("partition_hist", s);
    if (key_type == SJ_INT32)
      part_hist_kernel<int32_t, kColHistThreads><<<G, kColHistThreads, P * sizeof(int32_t), s>>>(src, pbits, chunk, vec, hist);
    else
      part_hist_kernel<int64_t, kColHistThreads><<<G, kColHistThreads, P * sizeof(int32_t), s>>>(src, pbits, chunk, vec, hist);
  }
  {
    KernelTimer timer("partition_scan", s);
    device_exclusive_scan<int32_t, int64_t>(hist, offs, nullptr, (int64_t)PG, tmp, s);
  }
  auto go = [&](auto k) -> sj_status {
    using K = decltype(k);
    const size_t smem = columns_smem(pbits);
    SJ_TRY(allow_smem((const void*)part_columns_kernel<K>, columns_smem(kMaxPartBits)));
    KernelTimer timer("partition_scatter", s);
    part_columns_kernel<K><<<G, kColThreads, smem, s>>>(static_cast<const K*>(keys), key_pairs, (uint32_t)n, pbits, (uint32_t)chunk, offs, cols);
    return SJ_OK;
  };
  if (cols.n > 0 && n > 0) SJ_TRY(key_type == SJ_INT32 ? go(int32_t{}) : go(int64_t{}));
  SJ_CUDA_TRY(cudaGetLastError());
  *d_total_out = offs + PG;
  *d_offs_out = offs;
  *grid_out = G;
  return SJ_OK;
}

// ------------------------------------------------------------------------------------------------
// Tile-local partition (the probe side): every tile of kColTile rows is sorted by partition and written
// back to its own rows, one column at a time through the staging buffer, in 16-byte pieces; its runs go to
// runs.off / runs.cnt[p * tiles + tile]. Rows that match nothing, those with a NULL key or one outside [kmin, kmax],
// are dropped: they are not written and the probe does not read them. No histogram, no scan, no write fronts.
// 64M int64 keys and one 8-byte payload, 16 partitions: 446 us, and the probe reads runs twice as long as with
// 2048-row tiles staged whole (479 us; unit probe 1,361 -> 1,300 us). A row's partition, then its slot, then the
// mark of a row that was dropped share a register: with a mask and a slot of their own 16 bytes spilled, and the test
// of the range took 465 us instead of 446 (454 without the test).
// ------------------------------------------------------------------------------------------------
__device__ __forceinline__ void stage_copy(const unsigned char* stage, void* dst, size_t at, uint32_t bytes) {
  uint4* d = reinterpret_cast<uint4*>(static_cast<char*>(dst) + at);
  const uint4* s = reinterpret_cast<const uint4*>(stage);
  for (uint32_t q = threadIdx.x; q < (bytes + 15) / 16; q += kColThreads) d[q] = s[q];
}

template <typename K>
__global__ void __launch_bounds__(kColThreads, kColCtasPerSm) part_local_kernel(const K* __restrict__ keys, bool key_pairs,
                                                                                const uint32_t* __restrict__ kvalid,
                                                                                int64_t kvoff, uint32_t n, int pbits,
                                                                                uint32_t n_tiles, std::make_unsigned_t<K> kmin,
                                                                                std::make_unsigned_t<K> span, K* okeys,
                                                                                int32_t* orid, PartColumns cols,
                                                                                LocalRuns runs) {
  if (!gate_open(runs.gate)) return;
  using U = std::conditional_t<sizeof(K) == 8, unsigned long long, unsigned int>;
  __shared__ __align__(16) unsigned char stage[kColTile * 8];
  __shared__ uint32_t s_wsum[kColThreads / 32], tcnt[1 << kMaxPartBits], tbase[1 << kMaxPartBits];
  const int P = 1 << pbits;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  for (int p = tid; p < P; p += kColThreads) tcnt[p] = 0;
  const U* ukeys = reinterpret_cast<const U*>(keys);
  uint64_t v[kColRows];
  uint32_t tile = blockIdx.x;
  if (tile < n_tiles) col_load_t(ukeys, key_pairs, tile * kColTile, n, v);
  __syncthreads();
  for (; tile < n_tiles; tile += gridDim.x) {
    const uint32_t t0 = tile * kColTile;
    const int tile_n = (int)min(n - t0, (uint32_t)kColTile);
    if (runs.zero_bits && tid * 32 < tile_n) runs.zero_bits[t0 / 32 + tid] = 0;
    // 1. rank every row that may match within its partition
    uint32_t pr[kColRows];  // partition << 16 | rank, ~0 for the others
#pragma unroll
    for (int j = 0; j < kColRows; ++j) {
      const int r = col_row(j, tid);
      pr[j] = 0xffffffffu;
      const bool in = (std::make_unsigned_t<K>)((std::make_unsigned_t<K>)v[j] - kmin) <= span;
      if (!(in & (r < tile_n)) || !bit_valid(kvalid, kvoff, (int64_t)t0 + r)) continue;
      const uint32_t p = (uint32_t)partition_of(key_u64<K>((K)v[j]), pbits);
      pr[j] = p << 16 | atomicAdd(&tcnt[p], 1u);
    }
    __syncthreads();
    // 2. exclusive scan of the tile's counts: the runs
    constexpr int kBins = (1 << kMaxPartBits) / kColThreads;
    uint32_t c[kBins], acc = 0;
#pragma unroll
    for (int q = 0; q < kBins; ++q) {
      const int p = tid * kBins + q;
      c[q] = p < P ? tcnt[p] : 0;
      acc += c[q];
    }
    const uint32_t incl = warp_inclusive_sum(acc);
    if (lane == 31) s_wsum[wid] = incl;
    __syncthreads();
    uint32_t run = incl - acc, valid = 0;
    for (int w = 0; w < kColThreads / 32; ++w) {
      run += w < wid ? s_wsum[w] : 0;
      valid += s_wsum[w];
    }
#pragma unroll
    for (int q = 0; q < kBins; ++q) {
      const int p = tid * kBins + q;
      if (p < P) {
        tbase[p] = run;
        tcnt[p] = 0;
        runs.off[(size_t)p * n_tiles + tile] = (int32_t)(t0 + run);
        runs.cnt[(size_t)p * n_tiles + tile] = (int32_t)c[q];
      }
      run += c[q];
    }
    __syncthreads();
    // 3. the keys, the payloads, the row ids
#pragma unroll
    for (int j = 0; j < kColRows; ++j) {
      if (pr[j] == 0xffffffffu) continue;
      pr[j] = tbase[pr[j] >> 16] + (pr[j] & 0xffffu);  // the sorted slot
      reinterpret_cast<K*>(stage)[pr[j]] = (K)v[j];
    }
    __syncthreads();
    auto next = [&](int q) {
      if (q < cols.n) col_load(cols.c[q], t0, n, v);
      else if (tile + gridDim.x < n_tiles) col_load_t(ukeys, key_pairs, (tile + gridDim.x) * kColTile, n, v);
    };
    next(0);
    stage_copy(stage, okeys, (size_t)t0 * sizeof(K), valid * (uint32_t)sizeof(K));
    __syncthreads();
    for (int q = 0; q < cols.n; ++q) {
      const int w = cols.c[q].width;
      if (w == 8) {
#pragma unroll
        for (int j = 0; j < kColRows; ++j)
          if (pr[j] < kColTile) reinterpret_cast<uint64_t*>(stage)[pr[j]] = v[j];
      } else {
#pragma unroll
        for (int j = 0; j < kColRows; ++j)
          if (pr[j] < kColTile) reinterpret_cast<uint32_t*>(stage)[pr[j]] = (uint32_t)v[j];
      }
      __syncthreads();
      next(q + 1);
      stage_copy(stage, cols.c[q].dst, (size_t)t0 * w, valid * w);
      __syncthreads();
    }
#pragma unroll
    for (int j = 0; j < kColRows; ++j)
      if (pr[j] < kColTile) reinterpret_cast<uint32_t*>(stage)[pr[j]] = t0 + col_row(j, tid);
    __syncthreads();
    stage_copy(stage, orid, (size_t)t0 * 4, valid * 4);
    __syncthreads();
  }
}

// The outputs start on 16 bytes and have room for whole 16-byte pieces.
sj_status local_partition(const PartSrc& src, int key_type, int pbits, int64_t kmin, int64_t kmax, const PartDst& dst,
                          const LocalRuns& runs, int device, cudaStream_t s) {
  if (!partition_plain_shape(src, dst)) return set_error(SJ_ERR_INVALID, "tile-local partition needs the plain shape");
  if (src.n == 0) return SJ_OK;
  static_assert(kColTile == kPartTileRows, "tile of the run tables");
  const uint32_t tiles = (uint32_t)((src.n + kColTile - 1) / kColTile);
  const int grid = (int)std::min<int64_t>(tiles, (int64_t)sm_count(device) * kColCtasPerSm);
  PartColumns cols{};
  for (int c = 0; c < src.n_pay; ++c)
    cols.c[cols.n++] = PartColumn{src.pay[c].data, nullptr, 0, dst.pay[c], src.pay[c].width, 0,
                                  (int16_t)((uintptr_t)src.pay[c].data % (2 * src.pay[c].width) == 0)};
  auto go = [&](auto k) {
    using K = decltype(k);
    using UK = std::make_unsigned_t<K>;
    KernelTimer timer("partition_scatter", s);
    part_local_kernel<K><<<grid, kColThreads, 0, s>>>(static_cast<const K*>(src.keys), (uintptr_t)src.keys % (2 * sizeof(K)) == 0,
                                                      src.kvalid, src.kvoff, (uint32_t)src.n, pbits, tiles, (UK)kmin, (UK)((UK)kmax - (UK)kmin),
                                                      static_cast<K*>(dst.keys), dst.rid, cols, runs);
  };
  if (key_type == SJ_INT32) go(int32_t{});
  else go(int64_t{});
  SJ_CUDA_TRY(cudaGetLastError());
  return SJ_OK;
}

}  // namespace sj
