// Which DISTINCT probe serves a gather, and the TMA-staged one. Outputs of plain columns go to the unit
// probe (sj_probe_units.cu):
//   build side: row ids plus up to 3 build payloads, either the fields of the table's row store (one
//               record per match) or plain 4/8-byte columns without NULLs gathered by row id;
//   probe side: row ids plus up to 2 plain 4/8-byte payload columns without NULLs.
// Other shapes (NULL payloads, 1/2-byte payloads, more columns) take the staged write-out kernel in
// sj_probe.cu.
#include <algorithm>

#include "sj_bulk.cuh"
#include "sj_device.cuh"
#include "sj_internal.h"
#include "sj_probe_direct.h"
#include "sj_probe_units.h"

namespace sj {

TableDev table_dev(const sj_table* t);

constexpr int kDirectThreads = 64;  // 2 warps: the reservation barriers wait on one other warp only
constexpr int kDirectWarps = kDirectThreads / 32;

__device__ __forceinline__ uint64_t ld_cs_w(const void* base, int64_t i, int w) {
  return w == 8 ? __ldcs(reinterpret_cast<const unsigned long long*>(base) + i)
                : (uint64_t)__ldcs(reinterpret_cast<const unsigned int*>(base) + i);
}
__device__ __forceinline__ uint64_t ld_nc_w(const void* a, int w) {
  return w == 8 ? __ldg(reinterpret_cast<const unsigned long long*>(a))
                : (uint64_t)__ldg(reinterpret_cast<const unsigned int*>(a));
}
__device__ __forceinline__ void st_cs_w(void* base, int64_t i, int w, uint64_t v) {
  if (w == 8) __stcs(reinterpret_cast<unsigned long long*>(base) + i, (unsigned long long)v);
  else __stcs(reinterpret_cast<unsigned int*>(base) + i, (unsigned int)v);
}

// One row-store record of 8, 16 or 32 bytes (the stride) in one load.
__device__ __forceinline__ void load_rec(const void* p, int stride, uint32_t (&w)[8]) {
  if (stride == 32) {
    asm("ld.global.nc.v8.u32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]), "=r"(w[4]), "=r"(w[5]), "=r"(w[6]), "=r"(w[7])
        : "l"(p));
  } else if (stride == 16) {
    const uint4 x = __ldg(reinterpret_cast<const uint4*>(p));
    w[0] = x.x; w[1] = x.y; w[2] = x.z; w[3] = x.w;
    w[4] = w[5] = w[6] = w[7] = 0;
  } else {
    const uint2 x = __ldg(reinterpret_cast<const uint2*>(p));
    w[0] = x.x; w[1] = x.y;
    w[2] = w[3] = w[4] = w[5] = w[6] = w[7] = 0;
  }
}

// ------------------------------------------------------------------------------------------------
// The probe with its streaming inputs staged by the TMA engine (opt-in). The probe rows of a tile
// (keys, partition row ids, probe payloads: contiguous ranges) are bulk-copied into a 3-stage
// shared-memory ring two tiles ahead of their use, so no lane waits on DRAM for them and no
// register holds them in flight; the lanes only wait on the table (bucket, then record) in L2.
// Stage of iteration i: i % 3; tile i+2 is issued right after iteration i's first CTA barrier,
// which every reader of that stage (iteration i-1) has passed. Only full tiles are staged; the
// last, partial tile of the probe reads global memory directly. A bounded mbarrier wait that runs
// out makes the whole CTA stop after its next barrier and marks the count negative (bit 63).
// ------------------------------------------------------------------------------------------------
constexpr int kTmaR = 2;
constexpr int kTmaTile = kDirectThreads * kTmaR;
constexpr int kTmaStages = 3;

struct TmaStage {
  int32_t key_off, rid_off, pay_off[kDirectMaxProbePayload], bytes;  // within a stage
};

template <typename K>
__host__ __device__ inline TmaStage tma_stage(const DirectArgs& a) {
  TmaStage st{};
  int o = 0;
  st.key_off = o;
  o += kTmaTile * (int)sizeof(K);
  st.rid_off = o;
  if (a.prid_map) o += kTmaTile * 4;
  for (int c = 0; c < kDirectMaxProbePayload; ++c) {
    st.pay_off[c] = o;
    if (c < a.n_pin) o += kTmaTile * a.pin_w[c];
  }
  st.bytes = (o + 127) & ~127;
  return st;
}

template <typename K, bool WIDE>
__global__ void __launch_bounds__(kDirectThreads, 4)
    probe_tma_kernel(TableDev t, const K* __restrict__ keys, const uint32_t* __restrict__ kv, int64_t kvoff,
                     int64_t n_host, const int64_t* d_n, DirectArgs a, TmaStage st) {
  using Ops = SlotOps<WIDE>;
  const uint64_t pol = a.l2_last ? l2_policy_evict_last() : 0ull;  // table loads' L2 policy
  constexpr int R = kTmaR;
  extern __shared__ __align__(128) unsigned char s_ring[];
  __shared__ __align__(8) uint64_t s_bar[kTmaStages];
  __shared__ unsigned s_wtot[kDirectWarps];
  __shared__ unsigned long long s_wbase[kDirectWarps];
  __shared__ int s_abort;
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const unsigned below = (1u << lane) - 1u;
  const int64_t n = d_n ? *d_n : n_host;
  const int64_t tiles = (n + kTmaTile - 1) / kTmaTile;
  const int64_t full_tiles = n / kTmaTile;
  const uint64_t kmask = ~((1ull << t.rbits) - 1);
  const int li = warp * (32 * R) + lane;  // row of group j inside a tile: li + 32 j

  auto issue = [&](int64_t tt, int sidx) {  // thread 0; tt < full_tiles
    unsigned char* sb = s_ring + sidx * st.bytes;
    uint32_t bytes = kTmaTile * (uint32_t)sizeof(K);
    if (a.prid_map) bytes += kTmaTile * 4;
    for (int c = 0; c < a.n_pin; ++c) bytes += kTmaTile * a.pin_w[c];
    mbar_arrive_expect_tx(&s_bar[sidx], bytes);
    bulk_copy_g2s(sb + st.key_off, keys + tt * kTmaTile, kTmaTile * sizeof(K), &s_bar[sidx]);
    if (a.prid_map) bulk_copy_g2s(sb + st.rid_off, a.prid_map + tt * kTmaTile, kTmaTile * 4, &s_bar[sidx]);
    for (int c = 0; c < a.n_pin; ++c)
      bulk_copy_g2s(sb + st.pay_off[c], static_cast<const char*>(a.pin[c]) + tt * kTmaTile * a.pin_w[c],
                    kTmaTile * a.pin_w[c], &s_bar[sidx]);
  };

  if (threadIdx.x == 0) {
    for (int q = 0; q < kTmaStages; ++q) mbar_init(&s_bar[q], 1);
    mbar_init_fence();
    s_abort = 0;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    if (blockIdx.x < full_tiles) issue(blockIdx.x, 0);
    if (blockIdx.x + gridDim.x < full_tiles) issue(blockIdx.x + gridDim.x, 1);
  }
  int it = 0;
  for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x, ++it) {
    const int sidx = it % kTmaStages;
    const unsigned char* sb = s_ring + sidx * st.bytes;
    const bool staged = tile < full_tiles;
    const int64_t r0 = tile * kTmaTile + li;
    bool ok = true;
    if (staged) ok = mbar_wait_bounded(&s_bar[sidx], (uint32_t)((it / kTmaStages) & 1), kBulkWaitPolls);
    K k[R];
#pragma unroll
    for (int j = 0; j < R; ++j) {
      const int64_t r = r0 + 32 * j;
      if (staged) k[j] = reinterpret_cast<const K*>(sb + st.key_off)[li + 32 * j];
      else k[j] = r < n ? __ldcs(keys + r) : (K)0;
    }
    uint32_t act = 0;
#pragma unroll
    for (int j = 0; j < R; ++j) {
      const int64_t r = r0 + 32 * j;
      if (ok && r < n && bit_valid(kv, kvoff, r) && in_range(t, k[j])) act |= 1u << j;
    }
    if (!ok) s_abort = 1;
    uint32_t b[R];
    uint64_t ks[R];
#pragma unroll
    for (int j = 0; j < R; ++j) {
      const uint64_t kb = key_u64<K>(k[j]);
      b[j] = home_bucket(t, kb);
      ks[j] = Ops::probe_key((uint64_t)(long long)k[j] - (uint64_t)t.kmin, kb, t.rbits);
    }
    int32_t pos[R];
    uint32_t hit = 0;
#pragma unroll
    for (int j = 0; j < R; ++j) pos[j] = 0;
    for (uint32_t step = 0; act && step <= t.segmask; ++step) {
      Bucket bk[R];
#pragma unroll
      for (int j = 0; j < R; ++j)
        if (act >> j & 1u) bk[j] = a.l2_last ? load_bucket_hint(t.slots, b[j], pol) : load_bucket<true>(t.slots, b[j]);
#pragma unroll
      for (int j = 0; j < R; ++j) {
        if (!(act >> j & 1u)) continue;
        int32_t pj;
        const bool m = Ops::match_distinct(bk[j], ks[j], kmask, t.rbits, pj);
        if (m) {
          pos[j] = pj;
          hit |= 1u << j;
        }
        if (m || Ops::open(bk[j])) act &= ~(1u << j);
        else b[j] = next_bucket(b[j], t.segmask);
      }
    }
    // build-side gather loads (the probe-side values stay in the stage until the stores)
    int32_t brid[R];
    uint64_t bv[kDirectMaxBuildPayload][R];
#pragma unroll
    for (int j = 0; j < R; ++j) {
      brid[j] = 0;
#pragma unroll
      for (int c = 0; c < kDirectMaxBuildPayload; ++c) bv[c][j] = 0;
      if (!(hit >> j & 1u)) continue;
      if (a.rec) {
        uint32_t w[8];
        load_rec(static_cast<const char*>(a.rec) + (int64_t)pos[j] * a.rec_stride, a.rec_stride, w);
        brid[j] = (int32_t)w[0];
#pragma unroll
        for (int c = 0; c < kDirectMaxBuildPayload; ++c) bv[c][j] = ((uint64_t)w[3 + 2 * c] << 32) | w[2 + 2 * c];
      } else {
        brid[j] = a.brid_map ? __ldg(reinterpret_cast<const int32_t*>(reinterpret_cast<const char*>(a.brid_map) +
                                                                       (int64_t)pos[j] * a.brid_stride))
                             : pos[j];
#pragma unroll
        for (int c = 0; c < kDirectMaxBuildPayload; ++c) {
          if (c < a.n_bin) {
            const int64_t i = a.bin_by_pos ? pos[j] : brid[j];
            bv[c][j] = ld_nc_w(static_cast<const char*>(a.bin[c]) + i * a.bin_stride[c], a.bin_w[c]);
          }
        }
      }
    }
    unsigned bal[R];
    unsigned wtot = 0;
#pragma unroll
    for (int j = 0; j < R; ++j) {
      bal[j] = __ballot_sync(kFullMask, (hit >> j) & 1u);
      wtot += __popc(bal[j]);
    }
    // CTA reservation; the first barrier also frees stage (it + 2) % 3 for tile it + 2
    if (lane == 0) s_wtot[warp] = wtot;
    __syncthreads();
    if (s_abort) break;
    if (threadIdx.x == 0) {
      const int64_t t2 = tile + 2 * (int64_t)gridDim.x;
      if (t2 < full_tiles) issue(t2, (it + 2) % kTmaStages);
    }
    if (warp == 0) {
      const unsigned v = lane < kDirectWarps ? s_wtot[lane] : 0u;
      unsigned incl = v;
#pragma unroll
      for (int d = 1; d < kDirectWarps; d <<= 1) {
        const unsigned o = __shfl_up_sync(kFullMask, incl, d);
        if (lane >= d) incl += o;
      }
      const unsigned tot = __shfl_sync(kFullMask, incl, kDirectWarps - 1);
      unsigned long long cb = 0;
      if (lane == 0 && tot) cb = atomicAdd(a.d_count, (unsigned long long)tot);
      cb = __shfl_sync(kFullMask, cb, 0);
      if (lane < kDirectWarps) s_wbase[lane] = cb + (incl - v);
    }
    __syncthreads();
    if (wtot == 0) continue;
    const unsigned long long base = s_wbase[warp];
    unsigned run = 0;
#pragma unroll
    for (int j = 0; j < R; ++j) {
      const int64_t p = (int64_t)(base + run + __popc(bal[j] & below));
      run += __popc(bal[j]);
      if (!(hit >> j & 1u) || p >= a.capacity) continue;
      const int64_t r = r0 + 32 * j;
      const int i = li + 32 * j;
      if (a.out_prid) {
        int32_t pr;
        if (!a.prid_map) pr = (int32_t)r;
        else if (staged) pr = reinterpret_cast<const int32_t*>(sb + st.rid_off)[i];
        else pr = __ldcs(a.prid_map + r);
        __stcs(a.out_prid + p, pr);
      }
      if (a.out_brid) __stcs(a.out_brid + p, brid[j]);
#pragma unroll
      for (int c = 0; c < kDirectMaxProbePayload; ++c) {
        if (c < a.n_pin) {
          uint64_t v;
          if (staged) v = a.pin_w[c] == 8 ? reinterpret_cast<const uint64_t*>(sb + st.pay_off[c])[i]
                                          : reinterpret_cast<const uint32_t*>(sb + st.pay_off[c])[i];
          else v = ld_cs_w(a.pin[c], r, a.pin_w[c]);
          st_cs_w(a.pout[c], p, a.pin_w[c], v);
        }
      }
#pragma unroll
      for (int c = 0; c < kDirectMaxBuildPayload; ++c)
        if (c < a.n_bin) st_cs_w(a.bout[c], p, a.bin_w[c], bv[c][j]);
    }
  }
  if (s_abort && threadIdx.x == 0) {
    atomicOr(a.d_count, 1ull << 63);
    // let copies still in flight land before the CTA's shared memory is released
    for (int q = 0; q < kTmaStages; ++q) mbar_wait_bounded(&s_bar[q], 0, 64);
  }
}

// ------------------------------------------------------------------------------------------------
// host side
// ------------------------------------------------------------------------------------------------
bool direct_args(const GatherArgs& g, DirectArgs& a) {
  if (g.n_pin > kDirectMaxProbePayload || g.n_bin > kDirectMaxBuildPayload) return false;
  a = DirectArgs{};
  a.out_prid = g.out_prid;
  a.out_brid = g.out_brid;
  a.prid_map = g.prid_map;
  a.capacity = g.capacity;
  a.d_count = g.d_count;
  a.matched = g.matched;
  a.n_pin = g.n_pin;
  a.n_bin = g.n_bin;
  for (int c = 0; c < g.n_pin; ++c) {
    const PayloadIn& in = g.pin[c];
    if (in.valid || in.valid8 || (in.width != 4 && in.width != 8) || in.stride != in.width) return false;
    a.pin[c] = in.data;
    a.pin_w[c] = in.width;
    a.pout[c] = g.pout[c].data;
  }
  if (g.n_bin > 0 && g.rec) {
    if (g.rec_stride != 8 && g.rec_stride != 16 && g.rec_stride != 32) return false;
    a.rec_std = 1;
    for (int c = 0; c < g.n_bin; ++c) {
      const int w = g.bin[c].width;
      if ((w != 4 && w != 8) || g.rec_voff[c] >= 0) return false;
      if (w != 8 || g.rec_off[c] != 8 + 8 * c) a.rec_std = 0;
      a.rec_off[c] = g.rec_off[c];
      a.bin_w[c] = w;
      a.bout[c] = g.bout[c].data;
    }
    a.rec = g.rec;
    a.rec_stride = g.rec_stride;
    return true;
  }
  a.brid_map = g.brid_map;
  a.brid_stride = g.brid_stride;
  a.bin_by_pos = g.bin_by_pos;
  for (int c = 0; c < g.n_bin; ++c) {
    const PayloadIn& in = g.bin[c];
    if (in.valid || in.valid8 || (in.width != 4 && in.width != 8)) return false;
    a.bin[c] = in.data;
    a.bin_stride[c] = in.stride;
    a.bin_w[c] = in.width;
    a.bout[c] = g.bout[c].data;
  }
  return true;
}

static bool al16(const void* p) { return ((uintptr_t)p & 15u) == 0; }

template <typename K, bool WIDE>
static void launch_tma(const sj_table* t, const sj_column& p, const int64_t* d_n, const DirectArgs& a,
                       cudaStream_t s) {
  const TmaStage st = tma_stage<K>(a);
  const size_t smem = (size_t)kTmaStages * st.bytes;
  if (smem > 48 * 1024)
    cudaFuncSetAttribute(probe_tma_kernel<K, WIDE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  int resident = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident, probe_tma_kernel<K, WIDE>, kDirectThreads, smem);
  const int64_t tiles = (p.num_rows + kTmaTile - 1) / kTmaTile;
  const int per_sm = std::min(std::max(1, resident), std::max(1, t->params.ctas_per_sm));
  const int grid = (int)std::max<int64_t>(1, std::min<int64_t>(tiles, (int64_t)sm_count(t->device) * per_sm));
  probe_tma_kernel<K, WIDE><<<grid, kDirectThreads, smem, s>>>(
      table_dev(t), static_cast<const K*>(p.data), p.validity, p.validity_offset, p.num_rows, d_n, a, st);
}

bool probe_direct(const sj_table* t, const sj_column& p, const int64_t* d_n, const GatherArgs& g, cudaStream_t s) {
  const sj_join_params& pr = t->params;
  if (pr.probe_kernel == SJ_PROBE_KERNEL_STAGED) return false;
  DirectArgs a;
  if (!direct_args(g, a)) return false;
  a.l2_last = pr.table_l2_priority == SJ_L2_EVICT_LAST;
  // AUTO takes plain loads: on the large 1:1 join the TMA ring's per-tile CTA barriers cost more than
  // the DRAM latency it hides (measured 1.96 vs 1.73 ms per 64M probe rows)
  bool tma = pr.probe_kernel == SJ_PROBE_KERNEL_DIRECT_TMA && (!a.rec || a.rec_std) && !a.matched;
  tma = tma && al16(p.data) && (!a.prid_map || al16(a.prid_map));
  for (int c = 0; c < a.n_pin; ++c) tma = tma && al16(a.pin[c]);
  if (tma) {
    KernelTimer timer("probe_direct", s);
    const bool wide = t->slot_kind == SJ_SLOT_WIDE128;
    if (t->key_type == SJ_INT32) {
      if (wide) launch_tma<int32_t, true>(t, p, d_n, a, s);
      else launch_tma<int32_t, false>(t, p, d_n, a, s);
    } else {
      if (wide) launch_tma<int64_t, true>(t, p, d_n, a, s);
      else launch_tma<int64_t, false>(t, p, d_n, a, s);
    }
    return true;
  }
  probe_units(t, p.data, p.validity, p.validity_offset, p.num_rows, d_n, nullptr, a, s);
  return true;
}

bool probe_runs_ok(const sj_table* t, const GatherArgs& g) {
  const sj_join_params& pr = t->params;
  if (pr.probe_kernel == SJ_PROBE_KERNEL_STAGED || pr.probe_kernel == SJ_PROBE_KERNEL_DIRECT_TMA) return false;
  DirectArgs a;
  return direct_args(g, a);
}

void probe_runs(const sj_table* t, const void* keys, int64_t n, const RunArgs& ra, const GatherArgs& g, cudaStream_t s) {
  DirectArgs a;
  direct_args(g, a);
  probe_units(t, keys, nullptr, 0, n, nullptr, &ra, a, s);
}

}  // namespace sj
