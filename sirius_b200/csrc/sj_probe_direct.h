// The direct write-out DISTINCT probe (sj_probe_direct.cu): its argument block and entry point.
#pragma once

#include "sj_device.cuh"
#include "sj_internal.h"

namespace sj {

constexpr int kDirectMaxProbePayload = 2;
constexpr int kDirectMaxBuildPayload = 3;

struct DirectArgs {
  int32_t* out_prid;
  int32_t* out_brid;
  const int32_t* prid_map;  // probe array index -> probe row id (partitioned probe), or NULL
  const int32_t* brid_map;  // table position -> build row id at brid_map + pos * brid_stride bytes
  int32_t brid_stride;
  int32_t bin_by_pos;       // build payload element index: table position (1) or build row id (0)
  const void* rec;          // row store (record = [row id | fields]) or NULL
  int32_t rec_stride;
  int32_t rec_std;          // fields are 8-byte at offsets 8, 16, 24 (else rec_off / bin_w)
  int16_t rec_off[kDirectMaxBuildPayload];
  int32_t n_pin, n_bin;
  const void* pin[kDirectMaxProbePayload];
  int32_t pin_w[kDirectMaxProbePayload];
  void* pout[kDirectMaxProbePayload];
  const void* bin[kDirectMaxBuildPayload];
  int32_t bin_stride[kDirectMaxBuildPayload];
  int32_t bin_w[kDirectMaxBuildPayload];
  void* bout[kDirectMaxBuildPayload];
  int64_t capacity;
  unsigned long long* d_count;
  uint32_t* matched;  // unit probe: bit of every probe row with a match (zero before if partitioned), or NULL
  int32_t l2_last;  // TMA-staged probe: table slot loads marked L2 evict_last
};

// Partition runs of a tile-local partition (local_partition): rows of partition p in tile i are
// [run_off[p * n_tiles + i], + run_cnt[p * n_tiles + i]).
struct RunArgs {
  const int32_t* run_off;
  const int32_t* run_cnt;
  uint32_t n_tiles;
  uint32_t P;
  uint32_t log2_pieces;  // a run is split into 2^log2_pieces units,
  uint32_t log2_join;    // or the runs of 2^log2_join consecutive tiles are one
};

// Fills `a` from a general gather description; false when the output shape needs the staged
// kernel (NULL payloads, 1/2-byte payloads, too many columns, other record layouts).
bool direct_args(const GatherArgs& g, DirectArgs& a);

// Launches the probe of DISTINCT table `t` when the shape allows and the table's parameters do not ask for
// the staged kernel; returns false (nothing launched) otherwise. `d_n`: device row count, or NULL.
bool probe_direct(const sj_table* t, const sj_column& p, const int64_t* d_n, const GatherArgs& g, cudaStream_t s);

// True when probe_runs serves this gather.
bool probe_runs_ok(const sj_table* t, const GatherArgs& g);

// Probe of tile-local partition runs: `keys` (n rows), the partition row ids and payloads in `g` are the
// partitioned arrays; the runs are walked partition after partition. Requires probe_runs_ok.
void probe_runs(const sj_table* t, const void* keys, int64_t n, const RunArgs& ra, const GatherArgs& g, cudaStream_t s);

}  // namespace sj
