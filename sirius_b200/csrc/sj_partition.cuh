// Radix partitioning shared by the build and the probe (implemented in sj_partition.cu).
#pragma once

#include "sj_device.cuh"
#include "sj_internal.h"

namespace sj {

constexpr int kMaxPartitionBits = 10;

struct PartSrc {
  const void* keys;
  const uint32_t* kvalid;
  int64_t kvoff;
  int64_t n;
  int32_t n_pay;
  PayloadIn pay[kMaxPayload];
};

// Outputs. stride == 0: rid / pay[c] / valid8[c] are plain arrays. stride > 0: they point at
// their fields inside one record array of `stride` bytes per row (the table's row store).
struct PartDst {
  void* keys;
  int32_t* rid;
  void* pay[kMaxPayload];
  uint8_t* valid8[kMaxPayload];
  int32_t stride;
};

size_t partition_scratch_bytes(int pbits, int device);
// Tile-local variant (one pass, no histogram): each tile of kPartTileRows rows is sorted by partition
// in place; off / cnt[p * tiles + tile] give partition p's rows of every tile. Only for
// plain outputs with at most 2 payloads of 4/8 bytes without NULLs. Rows with a NULL key or a key outside
// [kmin, kmax] (the table's range) are dropped. zero_bits: NULL, or one bit per row to clear on the way.
constexpr int kPartTileRows = 4096;
struct LocalRuns {
  int32_t* off;
  int32_t* cnt;
  uint32_t* zero_bits = nullptr;
  RangeGate gate;
};
sj_status local_partition(const PartSrc& src, int key_type, int pbits, int64_t kmin, int64_t kmax, const PartDst& dst,
                          const LocalRuns& runs, int device, cudaStream_t s);
bool partition_plain_shape(const PartSrc& src, const PartDst& dst);

sj_status radix_partition(const PartSrc& src, int key_type, int pbits, const PartDst& dst, void* scratch,
                          int device, cudaStream_t s, const int64_t** d_total_out, const int64_t** d_offs_out,
                          int* grid_out);

// Partitioning of columns alone (the partition operator): every row is valid, and no row ids or key
// copies are made. A column is `width` bytes per row at src, or one validity bit per row (bits != NULL)
// written as one byte; is_key: the partition key itself (same type), which must come first; pairs: src
// starts on a multiple of twice the width (row pairs are vector loads).
struct PartColumn {
  const void* src;
  const uint32_t* bits;
  int64_t voff;
  void* dst;
  int32_t width;
  int16_t is_key;
  int16_t pairs;
};
struct PartColumns {
  int32_t n;
  PartColumn c[2 * kMaxPayload];
};
sj_status partition_columns(const void* keys, int key_type, int64_t n, int pbits, const PartColumns& cols, void* scratch,
                            int device, cudaStream_t s, const int64_t** d_total_out, const int64_t** d_offs_out,
                            int* grid_out);

}  // namespace sj
