// The unit probe of DISTINCT tables (sj_probe_units.cu).
#pragma once

#include "sj_probe_direct.h"

namespace sj {

// Probes `n` rows (at most *d_n when d_n is given), or the partition runs `runs` of the probe arrays, into `t`
// for the gather `a`.
void probe_units(const sj_table* t, const void* keys, const uint32_t* kv, int64_t kvoff, int64_t n, const int64_t* d_n,
                 const RunArgs* runs, const DirectArgs& a, cudaStream_t s);

// Sets bit i of `words` for every probe row i with a match in `t` (any layout), from the partitioned arrays `keys` and
// `prid_map`, which lack the rows that cannot match. `words` must be zero before.
void find_units(const sj_table* t, const void* keys, int64_t n, const RunArgs& runs, const int32_t* prid_map,
                uint32_t* words, const RangeGate& gate, cudaStream_t s);

// GROUPED table: adds the matches of all probe rows to *d_total and, when m_ent is given, appends {probe row, group
// start} and the group size of the rows with matches to m_ent / m_cnt at *d_nent.
void match_units(const sj_table* t, const sj_column& p, int2* m_ent, int32_t* m_cnt, unsigned long long* d_nent,
                 unsigned long long* d_total, cudaStream_t s);

}  // namespace sj
