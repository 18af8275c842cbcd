// Interface of the tcgen05 corpus scan (topk_scan_sm100.cu) used by the top-k driver (topk.cu).
#pragma once

#include "common.cuh"

namespace phx {

struct TcScanArgs {
  long long rows;            // corpus rows of this shard
  long long row_offset;      // global id of local row 0
  int row_bytes, B;          // bytes of a corpus row (128 or 256), live queries (<= 256)
  int stride;                // sample pass: tiles 0, stride, 2*stride, ...
  float* gmax;               // sample pass out: [B][n_groups] maxima of 32-row groups
  long long n_groups;        // sampled tiles * 4
  const float* pivot;        // collect pass in: [B]
  unsigned long long* surv;  // collect pass out: [B][cap] keys ordered(score) << 32 | ~global_row
  int* counts;               // [B]
  int cap;
  // optional eligibility of the shard's rows: bit (r & 31) of mask[r >> 5] for shard-local row r = mask_row0 + row;
  // a row whose bit is clear is skipped like a row past the end.  null = every row is eligible
  const unsigned int* mask = nullptr;
  long long mask_row0 = 0;
  // int8 corpus (recsys_two_tower_model.py:2518-2533): score = bf16((float(int32 dot) * user_scale[u]) * row_scale[row]);
  // null = bf16 corpus
  const float* user_scale = nullptr;   // [B]
  const float* row_scale = nullptr;    // [rows]
  int scales_negative = 0;             // some row scale of the corpus is below zero
};

__device__ __forceinline__ bool row_eligible(const unsigned int* mask, long long mask_row0, long long row) {
  if (!mask) return true;
  const long long r = mask_row0 + row;
  return (mask[r >> 5] >> (r & 31)) & 1u;
}

// rows of 64 or 128 bf16, or of 128 or 256 int8
bool tc_scan_supported(int row_bytes);
// `queries`: [256][row_bytes], in the corpus' type
phx_status tc_scan_make_maps(CUtensorMap* map_corpus, CUtensorMap* map_users, const void* corpus, long long rows, int row_bytes,
                             const void* queries, std::string& err);
// mode 0 = sample pass (group maxima), 1 = collect pass (survivors).  expected: rows that the pivot is to let through for a query
phx_status tc_scan_launch(const CUtensorMap& map_corpus, const CUtensorMap& map_users, const TcScanArgs& a, int mode, double expected,
                          int num_sms, int* err_flag, cudaStream_t stream, std::string& err);

}  // namespace phx
