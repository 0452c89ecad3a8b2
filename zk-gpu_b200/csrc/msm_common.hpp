// Constants and small structs shared by the MSM kernels (msm_kernels.cuh) and the host plan
// (msm.hpp).
#pragma once
#include <cstdint>

namespace zkg {

constexpr uint32_t kNegBit = 0x80000000u;
constexpr uint32_t kNoKey = 0xffffffffu;
constexpr uint32_t kPadEntry = 0xffffffffu;  // a place of the sorted array without an entry (infinity)
// The scan over the slots: threads of a block, values of a thread.
constexpr int kScanBlock = 1024;
constexpr int kScanItems = 4;
constexpr int kScanTile = kScanBlock * kScanItems;
constexpr int kReduceThreads = 128;  // one running-sum block covers this many chunks of one window
constexpr int kMaxReduceLevels = 16;
// The last level takes at most this many values per window and is summed by marginals
// (msm_marginals) instead of further running sums: columns and rows of at most 64.
constexpr uint32_t kMarginalMax = 4096;

struct ReduceLevels {
  uint32_t count;                         // chunked levels
  uint32_t chunk_log;                     // buckets per running-sum thread = 2^chunk_log
  uint32_t tot_len[kMaxReduceLevels];     // tot values per window at each level
  uint32_t tot_offset[kMaxReduceLevels];  // start (in points) of level l's tot array; window stride = tot_len
};

}  // namespace zkg
