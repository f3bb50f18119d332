// Shared and tensor memory of the convolution's tile kernels.  Plain C++: tests read it without a GPU.
#pragma once
#include <algorithm>
#include <cstddef>
#include <cstdint>

namespace conv {

constexpr int BM = 128;                  // rows of a tile (UMMA M)
constexpr uint32_t A_BYTES = BM * 128;   // of a stage: 16 KB
constexpr int TMA_STAGES = 8;            // of the gather GEMM's ring, at most
constexpr int TMEM_COLUMNS = 512;        // of an SM
// Blocks that an SM is to hold.  1.3M rows of 64 -> 64 channels: 767 us, 907 with three.
constexpr int CONV_PER_SM = 4;

// Columns of tensor memory that a tile of n accumulator columns allocates: a power of two.
constexpr uint32_t tmem_columns(int n) { return n <= 32 ? 32u : n <= 64 ? 64u : n <= 128 ? 128u : 256u; }

struct GatherPlan {
  int per_sm, stages;
  uint32_t stage_bytes;
  size_t smem;                           // dynamic, of a block
};

// As many blocks on an SM as its shared and its tensor memory hold, up to CONV_PER_SM, of two stages or more, for tiles
// of `box` columns.
inline GatherPlan gather_plan(int box) {
  GatherPlan p{};
  const size_t fixed = 1024;                                    // alignment of the first stage
  p.stage_bytes = A_BYTES + (uint32_t)((box * 128 + 1023) & ~1023);
  for (p.per_sm = std::min(CONV_PER_SM, TMEM_COLUMNS / (int)tmem_columns(box));; p.per_sm--) {
    const size_t room = (227 << 10) / p.per_sm - 1536;          // the kernel's static arrays, the block's reserve
    p.stages = fixed < room ? (int)std::min<size_t>((room - fixed) / p.stage_bytes, TMA_STAGES) : 0;
    if (p.stages >= 2 || p.per_sm == 1) break;
  }
  p.smem = fixed + (size_t)p.stages * p.stage_bytes;
  return p;
}

}  // namespace conv
