// Shared and tensor memory of the convolution's tile kernels.  Plain C++: tests read it without a GPU.
#pragma once
#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <numeric>

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

// Whether a gather GEMM on the CUDA cores is faster with a thread per output than in tiles of 64 rows: where there is
// too little of it to fill the tiles' stages, one after another for every offset and 16 channels.  An estimate of both,
// in ns per kernel offset, fitted to 1,309 layers (FP32 and 16-bit, 200 to 200,000 rows, 1 to 256 channels in and out):
// - tiles: 1,350 a 16 channels while an SM's blocks are few, and 1.1 for 1,000 outputs (of columns padded to the tile's);
// - a thread per output: the longer of a thread's own chain and of what the SMs issue for all of them.  A warp's lanes
//   read rows of weights and of features, `conflicts` of them one after another: what lies in one bank, or a third of
//   the lines they touch.
// The choice takes at most 1.23 times what a thread per output takes, and at most 1.4 times the better one's time in all
// but one of them (1.53).  16 -> 32 channels FP32, 1,000 rows: 24 us by thread, 35 in tiles; 8,000 rows: 138 and 36.
// 144 -> 4 channels in 16 bits, 3,000 rows: 92 and 405.
inline bool simt_by_thread(int64_t rows, int kdim, int ncols, int elem_bytes) {
  const double outputs = (double)rows * ncols;
  const double bank = std::max(1, std::gcd(kdim * elem_bytes, 128) / 4);       // a power of two up to 32
  const double lines = std::min(1.0, kdim * elem_bytes / 128.0) / 3;           // of a row
  const double of_weights = std::max(1.0, std::min(ncols, 32) * std::max(bank / 32, lines));
  const double of_rows = std::max(1.0, 32.0 / ncols * std::max(bank / 32, lines));
  const double conflicts = ncols >= 32 ? of_weights + 1 : of_weights + of_rows + 3;
  const double work = std::max(24 + 1.5 * kdim, kdim * conflicts);
  constexpr double WAVE = 148 * 256;                                           // a block of 256 threads to every SM
  const double waves = (double)((int64_t)((outputs + WAVE - 1) / WAVE));
  const double by_thread = std::max(350 + 2.9 * work, waves * WAVE * work * 6.7e-5);
  const int padded = ncols <= 16 ? 16 : ncols <= 32 ? 32 : (ncols + 63) / 64 * 64;
  const double tiles = (kdim + 15) / 16 * (1350 + (double)rows * padded * 1.1e-3);
  return by_thread < tiles;
}

}  // namespace conv
