// Sparse convolution over voxel neighbour maps (ref: csrc/sparse_op/convolution_cuda.cu:52-282 and
// its caller models/ascn/utils.py:108-190): out[o] = sum_k in[i_k(o)] @ W[k] over the (input, output)
// pairs of every kernel offset k.
//
// The reference runs, per offset, a gather kernel into a dense buffer, a cuBLAS GEMM and a scatter-add
// kernel (27 x 3 launches and two buffers through HBM per layer).  Here the map is first turned into
// an output-major table (row o, offset k) -> input row or -1, and ONE kernel computes a 128-row tile
// of the output: for every offset the tile's 128 input rows are gathered straight into shared memory
// in the tensor core's K-major 128-byte-swizzled layout, the offset's weights beside them, and
// tcgen05.mma accumulates all offsets into the same TMEM accumulator (FP32); the epilogue reads TMEM
// once and writes each output row once -- no scatter, no atomics, no intermediate buffers.  The input
// gradient is the same kernel over the transposed table with W[k]^T; the weight gradient is a GEMM
// over the pairs of one offset (split over CTAs, partials reduced in a fixed order).
//
// Warp roles of the gather GEMM: at "tiles through TMA" below.  In the tile kernel of the weight gradient (288
// threads) warps 0-7 gather tiles into a ring of shared-memory stages and run the epilogue (warp w reads TMEM lanes
// 32(w%4).. = tile rows, column half w/4); warp 8 allocates TMEM and one of its lanes issues the MMAs.  Stages are
// handed over through mbarriers: "full" (arrivals after the stores and a proxy fence) and "empty" (tcgen05.commit of
// the MMAs that read the stage).  Every wait is bounded; on timeout the kernel records NGS_ERR_TIMEOUT, stops
// issuing, waits (bounded) for its copies and MMAs and releases its TMEM before returning.
#include <algorithm>
#include <cstdint>
#include <type_traits>
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include "conv_plan.h"
#include "conv_ring.h"
#include "ngs_common.cuh"

namespace conv {

constexpr int BK = 64;               // reduction elements per stage (128 bytes of 16-bit values)
constexpr int UK = 16;               // UMMA K of kind::f16
constexpr int PRODUCERS = 256;       // warps 0-7
constexpr int THREADS = PRODUCERS + 32;
constexpr int KMAX = 128;            // kernel offsets (5^3 = 125 at most)
constexpr long long WAIT_CYCLES = 4000000000ll;         // bound of one mbarrier wait (2 s or more)

NGS_DEV uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

NGS_DEV void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
NGS_DEV void mbar_arrive(uint64_t* bar) {
  asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.shared::cta.b64 st, [%0];\n\t}" ::"r"(smem_u32(bar)) : "memory");
}
NGS_DEV bool mbar_try(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait for the phase of the given parity to complete; false when the bound ran out or another
// thread of the CTA already gave up (abort flag in shared memory).
NGS_DEV bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* abort) {
  if (mbar_try(bar, parity)) return true;
  const long long t0 = clock64();
  while (!mbar_try(bar, parity)) {
    if (*abort) return false;
    if (clock64() - t0 > WAIT_CYCLES) {
      *abort = 1;
      return false;
    }
  }
  return true;
}

// Shared-memory matrix descriptor of a K-major tile with 128-byte swizzle: rows of 128 bytes, 8-row
// groups 1024 bytes apart (stride byte offset), leading byte offset 16 (unused by this layout but set
// as the canonical form has it), descriptor version 1, swizzle mode 2 (128 B).  The tile must start on
// a 1024-byte boundary; a K step inside the 128-byte row advances the start address.
NGS_DEV uint64_t kmajor_sw128_desc(uint32_t saddr) {
  return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) |
         ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}

// Shared-memory matrix descriptor of an MN-major tile with 128-byte swizzle: each 128-byte row holds 64
// consecutive M (or N) elements at one K index, 8 K rows form a 1024-byte swizzle atom (stride byte
// offset 1024 between the atoms along K), and the 64-element atoms along M sit 8 KB apart (leading
// byte offset: 64 K rows per stage).  A K step of 16 advances the start address by two atoms.
constexpr uint32_t MN_ATOM_BYTES = 64 * 128;
NGS_DEV uint64_t mnmajor_sw128_desc(uint32_t saddr) {
  return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)(MN_ATOM_BYTES >> 4) << 16) |
         ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}

// Instruction descriptor of kind::f16 with FP32 accumulation, both operands K-major.
// bf16: 1 = BF16 inputs, 0 = FP16 inputs (A and B always share the type).
NGS_DEV uint32_t f16_idesc(int m, int n, int bf16) {
  const uint32_t fmt = bf16 ? 1u : 0u;
  return (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}
// The same with both operands MN-major (bits 15 and 16).
NGS_DEV uint32_t f16_idesc_mn(int m, int n, int bf16) { return f16_idesc(m, n, bf16) | (1u << 15) | (1u << 16); }

NGS_DEV void umma_f16(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
      "l"(da), "l"(db), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Arrives on the mbarrier once every MMA issued so far by this thread has completed.
NGS_DEV void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}
NGS_DEV void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
NGS_DEV void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// Generic-proxy stores to shared memory become visible to the tensor core (async proxy).
NGS_DEV void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// 16 bytes from global to shared memory without passing through registers; zeros when !have.
NGS_DEV void cp_async16(uint32_t dst, const void* src, bool have) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.eq.u32 p, %2, 0;\n\tcp.async.cg.shared.global [%0], [%1], 16, p;\n\t}" ::"r"(dst),
      "l"(src), "r"((uint32_t)have)
      : "memory");
}
NGS_DEV void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int PENDING>
NGS_DEV void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(PENDING) : "memory");
}

// TMEM allocation by one whole warp; the column base lands in *dst (shared memory).
NGS_DEV void tmem_alloc(uint32_t* dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst)), "r"(ncols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
NGS_DEV void tmem_free(uint32_t base, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(ncols) : "memory");
}
// 16 consecutive FP32 columns of this thread's TMEM lane (warp w reads lanes 32w..32w+31).
NGS_DEV void tmem_ld16(uint32_t addr, float (&v)[16]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(addr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int j = 0; j < 16; j++) v[j] = __uint_as_float(r[j]);
}

// Byte offset of 16-byte chunk c of row r in a K-major 128-byte-swizzled tile (1024-byte aligned).
NGS_DEV uint32_t sw128(int r, int c) { return (uint32_t)(r * 128 + ((c ^ (r & 7)) << 4)); }

}  // namespace conv

// ----------------------------------------------------------------------------- gather tables
// Entry (row, k) of a table, at row * row_stride + k * k_stride: the source row paired with `row` at
// offset k (-1: none).  Pairs of offset k are nbmaps[starts[k] .. starts[k+1]) as (c0, c1) int32 pairs;
// key_col picks the column that indexes the table rows, the other column is the source.  mid >= 0:
// entry (row, mid) = row for every row (the reference's forward computes that offset as one dense
// product over all rows).
// The pairs of an offset usually come in the order of their rows, so with the offset outermost (k_stride
// = n_rows) a warp's entries are neighbours in memory, and so are a tile's when they are read; with the row
// outermost every entry is a 32-byte sector of its own.  1.3M rows, 24M pairs: 0.087 ms against 0.52.
__global__ void conv_table_kernel(const int32_t* __restrict__ nbmaps, const int64_t* __restrict__ starts, int K,
                                  int key_col, int64_t n_rows, int64_t row_stride, int64_t k_stride, int mid,
                                  int32_t* __restrict__ table) {
  const int k = blockIdx.y;
  const int64_t first = starts[k], end = starts[k + 1];
  if (k == mid) {
    for (int64_t r = ngs_gtid(); r < n_rows; r += ngs_gstride()) table[r * row_stride + k * k_stride] = (int32_t)r;
    return;
  }
  for (int64_t p = first + ngs_gtid(); p < end; p += ngs_gstride()) {
    const int32_t key = nbmaps[2 * p + key_col], src = nbmaps[2 * p + 1 - key_col];
    if (key < 0 || key >= n_rows) continue;    // the reference's scatter skips negative targets
    table[key * row_stride + k * k_stride] = src < 0 ? -1 : src;
  }
}

static int conv_table(const int32_t* nbmaps, const int64_t* starts_dev, int K, int key_col, int64_t n_rows,
                      int64_t row_stride, int64_t k_stride, int mid, int32_t* table, cudaStream_t st) {
  if (K < 1 || K > 128 || (key_col != 0 && key_col != 1) || n_rows < 0 || mid >= K || !starts_dev ||
      (n_rows > 0 && !table))
    return NGS_ERR_INVALID_ARG;
  if (n_rows > 0 && cudaMemsetAsync(table, 0xFF, (size_t)n_rows * K * sizeof(int32_t), st) != cudaSuccess)
    return ngs_set_cuda_error(cudaGetLastError());
  // the pair counts are on the device: about one thread per row and offset
  const dim3 grid(ngs_blocks(n_rows > 0 ? n_rows : 1, 256, 8), (unsigned)K);
  ngs_count_launch();
  conv_table_kernel<<<grid, 256, 0, st>>>(nbmaps, starts_dev, K, key_col, n_rows, row_stride, k_stride, mid, table);
  NGS_CHECK_LAUNCH();
  return NGS_OK;
}

extern "C" int ngs_conv_table(const int32_t* nbmaps, const int64_t* starts_dev, int K, int key_col, int64_t n_rows,
                              int mid, int32_t* table, ngs_stream s) {
  return conv_table(nbmaps, starts_dev, K, key_col, n_rows, K, 1, mid, table, (cudaStream_t)s);
}

extern "C" int ngs_conv_table_kmajor(const int32_t* nbmaps, const int64_t* starts_dev, int K, int key_col,
                                     int64_t n_rows, int mid, int32_t* table, ngs_stream s) {
  return conv_table(nbmaps, starts_dev, K, key_col, n_rows, 1, n_rows, mid, table, (cudaStream_t)s);
}

// ----------------------------------------------------------------------------- the tile kernel
// One CTA computes a 128 x N tile (N <= 256, a multiple of 16) of D = sum over `steps` of A_s B_s^T,
// every A_s (128 x 64) and B_s (N x 64) filled by the producers straight into a shared-memory stage
// (K-major, 128-byte swizzle), accumulated in TMEM by tcgen05.mma, and handed to the epilogue.
// Fill: the source of the tiles -- fill(step, a, b, tid) stores the stage's A and B rows (zeros where
// there is no data) and returns the number of valid reduction elements of the step (<= 64).  ASYNC: fill
// only issues asynchronous copies; the stage is handed over AHEAD steps later, so that a producer has the
// copies of AHEAD + 1 stages in flight (the ring has at least AHEAD + 1 stages).
// Store: store(row, col, v[16]) takes 16 consecutive accumulator columns of one tile row.
namespace conv {

struct TileShape {
  int steps;          // reduction steps of this tile (0: the tile is all zeros)
  int n;              // N of the MMA
  int stages;
  uint32_t stage_bytes;
};

constexpr int AHEAD = 2;

template <bool ASYNC, typename Fill, typename Store>
NGS_DEV void run_tile(const TileShape& t, uint8_t* smem, Fill& fill, Store& store, int bf16, int* error,
                      bool mn_major = false) {
  __shared__ uint64_t full_bar[8], empty_bar[8], done_bar;
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;
  __shared__ int ksteps_of[8];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int S = t.stages;
  const uint32_t ncols_alloc = tmem_columns(t.n);
  if (tid == 0) {
    for (int s = 0; s < S; s++) {
      mbar_init(&full_bar[s], PRODUCERS / 32);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(&done_bar, 1);
    abort_flag = 0;
  }
  if (warp == PRODUCERS / 32) tmem_alloc(&tmem_slot, ncols_alloc);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;

  if (tid < PRODUCERS) {
    // producers: fill the ring of stages (the ring position and its round are counted along: a division
    // by the stage count costs more instructions than a stage's copies)
    auto hand_over = [&](int st) {
      fence_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&full_bar[st]);
    };
    int s = 0, st = 0;
    uint32_t parity = 1u;                        // of the round before this one
    for (; s < t.steps; s++) {
      const bool go = s < S || mbar_wait(&empty_bar[st], parity, &abort_flag);
      if (!__all_sync(0xffffffffu, go)) break;
      uint8_t* a = smem + (size_t)st * t.stage_bytes;
      const int valid = fill(s, a, a + A_BYTES, tid);
      if (tid == 0) ksteps_of[st] = (valid + UK - 1) / UK;
      if constexpr (ASYNC) {
        cp_async_commit();
        if (s >= AHEAD) {
          cp_async_wait<AHEAD>();
          hand_over(st >= AHEAD ? st - AHEAD : st - AHEAD + S);
        }
      } else {
        hand_over(st);
      }
      if (++st == S) {
        st = 0;
        parity ^= 1u;
      }
    }
    if constexpr (ASYNC) {
      // the last stages; after an abort the copies still land before the shared memory is given up
      cp_async_wait<0>();
      if (s == t.steps)
        for (int r = max(0, s - AHEAD); r < s; r++) hand_over(r % S);
    }
  } else if (lane == 0) {
    // one thread issues the MMAs of every stage, then commits the stage back to the producers
    const uint32_t idesc = mn_major ? f16_idesc_mn(BM, t.n, bf16) : f16_idesc(BM, t.n, bf16);
    int st = 0;
    uint32_t parity = 0u;
    for (int s = 0; s < t.steps; s++) {
      if (!mbar_wait(&full_bar[st], parity, &abort_flag)) break;
      tc_fence_after();
      const uint32_t a = smem_u32(smem + (size_t)st * t.stage_bytes), b = a + A_BYTES;
      const int ks = ksteps_of[st];
      for (int kk = 0; kk < ks; kk++)
        umma_f16(tmem,
                 mn_major ? mnmajor_sw128_desc(a + kk * 2048) : kmajor_sw128_desc(a + kk * 32),
                 mn_major ? mnmajor_sw128_desc(b + kk * 2048) : kmajor_sw128_desc(b + kk * 32), idesc,
                 (s > 0 || kk > 0) ? 1u : 0u);
      umma_commit(&empty_bar[st]);
      if (++st == S) {
        st = 0;
        parity ^= 1u;
      }
    }
    umma_commit(&done_bar);        // arrives once everything issued above has completed
  }

  if (tid < PRODUCERS) {
    // epilogue: warp w reads TMEM lanes 32 (w % 4) .. (its tile rows), every other 16-column chunk
    bool ok = mbar_wait(&done_bar, 0u, &abort_flag);
    ok = __all_sync(0xffffffffu, ok) && !abort_flag;
    tc_fence_after();
    const int w = warp & 3, half = warp >> 2;
    const int row = 32 * w + lane;
    for (int cc = half; cc < t.n / 16; cc += 2) {
      float v[16];
      if (ok && t.steps > 0) {
        tmem_ld16(tmem + ((uint32_t)(32 * w) << 16) + (uint32_t)(cc * 16), v);
      } else {
#pragma unroll
        for (int j = 0; j < 16; j++) v[j] = 0.f;
      }
      if (ok) store(row, cc * 16, v);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (abort_flag) {
    int late = 0;                                // the MMAs issued end before their tensor memory is given up
    if (warp == PRODUCERS / 32 && lane == 0) mbar_wait(&done_bar, 0u, &late);
    if (tid == 0) atomicExch(error, NGS_ERR_TIMEOUT);
    __syncwarp();
  }
  if (warp == PRODUCERS / 32) {
    tc_fence_after();
    tmem_free(tmem, ncols_alloc);
  }
}

NGS_DEV uint4 ldg16(const uint16_t* p) { return __ldg(reinterpret_cast<const uint4*>(p)); }

NGS_DEV void st16_row(void* out, bool f32, int bf16, int64_t off, const float (&v)[16]) {
  if (f32) {
    float4* o = reinterpret_cast<float4*>(static_cast<float*>(out) + off);
#pragma unroll
    for (int j = 0; j < 4; j++) o[j] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
  } else {
    uint32_t p[8];
#pragma unroll
    for (int j = 0; j < 8; j++) {
      if (bf16) {
        const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
        p[j] = *reinterpret_cast<const uint32_t*>(&h);
      } else {
        const __half2 h = __floats2half2_rn(v[2 * j], v[2 * j + 1]);
        p[j] = *reinterpret_cast<const uint32_t*>(&h);
      }
    }
    uint4* o = reinterpret_cast<uint4*>(static_cast<uint16_t*>(out) + off);
    o[0] = make_uint4(p[0], p[1], p[2], p[3]);
    o[1] = make_uint4(p[4], p[5], p[6], p[7]);
  }
}

}  // namespace conv

// ----------------------------------------------------------------------------- tiles through TMA
// The tile kernel with most of its stages' bytes moved by TMA: two warps issue the copies (a row gather moves four
// rows of 128 bytes, zeros for rows and channels out of range, in the swizzled layout), one thread issues the MMAs,
// and the four warps of the epilogue copy the tile's last rows with cp.async meanwhile.  Both ways of copying have a
// rate of their own.  1.3M rows of 64 -> 64 channels, 27 offsets: 1,310 us with cp.async alone (the producers'
// instructions, 270 a step and warp), 1,128 with one warp issuing all rows by TMA (50 cycles a gather), 772 with four,
// 760 in this form.  What is left are issue slots (70 % busy) and the steps' waits for one another, not bytes: L2 runs at
// 31 % and DRAM at 7 % of their rates.
namespace conv {

constexpr int TMA_THREADS = 224;         // warps 0 and 6: TMA, warp 1: MMAs, warps 2-5: cp.async, then epilogue

NGS_DEV void mbar_expect(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
// Four rows of 128 bytes (the map's box: 64 elements, one row) at channel c.
NGS_DEV void tma_gather4(uint32_t dst, const CUtensorMap* map, int c, int r0, int r1, int r2, int r3, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile::gather4.mbarrier::complete_tx::bytes [%0], "
      "[%1, {%2, %3, %4, %5, %6}], [%7];" ::"r"(dst),
      "l"(map), "r"(c), "r"(r0), "r"(r1), "r"(r2), "r"(r3), "r"(smem_u32(bar))
      : "memory");
}
NGS_DEV void tma_tile(uint32_t dst, const CUtensorMap* map, int c, int r, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
      "l"(map), "r"(c), "r"(r), "r"(smem_u32(bar))
      : "memory");
}

// Every producer warp walks the steps for itself: next() finds its next step and returns the valid reduction elements
// (0: no more).  Issue: issue(a, bar, w) starts TMA warp w's copies into the stage, t.tx[w] bytes in all; copy(a, w)
// issues the cp.async of warp w of four.
struct TmaShape {
  int n, stages;
  uint32_t stage_bytes, tx[2];
};

template <typename Setup, typename Next, typename Issue, typename Copy, typename Store>
NGS_DEV void run_tile_tma(const TmaShape& t, uint8_t* smem, Setup& setup, Next& next, Issue& issue, Copy& copy, Store& store,
                          int bf16, int* error) {
  __shared__ uint64_t full_bar[TMA_STAGES], empty_bar[TMA_STAGES], done_bar;
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag, any_step;
  __shared__ int ksteps_of[TMA_STAGES];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int S = t.stages;
  const uint32_t ncols_alloc = tmem_columns(t.n);
  if (tid == 0) {
    for (int s = 0; s < S; s++) {
      mbar_init(&full_bar[s], 6);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(&done_bar, 2);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    abort_flag = 0;
    any_step = 0;
  }
  if (warp == 1) tmem_alloc(&tmem_slot, ncols_alloc);
  setup();
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;

  RingSpan open{0, 0};                           // steps whose TMA copies may still be on their way
  if (warp == 0 || warp == 6) {
    const int w = warp == 6;
    open = ring_walk(
        S, next,
        [&](int st, uint32_t parity, bool first) {
          const bool go = first || mbar_wait(&empty_bar[st], parity, &abort_flag);
          return __all_sync(0xffffffffu, go) != 0;
        },
        [&](int st, int valid) {
          if (lane == 0) {
            if (w == 0) ksteps_of[st] = (valid + UK - 1) / UK;   // 0: no more steps
            if (valid > 0 && t.tx[w] > 0) mbar_expect(&full_bar[st], t.tx[w]);
            else mbar_arrive(&full_bar[st]);
          }
          __syncwarp();
          if (valid > 0) issue(smem + (size_t)st * t.stage_bytes, &full_bar[st], w);
        });
  } else if (warp >= 2) {
    // a step's copies are handed over while the next one's are in flight (the ring has two stages or more)
    auto hand_over = [&](int st) {
      fence_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&full_bar[st]);
    };
    int st = 0, s = 0, last = -1;
    uint32_t parity = 1u;
    bool more = true;
    while (more) {
      more = next() > 0;
      const bool go = s < S || mbar_wait(&empty_bar[st], parity, &abort_flag);
      if (!__all_sync(0xffffffffu, go)) break;
      if (more) copy(smem + (size_t)st * t.stage_bytes, warp - 2);
      cp_async_commit();
      if (last >= 0) {
        cp_async_wait<1>();
        hand_over(last);
      }
      last = st;
      s++;
      if (++st == S) {
        st = 0;
        parity ^= 1u;
      }
    }
    cp_async_wait<0>();
    if (last >= 0) hand_over(last);
  } else if (warp == 1 && lane == 0) {
    const uint32_t idesc = f16_idesc(BM, t.n, bf16);
    int st = 0;
    uint32_t parity = 0u, accumulate = 0u;
    for (;;) {
      if (!mbar_wait(&full_bar[st], parity, &abort_flag)) break;
      tc_fence_after();
      const uint32_t a = smem_u32(smem + (size_t)st * t.stage_bytes), b = a + A_BYTES;
      const int ks = ksteps_of[st];
      if (ks == 0) break;
      for (int kk = 0; kk < ks; kk++) {
        umma_f16(tmem, kmajor_sw128_desc(a + kk * 32), kmajor_sw128_desc(b + kk * 32), idesc, accumulate);
        accumulate = 1u;
      }
      umma_commit(&empty_bar[st]);
      if (++st == S) {
        st = 0;
        parity ^= 1u;
      }
    }
    any_step = (int)accumulate;
    umma_commit(&done_bar);        // arrives once everything issued above has completed,
    mbar_arrive(&done_bar);        // and here for any_step
  }

  if (warp >= 2 && warp < 6) {
    // warp w reads TMEM lanes 32 (w % 4) ..: its tile rows
    bool ok = mbar_wait(&done_bar, 0u, &abort_flag);
    ok = __all_sync(0xffffffffu, ok) && !abort_flag;
    tc_fence_after();
    const int w = warp & 3, row = 32 * w + lane;
    const bool any = any_step != 0;
    for (int cc = 0; cc < t.n / 16; cc++) {
      float v[16];
      if (ok && any) {
        tmem_ld16(tmem + ((uint32_t)(32 * w) << 16) + (uint32_t)(cc * 16), v);
      } else {
#pragma unroll
        for (int j = 0; j < 16; j++) v[j] = 0.f;
      }
      if (ok) store(row, cc * 16, v);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (abort_flag) {
    // what is in flight ends before the shared and the tensor memory are given up; once one of a thread's waits has
    // run its full time, the others are not waited for again
    int late = 0;
    if ((warp == 0 || warp == 6) && lane == 0)
      for (int r = open.first; r < open.last; r++) mbar_wait(&full_bar[r % S], (uint32_t)(r / S) & 1u, &late);
    if (warp == 1 && lane == 0) mbar_wait(&done_bar, 0u, &late);
    if (tid == 0) atomicExch(error, NGS_ERR_TIMEOUT);
    __syncwarp();
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_free(tmem, ncols_alloc);
  }
}

}  // namespace conv

// ----------------------------------------------------------------------------- gather GEMM (forward, input grad)
// out[r, n] = sum over offsets k with table[r, k] = i >= 0 of sum_c x[i, c] * bt[k, n, c]
// (forward: x = input features, bt = W[k]^T; input gradient: x = output gradient, table transposed,
// bt = W[k] as stored).  Grid: (row tiles, column tiles of 256).
struct GatherGemm {
  const uint16_t* x;
  int64_t n_src;
  int kdim;
  const int32_t* table;
  int64_t row_stride, k_stride;   // of the table: entry (row, k) at row * row_stride + k * k_stride
  int64_t n_rows;
  int K;
  const uint16_t* bt;
  int ncols;
  void* out;
  int out_f32;
  int bf16;
  int stages;
  uint32_t stage_bytes;
  int* error;
  int32_t oob;
};

// CP: rows of a tile that are copied with cp.async (a multiple of 16), the others by TMA.  48: 1.3M rows of 64 -> 64
// channels 776, 767 and 800 us with 32, 48 and 64 rows.  TMA gathers rows of an odd number of 16-byte pieces (8 channels
// more than a multiple of 16) at a fraction of its rate: these take 64, and 96 where an SM has more than one tile.
// 300,000 rows, us with 48 / 64 / 96 / 128 rows: 8 -> 16 channels 305 / 247 / 162 / 182, 72 -> 128 channels 544 / 479
// / 406 / 466; 10,000 rows: 28 / 26 / 26 / 31 and 53 / 48 / 56 / 65.
template <int CP>
__global__ void __launch_bounds__(conv::TMA_THREADS) conv_gather_gemm_kernel(const __grid_constant__ GatherGemm g,
                                                                            const __grid_constant__ CUtensorMap xmap,
                                                                            const __grid_constant__ CUtensorMap bmap) {
  using namespace conv;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  const int tid = threadIdx.x, lane = tid & 31;
  const int64_t r0 = (int64_t)blockIdx.x * BM;
  const int n0 = blockIdx.y * 256, rows = (int)min((int64_t)BM, g.n_rows - r0);
  const unsigned n_src = (unsigned)g.n_src;
  constexpr int TMA_ROWS = BM - CP;
  constexpr uint32_t half = TMA_ROWS / 8 * 512;         // bytes of a TMA warp's gathers
  TmaShape t{min(256, g.ncols - n0), g.stages, g.stage_bytes, {half + (uint32_t)min(256, g.ncols) * 128u, half}};

  // entries of rows 4 lane .. 4 lane + 3 at an offset: `oob`, a row out of the map's range (zeros), for missing ones
  const int32_t* const te = g.table + (r0 + 4 * lane) * g.row_stride;
  const int left = rows - 4 * lane;
  auto entries = [&](int k) {
    int v[4];
#pragma unroll
    for (int j = 0; j < 4; j++) v[j] = j < left && k < g.K ? __ldg(te + j * g.row_stride + k * g.k_stride) : -1;
    return make_int4(v[0], v[1], v[2], v[3]);
  };
  // the offsets with at least one pair in this tile (empty offsets cost nothing), each in chunks of 64 channels; the
  // next three offsets' entries are on their way meanwhile
  int k = -1, c0 = g.kdim;
  int4 src = make_int4(0, 0, 0, 0), ahead[3];
  auto setup = [&] {
#pragma unroll
    for (int i = 0; i < 3; i++) ahead[i] = entries(i);
  };
  auto next = [&]() -> int {
    if (c0 + BK < g.kdim) {
      c0 += BK;
      return min(BK, g.kdim - c0);
    }
    c0 = 0;
    do {
      if (++k >= g.K) return 0;
      src = ahead[0];
      ahead[0] = ahead[1];
      ahead[1] = ahead[2];
      ahead[2] = entries(k + 3);
      src.x = (unsigned)src.x < n_src ? src.x : g.oob;
      src.y = (unsigned)src.y < n_src ? src.y : g.oob;
      src.z = (unsigned)src.z < n_src ? src.z : g.oob;
      src.w = (unsigned)src.w < n_src ? src.w : g.oob;
    } while (!__any_sync(0xffffffffu, src.x != g.oob || src.y != g.oob || src.z != g.oob || src.w != g.oob));
    return min(BK, g.kdim);
  };
  auto issue = [&](uint8_t* a, uint64_t* bar, int w) {
    const uint32_t sa = smem_u32(a);
    if (w == 0 && lane == 31) tma_tile(sa + A_BYTES, &bmap, c0, k * g.ncols + n0, bar);
    if (lane / (TMA_ROWS / 8) == w) tma_gather4(sa + lane * 512, &xmap, c0, src.x, src.y, src.z, src.w, bar);
  };
  // eight lanes per row, one 16-byte piece each
  auto copy = [&](uint8_t* a, int w) {
    const uint32_t sa = smem_u32(a);
    const int piece = lane & 7, of4 = lane >> 3, e = c0 + piece * 8, quad0 = (TMA_ROWS + w * (CP / 4)) / 4;
#pragma unroll
    for (int j = 0; j < CP / 16; j++) {
      const int x = __shfl_sync(0xffffffffu, src.x, quad0 + j), y = __shfl_sync(0xffffffffu, src.y, quad0 + j);
      const int z = __shfl_sync(0xffffffffu, src.z, quad0 + j), u = __shfl_sync(0xffffffffu, src.w, quad0 + j);
      const int32_t v = of4 < 2 ? (of4 == 0 ? x : y) : (of4 == 2 ? z : u);
      const bool have = v != g.oob && e < g.kdim;
      cp_async16(sa + sw128((quad0 + j) * 4 + of4, piece), have ? g.x + (int64_t)v * g.kdim + e : g.x, have);
    }
  };
  auto store = [&](int row, int col, const float (&v)[16]) {
    if (row < rows) st16_row(g.out, g.out_f32 != 0, g.bf16, (r0 + row) * g.ncols + n0 + col, v);
  };
  run_tile_tma(t, smem, setup, next, issue, copy, store, g.bf16, g.error);
}

// ----------------------------------------------------------------------------- weight gradient
// part[k, split, m, n] = sum over the pairs p of offset k in the split's range of
// x[in(p), m0 + m] * gy[out(p), n0 + n]: A = the pairs' input rows transposed (rows m = input
// channels, reduction over pairs), B = their output-gradient rows transposed.  Grid: (splits,
// offsets, channel tiles).  The splits are summed in order by conv_wgrad_reduce_kernel.
struct WeightGrad {
  const uint16_t* x;         // [n_in, cin]
  const uint16_t* gy;        // [n_out, cout]
  int64_t n_in, n_out;
  int cin, cout;
  const int32_t* nbmaps;     // [P, 2]
  const int64_t* starts;     // [K + 1]
  int in_col;                // column of the input row in a pair (the other is the output row)
  int K;
  int splits;
  int m_tiles;               // ceil(cin / 128)
  float* part;               // [K, splits, cin, cout]
  int mn;                    // channels in multiples of 64: rows copied as they are into MN-major stages
  int bf16;
  int stages;
  uint32_t stage_bytes;
  int* error;
};

__global__ void __launch_bounds__(conv::THREADS, 1) conv_wgrad_kernel(const __grid_constant__ WeightGrad g) {
  using namespace conv;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  const int tid = threadIdx.x;
  const int split = blockIdx.x, k = blockIdx.y;
  const int m0 = (blockIdx.z % g.m_tiles) * BM, n0 = (blockIdx.z / g.m_tiles) * 256;
  const int N = min(256, g.cout - n0);
  const int64_t p_begin = __ldg(g.starts + k), p_count = __ldg(g.starts + k + 1) - p_begin;
  // this split's pairs, in whole chunks of 64
  const int64_t chunks = (p_count + BK - 1) / BK;
  const int64_t per = (chunks + g.splits - 1) / g.splits;
  const int64_t c_begin = min(chunks, (int64_t)split * per), c_end = min(chunks, c_begin + per);
  TileShape t{(int)(c_end - c_begin), N, g.stages, g.stage_bytes};

  // producer p: pair column kk = p % 64 of the stage, channel quarter q = p / 64 of the A rows (32
  // input channels) and of the B rows (N / 4 output channels); 16-bit values stored transposed
  auto fill = [&](int s, uint8_t* a, uint8_t* b, int p) -> int {
    const int64_t pc = (c_begin + s) * BK;              // first pair of the step (relative to p_begin)
    const int kk = p & 63, q = p >> 6;
    const int64_t pair = pc + kk;
    int32_t xi = -1, yo = -1;
    if (pair < p_count) {
      xi = __ldg(g.nbmaps + 2 * (p_begin + pair) + g.in_col);
      yo = __ldg(g.nbmaps + 2 * (p_begin + pair) + 1 - g.in_col);
    }
    const bool hx = xi >= 0 && xi < g.n_in, hy = yo >= 0 && yo < g.n_out;
    uint16_t* a16 = reinterpret_cast<uint16_t*>(a);
    uint16_t* b16 = reinterpret_cast<uint16_t*>(b);
    const int chunk = kk >> 3, within = kk & 7;
    for (int m = q * 32; m < q * 32 + 32; m++) {
      const int c = m0 + m;
      const uint16_t v = (hx && c < g.cin) ? __ldg(g.x + (int64_t)xi * g.cin + c) : (uint16_t)0;
      a16[(sw128(m, chunk) >> 1) + within] = v;
    }
    const int nq = N / 4;
    for (int n = q * nq; n < q * nq + nq; n++) {
      const int c = n0 + n;
      const uint16_t v = hy ? __ldg(g.gy + (int64_t)yo * g.cout + c) : (uint16_t)0;
      b16[(sw128(n, chunk) >> 1) + within] = v;
    }
    return (int)min((int64_t)BK, p_count - pc);
  };
  // MN-major form: the stage's K index is the pair, each 128-byte row 64 consecutive channels of one
  // pair, so a producer copies 16-byte pieces of its pairs' rows as they are (no transposition): eight
  // producers per 128 bytes, two pairs each.  Channels past cin are zeroed once, before the first step.
  const int prow = tid >> 3, pchunk = tid & 7;
  const int a_atoms = min(2, (g.cin - m0) / 64), b_atoms = N / 64;
  auto pairs = [&](int s, int32_t (&xi)[2], int32_t (&yo)[2]) {
#pragma unroll
    for (int j = 0; j < 2; j++) {
      const int64_t pair = (c_begin + s) * BK + prow + 32 * j;
      xi[j] = yo[j] = -1;
      if (pair < p_count) {
        xi[j] = __ldg(g.nbmaps + 2 * (p_begin + pair) + g.in_col);
        yo[j] = __ldg(g.nbmaps + 2 * (p_begin + pair) + 1 - g.in_col);
      }
    }
  };
  int32_t nx[2] = {-1, -1}, ny[2] = {-1, -1};
  const uint32_t at = sw128(prow, pchunk);
  const unsigned n_in = (unsigned)g.n_in, n_out = (unsigned)g.n_out;
  const uint16_t *x0 = g.x + m0 + pchunk * 8, *y0 = g.gy + n0 + pchunk * 8;
  if (g.mn) {
    if (a_atoms < 2)
      for (int st = 0; st < g.stages; st++)
        for (int i = tid; i < (int)MN_ATOM_BYTES / 16; i += THREADS)
          *reinterpret_cast<uint4*>(smem + (size_t)st * g.stage_bytes + MN_ATOM_BYTES + i * 16) = make_uint4(0, 0, 0, 0);
    fence_async_smem();
    if (tid < PRODUCERS && t.steps > 0) pairs(0, nx, ny);
  }
  auto fill_mn = [&](int s, uint8_t* a, uint8_t* b, int p) -> int {
    int32_t xi[2], yo[2];
#pragma unroll
    for (int j = 0; j < 2; j++) {
      xi[j] = nx[j];
      yo[j] = ny[j];
    }
    const uint32_t sa = smem_u32(a), sb = smem_u32(b);
    if (s + 1 < t.steps) pairs(s + 1, nx, ny);
#pragma unroll
    for (int j = 0; j < 2; j++) {
      const bool hx = (unsigned)xi[j] < n_in, hy = (unsigned)yo[j] < n_out;
      const uint16_t* xr = hx ? x0 + (int64_t)xi[j] * g.cin : g.x;
      const uint16_t* yr = hy ? y0 + (int64_t)yo[j] * g.cout : g.gy;
      for (int c = 0; c < a_atoms; c++) cp_async16(sa + c * MN_ATOM_BYTES + at + j * 4096, xr + (hx ? c * 64 : 0), hx);
      for (int c = 0; c < b_atoms; c++) cp_async16(sb + c * MN_ATOM_BYTES + at + j * 4096, yr + (hy ? c * 64 : 0), hy);
    }
    return (int)min((int64_t)BK, p_count - (c_begin + s) * BK);
  };
  float* part = g.part + ((int64_t)k * g.splits + split) * g.cin * g.cout;
  auto store = [&](int row, int col, const float (&v)[16]) {
    if (m0 + row < g.cin) {
      float4* o = reinterpret_cast<float4*>(part + (int64_t)(m0 + row) * g.cout + n0 + col);
#pragma unroll
      for (int j = 0; j < 4; j++) o[j] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
    }
  };
  if (g.mn) run_tile<true>(t, smem, fill_mn, store, g.bf16, g.error, true);
  else run_tile<false>(t, smem, fill, store, g.bf16, g.error);
}

// grad_w[k, c, n] = sum over splits (in order) of part[k, split, c, n]; FP32 or 16-bit out.
__global__ void conv_wgrad_reduce_kernel(const float* __restrict__ part, int K, int splits, int64_t cc, void* out,
                                         int out_f32, int bf16) {
  const int64_t total = (int64_t)K * cc;
  for (int64_t e = ngs_gtid(); e < total; e += ngs_gstride()) {
    const int64_t k = e / cc, j = e % cc;
    float acc = 0.f;
    for (int s = 0; s < splits; s++) acc += part[(k * splits + s) * cc + j];
    if (out_f32) static_cast<float*>(out)[e] = acc;
    else if (bf16) static_cast<__nv_bfloat16*>(out)[e] = __float2bfloat16_rn(acc);
    else static_cast<__half*>(out)[e] = __float2half_rn(acc);
  }
}

// ----------------------------------------------------------------------------- CUDA-core path
// FP32 inputs (the reference's path outside autocast is an FP32 cuBLAS GEMM, so FP32 stays FP32 here)
// and 16-bit shapes the tensor-core tiles do not take (kdim not a multiple of 8, ncols not a multiple
// of 16): FP32 multiply-adds on 4 x 4 outputs per thread, both operands staged through shared memory.
template <typename T>
NGS_DEV float to_f(T v) { return (float)v; }
template <>
NGS_DEV float to_f<__half>(__half v) { return __half2float(v); }
template <>
NGS_DEV float to_f<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }

template <typename T>
NGS_DEV void put(void* out, int64_t i, float v, bool f32) {
  if (f32) static_cast<float*>(out)[i] = v;
  else if constexpr (sizeof(T) == 2) static_cast<T*>(out)[i] = (T)v;
  else static_cast<float*>(out)[i] = v;
}

// Elements c .. c + 3 of a row of len elements as FP32, zero past its end; one 16-byte load for FP32
// rows that allow it (vec: len a multiple of 4 and the base 16-byte aligned).
template <typename T>
NGS_DEV float4 load4(const T* __restrict__ row, int c, int len, bool vec) {
  if constexpr (sizeof(T) == 4) {
    if (vec) return c < len ? __ldg(reinterpret_cast<const float4*>(row + c)) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  float4 v;
  v.x = c < len ? to_f(row[c]) : 0.f;
  v.y = c + 1 < len ? to_f(row[c + 1]) : 0.f;
  v.z = c + 2 < len ? to_f(row[c + 2]) : 0.f;
  v.w = c + 3 < len ? to_f(row[c + 3]) : 0.f;
  return v;
}
NGS_DEV bool finite4(float4 v) { return isfinite(v.x) && isfinite(v.y) && isfinite(v.z) && isfinite(v.w); }

// A tile of BM output rows x BN columns.  Per kernel offset that some row of the tile has, and per slice
// of CK channels: the rows gathered and the offset's weights into shared memory (both with the channel
// outermost), the next stage's loads in flight in registers while this one is multiplied.  A thread's
// sums run over the offsets and channels in order, as one thread per output would run them.  A missing
// row is staged as zeros, which adds nothing unless a weight is infinite or NaN: a stage with such a
// weight takes the rows one by one.
// What bounds it is the gather's latency over some 30 stages a tile.  Measured, FP32, 16 -> 32 channels,
// 44,595 rows, 702,000 pairs: forward 0.063 ms and input gradient 0.105 ms, against 0.83 ms each with one
// thread per output that reads its rows and weights for itself.
template <typename T, int BM, int BN, int CK>
__global__ void __launch_bounds__(BM* BN / 16) conv_gather_gemm_simt_kernel(
    const T* __restrict__ x, int64_t n_src, int kdim, const int32_t* __restrict__ table, int64_t row_stride,
    int64_t k_stride, int64_t n_rows, int K, const T* __restrict__ bt, int ncols, void* out, int out_f32, int vec) {
  constexpr int NT = BM * BN / 16;
  constexpr int NA = BM * CK / 4 / NT, NB = (BN * CK / 4 + NT - 1) / NT;
  __shared__ __align__(16) float As[CK][BM + 4];
  __shared__ __align__(16) float Bs[CK][BN + 4];
  __shared__ int s_valid[BM];
  __shared__ unsigned s_any[(conv::KMAX + 31) / 32];
  const int t = threadIdx.x, tx = t % (BN / 4), ty = t / (BN / 4);
  const int64_t r0 = (int64_t)blockIdx.x * BM;
  const int n0 = blockIdx.y * BN;
  for (int k = t; k < (conv::KMAX + 31) / 32; k += NT) s_any[k] = 0u;
  __syncthreads();
  const int rows = (int)min((int64_t)BM, n_rows - r0);
  for (int e = t; e < BM * K; e += NT) {
    const int row = e % BM, k = e / BM;
    if (row >= rows) continue;
    const int32_t src = table[(r0 + row) * row_stride + k * k_stride];
    if (src >= 0 && src < n_src) atomicOr(&s_any[k >> 5], 1u << (k & 31));
  }
  __syncthreads();
  auto next_k = [&](int k) {
    for (k++; k < K; k++)
      if ((s_any[k >> 5] >> (k & 31)) & 1u) break;
    return k;
  };
  float4 ra[NA], rb[NB];
  bool va = false;
  auto fetch = [&](int k, int c0) {
#pragma unroll
    for (int j = 0; j < NA; j++) {
      const int e = t + j * NT, row = e % BM, c = c0 + e / BM * 4;
      const int32_t src = row < rows ? __ldg(table + (r0 + row) * row_stride + k * k_stride) : -1;
      const bool ok = src >= 0 && src < n_src;
      if (j == 0) va = ok;                            // thread t < BM stages row t first
      ra[j] = ok ? load4<T>(x + (int64_t)src * kdim, c, kdim, vec) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int j = 0; j < NB; j++) {
      const int e = t + j * NT, n = e % BN, c = c0 + e / BN * 4;
      rb[j] = e < BN * CK / 4 && n0 + n < ncols ? load4<T>(bt + ((int64_t)k * ncols + n0 + n) * kdim, c, kdim, vec)
                                               : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  };
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) acc[i][j] = 0.f;
  int k = next_k(-1), c0 = 0;
  if (k < K) fetch(k, c0);
  while (k < K) {
    int odd = 0;
#pragma unroll
    for (int j = 0; j < NA; j++) {
      const int e = t + j * NT, row = e % BM, c = e / BM * 4;
      As[c][row] = ra[j].x;
      As[c + 1][row] = ra[j].y;
      As[c + 2][row] = ra[j].z;
      As[c + 3][row] = ra[j].w;
    }
    if (t < BM) s_valid[t] = va;
#pragma unroll
    for (int j = 0; j < NB; j++) {
      const int e = t + j * NT, n = e % BN, c = e / BN * 4;
      if (e < BN * CK / 4) {
        Bs[c][n] = rb[j].x;
        Bs[c + 1][n] = rb[j].y;
        Bs[c + 2][n] = rb[j].z;
        Bs[c + 3][n] = rb[j].w;
        odd |= !finite4(rb[j]);
      }
    }
    odd = __syncthreads_or(odd);
    c0 += CK;
    if (c0 >= kdim) {
      c0 = 0;
      k = next_k(k);
    }
    if (k < K) fetch(k, c0);                          // the next stage, while this one is multiplied
    bool use[4] = {true, true, true, true};
    if (odd) {
#pragma unroll
      for (int i = 0; i < 4; i++) use[i] = s_valid[ty * 4 + i] != 0;
    }
#pragma unroll 16
    for (int c = 0; c < CK; c++) {
      const float4 a4 = *reinterpret_cast<const float4*>(&As[c][ty * 4]);
      const float4 b4 = *reinterpret_cast<const float4*>(&Bs[c][tx * 4]);
      const float av[4] = {a4.x, a4.y, a4.z, a4.w}, bv[4] = {b4.x, b4.y, b4.z, b4.w};
      if (!odd) {
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
          for (int j = 0; j < 4; j++) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
      } else {
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
          for (int j = 0; j < 4; j++)
            if (use[i]) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const int row = ty * 4 + i;
    if (row >= rows) continue;
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int n = n0 + tx * 4 + j;
      if (n < ncols) put<T>(out, (r0 + row) * ncols + n, acc[i][j], out_f32 != 0);
    }
  }
}

// One thread per output, for layers too small to fill the tiles' pipeline: the same multiply-adds in the same order (a
// missing row is skipped instead of added as zeros).  STAGED: the table's entries of a block's rows go through shared
// memory, THREAD_OFFSETS offsets at a time.  Read by every thread for itself they are a sector each in a table with the
// offset outermost, and at few channels in they take longer than the rows.  Over 1,309 layers the staged form takes
// 0.9 to 1.0 times the other's (median by columns) from 4 columns on, and 1.1 times for fewer, whose block has as
// many rows as outputs.  FP32, staged and directly: 4 -> 16 channels, 3,000 rows 11.2 and 12.7 us; 24 -> 1, 150,000
// rows 191 and 101.
constexpr int THREAD_BLOCK = 256, THREAD_OFFSETS = 32, STAGED_COLUMNS = 4;

template <typename T, bool STAGED>
__global__ void __launch_bounds__(THREAD_BLOCK) conv_gather_gemm_thread_kernel(
    const T* __restrict__ x, int64_t n_src, int kdim, const int32_t* __restrict__ table, int64_t row_stride,
    int64_t k_stride, int64_t n_rows, int K, const T* __restrict__ bt, int ncols, void* out, int out_f32) {
  extern __shared__ int32_t s_entry[];         // [offset][row]
  const int64_t total = n_rows * ncols;
  for (int64_t e0 = (int64_t)blockIdx.x * THREAD_BLOCK; e0 < total; e0 += (int64_t)gridDim.x * THREAD_BLOCK) {
    const int64_t r0 = e0 / ncols;
    const int rows = (int)(min(e0 + THREAD_BLOCK, total) - 1 - r0 * ncols) / ncols + 1;
    const int own = (int)(e0 - r0 * ncols) + threadIdx.x, row = min(own / ncols, rows - 1), n = own - own / ncols * ncols;
    float acc = 0.f;
    auto add = [&](int k, int32_t src) {
      if (src < 0 || src >= n_src) return;
      const T* xr = x + (int64_t)src * kdim;
      const T* br = bt + ((int64_t)k * ncols + n) * kdim;
      for (int c = 0; c < kdim; c++) acc = fmaf(to_f(xr[c]), to_f(br[c]), acc);
    };
    if constexpr (STAGED) {
      for (int k0 = 0; k0 < K; k0 += THREAD_OFFSETS) {
        const int ks = min(THREAD_OFFSETS, K - k0);
        __syncthreads();
        for (int i = threadIdx.x; i < rows * ks; i += THREAD_BLOCK) {
          const int k = i / rows;
          s_entry[i] = __ldg(table + (r0 + i - k * rows) * row_stride + (k0 + k) * k_stride);
        }
        __syncthreads();
        for (int k = 0; k < ks; k++) add(k0 + k, s_entry[k * rows + row]);
      }
    } else {
      for (int k = 0; k < K; k++) add(k, __ldg(table + (r0 + row) * row_stride + k * k_stride));
    }
    if (e0 + threadIdx.x < total) put<T>(out, e0 + threadIdx.x, acc, out_f32 != 0);
  }
}

// Weight gradient: per offset a BM x BN tile of channels, the offset's pairs split over blockIdx.x (a
// partial per split, added in split order by conv_wgrad_reduce_kernel), a stage of 64 pairs in shared
// memory.  Tiles smaller than 128 threads' work are kept by several groups of threads, each on its share
// of a stage's pairs, added in group order.  A pair outside the feature maps is staged as two rows of
// zeros.  Measured on the same layer: 0.05 ms, against 7.8 ms with one thread per weight walking all pairs
// of its offset; the partial sums are short, so the error against 64 bits fell from 2.9e-6 to 4.1e-7.
constexpr int SIMT_PAIRS = 64;

template <typename T, int BM, int BN>
__global__ void __launch_bounds__(BM* BN / 16 < 128 ? 128 : BM * BN / 16) conv_wgrad_simt_kernel(
    const T* __restrict__ x, const T* __restrict__ gy, int64_t n_in, int64_t n_out, int cin, int cout,
    const int32_t* __restrict__ nbmaps, const int64_t* __restrict__ starts, int in_col, float* __restrict__ part,
    void* out, int out_f32, int vec_x, int vec_y) {
  constexpr int TT = BM * BN / 16, NT = TT < 128 ? 128 : TT, GROUPS = NT / TT;
  constexpr int NA = SIMT_PAIRS * BM / 4 / NT, NB = SIMT_PAIRS * BN / 4 / NT;
  union Stage {
    struct {
      float a[SIMT_PAIRS][BM];
      float b[SIMT_PAIRS][BN];
    } s;
    float sum[GROUPS][BM * BN];
  };
  __shared__ __align__(16) Stage sh;
  const int t = threadIdx.x, g = t / TT, tx = t % TT % (BN / 4), ty = t % TT / (BN / 4);
  const int k = blockIdx.y, split = blockIdx.x, splits = gridDim.x;
  const int nt = (cout + BN - 1) / BN, m0 = blockIdx.z / nt * BM, n0 = blockIdx.z % nt * BN;
  const int64_t first = starts[k], count = starts[k + 1] - first;
  const int64_t chunks = (count + SIMT_PAIRS - 1) / SIMT_PAIRS;
  const int64_t p_end = first + min(count, chunks * (split + 1) / splits * SIMT_PAIRS);
  int64_t p0 = first + chunks * split / splits * SIMT_PAIRS;
  float4 ra[NA], rb[NB];
  auto fetch = [&](int64_t p) {
#pragma unroll
    for (int j = 0; j < NA; j++) {
      const int e = t + j * NT, c = e % (BM / 4) * 4;
      const int64_t q = p + e / (BM / 4);
      ra[j] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (q < p_end) {
        const int32_t i = nbmaps[2 * q + in_col], o = nbmaps[2 * q + 1 - in_col];
        if (i >= 0 && i < n_in && o >= 0 && o < n_out) ra[j] = load4<T>(x + (int64_t)i * cin, m0 + c, cin, vec_x);
      }
    }
#pragma unroll
    for (int j = 0; j < NB; j++) {
      const int e = t + j * NT, c = e % (BN / 4) * 4;
      const int64_t q = p + e / (BN / 4);
      rb[j] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (q < p_end) {
        const int32_t i = nbmaps[2 * q + in_col], o = nbmaps[2 * q + 1 - in_col];
        if (i >= 0 && i < n_in && o >= 0 && o < n_out) rb[j] = load4<T>(gy + (int64_t)o * cout, n0 + c, cout, vec_y);
      }
    }
  };
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) acc[i][j] = 0.f;
  if (p0 < p_end) fetch(p0);
  for (; p0 < p_end; p0 += SIMT_PAIRS) {
#pragma unroll
    for (int j = 0; j < NA; j++) {
      const int e = t + j * NT;
      *reinterpret_cast<float4*>(&sh.s.a[e / (BM / 4)][e % (BM / 4) * 4]) = ra[j];
    }
#pragma unroll
    for (int j = 0; j < NB; j++) {
      const int e = t + j * NT;
      *reinterpret_cast<float4*>(&sh.s.b[e / (BN / 4)][e % (BN / 4) * 4]) = rb[j];
    }
    __syncthreads();
    if (p0 + SIMT_PAIRS < p_end) fetch(p0 + SIMT_PAIRS);
#pragma unroll 8
    for (int p = g; p < SIMT_PAIRS; p += GROUPS) {
      const float4 a4 = *reinterpret_cast<const float4*>(&sh.s.a[p][ty * 4]);
      const float4 b4 = *reinterpret_cast<const float4*>(&sh.s.b[p][tx * 4]);
      const float av[4] = {a4.x, a4.y, a4.z, a4.w}, bv[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) sh.sum[g][(ty * 4 + i) * BN + tx * 4 + j] = acc[i][j];
  __syncthreads();
  for (int e = t; e < BM * BN; e += NT) {
    const int m = m0 + e / BN, n = n0 + e % BN;
    if (m >= cin || n >= cout) continue;
    float v = 0.f;
#pragma unroll
    for (int h = 0; h < GROUPS; h++) v += sh.sum[h][e];
    if (part) part[(((int64_t)k * splits + split) * cin + m) * cout + n] = v;
    else put<T>(out, ((int64_t)k * cin + m) * cout + n, v, out_f32 != 0);
  }
}

template <typename T>
__global__ void conv_transpose_kernel(const T* __restrict__ w, int K, int a, int b, T* __restrict__ wt) {
  const int64_t total = (int64_t)K * a * b;
  for (int64_t e = ngs_gtid(); e < total; e += ngs_gstride()) {
    const int64_t k = e / ((int64_t)a * b), i = (e / b) % a, j = e % b;
    wt[(k * b + j) * a + i] = w[e];
  }
}

// ----------------------------------------------------------------------------- host entry points
namespace {

bool aligned16(const void* p) { return ((uintptr_t)p & 15u) == 0; }

// The tensor map of `rows` rows of `width` 16-bit elements, in boxes of 64 elements and `box` rows, swizzled over 128
// bytes, zeros out of range.  false where the driver refuses it.
bool rows_map(CUtensorMap& map, const void* base, int64_t width, int64_t rows, int box) {
  using Encode = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                              const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                              CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
  static const Encode encode = [] {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult found;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &found) != cudaSuccess ||
        found != cudaDriverEntryPointSuccess)
      fn = nullptr;
    return reinterpret_cast<Encode>(fn);
  }();
  if (!encode) return false;
  const cuuint64_t dims[2] = {(cuuint64_t)width, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)width * 2};
  const cuuint32_t boxes[2] = {conv::BK, (cuuint32_t)box}, steps[2] = {1, 1};
  return encode(&map, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, const_cast<void*>(base), dims, strides, boxes, steps,
                CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Dynamic shared memory of a tile kernel's block, at most (of 227 KB; the static arrays take the rest).  The kernels'
// limit is always set to this: threads share it, and one with a smaller need would lower it under another's launch.
constexpr int SMEM_MOST = 226 << 10;

// Stages of the ring for an N-column tile, and the dynamic shared memory of the launch.
void tile_plan(int n, int& stages, uint32_t& stage_bytes, size_t& smem) {
  const uint32_t nb = (uint32_t)((n + 7) / 8 * 8) * 128u;
  stage_bytes = (conv::A_BYTES + nb + 1023u) & ~1023u;
  stages = (int)((200u * 1024u) / stage_bytes);
  if (stages > 4) stages = 4;
  if (stages < 2) stages = 2;
  smem = (size_t)stages * stage_bytes + 1024;        // + alignment of the first stage to 1024 bytes
}

// Column tile of the CUDA-core kernels: the smallest of 16, 32 and 64 that holds the columns (a narrower
// tile than the columns need would gather the rows once more, a wider one multiplies zeros).
template <typename T, int BM, int BN>
int simt_gemm_tile(const GatherGemm& g, cudaStream_t st) {
  const dim3 grid((unsigned)((g.n_rows + BM - 1) / BM), (unsigned)((g.ncols + BN - 1) / BN));
  const T* x = reinterpret_cast<const T*>(g.x);
  const T* bt = reinterpret_cast<const T*>(g.bt);
  // slices of 32 channels where there are more than 16: half the stages, and a stage is a round trip
  const int vec = g.kdim % 4 == 0 && aligned16(x) && aligned16(bt);
  ngs_count_launch();
  if (g.kdim <= 16)
    conv_gather_gemm_simt_kernel<T, BM, BN, 16><<<grid, BM * BN / 16, 0, st>>>(
        x, g.n_src, g.kdim, g.table, g.row_stride, g.k_stride, g.n_rows, g.K, bt, g.ncols, g.out, g.out_f32, vec);
  else
    conv_gather_gemm_simt_kernel<T, BM, BN, 32><<<grid, BM * BN / 16, 0, st>>>(
        x, g.n_src, g.kdim, g.table, g.row_stride, g.k_stride, g.n_rows, g.K, bt, g.ncols, g.out, g.out_f32, vec);
  NGS_CHECK_LAUNCH();
  return NGS_OK;
}

template <typename T>
int simt_gemm(const GatherGemm& g, cudaStream_t st) {
  if (conv::simt_by_thread(g.n_rows, g.kdim, g.ncols, sizeof(T))) {
    ngs_count_launch();
    const bool staged = g.ncols >= STAGED_COLUMNS;
    const int rows = (THREAD_BLOCK - 1) / g.ncols + 2;                 // of a block's outputs, at most
    const auto kernel = staged ? conv_gather_gemm_thread_kernel<T, true> : conv_gather_gemm_thread_kernel<T, false>;
    kernel<<<ngs_blocks(g.n_rows * g.ncols, THREAD_BLOCK), THREAD_BLOCK,
             staged ? rows * std::min(g.K, THREAD_OFFSETS) * sizeof(int32_t) : 0, st>>>(
        reinterpret_cast<const T*>(g.x), g.n_src, g.kdim, g.table, g.row_stride, g.k_stride, g.n_rows, g.K,
        reinterpret_cast<const T*>(g.bt), g.ncols, g.out, g.out_f32);
    NGS_CHECK_LAUNCH();
    return NGS_OK;
  }
  if (g.ncols <= 16) return simt_gemm_tile<T, 64, 16>(g, st);
  if (g.ncols <= 32) return simt_gemm_tile<T, 64, 32>(g, st);
  return simt_gemm_tile<T, 64, 64>(g, st);
}

// Splits of an offset's pairs, each with a partial result in the workspace: of at least `least` pairs each, at most 64.
int wgrad_splits(int64_t max_pairs, int64_t least) {
  const int64_t s = (max_pairs + least - 1) / least;
  return (int)(s < 1 ? 1 : (s > 64 ? 64 : s));
}

// On the tensor cores splits of 2,048 pairs; on the CUDA cores of 512 while offsets, channel tiles and splits together
// are no more than SIMT_BLOCKS, some 16 blocks an SM: more of them add partials to write and to read, not blocks that
// run.
constexpr int SIMT_BLOCKS = 2400;

int simt_tile(int channels) { return channels <= 16 ? 16 : channels <= 32 ? 32 : 64; }

int simt_splits(int K, int cin, int cout, int64_t max_pairs) {
  const int bm = simt_tile(cin), bn = simt_tile(cout);
  const int64_t tiles = (int64_t)K * ((cin + bm - 1) / bm) * ((cout + bn - 1) / bn);
  return (int)std::min<int64_t>(wgrad_splits(max_pairs, 512), (SIMT_BLOCKS + tiles - 1) / tiles);
}

bool wgrad_tensor_cores(int cout, int dtype) { return (dtype == NGS_F16 || dtype == NGS_BF16) && cout % 16 == 0; }

template <typename T, int BM, int BN>
void simt_wgrad_tile(const void* x, const void* gy, int64_t n_in, int64_t n_out, int cin, int cout,
                     const int32_t* nbmaps, const int64_t* starts, int in_col, int K, int splits, float* part,
                     void* out, int out_f32, cudaStream_t st) {
  const dim3 grid((unsigned)splits, (unsigned)K, (unsigned)(((cin + BM - 1) / BM) * ((cout + BN - 1) / BN)));
  ngs_count_launch();
  conv_wgrad_simt_kernel<T, BM, BN><<<grid, BM * BN / 16 < 128 ? 128 : BM * BN / 16, 0, st>>>(
      static_cast<const T*>(x), static_cast<const T*>(gy), n_in, n_out, cin, cout, nbmaps, starts, in_col, part, out,
      out_f32, cin % 4 == 0 && aligned16(x), cout % 4 == 0 && aligned16(gy));
}

template <typename T>
int simt_wgrad(const void* x, const void* gy, int64_t n_in, int64_t n_out, int cin, int cout, const int32_t* nbmaps,
               const int64_t* starts, int in_col, int K, int64_t max_pairs, void* out, int out_f32, void* ws,
               size_t ws_bytes, cudaStream_t st) {
  // as many splits as the workspace holds partials for, one (written in place) without a workspace
  const size_t one = (size_t)K * cin * cout * sizeof(float);
  const int splits = ws && aligned16(ws) ? (int)std::max<size_t>(1, std::min<size_t>(simt_splits(K, cin, cout, max_pairs), ws_bytes / one)) : 1;
  float* part = splits > 1 ? static_cast<float*>(ws) : nullptr;
  auto go = [&](auto bm, auto bn) {
    simt_wgrad_tile<T, decltype(bm)::value, decltype(bn)::value>(x, gy, n_in, n_out, cin, cout, nbmaps, starts, in_col,
                                                                 K, splits, part, out, out_f32, st);
  };
  auto with_bm = [&](auto bm) {
    if (simt_tile(cout) == 16) go(bm, std::integral_constant<int, 16>{});
    else if (simt_tile(cout) == 32) go(bm, std::integral_constant<int, 32>{});
    else go(bm, std::integral_constant<int, 64>{});
  };
  if (simt_tile(cin) == 16) with_bm(std::integral_constant<int, 16>{});
  else if (simt_tile(cin) == 32) with_bm(std::integral_constant<int, 32>{});
  else with_bm(std::integral_constant<int, 64>{});
  NGS_CHECK_LAUNCH();
  if (part) {
    ngs_count_launch();
    conv_wgrad_reduce_kernel<<<ngs_blocks((int64_t)K * cin * cout, 256), 256, 0, st>>>(
        part, K, splits, (int64_t)cin * cout, out, out_f32, std::is_same<T, __nv_bfloat16>::value);
    NGS_CHECK_LAUNCH();
  }
  return NGS_OK;
}

}  // namespace

extern "C" int ngs_conv_transpose_weight(const void* w, int K, int a, int b, int dtype, void* wt, ngs_stream s) {
  if (!w || !wt || K < 1 || a < 1 || b < 1 || dtype < NGS_F16 || dtype > NGS_F32) return NGS_ERR_INVALID_ARG;
  cudaStream_t st = (cudaStream_t)s;
  const int64_t total = (int64_t)K * a * b;
  ngs_count_launch();
  if (dtype == NGS_F32)
    conv_transpose_kernel<float><<<ngs_blocks(total, 256), 256, 0, st>>>(static_cast<const float*>(w), K, a, b,
                                                                        static_cast<float*>(wt));
  else
    conv_transpose_kernel<uint16_t><<<ngs_blocks(total, 256), 256, 0, st>>>(static_cast<const uint16_t*>(w), K, a, b,
                                                                           static_cast<uint16_t*>(wt));
  NGS_CHECK_LAUNCH();
  return NGS_OK;
}

extern "C" int ngs_conv_tensor_core_ok(int kdim, int ncols, int dtype) {
  return (dtype == NGS_F16 || dtype == NGS_BF16) && kdim >= 8 && kdim % 8 == 0 && ncols >= 16 && ncols % 16 == 0;
}

static int conv_gather_gemm(const void* x, int64_t n_src, int kdim, const int32_t* table, int64_t row_stride,
                            int64_t k_stride, int64_t n_rows, int K, const void* bt, int ncols, int dtype, void* out,
                            int out_f32, int* error_dev, cudaStream_t st) {
  if (n_src < 0 || n_rows < 0 || kdim < 1 || ncols < 1 || K < 1 || K > conv::KMAX || dtype < NGS_F16 ||
      dtype > NGS_F32 || (n_rows > 0 && (!table || !out || !bt)) || (n_src > 0 && !x) || !error_dev)
    return NGS_ERR_INVALID_ARG;
  if (n_rows == 0) return NGS_OK;
  GatherGemm g{};
  g.x = static_cast<const uint16_t*>(n_src > 0 ? x : bt);   // a valid address also where every row is missing
  g.n_src = n_src;
  g.kdim = kdim;
  g.table = table;
  g.row_stride = row_stride;
  g.k_stride = k_stride;
  g.n_rows = n_rows;
  g.K = K;
  g.bt = static_cast<const uint16_t*>(bt);
  g.ncols = ncols;
  g.out = out;
  g.out_f32 = out_f32 || dtype == NGS_F32;
  g.bf16 = dtype == NGS_BF16;
  g.error = error_dev;
  CUtensorMap xmap, bmap;
  const int box = std::min(ncols, 256);
  if (!ngs_conv_tensor_core_ok(kdim, ncols, dtype) || !aligned16(x) || !aligned16(bt) || !aligned16(out) ||
      !rows_map(xmap, g.x, kdim, std::max<int64_t>(n_src, 1), 1) || !rows_map(bmap, bt, kdim, (int64_t)K * ncols, box)) {
    if (dtype == NGS_F32) return simt_gemm<float>(g, st);
    if (dtype == NGS_BF16) return simt_gemm<__nv_bfloat16>(g, st);
    return simt_gemm<__half>(g, st);
  }
  g.oob = n_src < 0x7fffffff ? (int32_t)std::max<int64_t>(n_src, 1) : -1;
  const conv::GatherPlan plan = conv::gather_plan(box);
  g.stages = plan.stages;
  g.stage_bytes = plan.stage_bytes;
  const auto kernel = kdim % 16 == 0 ? conv_gather_gemm_kernel<48>
                      : n_rows <= (int64_t)ngs_num_sms() * conv::BM ? conv_gather_gemm_kernel<64> : conv_gather_gemm_kernel<96>;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_MOST) != cudaSuccess)
    return ngs_set_cuda_error(cudaGetLastError());
  const dim3 grid((unsigned)((n_rows + conv::BM - 1) / conv::BM), (unsigned)((ncols + 255) / 256));
  ngs_count_launch();
  kernel<<<grid, conv::TMA_THREADS, plan.smem, st>>>(g, xmap, bmap);
  NGS_CHECK_LAUNCH();
  return NGS_OK;
}

extern "C" int ngs_conv_gather_gemm(const void* x, int64_t n_src, int kdim, const int32_t* table, int64_t n_rows, int K,
                                    const void* bt, int ncols, int dtype, void* out, int out_f32, int* error_dev,
                                    ngs_stream s) {
  return conv_gather_gemm(x, n_src, kdim, table, K, 1, n_rows, K, bt, ncols, dtype, out, out_f32, error_dev,
                          (cudaStream_t)s);
}

extern "C" int ngs_conv_gather_gemm_kmajor(const void* x, int64_t n_src, int kdim, const int32_t* table,
                                           int64_t n_rows, int K, const void* bt, int ncols, int dtype, void* out,
                                           int out_f32, int* error_dev, ngs_stream s) {
  return conv_gather_gemm(x, n_src, kdim, table, 1, n_rows, n_rows, K, bt, ncols, dtype, out, out_f32, error_dev,
                          (cudaStream_t)s);
}

extern "C" size_t ngs_conv_weight_grad_ws_bytes(int K, int cin, int cout, int64_t max_pairs) {
  return (size_t)K * wgrad_splits(max_pairs, 2048) * cin * cout * sizeof(float);
}

extern "C" size_t ngs_conv_weight_grad_ws_bytes_of(int K, int cin, int cout, int64_t max_pairs, int dtype) {
  if (K < 1 || cin < 1 || cout < 1 || max_pairs < 0) return 0;
  const int splits = wgrad_tensor_cores(cout, dtype) ? wgrad_splits(max_pairs, 2048) : simt_splits(K, cin, cout, max_pairs);
  return (size_t)K * splits * cin * cout * sizeof(float);
}

extern "C" int ngs_conv_weight_grad(const void* x, int64_t n_in, int cin, const void* gy, int64_t n_out, int cout,
                                    const int32_t* nbmaps, const int64_t* starts_dev, int K, int64_t max_pairs,
                                    int in_col, int dtype, void* grad_w, int out_f32, void* ws, size_t ws_bytes,
                                    int* error_dev, ngs_stream s) {
  if (n_in < 0 || n_out < 0 || cin < 1 || cout < 1 || K < 1 || K > conv::KMAX || max_pairs < 0 ||
      (in_col != 0 && in_col != 1) || dtype < NGS_F16 || dtype > NGS_F32 || !starts_dev || !grad_w || !error_dev ||
      (max_pairs > 0 && !nbmaps) || (n_in > 0 && !x) || (n_out > 0 && !gy))
    return NGS_ERR_INVALID_ARG;
  cudaStream_t st = (cudaStream_t)s;
  if (!wgrad_tensor_cores(cout, dtype) || !aligned16(grad_w)) {
    if (dtype == NGS_F32)
      return simt_wgrad<float>(x, gy, n_in, n_out, cin, cout, nbmaps, starts_dev, in_col, K, max_pairs, grad_w, 1, ws,
                               ws_bytes, st);
    if (dtype == NGS_BF16)
      return simt_wgrad<__nv_bfloat16>(x, gy, n_in, n_out, cin, cout, nbmaps, starts_dev, in_col, K, max_pairs, grad_w,
                                       out_f32, ws, ws_bytes, st);
    return simt_wgrad<__half>(x, gy, n_in, n_out, cin, cout, nbmaps, starts_dev, in_col, K, max_pairs, grad_w, out_f32,
                              ws, ws_bytes, st);
  }
  const int splits = wgrad_splits(max_pairs, 2048);
  const size_t need = (size_t)K * splits * cin * cout * sizeof(float);
  if (!ws || ws_bytes < need) return NGS_ERR_OOM;
  WeightGrad g{};
  g.x = static_cast<const uint16_t*>(n_in > 0 ? x : grad_w);     // a valid address also where every pair is skipped
  g.gy = static_cast<const uint16_t*>(n_out > 0 ? gy : grad_w);
  g.n_in = n_in;
  g.n_out = n_out;
  g.cin = cin;
  g.cout = cout;
  g.nbmaps = nbmaps;
  g.starts = starts_dev;
  g.in_col = in_col;
  g.K = K;
  g.splits = splits;
  g.m_tiles = (cin + conv::BM - 1) / conv::BM;
  g.part = static_cast<float*>(ws);
  g.mn = cin % 64 == 0 && cout % 64 == 0 && aligned16(x) && aligned16(gy);
  g.bf16 = dtype == NGS_BF16;
  g.error = error_dev;
  size_t smem = 0;
  tile_plan(cout < 256 ? cout : 256, g.stages, g.stage_bytes, smem);
  if (cudaFuncSetAttribute(conv_wgrad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_MOST) != cudaSuccess)
    return ngs_set_cuda_error(cudaGetLastError());
  const dim3 grid((unsigned)g.splits, (unsigned)K, (unsigned)(g.m_tiles * ((cout + 255) / 256)));
  ngs_count_launch();
  conv_wgrad_kernel<<<grid, conv::THREADS, smem, st>>>(g);
  NGS_CHECK_LAUNCH();
  ngs_count_launch();
  conv_wgrad_reduce_kernel<<<ngs_blocks((int64_t)K * cin * cout, 256), 256, 0, st>>>(g.part, K, g.splits, (int64_t)cin * cout, grad_w,
                                                                  out_f32, g.bf16);
  NGS_CHECK_LAUNCH();
  return NGS_OK;
}
