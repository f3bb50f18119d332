// Galerkin assembly of the screened-Poisson system on one level
// (jspsr/core/reconstructor.py:122-189, jspsr/bases/bezier_tensor.py:75-121).
//
// Layout: CSR over the lexicographically sorted voxels of the level; the
// columns of a row are its present neighbours in the 5x5x5 stencil, in
// lexicographic offset order, hence sorted.  A 128-bit mask per row records
// which of the 125 offsets are present, so the CSR slot of any (row, offset)
// pair is rowptr + popc(mask below offset) -- the screening Gram product
// therefore adds straight into the matrix instead of going through the
// reference's second hash table keyed by (row, col) pairs.
#include "ngs_common.cuh"


// ----------------------------------------------------------------------------- structure
// One warp per row: lane l < 25 owns the stencil column (dx, dy) = (l / 5 - 2, l % 5 - 2) and its
// five cells along z (offsets o = 5 l .. 5 l + 4 in lexicographic order), found with one or two
// bitmap words; a warp scan of the lanes' counts gives every lane its first CSR slot, so the row's
// entries are written by consecutive lanes.
NGS_DEV void stencil_column(const ngs_grid& g, const int32_t* __restrict__ coords, int64_t i, int lane,
                            int32_t (&r)[5]) {
  const int cx = coords[i * 3], cy = coords[i * 3 + 1], cz = coords[i * 3 + 2];
  if (lane < 25)
    grid_rows_zrun<5>(g, cx + (lane / 5 - 2) * g.stride, cy + (lane % 5 - 2) * g.stride, cz - 2 * g.stride, r);
  else
    for (int t = 0; t < 5; t++) r[t] = -1;
}

__global__ void stencil_count_kernel(ngs_grid g, const int32_t* __restrict__ coords, int64_t V,
                                     uint4* __restrict__ masks, int64_t* __restrict__ counts) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t i = ngs_gtid() >> 5; i < V; i += warps) {
    int32_t r[5];
    stencil_column(g, coords, i, lane, r);
    // lane l's column fills mask bits 5l .. 5l+4 (cell t of the column at bit 5l + t); each of the
    // four 32-bit words is the OR of the lanes' shifted patterns
    unsigned pat = 0u;
#pragma unroll
    for (int t = 0; t < 5; t++) pat |= (r[t] >= 0 ? 1u : 0u) << t;
    const int lo = 5 * lane;
    unsigned w[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const int sh = lo - 32 * k;             // position of the pattern's bit 0 in word k
      const unsigned part = sh >= 32 || sh <= -5 ? 0u : (sh >= 0 ? pat << sh : pat >> -sh);
      w[k] = __reduce_or_sync(0xffffffffu, part);
    }
    const unsigned total = __reduce_add_sync(0xffffffffu, (unsigned)__popc(pat));
    if (lane == 0) {
      masks[i] = make_uint4(w[0], w[1], w[2], w[3]);
      counts[i] = (int64_t)total;
    }
  }
}

__global__ void stencil_fill_kernel(ngs_grid g, const int32_t* __restrict__ coords, int64_t V,
                                    const uint4* __restrict__ masks, const int64_t* __restrict__ rowptr,
                                    const double* __restrict__ stencil, int32_t* __restrict__ cols,
                                    double* __restrict__ vals, int64_t* __restrict__ diag_slot) {
  __shared__ double st[125];
  for (int t = threadIdx.x; t < 125; t += blockDim.x) st[t] = stencil[t];
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t i = ngs_gtid() >> 5; i < V; i += warps) {
    int32_t r[5];
    stencil_column(g, coords, i, lane, r);
    int c = 0;
#pragma unroll
    for (int t = 0; t < 5; t++) c += r[t] >= 0 ? 1 : 0;
    int pre = c;                                      // inclusive warp scan of the counts
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, pre, d);
      if (lane >= d) pre += y;
    }
    int64_t slot = rowptr[i] + (pre - c);
#pragma unroll
    for (int t = 0; t < 5; t++) {
      if (r[t] < 0) continue;
      const int o = 5 * lane + t;
      cols[slot] = r[t];
      vals[slot] = st[o];
      if (o == 62) diag_slot[i] = slot;
      slot++;
    }
  }
}

extern "C" int ngs_stencil_count(ngs_grid g, const int32_t* coords, int64_t V, uint32_t* masks, int64_t* counts,
                                 ngs_stream s) {
  if (!g.words || V < 0 || (V > 0 && (!coords || !masks || !counts))) return NGS_ERR_INVALID_ARG;
  if (V == 0) return NGS_OK;
  { ngs_count_launch(); stencil_count_kernel<<<ngs_blocks(V * 32, 256), 256, 0, (cudaStream_t)s>>>(g, coords, V, reinterpret_cast<uint4*>(masks),
                                                                       counts); }
  NGS_CHECK_LAUNCH();
  return NGS_OK;
}

extern "C" int ngs_stencil_fill(ngs_grid g, const int32_t* coords, int64_t V, const uint32_t* masks,
                                const int64_t* rowptr, const double* stencil125, int32_t* cols, double* vals,
                                int64_t* diag_slot, ngs_stream s) {
  if (!g.words || V < 0 || (V > 0 && (!coords || !masks || !rowptr || !stencil125 || !cols || !vals || !diag_slot)))
    return NGS_ERR_INVALID_ARG;
  if (V == 0) return NGS_OK;
  { ngs_count_launch(); stencil_fill_kernel<<<ngs_blocks(V * 32, 256), 256, 0, (cudaStream_t)s>>>(
      g, coords, V, reinterpret_cast<const uint4*>(masks), rowptr, stencil125, cols, vals, diag_slot); }
  NGS_CHECK_LAUNCH();
  return NGS_OK;
}

// ----------------------------------------------------------------------------- screening
// One warp per point; lane a (< 27) owns the point's neighbour a and adds
// w * phi_a * phi_b into row a for every present neighbour b.
__global__ void screen_gram_kernel(const int32_t* __restrict__ rows, const float* __restrict__ phi, int64_t n,
                                   const float* __restrict__ w, const uint4* __restrict__ masks,
                                   const int64_t* __restrict__ rowptr, double scale, double* __restrict__ vals) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t p = ngs_gtid() >> 5; p < n; p += warps) {
    const int32_t ra = lane < 27 ? rows[p * 27 + lane] : -1;
    const float pa = lane < 27 ? phi[p * 27 + lane] : 0.f;
    const double sa = scale * (double)(w ? w[p] : 1.f) * (double)pa;
    uint4 m = make_uint4(0, 0, 0, 0);
    int64_t base = 0;
    if (ra >= 0) {
      m = masks[ra];
      base = rowptr[ra];
    }
    const int ax = lane / 9, ay = (lane / 3) % 3, az = lane % 3;
#pragma unroll 3
    for (int b = 0; b < 27; b++) {
      const int32_t rb = __shfl_sync(0xffffffffu, ra, b);
      const float pb = __shfl_sync(0xffffffffu, pa, b);
      if (ra < 0 || rb < 0) continue;
      const int bx = b / 9, by = (b / 3) % 3, bz = b % 3;
      const int o = (bx - ax + 2) * 25 + (by - ay + 2) * 5 + (bz - az + 2);
      atomicAdd(vals + base + popc_below(m, o), sa * (double)pb);
    }
  }
}

extern "C" int ngs_screen_gram(const int32_t* rows, const float* phi, int64_t n, const float* w, const uint32_t* masks,
                               const int64_t* rowptr, double scale, double* vals, ngs_stream s) {
  if (n < 0 || (n > 0 && (!rows || !phi || !masks || !rowptr || !vals))) return NGS_ERR_INVALID_ARG;
  if (n == 0) return NGS_OK;
  { ngs_count_launch(); screen_gram_kernel<<<ngs_blocks(n * 32, 256), 256, 0, (cudaStream_t)s>>>(
      rows, phi, n, w, reinterpret_cast<const uint4*>(masks), rowptr, scale, vals); }
  NGS_CHECK_LAUNCH();
  return NGS_OK;
}

// The cell key of each point: its first present neighbour row * 27 + that neighbour's position, or
// -1 when none of the 27 is present.  Points in one cell share all 27 rows, so the key identifies
// the cell (the cell is the first present neighbour's voxel minus that position's offset).
__global__ void point_cell_keys_kernel(const int32_t* __restrict__ rows, int64_t n, int64_t* __restrict__ keys) {
  for (int64_t p = ngs_gtid(); p < n; p += ngs_gstride()) {
    int64_t key = -1;
    for (int a = 0; a < 27; a++) {
      const int32_t r = rows[p * 27 + a];
      if (r >= 0) {
        key = (int64_t)r * 27 + a;
        break;
      }
    }
    keys[p] = key;
  }
}

extern "C" int ngs_point_cell_keys(const int32_t* rows, int64_t n, int64_t* keys, ngs_stream s) {
  if (n < 0 || (n > 0 && (!rows || !keys))) return NGS_ERR_INVALID_ARG;
  if (n == 0) return NGS_OK;
  { ngs_count_launch(); point_cell_keys_kernel<<<ngs_blocks(n, 256), 256, 0, (cudaStream_t)s>>>(rows, n, keys); }
  NGS_CHECK_LAUNCH();
  return NGS_OK;
}

// Points sorted by cell key: each warp takes a contiguous share of the sorted positions, lane a (< 27)
// works for the cell's neighbour a, and a run of equal keys within the share is summed in registers and
// added at its end.  Positions per warp: enough warps for every SM first, then longer shares (fewer runs
// cut, fewer atomics on the rows of coarse levels, where millions of points share a cell).
static int64_t group_share(int64_t n, int warps_per_sm, int64_t most) {
  const int64_t want = (int64_t)ngs_num_sms() * warps_per_sm, share = (n + want - 1) / want;
  return share < 1 ? 1 : (share > most ? most : share);
}
constexpr int GROUP_BATCH = 8;             // points whose 27 values are in flight together
constexpr int GROUP_WARPS = 4;

// Walks a warp's share of the sorted positions, 32 at a time (one position per lane, coalesced), their
// values phi[point, lane] GROUP_BATCH at a time (through `stage`, GROUP_BATCH rows of 32):
// head(point) at the first point of every run, add(scale_p, value) at every point, tail() after the last one
// of a run.  scale_p = scale * w[p] * field[p].
template <typename Head, typename Add, typename Tail>
NGS_DEV void walk_groups(float (*stage)[32], const float* __restrict__ phi, int64_t n, const float* __restrict__ w,
                         const float* __restrict__ field, const int64_t* __restrict__ order,
                         const int64_t* __restrict__ keys, double scale, int64_t share, Head head, Add add, Tail tail) {
  const int lane = threadIdx.x & 31, la = min(lane, 26);          // lanes 27 .. 31 follow lane 26
  const int64_t begin = (ngs_gtid() >> 5) * share, end = min(n, begin + share);
  int64_t last = -1;                                              // key of the open run
  for (int64_t i = begin; i < end; i += 32) {                     // warp-uniform
    const int64_t key = i + lane < end ? keys[i + lane] : -1;
    const int32_t p = key >= 0 ? (int32_t)order[i + lane] : 0;
    double sp = scale;
    if (key >= 0 && w) sp *= (double)w[p];
    if (key >= 0 && field) sp *= (double)field[p];
    int64_t prev = __shfl_up_sync(0xffffffffu, key, 1);
    if (lane == 0) prev = last;
    const unsigned valid = __ballot_sync(0xffffffffu, key >= 0);
    const unsigned heads = __ballot_sync(0xffffffffu, key >= 0 && key != prev);
    const int m = 32 - __clz(valid);
    for (int j0 = 0; j0 < m; j0 += GROUP_BATCH) {
      float v[GROUP_BATCH];
#pragma unroll
      for (int j = 0; j < GROUP_BATCH; j++) {
        const int32_t q = __shfl_sync(0xffffffffu, p, j0 + j);
        v[j] = (valid >> (j0 + j)) & 1u ? phi[(int64_t)q * 27 + la] : 0.f;
      }
      __syncwarp();
#pragma unroll
      for (int j = 0; j < GROUP_BATCH; j++) stage[j][lane] = v[j];
      // not unrolled: the code that ends a run is there once
#pragma unroll 1
      for (int j = j0; j < min(m, j0 + GROUP_BATCH); j++) {
        if (!((valid >> j) & 1u)) continue;
        if ((heads >> j) & 1u) {
          if (last >= 0) tail();
          last = 0;
          head(__shfl_sync(0xffffffffu, p, j));
        }
        add(__shfl_sync(0xffffffffu, sp, j), stage[j - j0][lane]);
      }
    }
    if (valid) last = __shfl_sync(0xffffffffu, key, m - 1);
  }
  if (last >= 0) tail();
}

// The same sum with the points grouped by their 27-voxel neighbourhood: points in one cell share all
// 27 rows, so each (row, column) slot takes one atomic per run instead of one per point.  order / keys:
// the points sorted by key = first present row * 27 + its position (-1: no voxel), a key that fixes the
// cell.  The Gram is symmetric and 27 is odd: lane a sums the 14 pairs (a, a + t mod 27), t = 0 .. 13, which
// are all pairs once (each value converted to FP64 once, by its own lane); at the end of a run the sums go
// through shared memory to the lanes that add them to their rows.  On fine levels (1 to 3 points a run) the
// 729 atomics of a run bound it, on coarse ones the shuffles.  Measured: 5M points, 11 levels: 26 ms, of
// which 1.0 each on the 8 coarse levels (101 ms with a warp per sorted position and 27 conversions and
// products per lane and point); 300,000 points, 4 levels: 2.15 ms (2.09).  The code that ends a run has to
// stay small and be there once: unrolled over the points of a batch it took 4.9 to 13 ms.
struct GramRow {
  ulonglong2 mask;                         // of the row's stencil offsets
  int64_t base;                            // its first slot, -1: no such row
};

__global__ void __launch_bounds__(GROUP_WARPS * 32, 6) screen_gram_grouped_kernel(
    const int32_t* __restrict__ rows, const float* __restrict__ phi, int64_t n, const float* __restrict__ w,
    const int64_t* __restrict__ order, const int64_t* __restrict__ keys, const uint4* __restrict__ masks,
    const int64_t* __restrict__ rowptr, double scale, double* __restrict__ vals, int64_t share) {
  __shared__ GramRow s_row[GROUP_WARPS][27];
  __shared__ double s_sum[GROUP_WARPS][14][27];
  __shared__ float s_stage[GROUP_WARPS][GROUP_BATCH][32];
  const int lane = threadIdx.x & 31, la = min(lane, 26);
  double(*sum)[27] = s_sum[threadIdx.x >> 5];
  const int ob = 62 + la / 9 * 25 + (la / 3) % 3 * 5 + la % 3;    // offset of (a, b): ob - the same sum of a
  GramRow* row = s_row[threadIdx.x >> 5];
  double acc[14];
#pragma unroll
  for (int t = 0; t < 14; t++) acc[t] = 0.0;
  int32_t rb = -1;
  walk_groups(
      s_stage[threadIdx.x >> 5], phi, n, w, nullptr, order, keys, 1.0, share, [&](int32_t p) { rb = rows[(int64_t)p * 27 + la]; },
      [&](double sp, float v) {
        const double pa = (double)v, sa = sp * pa;
        acc[0] += sa * pa;
#pragma unroll
        for (int t = 1; t < 14; t++)
          acc[t] += sa * __shfl_sync(0xffffffffu, pa, la + t < 27 ? la + t : la + t - 27);
      },
      [&]() {
        __syncwarp();
#pragma unroll
        for (int t = 0; t < 14; t++) {
          if (lane < 27) sum[t][lane] = acc[t];
          acc[t] = 0.0;
        }
        if (lane < 27) {
          row[lane].base = rb >= 0 ? rowptr[rb] : -1;
          if (rb >= 0) row[lane].mask = *reinterpret_cast<const ulonglong2*>(masks + rb);
        }
        __syncwarp();
        // one row a at a time, lane b adding to column b: the row's 27 slots lie in 9 runs of 3, some 10
        // sectors to an atomic instruction (with a row per lane each slot is a sector of its own)
#pragma unroll 3
        for (int a = 0; a < 27; a++) {
          const ulonglong2 m = row[a].mask;
          if (row[a].base < 0 || lane >= 27 || rb < 0) continue;
          const int t = la >= a ? la - a : la - a + 27;           // b = a + t mod 27, or a = b + (27 - t) mod 27
          const double v = t < 14 ? sum[t][a] : sum[27 - t][la];
          const int o = ob - (a / 9 * 25 + (a / 3) % 3 * 5 + a % 3);
          const int below = o < 64 ? __popcll(m.x & ((1ull << o) - 1ull))
                                   : __popcll(m.x) + __popcll(m.y & ((1ull << (o - 64)) - 1ull));
          atomicAdd(vals + row[a].base + below, scale * v);
        }
      });
}

extern "C" int ngs_screen_gram_grouped(const int32_t* rows, const float* phi, int64_t n, const float* w,
                                       const int64_t* order, const int64_t* keys, const uint32_t* masks,
                                       const int64_t* rowptr, double scale, double* vals, ngs_stream s) {
  if (n < 0 || (n > 0 && (!rows || !phi || !order || !keys || !masks || !rowptr || !vals))) return NGS_ERR_INVALID_ARG;
  if (n == 0) return NGS_OK;
  const int64_t share = group_share(n, 32, 128);
  { ngs_count_launch(); screen_gram_grouped_kernel<<<(unsigned)((n + GROUP_WARPS * share - 1) / (GROUP_WARPS * share)), GROUP_WARPS * 32, 0,
                                                    (cudaStream_t)s>>>(
      rows, phi, n, w, order, keys, reinterpret_cast<const uint4*>(masks), rowptr, scale, vals, share); }
  NGS_CHECK_LAUNCH();
  return NGS_OK;
}

__global__ void screen_rhs_kernel(const int32_t* __restrict__ rows, const float* __restrict__ phi, int64_t n,
                                  const float* __restrict__ w, const float* __restrict__ field, double scale,
                                  double* __restrict__ rhs) {
  const int64_t total = n * 27;
  for (int64_t t = ngs_gtid(); t < total; t += ngs_gstride()) {
    const int32_t r = rows[t];
    if (r < 0) continue;
    const int64_t p = t / 27;
    double v = scale * (double)phi[t];
    if (w) v *= (double)w[p];
    if (field) v *= (double)field[p];
    atomicAdd(rhs + r, v);
  }
}

// Screening RHS terms over the points sorted by cell key (the Gram's order / keys), shared out to the
// warps as the Gram's points are: lane a sums the run's terms of neighbour a, one atomic per (run, row).
// (A point per lane and a segmented warp scan per neighbour took 270 shuffles for 32 points; here a point
// costs one load and one multiply-add per lane: 300,000 points, 7 launches: 0.30 ms against 0.42; 5M points,
// 21 launches: 8.5 against 26.8.)
__global__ void __launch_bounds__(GROUP_WARPS * 32) screen_rhs_grouped_kernel(
    const int32_t* __restrict__ rows, const float* __restrict__ phi, int64_t n, const float* __restrict__ w,
    const float* __restrict__ field, const int64_t* __restrict__ order, const int64_t* __restrict__ keys,
    double scale, double* __restrict__ rhs, int64_t share) {
  __shared__ float s_stage[GROUP_WARPS][GROUP_BATCH][32];
  const int lane = threadIdx.x & 31, la = min(lane, 26);
  double acc = 0.0;
  int32_t r = -1;
  walk_groups(
      s_stage[threadIdx.x >> 5], phi, n, w, field, order, keys, scale, share, [&](int32_t p) { r = rows[(int64_t)p * 27 + la]; },
      [&](double sp, float v) { acc += sp * (double)v; },
      [&]() {
        if (lane < 27 && r >= 0) atomicAdd(rhs + r, acc);
        acc = 0.0;
      });
}

extern "C" int ngs_screen_rhs_grouped(const int32_t* rows, const float* phi, int64_t n, const float* w,
                                      const float* field, const int64_t* order, const int64_t* keys, double scale,
                                      double* rhs, ngs_stream s) {
  if (n < 0 || (n > 0 && (!rows || !phi || !order || !keys || !rhs))) return NGS_ERR_INVALID_ARG;
  if (n == 0) return NGS_OK;
  const int64_t share = group_share(n, 48, 256);
  { ngs_count_launch(); screen_rhs_grouped_kernel<<<(unsigned)((n + GROUP_WARPS * share - 1) / (GROUP_WARPS * share)), GROUP_WARPS * 32, 0,
                                                    (cudaStream_t)s>>>(
      rows, phi, n, w, field, order, keys, scale, rhs, share); }
  NGS_CHECK_LAUNCH();
  return NGS_OK;
}

extern "C" int ngs_screen_rhs(const int32_t* rows, const float* phi, int64_t n, const float* w, double scale,
                              double* rhs, ngs_stream s) {
  if (n < 0 || (n > 0 && (!rows || !phi || !rhs))) return NGS_ERR_INVALID_ARG;
  if (n == 0) return NGS_OK;
  { ngs_count_launch(); screen_rhs_kernel<<<ngs_blocks(n * 27, 256), 256, 0, (cudaStream_t)s>>>(rows, phi, n, w, nullptr, scale, rhs); }
  NGS_CHECK_LAUNCH();
  return NGS_OK;
}

extern "C" int ngs_correction_screen(const int32_t* rows, const float* phi, int64_t n, const float* w,
                                     const float* field, double scale, double* rhs, ngs_stream s) {
  if (n < 0 || (n > 0 && (!rows || !phi || !field || !rhs))) return NGS_ERR_INVALID_ARG;
  if (n == 0) return NGS_OK;
  { ngs_count_launch(); screen_rhs_kernel<<<ngs_blocks(n * 27, 256), 256, 0, (cudaStream_t)s>>>(rows, phi, n, w, field, -scale, rhs); }
  NGS_CHECK_LAUNCH();
  return NGS_OK;
}

// ----------------------------------------------------------------------------- RHS from normals
// target stride >= data stride: scatter from every data voxel to the 27 target voxels around the
// target cell that holds the data voxel's centre (get_coords_neighbours, _hash_backend.py:194-228).
// Data voxels come in lexicographic order, so consecutive ones often share the target cell (always, for a
// coarse target level): a warp takes a contiguous share of them, lane k (< 27) sums the terms of the cell's
// neighbour k and adds them when the cell changes.  The voxels' coordinates are read and their table
// values looked up 32 voxels at a time, one per lane, and passed to the neighbours' lanes through shared
// memory: nine reads and a dozen FP64 operations per voxel and lane.  (A voxel per lane and a segmented
// warp scan per neighbour took 270 shuffles for 32 voxels; lanes that look the tables up themselves took
// more time for level ratios from 16 on.)
// 1.2M data voxels and 3 target levels: 0.59 ms in all against 0.75; a room's 10.6M and 10: 12.6 against 68.7.
constexpr int SCATTER_WARPS = 4;
__global__ void __launch_bounds__(SCATTER_WARPS * 32) rhs_scatter_kernel(
    const int32_t* __restrict__ dc, int64_t nd, int sd, const float* __restrict__ nrm, ngs_grid tg,
    const double* __restrict__ tc, const double* __restrict__ tgv, int tab_len, double* __restrict__ rhs,
    int64_t share) {
  __shared__ double s_tab[SCATTER_WARPS][21][33];                 // [axis * 6 + k * 2 + (c, g)], [18 + axis]: normal
  __shared__ double s_open[SCATTER_WARPS][4][32];
  __shared__ int s_cell[SCATTER_WARPS][4][4];
  double(*tab)[33] = s_tab[threadIdx.x >> 5];
  const int st = tg.stride, M = st / sd;
  const int lane = threadIdx.x & 31, la = min(lane, 26);          // lanes 27 .. 31 follow lane 26 and add nothing
  const int kx = la / 9, ky = (la / 3) % 3, kz = la % 3;
  const int64_t begin = (ngs_gtid() >> 5) * share, end = min(nd, begin + share);
  // Four cells are open at a time, by the low bits of their place along z: a column of voxels that meets a
  // floor and a ceiling goes back and forth between two cells, and on a coarse level every flush adds to
  // the same few rows (10.6M voxels of a room onto 256: 7.8 ms with one open cell, 0.8 with four).
  double(*open_sum)[32] = s_open[threadIdx.x >> 5];
  int(*cell)[4] = s_cell[threadIdx.x >> 5];                       // x, y, z of the open cells, and whether there is one
  if (lane < 4) cell[lane][3] = 0;
  __syncwarp();
  double acc = 0.0;
  int cur = -1;                                                   // the cell that acc belongs to
  auto flush = [&](int e, double v) {
    const int64_t t = grid_row(tg, cell[e][0] + (kx - 1) * st, cell[e][1] + (ky - 1) * st, cell[e][2] + (kz - 1) * st);
    if (lane < 27 && t >= 0 && v != 0.0) atomicAdd(rhs + t, -v);
  };
  int p0 = 0, p1 = 0, p2 = 0;                                     // the voxel before this batch
  for (int64_t i = begin; i < end; i += 32) {                     // warp-uniform
    const int64_t v = min(i + lane, end - 1);
    int q[3];
    __syncwarp();
#pragma unroll
    for (int a = 0; a < 3; a++) {
      const int c = dc[v * 3 + a];
      q[a] = (int)floorf(((float)c + 0.5f * (float)sd) / (float)st) * st;
#pragma unroll
      for (int k = 0; k < 3; k++) {
        // rel = (k-1)*M + (q - c)/sd + (M-1)/2 ; idx = rel + (3M-1)/2  (integer)
        const int idx = (k - 1) * M + (q[a] - c) / sd + 2 * M - 1;
        const bool ok = idx >= 0 && idx < tab_len;
        tab[a * 6 + k * 2][lane] = ok ? __ldg(tc + idx) : 0.0;
        tab[a * 6 + k * 2 + 1][lane] = ok ? __ldg(tgv + idx) : 0.0;
      }
      tab[18 + a][lane] = nrm[v * 3 + a];
    }
    __syncwarp();
    int u0 = __shfl_up_sync(0xffffffffu, q[0], 1), u1 = __shfl_up_sync(0xffffffffu, q[1], 1),
        u2 = __shfl_up_sync(0xffffffffu, q[2], 1);
    if (lane == 0) {
      u0 = p0;
      u1 = p1;
      u2 = p2;
    }
    const int m = (int)min((int64_t)32, end - i);
    unsigned heads = __ballot_sync(0xffffffffu, q[0] != u0 || q[1] != u1 || q[2] != u2);
    if (cur < 0) heads |= 1u;
    p0 = __shfl_sync(0xffffffffu, q[0], 31);
    p1 = __shfl_sync(0xffffffffu, q[1], 31);
    p2 = __shfl_sync(0xffffffffu, q[2], 31);
#pragma unroll 1
    for (int j = 0; j < m; j++) {
      if ((heads >> j) & 1u) {
        const int c0 = __shfl_sync(0xffffffffu, q[0], j), c1 = __shfl_sync(0xffffffffu, q[1], j),
                  c2 = __shfl_sync(0xffffffffu, q[2], j);
        const int e = (c2 >> tg.log2_stride) & 3;
        if (cur >= 0) open_sum[cur][lane] = acc;
        const bool taken = cell[e][3] != 0;
        const bool same = taken && cell[e][0] == c0 && cell[e][1] == c1 && cell[e][2] == c2;
        acc = taken ? open_sum[e][lane] : 0.0;
        if (!same) {
          if (taken) flush(e, acc);
          acc = 0.0;
          __syncwarp();
          if (lane == 0) {
            cell[e][0] = c0;
            cell[e][1] = c1;
            cell[e][2] = c2;
            cell[e][3] = 1;
          }
          __syncwarp();
        }
        cur = e;
      }
      const double cx = tab[kx * 2][j], cy = tab[6 + ky * 2][j], cz = tab[12 + kz * 2][j];
      acc += tab[18][j] * tab[kx * 2 + 1][j] * cy * cz + tab[19][j] * cx * tab[6 + ky * 2 + 1][j] * cz +
             tab[20][j] * cx * cy * tab[12 + kz * 2 + 1][j];
    }
  }
  if (cur >= 0) open_sum[cur][lane] = acc;
#pragma unroll 1
  for (int e = 0; e < 4; e++)
    if (cell[e][3]) flush(e, open_sum[e][lane]);
}

// target stride < data stride (coarse data, fine target): gather per target voxel over the coarse
// data voxels whose centre lies within 1.5 fine voxels (the inverted map, _hash_backend.py:254-262).
__global__ void rhs_gather_kernel(ngs_grid dg, const float* __restrict__ nrm, const int32_t* __restrict__ tcoords,
                                  int64_t nt, int st, const double* __restrict__ tc, const double* __restrict__ tgv,
                                  int tab_len, double* __restrict__ rhs) {
  const int sd = dg.stride, M = sd / st;
  for (int64_t i = ngs_gtid(); i < nt; i += ngs_gstride()) {
    int q[3], c[3];
#pragma unroll
    for (int a = 0; a < 3; a++) {
      c[a] = tcoords[i * 3 + a];
      q[a] = (int)floorf(((float)c[a] + 0.5f * (float)st) / (float)sd) * sd;
    }
    double acc = 0.0;
    for (int kx = -1; kx <= 1; kx++)
      for (int ky = -1; ky <= 1; ky++)
        for (int kz = -1; kz <= 1; kz++) {
          const int k[3] = {kx, ky, kz};
          double cv[3], gv[3];
          bool ok = true;
#pragma unroll
          for (int a = 0; a < 3; a++) {
            // nt = k*M + (q - c)/st + (M-1)/2 (fine units), keep |nt| < 1.5;
            // rel = -nt * st / sd ; idx = rel * M + M/2 + 0.5 = -nt + M/2 + 0.5 (integer)
            const int two_nt = 2 * (k[a] * M + (q[a] - c[a]) / st) + (M - 1);
            ok &= (two_nt > -3 - 1 && two_nt < 3 + 1) && (abs(two_nt) <= 3);
            const int idx = (-two_nt + M + 1) / 2;
            ok &= (idx >= 0 && idx < tab_len);
            cv[a] = ok ? tc[idx] : 0.0;
            gv[a] = ok ? tgv[idx] : 0.0;
          }
          if (!ok) continue;
          const int64_t d = grid_row(dg, q[0] + kx * sd, q[1] + ky * sd, q[2] + kz * sd);
          if (d < 0) continue;
          const double n0 = nrm[d * 3], n1 = nrm[d * 3 + 1], n2 = nrm[d * 3 + 2];
          acc += n0 * gv[0] * cv[1] * cv[2] + n1 * cv[0] * gv[1] * cv[2] + n2 * cv[0] * cv[1] * gv[2];
        }
    rhs[i] -= acc;
  }
}

// target stride == data stride: every data voxel D scatters to the targets D + k stride, k in
// {-1, 0, 1}^3, so each target T gathers from the data voxels T - k stride instead -- 9 runs of 3
// cells along z, no atomics, a fixed summation order.  The table index of offset k is k + 1.
__global__ void rhs_same_level_kernel(ngs_grid dg, const float* __restrict__ nrm, const int32_t* __restrict__ tcoords,
                                      int64_t nt, const double* __restrict__ tc, const double* __restrict__ tgv,
                                      double* __restrict__ rhs) {
  const int s = dg.stride;
  for (int64_t i = ngs_gtid(); i < nt; i += ngs_gstride()) {
    const int c0 = tcoords[i * 3], c1 = tcoords[i * 3 + 1], c2 = tcoords[i * 3 + 2];
    double acc = 0.0;
#pragma unroll
    for (int jx = -1; jx <= 1; jx++)
#pragma unroll
      for (int jy = -1; jy <= 1; jy++) {
        int32_t r[3];
        grid_rows_zrun<3>(dg, c0 + jx * s, c1 + jy * s, c2 - s, r);
#pragma unroll
        for (int jz = -1; jz <= 1; jz++) {
          const int32_t d = r[jz + 1];
          if (d < 0) continue;
          // data voxel D = T + j s sees the target at offset k = -j: table index 1 - j
          const double cx = tc[1 - jx], cy = tc[1 - jy], cz = tc[1 - jz];
          const double gx = tgv[1 - jx], gy = tgv[1 - jy], gz = tgv[1 - jz];
          const double n0 = nrm[(int64_t)d * 3], n1 = nrm[(int64_t)d * 3 + 1], n2 = nrm[(int64_t)d * 3 + 2];
          acc += n0 * gx * cy * cz + n1 * cx * gy * cz + n2 * cx * cy * gz;
        }
      }
    rhs[i] -= acc;
  }
}

extern "C" int ngs_rhs_normals(ngs_grid data_grid, const int32_t* data_coords, int64_t n_data, const float* normals,
                               ngs_grid tgt_grid, const int32_t* tgt_coords, int64_t n_tgt, const double* tab_c,
                               const double* tab_g, int tab_len, double* rhs, ngs_stream s) {
  if (!normals || !tab_c || !tab_g || !rhs || tab_len <= 0) return NGS_ERR_INVALID_ARG;
  cudaStream_t st = (cudaStream_t)s;
  if (tgt_grid.stride == data_grid.stride && tgt_coords && data_grid.words && tab_len == 3) {
    if (n_tgt <= 0 || n_data <= 0) return NGS_OK;
    { ngs_count_launch(); rhs_same_level_kernel<<<ngs_blocks(n_tgt, 128), 128, 0, st>>>(data_grid, normals, tgt_coords, n_tgt,
                                                                                       tab_c, tab_g, rhs); }
  } else if (tgt_grid.stride >= data_grid.stride) {
    if (n_data <= 0) return NGS_OK;
    if (!data_coords || !tgt_grid.words) return NGS_ERR_INVALID_ARG;
    // shares of 32 to 1024 voxels: enough warps first, then longer runs
    int64_t share = (n_data + 32 * (int64_t)ngs_num_sms() - 1) / (32 * (int64_t)ngs_num_sms());
    share = ((share < 32 ? 32 : (share > 1024 ? 1024 : share)) + 31) & ~(int64_t)31;
    { ngs_count_launch(); rhs_scatter_kernel<<<(unsigned)((n_data + SCATTER_WARPS * share - 1) / (SCATTER_WARPS * share)),
                                             SCATTER_WARPS * 32, 0, st>>>(
        data_coords, n_data, data_grid.stride, normals, tgt_grid, tab_c, tab_g, tab_len, rhs, share); }
  } else {
    if (n_tgt <= 0) return NGS_OK;
    if (!tgt_coords || !data_grid.words) return NGS_ERR_INVALID_ARG;
    { ngs_count_launch(); rhs_gather_kernel<<<ngs_blocks(n_tgt, 128), 128, 0, st>>>(data_grid, normals, tgt_coords, n_tgt, tgt_grid.stride,
                                                              tab_c, tab_g, tab_len, rhs); }
  }
  NGS_CHECK_LAUNCH();
  return NGS_OK;
}

// ----------------------------------------------------------------------------- cross-level correction
// rhs_fine[i] -= sum over the 125 coarse neighbours j of K(i, j) * x_coarse[j]
// (reconstructor.py:153-168, stiffness part; computed matrix-free).
// 64 registers (eight 128-thread blocks per SM, no spills): more resident warps to wait on the bitmap
// runs and gathers (0.89 -> 0.82 ms for the 300k cloud).
__global__ void __launch_bounds__(128, 8) correction_kernel(const int32_t* __restrict__ fc, int64_t nf, int sf, ngs_grid cg,
                                  const float* __restrict__ x, const double* __restrict__ tc,
                                  const double* __restrict__ tg, int tab_len, double* __restrict__ rhs) {
  extern __shared__ double tabs[];
  for (int t = threadIdx.x; t < tab_len; t += blockDim.x) {
    tabs[t] = tc[t];
    tabs[tab_len + t] = tg[t];
  }
  __syncthreads();
  const int sc = cg.stride, M = sc / sf;
  for (int64_t i = ngs_gtid(); i < nf; i += ngs_gstride()) {
    int q[3], base[3];
#pragma unroll
    for (int a = 0; a < 3; a++) {
      const int c = fc[i * 3 + a];
      q[a] = (int)floorf(((float)c + 0.5f * (float)sf) / (float)sc) * sc;
      // idx = rel + 1.5M + 0.5 with rel = k*M + (q - c)/sf + (M-1)/2  ->  k*M + (q - c)/sf + 2M
      base[a] = (q[a] - c) / sf + 2 * M;
    }
    double acc = 0.0;
    for (int kx = -2; kx <= 2; kx++) {
      const int ix = kx * M + base[0];
      if (ix < 0 || ix >= tab_len) continue;
      for (int ky = -2; ky <= 2; ky++) {
        const int iy = ky * M + base[1];
        if (iy < 0 || iy >= tab_len) continue;
        int32_t rz[5];                       // the 5 coarse cells along z, one or two bitmap words
        grid_rows_zrun<5>(cg, q[0] + kx * sc, q[1] + ky * sc, q[2] - 2 * sc, rz);
        // K = g_x c_y c_z + c_x g_y c_z + c_x c_y g_z = A c_z + B g_z for the column (kx, ky)
        const double A = tabs[tab_len + ix] * tabs[iy] + tabs[ix] * tabs[tab_len + iy];
        const double B = tabs[ix] * tabs[iy];
#pragma unroll
        for (int kz = -2; kz <= 2; kz++) {
          const int iz = kz * M + base[2];
          if (iz < 0 || iz >= tab_len) continue;
          const int64_t j = rz[kz + 2];
          if (j < 0) continue;
          acc += (A * tabs[iz] + B * tabs[tab_len + iz]) * (double)x[j];
        }
      }
    }
    rhs[i] -= acc;
  }
}

extern "C" int ngs_correction_stiffness(const int32_t* fine_coords, int64_t n_fine, int fine_stride, ngs_grid cg,
                                        const float* x_coarse, const double* tab_c, const double* tab_g, int tab_len,
                                        double* rhs, ngs_stream s) {
  // tables of 3M + 2 entries each: level ratios M up to 2^12 (13 levels) fit one block's shared memory
  constexpr int MOST = 12290;
  if (n_fine < 0 || fine_stride <= 0 || cg.stride <= fine_stride || tab_len <= 0 || tab_len > MOST)
    return NGS_ERR_INVALID_ARG;
  if (n_fine == 0) return NGS_OK;
  if (!fine_coords || !cg.words || !x_coarse || !tab_c || !tab_g || !rhs) return NGS_ERR_INVALID_ARG;
  const size_t smem = 2 * (size_t)tab_len * sizeof(double);
  if (smem > 48 * 1024) {
    // the same limit for every call: another thread's launch may stand between this one's two steps
    const cudaError_t e = cudaFuncSetAttribute(correction_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               2 * MOST * (int)sizeof(double));
    if (e != cudaSuccess) return ngs_set_cuda_error(e);
  }
  { ngs_count_launch(); correction_kernel<<<ngs_blocks(n_fine, 128), 128, smem, (cudaStream_t)s>>>(
      fine_coords, n_fine, fine_stride, cg, x_coarse, tab_c, tab_g, tab_len, rhs); }
  NGS_CHECK_LAUNCH();
  return NGS_OK;
}

// ----------------------------------------------------------------------------- finish
__global__ void finish_kernel(const double* __restrict__ v64, int64_t nnz, const int64_t* __restrict__ diag_slot,
                              int64_t V, float* __restrict__ v32, float* __restrict__ inv_diag) {
  for (int64_t i = ngs_gtid(); i < nnz; i += ngs_gstride()) v32[i] = (float)v64[i];
  for (int64_t i = ngs_gtid(); i < V; i += ngs_gstride()) inv_diag[i] = (float)(1.0 / v64[diag_slot[i]]);
}

extern "C" int ngs_finish_system(const double* vals64, int64_t nnz, const int64_t* diag_slot, int64_t V, float* vals32,
                                 float* inv_diag, ngs_stream s) {
  if (nnz < 0 || V < 0 || (nnz > 0 && (!vals64 || !vals32)) || (V > 0 && (!diag_slot || !inv_diag)))
    return NGS_ERR_INVALID_ARG;
  if (nnz == 0 && V == 0) return NGS_OK;
  { ngs_count_launch(); finish_kernel<<<ngs_blocks(nnz > V ? nnz : V, 256), 256, 0, (cudaStream_t)s>>>(vals64, nnz, diag_slot, V, vals32,
                                                                                inv_diag); }
  NGS_CHECK_LAUNCH();
  return NGS_OK;
}

__global__ void inv_diag_kernel(const double* __restrict__ v64, const int64_t* __restrict__ diag_slot, int64_t n,
                                float* __restrict__ inv_diag) {
  for (int64_t i = ngs_gtid(); i < n; i += ngs_gstride()) inv_diag[i] = (float)(1.0 / v64[diag_slot[i]]);
}

// 1 / (sum of a row's entries on the diagonal) of any CSR, eight lanes a row.  As torch operations (row of every
// entry, mask, two selections with their synchronisations, scatter) this took 0.30 of the 1.72 ms of a direct-solve
// replacement with 7M entries; bound by the 12 bytes of an entry's column (and the values on the diagonal).
__global__ void diag_inv_kernel(const int64_t* __restrict__ rp, const int32_t* __restrict__ cols,
                                const double* __restrict__ vals, int64_t n, float* __restrict__ inv_diag) {
  const int sub = threadIdx.x & 7;
  const unsigned mask = 0xffu << (threadIdx.x & 24);
  for (int64_t row = ngs_gtid() >> 3; row < n; row += ngs_gstride() >> 3) {
    double d = 0.0;
    const int64_t end = rp[row + 1];
#pragma unroll 4
    for (int64_t j = rp[row] + sub; j < end; j += 8)
      if (cols[j] == row) d += vals[j];
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) d += __shfl_xor_sync(mask, d, o);
    if (sub == 0) inv_diag[row] = (float)(1.0 / d);
  }
}

extern "C" int ngs_csr_diag_inv(const int64_t* rowptr, const int32_t* cols, const double* vals64, int64_t n,
                                float* inv_diag, ngs_stream s) {
  if (n < 0 || (n > 0 && (!rowptr || !cols || !vals64 || !inv_diag))) return NGS_ERR_INVALID_ARG;
  if (n == 0) return NGS_OK;
  { ngs_count_launch(); diag_inv_kernel<<<ngs_blocks(n * 8, 256), 256, 0, (cudaStream_t)s>>>(rowptr, cols, vals64, n, inv_diag); }
  NGS_CHECK_LAUNCH();
  return NGS_OK;
}

extern "C" int ngs_csr_inv_diag(const double* vals64, const int64_t* diag_slot, int64_t n, float* inv_diag,
                                ngs_stream s) {
  if (n < 0 || (n > 0 && (!vals64 || !diag_slot || !inv_diag))) return NGS_ERR_INVALID_ARG;
  if (n == 0) return NGS_OK;
  { ngs_count_launch(); inv_diag_kernel<<<ngs_blocks(n, 256), 256, 0, (cudaStream_t)s>>>(vals64, diag_slot, n, inv_diag); }
  NGS_CHECK_LAUNCH();
  return NGS_OK;
}
