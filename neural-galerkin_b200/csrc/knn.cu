// Exact k-nearest-neighbour search and signed distance from oriented points, on a uniform cell grid.
//
// Replaces the FLANN-derived CUDA k-d tree of the reference (csrc/common/kdtree_cuda.cu:1071-1279,
// built and queried by ext/sdfgen/sdf_from_points.cu:70-116) and its voting kernel
// (ext/sdfgen/sdf_from_points.cu:31-68): the ground-truth occupancy of the training loop
// (models/full_net.py:135-142 calls it with k = 8, stdv = 0.02).
//
// Layout: the reference points are bucketed by a cubic cell of side h.  The occupied cells form a
// rank bitmap (ngs_grid, stride 1 in cell units), so a cell's bucket is found with one 128-bit load;
// a counting sort (counts by atomics, an exclusive scan, a scatter) lays the points out cell by cell.
// A query walks Chebyshev rings of cells around its own cell, keeping the k best (squared distance,
// point index) pairs in registers -- ties broken by the smaller index, so the result does not depend
// on the order of points inside a bucket -- and stops once k are held and the k-th distance is at
// most r h: every point of ring r + 1 or beyond is farther than r h from a query inside the centre
// cell.  The ring walk is clipped to the grid's box, and ends when the box is covered.
//
// This grid walk serves callers of the C ABI that keep a cell index; jspsr.sdfgen uses the box tree at the
// end of this file.
//
// The signed distance follows the reference exactly: magnitude from the nearest neighbour p0,
// |n0 . (q - p0)| when |q - p0| < stdv, else |q - p0|; sign negative unless more than k / 2 of the
// k neighbours see the query on the positive side of their normal (n . (q - p) > 0).
#include "ngs_common.cuh"
#include "scan.cuh"

constexpr int KNN_MAX_K = 32;

__global__ void knn_mark_cells_kernel(ngs_grid g, const float* __restrict__ xyz, int64_t n, float inv_h) {
  unsigned long long* words = reinterpret_cast<unsigned long long*>(g.words);
  for (int64_t i = ngs_gtid(); i < n; i += ngs_gstride()) {
    int bit;
    const int64_t w = grid_word_index(g, (int)floorf(xyz[3 * i] * inv_h), (int)floorf(xyz[3 * i + 1] * inv_h),
                                      (int)floorf(xyz[3 * i + 2] * inv_h), &bit);
    if (w >= 0) atomicOr(words + 2 * w + 1, 1ull << bit);
  }
}

__global__ void knn_bucket_kernel(ngs_grid g, const float* __restrict__ xyz, int64_t n, float inv_h,
                                  int32_t* __restrict__ cell_of, int32_t* __restrict__ cell_count) {
  for (int64_t i = ngs_gtid(); i < n; i += ngs_gstride()) {
    const int64_t r = grid_row(g, (int)floorf(xyz[3 * i] * inv_h), (int)floorf(xyz[3 * i + 1] * inv_h),
                               (int)floorf(xyz[3 * i + 2] * inv_h));
    cell_of[i] = (int32_t)r;
    if (r >= 0) atomicAdd(cell_count + r, 1);
  }
}

__global__ void knn_scatter_kernel(const int32_t* __restrict__ cell_of, int64_t n, const int64_t* __restrict__ start,
                                   int32_t* __restrict__ cursor, int32_t* __restrict__ sorted) {
  for (int64_t i = ngs_gtid(); i < n; i += ngs_gstride()) {
    const int32_t c = cell_of[i];
    if (c >= 0) sorted[start[c] + atomicAdd(cursor + c, 1)] = (int32_t)i;
  }
}

// (d2, idx) ordering: smaller distance first, then smaller index
NGS_DEV bool knn_less(float da, int ia, float db, int ib) { return da < db || (da == db && ia < ib); }

__global__ void knn_sdf_kernel(ngs_grid g, const int64_t* __restrict__ start, const int32_t* __restrict__ sorted,
                               const float* __restrict__ ref, const float* __restrict__ nrm,
                               const float* __restrict__ q, int64_t nq, float inv_h, float h, int k, float stdv,
                               int32_t* __restrict__ idx_out, float* __restrict__ d2_out, float* __restrict__ sdf_out) {
  for (int64_t i = ngs_gtid(); i < nq; i += ngs_gstride()) {
    const float px = q[3 * i], py = q[3 * i + 1], pz = q[3 * i + 2];
    const int cx = (int)floorf(px * inv_h), cy = (int)floorf(py * inv_h), cz = (int)floorf(pz * inv_h);
    const int lo[3] = {g.origin[0], g.origin[1], g.origin[2]};
    const int hi[3] = {g.origin[0] + g.dims[0] - 1, g.origin[1] + g.dims[1] - 1, g.origin[2] + g.dims[2] - 1};
    const int c[3] = {cx, cy, cz};
    int rmax = 0;
#pragma unroll
    for (int a = 0; a < 3; a++) rmax = max(rmax, max(c[a] - lo[a], hi[a] - c[a]));
    float bd[KNN_MAX_K];
    int bi[KNN_MAX_K];
    int cnt = 0;
    for (int r = 0; r <= rmax; r++) {
      const int x0 = max(cx - r, lo[0]), x1 = min(cx + r, hi[0]);
      const int y0 = max(cy - r, lo[1]), y1 = min(cy + r, hi[1]);
      for (int x = x0; x <= x1; x++) {
        for (int y = y0; y <= y1; y++) {
          const bool side = abs(x - cx) == r || abs(y - cy) == r;
          // on the ring: every z of the column when x or y is at distance r, else only cz -+ r
          for (int z = side ? cz - r : cz - r; z <= cz + r; z += (side || r == 0) ? 1 : 2 * r) {
            if (z < lo[2] || z > hi[2]) continue;
            const int64_t cell = grid_row(g, x, y, z);
            if (cell < 0) continue;
            for (int64_t t = start[cell]; t < start[cell + 1]; t++) {
              const int pid = sorted[t];
              const float dx = ref[3 * pid] - px, dy = ref[3 * pid + 1] - py, dz = ref[3 * pid + 2] - pz;
              const float d2 = dx * dx + dy * dy + dz * dz;
              if (cnt == k && !knn_less(d2, pid, bd[k - 1], bi[k - 1])) continue;
              int s = cnt < k ? cnt++ : k - 1;     // insertion into the sorted list
              while (s > 0 && knn_less(d2, pid, bd[s - 1], bi[s - 1])) {
                bd[s] = bd[s - 1];
                bi[s] = bi[s - 1];
                s--;
              }
              bd[s] = d2;
              bi[s] = pid;
            }
          }
        }
      }
      const float reach = (float)r * h;
      if (cnt == k && bd[k - 1] <= reach * reach) break;
    }
    if (idx_out)
      for (int j = 0; j < k; j++) idx_out[i * k + j] = j < cnt ? bi[j] : -1;
    if (d2_out)
      for (int j = 0; j < k; j++) d2_out[i * k + j] = j < cnt ? bd[j] : INFINITY;
    if (sdf_out) {
      float sdf = 0.f;
      int pos = 0;
      for (int j = 0; j < cnt; j++) {
        const int pid = bi[j];
        const float rx = px - ref[3 * pid], ry = py - ref[3 * pid + 1], rz = pz - ref[3 * pid + 2];
        const float d = nrm[3 * pid] * rx + nrm[3 * pid + 1] * ry + nrm[3 * pid + 2] * rz;
        if (j == 0) {
          const float len = sqrtf(rx * rx + ry * ry + rz * rz);
          sdf = len < stdv ? fabsf(d) : len;
        }
        if (d > 0.f) pos++;
      }
      sdf_out[i] = pos <= k / 2 ? -sdf : sdf;
    }
  }
}

extern "C" int ngs_knn_mark_cells(ngs_grid g, const float* xyz, int64_t n, float inv_h, ngs_stream s) {
  if (!g.words || g.stride != 1 || n < 0 || (n > 0 && !xyz) || !(inv_h > 0.f)) return NGS_ERR_INVALID_ARG;
  if (n == 0) return NGS_OK;
  { ngs_count_launch(); knn_mark_cells_kernel<<<ngs_blocks(n, 256), 256, 0, (cudaStream_t)s>>>(g, xyz, n, inv_h); }
  NGS_CHECK_LAUNCH();
  return NGS_OK;
}

extern "C" int ngs_knn_bucket(ngs_grid g, const float* xyz, int64_t n, float inv_h, int32_t* cell_of,
                              int32_t* cell_count, ngs_stream s) {
  if (!g.words || g.stride != 1 || n < 0 || (n > 0 && (!xyz || !cell_of || !cell_count)) || !(inv_h > 0.f))
    return NGS_ERR_INVALID_ARG;
  if (n == 0) return NGS_OK;
  { ngs_count_launch(); knn_bucket_kernel<<<ngs_blocks(n, 256), 256, 0, (cudaStream_t)s>>>(g, xyz, n, inv_h, cell_of, cell_count); }
  NGS_CHECK_LAUNCH();
  return NGS_OK;
}

extern "C" int ngs_knn_scatter(const int32_t* cell_of, int64_t n, const int64_t* start, int32_t* cursor, int32_t* sorted,
                               ngs_stream s) {
  if (n < 0 || (n > 0 && (!cell_of || !start || !cursor || !sorted))) return NGS_ERR_INVALID_ARG;
  if (n == 0) return NGS_OK;
  { ngs_count_launch(); knn_scatter_kernel<<<ngs_blocks(n, 256), 256, 0, (cudaStream_t)s>>>(cell_of, n, start, cursor, sorted); }
  NGS_CHECK_LAUNCH();
  return NGS_OK;
}

extern "C" int ngs_knn_sdf(ngs_grid g, const int64_t* start, const int32_t* sorted, const float* ref_xyz,
                           const float* ref_normal, const float* queries, int64_t nq, float inv_h, float h, int k,
                           float stdv, int32_t* idx_out, float* d2_out, float* sdf_out, ngs_stream s) {
  if (!g.words || g.stride != 1 || nq < 0 || k < 1 || k > KNN_MAX_K || !(inv_h > 0.f) || !start || !sorted ||
      !ref_xyz || (nq > 0 && !queries) || (sdf_out && !ref_normal))
    return NGS_ERR_INVALID_ARG;
  if (nq == 0) return NGS_OK;
  { ngs_count_launch(); knn_sdf_kernel<<<ngs_blocks(nq, 128), 128, 0, (cudaStream_t)s>>>(
      g, start, sorted, ref_xyz, ref_normal, queries, nq, inv_h, h, k, stdv, idx_out, d2_out, sdf_out); }
  NGS_CHECK_LAUNCH();
  return NGS_OK;
}

// ----------------------------------------------------------------------------- box tree
// The queries of jspsr.sdfgen: the points in Morton order of a cube of cells, 32 to a leaf, under a
// 32-ary tree of bounding boxes; one warp per query.  A node's children are tested 32 at a time, one per
// lane, and visited nearest first; a child is skipped once its box is farther than the k-th best point.
// The list of the k best lives in the lanes (lane j: the j-th), so a leaf costs one distance per lane
// and a few shuffles per point that enters the list.
//
// The ring walk above reads every cell of the rings between a query and its neighbours: a query a
// tenth of the scene off the surface reads ~10^5 empty cells and holds up its warp.  What bounds the tree
// walk is the chain of box test -> choice of the nearest child -> next box test, 3 to 5 levels deep, and
// the shuffles of the list.  Measured (60,000 points on a torus, 100,000 queries, 1 in 16 anywhere in the
// cube around it, k = 8, signed distance): build and queries 0.45 ms, the grid walk 376 ms (with
// every point inserted one by one, and cells of 16 points instead of 2: 0.65 ms).
//
// Exactness: a box's squared distance is formed from lo - q or hi - q by the operations that form a
// point's from p - q.  Each rounds monotonically, so no point of a box is nearer than its box, and skipping
// boxes strictly farther than the k-th best loses neither a neighbour nor a tie (ties go to the smaller
// index, whatever the order of the visit).
constexpr int KNN_TREE_LEVELS = 7;          // 32^7 > 2^31 points
constexpr int KNN_TREE_WARPS = 4;

struct KnnTree {
  const float4* pts;                        // x, y, z, bits of the point's index
  const float4* box;                        // two per node: (lo, -), (hi, -); level 0 = leaves
  int64_t n;
  int64_t off[KNN_TREE_LEVELS];             // first node of each level
  int64_t cnt[KNN_TREE_LEVELS];
  int levels;                               // the last level has at most 32 nodes
};

static int64_t knn_align(int64_t v) { return (v + 255) & ~(int64_t)255; }

static KnnTree knn_tree_layout(int64_t n, void* mem) {
  KnnTree t{};
  t.n = n;
  t.pts = static_cast<const float4*>(mem);
  t.box = reinterpret_cast<const float4*>(static_cast<char*>(mem) + knn_align(n * 16));
  int64_t c = n, off = 0;
  do {
    c = (c + 31) / 32;
    t.off[t.levels] = off;
    t.cnt[t.levels++] = c;
    off += c;
  } while (c > 32);
  return t;
}

extern "C" size_t ngs_knn_tree_bytes(int64_t n) {
  if (n < 1 || n > (int64_t)0x7fffffff) return 0;
  const KnnTree t = knn_tree_layout(n, nullptr);
  return (size_t)(knn_align(n * 16) + (t.off[t.levels - 1] + t.cnt[t.levels - 1]) * 32);
}

// Cells per axis 2^bits: about 2 points per occupied cell for points on a surface, at most 512.
static int knn_tree_bits(int64_t n) {
  int b = 2;
  while (b < 9 && ((int64_t)2 << (2 * b)) < n) b++;
  return b;
}

struct KnnScratch {
  float* bbox;
  GridWord* words;
  int64_t nwords;
  int32_t *cell, *count, *cursor;
  int64_t* start;
  void* scan;
  size_t scan_bytes;
  int bits;
};

static size_t knn_scratch_layout(int64_t n, void* mem, KnnScratch& s) {
  char* p = static_cast<char*>(mem);
  size_t at = 0;
  auto take = [&](int64_t bytes) {
    char* r = p + at;
    at += (size_t)knn_align(bytes);
    return r;
  };
  s.bits = knn_tree_bits(n);
  s.nwords = ((int64_t)1 << (3 * s.bits)) / 64;
  s.words = reinterpret_cast<GridWord*>(take(s.nwords * 16));
  s.count = reinterpret_cast<int32_t*>(take(n * 4));
  s.cursor = reinterpret_cast<int32_t*>(take(n * 4));
  s.cell = reinterpret_cast<int32_t*>(take(n * 4));
  s.start = reinterpret_cast<int64_t*>(take(n * 8));
  s.bbox = reinterpret_cast<float*>(take(6 * 4));
  s.scan_bytes = ngs_scan_ws_bytes(s.nwords > n ? s.nwords : n);
  s.scan = take((int64_t)s.scan_bytes);
  return at;
}

extern "C" size_t ngs_knn_tree_scratch_bytes(int64_t n) {
  KnnScratch s;
  return n < 1 || n > (int64_t)0x7fffffff ? 0 : knn_scratch_layout(n, nullptr, s);
}

NGS_DEV unsigned spread3(unsigned v) {       // bit i of v to bit 3 i
  unsigned r = 0;
#pragma unroll
  for (int i = 0; i < 9; i++) r |= ((v >> i) & 1u) << (3 * i);
  return r;
}

// Morton code of the point's cell in the cube over the bounding box (every value ends in the cube).
NGS_DEV unsigned knn_code(const float* __restrict__ p, const float* __restrict__ bbox, int bits) {
  const float ext = fmaxf(fmaxf(bbox[3] - bbox[0], bbox[4] - bbox[1]), bbox[5] - bbox[2]);
  const float scale = ext > 0.f ? (float)(1 << bits) / ext : 0.f;
  unsigned code = 0;
#pragma unroll
  for (int a = 0; a < 3; a++) {
    const int c = (int)fminf(fmaxf((p[a] - bbox[a]) * scale, 0.f), (float)((1 << bits) - 1));
    code |= spread3((unsigned)c) << (2 - a);
  }
  return code;
}

__global__ void knn_tree_mark_kernel(const float* __restrict__ xyz, int64_t n, const float* __restrict__ bbox,
                                     int bits, GridWord* __restrict__ words, int32_t* __restrict__ cell) {
  for (int64_t i = ngs_gtid(); i < n; i += ngs_gstride()) {
    const unsigned code = knn_code(xyz + 3 * i, bbox, bits);
    cell[i] = (int32_t)code;
    atomicOr(&words[code >> 6].bits, 1ull << (code & 63));
  }
}

struct KnnWordPopc {
  const GridWord* w;
  NGS_DEV int64_t operator()(int64_t i) const { return __popcll(w[i].bits); }
};
struct KnnWordRank {
  GridWord* w;
  NGS_DEV void operator()(int64_t i, int64_t v) const { w[i].rank = (uint32_t)v; }
};
struct KnnLoadI32 {
  const int32_t* p;
  NGS_DEV int64_t operator()(int64_t i) const { return (int64_t)p[i]; }
};
struct KnnStoreI64 {
  int64_t* p;
  NGS_DEV void operator()(int64_t i, int64_t v) const { p[i] = v; }
};

__global__ void knn_tree_bucket_kernel(const GridWord* __restrict__ words, int64_t n, int32_t* __restrict__ cell,
                                       int32_t* __restrict__ count) {
  for (int64_t i = ngs_gtid(); i < n; i += ngs_gstride()) {
    const unsigned code = (unsigned)cell[i];
    const GridWord w = words[code >> 6];
    const int32_t r = (int32_t)w.rank + __popcll(w.bits & ((1ull << (code & 63)) - 1ull));
    cell[i] = r;
    atomicAdd(count + r, 1);
  }
}

__global__ void knn_tree_scatter_kernel(const float* __restrict__ xyz, int64_t n, const int32_t* __restrict__ cell,
                                        const int64_t* __restrict__ start, int32_t* __restrict__ cursor,
                                        float4* __restrict__ pts) {
  for (int64_t i = ngs_gtid(); i < n; i += ngs_gstride()) {
    const int32_t c = cell[i];
    pts[start[c] + atomicAdd(cursor + c, 1)] =
        make_float4(xyz[3 * i], xyz[3 * i + 1], xyz[3 * i + 2], __int_as_float((int)i));
  }
}

// Boxes of one level: a warp per node, a lane per child (points for level 0, nodes of the level below
// otherwise).
__global__ void knn_tree_box_kernel(const float4* __restrict__ pts, const float4* __restrict__ child, int64_t n_child,
                                    float4* __restrict__ out, int64_t n_node) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t b = ngs_gtid() >> 5; b < n_node; b += warps) {
    const int64_t c = min(b * 32 + lane, n_child - 1);
    float4 lo, hi;
    if (pts) {
      lo = hi = pts[c];
    } else {
      lo = child[2 * c];
      hi = child[2 * c + 1];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      lo.x = fminf(lo.x, __shfl_xor_sync(0xffffffffu, lo.x, o));
      lo.y = fminf(lo.y, __shfl_xor_sync(0xffffffffu, lo.y, o));
      lo.z = fminf(lo.z, __shfl_xor_sync(0xffffffffu, lo.z, o));
      hi.x = fmaxf(hi.x, __shfl_xor_sync(0xffffffffu, hi.x, o));
      hi.y = fmaxf(hi.y, __shfl_xor_sync(0xffffffffu, hi.y, o));
      hi.z = fmaxf(hi.z, __shfl_xor_sync(0xffffffffu, hi.z, o));
    }
    if (lane == 0) {
      out[2 * b] = make_float4(lo.x, lo.y, lo.z, 0.f);
      out[2 * b + 1] = make_float4(hi.x, hi.y, hi.z, 0.f);
    }
  }
}

// Squared distance in the grid walk's order of operations; NaN sorts with infinity.
NGS_DEV float knn_d2(float dx, float dy, float dz) {
  const float d = __fmaf_rn(dz, dz, __fmaf_rn(dx, dx, __fmul_rn(dy, dy)));
  return d == d ? d : INFINITY;
}
// Distance and index as one ordered number: the bits of a distance, which is never negative, order as the
// distance does.
NGS_DEV unsigned long long knn_key(float d, int i) {
  return (unsigned long long)__float_as_uint(d) << 32 | (unsigned)i;
}
constexpr unsigned long long KNN_NONE = 0x7f8000007fffffffull;        // (infinity, INT_MAX): after every point

// One step of a bitonic network over the warp: lane keeps the smaller of the pair (lane, lane ^ o) if `low`.
NGS_DEV unsigned long long knn_exchange(unsigned long long v, int o, bool low) {
  const unsigned long long w = __shfl_xor_sync(0xffffffffu, v, o);
  return (w < v) == low ? w : v;
}
// Distance along one axis from q to [lo, hi] (0 inside; a NaN query stays NaN).
NGS_DEV float knn_gap(float lo, float hi, float q) { return q < lo ? lo - q : (q > hi ? q - hi : q - q); }

__global__ void __launch_bounds__(KNN_TREE_WARPS * 32) knn_tree_query_kernel(
    const __grid_constant__ KnnTree t, const float* __restrict__ ref, const float* __restrict__ nrm,
    const float* __restrict__ q, int64_t nq, int k, float stdv, int32_t* __restrict__ idx_out,
    float* __restrict__ d2_out, float* __restrict__ sdf_out) {
  // per level of the walk: the children's distances (a lane each), those still to visit, and the node
  __shared__ float s_d[KNN_TREE_WARPS][KNN_TREE_LEVELS][32];
  __shared__ unsigned s_left[KNN_TREE_WARPS][KNN_TREE_LEVELS];
  __shared__ int s_node[KNN_TREE_WARPS][KNN_TREE_LEVELS];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t warps = (int64_t)gridDim.x * KNN_TREE_WARPS;
  for (int64_t i = (int64_t)blockIdx.x * KNN_TREE_WARPS + w; i < nq; i += warps) {
    const float px = q[3 * i], py = q[3 * i + 1], pz = q[3 * i + 2];
    unsigned long long mine = KNN_NONE;      // lane j: the j-th best point
    unsigned long long last = KNN_NONE;      // the k-th best
    float kd = INFINITY;
    int lev = t.levels - 1, node = 0;        // node: the parent whose children at level lev are tested
    bool fresh = true;
    while (lev < t.levels) {
      if (fresh) {
        const int64_t c = (int64_t)node * 32 + lane;
        float d = INFINITY;
        const bool have = c < t.cnt[lev];
        if (have) {
          const float4 lo = __ldg(t.box + 2 * (t.off[lev] + c)), hi = __ldg(t.box + 2 * (t.off[lev] + c) + 1);
          d = knn_d2(knn_gap(lo.x, hi.x, px), knn_gap(lo.y, hi.y, py), knn_gap(lo.z, hi.z, pz));
        }
        const unsigned left = __ballot_sync(0xffffffffu, have && d <= kd);
        s_d[w][lev][lane] = d;
        if (lane == 0) {
          s_left[w][lev] = left;
          s_node[w][lev] = node;
        }
        __syncwarp();
        fresh = false;
      }
      // the nearest child still to visit; one beyond the k-th best ends the node
      const float d = s_d[w][lev][lane];
      const unsigned left = s_left[w][lev];
      const unsigned key = (left >> lane) & 1u ? __float_as_uint(d) : 0xffffffffu;
      const unsigned best = __reduce_min_sync(0xffffffffu, key);
      if (left == 0u || __uint_as_float(best) > kd) {
        lev++;
        __syncwarp();
        continue;
      }
      const int pick = __ffs(__ballot_sync(0xffffffffu, key == best)) - 1;
      if (lane == 0) s_left[w][lev] = left & ~(1u << pick);
      const int child = s_node[w][lev] * 32 + pick;
      __syncwarp();
      if (lev > 0) {
        lev--;
        node = child;
        fresh = true;
        continue;
      }
      // a leaf: one point per lane.  A few that enter the list are inserted one after another; more (the
      // first leaf, above all) are sorted and merged with the list, some 150 instructions against 25 each
      const int64_t c = (int64_t)child * 32 + lane;
      unsigned long long pt = KNN_NONE;
      if (c < t.n) {
        const float4 p = __ldg(t.pts + c);
        pt = knn_key(knn_d2(p.x - px, p.y - py, p.z - pz), __float_as_int(p.w));
      }
      unsigned cand = __ballot_sync(0xffffffffu, pt < last);
      if (__popc(cand) > 6) {
#pragma unroll
        for (int size = 2; size <= 32; size <<= 1)
#pragma unroll
          for (int o = size >> 1; o > 0; o >>= 1) pt = knn_exchange(pt, o, ((lane & o) == 0) == ((lane & size) == 0));
        // the list and the reversed leaf: the 32 smallest of both form a bitonic sequence
        pt = __shfl_xor_sync(0xffffffffu, pt, 31);
        mine = pt < mine ? pt : mine;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mine = knn_exchange(mine, o, (lane & o) == 0);
        last = __shfl_sync(0xffffffffu, mine, k - 1);
        cand = 0u;
      }
      while (cand) {
        const unsigned long long p = __shfl_sync(0xffffffffu, pt, __ffs(cand) - 1);
        const unsigned long long up = __shfl_up_sync(0xffffffffu, mine, 1);
        const int at = __popc(__ballot_sync(0xffffffffu, mine < p));     // sorted: lanes 0 .. at - 1
        mine = lane > at ? up : (lane == at ? p : mine);
        last = __shfl_sync(0xffffffffu, mine, k - 1);
        cand &= cand - 1u;
        cand &= __ballot_sync(0xffffffffu, pt < last);
      }
      kd = __uint_as_float((unsigned)(last >> 32));
    }
    const float bd = __uint_as_float((unsigned)(mine >> 32));
    const int bi = (int)(unsigned)mine;
    const bool have = lane < k && mine != KNN_NONE;
    if (lane < k) {
      if (idx_out) idx_out[i * k + lane] = have ? bi : -1;
      if (d2_out) d2_out[i * k + lane] = have && px + py + pz != px + py + pz && bd == INFINITY ? NAN : bd;
    }
    if (sdf_out) {
      float rx = 0.f, ry = 0.f, rz = 0.f, d = 0.f;
      if (have) {
        rx = px - ref[3 * (int64_t)bi];
        ry = py - ref[3 * (int64_t)bi + 1];
        rz = pz - ref[3 * (int64_t)bi + 2];
        d = nrm[3 * (int64_t)bi] * rx + nrm[3 * (int64_t)bi + 1] * ry + nrm[3 * (int64_t)bi + 2] * rz;
      }
      const int pos = __popc(__ballot_sync(0xffffffffu, have && d > 0.f));
      if (lane == 0) {
        const float len = sqrtf(rx * rx + ry * ry + rz * rz);
        const float sdf = have ? (len < stdv ? fabsf(d) : len) : 0.f;
        sdf_out[i] = pos <= k / 2 ? -sdf : sdf;
      }
    }
  }
}

extern "C" int ngs_knn_tree_build(const float* xyz, int64_t n, void* tree, size_t tree_bytes, void* scratch,
                                  size_t scratch_bytes, ngs_stream s) {
  if (n < 1 || n > (int64_t)0x7fffffff || !xyz || !tree || !scratch ||
      ((reinterpret_cast<uintptr_t>(tree) | reinterpret_cast<uintptr_t>(scratch)) & 15u))
    return NGS_ERR_INVALID_ARG;
  if (tree_bytes < ngs_knn_tree_bytes(n) || scratch_bytes < ngs_knn_tree_scratch_bytes(n)) return NGS_ERR_OOM;
  cudaStream_t st = (cudaStream_t)s;
  const KnnTree t = knn_tree_layout(n, tree);
  KnnScratch c;
  knn_scratch_layout(n, scratch, c);
  float4* pts = const_cast<float4*>(t.pts);
  float4* box = const_cast<float4*>(t.box);
  int rc = ngs_points_bbox(xyz, n, c.bbox, s);
  if (rc != NGS_OK) return rc;
  // words, counts and cursors lie at the front of the scratch, one after another
  cudaMemsetAsync(c.words, 0, (size_t)(reinterpret_cast<char*>(c.cell) - reinterpret_cast<char*>(c.words)), st);
  const unsigned grid = ngs_blocks(n, 256);
  { ngs_count_launch(); knn_tree_mark_kernel<<<grid, 256, 0, st>>>(xyz, n, c.bbox, c.bits, c.words, c.cell); }
  rc = ngs_scan(KnnWordPopc{c.words}, KnnWordRank{c.words}, c.nwords, nullptr, c.scan, c.scan_bytes, st);
  if (rc != NGS_OK) return rc;
  { ngs_count_launch(); knn_tree_bucket_kernel<<<grid, 256, 0, st>>>(c.words, n, c.cell, c.count); }
  rc = ngs_scan(KnnLoadI32{c.count}, KnnStoreI64{c.start}, n, nullptr, c.scan, c.scan_bytes, st);
  if (rc != NGS_OK) return rc;
  { ngs_count_launch(); knn_tree_scatter_kernel<<<grid, 256, 0, st>>>(xyz, n, c.cell, c.start, c.cursor, pts); }
  for (int l = 0; l < t.levels; l++) {
    ngs_count_launch();
    knn_tree_box_kernel<<<ngs_blocks(t.cnt[l] * 32, 256), 256, 0, st>>>(
        l == 0 ? pts : nullptr, l == 0 ? nullptr : box + 2 * t.off[l - 1], l == 0 ? n : t.cnt[l - 1],
        box + 2 * t.off[l], t.cnt[l]);
  }
  NGS_CHECK_LAUNCH();
  return NGS_OK;
}

extern "C" int ngs_knn_tree_query(const void* tree, size_t tree_bytes, const float* ref_xyz, int64_t n,
                                  const float* ref_normal, const float* queries, int64_t nq, int k, float stdv,
                                  int32_t* idx_out, float* d2_out, float* sdf_out, ngs_stream s) {
  if (n < 1 || n > (int64_t)0x7fffffff || !tree || (reinterpret_cast<uintptr_t>(tree) & 15u) || !ref_xyz || nq < 0 ||
      k < 1 || k > KNN_MAX_K || (nq > 0 && !queries) || (sdf_out && !ref_normal))
    return NGS_ERR_INVALID_ARG;
  if (tree_bytes < ngs_knn_tree_bytes(n)) return NGS_ERR_OOM;
  if (nq == 0) return NGS_OK;
  const KnnTree t = knn_tree_layout(n, const_cast<void*>(tree));
  {
    ngs_count_launch();
    knn_tree_query_kernel<<<ngs_blocks(nq * 32, KNN_TREE_WARPS * 32), KNN_TREE_WARPS * 32, 0, (cudaStream_t)s>>>(
        t, ref_xyz, ref_normal, queries, nq, k, stdv, idx_out, d2_out, sdf_out);
  }
  NGS_CHECK_LAUNCH();
  return NGS_OK;
}
