// Terms of the Galerkin system of a learned (additive) basis and their derivatives
// (jspsr/bases/additive.py:55-414): per axis B(x) = sum_k m_k q_k(x) with a voxel's coefficients
// m[3 k + axis]; a pair's stiffness and divergence are bilinear and linear forms of them through tables.
//
// Every kernel reads the coefficients by voxel id and sums a term straight into what it belongs to (a CSR
// slot, a right-hand side, a coefficient gradient).  Bound: launches and latency at the sizes of a shape
// (1e4 voxels, 1e6 pairs).  As torch operations around a pair kernel, a term gathered two rows of 3 C floats per
// pair, and its gradient scattered as many through a sort; a training step of four shapes of 3,000 points made
// some 10,000 launches and 150 synchronisations, bound by the host: 238.6 ms, 93.1 with these kernels, of which the
// solves take 30.  Per launch at 1e5 to 5e5 pairs of ten components: values 108 us (pair kernel alone) -> 45,
// gradient 147 us and a sorted scatter of 107 -> 158.
//
// Gradients: a lane works one pair and stages its row of 3 C floats; the warp then adds the rows with a lane per
// column (consecutive words, and rows of one voxel next to each other summed first), instead of 3 C strided
// atomics per pair.  The pair kernels hold the tables in shared memory and are compiled per component count, so
// that a pair's coefficients stay in registers.
#include "ngs_common.cuh"

constexpr int BASIS_MOST = 32;        // components of a basis
constexpr int PAIR_MOST = 12;         // of one whose pair terms run here (registers: three arrays of C floats)
constexpr int ROWS_SMEM = 4 * 4 * 32 * (3 * BASIS_MOST + 1);   // staged rows of a block of 128 threads, at most

// ----------------------------------------------------------------------------- components
struct BasisComps {
  int count;
  int kind[BASIS_MOST];               // ngs_basis_comps
  float a[BASIS_MOST], b[BASIS_MOST];
};

NGS_DEV float comp_value(const BasisComps& c, int k, float x) {
  switch (c.kind[k]) {
    case NGS_COMP_POWER: {
      const float p = c.a[k];
      if (p == 0.f) return 1.f;
      if (p == 1.f) return x;
      if (p == 2.f) return x * x;
      if (p == 3.f) return x * x * x;
      return powf(x, p);
    }
    case NGS_COMP_SIN:
      return sinf(__fadd_rn(__fmul_rn(c.a[k], x), c.b[k]));
    default: {                        // the quadratic B-spline, times two
      if (x >= -1.5f && x < -0.5f) return (x + 1.5f) * (x + 1.5f);
      if (x >= -0.5f && x < 0.5f) return 1.5f - 2.f * (x * x);
      if (x >= 0.5f && x < 1.5f) return (x - 1.5f) * (x - 1.5f);
      return 0.f;
    }
  }
}

static bool comps_of(const ngs_basis_comps* in, BasisComps& out) {
  if (!in || in->count < 1 || in->count > BASIS_MOST) return false;
  out = BasisComps{};
  out.count = in->count;
  for (int k = 0; k < in->count; k++) {
    if (in->kind[k] < NGS_COMP_POWER || in->kind[k] > NGS_COMP_BEZIER) return false;
    out.kind[k] = in->kind[k];
    out.a[k] = in->a[k];
    out.b[k] = in->b[k];
  }
  return true;
}

// A thread per (row, axis): values with the row's own coefficients, and their gradient.
__global__ void basis_axes_kernel(const __grid_constant__ BasisComps c, const float* __restrict__ coef,
                                  const float* __restrict__ x, int64_t m, float* __restrict__ f) {
  for (int64_t t = ngs_gtid(); t < 3 * m; t += ngs_gstride()) {
    const int64_t row = t / 3;
    const float* cr = coef + row * 3 * c.count + (t - 3 * row);
    const float xv = x[t];
    float s = 0.f;
    for (int k = 0; k < c.count; k++) s = __fadd_rn(s, __fmul_rn(comp_value(c, k, xv), cr[3 * k]));
    f[t] = s;
  }
}

__global__ void basis_axes_grad_kernel(const __grid_constant__ BasisComps c, const float* __restrict__ x,
                                       const float* __restrict__ grad, int64_t m, float* __restrict__ gcoef) {
  for (int64_t t = ngs_gtid(); t < 3 * m; t += ngs_gstride()) {
    const int64_t row = t / 3;
    float* gr = gcoef + row * 3 * c.count + (t - 3 * row);
    const float xv = x[t], g = grad[t];
    for (int k = 0; k < c.count; k++) gr[3 * k] = g * comp_value(c, k, xv);
  }
}

// B(p) of every (point, slot): the product of the axes' values, 0 where the slot has no voxel.
__global__ void basis_phi_kernel(const __grid_constant__ BasisComps c, const float* __restrict__ coef,
                                 const int32_t* __restrict__ rows, const float* __restrict__ local, int64_t m,
                                 float* __restrict__ phi) {
  for (int64_t t = ngs_gtid(); t < m; t += ngs_gstride()) {
    const int32_t row = rows[t];
    float out = 0.f;
    if (row >= 0) {
      const float* cr = coef + (int64_t)row * 3 * c.count;
      float f[3] = {0.f, 0.f, 0.f};
      const float x[3] = {local[3 * t], local[3 * t + 1], local[3 * t + 2]};
      for (int k = 0; k < c.count; k++)
#pragma unroll
        for (int v = 0; v < 3; v++) f[v] = __fadd_rn(f[v], __fmul_rn(comp_value(c, k, x[v]), cr[3 * k + v]));
      out = f[0] * f[1] * f[2];
    }
    phi[t] = out;
  }
}

// Sums rows of 3 C floats staged by a warp's lanes (one row each, stride `pitch`) into dst[id]: lane = column,
// so that a row goes out as consecutive words, and rows of one id next to each other are summed first.
NGS_DEV void add_rows(const float* stage, int pitch, int width, int64_t id, float* __restrict__ dst) {
  const int lane = threadIdx.x & 31;
  const unsigned live = __ballot_sync(0xffffffffu, id >= 0);
  for (int c0 = 0; c0 < width; c0 += 32) {
    const int c = c0 + lane;
    float run = 0.f;
    int64_t cur = -1;
    for (unsigned left = live; left; left &= left - 1) {
      const int p = __ffs(left) - 1;
      const int64_t q = __shfl_sync(0xffffffffu, id, p);
      if (q != cur) {
        if (cur >= 0 && c < width) atomicAdd(dst + cur * width + c, run);
        cur = q;
        run = 0.f;
      }
      if (c < width) run += stage[p * pitch + c];
    }
    if (cur >= 0 && c < width) atomicAdd(dst + cur * width + c, run);
  }
}

// Coefficient gradient of the point values: dL/dB(p) of slot row i is lambda_i A_p + x_i B_p.
__global__ void basis_phi_grad_kernel(const __grid_constant__ BasisComps c, const float* __restrict__ coef,
                                      const int32_t* __restrict__ rows, const float* __restrict__ local, int64_t m,
                                      const double* __restrict__ lam, const double* __restrict__ xs,
                                      const double* __restrict__ pa, const double* __restrict__ pb,
                                      float* __restrict__ gcoef) {
  extern __shared__ float smem[];
  const int lane = threadIdx.x & 31, width = 3 * c.count, pitch = width | 1;
  float* own = smem + (int64_t)(threadIdx.x >> 5) * 32 * pitch;
  const int64_t step = ngs_gstride();
  for (int64_t t0 = ngs_gtid() - lane; t0 < m; t0 += step) {            // warp-uniform
    const int64_t t = t0 + lane;
    const int32_t row = t < m ? rows[t] : -1;
    if (row >= 0) {
      const float* cr = coef + (int64_t)row * width;
      float f[3] = {0.f, 0.f, 0.f};
      const float x[3] = {local[3 * t], local[3 * t + 1], local[3 * t + 2]};
      for (int k = 0; k < c.count; k++)
#pragma unroll
        for (int v = 0; v < 3; v++) {
          const float q = comp_value(c, k, x[v]);
          own[lane * pitch + 3 * k + v] = q;
          f[v] = __fadd_rn(f[v], __fmul_rn(q, cr[3 * k + v]));
        }
      const int64_t p = t / 27;
      const float g = (float)(lam[row] * pa[p] + xs[row] * pb[p]);
      const float gv[3] = {(g * f[2]) * f[1], (g * f[2]) * f[0], g * (f[0] * f[1])};
      for (int k = 0; k < c.count; k++)
#pragma unroll
        for (int v = 0; v < 3; v++) own[lane * pitch + 3 * k + v] *= gv[v];
    }
    __syncwarp();
    add_rows(own, pitch, width, row, gcoef);
    __syncwarp();
  }
}

// ----------------------------------------------------------------------------- stiffness of voxel pairs
struct PairArgs {
  const float *ff, *dd;               // [C, C, R] integrals of q q and q' q' by offset
  const float *cs, *ct;               // coefficients of the sources' and the targets' level
  const int64_t* sid;
  const void* tid;
  const float* rel;                   // [pairs, 3]
  int64_t pairs;
  float fscale, dscale, add;          // scales of the tables; the offset of rel in them
  int R, tid32;
  double* out;                        // per pair, or
  const double* x;                    // y[target or source] -= value * x[the other]
  double* y;
  int transposed;
  const double *lam, *xs;             // gradient: dL/dvalue = -lambda[source] x[target]
  float *gs, *gt;                     // (either may be null)
};

NGS_DEV int64_t pair_target(const PairArgs& a, int64_t t) {
  return a.tid32 ? (int64_t)static_cast<const int32_t*>(a.tid)[t] : static_cast<const int64_t*>(a.tid)[t];
}

template <int C>
NGS_DEV void pair_tables(const PairArgs& a, float2* tab) {
  for (int i = threadIdx.x; i < C * C * a.R; i += blockDim.x) tab[i] = make_float2(a.ff[i] * a.fscale, a.dd[i] * a.dscale);
  __syncthreads();
}

// p = <q q>, q = <q' q'> of one axis; both 0 outside the tables.
template <int C>
NGS_DEV void pair_axis(const PairArgs& a, const float2* tab, const float* cs, const float* ct, float rel, float& p, float& q,
                       int& r) {
  const float at = rintf(rel + a.add);
  const bool ok = at >= 0.f && at < (float)a.R;
  r = ok ? (int)at : -1;
  p = q = 0.f;
  if (!ok) return;
  float t[C];
#pragma unroll
  for (int k = 0; k < C; k++) t[k] = ct[3 * k];
#pragma unroll
  for (int si = 0; si < C; si++) {
    float fp = 0.f, fq = 0.f;
#pragma unroll
    for (int ti = 0; ti < C; ti++) {
      const float2 w = tab[(si * C + ti) * a.R + r];
      fp += w.x * t[ti];
      fq += w.y * t[ti];
    }
    const float s = cs[3 * si];
    p += s * fp;
    q += s * fq;
  }
}

template <int C>
__global__ void __launch_bounds__(128) basis_pairs_kernel(const __grid_constant__ PairArgs a) {
  extern __shared__ float smem[];
  float2* tab = reinterpret_cast<float2*>(smem);
  pair_tables<C>(a, tab);
  for (int64_t t = ngs_gtid(); t < a.pairs; t += ngs_gstride()) {
    const int64_t s = a.sid[t], d = pair_target(a, t);
    float p[3], q[3];
    int r;
#pragma unroll 1
    for (int v = 0; v < 3; v++) {
      float pv, qv;
      pair_axis<C>(a, tab, a.cs + s * 3 * C + v, a.ct + d * 3 * C + v, a.rel[3 * t + v], pv, qv, r);
      if (v == 0) p[0] = pv, q[0] = qv;
      else if (v == 1) p[1] = pv, q[1] = qv;
      else p[2] = pv, q[2] = qv;
    }
    const double k = (double)(q[0] * p[1] * p[2] + p[0] * q[1] * p[2] + p[0] * p[1] * q[2]);
    if (a.out) a.out[t] = k;
    else if (a.transposed) atomicAdd(a.y + d, -(k * a.x[s]));
    else atomicAdd(a.y + s, -(k * a.x[d]));
  }
}

template <int C>
__global__ void __launch_bounds__(128) basis_pairs_grad_kernel(const __grid_constant__ PairArgs a) {
  extern __shared__ float smem[];
  constexpr int W = 3 * C, PITCH = W | 1;
  float2* tab = reinterpret_cast<float2*>(smem);
  float* own = smem + 2 * C * C * a.R + (threadIdx.x >> 5) * 64 * PITCH;      // rows of the sources, of the targets
  pair_tables<C>(a, tab);
  const int lane = threadIdx.x & 31;
  const int64_t step = ngs_gstride();
  for (int64_t t0 = ngs_gtid() - lane; t0 < a.pairs; t0 += step) {            // warp-uniform
    const int64_t t = t0 + lane;
    int64_t s = -1, d = -1;
    if (t < a.pairs) {
      s = a.sid[t];
      d = pair_target(a, t);
      float p[3], q[3];
      int r[3];
#pragma unroll 1
      for (int v = 0; v < 3; v++) {
        float pv, qv;
        int rv;
        pair_axis<C>(a, tab, a.cs + s * W + v, a.ct + d * W + v, a.rel[3 * t + v], pv, qv, rv);
        if (v == 0) p[0] = pv, q[0] = qv, r[0] = rv;
        else if (v == 1) p[1] = pv, q[1] = qv, r[1] = rv;
        else p[2] = pv, q[2] = qv, r[2] = rv;
      }
      const float g = (float)(-(a.lam[s] * a.xs[d]));
#pragma unroll 1
      for (int v = 0; v < 3; v++) {
        const float p1 = v == 0 ? p[1] : p[0], q1 = v == 0 ? q[1] : q[0];
        const float p2 = v == 2 ? p[1] : p[2], q2 = v == 2 ? q[1] : q[2];
        const int rv = v == 0 ? r[0] : v == 1 ? r[1] : r[2];
        const float gq = rv >= 0 ? g * p1 * p2 : 0.f, gp = rv >= 0 ? g * q1 * p2 + g * p1 * q2 : 0.f;
        const int o = rv >= 0 ? rv : 0;
        float cs[C], ct[C], acc[C];
#pragma unroll
        for (int k = 0; k < C; k++) {
          cs[k] = a.cs[s * W + 3 * k + v];
          ct[k] = a.ct[d * W + 3 * k + v];
          acc[k] = 0.f;
        }
#pragma unroll
        for (int si = 0; si < C; si++) {
          float sum = 0.f;
#pragma unroll
          for (int ti = 0; ti < C; ti++) {
            const float2 w = tab[(si * C + ti) * a.R + o];
            const float m = gp * w.x + gq * w.y;
            sum += m * ct[ti];
            acc[ti] += m * cs[si];
          }
          own[lane * PITCH + 3 * si + v] = sum;
        }
#pragma unroll
        for (int k = 0; k < C; k++) own[(32 + lane) * PITCH + 3 * k + v] = acc[k];
      }
    }
    __syncwarp();
    if (a.gs) add_rows(own, PITCH, W, s, a.gs);
    if (a.gt) add_rows(own + 32 * PITCH, PITCH, W, d, a.gt);
    __syncwarp();
  }
}

// Shared memory of a pair kernel's block, at most.  A kernel's limit is set to the most that any call can need, never
// to a call's own need: threads share it, and one with small tables would lower it under another's launch.
constexpr int PAIR_SMEM = 200 << 10;

template <int C>
static int launch_pairs(const PairArgs& a, bool grad, cudaStream_t st) {
  const size_t tab = sizeof(float2) * C * C * a.R;
  const size_t smem = tab + (grad ? sizeof(float) * 4 * 64 * ((3 * C) | 1) : 0);
  const void* f = grad ? (const void*)basis_pairs_grad_kernel<C> : (const void*)basis_pairs_kernel<C>;
  if (smem > 48 << 10) {
    const cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, PAIR_SMEM);
    if (e != cudaSuccess) return ngs_set_cuda_error(e);
  }
  void* args[] = {const_cast<PairArgs*>(&a)};
  ngs_count_launch();
  const cudaError_t e = cudaLaunchKernel(f, dim3(ngs_blocks(a.pairs, 128, 8)), dim3(128), args, smem, st);
  return e == cudaSuccess ? NGS_OK : ngs_set_cuda_error(e);
}

// Bytes of shared memory of the gradient kernel (the larger of the two) fit a block.
extern "C" int ngs_basis_pairs_fit(int C, int R) {
  return C >= 1 && C <= PAIR_MOST && R >= 1 &&
         8ll * C * C * R + 4ll * 4 * 64 * ((3 * C) | 1) <= PAIR_SMEM;
}

extern "C" int ngs_basis_pairs(const ngs_basis_pair_term* p, int grad, ngs_stream s) {
  if (!p || p->pairs < 0 || !ngs_basis_pairs_fit(p->C, p->R)) return NGS_ERR_INVALID_ARG;
  if (p->pairs == 0) return NGS_OK;
  if (!p->ff || !p->dd || !p->cs || !p->ct || !p->sid || !p->tid || !p->rel) return NGS_ERR_INVALID_ARG;
  if (grad ? (!p->lam || !p->xs || (!p->gs && !p->gt)) : (!p->out && (!p->x || !p->y))) return NGS_ERR_INVALID_ARG;
  PairArgs a{p->ff, p->dd, p->cs, p->ct, p->sid, p->tid, p->rel, p->pairs, p->fscale, p->dscale, p->add, p->R, p->tid32,
             p->out, p->x, p->y, p->transposed, p->lam, p->xs, p->gs, p->gt};
  cudaStream_t st = (cudaStream_t)s;
  switch (p->C) {
    case 1: return launch_pairs<1>(a, grad, st);
    case 2: return launch_pairs<2>(a, grad, st);
    case 3: return launch_pairs<3>(a, grad, st);
    case 4: return launch_pairs<4>(a, grad, st);
    case 5: return launch_pairs<5>(a, grad, st);
    case 6: return launch_pairs<6>(a, grad, st);
    case 7: return launch_pairs<7>(a, grad, st);
    case 8: return launch_pairs<8>(a, grad, st);
    case 9: return launch_pairs<9>(a, grad, st);
    case 10: return launch_pairs<10>(a, grad, st);
    case 11: return launch_pairs<11>(a, grad, st);
    default: return launch_pairs<12>(a, grad, st);
  }
}

// ----------------------------------------------------------------------------- divergence of voxel data
// -int grad B_t . n_v per pair (v, t): p_a = sum_k m_k f_k[r_a] scale, q_a = sum_k m_k f'_k[r_a].
struct DivArgs {
  const float* f[BASIS_MOST];
  const float* df[BASIS_MOST];
  int C, len;
  const float *coef, *data, *rel;
  const int64_t *vid, *tid;
  int64_t pairs;
  float mul, add, scale;
  double* b;                          // b[t] += value, or the gradient of sum lambda_t value:
  const double* lam;
  float *gcoef, *gdata;               // (either may be null)
};

NGS_DEV int div_offset(const DivArgs& a, float rel) {
  const float at = rintf(rel * a.mul + a.add);
  return at >= 0.f && at < (float)a.len ? (int)at : -1;
}

template <bool GRAD>
__global__ void __launch_bounds__(128) basis_divergence_kernel(const __grid_constant__ DivArgs a) {
  extern __shared__ float smem[];
  const int lane = threadIdx.x & 31, width = 3 * a.C, pitch = width | 1;
  float* own = smem + (int64_t)(threadIdx.x >> 5) * 32 * pitch;
  const int64_t step = ngs_gstride();
  for (int64_t t0 = ngs_gtid() - lane; t0 < a.pairs; t0 += step) {            // warp-uniform
    const int64_t t = t0 + lane;
    int64_t target = -1;
    if (t < a.pairs) {
      target = a.tid[t];
      const int64_t v = a.vid[t];
      const float* cr = a.coef + target * width;
      float p[3] = {0.f, 0.f, 0.f}, q[3] = {0.f, 0.f, 0.f}, n[3];
      int r[3];
#pragma unroll
      for (int x = 0; x < 3; x++) {
        n[x] = -a.data[3 * v + x];
        r[x] = div_offset(a, a.rel[3 * t + x]);
        if (r[x] < 0) p[x] = q[x] = __int_as_float(0x7fc00000);               // a pair no table covers
      }
      for (int k = 0; k < a.C; k++)
#pragma unroll
        for (int x = 0; x < 3; x++)
          if (r[x] >= 0) {
            const float c = cr[3 * k + x];
            p[x] += c * (__ldg(a.f[k] + r[x]) * a.scale);
            q[x] += c * __ldg(a.df[k] + r[x]);
          }
      if constexpr (!GRAD) {
        const float out = n[0] * q[0] * p[1] * p[2] + n[1] * p[0] * q[1] * p[2] + n[2] * p[0] * p[1] * q[2];
        atomicAdd(a.b + target, (double)out);
      } else {
        const float g = (float)a.lam[target];
        if (a.gdata) {
          atomicAdd(a.gdata + 3 * v, -(g * q[0] * p[1] * p[2]));
          atomicAdd(a.gdata + 3 * v + 1, -(g * p[0] * q[1] * p[2]));
          atomicAdd(a.gdata + 3 * v + 2, -(g * p[0] * p[1] * q[2]));
        }
        if (a.gcoef) {
          const float gq[3] = {g * n[0] * p[1] * p[2], g * n[1] * p[0] * p[2], g * n[2] * p[0] * p[1]};
          const float gp[3] = {g * (n[1] * q[1] * p[2] + n[2] * p[1] * q[2]), g * (n[0] * q[0] * p[2] + n[2] * p[0] * q[2]),
                               g * (n[0] * q[0] * p[1] + n[1] * p[0] * q[1])};
          for (int k = 0; k < a.C; k++)
#pragma unroll
            for (int x = 0; x < 3; x++)
              own[lane * pitch + 3 * k + x] = r[x] >= 0 ? gp[x] * (__ldg(a.f[k] + r[x]) * a.scale) + gq[x] * __ldg(a.df[k] + r[x])
                                                        : gp[x] + gq[x];
        }
      }
    }
    if constexpr (GRAD)
      if (a.gcoef) {
        __syncwarp();
        add_rows(own, pitch, width, target, a.gcoef);
        __syncwarp();
      }
  }
}

extern "C" int ngs_basis_divergence(const ngs_basis_div_term* p, int grad, ngs_stream s) {
  if (!p || p->pairs < 0 || p->C < 1 || p->C > BASIS_MOST || p->len < 1) return NGS_ERR_INVALID_ARG;
  if (p->pairs == 0) return NGS_OK;
  if (!p->coef || !p->data || !p->rel || !p->vid || !p->tid) return NGS_ERR_INVALID_ARG;
  if (grad ? (!p->lam || (!p->gcoef && !p->gdata)) : !p->b) return NGS_ERR_INVALID_ARG;
  DivArgs a{};
  for (int k = 0; k < p->C; k++) {
    if (!p->f[k] || !p->df[k]) return NGS_ERR_INVALID_ARG;
    a.f[k] = p->f[k];
    a.df[k] = p->df[k];
  }
  a.C = p->C, a.len = p->len;
  a.coef = p->coef, a.data = p->data, a.rel = p->rel, a.vid = p->vid, a.tid = p->tid, a.pairs = p->pairs;
  a.mul = p->mul, a.add = p->add, a.scale = p->scale;
  a.b = p->b, a.lam = p->lam, a.gcoef = p->gcoef, a.gdata = p->gdata;
  const unsigned grid = ngs_blocks(a.pairs, 128, 8);
  const size_t smem = sizeof(float) * 4 * 32 * ((3 * a.C) | 1);               // at most ROWS_SMEM
  ngs_count_launch();
  if (grad) {
    if (smem > 48 << 10) cudaFuncSetAttribute(basis_divergence_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, ROWS_SMEM);
    basis_divergence_kernel<true><<<grid, 128, smem, (cudaStream_t)s>>>(a);
  } else {
    basis_divergence_kernel<false><<<grid, 128, 0, (cudaStream_t)s>>>(a);
  }
  NGS_CHECK_LAUNCH();
  return NGS_OK;
}

// ----------------------------------------------------------------------------- values at the points
extern "C" int ngs_basis_axes(const ngs_basis_comps* comps, const float* coef, const float* x, int64_t m, float* f,
                              ngs_stream s) {
  BasisComps c;
  if (m < 0 || !comps_of(comps, c)) return NGS_ERR_INVALID_ARG;
  if (m == 0) return NGS_OK;
  if (!coef || !x || !f) return NGS_ERR_INVALID_ARG;
  { ngs_count_launch(); basis_axes_kernel<<<ngs_blocks(3 * m, 256), 256, 0, (cudaStream_t)s>>>(c, coef, x, m, f); }
  NGS_CHECK_LAUNCH();
  return NGS_OK;
}

extern "C" int ngs_basis_axes_grad(const ngs_basis_comps* comps, const float* x, const float* grad, int64_t m,
                                   float* gcoef, ngs_stream s) {
  BasisComps c;
  if (m < 0 || !comps_of(comps, c)) return NGS_ERR_INVALID_ARG;
  if (m == 0) return NGS_OK;
  if (!x || !grad || !gcoef) return NGS_ERR_INVALID_ARG;
  { ngs_count_launch(); basis_axes_grad_kernel<<<ngs_blocks(3 * m, 256), 256, 0, (cudaStream_t)s>>>(c, x, grad, m, gcoef); }
  NGS_CHECK_LAUNCH();
  return NGS_OK;
}

extern "C" int ngs_basis_phi(const ngs_basis_comps* comps, const float* coef, const int32_t* rows, const float* local,
                             int64_t n_points, float* phi, ngs_stream s) {
  BasisComps c;
  if (n_points < 0 || !comps_of(comps, c)) return NGS_ERR_INVALID_ARG;
  if (n_points == 0) return NGS_OK;
  if (!coef || !rows || !local || !phi) return NGS_ERR_INVALID_ARG;
  const int64_t m = 27 * n_points;
  { ngs_count_launch(); basis_phi_kernel<<<ngs_blocks(m, 128), 128, 0, (cudaStream_t)s>>>(c, coef, rows, local, m, phi); }
  NGS_CHECK_LAUNCH();
  return NGS_OK;
}

extern "C" int ngs_basis_phi_grad(const ngs_basis_comps* comps, const float* coef, const int32_t* rows, const float* local,
                                  int64_t n_points, const double* lam, const double* xs, const double* pa,
                                  const double* pb, float* gcoef, ngs_stream s) {
  BasisComps c;
  if (n_points < 0 || !comps_of(comps, c)) return NGS_ERR_INVALID_ARG;
  if (n_points == 0) return NGS_OK;
  if (!coef || !rows || !local || !lam || !xs || !pa || !pb || !gcoef) return NGS_ERR_INVALID_ARG;
  const int64_t m = 27 * n_points;
  const size_t smem = sizeof(float) * 4 * 32 * ((3 * c.count) | 1);
  if (smem > 48 << 10) cudaFuncSetAttribute(basis_phi_grad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, ROWS_SMEM);
  { ngs_count_launch(); basis_phi_grad_kernel<<<ngs_blocks(m, 128, 8), 128, smem, (cudaStream_t)s>>>(c, coef, rows, local, m, lam, xs, pa, pb,
                                                                                        gcoef); }
  NGS_CHECK_LAUNCH();
  return NGS_OK;
}

// A warp per point, a lane per slot.
__global__ void point_sum64_kernel(const float* __restrict__ phi, const int32_t* __restrict__ rows, int64_t n,
                                   const double* __restrict__ x, double* __restrict__ out) {
  const int lane = threadIdx.x & 31;
  for (int64_t p = ngs_gtid() >> 5; p < n; p += ngs_gstride() >> 5) {
    const int32_t r = lane < 27 ? rows[27 * p + lane] : -1;
    double v = r >= 0 ? (double)phi[27 * p + lane] * x[r] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) out[p] = v;
  }
}

__global__ void point_spread64_kernel(const float* __restrict__ phi, const int32_t* __restrict__ rows, int64_t n,
                                      const double* __restrict__ w, double scale, double* __restrict__ out) {
  const int lane = threadIdx.x & 31;
  for (int64_t p = ngs_gtid() >> 5; p < n; p += ngs_gstride() >> 5) {
    const int32_t r = lane < 27 ? rows[27 * p + lane] : -1;
    if (r >= 0) atomicAdd(out + r, scale * ((double)phi[27 * p + lane] * w[p]));
  }
}

extern "C" int ngs_point_sum64(const float* phi, const int32_t* rows, int64_t n, const double* x, double* out, ngs_stream s) {
  if (n < 0 || (n > 0 && (!phi || !rows || !x || !out))) return NGS_ERR_INVALID_ARG;
  if (n == 0) return NGS_OK;
  { ngs_count_launch(); point_sum64_kernel<<<ngs_blocks(n * 32, 256), 256, 0, (cudaStream_t)s>>>(phi, rows, n, x, out); }
  NGS_CHECK_LAUNCH();
  return NGS_OK;
}

extern "C" int ngs_point_spread64(const float* phi, const int32_t* rows, int64_t n, const double* w, double scale,
                                  double* out, ngs_stream s) {
  if (n < 0 || (n > 0 && (!phi || !rows || !w || !out))) return NGS_ERR_INVALID_ARG;
  if (n == 0) return NGS_OK;
  { ngs_count_launch(); point_spread64_kernel<<<ngs_blocks(n * 32, 256), 256, 0, (cudaStream_t)s>>>(phi, rows, n, w, scale, out); }
  NGS_CHECK_LAUNCH();
  return NGS_OK;
}
