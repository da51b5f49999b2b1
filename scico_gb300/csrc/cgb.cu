// Unrolled fixed-iteration CG block of the MoDL network with a hand-written
// backward: scico.flax.inverse.cg_solver (scico/flax/inverse.py:113-158) on
// (s H^T H + lam I) x = b for nsys independent images sharing the 2D
// projector H (s = gram_scale, e.g. c^2 for a projector scaled by c), and the
// reverse-mode recurrence of its K steps.
//
// Forward step k (float32 vectors, float64 scalars, per system):
//   Ap_k = s H^T H p_k + lam p_k;  d_k = <p_k, Ap_k>;  a_k = num_k / d_k
//   x += a_k p_k;  r_{k+1} = r_k - a_k Ap_k;  num_{k+1} = <r_{k+1}, r_{k+1}>
//   b_k = num_{k+1} / num_k;  p_{k+1} = r_{k+1} + b_k p_k
// with r_0 = b - A x_0, p_0 = r_0.  The tape keeps p_k, Ap_k, r_k and the
// scalars; with recompute it keeps only the scalars, and the backward reruns
// the forward from the block's inputs (its checkpoint) into the workspace.
//
// Backward step k, adjoints xb, rb, pb (of p_{k+1}), numb (of num_{k+1}):
//   bb = <pb, p_k>;  numb' = numb + bb / num_k;  nk = -bb num_{k+1} / num_k^2
//   rb += pb + 2 numb' r_{k+1};  ab = <xb, p_k> - <rb, Ap_k>
//   nk += ab / d_k;  db = -ab num_k / d_k^2
//   Apb = -a_k rb + db p_k;  lamb += <Apb, p_k>
//   pb = b_k pb + a_k xb + db Ap_k + A Apb;  numb = nk
// then rb_0 = rb + pb + 2 numb r_0 is the gradient of b, xb - A rb_0 that of
// x_0 and -<rb_0, x_0> is added to lamb.  Reductions are deterministic
// (fixed per-system trees), no float atomics.
#include <math.h>

#include <algorithm>

#include "kernels.cuh"

namespace {

constexpr int NT = ct::kReduceThreads;

// Per-system scalar block (doubles): running values, then one record per step.
enum { C_NUM = 0, C_NUMB = 1, C_LAMB = 2, C_NK = 3, C_DB = 4, C_HEAD = 8, C_REC = 5 };
enum { R_NUM = 0, R_D = 1, R_A = 2, R_B = 3, R_NUMN = 4 };

struct Sys {
  int nsys, nb;
  size_t n;
  int stride;  // doubles per system in the scalar block
};

__device__ __forceinline__ double* sys_scal(double* scal, const Sys& s, int sy) { return scal + (size_t)sy * s.stride; }
__device__ __forceinline__ double* rec(double* scal, const Sys& s, int sy, int k) {
  return sys_scal(scal, s, sy) + C_HEAD + C_REC * k;
}

// Reduction of K (<= 4) sums over the blocks of one system (grid = (nb, nsys),
// nb <= 64); true in thread 0 of the system's last block.  The block's first
// warp adds the threads' values as ct::block_reduce does and finishes alone: no
// block-wide barrier stands between the ticket and the result, and the last
// block's sum over the partials is that warp's too (16 images below: 2.82 ms
// with per-warp shuffle trees against 2.88 with grid_reduce_last as it was,
// 2.80 with the adds in one warp).
template <int K>
__device__ __forceinline__ void warp_sums(double (&v)[K]) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
    for (int k = 0; k < K; ++k) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
  }
}

template <int K>
__device__ __forceinline__ bool sys_reduce(double (&v)[K], double* partials, unsigned int* tickets, const Sys& s,
                                           double (&out)[K]) {
  __shared__ double red[K][NT];
  const int lane = threadIdx.x;
#pragma unroll
  for (int k = 0; k < K; ++k) red[k][threadIdx.x] = v[k];
  __syncthreads();
  if (threadIdx.x >= 32) return false;
  double* part = partials + (size_t)blockIdx.y * 4 * s.nb;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const double* r = red[k] + lane;
    v[k] = ((r[0] + r[32]) + (r[64] + r[96])) + ((r[128] + r[160]) + (r[192] + r[224]));
  }
  warp_sums<K>(v);
  int last = 0;
  if (lane == 0) {
#pragma unroll
    for (int k = 0; k < K; ++k) part[(size_t)K * blockIdx.x + k] = v[k];
    __threadfence();
    last = atomicAdd(tickets + blockIdx.y, 1u) == gridDim.x - 1;
  }
  if (!__shfl_sync(0xffffffffu, last, 0)) return false;
  __threadfence();
#pragma unroll
  for (int k = 0; k < K; ++k) {
    double a = lane < s.nb ? __ldcg(part + (size_t)K * lane + k) : 0.0;
    if (lane + 32 < s.nb) a += __ldcg(part + (size_t)K * (lane + 32) + k);
    out[k] = a;
  }
  warp_sums<K>(out);
  if (lane != 0) return false;
  tickets[blockIdx.y] = 0u;
  return true;
}

// The element passes below are read and write streams of a few vectors with one
// or two float64 dots.  A thread takes kE = 8 elements at a time in accesses of
// W (4: 128 bits, where the image size and every array allow it; else 1), all
// loads of a group before its arithmetic, so that one memory latency covers a
// whole image of 256^2 (32 blocks); dots go through ct::dot_group.
// H^T H v is taken as the adjoint left it: the view splits are summed here, in
// split order, instead of by a pass of their own.  16 images of 256^2, 6 steps,
// forward and backward: 3.24 -> 2.80 ms with the projections, which did not
// change (3.00 ms with each element's dot term converted to float64); one image
// of 256^2 0.95 -> 0.68 ms, odd sizes (5 x 255^2, W = 1) 1.27 -> 1.04 ms.
constexpr int kE = 8;

struct Gram {        // H^T H v: `ns` partial images `stride` floats apart
  const float* t;
  int ns;
  size_t stride;
};

template <int W>
__device__ __forceinline__ void ld(const float* p, size_t e0, size_t step, size_t end, float (&v)[kE]) {
#pragma unroll
  for (int u = 0; u < kE / W; ++u) {
    const size_t e = e0 + u * step;
    if constexpr (W == 4) {
      const float4 q = e < end ? *reinterpret_cast<const float4*>(p + e) : make_float4(0.f, 0.f, 0.f, 0.f);
      v[4 * u] = q.x, v[4 * u + 1] = q.y, v[4 * u + 2] = q.z, v[4 * u + 3] = q.w;
    } else {
      v[u] = e < end ? p[e] : 0.0f;
    }
  }
}

template <int W>
__device__ __forceinline__ void st(float* p, size_t e0, size_t step, size_t end, const float (&v)[kE]) {
#pragma unroll
  for (int u = 0; u < kE / W; ++u) {
    const size_t e = e0 + u * step;
    if (e < end) {
      if constexpr (W == 4)
        *reinterpret_cast<float4*>(p + e) = make_float4(v[4 * u], v[4 * u + 1], v[4 * u + 2], v[4 * u + 3]);
      else
        p[e] = v[u];
    }
  }
}

template <int W>
__device__ __forceinline__ void ld(const Gram& g, size_t e0, size_t step, size_t end, float (&v)[kE]) {
  ld<W>(g.t, e0, step, end, v);
#pragma unroll 4
  for (int k = 1; k < g.ns; ++k) {
    float w[kE];
    ld<W>(g.t + (size_t)k * g.stride, e0, step, end, w);
#pragma unroll
    for (int j = 0; j < kE; ++j) v[j] = ct::fadd(v[j], w[j]);
  }
}

#define FOR_SYS(W, e, s)                                                                           \
  const int sy = blockIdx.y;                                                                       \
  const size_t end = (size_t)(sy + 1) * (s).n, step = (size_t)(s).nb * NT * (W);                   \
  for (size_t e = (size_t)sy * (s).n + ((size_t)blockIdx.x * NT + threadIdx.x) * (W); e < end;     \
       e += (kE / (W)) * step)
#define EACH(j) _Pragma("unroll") for (int j = 0; j < kE; ++j)

// x = x0 (or 0);  r_0 = p_0 = b - (gs t + lam x0) (or b);  num = <r_0, r_0>.
template <int W>
__global__ void __launch_bounds__(NT)
    k_cgb_init(const float* __restrict__ b, Gram t, const float* x0, float* x, float* __restrict__ r0,
               float* __restrict__ p0, float gs, float lam, Sys s, double* __restrict__ scal,
               double* __restrict__ partials, unsigned int* __restrict__ tickets) {
  ct::grid_dep_wait();  // before any global access (dependent launch)
  ct::grid_dep_trigger();
  double nn = 0.0;
  FOR_SYS(W, e, s) {
    float r[kE], xv[kE] = {};
    ld<W>(b, e, step, end, r);
    if (x0) {
      float tv[kE];
      ld<W>(t, e, step, end, tv);
      ld<W>(x0, e, step, end, xv);
      EACH(j) r[j] = ct::fsub(r[j], ct::fadd(ct::fmul(gs, tv[j]), ct::fmul(lam, xv[j])));
    }
    st<W>(x, e, step, end, xv);
    st<W>(r0, e, step, end, r);
    st<W>(p0, e, step, end, r);
    nn += ct::dot_group(r, r);
  }
  double v[1] = {nn}, out[1];
  if (sys_reduce<1>(v, partials, tickets, s, out)) sys_scal(scal, s, sy)[C_NUM] = out[0];
}

// Ap = gs t + lam p (t = H^T H p), d = <p, Ap>, a = num / d.
template <int W>
__global__ void __launch_bounds__(NT)
    k_cgb_ap(Gram t, const float* __restrict__ p, float* __restrict__ ap, float gs, float lam, int k, Sys s,
             double* __restrict__ scal, double* __restrict__ partials, unsigned int* __restrict__ tickets) {
  ct::grid_dep_wait();  // before any global access (dependent launch)
  ct::grid_dep_trigger();
  double d = 0.0;
  FOR_SYS(W, e, s) {
    float a[kE], pv[kE];
    ld<W>(p, e, step, end, pv);
    ld<W>(t, e, step, end, a);
    EACH(j) a[j] = ct::fadd(ct::fmul(gs, a[j]), ct::fmul(lam, pv[j]));
    st<W>(ap, e, step, end, a);
    d += ct::dot_group(pv, a);
  }
  double v[1] = {d}, out[1];
  if (sys_reduce<1>(v, partials, tickets, s, out)) {
    const double num = sys_scal(scal, s, sy)[C_NUM];
    double* r = rec(scal, s, sy, k);
    r[R_NUM] = num;
    r[R_D] = out[0];
    r[R_A] = num / out[0];
  }
}

// x += a p; r' = r - a Ap; num' = <r', r'>; b = num' / num.
template <int W>
__global__ void __launch_bounds__(NT)
    k_cgb_upd(float* __restrict__ x, const float* __restrict__ r, float* __restrict__ rn, const float* __restrict__ p,
              const float* __restrict__ ap, int k, Sys s, double* __restrict__ scal, double* __restrict__ partials,
              unsigned int* __restrict__ tickets) {
  ct::grid_dep_wait();  // before any global access (dependent launch)
  ct::grid_dep_trigger();
  const float a = (float)rec(scal, s, blockIdx.y, k)[R_A];
  double nn = 0.0;
  FOR_SYS(W, e, s) {
    float xv[kE], rv[kE], pv[kE], av[kE];
    ld<W>(x, e, step, end, xv);
    ld<W>(p, e, step, end, pv);
    ld<W>(r, e, step, end, rv);
    ld<W>(ap, e, step, end, av);
    EACH(j) {
      xv[j] = ct::fadd(xv[j], ct::fmul(a, pv[j]));
      rv[j] = ct::fsub(rv[j], ct::fmul(a, av[j]));
    }
    st<W>(x, e, step, end, xv);
    st<W>(rn, e, step, end, rv);
    nn += ct::dot_group(rv, rv);
  }
  double v[1] = {nn}, out[1];
  if (sys_reduce<1>(v, partials, tickets, s, out)) {
    double* rr = rec(scal, s, sy, k);
    rr[R_NUMN] = out[0];
    rr[R_B] = out[0] / rr[R_NUM];
    sys_scal(scal, s, sy)[C_NUM] = out[0];
  }
}

// p' = r' + b p.
template <int W>
__global__ void __launch_bounds__(NT)
    k_cgb_dir(const float* __restrict__ rn, const float* __restrict__ p, float* __restrict__ pn, int k, Sys s,
              double* __restrict__ scal) {
  ct::grid_dep_wait();  // before any global access (dependent launch)
  ct::grid_dep_trigger();
  const float bt = (float)rec(scal, s, blockIdx.y, k)[R_B];
  FOR_SYS(W, e, s) {
    float rv[kE], pv[kE];
    ld<W>(rn, e, step, end, rv);
    ld<W>(p, e, step, end, pv);
    EACH(j) pv[j] = ct::fadd(rv[j], ct::fmul(bt, pv[j]));
    st<W>(pn, e, step, end, pv);
  }
}

// The backward's running scalars (numb, lamb) start at zero.
__global__ void k_cgb_reset(double* __restrict__ scal, Sys s) {
  for (int sy = threadIdx.x; sy < s.nsys; sy += blockDim.x) {
    scal[(size_t)sy * s.stride + C_NUMB] = 0.0;
    scal[(size_t)sy * s.stride + C_LAMB] = 0.0;
  }
}

// pb += gs t + lam Apb (the A Apb term of the previous backward step; pb = 0
// and no such term in the first, t.t == null);  bb = <pb, p_k>,
// numb' = numb + bb / num_k, nk = -bb num_{k+1} / num_k^2.
template <int W>
__global__ void __launch_bounds__(NT)
    k_cgb_b1(float* __restrict__ pb, Gram t, const float* __restrict__ apb, float gs, float lam,
             const float* __restrict__ pk, int k, Sys s, double* __restrict__ scal, double* __restrict__ partials,
             unsigned int* __restrict__ tickets) {
  ct::grid_dep_wait();  // before any global access (dependent launch)
  ct::grid_dep_trigger();
  double bb = 0.0;
  FOR_SYS(W, e, s) {
    float v[kE] = {}, pv[kE];
    ld<W>(pk, e, step, end, pv);
    if (t.t) {
      float tv[kE], gv[kE];
      ld<W>(pb, e, step, end, v);
      ld<W>(apb, e, step, end, gv);
      ld<W>(t, e, step, end, tv);
      EACH(j) v[j] = ct::fadd(v[j], ct::fadd(ct::fmul(gs, tv[j]), ct::fmul(lam, gv[j])));
    }
    st<W>(pb, e, step, end, v);
    bb += ct::dot_group(v, pv);
  }
  double v[1] = {bb}, out[1];
  if (sys_reduce<1>(v, partials, tickets, s, out)) {
    double* c = sys_scal(scal, s, sy);
    const double* r = rec(scal, s, sy, k);
    c[C_NUMB] += out[0] / r[R_NUM];
    c[C_NK] = -out[0] * r[R_NUMN] / (r[R_NUM] * r[R_NUM]);
  }
}

// rb += pb + 2 numb' r_{k+1} (rb = 0 before the first step);
// ab = <xb, p_k> - <rb, Ap_k>;  numb = nk + ab / d_k;  db = -ab num_k / d_k^2.
template <int W>
__global__ void __launch_bounds__(NT)
    k_cgb_b2(float* __restrict__ rb, int first, const float* __restrict__ pb, const float* __restrict__ rn,
             const float* __restrict__ xb, const float* __restrict__ pk, const float* __restrict__ apk, int k, Sys s,
             double* __restrict__ scal, double* __restrict__ partials, unsigned int* __restrict__ tickets) {
  ct::grid_dep_wait();  // before any global access (dependent launch)
  ct::grid_dep_trigger();
  const float tn = (float)(2.0 * sys_scal(scal, s, blockIdx.y)[C_NUMB]);
  double s_xp = 0.0, s_ra = 0.0;
  FOR_SYS(W, e, s) {
    float v[kE] = {}, w[kE], q[kE], xv[kE], pv[kE], av[kE];
    if (!first) ld<W>(rb, e, step, end, v);
    ld<W>(pb, e, step, end, w);
    ld<W>(rn, e, step, end, q);
    ld<W>(xb, e, step, end, xv);
    ld<W>(pk, e, step, end, pv);
    ld<W>(apk, e, step, end, av);
    EACH(j) v[j] = ct::fadd(ct::fadd(v[j], w[j]), ct::fmul(tn, q[j]));
    st<W>(rb, e, step, end, v);
    s_xp += ct::dot_group(xv, pv);
    s_ra += ct::dot_group(v, av);
  }
  double v[2] = {s_xp, s_ra}, out[2];
  if (sys_reduce<2>(v, partials, tickets, s, out)) {
    double* c = sys_scal(scal, s, sy);
    const double* r = rec(scal, s, sy, k);
    const double ab = out[0] - out[1];
    c[C_NUMB] = c[C_NK] + ab / r[R_D];
    c[C_DB] = -ab * r[R_NUM] / (r[R_D] * r[R_D]);
  }
}

// Apb = -a_k rb + db p_k;  pb = b_k pb + a_k xb + db Ap_k;  lamb += <Apb, p_k>.
template <int W>
__global__ void __launch_bounds__(NT)
    k_cgb_b3(const float* __restrict__ rb, const float* __restrict__ xb, float* __restrict__ pb,
             float* __restrict__ apb, const float* __restrict__ pk, const float* __restrict__ apk, int k, Sys s,
             double* __restrict__ scal, double* __restrict__ partials, unsigned int* __restrict__ tickets) {
  ct::grid_dep_wait();  // before any global access (dependent launch)
  ct::grid_dep_trigger();
  const double* r = rec(scal, s, blockIdx.y, k);
  const float a = (float)r[R_A], bt = (float)r[R_B], db = (float)sys_scal(scal, s, blockIdx.y)[C_DB];
  double lb = 0.0;
  FOR_SYS(W, e, s) {
    float g[kE], xv[kE], bv[kE], pv[kE], av[kE];
    ld<W>(rb, e, step, end, g);
    ld<W>(pk, e, step, end, pv);
    ld<W>(pb, e, step, end, bv);
    ld<W>(xb, e, step, end, xv);
    ld<W>(apk, e, step, end, av);
    EACH(j) {
      g[j] = ct::fadd(ct::fmul(-a, g[j]), ct::fmul(db, pv[j]));
      bv[j] = ct::fadd(ct::fadd(ct::fmul(bt, bv[j]), ct::fmul(a, xv[j])), ct::fmul(db, av[j]));
    }
    st<W>(apb, e, step, end, g);
    st<W>(pb, e, step, end, bv);
    lb += ct::dot_group(g, pv);
  }
  double v[1] = {lb}, out[1];
  if (sys_reduce<1>(v, partials, tickets, s, out)) sys_scal(scal, s, sy)[C_LAMB] += out[0];
}

// gb = rb + (pb + gs t + lam Apb) + 2 numb r_0 (the adjoint of r_0, which is
// that of b); rb = pb = 0 and no A Apb term where no step ran (t.t == null).
template <int W>
__global__ void __launch_bounds__(NT)
    k_cgb_rb0(const float* __restrict__ rb, const float* __restrict__ pb, Gram t, const float* __restrict__ apb,
              float gs, float lam, const float* __restrict__ r0, float* __restrict__ gb, Sys s,
              double* __restrict__ scal) {
  ct::grid_dep_wait();  // before any global access (dependent launch)
  ct::grid_dep_trigger();
  const float tn = (float)(2.0 * sys_scal(scal, s, blockIdx.y)[C_NUMB]);
  FOR_SYS(W, e, s) {
    float v[kE] = {}, w[kE] = {}, q[kE];
    ld<W>(r0, e, step, end, q);
    if (t.t) {
      float tv[kE], gv[kE];
      ld<W>(rb, e, step, end, v);
      ld<W>(pb, e, step, end, w);
      ld<W>(apb, e, step, end, gv);
      ld<W>(t, e, step, end, tv);
      EACH(j) w[j] = ct::fadd(w[j], ct::fadd(ct::fmul(gs, tv[j]), ct::fmul(lam, gv[j])));
    }
    EACH(j) v[j] = ct::fadd(ct::fadd(v[j], w[j]), ct::fmul(tn, q[j]));
    st<W>(gb, e, step, end, v);
  }
}

// gx0 = xb - (gs t + lam gb) (t = H^T H gb, gx0 may be null);  lamb -= <gb, x0>.
template <int W>
__global__ void __launch_bounds__(NT)
    k_cgb_x0(const float* __restrict__ xb, Gram t, const float* __restrict__ gb, const float* __restrict__ x0,
             float* __restrict__ gx0, float gs, float lam, Sys s, double* __restrict__ scal,
             double* __restrict__ partials, unsigned int* __restrict__ tickets) {
  ct::grid_dep_wait();  // before any global access (dependent launch)
  ct::grid_dep_trigger();
  double lb = 0.0;
  FOR_SYS(W, e, s) {
    float g[kE], xv[kE];
    ld<W>(gb, e, step, end, g);
    ld<W>(x0, e, step, end, xv);
    if (gx0) {
      float tv[kE], bv[kE];
      ld<W>(xb, e, step, end, bv);
      ld<W>(t, e, step, end, tv);
      EACH(j) bv[j] = ct::fsub(bv[j], ct::fadd(ct::fmul(gs, tv[j]), ct::fmul(lam, g[j])));
      st<W>(gx0, e, step, end, bv);
    }
    lb += ct::dot_group(g, xv);
  }
  double v[1] = {lb}, out[1];
  if (sys_reduce<1>(v, partials, tickets, s, out)) sys_scal(scal, s, sy)[C_LAMB] -= out[0];
}

// glam = sum of the systems' lamb, in system order.
__global__ void k_cgb_lamsum(const double* __restrict__ scal, Sys s, double* __restrict__ glam) {
  double acc = 0.0;
  for (int sy = 0; sy < s.nsys; ++sy) acc += scal[(size_t)sy * s.stride + C_LAMB];
  *glam = acc;
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------

#define CT_TRY(expr)              \
  do {                            \
    ct_status _st = (expr);       \
    if (_st != CT_OK) return _st; \
  } while (0)

struct Plan {
  Sys s;
  ct::Proj2dPlan p2;
  size_t vec;  // bytes of one batched vector
  size_t tape_vectors, tape_scal, tape_total;
  size_t ws_red, ws_proj, ws_sino, ws_tmp, ws_recompute, ws_total;
};

// Tape: P[K], AP[K], R[K+1] (none with recompute), then the scalars.
// Workspace: reduction area, projector scratch, sinogram, t and the
// backward's rb, pb, apb, xb (where a gradient is written over gx); with recompute also P, AP, R and x.
Plan plan_of(const ct_cg_block_desc* d) {
  Plan P;
  const size_t n = (size_t)d->geom.rows * d->geom.cols;
  const int K = d->maxiter;
  P.s.nsys = d->nsys;
  P.s.n = n;
  P.s.nb = (int)std::min<size_t>(64, std::max<size_t>(1, (n + 8 * NT - 1) / (8 * NT)));
  P.s.stride = C_HEAD + C_REC * K;
  P.p2 = ct::proj2d_plan(&d->geom, d->nsys);
  P.vec = ct::round_up((size_t)d->nsys * n * sizeof(float), 256);
  const size_t vectors = (size_t)(3 * K + 1) * P.vec;
  P.tape_vectors = d->recompute ? 0 : vectors;
  P.tape_scal = ct::round_up((size_t)d->nsys * P.s.stride * sizeof(double), 256);
  P.tape_total = P.tape_vectors + P.tape_scal;
  P.ws_red = ct::round_up((size_t)d->nsys * sizeof(unsigned int), 256) +
             ct::round_up((size_t)d->nsys * 4 * P.s.nb * sizeof(double), 256);
  P.ws_proj = ct::round_up(std::max<size_t>(std::max(P.p2.fwd_bytes, P.p2.adj_ws_bytes), 256), 256);
  P.ws_sino = ct::round_up((size_t)d->nsys * d->geom.n_views * d->geom.det_count * sizeof(float), 256);
  P.ws_tmp = 5 * P.vec;
  P.ws_recompute = d->recompute ? vectors + P.vec : 0;
  P.ws_total = P.ws_red + P.ws_proj + P.ws_sino + P.ws_tmp + P.ws_recompute;
  return P;
}

ct_status check(const ct_cg_block_desc* d, const char* who) {
  if (!d) return ct::fail(CT_ERR_INVALID_ARG, "%s: null descriptor", who);
  CT_TRY(ct::proj2d_check(&d->geom, who));
  if (d->nsys <= 0 || d->maxiter < 0)
    return ct::fail(CT_ERR_INVALID_ARG, "%s: nsys=%d maxiter=%d", who, d->nsys, d->maxiter);
  if (d->nsys > 65535) return ct::fail(CT_ERR_UNSUPPORTED, "%s: nsys=%d above 65535", who, d->nsys);
  return CT_OK;
}

struct Bufs {
  unsigned int* tickets;
  double* partials;
  float* proj_ws;
  float* sino;
  float *t, *rb, *pb, *apb, *xb;
  float *P, *AP, *R, *x;  // iterates: the tape's, or the workspace's with recompute
  double* scal;
};

Bufs bufs(const ct_cg_block_desc* d, const Plan& P, void* tape, void* ws, float* x_out) {
  Bufs B{};
  char* w = static_cast<char*>(ws);
  B.tickets = reinterpret_cast<unsigned int*>(w);
  B.partials = reinterpret_cast<double*>(w + ct::round_up((size_t)d->nsys * sizeof(unsigned int), 256));
  char* q = w + P.ws_red;
  B.proj_ws = reinterpret_cast<float*>(q);
  q += P.ws_proj;
  B.sino = reinterpret_cast<float*>(q);
  q += P.ws_sino;
  B.t = reinterpret_cast<float*>(q);
  B.rb = reinterpret_cast<float*>(q + P.vec);
  B.pb = reinterpret_cast<float*>(q + 2 * P.vec);
  B.apb = reinterpret_cast<float*>(q + 3 * P.vec);
  B.xb = reinterpret_cast<float*>(q + 4 * P.vec);
  q += P.ws_tmp;
  char* vec = d->recompute ? q : static_cast<char*>(tape);
  const int K = d->maxiter;
  B.P = reinterpret_cast<float*>(vec);
  B.AP = reinterpret_cast<float*>(vec + (size_t)K * P.vec);
  B.R = reinterpret_cast<float*>(vec + (size_t)2 * K * P.vec);
  B.x = d->recompute ? reinterpret_cast<float*>(vec + (size_t)(3 * K + 1) * P.vec) : x_out;
  B.scal = reinterpret_cast<double*>(static_cast<char*>(tape) + P.tape_vectors);
  return B;
}

float* at(float* base, const Plan& P, int k) {
  return reinterpret_cast<float*>(reinterpret_cast<char*>(base) + (size_t)k * P.vec);
}

// t = H^T H v for the batch: forward projection, then the adjoint, whose view
// splits the next pass sums.  v is the output of one of this file's kernels
// (dependent) or the caller's.
ct_status gram(const ct_cg_block_desc* d, const Plan& P, const Bufs& B, const float* v, Gram& t, cudaStream_t s,
               bool dependent) {
  CT_TRY(ct::proj2d_fwd_launch(&d->geom, P.p2, v, B.sino, d->nsys, B.proj_ws, s, nullptr, dependent));
  CT_TRY(ct::proj2d_adj_launch(&d->geom, P.p2, B.sino, B.t, B.proj_ws, d->nsys, s, nullptr, true));
  t = Gram{P.p2.nsplit > 1 ? B.proj_ws : B.t, P.p2.nsplit, (size_t)d->nsys * P.s.n};
  return CT_OK;
}

// A pass over all systems in its W = 4 form where `vec`, else in its W = 1 form.
template <class... K, class... A>
ct_status pass(const char* name, const Plan& P, cudaStream_t s, bool dependent, int vec, void (*k4)(K...),
               void (*k1)(K...), A... args) {
  const dim3 g((unsigned)P.s.nb, (unsigned)P.s.nsys, 1);
  return ct::cuda_check(ct::launch_k(vec ? k4 : k1, g, dim3(NT), 0, s, dependent, args...), name);
}
#define PASS(k, dependent, vec, ...) CT_TRY(pass(#k, P, s, dependent, vec, k<4>, k<1>, __VA_ARGS__))

ct_status forward(const ct_cg_block_desc* d, const Plan& P, const Bufs& B, const float* b, float lam,
                  const float* x0, cudaStream_t s) {
  const float gs = d->gram_scale;
  const int vec = ct::quad_ok(P.s.n, b, x0, B.x);  // the tape and workspace vectors are 256-B aligned
  Gram t{};
  if (x0) CT_TRY(gram(d, P, B, x0, t, s, false));
  const int K = d->maxiter;
  PASS(k_cgb_init, x0 != nullptr, vec, b, t, x0, B.x, at(B.R, P, 0), K > 0 ? at(B.P, P, 0) : B.pb, gs, lam, P.s,
       B.scal, B.partials, B.tickets);
  for (int k = 0; k < K; ++k) {
    float* pk = at(B.P, P, k);
    float* apk = at(B.AP, P, k);
    CT_TRY(gram(d, P, B, pk, t, s, true));
    PASS(k_cgb_ap, true, vec, t, pk, apk, gs, lam, k, P.s, B.scal, B.partials, B.tickets);
    PASS(k_cgb_upd, true, vec, B.x, at(B.R, P, k), at(B.R, P, k + 1), pk, apk, k, P.s, B.scal, B.partials, B.tickets);
    if (k + 1 < K)
      PASS(k_cgb_dir, true, vec, at(B.R, P, k + 1), pk, at(B.P, P, k + 1), k, P.s, B.scal);
  }
  return CT_OK;
}

ct_status buffers_check(const Plan& P, void* tape, size_t tape_bytes, void* ws, size_t ws_bytes, const char* who) {
  if (!tape || tape_bytes < P.tape_total || !ct::aligned(tape, 256))
    return ct::fail(CT_ERR_WORKSPACE, "%s: tape needs %zu bytes (256-B aligned), got %zu", who, P.tape_total,
                    tape_bytes);
  if (!ws || ws_bytes < P.ws_total || !ct::aligned(ws, 256))
    return ct::fail(CT_ERR_WORKSPACE, "%s: workspace needs %zu bytes (256-B aligned), got %zu", who, P.ws_total,
                    ws_bytes);
  return CT_OK;
}

}  // namespace

extern "C" {

ct_status ct_cg_block_workspace(const ct_cg_block_desc* d, size_t* tape_bytes, size_t* ws_bytes) {
  CT_TRY(check(d, "ct_cg_block_workspace"));
  const Plan P = plan_of(d);
  if (tape_bytes) *tape_bytes = P.tape_total;
  if (ws_bytes) *ws_bytes = P.ws_total;
  return CT_OK;
}

ct_status ct_cg_block_fwd(const ct_cg_block_desc* d, const float* b, float lam, const float* x0, float* x,
                          void* tape, size_t tape_bytes, void* workspace, size_t workspace_bytes,
                          ct_stream_t stream) {
  const char* who = "ct_cg_block_fwd";
  CT_TRY(check(d, who));
  if (!b || !x) return ct::fail(CT_ERR_INVALID_ARG, "%s: null array", who);
  const Plan P = plan_of(d);
  CT_TRY(buffers_check(P, tape, tape_bytes, workspace, workspace_bytes, who));
  CT_TRY(ct::proj2d_prepare(P.p2));
  cudaStream_t s = ct::as_stream(stream);
  CT_TRY(ct::cuda_check(cudaMemsetAsync(workspace, 0, P.ws_red, s), "reduction init"));
  const Bufs B = bufs(d, P, tape, workspace, x);
  CT_TRY(forward(d, P, B, b, lam, x0, s));
  if (d->recompute)
    CT_TRY(ct::cuda_check(
        cudaMemcpyAsync(x, B.x, (size_t)d->nsys * P.s.n * sizeof(float), cudaMemcpyDeviceToDevice, s), "x copy"));
  return CT_OK;
}

ct_status ct_cg_block_bwd(const ct_cg_block_desc* d, const float* gx, const float* b, float lam, const float* x0,
                          void* tape, size_t tape_bytes, float* gb, float* gx0, double* glam, void* workspace,
                          size_t workspace_bytes, ct_stream_t stream) {
  const char* who = "ct_cg_block_bwd";
  CT_TRY(check(d, who));
  if (!gx || !gb || !glam) return ct::fail(CT_ERR_INVALID_ARG, "%s: null array", who);
  if (d->recompute && !b) return ct::fail(CT_ERR_INVALID_ARG, "%s: recompute needs b", who);
  if (gx0 && !x0) return ct::fail(CT_ERR_INVALID_ARG, "%s: gx0 without x0", who);
  const Plan P = plan_of(d);
  CT_TRY(buffers_check(P, tape, tape_bytes, workspace, workspace_bytes, who));
  CT_TRY(ct::proj2d_prepare(P.p2));
  cudaStream_t s = ct::as_stream(stream);
  CT_TRY(ct::cuda_check(cudaMemsetAsync(workspace, 0, P.ws_red, s), "reduction init"));
  const Bufs B = bufs(d, P, tape, workspace, nullptr);
  if (d->recompute) CT_TRY(forward(d, P, B, b, lam, x0, s));  // the iterates from the block's inputs
  const float gs = d->gram_scale;
  const size_t nbytes = (size_t)d->nsys * P.s.n * sizeof(float);
  auto over = [&](const float* p) {
    const char *u = reinterpret_cast<const char*>(gx), *w = reinterpret_cast<const char*>(p);
    return p && u < w + nbytes && w < u + nbytes;
  };
  if (over(gb) || over(gx0)) {  // gx is read to the end
    CT_TRY(ct::cuda_check(cudaMemcpyAsync(B.xb, gx, nbytes, cudaMemcpyDeviceToDevice, s), "gx copy"));
    gx = B.xb;
  }
  const int vec = ct::quad_ok(P.s.n, gx, x0, gb, gx0);
  k_cgb_reset<<<1, 256, 0, s>>>(B.scal, P.s);
  CT_TRY(ct::launch_check("k_cgb_reset"));
  const int K = d->maxiter;
  Gram t{};  // H^T H apb of the previous backward step
  for (int k = K - 1; k >= 0; --k) {
    const float* pk = at(B.P, P, k);
    const float* apk = at(B.AP, P, k);
    const int first = k == K - 1;
    PASS(k_cgb_b1, !first, vec, B.pb, t, B.apb, gs, lam, pk, k, P.s, B.scal, B.partials, B.tickets);
    PASS(k_cgb_b2, true, vec, B.rb, first, B.pb, at(B.R, P, k + 1), gx, pk, apk, k, P.s, B.scal, B.partials,
         B.tickets);
    PASS(k_cgb_b3, true, vec, B.rb, gx, B.pb, B.apb, pk, apk, k, P.s, B.scal, B.partials, B.tickets);
    CT_TRY(gram(d, P, B, B.apb, t, s, true));
  }
  PASS(k_cgb_rb0, K > 0, vec, B.rb, B.pb, t, B.apb, gs, lam, at(B.R, P, 0), gb, P.s, B.scal);
  if (x0) {
    CT_TRY(gram(d, P, B, gb, t, s, true));
    PASS(k_cgb_x0, true, vec, gx, t, gb, x0, gx0, gs, lam, P.s, B.scal, B.partials, B.tickets);
  }
  k_cgb_lamsum<<<1, 1, 0, s>>>(B.scal, P.s, glam);
  return ct::launch_check("k_cgb_lamsum");
}

}  // extern "C"
