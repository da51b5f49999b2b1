// Finite differences (scico FiniteDifference), their adjoint, and the
// L2,1 / L1 proximal operators and norms (scico/functional/_norm.py).
#include <math.h>

#include <algorithm>

#include "common.cuh"

namespace {

struct FdBlock {
  int axis;    // differenced axis (0..2 of the 3-D padded shape)
  int M;       // output length along that axis
  size_t off;  // element offset of this block in the concatenated output
  size_t count;
};

struct FdParams {
  int n[3];  // padded 3-D input shape
  int nblocks;
  FdBlock blk[3];
  int prepend, append, circular;
  size_t in_count;   // elements of one input
  size_t out_count;  // elements of one output (all blocks)
};

ct_status make_fd(const ct_fd_desc* d, FdParams& p, const char* who) {
  if (!d) return ct::fail(CT_ERR_INVALID_ARG, "%s: null descriptor", who);
  if (d->ndim < 1 || d->ndim > 3) return ct::fail(CT_ERR_UNSUPPORTED, "%s: ndim=%d", who, d->ndim);
  if (d->naxes < 1 || d->naxes > d->ndim)
    return ct::fail(CT_ERR_INVALID_ARG, "%s: naxes=%d", who, d->naxes);
  if (d->prepend < -1 || d->prepend > 1 || d->append < -1 || d->append > 1)
    return ct::fail(CT_ERR_INVALID_ARG, "%s: prepend/append must be -1, 0 or 1", who);
  if (d->circular && (d->prepend != -1 || d->append != -1))
    return ct::fail(CT_ERR_INVALID_ARG, "%s: circular needs prepend = append = None", who);
  const int pad = 3 - d->ndim;
  for (int k = 0; k < 3; ++k) p.n[k] = 1;
  for (int k = 0; k < d->ndim; ++k) {
    if (d->shape[k] <= 0) return ct::fail(CT_ERR_SHAPE, "%s: shape[%d]=%d", who, k, d->shape[k]);
    p.n[pad + k] = d->shape[k];
  }
  p.prepend = d->prepend;
  p.append = d->append;
  p.circular = d->circular ? 1 : 0;
  p.nblocks = d->naxes;
  p.in_count = (size_t)p.n[0] * p.n[1] * p.n[2];
  size_t off = 0;
  for (int k = 0; k < d->naxes; ++k) {
    const int ax = d->axes[k];
    if (ax < 0 || ax >= d->ndim) return ct::fail(CT_ERR_INVALID_ARG, "%s: axis %d", who, ax);
    for (int q = 0; q < k; ++q)
      if (d->axes[q] == ax) return ct::fail(CT_ERR_INVALID_ARG, "%s: repeated axis %d", who, ax);
    const int a3 = pad + ax;
    const int n = p.n[a3];
    int M = p.circular ? n : n + (p.prepend >= 0) + (p.append >= 0) - 1;
    if (M < 0) M = 0;
    p.blk[k].axis = a3;
    p.blk[k].M = M;
    p.blk[k].off = off;
    p.blk[k].count = p.in_count / n * M;
    off += p.blk[k].count;
  }
  p.out_count = off;
  return CT_OK;
}

// ---------------------------------------------------------------------------
// Same-shape differences (circular, or exactly one end extended: every output
// block has the input's shape), the form of every regulariser here.  Bound by
// memory; what cost the time before was index arithmetic (two 64-bit divisions
// an element) and one element in flight per thread.
//
// Rows of a whole number of quads in aligned arrays (k_fd_*_quads): a thread
// takes four elements of a row, whose coordinates cost two 32-bit multiply-high
// divisions a quad, and its six loads are all in flight.  Other rows of at
// least a warp (k_fd_rows): a warp takes up to kFdU elements a lane of one
// row (the last axis), so the position along the other axes, and with it the
// offset to the neighbour and the test for the line's end, is the same for
// the whole warp and costs nothing per element.  Shorter ones (k_fd_*_flat) would
// leave lanes idle: there a thread takes kFdU elements of the flat array
// kFdT apart, or one (one_each: 17 x 19 x 23 2.9 / 3.9 -> 1.9 / 2.1 us).  A copied end's second term is behind a branch that few threads
// take: as a select it cost the adjoint more than its loads (192^3 in quads 22.3 us).
// 192^3, three axes (forward / adjoint): 177 / 150 us with the divisions of
// k_fd_fwd / k_fd_adj, 43 / 62 us flat, 18.8 / 27.7 us by rows, 17.4 / 19.9 us
// in quads (113 MB each: 17 us of measured bandwidth); 300 x 200 x 100 17.7 /
// 21.5 by rows, 12.7 / 13.7 in quads; 100 x 100 x 20 3.7 / 4.2 flat, 2.0 / 2.1.
// ---------------------------------------------------------------------------
constexpr int kFdT = 256;  // threads of a block
constexpr int kFdU = 4;    // elements per thread

// One element a thread where the SMs hold a thread for each (eight CTAs of 256 an
// SM): there a thread's second element only lengthens the launch.
bool one_each(size_t n) { return n <= (size_t)ct::sm_count() * 8 * 256; }

// Division of 31-bit unsigned numbers by a fixed divisor: q = (mulhi(e, m) + e) >> s.
struct FastDiv {
  uint32_t d, m, s;
};
FastDiv fast_div(uint32_t d) {
  FastDiv f{d, 0, 0};
  while ((1u << f.s) < d && f.s < 31) ++f.s;
  f.m = (uint32_t)((((1ull << f.s) - d) << 32) / d + 1);
  return f;
}
__device__ __forceinline__ uint32_t div_by(const FastDiv& f, uint32_t e) { return (__umulhi(e, f.m) + e) >> f.s; }

struct FdSame {
  uint32_t count;  // elements of one input
  FastDiv n2, n1;
  int n[3];
  int axis[3];
  uint32_t stride[3];  // of axis[k]
  int mode;            // 0 circular, 1 append, 2 prepend
  int zero;            // extended sample: 0 = copy of the end, 1 = zero
  // by rows: elements a lane, chunks of 32 per_lane elements in a row, their total
  int per_lane;
  uint32_t units;
  FastDiv chunks;
};

// True when `p` is same-shape and every index fits 31 bits (the descriptor's
// divisors must be below 2^31 for fast_div).
bool make_same(const FdParams& p, FdSame& q) {
  const bool pre = p.prepend >= 0, app = p.append >= 0;
  if (!p.circular && pre == app) return false;
  if (p.in_count >= (1ull << 31)) return false;
  q.count = (uint32_t)p.in_count;
  q.n1 = fast_div((uint32_t)p.n[1]);
  q.n2 = fast_div((uint32_t)p.n[2]);
  for (int k = 0; k < 3; ++k) q.n[k] = p.n[k];
  for (int k = 0; k < p.nblocks; ++k) {
    q.axis[k] = p.blk[k].axis;
    q.stride[k] = q.axis[k] == 2 ? 1u : (q.axis[k] == 1 ? (uint32_t)p.n[2] : (uint32_t)p.n[1] * (uint32_t)p.n[2]);
  }
  q.mode = p.circular ? 0 : (app ? 1 : 2);
  q.zero = p.circular ? 0 : (app ? p.append : p.prepend);
  // the elements a lane takes: whichever of 1..kFdU leaves the fewest lanes of
  // a row's last chunk idle, the most of those
  int best = 0;
  uint32_t least = 0xffffffffu;
  for (int u = 1; u <= kFdU; ++u) {
    const uint32_t span = 32u * u, used = ((uint32_t)p.n[2] + span - 1) / span * span;
    if (used <= least) {
      least = used;
      best = u;
    }
  }
  q.per_lane = best;
  const uint32_t chunks = ((uint32_t)p.n[2] + 32u * best - 1) / (32u * best);
  q.chunks = fast_div(chunks);
  q.units = (uint32_t)(p.in_count / p.n[2]) * chunks;
  return true;
}

__device__ __forceinline__ void fd_coords(const FdSame& q, uint32_t e, int (&c)[3]) {
  const uint32_t r = div_by(q.n2, e);
  c[2] = (int)(e - r * (uint32_t)q.n[2]);
  c[0] = (int)div_by(q.n1, r);
  c[1] = (int)(r - (uint32_t)c[0] * (uint32_t)q.n[1]);
}

// out[k][e] = (next) - (this) along axis k, next the circular neighbour or the
// extended sample at the end (append), or (this) - (previous) (prepend).
template <int NB, int U>
__global__ void __launch_bounds__(kFdT) k_fd_fwd_flat(const float* __restrict__ x, float* __restrict__ out, const FdSame q) {
  x += (size_t)blockIdx.y * q.count;
  out += (size_t)blockIdx.y * NB * q.count;
  const uint32_t e0 = blockIdx.x * (uint32_t)(kFdT * U) + threadIdx.x;
  float xc[U], xn[U][NB];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const uint32_t e = min(e0 + u * kFdT, q.count - 1);  // loads stay unconditional, all in flight
    int c[3];
    fd_coords(q, e, c);
    xc[u] = __ldg(x + e);
#pragma unroll
    for (int k = 0; k < NB; ++k) {
      const int a = q.axis[k], ca = a == 2 ? c[2] : (a == 1 ? c[1] : c[0]), na = a == 2 ? q.n[2] : (a == 1 ? q.n[1] : q.n[0]);
      const bool end = q.mode == 2 ? ca == 0 : ca == na - 1;
      // mode 0 wraps to the line's start; an extended end reads its own sample
      const uint32_t at = end ? (q.mode == 0 ? e - (uint32_t)ca * q.stride[k] : e)
                              : (q.mode == 2 ? e - q.stride[k] : e + q.stride[k]);
      const float v = __ldg(x + at);
      xn[u][k] = end && q.zero ? 0.0f : v;
    }
  }
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const uint32_t e = e0 + u * kFdT;
    if (e >= q.count) break;
#pragma unroll
    for (int k = 0; k < NB; ++k)
      out[(size_t)k * q.count + e] = q.mode == 2 ? ct::fsub(xc[u], xn[u][k]) : ct::fsub(xn[u][k], xc[u]);
  }
}

// x[e] = sum over axes, in axis order, of the extended line's cotangents
// ce[t] = d[t-1] - d[t] (terms off the line are 0) at the positions holding
// x[e]; an end copied by the extension holds two, added in position order
// (k_fd_adj below states the rule in general).
template <int NB, int U>
__global__ void __launch_bounds__(kFdT) k_fd_adj_flat(const float* __restrict__ d, float* __restrict__ x, const FdSame q) {
  d += (size_t)blockIdx.y * NB * q.count;
  x += (size_t)blockIdx.y * q.count;
  const uint32_t e0 = blockIdx.x * (uint32_t)(kFdT * U) + threadIdx.x;
  float dc[U][NB], dn[U][NB];
  unsigned two = 0;  // bit u*NB + k: the sample is a copied end
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const uint32_t e = min(e0 + u * kFdT, q.count - 1);  // loads stay unconditional, all in flight
    int c[3];
    fd_coords(q, e, c);
#pragma unroll
    for (int k = 0; k < NB; ++k) {
      const float* dk = d + (size_t)k * q.count;
      const int a = q.axis[k], ca = a == 2 ? c[2] : (a == 1 ? c[1] : c[0]), na = a == 2 ? q.n[2] : (a == 1 ? q.n[1] : q.n[0]);
      // the neighbour of the cotangent pair: the previous difference
      // (circular, append) or the next one (prepend)
      const bool off = q.mode == 2 ? ca == na - 1 : ca == 0;
      const uint32_t at = off ? (q.mode == 0 ? e + (uint32_t)(na - 1) * q.stride[k] : e)
                              : (q.mode == 2 ? e + q.stride[k] : e - q.stride[k]);
      const float v = __ldg(dk + at);
      dc[u][k] = __ldg(dk + e);
      dn[u][k] = off && q.mode != 0 ? 0.0f : v;
      const bool copied = q.mode != 0 && !q.zero && (q.mode == 2 ? ca == 0 : ca == na - 1);
      if (copied) two |= 1u << (u * NB + k);
    }
  }
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const uint32_t e = e0 + u * kFdT;
    if (e >= q.count) break;
    float acc = 0.0f;
#pragma unroll
    for (int k = 0; k < NB; ++k) {
      const bool cp = (two >> (u * NB + k)) & 1u;
      float v;
      if (q.mode == 2) {
        v = ct::fsub(dc[u][k], dn[u][k]);
        if (cp) v = ct::fadd(ct::fsub(0.0f, dc[u][k]), v);  // position 0 first
      } else {
        v = ct::fsub(dn[u][k], dc[u][k]);
        if (cp) v = ct::fadd(v, dc[u][k]);  // then the position past the end: d[n-1] - 0
      }
      acc = k == 0 ? v : ct::fadd(acc, v);
    }
    x[e] = acc;
  }
}

// This warp's row and the lane's first element of it; false past the end.
struct FdRow {
  uint32_t row, c0, c1, c2;  // row index, coordinates (c2: the lane's first element)
};
__device__ __forceinline__ bool fd_row(const FdSame& q, FdRow& r) {
  const uint32_t w = blockIdx.x * (kFdT / 32) + (threadIdx.x >> 5);
  if (w >= q.units) return false;
  r.row = div_by(q.chunks, w);
  r.c0 = div_by(q.n1, r.row);
  r.c1 = r.row - r.c0 * (uint32_t)q.n[1];
  r.c2 = (w - r.row * q.chunks.d) * 32u * (uint32_t)q.per_lane + (threadIdx.x & 31);
  return true;
}

// The forward and the adjoint below, by rows; U = FdSame::per_lane, MODE =
// FdSame::mode.  FULL: the warp's whole chunk lies in the row, so every load
// is unconditional at an immediate offset from its axis's base address.
template <int NB, int U, int MODE, bool FULL>
__device__ __forceinline__ void fd_fwd_row(const float* __restrict__ x, float* __restrict__ out, const FdSame& q,
                                           const FdRow& r) {
  constexpr bool back = MODE == 2, wrap = MODE == 0;
  const int n2 = q.n[2], c = (int)r.c2;
  const float* __restrict__ xp = x + (size_t)blockIdx.y * q.count + r.row * (uint32_t)n2 + c;
  float xc[U], xn[NB][U];
#pragma unroll
  for (int u = 0; u < U; ++u)
    if (FULL || c + 32 * u < n2) xc[u] = __ldg(xp + 32 * u);
#pragma unroll
  for (int k = 0; k < NB; ++k) {
    const int a = q.axis[k];
    if (a == 2) {
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (FULL || c + 32 * u < n2) {
          const bool end = back ? c + 32 * u == 0 : c + 32 * u == n2 - 1;
          const int off = end ? (wrap ? -(c + 32 * u) : 0) : (back ? -1 : 1);
          xn[k][u] = __ldg(xp + 32 * u + off);
          if (!wrap && end && q.zero) xn[k][u] = 0.0f;
        }
    } else {
      const int ca = (int)(a == 1 ? r.c1 : r.c0), na = a == 1 ? q.n[1] : q.n[0];
      const bool end = back ? ca == 0 : ca == na - 1;
      const ptrdiff_t st = (ptrdiff_t)q.stride[k];
      const float* __restrict__ np = xp + (end ? (wrap ? -(ptrdiff_t)ca * st : 0) : (back ? -st : st));
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (FULL || c + 32 * u < n2) {
          xn[k][u] = __ldg(np + 32 * u);
          if (!wrap && end && q.zero) xn[k][u] = 0.0f;
        }
    }
  }
  float* __restrict__ op = out + (size_t)blockIdx.y * NB * q.count + r.row * (uint32_t)n2 + c;
#pragma unroll
  for (int k = 0; k < NB; ++k)
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (FULL || c + 32 * u < n2)
        op[(size_t)k * q.count + 32 * u] = back ? ct::fsub(xc[u], xn[k][u]) : ct::fsub(xn[k][u], xc[u]);
}

template <int NB, int U, int MODE, bool FULL>
__device__ __forceinline__ void fd_adj_row(const float* __restrict__ d, float* __restrict__ x, const FdSame& q,
                                           const FdRow& r) {
  constexpr bool fwd = MODE == 2, wrap = MODE == 0;
  const int n2 = q.n[2], c = (int)r.c2;
  const float* __restrict__ dp = d + (size_t)blockIdx.y * NB * q.count + r.row * (uint32_t)n2 + c;
  float dc[NB][U], dn[NB][U];
#pragma unroll
  for (int k = 0; k < NB; ++k) {
    const float* __restrict__ dk = dp + (size_t)k * q.count;
    const int a = q.axis[k];
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (FULL || c + 32 * u < n2) dc[k][u] = __ldg(dk + 32 * u);
    if (a == 2) {
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (FULL || c + 32 * u < n2) {
          const bool off = fwd ? c + 32 * u == n2 - 1 : c + 32 * u == 0;
          const int at = off ? (wrap ? n2 - 1 : 0) : (fwd ? 1 : -1);
          dn[k][u] = __ldg(dk + 32 * u + at);
          if (!wrap && off) dn[k][u] = 0.0f;
        }
    } else {
      const int ca = (int)(a == 1 ? r.c1 : r.c0), na = a == 1 ? q.n[1] : q.n[0];
      const bool off = fwd ? ca == na - 1 : ca == 0;
      const ptrdiff_t st = (ptrdiff_t)q.stride[k];
      const float* __restrict__ np = dk + (off ? (wrap ? (ptrdiff_t)(na - 1) * st : 0) : (fwd ? st : -st));
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (FULL || c + 32 * u < n2) {
          dn[k][u] = __ldg(np + 32 * u);
          if (!wrap && off) dn[k][u] = 0.0f;
        }
    }
  }
  float* __restrict__ op = x + (size_t)blockIdx.y * q.count + r.row * (uint32_t)n2 + c;
  float acc[U];
#pragma unroll
  for (int k = 0; k < NB; ++k) {
    float v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) v[u] = fwd ? ct::fsub(dc[k][u], dn[k][u]) : ct::fsub(dn[k][u], dc[k][u]);
    if (!wrap && !q.zero) {  // a copied end: position 0 first, or then the position past the end (d[n-1] - 0)
      const int a = q.axis[k];
      const int ca = (int)(a == 1 ? r.c1 : r.c0), na = a == 1 ? q.n[1] : q.n[0];
      if (a == 2 || (fwd ? ca == 0 : ca == na - 1)) {
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (a != 2 || (fwd ? c + 32 * u == 0 : c + 32 * u == n2 - 1))
            v[u] = fwd ? ct::fadd(ct::fsub(0.0f, dc[k][u]), v[u]) : ct::fadd(v[u], dc[k][u]);
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) acc[u] = k == 0 ? v[u] : ct::fadd(acc[u], v[u]);
  }
#pragma unroll
  for (int u = 0; u < U; ++u)
    if (FULL || c + 32 * u < n2) op[32 * u] = acc[u];
}

template <int NB, int U, int MODE, bool ADJ>
__global__ void __launch_bounds__(kFdT) k_fd_rows(const float* __restrict__ src, float* __restrict__ dst, const FdSame q) {
  FdRow r;
  if (!fd_row(q, r)) return;
  const bool full = (int)(r.c2 | 31u) + 32 * (U - 1) < q.n[2];  // c2 of lane 0 is a multiple of 32
  if (ADJ) {
    if (full)
      fd_adj_row<NB, U, MODE, true>(src, dst, q, r);
    else
      fd_adj_row<NB, U, MODE, false>(src, dst, q, r);
  } else {
    if (full)
      fd_fwd_row<NB, U, MODE, true>(src, dst, q, r);
    else
      fd_fwd_row<NB, U, MODE, false>(src, dst, q, r);
  }
}

// Quads (rows of a whole number of them, 16-byte aligned arrays): a thread takes four consecutive elements, its
// neighbours along the last axis from the quad itself and one more element.
template <int NB, int MODE>
__global__ void __launch_bounds__(kFdT) k_fd_fwd_quads(const float* __restrict__ x, float* __restrict__ out, const FdSame q) {
  constexpr bool back = MODE == 2, wrap = MODE == 0;
  const uint32_t e = 4 * (blockIdx.x * (uint32_t)kFdT + threadIdx.x);
  if (e >= q.count) return;
  int c[3];
  fd_coords(q, e, c);
  const float* __restrict__ xp = x + (size_t)blockIdx.y * q.count + e;
  const float4 x4 = __ldg(reinterpret_cast<const float4*>(xp));
  const float xc[4] = {x4.x, x4.y, x4.z, x4.w};
  float xn[NB][4];
#pragma unroll
  for (int k = 0; k < NB; ++k) {
    const int a = q.axis[k];
    if (a == 2) {
      const bool end = back ? c[2] == 0 : c[2] + 4 == q.n[2];
      const int at = back ? (end ? (wrap ? q.n[2] - 1 : 0) : -1) : (end ? (wrap ? 4 - q.n[2] : 3) : 4);
      float far = __ldg(xp + at);
      if (!wrap && end && q.zero) far = 0.0f;
#pragma unroll
      for (int j = 0; j < 4; ++j) xn[k][j] = back ? (j > 0 ? xc[j > 0 ? j - 1 : 0] : far) : (j < 3 ? xc[j < 3 ? j + 1 : 3] : far);
    } else {
      const int ca = a == 1 ? c[1] : c[0], na = a == 1 ? q.n[1] : q.n[0];
      const bool end = back ? ca == 0 : ca == na - 1;
      const ptrdiff_t sd = (ptrdiff_t)q.stride[k];
      const float4 f = __ldg(reinterpret_cast<const float4*>(xp + (end ? (wrap ? -(ptrdiff_t)ca * sd : 0) : (back ? -sd : sd))));
      xn[k][0] = f.x, xn[k][1] = f.y, xn[k][2] = f.z, xn[k][3] = f.w;
      if (!wrap && end && q.zero) {
#pragma unroll
        for (int j = 0; j < 4; ++j) xn[k][j] = 0.0f;
      }
    }
  }
  float* __restrict__ op = out + (size_t)blockIdx.y * NB * q.count + e;
#pragma unroll
  for (int k = 0; k < NB; ++k) {
    float v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = back ? ct::fsub(xc[j], xn[k][j]) : ct::fsub(xn[k][j], xc[j]);
    *reinterpret_cast<float4*>(op + (size_t)k * q.count) = make_float4(v[0], v[1], v[2], v[3]);
  }
}

template <int NB, int MODE>
__global__ void __launch_bounds__(kFdT) k_fd_adj_quads(const float* __restrict__ d, float* __restrict__ x, const FdSame q) {
  constexpr bool fwd = MODE == 2, wrap = MODE == 0;
  const uint32_t e = 4 * (blockIdx.x * (uint32_t)kFdT + threadIdx.x);
  if (e >= q.count) return;
  int c[3];
  fd_coords(q, e, c);
  const float* __restrict__ dp = d + (size_t)blockIdx.y * NB * q.count + e;
  float dc[NB][4], dn[NB][4];
#pragma unroll
  for (int k = 0; k < NB; ++k) {
    const float* __restrict__ dk = dp + (size_t)k * q.count;
    const int a = q.axis[k];
    const float4 f = __ldg(reinterpret_cast<const float4*>(dk));
    dc[k][0] = f.x, dc[k][1] = f.y, dc[k][2] = f.z, dc[k][3] = f.w;
    if (a == 2) {
      const bool off = fwd ? c[2] + 4 == q.n[2] : c[2] == 0;
      float far = __ldg(dk + (off ? (wrap ? q.n[2] - 1 : 0) : (fwd ? 4 : -1)));
      if (!wrap && off) far = 0.0f;
#pragma unroll
      for (int j = 0; j < 4; ++j) dn[k][j] = fwd ? (j < 3 ? dc[k][j < 3 ? j + 1 : 3] : far) : (j > 0 ? dc[k][j > 0 ? j - 1 : 0] : far);
    } else {
      const int ca = a == 1 ? c[1] : c[0], na = a == 1 ? q.n[1] : q.n[0];
      const bool off = fwd ? ca == na - 1 : ca == 0;
      const ptrdiff_t sd = (ptrdiff_t)q.stride[k];
      const float4 g = __ldg(reinterpret_cast<const float4*>(dk + (off ? (wrap ? (ptrdiff_t)(na - 1) * sd : 0) : (fwd ? sd : -sd))));
      dn[k][0] = g.x, dn[k][1] = g.y, dn[k][2] = g.z, dn[k][3] = g.w;
      if (!wrap && off) {
#pragma unroll
        for (int j = 0; j < 4; ++j) dn[k][j] = 0.0f;
      }
    }
  }
  float acc[4];
#pragma unroll
  for (int k = 0; k < NB; ++k) {
    float v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = fwd ? ct::fsub(dc[k][j], dn[k][j]) : ct::fsub(dn[k][j], dc[k][j]);
    if (!wrap && !q.zero) {  // a copied end: position 0 first, or then the position past the end (d[n-1] - 0)
      const int a = q.axis[k];
      const int ca = a == 2 ? (fwd ? c[2] : c[2] + 3) : (a == 1 ? c[1] : c[0]);
      const int na = a == 2 ? q.n[2] : (a == 1 ? q.n[1] : q.n[0]);
      if (fwd ? ca == 0 : ca == na - 1) {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (a != 2 || j == (fwd ? 0 : 3))
            v[j] = fwd ? ct::fadd(ct::fsub(0.0f, dc[k][j]), v[j]) : ct::fadd(v[j], dc[k][j]);
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[j] = k == 0 ? v[j] : ct::fadd(acc[j], v[j]);
  }
  *reinterpret_cast<float4*>(x + (size_t)blockIdx.y * q.count + e) = make_float4(acc[0], acc[1], acc[2], acc[3]);
}

// Launch of the same-shape kernels.
template <bool ADJ, int NB, int U>
void fd_rows_launch(const float* src, float* dst, const FdSame& q, dim3 g, cudaStream_t s) {
  if (q.mode == 0)
    k_fd_rows<NB, U, 0, ADJ><<<g, kFdT, 0, s>>>(src, dst, q);
  else if (q.mode == 1)
    k_fd_rows<NB, U, 1, ADJ><<<g, kFdT, 0, s>>>(src, dst, q);
  else
    k_fd_rows<NB, U, 2, ADJ><<<g, kFdT, 0, s>>>(src, dst, q);
}

template <bool ADJ, int NB>
ct_status fd_same_launch(const float* src, float* dst, const FdSame& q, int batch, cudaStream_t s) {
  if (q.n[2] % 4 == 0 && ct::aligned(src, 16) && ct::aligned(dst, 16)) {
    const dim3 g((q.count / 4 + kFdT - 1) / kFdT, batch);
    if constexpr (ADJ) {
      auto f = q.mode == 0 ? k_fd_adj_quads<NB, 0> : (q.mode == 1 ? k_fd_adj_quads<NB, 1> : k_fd_adj_quads<NB, 2>);
      f<<<g, kFdT, 0, s>>>(src, dst, q);
    } else {
      auto f = q.mode == 0 ? k_fd_fwd_quads<NB, 0> : (q.mode == 1 ? k_fd_fwd_quads<NB, 1> : k_fd_fwd_quads<NB, 2>);
      f<<<g, kFdT, 0, s>>>(src, dst, q);
    }
    return ct::launch_check("k_fd_quads");
  }
  if (q.n[2] >= 32) {
    const dim3 g((q.units + kFdT / 32 - 1) / (kFdT / 32), batch);
    switch (q.per_lane) {
      case 1: fd_rows_launch<ADJ, NB, 1>(src, dst, q, g, s); break;
      case 2: fd_rows_launch<ADJ, NB, 2>(src, dst, q, g, s); break;
      case 3: fd_rows_launch<ADJ, NB, 3>(src, dst, q, g, s); break;
      default: fd_rows_launch<ADJ, NB, 4>(src, dst, q, g, s); break;
    }
    return ct::launch_check("k_fd_rows");
  }
  const int u = one_each(q.count) ? 1 : kFdU;
  const dim3 g((q.count + kFdT * u - 1) / (kFdT * u), batch);
  if constexpr (ADJ) {
    auto f = u == 1 ? k_fd_adj_flat<NB, 1> : k_fd_adj_flat<NB, kFdU>;
    f<<<g, kFdT, 0, s>>>(src, dst, q);
  } else {
    auto f = u == 1 ? k_fd_fwd_flat<NB, 1> : k_fd_fwd_flat<NB, kFdU>;
    f<<<g, kFdT, 0, s>>>(src, dst, q);
  }
  return ct::launch_check(ADJ ? "k_fd_adj_flat" : "k_fd_fwd_flat");
}

// Value of the extended line e (prepend/append applied) at position t.
__device__ __forceinline__ float fd_ext(const float* __restrict__ x, size_t stride, int n, int P,
                                        int prepend, int append, int t) {
  if (t < P) return prepend == 0 ? __ldg(x) : 0.0f;
  const int s = t - P;
  if (s < n) return __ldg(x + (size_t)s * stride);
  return append == 0 ? __ldg(x + (size_t)(n - 1) * stride) : 0.0f;
}

__global__ void k_fd_fwd(const float* __restrict__ x, float* __restrict__ out, FdParams p,
                         int batch) {
  const size_t total = p.out_count * batch;
  for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < total;
       e += (size_t)gridDim.x * blockDim.x) {
    const size_t bi = e / p.out_count;
    size_t r = e - bi * p.out_count;
    int k = 0;
    while (k + 1 < p.nblocks && r >= p.blk[k + 1].off) ++k;
    r -= p.blk[k].off;
    const FdBlock& B = p.blk[k];
    int dims[3] = {p.n[0], p.n[1], p.n[2]};
    dims[B.axis] = B.M;
    const int c2 = (int)(r % dims[2]);
    const size_t r1 = r / dims[2];
    const int c1 = (int)(r1 % dims[1]);
    const int c0 = (int)(r1 / dims[1]);
    int c[3] = {c0, c1, c2};
    const int m = c[B.axis];
    const int n = p.n[B.axis];
    size_t stride = 1;
    for (int q = 2; q > B.axis; --q) stride *= p.n[q];
    c[B.axis] = 0;
    const float* line = x + bi * p.in_count + ((size_t)c[0] * p.n[1] + c[1]) * p.n[2] + c[2];
    float v;
    if (p.circular) {
      const int m1 = (m + 1 == n) ? 0 : m + 1;
      v = ct::fsub(__ldg(line + (size_t)m1 * stride), __ldg(line + (size_t)m * stride));
    } else {
      const int P = p.prepend >= 0 ? 1 : 0;
      v = ct::fsub(fd_ext(line, stride, n, P, p.prepend, p.append, m + 1),
                   fd_ext(line, stride, n, P, p.prepend, p.append, m));
    }
    out[e] = v;
  }
}

// Adjoint, as jax.linear_transpose builds it from the forward's jnp.diff:
// extended-line position q gets the cotangent ce[q] = d[q-1] - d[q] (a term
// outside 0..M-1 is 0), and x[t] = sum over blocks (axis order) of the sum,
// in position order, of ce[q] over the run [qa, qb] of positions holding
// x[t] -- one position inside the line, two at an end copied by prepend=0 /
// append=0 (the float32 sum (d[0] - d[1]) - d[0] is not -d[1] in general).
__global__ void k_fd_adj(const float* __restrict__ d, float* __restrict__ x, FdParams p,
                         int batch) {
  const size_t total = p.in_count * batch;
  const int P = p.prepend >= 0 ? 1 : 0;
  for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < total;
       e += (size_t)gridDim.x * blockDim.x) {
    const size_t bi = e / p.in_count;
    const size_t r = e - bi * p.in_count;
    const int c2 = (int)(r % p.n[2]);
    const size_t r1 = r / p.n[2];
    const int c1 = (int)(r1 % p.n[1]);
    const int c0 = (int)(r1 / p.n[1]);
    float acc = 0.0f;
    for (int k = 0; k < p.nblocks; ++k) {
      const FdBlock& B = p.blk[k];
      int c[3] = {c0, c1, c2};
      const int t = c[B.axis];
      const int n = p.n[B.axis];
      int dims[3] = {p.n[0], p.n[1], p.n[2]};
      dims[B.axis] = B.M;
      size_t stride = 1;
      for (int q = 2; q > B.axis; --q) stride *= dims[q];
      c[B.axis] = 0;
      const float* line =
          d + bi * p.out_count + B.off + ((size_t)c[0] * dims[1] + c[1]) * dims[2] + c[2];
      float v;
      if (p.circular) {
        const int tm = (t == 0) ? n - 1 : t - 1;
        v = ct::fsub(__ldg(line + (size_t)tm * stride), __ldg(line + (size_t)t * stride));
      } else {
        const int qa = (p.prepend == 0 && t == 0) ? 0 : t + P;
        const int qb = (p.append == 0 && t == n - 1) ? n + P : t + P;
        auto ce = [&](int q) {
          const float lo = (q - 1 >= 0 && q - 1 < B.M) ? __ldg(line + (size_t)(q - 1) * stride) : 0.0f;
          const float hi = (q >= 0 && q < B.M) ? __ldg(line + (size_t)q * stride) : 0.0f;
          return ct::fsub(lo, hi);
        };
        v = ce(qa);
        for (int q = qa + 1; q <= qb; ++q) v = ct::fadd(v, ce(q));
      }
      acc = (k == 0) ? v : ct::fadd(acc, v);
    }
    x[e] = acc;
  }
}

// Single-level shift-invariant Haar transform over the descriptor's axes
// (HaarTransform / SingleAxisHaarTransform, scico/functional/_tvnorm.py:
// 458-538), output (naxes, 2, *shape) per batch item: for axis k,
// w[k][0] = r (x + x[next]) and w[k][1] = r (x[next] - x), x[next] the
// circularly next sample along the axis, r = float32(1/sqrt 2); every sum and
// product rounded on its own (the reference's separate float32 operations).
__global__ void k_haar_fwd(const float* __restrict__ x, float* __restrict__ w, FdParams p, float r,
                           int batch) {
  const size_t per = 2 * (size_t)p.nblocks * p.in_count;
  const size_t total = per * batch;
  for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < total;
       e += (size_t)gridDim.x * blockDim.x) {
    const size_t bi = e / per;
    size_t rem = e - bi * per;
    const int k = (int)(rem / (2 * p.in_count));
    rem -= (size_t)k * 2 * p.in_count;
    const int comp = (int)(rem / p.in_count);
    const size_t idx = rem - (size_t)comp * p.in_count;
    const int ax = p.blk[k].axis;
    const int c2 = (int)(idx % p.n[2]);
    const size_t r1 = idx / p.n[2];
    const int c[3] = {(int)(r1 / p.n[1]), (int)(r1 % p.n[1]), c2};
    size_t stride = 1;
    for (int q = 2; q > ax; --q) stride *= p.n[q];
    const float* xb = x + bi * p.in_count;
    const float xc = __ldg(xb + idx);
    const size_t in = c[ax] + 1 == p.n[ax] ? idx - (size_t)c[ax] * stride : idx + stride;
    const float xn = __ldg(xb + in);
    w[e] = comp == 0 ? ct::fmul(r, ct::fadd(xc, xn)) : ct::fmul(r, ct::fsub(xn, xc));
  }
}

// Its adjoint: x = sum over axes, in axis order, of
// r (lo + lo[prev]) + r (hi[prev] - hi), [prev] the circularly previous
// sample along the axis.
__global__ void k_haar_adj(const float* __restrict__ w, float* __restrict__ x, FdParams p, float r,
                           int batch) {
  const size_t total = p.in_count * batch;
  const size_t per = 2 * (size_t)p.nblocks * p.in_count;
  for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < total;
       e += (size_t)gridDim.x * blockDim.x) {
    const size_t bi = e / p.in_count;
    const size_t idx = e - bi * p.in_count;
    const int c2 = (int)(idx % p.n[2]);
    const size_t r1 = idx / p.n[2];
    const int c[3] = {(int)(r1 / p.n[1]), (int)(r1 % p.n[1]), c2};
    float acc = 0.0f;
    for (int k = 0; k < p.nblocks; ++k) {
      const int ax = p.blk[k].axis;
      size_t stride = 1;
      for (int q = 2; q > ax; --q) stride *= p.n[q];
      const size_t ip = c[ax] == 0 ? idx + (size_t)(p.n[ax] - 1) * stride : idx - stride;
      const float* lo = w + bi * per + (size_t)k * 2 * p.in_count;
      const float* hi = lo + p.in_count;
      const float t = ct::fadd(ct::fmul(r, ct::fadd(__ldg(lo + idx), __ldg(lo + ip))),
                               ct::fmul(r, ct::fsub(__ldg(hi + ip), __ldg(hi + idx))));
      acc = k == 0 ? t : ct::fadd(acc, t);
    }
    x[e] = acc;
  }
}

int grid_for(size_t n, int threads) {
  const size_t want = (n + threads - 1) / threads;
  const size_t cap = (size_t)ct::sm_count() * 16;
  return (int)std::max<size_t>(1, std::min(want, cap));
}

// Shrink one vector of NC components (values v, component order): L21Norm._prox
// (_norm.py:254-263): len = sqrt(sum_c v_c^2); dir = v/len (0 where len == 0);
// nl = len - lam; nl = 0.5 (nl + |nl|); v = nl * dir.
template <int NC>
__device__ __forceinline__ void l21_shrink(float (&v)[NC], float lam) {
  float ss = ct::fmul(v[0], v[0]);
#pragma unroll
  for (int c = 1; c < NC; ++c) ss = ct::fadd(ss, ct::fmul(v[c], v[c]));
  const float len = __fsqrt_rn(ss);
  float nl = ct::fsub(len, lam);
  nl = ct::fmul(0.5f, ct::fadd(nl, fabsf(nl)));
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    const float dir = (len != 0.0f) ? __fdiv_rn(v[c], len) : 0.0f;
    v[c] = ct::fmul(nl, dir);
  }
}

// The prox of up to three components (every image gradient): the components
// are read once and kept in registers, U vectors in flight per thread: kPxU, or one
// (one_each).  3 x 192^3: 43 -> 27.7 us, the time of a copy; 3 x 64 x 64 x 3 2.5 us
// before, 3.1 with four, 2.1 with one.
constexpr int kPxU = 4;
template <int NC, int U>
__global__ void __launch_bounds__(256) k_l21_prox_few(const float* __restrict__ v, float* __restrict__ out, size_t n,
                                                      float lam) {
  const size_t e0 = (size_t)blockIdx.x * (256 * U) + threadIdx.x;
  float r[U][NC];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const size_t e = min(e0 + u * 256, n - 1);
#pragma unroll
    for (int c = 0; c < NC; ++c) r[u][c] = __ldg(v + (size_t)c * n + e);
  }
#pragma unroll
  for (int u = 0; u < U; ++u)
    if (e0 + u * 256 < n) {
      l21_shrink<NC>(r[u], lam);
#pragma unroll
      for (int c = 0; c < NC; ++c) out[(size_t)c * n + e0 + u * 256] = r[u][c];
    }
}

// The same for any number of components (two passes over them).
__global__ void k_l21_prox(const float* __restrict__ v, float* __restrict__ out, int ncomp,
                           size_t n, float lam) {
  for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < n;
       e += (size_t)gridDim.x * blockDim.x) {
    float ss = 0.0f;
    for (int c = 0; c < ncomp; ++c) {
      const float x = v[(size_t)c * n + e];
      const float sq = ct::fmul(x, x);
      ss = (c == 0) ? sq : ct::fadd(ss, sq);
    }
    const float len = __fsqrt_rn(ss);
    float nl = ct::fsub(len, lam);
    nl = ct::fmul(0.5f, ct::fadd(nl, fabsf(nl)));
    for (int c = 0; c < ncomp; ++c) {
      const float x = v[(size_t)c * n + e];
      const float dir = (len != 0.0f) ? __fdiv_rn(x, len) : 0.0f;
      out[(size_t)c * n + e] = ct::fmul(nl, dir);
    }
  }
}

// L1 prox (L1Norm.prox, _norm.py:110-116): sign(v) * 0.5 (t + |t|), t = |v| - lam.
__device__ __forceinline__ float l1_shrink(float x, float lam) {
  float t = ct::fsub(fabsf(x), lam);
  t = ct::fmul(0.5f, ct::fadd(t, fabsf(t)));
  const float sg = (x > 0.0f) ? 1.0f : ((x < 0.0f) ? -1.0f : (x == 0.0f ? 0.0f : x));
  return ct::fmul(sg, t);
}

__global__ void k_l1_prox(const float* __restrict__ v, float* __restrict__ out, size_t n,
                          float lam) {
  for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < n;
       e += (size_t)gridDim.x * blockDim.x) {
    out[e] = l1_shrink(v[e], lam);
  }
}

// ---------------------------------------------------------------------------
// TV prox in one pass (TVNorm.prox, scico/functional/_tvnorm.py:190-237): the
// shift-invariant Haar transform of v (edge-padded by one sample on every
// differenced axis unless circular), the base norm's prox on its highpass part
// (on the region without the padding), the adjoint transform cropped back,
// times 1/K.  Output e along axis k needs lowpass and shrunk highpass at e and
// at the sample before it, and nothing else, so nothing goes through memory
// but v and the result: a thread evaluates both positions of every axis.  Each
// sum, product, root and quotient is the one that ct_haar_fwd, ct_l21_prox /
// ct_l1_prox and ct_haar_adj round, in their order: same bits.  Bound by the
// divisions and roots (L2,1) or by launch latency at small sizes; the composed
// path took eight launches and passed over 2 naxes arrays: 512^2, L2,1, edge
// padding 40 us of kernels (and 280 us of launches around them) -> 5 us.
// ---------------------------------------------------------------------------
struct TvArgs {
  const float* x;
  float* out;
  FdSame q;      // axes, strides, mode 0 = circular, 1 = edge-padded
  float r, thr, inv_k;
};

template <int NB, bool ISO>
__global__ void __launch_bounds__(256) k_tv_prox(const TvArgs a) {
  const FdSame& q = a.q;
  const uint32_t e = blockIdx.x * 256u + threadIdx.x;
  if (e >= q.count) return;
  const float* __restrict__ x = a.x + (size_t)blockIdx.y * q.count;
  int c[3];
  fd_coords(q, e, c);
  int ca[NB], na[NB];
#pragma unroll
  for (int k = 0; k < NB; ++k) {
    const int ax = q.axis[k];
    ca[k] = ax == 2 ? c[2] : (ax == 1 ? c[1] : c[0]);
    na[k] = ax == 2 ? q.n[2] : (ax == 1 ? q.n[1] : q.n[0]);
  }
  // the sample after position p along axis k, whose coordinate there is t
  auto next = [&](uint32_t p, int k, int t) {
    const uint32_t at = t + 1 < na[k] ? p + q.stride[k] : (q.mode == 0 ? p - (uint32_t)t * q.stride[k] : p);
    return __ldg(x + at);
  };
  const float xe = __ldg(x + e);
  float lo[NB], hi[NB];
#pragma unroll
  for (int k = 0; k < NB; ++k) {
    const float xn = next(e, k, ca[k]);
    lo[k] = ct::fmul(a.r, ct::fadd(xe, xn));
    hi[k] = ct::fmul(a.r, ct::fsub(xn, xe));
  }
  if (ISO) {
    l21_shrink<NB>(hi, a.thr);
  } else {
#pragma unroll
    for (int k = 0; k < NB; ++k) hi[k] = l1_shrink(hi[k], a.thr);
  }
  float acc = 0.0f;
#pragma unroll
  for (int k = 0; k < NB; ++k) {
    // the position before e along axis k: at the line's start the circular
    // wrap, or the padding sample (a copy of the line's end, not shrunk)
    const bool first = ca[k] == 0;
    const uint32_t p = first ? e + (uint32_t)(na[k] - 1) * q.stride[k] : e - q.stride[k];
    const float xp = __ldg(x + p);
    const float lop = ct::fmul(a.r, ct::fadd(xp, xe));
    float hip = ct::fmul(a.r, ct::fsub(xe, xp));
    if (!(first && q.mode != 0)) {
      if (ISO) {
        float v[NB];
#pragma unroll
        for (int j = 0; j < NB; ++j) v[j] = j == k ? hip : ct::fmul(a.r, ct::fsub(next(p, j, ca[j]), xp));
        l21_shrink<NB>(v, a.thr);
        hip = v[k];
      } else {
        hip = l1_shrink(hip, a.thr);
      }
    }
    const float t = ct::fadd(ct::fmul(a.r, ct::fadd(lo[k], lop)), ct::fmul(a.r, ct::fsub(hip, hi[k])));
    acc = k == 0 ? t : ct::fadd(acc, t);
  }
  a.out[(size_t)blockIdx.y * q.count + e] = ct::fmul(a.inv_k, acc);
}

// sum_e sqrt(sum_c v_c^2) (ncomp > 0) or sum_e |v_e| (ncomp == 0), float64.
__global__ void __launch_bounds__(ct::kReduceThreads)
    k_l21_norm(const float* __restrict__ v, int ncomp, size_t n, double* __restrict__ out,
               double* __restrict__ partials, unsigned int* __restrict__ ticket) {
  double acc = 0.0;
  for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < n;
       e += (size_t)gridDim.x * blockDim.x) {
    if (ncomp == 0) {
      acc += fabs((double)v[e]);
    } else {
      float ss = 0.0f;
      for (int c = 0; c < ncomp; ++c) {
        const float x = v[(size_t)c * n + e];
        const float sq = ct::fmul(x, x);
        ss = (c == 0) ? sq : ct::fadd(ss, sq);
      }
      acc += (double)__fsqrt_rn(ss);
    }
  }
  double part[1] = {acc}, tot[1];
  if (ct::grid_reduce_last<ct::kReduceThreads, 1>(part, partials, ticket, tot)) *out = tot[0];
}

}  // namespace

extern "C" {

ct_status ct_fd_out_count(const ct_fd_desc* d, int64_t* count) {
  FdParams p{};
  ct_status st = make_fd(d, p, "ct_fd_out_count");
  if (st != CT_OK) return st;
  if (!count) return ct::fail(CT_ERR_INVALID_ARG, "ct_fd_out_count: null count");
  *count = (int64_t)p.out_count;
  return CT_OK;
}

ct_status ct_fd_fwd(const ct_fd_desc* d, const float* x, float* out, int32_t batch,
                    ct_stream_t stream) {
  FdParams p{};
  ct_status st = make_fd(d, p, "ct_fd_fwd");
  if (st != CT_OK) return st;
  if (!x || !out) return ct::fail(CT_ERR_INVALID_ARG, "ct_fd_fwd: null array");
  if (batch <= 0) return ct::fail(CT_ERR_INVALID_ARG, "ct_fd_fwd: batch=%d", batch);
  const size_t total = p.out_count * batch;
  if (total == 0) return CT_OK;
  FdSame q{};
  if (batch <= 65535 && make_same(p, q)) {
    cudaStream_t s = ct::as_stream(stream);
    if (p.nblocks == 1) return fd_same_launch<false, 1>(x, out, q, batch, s);
    if (p.nblocks == 2) return fd_same_launch<false, 2>(x, out, q, batch, s);
    return fd_same_launch<false, 3>(x, out, q, batch, s);
  }
  k_fd_fwd<<<grid_for(total, 256), 256, 0, ct::as_stream(stream)>>>(x, out, p, batch);
  return ct::launch_check("k_fd_fwd");
}

ct_status ct_fd_adj(const ct_fd_desc* d, const float* dx, float* x, int32_t batch,
                    ct_stream_t stream) {
  FdParams p{};
  ct_status st = make_fd(d, p, "ct_fd_adj");
  if (st != CT_OK) return st;
  if (!x || !dx) return ct::fail(CT_ERR_INVALID_ARG, "ct_fd_adj: null array");
  if (batch <= 0) return ct::fail(CT_ERR_INVALID_ARG, "ct_fd_adj: batch=%d", batch);
  const size_t total = p.in_count * batch;
  FdSame q{};
  if (batch <= 65535 && make_same(p, q)) {
    cudaStream_t s = ct::as_stream(stream);
    if (p.nblocks == 1) return fd_same_launch<true, 1>(dx, x, q, batch, s);
    if (p.nblocks == 2) return fd_same_launch<true, 2>(dx, x, q, batch, s);
    return fd_same_launch<true, 3>(dx, x, q, batch, s);
  }
  k_fd_adj<<<grid_for(total, 256), 256, 0, ct::as_stream(stream)>>>(dx, x, p, batch);
  return ct::launch_check("k_fd_adj");
}

ct_status ct_haar_fwd(const ct_fd_desc* d, const float* x, float* w, int32_t batch, ct_stream_t stream) {
  FdParams p{};
  ct_status st = make_fd(d, p, "ct_haar_fwd");
  if (st != CT_OK) return st;
  if (!x || !w) return ct::fail(CT_ERR_INVALID_ARG, "ct_haar_fwd: null array");
  if (batch <= 0) return ct::fail(CT_ERR_INVALID_ARG, "ct_haar_fwd: batch=%d", batch);
  const size_t total = 2 * (size_t)p.nblocks * p.in_count * batch;
  k_haar_fwd<<<grid_for(total, 256), 256, 0, ct::as_stream(stream)>>>(x, w, p, (float)(1.0 / sqrt(2.0)), batch);
  return ct::launch_check("k_haar_fwd");
}

ct_status ct_haar_adj(const ct_fd_desc* d, const float* w, float* x, int32_t batch, ct_stream_t stream) {
  FdParams p{};
  ct_status st = make_fd(d, p, "ct_haar_adj");
  if (st != CT_OK) return st;
  if (!x || !w) return ct::fail(CT_ERR_INVALID_ARG, "ct_haar_adj: null array");
  if (batch <= 0) return ct::fail(CT_ERR_INVALID_ARG, "ct_haar_adj: batch=%d", batch);
  const size_t total = p.in_count * batch;
  k_haar_adj<<<grid_for(total, 256), 256, 0, ct::as_stream(stream)>>>(w, x, p, (float)(1.0 / sqrt(2.0)), batch);
  return ct::launch_check("k_haar_adj");
}

ct_status ct_tv_prox(const ct_fd_desc* d, const float* v, float* out, int32_t iso, float thr, int32_t batch,
                     ct_stream_t stream) {
  FdParams p{};
  ct_status st = make_fd(d, p, "ct_tv_prox");
  if (st != CT_OK) return st;
  if (!v || !out) return ct::fail(CT_ERR_INVALID_ARG, "ct_tv_prox: null array");
  if (batch <= 0) return ct::fail(CT_ERR_INVALID_ARG, "ct_tv_prox: batch=%d", batch);
  if (!p.circular && (p.append != 0 || p.prepend >= 0))
    return ct::fail(CT_ERR_INVALID_ARG, "ct_tv_prox: the differences are circular or have append = 0");
  TvArgs a{};
  if (batch > 65535 || !make_same(p, a.q))
    return ct::fail(CT_ERR_UNSUPPORTED, "ct_tv_prox: batch above 65535 or an array of 2^31 elements or more");
  a.x = v;
  a.out = out;
  a.r = (float)(1.0 / sqrt(2.0));
  a.thr = thr;
  a.inv_k = (float)(1.0 / (2.0 * p.nblocks));
  const dim3 g((a.q.count + 255) / 256, batch);
  cudaStream_t s = ct::as_stream(stream);
  switch (2 * p.nblocks + (iso ? 1 : 0)) {
    case 2: k_tv_prox<1, false><<<g, 256, 0, s>>>(a); break;
    case 3: k_tv_prox<1, true><<<g, 256, 0, s>>>(a); break;
    case 4: k_tv_prox<2, false><<<g, 256, 0, s>>>(a); break;
    case 5: k_tv_prox<2, true><<<g, 256, 0, s>>>(a); break;
    case 6: k_tv_prox<3, false><<<g, 256, 0, s>>>(a); break;
    default: k_tv_prox<3, true><<<g, 256, 0, s>>>(a); break;
  }
  return ct::launch_check("k_tv_prox");
}

ct_status ct_l21_prox(const float* v, float* out, int32_t ncomp, int64_t n, float lam,
                      ct_stream_t stream) {
  if (!v || !out) return ct::fail(CT_ERR_INVALID_ARG, "ct_l21_prox: null array");
  if (ncomp < 1 || n < 0)
    return ct::fail(CT_ERR_INVALID_ARG, "ct_l21_prox: ncomp=%d n=%lld", ncomp, (long long)n);
  if (n == 0) return CT_OK;
  const int u = one_each((size_t)n) ? 1 : kPxU;
  const size_t blocks = ((size_t)n + 256 * u - 1) / (256 * u);
  if (ncomp <= 3 && blocks < (1ull << 31)) {
    auto launch = [&](auto one, auto four) {
      (u == 1 ? one : four)<<<(unsigned)blocks, 256, 0, ct::as_stream(stream)>>>(v, out, (size_t)n, lam);
    };
    if (ncomp == 1)
      launch(k_l21_prox_few<1, 1>, k_l21_prox_few<1, kPxU>);
    else if (ncomp == 2)
      launch(k_l21_prox_few<2, 1>, k_l21_prox_few<2, kPxU>);
    else
      launch(k_l21_prox_few<3, 1>, k_l21_prox_few<3, kPxU>);
    return ct::launch_check("k_l21_prox_few");
  }
  k_l21_prox<<<grid_for((size_t)n, 256), 256, 0, ct::as_stream(stream)>>>(v, out, ncomp,
                                                                           (size_t)n, lam);
  return ct::launch_check("k_l21_prox");
}

ct_status ct_l1_prox(const float* v, float* out, int64_t n, float lam, ct_stream_t stream) {
  if (!v || !out) return ct::fail(CT_ERR_INVALID_ARG, "ct_l1_prox: null array");
  if (n < 0) return ct::fail(CT_ERR_INVALID_ARG, "ct_l1_prox: n=%lld", (long long)n);
  if (n == 0) return CT_OK;
  k_l1_prox<<<grid_for((size_t)n, 256), 256, 0, ct::as_stream(stream)>>>(v, out, (size_t)n, lam);
  return ct::launch_check("k_l1_prox");
}

ct_status ct_l21_norm(const float* v, int32_t ncomp, int64_t n, double* out_dev, void* workspace,
                      size_t workspace_bytes, ct_stream_t stream) {
  if (!v || !out_dev) return ct::fail(CT_ERR_INVALID_ARG, "ct_l21_norm: null pointer");
  if (ncomp < 0 || n < 0)
    return ct::fail(CT_ERR_INVALID_ARG, "ct_l21_norm: ncomp=%d n=%lld", ncomp, (long long)n);
  if (!workspace || workspace_bytes < ct::kReduceWorkspace || !ct::aligned(workspace, 256))
    return ct::fail(CT_ERR_WORKSPACE, "ct_l21_norm: need %zu bytes", ct::kReduceWorkspace);
  unsigned int* ticket = static_cast<unsigned int*>(workspace);
  double* partials = reinterpret_cast<double*>(static_cast<char*>(workspace) + 256);
  k_l21_norm<<<ct::kReduceBlocks, ct::kReduceThreads, 0, ct::as_stream(stream)>>>(
      v, ncomp, (size_t)n, out_dev, partials, ticket);
  return ct::launch_check("k_l21_norm");
}

}  // extern "C"
