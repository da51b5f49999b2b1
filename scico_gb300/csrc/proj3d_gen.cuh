// GENERAL 3D projector kernels (any matrices), included by proj3d.cu.
//
// Forward.  A view marches along the axis a on which its ray direction is
// largest; (p, q) are the other two axes.  Voxels are taken in sheared windows
// of kWin x kWin voxels of the (p, q) plane: plane ia shifts every window by
// s(ia) = round(d ia), d the ray's slope in voxels per plane, so that the
// footprints of a window's voxels stay inside one small detector tile over the
// whole depth, and each voxel lies in exactly one window.  One warp owns a
// window (or a segment of its planes) and its tile, in shared memory, so no
// two warps ever add to the same number and nothing is atomic:
//  * a voxel whose footprint starts at detector pixel (u0, u1) adds its four
//    products to the float4 of slot (u0, u1), by one 16-byte load and store;
//  * the 32 lanes take an 8 x 4 lattice of the plane's voxels, two apart, and a
//    second one beside it: 64 voxels on 64 different slots, so both loads go
//    out before the first store (checked per view from the matrix; views where
//    it does not hold take the step in two or four phases of lanes that are
//    further apart);
//  * axis 2 as the marching axis would read the volume across its rows: those
//    views read a copy with that axis outermost.
//  * the row stride of the slots is the one of eight that spreads eight
//    neighbouring lanes best over the eight 16-byte bank groups.
// The tile's pixels (the sum of up to four slots' parts) go to a scratch, and
// k_p3_gen_gather adds, per detector pixel, the windows that cover it, in
// window order.  The products and weights are the reference's float32
// expressions; only the order of the sums differs from a detector-driven
// march.  The march (k_p3_gen_march: each pixel searches, plane by plane, the
// voxels that can reach it: two divisions and some twenty tests for each four
// hits) stays for views outside the tile's bounds (voxels above ~1.2 detector
// pixels or below 1/4) and for callers without scratch.
// Bound by the shared-memory and load pipe (9 cycles of 16-byte accesses and 4
// of loads a step of 32 voxels).  97 x 128 x 111 voxels, 60 tilted views on
// 128 x 181: the march 2754 us, this 295 us.
#pragma once

namespace ct {
namespace {

constexpr int kWin = 16;         // window edge (voxels)
constexpr int kSlots = 640;      // float4 slots of a warp's tile: 24 x 24 for voxels of one pixel at any angle
constexpr int kTilePix = 704;    // pixels of a tile in the scratch
constexpr float kTileSlack = 0.0625f;  // rounding of positions and shifts, in pixels
constexpr int kGenWarps = 4;     // five CTAs of 41 KB tiles an SM
constexpr int kGatherWarps = 8;

__device__ __forceinline__ unsigned long long g_pk(float lo, float hi) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void g_upk(unsigned long long v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
// Paired float32 operations, each half rounded as the scalar one.
__device__ __forceinline__ unsigned long long g_add(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ unsigned long long g_sub(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ unsigned long long g_add_down(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("add.rm.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ unsigned long long g_add_up(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("add.rp.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ unsigned long long g_mul(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ unsigned long long g_fma(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

// 1.5 2^23: adding it rounds to an integer, whose value is the sum's low bits.
constexpr float kGMagic = 12582912.0f;
constexpr int kGMagicBits = 0x4B400000;

// Footprint of a voxel from its rounded position pair px = (Px_0, Px_1): the
// first detector pixel as magic bits and the four weights (t0 t1, t0 s1, s0 t1,
// s0 s1) times 4, as in edge3 with s = 0.5 - t: floor and ceil are a rounding
// down and up of left + 1.5 2^23 (|left| < 2^22).
struct Foot {
  int u0, u1;  // kGMagicBits + floor(left)
  unsigned long long w0, w1;  // (w00, w01), (w10, w11)
};
// The first pixel's bits and ceil(left) - left of both axes.
__device__ __forceinline__ void foot_edges(unsigned long long px, int& u0, int& u1, float& t0, float& t1) {
  const unsigned long long magic = g_pk(kGMagic, kGMagic);
  const unsigned long long left = g_sub(px, g_pk(0.25f, 0.25f));
  const unsigned long long fl = g_add_down(left, magic);
  const unsigned long long up = g_sub(g_add_up(left, magic), magic);
  float f0, f1;
  g_upk(g_sub(up, left), t0, t1);
  g_upk(fl, f0, f1);
  u0 = __float_as_int(f0);
  u1 = __float_as_int(f1);
}
__device__ __forceinline__ Foot footprint(unsigned long long px) {
  Foot f;
  float t0, t1;
  foot_edges(px, f.u0, f.u1, t0, t1);
  t0 = fminf(t0, 0.5f);
  t1 = fminf(t1, 0.5f);
  const float s0 = fsub(0.5f, t0), s1 = fsub(0.5f, t1);
  // (a b) 4 = a (4 b) exactly
  const unsigned long long q1 = g_pk(fmul(4.0f, t1), fmul(4.0f, s1));
  f.w0 = g_mul(g_pk(t0, t0), q1);
  f.w1 = g_mul(g_pk(s0, s0), q1);
  return f;
}

// One view's windows and tiles (the same numbers in every kernel: products and
// sums are rounded one by one, not contracted).
struct GenView {
  int ok;            // the window kernels take this view
  int phases;        // lanes of a step share no slot within a phase (1, 2 or 4)
  int ax;            // marching axis
  int na, np, nq;    // extents along a, p, q
  float ma0, ma1, mp0, mp1, mq0, mq1, c0, c1;  // matrix columns by role, translation
  float dp, dq;      // window shift per plane
  int I0, nI, J0, nJ;  // window index ranges
  int T0, T1, LD;    // slots of a tile: rows, columns, row stride
  float b0, b1;      // tile origin of window (0, 0) before rounding
  float i00, i01, i10, i11;  // (1 / kWin) inverse of the (p, q) columns
};

__host__ __device__ __forceinline__ float gen_div(float a, float b) {
#ifdef __CUDA_ARCH__
  return __fdiv_rn(a, b);
#else
  return a / b;
#endif
}

__host__ __device__ __forceinline__ int gen_shift(float d, int ia) {
  return (int)floorf(fadd(fmul(d, (float)ia), 0.5f));
}

__device__ __forceinline__ void gen_tile_base(const GenView& g, int I, int J, int& b0, int& b1) {
  const float x = (float)(kWin * I), y = (float)(kWin * J);
  b0 = (int)floorf(fadd(g.b0, fadd(fmul(g.mp0, x), fmul(g.mq0, y))));
  b1 = (int)floorf(fadd(g.b1, fadd(fmul(g.mp1, x), fmul(g.mq1, y))));
}

// Everything of a view's plan but phases and LD; returns the tests of `ok` that
// concern the view as a whole.
__host__ __device__ inline bool gen_view_base(GenView& g, const float* m, int n0, int n1, int n2, int nwin) {
  auto pick = [&](int k) { return k == 0 ? n0 : (k == 1 ? n1 : n2); };
  auto least = [](int a, int b) { return a < b ? a : b; };
  auto most = [](int a, int b) { return a > b ? a : b; };
  g.ax = (int)m[8];
  const int p = g.ax == 0 ? 1 : 0, q = g.ax == 2 ? 1 : 2;
  g.na = pick(g.ax);
  g.np = pick(p);
  g.nq = pick(q);
  g.ma0 = m[g.ax];
  g.ma1 = m[4 + g.ax];
  g.mp0 = m[p];
  g.mp1 = m[4 + p];
  g.mq0 = m[q];
  g.mq1 = m[4 + q];
  g.c0 = m[3];
  g.c1 = m[7];
  const float det = fsub(fmul(g.mp0, g.mq1), fmul(g.mq0, g.mp1));
  g.dp = -gen_div(fsub(fmul(g.mq1, g.ma0), fmul(g.mq0, g.ma1)), det);
  g.dq = -gen_div(fsub(fmul(g.mp0, g.ma1), fmul(g.mp1, g.ma0)), det);
  const float w = 1.0f / kWin;
  g.i00 = gen_div(fmul(w, g.mq1), det);
  g.i01 = -gen_div(fmul(w, g.mq0), det);
  g.i10 = -gen_div(fmul(w, g.mp1), det);
  g.i11 = gen_div(fmul(w, g.mp0), det);
  // coordinates small enough for the slack, a sane shear
  const float r0 = fabsf(g.ma0) * g.na + fabsf(g.mp0) * g.np + fabsf(g.mq0) * g.nq + fabsf(g.c0);
  const float r1 = fabsf(g.ma1) * g.na + fabsf(g.mp1) * g.np + fabsf(g.mq1) * g.nq + fabsf(g.c1);
  bool ok = r0 < 32768.0f && r1 < 32768.0f && fabsf(g.dp) < 1.01f && fabsf(g.dq) < 1.01f;
  // the gather's window index of a pixel, off by less than its margin of 0.01:
  // the terms that cancel in it, each good to a few units of rounding
  // (nearly parallel matrix rows make them many times the index)
  const float P = (float)g.np + (float)g.na, Q = (float)g.nq + (float)g.na;
  const float y0 = fabsf(g.mp0) * P + fabsf(g.mq0) * Q, y1 = fabsf(g.mp1) * P + fabsf(g.mq1) * Q;
  ok = ok && 0x1p-20f * (fabsf(g.i00) * y0 + fabsf(g.i01) * y1) <= 0.01f &&
       0x1p-20f * (fabsf(g.i10) * y0 + fabsf(g.i11) * y1) <= 0.01f;
  // shift range over the planes, window ranges
  const int ep = ok ? gen_shift(g.dp, g.na - 1) : 0, eq = ok ? gen_shift(g.dq, g.na - 1) : 0;
  auto fdiv = [](int a) { return a >= 0 ? a / kWin : -((-a + kWin - 1) / kWin); };
  g.I0 = fdiv(-most(0, ep));
  g.nI = fdiv(g.np - 1 - least(0, ep)) - g.I0 + 1;
  g.J0 = fdiv(-most(0, eq));
  g.nJ = fdiv(g.nq - 1 - least(0, eq)) - g.J0 + 1;
  ok = ok && (long long)g.nI * g.nJ <= nwin;
  // footprint of a window: its voxels' left positions span
  // [min, max] of kWin (mp x + mq y), x, y in [0, 1] (half a voxel of shift
  // rounding on either side included)
  const float fw = (float)kWin;
  const float e0 = fadd(fmul(fw, fabsf(g.mp0)), fmul(fw, fabsf(g.mq0)));
  const float e1 = fadd(fmul(fw, fabsf(g.mp1)), fmul(fw, fabsf(g.mq1)));
  ok = ok && e0 < 512.0f && e1 < 512.0f;
  g.T0 = ok ? (int)ceilf(fadd(e0, 2.0f * kTileSlack)) + 1 : 1;
  g.T1 = ok ? (int)ceilf(fadd(e1, 2.0f * kTileSlack)) + 1 : 1;
  ok = ok && g.T0 * g.T1 <= kSlots && (g.T0 + 1) * (g.T1 + 1) <= kTilePix;
  const float l0 = fadd(fmul(fw, fminf(g.mp0, 0.0f)), fmul(fw, fminf(g.mq0, 0.0f)));
  const float l1 = fadd(fmul(fw, fminf(g.mp1, 0.0f)), fmul(fw, fminf(g.mq1, 0.0f)));
  g.b0 = fadd(fadd(fadd(g.c0, fmul(0.5f, g.ma0)), -0.25f - kTileSlack), l0);
  g.b1 = fadd(fadd(fadd(g.c1, fmul(0.5f, g.ma1)), -0.25f - kTileSlack), l1);
  return ok;
}

// Plane ia's shift keeps its voxels inside the tile: the windows' footprint moves
// by at most half a voxel either way, as e0 and e1 allow, and a quarter of the
// slack.  The shears are quotients of differences, which nearly parallel matrix rows
// leave few digits of; over the planes that adds up to whole pixels.
__host__ __device__ inline bool gen_plane_fits(const GenView& g, int ia) {
  const float sp = (float)gen_shift(g.dp, ia), sq = (float)gen_shift(g.dq, ia), xa = (float)ia;
  const float d0 = fadd(fmul(g.ma0, xa), fadd(fmul(g.mp0, sp), fmul(g.mq0, sq)));
  const float d1 = fadd(fmul(g.ma1, xa), fadd(fmul(g.mp1, sp), fmul(g.mq1, sq)));
  return fabsf(d0) <= fadd(fmul(0.5f, fadd(fabsf(g.mp0), fabsf(g.mq0))), 0.25f * kTileSlack) &&
         fabsf(d1) <= fadd(fmul(0.5f, fadd(fabsf(g.mp1), fabsf(g.mq1))), 0.25f * kTileSlack);
}

// The voxels of a step sit 2 apart: displacements (2 di, 2 dj), half plane, number k
// of kLattice; two share a slot only where both components stay below one pixel.
// Returns 0 where they cannot, else 1, + 2 where di + dj is even, + 4 where both are.
constexpr int kLattice = 15 * 8;
__host__ __device__ inline int gen_lattice(const GenView& g, int k) {
  const int dj = k / 15, di = k % 15 - 7;
  if (dj == 0 && di <= 0) return 0;
  const float x = 2.0f * di, y = 2.0f * dj;
  const float d0 = fabsf(fadd(fmul(g.mp0, x), fmul(g.mq0, y))), d1 = fabsf(fadd(fmul(g.mp1, x), fmul(g.mq1, y)));
  if (fmaxf(d0, d1) >= 1.0f + 2.0f * kTileSlack) return 0;
  return 1 + (((di + dj) & 1) == 0 ? 2 : 0) + ((di & 1) == 0 && (dj & 1) == 0 ? 4 : 0);
}

// By all 32 lanes of one warp; valid in every lane.
__device__ GenView gen_view(const float* __restrict__ m, int n0, int n1, int n2, int nwin, bool turned) {
  const int lane = threadIdx.x & 31;
  GenView g;
  bool ok = gen_view_base(g, m, n0, n1, n2, nwin) && (turned || g.ax != 2);
  if (ok) {  // the same in every lane
    bool fits = true;
    for (int ia = lane; ia < g.na; ia += 32) fits = fits && gen_plane_fits(g, ia);
    ok = __all_sync(0xffffffffu, fits);
  }
  int shared = 0;
  for (int k = lane; k < kLattice; k += 32) shared |= gen_lattice(g, k);
  shared = __reduce_or_sync(0xffffffffu, shared);
  g.phases = !(shared & 1) ? 1 : (!(shared & 2) ? 2 : 4);
  ok = ok && !(shared & 4);
  // row stride: lane = (candidate, starting phase); the bank groups that eight
  // lanes in a row along q meet
  const int cand = lane & 7;
  int cost = 0;
  {
    const int ld = g.T1 + cand;
    const float f = 0.25f * (float)(lane >> 3);
    unsigned lo = 0, most = 0;  // 4-bit counters of the 8 bank groups
    for (int i = 0; i < 8; ++i) {
      const int r = (int)floorf(2.0f * i * g.mq0 + f), c = (int)floorf(2.0f * i * g.mq1 + f);
      const unsigned b = (unsigned)(r * ld + c) & 7u;
      lo += 1u << (4 * b);
      most = max(most, (lo >> (4 * b)) & 15u);
    }
    cost = (int)most;
  }
  cost += __shfl_xor_sync(0xffffffffu, cost, 8);
  cost += __shfl_xor_sync(0xffffffffu, cost, 16);
  cost = (g.T0 * (g.T1 + cand) <= kSlots ? cost : 1000) * 8 + cand;
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) cost = min(cost, __shfl_xor_sync(0xffffffffu, cost, o));
  g.LD = g.T1 + (cost & 7);
  g.ok = ok ? 1 : 0;
  return g;
}

// gen_view's `ok` on the host (the table as ct_proj3d_views wrote it).
inline bool gen_view_fits(const float* m, int n0, int n1, int n2, int nwin) {
  GenView g;
  if (!gen_view_base(g, m, n0, n1, n2, nwin)) return false;
  for (int ia = 0; ia < g.na; ++ia)
    if (!gen_plane_fits(g, ia)) return false;
  for (int k = 0; k < kLattice; ++k)
    if (gen_lattice(g, k) & 4) return false;
  return true;
}

struct GenFwdArgs {
  const float* vol;
  const float* vol_t;     // [axis 2][axis 0][axis 1]
  const GenView* plan;    // per view
  float* part;            // [view of the launch][segment][window][kTilePix]
  float* proj;
  int n0, n1, n2, R, C;
  int v0;          // first view of the launch
  int nwin, nseg;  // windows of a view (bound), segments of the planes
  const double* skip;
};

// What a forward needs before its windows: the views' plans (the first
// ceil(V / 8) blocks, a warp per view) and, where a view marches along axis 2, the
// volume with that axis outermost, out[k][r] = in[r][k] (rows = n0 n1), a 32 x 32
// piece per further block.  out null: no copy, and no windows for those views.
__global__ void __launch_bounds__(256) k_p3_gen_setup(const float* __restrict__ views, GenView* __restrict__ plan,
                                                      const float* __restrict__ in, float* __restrict__ out, int n0,
                                                      int n1, int n2, int V, int nwin, const double* skip) {
  if (skip && *skip != 0.0) return;
  const unsigned plan_blocks = (V + 7) / 8;
  if (blockIdx.x < plan_blocks) {
    const int v = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (v >= V) return;
    const GenView g = gen_view(views + (size_t)v * kVT, n0, n1, n2, nwin, out != nullptr);
    if ((threadIdx.x & 31) == 0) plan[v] = g;
    return;
  }
  int along = 0;
  for (int v = threadIdx.x; v < V; v += 256) along |= views[(size_t)v * kVT + 8] == 2.0f;
  if (!__syncthreads_or(along)) return;
  __shared__ float t[32][33];
  const int rows = n0 * n1;
  const unsigned piece = blockIdx.x - plan_blocks, nk = (n2 + 31) / 32, br = piece / nk, bk = piece - br * nk;
  const int lx = threadIdx.x & 31, ly = threadIdx.x >> 5;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int r = br * 32 + ly + 8 * q, k = bk * 32 + lx;
    if (r < rows && k < n2) t[ly + 8 * q][lx] = __ldg(in + (size_t)r * n2 + k);
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int k = bk * 32 + ly + 8 * q, r = br * 32 + lx;
    if (r < rows && k < n2) out[(size_t)k * rows + r] = t[lx][ly + 8 * q];
  }
}

__device__ __forceinline__ void lds_pairs(uint32_t a, unsigned long long& x, unsigned long long& y) {
  asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(x), "=l"(y) : "r"(a) : "memory");
}
__device__ __forceinline__ void sts_pairs(uint32_t a, unsigned long long x, unsigned long long y) {
  asm volatile("st.shared.v2.b64 [%0], {%1, %2};" ::"r"(a), "l"(x), "l"(y) : "memory");
}

// The planes [zb, ze) of window (I, J) into the warp's tile at shared address
// `tile`.  LAST: the marching axis is axis 2, whose product is added last
// (((m0 x0 + m1 x1) + m2 x2) + m3).  Voxels of a row (axis q) are contiguous.
template <bool LAST>
__device__ __forceinline__ void gen_window(const GenFwdArgs& a, const GenView& g, int I, int J, int zb, int ze,
                                           int base0, int base1, uint32_t tile) {
  const int lane = threadIdx.x & 31, li = lane & 7, lj = lane >> 3;
  const ptrdiff_t sa = LAST ? (ptrdiff_t)a.n0 * a.n1 : (g.ax == 0 ? (ptrdiff_t)a.n1 * a.n2 : a.n2);
  const ptrdiff_t sp = LAST ? a.n1 : (g.ax == 0 ? a.n2 : (ptrdiff_t)a.n1 * a.n2);
  const float* __restrict__ vol = LAST ? a.vol_t : a.vol;
  const unsigned long long cc = g_pk(g.c0, g.c1);
  const uint32_t ld16 = 16u * (uint32_t)g.LD;
  const uint32_t origin = tile - ld16 * (uint32_t)(kGMagicBits + base0) - 16u * (uint32_t)(kGMagicBits + base1);
  const int colour = g.phases == 1 ? 0 : (g.phases == 2 ? (li + lj) & 1 : (li & 1) | ((lj & 1) << 1));
  // the lane's eight voxels of a plane: x[4 f + 2 e + h] at (p, q) =
  // (p0 + 2 lj + e + 8 h, q0 + 2 li + f): eight lanes along a row, so that a
  // load meets four rows
  auto load = [&](int ia, float (&x)[8], int& p0, int& q0) {
    p0 = gen_shift(g.dp, ia) + kWin * I;
    q0 = gen_shift(g.dq, ia) + kWin * J;
    if (p0 >= g.np || p0 + kWin <= 0 || q0 >= g.nq || q0 + kWin <= 0) return false;  // warp-uniform
    const int p = p0 + 2 * lj, q = q0 + 2 * li;
    const float* __restrict__ v = vol + ia * sa + p * sp + q;
    const bool inside = p0 >= 0 && p0 + kWin <= g.np && q0 >= 0 && q0 + kWin <= g.nq;  // warp-uniform
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int dp = (k >> 1) + 8 * (k & 1);
      const float* __restrict__ row = v + dp * sp;
      if (inside) {
        x[k] = __ldg(row);
        x[4 + k] = __ldg(row + 1);
      } else {
        const bool in = (unsigned)(p + dp) < (unsigned)g.np;
        x[k] = in && (unsigned)q < (unsigned)g.nq ? __ldg(row) : 0.0f;
        x[4 + k] = in && (unsigned)(q + 1) < (unsigned)g.nq ? __ldg(row + 1) : 0.0f;
      }
    }
    return true;
  };
  float xc[8], xn[8];
  int p0 = 0, q0 = 0, pn = 0, qn = 0;
  bool cur = load(zb, xc, p0, q0);
  for (int ia = zb; ia < ze; ++ia) {
    bool nxt = false;
    if (ia + 1 < ze) nxt = load(ia + 1, xn, pn, qn);
    if (cur) {
      const float xa = (float)ia + 0.5f;
      const unsigned long long A = g_pk(fmul(g.ma0, xa), fmul(g.ma1, xa));
      unsigned long long P[4], Q[2];  // P[2 e + h], Q[f]
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float xp = (float)(p0 + 2 * lj + (k >> 1) + 8 * (k & 1)) + 0.5f;
        P[k] = g_pk(fmul(g.mp0, xp), fmul(g.mp1, xp));
        if (!LAST) P[k] = g_add(A, P[k]);
      }
#pragma unroll
      for (int f = 0; f < 2; ++f) {
        const float xq = (float)(q0 + 2 * li + f) + 0.5f;
        Q[f] = g_pk(fmul(g.mq0, xq), fmul(g.mq1, xq));
      }
      // voxels t and t + 1 of the lane: footprints, slot addresses; the next
      // two are worked out while this pair's slots are on their way
      Foot ft[2];
      uint32_t at[2];
      auto feet = [&](int t, Foot (&f)[2], uint32_t (&w)[2]) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          unsigned long long px = g_add(P[(t & 2) + h], Q[t >> 2]);
          if (LAST) px = g_add(px, A);
          f[h] = footprint(g_add(px, cc));
          w[h] = origin + ld16 * (uint32_t)f[h].u0 + 16u * (uint32_t)f[h].u1;
        }
      };
      feet(0, ft, at);
#pragma unroll
      for (int t = 0; t < 8; t += 2) {
        Foot fn[2];
        uint32_t an[2] = {0u, 0u};
        const unsigned long long xx[2] = {g_pk(xc[t], xc[t]), g_pk(xc[t + 1], xc[t + 1])};
        if (g.phases == 1) {
          unsigned long long s0, r0, s1, r1;
          lds_pairs(at[0], s0, r0);
          lds_pairs(at[1], s1, r1);
          if (t < 6) feet(t + 2, fn, an);
          sts_pairs(at[0], g_fma(ft[0].w0, xx[0], s0), g_fma(ft[0].w1, xx[0], r0));
          sts_pairs(at[1], g_fma(ft[1].w0, xx[1], s1), g_fma(ft[1].w1, xx[1], r1));
          __syncwarp();
        } else {
          if (t < 6) feet(t + 2, fn, an);
#pragma unroll
          for (int h = 0; h < 2; ++h)
            for (int ph = 0; ph < g.phases; ++ph) {
              if (colour == ph) {
                unsigned long long s, r;
                lds_pairs(at[h], s, r);
                sts_pairs(at[h], g_fma(ft[h].w0, xx[h], s), g_fma(ft[h].w1, xx[h], r));
              }
              __syncwarp();
            }
        }
        if (t < 6) {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            ft[h] = fn[h];
            at[h] = an[h];
          }
        }
      }
    }
    cur = nxt;
    p0 = pn;
    q0 = qn;
#pragma unroll
    for (int t = 0; t < 8; ++t) xc[t] = xn[t];
  }
}

// grid = (ceil(nwin nseg / kGenWarps), views of the launch), a warp per window
// and segment.
__global__ void __launch_bounds__(kGenWarps * 32, 5) k_p3_gen_windows(const GenFwdArgs a) {
  if (a.skip && *a.skip != 0.0) return;
  extern __shared__ __align__(16) float4 slots[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, vi = blockIdx.y;
  const GenView& gp = a.plan[a.v0 + vi];
  const int task = blockIdx.x * kGenWarps + warp, per = gp.nI * gp.nJ;
  if (!gp.ok || task >= per * a.nseg) return;
  const GenView g = gp;
  const int seg = task / per, w = task - seg * per;
  const int I = g.I0 + w / g.nJ, J = g.J0 + w % g.nJ;
  int base0, base1;
  gen_tile_base(g, I, J, base0, base1);
  // tiles off the detector are never read
  if (base0 >= a.R || base0 + g.T0 < 0 || base1 >= a.C || base1 + g.T1 < 0) return;
  float4* S = slots + warp * kSlots;
  for (int e = lane; e < g.T0 * g.LD; e += 32) S[e] = make_float4(0.f, 0.f, 0.f, 0.f);
  __syncwarp();
  const int zb = (int)((long long)g.na * seg / a.nseg), ze = (int)((long long)g.na * (seg + 1) / a.nseg);
  const uint32_t tile = (uint32_t)__cvta_generic_to_shared(S);
  if (zb < ze) {
    if (g.ax == 2)
      gen_window<true>(a, g, I, J, zb, ze, base0, base1, tile);
    else
      gen_window<false>(a, g, I, J, zb, ze, base0, base1, tile);
  }
  __syncwarp();
  // pixel (r, c): its own slot's first part, the left neighbour's second, the
  // upper one's third and the upper left one's fourth
  float* __restrict__ o = a.part + (((size_t)vi * a.nseg + seg) * a.nwin + w) * kTilePix;
  const int pc = g.T1 + 1, npix = (g.T0 + 1) * pc;
  for (int e = lane; e < npix; e += 32) {
    const int r = e / pc, c = e - r * pc;
    const float4* row = S + r * g.LD;
    float s = 0.0f;
    if (r < g.T0 && c < g.T1) s = row[c].x;
    if (r < g.T0 && c > 0) s += row[c - 1].y;
    if (r > 0 && c < g.T1) s += (row - g.LD)[c].z;
    if (r > 0 && c > 0) s += (row - g.LD)[c - 1].w;
    o[e] = s;
  }
}

// proj[v][r][c] = the windows covering (r, c): a thread finds the few that can
// from the inverse of the in-plane map (two by two for voxels of one pixel) and
// loads them together, adding in a fixed order.
// grid = (ceil(C / 32) ceil(R / kGatherWarps), views of the launch).
__global__ void __launch_bounds__(kGatherWarps * 32) k_p3_gen_gather(const GenFwdArgs a) {
  if (a.skip && *a.skip != 0.0) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, vi = blockIdx.y;
  const unsigned cols = (a.C + 31) / 32, by = blockIdx.x / cols, bx = blockIdx.x - by * cols;
  const GenView& g = a.plan[a.v0 + vi];
  if (!g.ok) return;
  const int r = (int)by * kGatherWarps + warp, c = (int)bx * 32 + lane;
  if (r >= a.R || c >= a.C) return;
  // a tap at (r, c) comes from left positions within one pixel of it
  const float y0 = (float)r - (g.c0 + 0.5f * g.ma0 - 0.25f), y1 = (float)c - (g.c1 + 0.5f * g.ma1 - 0.25f);
  const float x = g.i00 * y0 + g.i01 * y1, y = g.i10 * y0 + g.i11 * y1;
  const float mx = 1.25f * (fabsf(g.i00) + fabsf(g.i01)) + 0.01f, my = 1.25f * (fabsf(g.i10) + fabsf(g.i11)) + 0.01f;
  const int I0 = g.I0, J0 = g.J0, nJ = g.nJ, T0 = g.T0, T1 = g.T1, pc = T1 + 1;
  const int Ia = max(I0, (int)floorf(x - mx)), Ib = min(I0 + g.nI - 1, (int)floorf(x + mx));
  const int Ja = max(J0, (int)floorf(y - my)), Jb = min(J0 + nJ - 1, (int)floorf(y + my));
  const size_t seg_stride = (size_t)a.nwin * kTilePix;
  const float* __restrict__ pv = a.part + (size_t)vi * a.nseg * seg_stride;
  float acc = 0.0f;
  for (int I = Ia; I <= Ib; I += 2) {
    for (int J = Ja; J <= Jb; J += 2) {
      const float* q[4];
      bool in[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int Ik = I + (k >> 1), Jk = J + (k & 1);
        int base0, base1;
        gen_tile_base(g, Ik, Jk, base0, base1);
        const int rr = r - base0, c2 = c - base1;
        in[k] = Ik <= Ib && Jk <= Jb && (unsigned)rr <= (unsigned)T0 && (unsigned)c2 <= (unsigned)T1;
        q[k] = pv + (ptrdiff_t)((Ik - I0) * nJ + (Jk - J0)) * kTilePix + rr * pc + c2;
      }
      for (int seg = 0; seg < a.nseg; seg += 2) {
        float v[2][4];
#pragma unroll
        for (int u = 0; u < 2; ++u)
#pragma unroll
          for (int k = 0; k < 4; ++k)
            v[u][k] = in[k] && seg + u < a.nseg ? __ldg(q[k] + (size_t)(seg + u) * seg_stride) : 0.0f;
#pragma unroll
        for (int u = 0; u < 2; ++u)
#pragma unroll
          for (int k = 0; k < 4; ++k) acc += v[u][k];
      }
    }
  }
  a.proj[((size_t)(a.v0 + vi) * a.R + r) * a.C + c] = acc;
}

// ---------------------------------------------------------------------------
// GENERAL adjoint (_back_project_single, _xray3d.py:192-204): a CTA owns a
// brick of kBrick^3 voxels, a thread a column of kBrick along axis 0, and runs
// over the views in order.  Per view it stages the detector tile that the
// brick's footprints can touch, one view ahead and zero off the detector, as
// float4s of a slot's four pixels, (y[r][c], y[r+1][c]) and (y[r][c+1], y[r+1][c+1]),
// so that a voxel is one 16-byte shared load, w0 y0 + w1 y1 between columns and then
// rows, and one addition to its sum, without tests, divisions or conversions.
// Each product and sum is rounded at the size of the voxel's own taps, and a pixel of
// weight 0 adds nothing, however large (an interpolation from differences of the
// pixels, three operations less, would round at the size of the larger).  The rows'
// stride is 1 or 7 modulo 8 by the sign of the two steps along axis 2, so that
// eight neighbouring lanes walk monotonically over the eight 16-byte bank
// groups.  Views whose tile does not fit (voxels above ~1.3 detector pixels)
// gather from global memory.  Bound by the FP32 pipe (some 25 operations a voxel
// and view).  97 x 128 x 111 voxels, 60 views: one voxel a thread with four
// scalar gathers 238 us; bricks with the four weights formed and four multiply-adds
// into the sum 163 us; interpolated as here 157 us, in three view splits 141 us, with
// positions times two, whose edges are the weights without a further step, 135 us; error
// against 64 bits 1.8e-7 -> 5.9e-8.
// ---------------------------------------------------------------------------
constexpr int kBrick = 16;

// A voxel's value between the columns (y[r][c], y[r+1][c]), (y[r][c+1], y[r+1][c+1])
// and then the rows: weights s of each axis's first pixel and 1 - s of its second.
__device__ __forceinline__ float gen_interp(unsigned long long y0, unsigned long long y1, float s0, float s1) {
  const float o0 = fsub(1.0f, s0), o1 = fsub(1.0f, s1);
  float r0, r1;
  g_upk(g_fma(y0, g_pk(s1, s1), g_mul(y1, g_pk(o1, o1))), r0, r1);
  return fmaf(r0, s0, fmul(r1, o0));
}

// First pixel and its weight 2 min(ceil(left) - left, 0.5) on both axes, from twice
// the rounded position (from a matrix times two: the same roundings): adding 1.5 2^24
// rounds to an even number, so the difference of the rounding up is the weight.
constexpr float kGMagic2 = 25165824.0f;
constexpr int kGMagic2Bits = 0x4BC00000;
__device__ __forceinline__ void twice_edges(unsigned long long px2, int& u0, int& u1, float& s0, float& s1) {
  const unsigned long long magic = g_pk(kGMagic2, kGMagic2);
  const unsigned long long left2 = g_sub(px2, g_pk(0.5f, 0.5f));
  float f0, f1, a0, a1, l0, l1;
  g_upk(g_add_down(left2, magic), f0, f1);
  g_upk(g_sub(g_add_up(left2, magic), magic), a0, a1);
  g_upk(left2, l0, l1);
  s0 = __saturatef(fsub(a0, l0));
  s1 = __saturatef(fsub(a1, l1));
  u0 = __float_as_int(f0);
  u1 = __float_as_int(f1);
}

// The same of the view `y` in global memory, zero off the detector.
__device__ __forceinline__ float gen_gathered(const float* __restrict__ y, int R, int C, int u0, int u1, float t0,
                                              float t1) {
  const bool r0 = u0 >= 0 && u0 < R, r1 = u0 + 1 >= 0 && u0 + 1 < R;
  const bool c0 = u1 >= 0 && u1 < C, c1 = u1 + 1 >= 0 && u1 + 1 < C;
  const float y00 = r0 && c0 ? __ldg(y + (size_t)u0 * C + u1) : 0.0f;
  const float y10 = r1 && c0 ? __ldg(y + (size_t)(u0 + 1) * C + u1) : 0.0f;
  const float y01 = r0 && c1 ? __ldg(y + (size_t)u0 * C + u1 + 1) : 0.0f;
  const float y11 = r1 && c1 ? __ldg(y + (size_t)(u0 + 1) * C + u1 + 1) : 0.0f;
  return gen_interp(g_pk(y00, y10), g_pk(y01, y11), __saturatef(fadd(t0, t0)), __saturatef(fadd(t1, t1)));
}

constexpr int kAdjSlots = 1024;  // float4 slots of a staged tile
constexpr int kAdjChunk = 32;    // views whose tiles are laid out at once

struct GenAdjView {
  float m[8];  // the matrix times two
  int base0, base1, T0, LD;
  int ok;      // the tile fits; 2: it lies inside the detector as well
  unsigned inv;  // e / LD = (e inv) >> 16 for e < kAdjSlots
};

// grid = (bricks, view splits).
__global__ void __launch_bounds__(256, 3) k_p3_gen_adj(const float* __restrict__ proj, float* __restrict__ out,
                                                       const float* __restrict__ views, int n0, int n1, int n2, int V,
                                                       int R, int C, int per_split, size_t split_stride,
                                                       const double* skip) {
  if (skip && *skip != 0.0) return;
  __shared__ __align__(16) float4 sy[2][kAdjSlots];
  __shared__ GenAdjView tv[kAdjChunk];
  const int tid = threadIdx.x;
  const unsigned nb1 = (n1 + kBrick - 1) / kBrick, nb2 = (n2 + kBrick - 1) / kBrick;
  const int split = blockIdx.y;
  const unsigned r12 = blockIdx.x / nb2;
  const int b0 = (int)(r12 / nb1) * kBrick, b1 = (int)(r12 % nb1) * kBrick, b2 = (int)(blockIdx.x - r12 * nb2) * kBrick;
  const int i1 = b1 + (tid >> 4), i2 = b2 + (tid & 15);
  const float x1 = (float)i1 + 0.5f, x2 = (float)i2 + 0.5f;
  const int vs = split * per_split, ve = min(V, vs + per_split);
  float acc[kBrick];
#pragma unroll
  for (int k = 0; k < kBrick; ++k) acc[k] = 0.0f;

  constexpr int kStage = kAdjSlots / 256;
  float4 st[kStage];
  // the slots tid + 256 k of view `v`'s tile (tv entry t) into registers
  auto stage_load = [&](int v, const GenAdjView& t) {
    const float* __restrict__ y = proj + (size_t)v * R * C;
    const int n = t.T0 * t.LD;
#pragma unroll
    for (int k = 0; k < kStage; ++k) {
      const int e = tid + 256 * k;
      if (e < n) {
        const int r = (int)((unsigned)e * t.inv >> 16), c = e - r * t.LD;
        const int gr = t.base0 + r, gc = t.base1 + c;
        const float* __restrict__ q = y + (ptrdiff_t)gr * C + gc;
        if (t.ok == 2) {
          st[k] = make_float4(__ldg(q), __ldg(q + 1), __ldg(q + C), __ldg(q + C + 1));
        } else {
          const bool r0 = (unsigned)gr < (unsigned)R, r1 = (unsigned)(gr + 1) < (unsigned)R;
          const bool c0 = (unsigned)gc < (unsigned)C, c1 = (unsigned)(gc + 1) < (unsigned)C;
          st[k].x = r0 && c0 ? __ldg(q) : 0.0f;
          st[k].y = r0 && c1 ? __ldg(q + 1) : 0.0f;
          st[k].z = r1 && c0 ? __ldg(q + C) : 0.0f;
          st[k].w = r1 && c1 ? __ldg(q + C + 1) : 0.0f;
        }
      }
    }
  };
  auto stage_store = [&](int buf, const GenAdjView& t) {
    const int n = t.T0 * t.LD;
#pragma unroll
    for (int k = 0; k < kStage; ++k)
      if (tid + 256 * k < n)
        sy[buf][tid + 256 * k] = make_float4(st[k].x, st[k].z, st[k].y, st[k].w);
  };

  for (int vc = vs; vc < ve; vc += kAdjChunk) {
    const int nv = min(kAdjChunk, ve - vc);
    __syncthreads();  // the previous chunk's entries and tiles are done with
    if (tid < nv) {
      GenAdjView& t = tv[tid];
      const float* m = views + (size_t)(vc + tid) * kVT;
#pragma unroll
      for (int q = 0; q < 8; ++q) t.m[q] = 2.0f * m[q];
      float lo[2], ext[2], mag = 0.0f;
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const float a0 = m[4 * r], a1 = m[4 * r + 1], a2 = m[4 * r + 2];
        lo[r] = m[4 * r + 3] + a0 * ((float)b0 + 0.5f) + a1 * ((float)b1 + 0.5f) + a2 * ((float)b2 + 0.5f) - 0.25f +
                (kBrick - 1) * (fminf(a0, 0.0f) + fminf(a1, 0.0f) + fminf(a2, 0.0f)) - kTileSlack;
        ext[r] = (kBrick - 1) * (fabsf(a0) + fabsf(a1) + fabsf(a2)) + 2.0f * kTileSlack;
        mag = fmaxf(mag, fabsf(m[4 * r + 3]) + fabsf(a0) * (n0 + kBrick) + fabsf(a1) * (n1 + kBrick) + fabsf(a2) * (n2 + kBrick));
      }
      const bool small = mag < 32768.0f && ext[0] < 512.0f && ext[1] < 512.0f;
      const int T0 = small ? (int)ceilf(ext[0]) + 1 : 1, T1 = small ? (int)ceilf(ext[1]) + 1 : 1;
      const int want = m[2] * m[6] >= 0.0f ? 1 : 7;
      int LD = T1;
      while ((LD & 7) != want) ++LD;
      t.base0 = small ? (int)floorf(lo[0]) : 0;
      t.base1 = small ? (int)floorf(lo[1]) : 0;
      t.T0 = T0;
      t.LD = LD;
      t.inv = 65536u / (unsigned)LD + 1u;
      const bool fits = small && T0 * LD <= kAdjSlots && LD < 64;
      const bool inside = t.base0 >= 0 && t.base1 >= 0 && t.base0 + T0 < R && t.base1 + LD < C;
      t.ok = !fits ? 0 : (inside ? 2 : 1);
    }
    __syncthreads();
    if (tv[0].ok) {
      stage_load(vc, tv[0]);
      stage_store(0, tv[0]);
    }
    __syncthreads();
    for (int vi = 0; vi < nv; ++vi) {
      const GenAdjView& t = tv[vi];
      const bool next = vi + 1 < nv && tv[vi + 1].ok;
      if (next) stage_load(vc + vi + 1, tv[vi + 1]);
      const float m0 = t.m[0], m4 = t.m[4];
      if (t.ok) {
        const unsigned long long P = g_pk(fmul(t.m[1], x1), fmul(t.m[5], x1)), Q = g_pk(fmul(t.m[2], x2), fmul(t.m[6], x2));
        const unsigned long long cc = g_pk(t.m[3], t.m[7]);
        const uint32_t ld16 = 16u * (uint32_t)t.LD;
        const uint32_t origin = (uint32_t)__cvta_generic_to_shared(&sy[vi & 1][0]) -
                                ld16 * (uint32_t)(kGMagic2Bits + t.base0) - 16u * (uint32_t)(kGMagic2Bits + t.base1);
#pragma unroll
        for (int k = 0; k < kBrick; k += 2) {
          float v[2];
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const float x0 = (float)(b0 + k + h) + 0.5f;
            const unsigned long long A = g_pk(fmul(m0, x0), fmul(m4, x0));
            int u0, u1;
            float s0, s1;
            twice_edges(g_add(g_add(g_add(A, P), Q), cc), u0, u1, s0, s1);
            unsigned long long y0, y1;
            lds_pairs(origin + ld16 * (uint32_t)u0 + 16u * (uint32_t)u1, y0, y1);
            v[h] = gen_interp(y0, y1, s0, s1);
          }
          g_upk(g_add(g_pk(acc[k], acc[k + 1]), g_pk(v[0], v[1])), acc[k], acc[k + 1]);
        }
      } else {
        const float* y = proj + (size_t)(vc + vi) * R * C;
#pragma unroll
        for (int k = 0; k < kBrick; ++k) {
          const float x0 = (float)(b0 + k) + 0.5f;
          int u0, u1;
          float t0, t1;
          edge3(0.5f * px3(m0, t.m[1], t.m[2], t.m[3], x0, x1, x2), u0, t0);
          edge3(0.5f * px3(m4, t.m[5], t.m[6], t.m[7], x0, x1, x2), u1, t1);
          acc[k] = fadd(acc[k], gen_gathered(y, R, C, u0, u1, t0, t1));
        }
      }
      if (next) stage_store((vi + 1) & 1, tv[vi + 1]);
      __syncthreads();
    }
  }
  if (i1 >= n1 || i2 >= n2) return;
  float* __restrict__ o = out + (size_t)split * split_stride + ((size_t)b0 * n1 + i1) * n2 + i2;
#pragma unroll
  for (int k = 0; k < kBrick; ++k)
    if (b0 + k < n0) o[(size_t)k * n1 * n2] = acc[k];
}

// The same sums with a voxel per thread, four gathers a view from global memory, for
// volumes too small for their bricks to keep the SMs busy: a brick's chain of
// 16 voxels a thread and two barriers takes some 1.2 us a view, a voxel 0.28 us.
// grid = (ceil(voxels / 256), view splits).
__global__ void __launch_bounds__(256) k_p3_gen_adj_voxels(const float* __restrict__ proj, float* __restrict__ out,
                                                           const float* __restrict__ views, int n0, int n1, int n2,
                                                           int V, int R, int C, int per_split, size_t split_stride,
                                                           const double* skip) {
  if (skip && *skip != 0.0) return;
  __shared__ float sm[kAdjChunk * 8];
  const unsigned n = (unsigned)n0 * (unsigned)n1 * (unsigned)n2;
  const unsigned e = blockIdx.x * 256u + threadIdx.x;
  const int split = blockIdx.y;
  const int vs = split * per_split, ve = min(V, vs + per_split);
  const unsigned r = e / (unsigned)n2;
  const float x0 = (float)(r / (unsigned)n1) + 0.5f, x1 = (float)(r % (unsigned)n1) + 0.5f,
              x2 = (float)(e - r * (unsigned)n2) + 0.5f;
  float acc = 0.0f;
  for (int vc = vs; vc < ve; vc += kAdjChunk) {
    const int nv = min(kAdjChunk, ve - vc);
    __syncthreads();
    for (int q = threadIdx.x; q < nv * 8; q += 256) sm[q] = views[(size_t)(vc + q / 8) * kVT + (q & 7)];
    __syncthreads();
    if (e >= n) continue;
    for (int vi = 0; vi < nv; ++vi) {
      const float* m = sm + vi * 8;
      int u0, u1;
      float t0, t1;
      edge3(px3(m[0], m[1], m[2], m[3], x0, x1, x2), u0, t0);
      edge3(px3(m[4], m[5], m[6], m[7], x0, x1, x2), u1, t1);
      acc = fadd(acc, gen_gathered(proj + (size_t)(vc + vi) * R * C, R, C, u0, u1, t0, t1));
    }
  }
  if (e < n) out[(size_t)split * split_stride + e] = acc;
}

}  // namespace
}  // namespace ct
