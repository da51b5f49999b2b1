// 3D parallel-beam X-ray projector: XRayTransform3D.project / back_project
// (scico/linop/xray/_xray3d.py:95-266) for sm_103a.
//
// Weight model (_calc_weights, :206-266).  Voxel (i0, i1, i2) has its centre
// at x = (i0+0.5, i1+0.5, i2+0.5) and lands on the detector at
//   Px_r = ((M[r][0]*x0 + M[r][1]*x1) + M[r][2]*x2) + M[r][3]      (r = 0, 1)
// in float32, each operation rounded.  left = Px - 0.25,
// to_next t = min(ceil(left) - left, 0.5), ul = floor(left), and the four taps
//   (ul0,   ul1)   t0*t1*4          (ul0+1, ul1)   (0.5-t0)*t1*4
//   (ul0,   ul1+1) t0*(0.5-t1)*4    (ul0+1, ul1+1) (0.5-t0)*(0.5-t1)*4
// each zeroed when its detector pixel is out of range.  Every kernel here
// evaluates these expressions with the same float32 operations in the same
// order (no contraction) up to to_next, so forward and adjoint place every voxel
// alike and agree bit for bit in each axis's two weights; the GENERAL adjoint
// multiplies a pixel by the one and then the other (rounded after each) instead
// of by their rounded product.
//
// Two geometry kinds (ct_proj3d_views classifies):
//  * AXIS0 -- rotation about volume axis 0, slice i on detector row
//    i + row_offset with t0 = 0.5.  Then ul = 2*t1, ll = 2*(0.5-t1) (both
//    exact) and the two other taps are zero, and the column weights of pixel
//    (i1, i2) are the same for every slice.  The kernels compute each column
//    weight once per view and tile and apply it to up to 128 slices at a time:
//      forward  k_p3_ax0_fwd: lanes = slices (up to four each); a warp walks a
//               16x16 pixel tile (staged in shared memory, [pixel][slice]) in
//               the per-view detector order of the order table, carrying the
//               two open bins in registers; each completed bin is added into
//               the warp's own slices of a [group][view][col][slice]
//               accumulator in global memory (old values loaded three bins
//               ahead), which k_p3_ax0_rows transposes into the sinogram.
//      adjoint  k_p3_ax0_adj: lanes = slices (up to four each), a warp owns
//               4x4 pixels; the view's detector columns are staged as
//               [column][slice] and kept in registers from pixel to pixel.
//  * GENERAL -- any matrices: proj3d_gen.cuh.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <map>
#include <mutex>
#include <tuple>
#include <type_traits>
#include <vector>

#include "kernels.cuh"

namespace ct {
namespace {

constexpr int kVT = CT_VIEW3D_STRIDE;
constexpr int kOrd = CT_PROJ3D_ORDER;
constexpr int kTileJ = 16, kTileK = 16;  // AXIS0 forward pixel tile (axis 1 x axis 2)
constexpr int kFwdPad = 64;  // slices of the forward accumulator are padded to this
constexpr int kWalkGroup = 4;   // walk entries tested together for a new bin

static_assert(kTileJ * kTileK == kOrd, "order table covers one tile");

// Device error word of the 3D kernels' internal checks (bit 0: forward tile
// span, bit 1: adjoint window span).
__device__ int g_proj3d_err = 0;

int* errflag3_ptr() {
  static int* cached[64] = {nullptr};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
  if (!cached[dev]) {
    int* p = nullptr;
    if (cudaGetSymbolAddress((void**)&p, g_proj3d_err) != cudaSuccess) return nullptr;
    cached[dev] = p;
  }
  return cached[dev];
}

// Detector coordinate of voxel centre (x0, x1, x2) on detector axis r of a
// view (_xray3d.py:214-219), rounded like the reference's float32 expression.
__device__ __forceinline__ float px3(float m0, float m1, float m2, float m3, float x0, float x1,
                                     float x2) {
  return fadd(fadd(fadd(fmul(m0, x0), fmul(m1, x1)), fmul(m2, x2)), m3);
}

// left = Px - w/2, to_next = min(ceil(left) - left, w), ul = floor(left)
// with w = 0.5 (:222-225).
__device__ __forceinline__ void edge3(float px, int& ul, float& t) {
  const float left = fsub(px, 0.25f);
  t = fminf(fsub(ceilf(left), left), 0.5f);
  ul = (int)floorf(left);
}

// 4-byte global -> shared copy that bypasses registers; zero-fills when
// `valid` is false (source size 0, nothing is read).
__device__ __forceinline__ void cp_async4(uint32_t dst, const float* src, bool valid) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src),
               "r"(valid ? 4 : 0)
               : "memory");
}

__device__ __forceinline__ void cp_async4_all(uint32_t dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}

__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.wait_all;" ::: "memory");
}

}  // namespace
}  // namespace ct

#include "proj3d_gen.cuh"

namespace ct {
namespace {

// ---------------------------------------------------------------------------
// AXIS0 forward
// ---------------------------------------------------------------------------
struct Ax0FwdArgs {
  const float* vol;  // (S, NJ, NK)
  float* acc_out;    // [G][V][C][Spad]
  const float* views;
  const uint16_t* order;
  int S, NJ, NK, V, C, Spad;
  int tiles_k, n_tiles, G;
  int* errflag;
  const double* skip;  // device flag: return at once when non-zero (may be null)
};

// Bin range of one 16x16 tile for one view.  Every operation of the rounded
// Px is monotone in each pixel index, so the tile's extremes are at corner
// pixels; floor(left) of those, widened by one bin below and two above
// (room for the second tap and the carried bin), gives [lo, hi).
__device__ __forceinline__ void tile_bins(float m11, float m12, float m13, int j0, int k0,
                                          int& lo, int& hi) {
  const float ja = (float)j0 + 0.5f, jb = (float)(j0 + kTileJ - 1) + 0.5f;
  const float ka = (float)k0 + 0.5f, kb = (float)(k0 + kTileK - 1) + 0.5f;
  const float a0 = fmul(m11, ja), a1 = fmul(m11, jb);
  const float b0 = fmul(m12, ka), b1 = fmul(m12, kb);
  const float pmin = fadd(fminf(a0, a1) + fminf(b0, b1), m13);
  const float pmax = fadd(fmaxf(a0, a1) + fmaxf(b0, b1), m13);
  lo = (int)floorf(pmin - 0.25f) - 1;
  hi = (int)floorf(pmax - 0.25f) + 3;
}

// Tile order of the forward: Z-order (Morton) over the tile grid's
// power-of-two bounding box, axis-2 tile bit lowest, the longer side's
// surplus bits on top.  A tile group takes a run of consecutive tiles in this
// order, a compact patch of the image, so that for every view the tiles it
// visits one after another touch overlapping detector columns and the
// accumulator's read-modify-write stays in L2.
__device__ __forceinline__ int bit_len(int n) {  // bits of n - 1 (0 for n <= 1)
  return n <= 1 ? 0 : 32 - __clz(n - 1);
}
__device__ __forceinline__ void zorder_decode(int code, int bj, int bk, int& tj, int& tk) {
  const int m = min(bj, bk);
  tj = 0;
  tk = 0;
  for (int b = 0; b < m; ++b) {
    tk |= ((code >> (2 * b)) & 1) << b;
    tj |= ((code >> (2 * b + 1)) & 1) << b;
  }
  const int rest = code >> (2 * m);
  if (bj > m) tj |= rest << m;
  else tk |= rest << m;
}
// Tiles of the grid [0, nj) x [0, nk) inside the box [j, j + sj) x [k, k + sk).
__device__ __forceinline__ int tiles_in(int j, int sj, int k, int sk, int nj, int nk) {
  return max(0, min(nj, j + sj) - j) * max(0, min(nk, k + sk) - k);
}
// Code of the r-th tile of the grid in Z-order (r < nj * nk): descend the
// surplus blocks, then the quadrants, counting the grid tiles each holds.
__device__ int zorder_select(int r, int nj, int nk) {
  const int bj = bit_len(nj), bk = bit_len(nk), m = min(bj, bk);
  const int sq = 1 << m;
  int code = 0, j = 0, k = 0;
  const int nblk = 1 << (max(bj, bk) - m);
  for (int blk = 0; blk < nblk; ++blk) {
    const int jb = bj > m ? blk * sq : 0, kb = bj > m ? 0 : blk * sq;
    const int c = tiles_in(jb, sq, kb, sq, nj, nk);
    if (r < c) {
      code = blk << (2 * m);
      j = jb;
      k = kb;
      break;
    }
    r -= c;
  }
  for (int l = m - 1; l >= 0; --l) {
    const int s = 1 << l;
    for (int q = 0; q < 4; ++q) {
      const int dj = q >> 1, dk = q & 1;
      const int c = tiles_in(j + dj * s, s, k + dk * s, s, nj, nk);
      if (r < c || q == 3) {
        code |= q << (2 * l);
        j += dj * s;
        k += dk * s;
        break;
      }
      r -= c;
    }
  }
  return code;
}

// SL consecutive floats as one shared or global access.
template <int SL>
struct FwdVec {
  float x[SL];
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int i = 0; i < SL; ++i) x[i] = 0.0f;
  }
  // sums and differences by pairs (each half rounded as the scalar operation)
  __device__ __forceinline__ FwdVec plus(const FwdVec& b) const {
    FwdVec r;
    if constexpr (SL > 1) {
#pragma unroll
      for (int i = 0; i < SL; i += 2) g_upk(g_add(g_pk(x[i], x[i + 1]), g_pk(b.x[i], b.x[i + 1])), r.x[i], r.x[i + 1]);
    } else {
      r.x[0] = x[0] + b.x[0];
    }
    return r;
  }
  __device__ __forceinline__ FwdVec minus(const FwdVec& b) const {
    FwdVec r;
    if constexpr (SL > 1) {
#pragma unroll
      for (int i = 0; i < SL; i += 2) g_upk(g_sub(g_pk(x[i], x[i + 1]), g_pk(b.x[i], b.x[i + 1])), r.x[i], r.x[i + 1]);
    } else {
      r.x[0] = x[0] - b.x[0];
    }
    return r;
  }
  // this += w x, sx += x
  __device__ __forceinline__ void add(float w, const FwdVec& v, FwdVec& sx) {
    if constexpr (SL > 1) {
      const unsigned long long ww = g_pk(w, w);
#pragma unroll
      for (int i = 0; i < SL; i += 2) {
        const unsigned long long xx = g_pk(v.x[i], v.x[i + 1]);
        g_upk(g_fma(ww, xx, g_pk(x[i], x[i + 1])), x[i], x[i + 1]);
        g_upk(g_add(g_pk(sx.x[i], sx.x[i + 1]), xx), sx.x[i], sx.x[i + 1]);
      }
    } else {
      x[0] = fmaf(w, v.x[0], x[0]);
      sx.x[0] += v.x[0];
    }
  }
  static __device__ __forceinline__ FwdVec shared(uint32_t at) {
    FwdVec v;
    if constexpr (SL == 4)
      asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x[0]), "=f"(v.x[1]), "=f"(v.x[2]), "=f"(v.x[3]) : "r"(at));
    else if constexpr (SL == 2)
      asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x[0]), "=f"(v.x[1]) : "r"(at));
    else
      asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v.x[0]) : "r"(at));
    return v;
  }
  static __device__ __forceinline__ FwdVec global(const float* p) {
    FwdVec v;
    if constexpr (SL == 4) {
      const float4 f = __ldcg(reinterpret_cast<const float4*>(p));
      v.x[0] = f.x;
      v.x[1] = f.y;
      v.x[2] = f.z;
      v.x[3] = f.w;
    } else if constexpr (SL == 2) {
      const float2 f = __ldcg(reinterpret_cast<const float2*>(p));
      v.x[0] = f.x;
      v.x[1] = f.y;
    } else {
      v.x[0] = __ldcg(p);
    }
    return v;
  }
  __device__ __forceinline__ void store(float* p) const {
    if constexpr (SL == 4)
      __stcg(reinterpret_cast<float4*>(p), make_float4(x[0], x[1], x[2], x[3]));
    else if constexpr (SL == 2)
      __stcg(reinterpret_cast<float2*>(p), make_float2(x[0], x[1]));
    else
      __stcg(p, x[0]);
  }
};

__host__ __device__ constexpr int fwd_row(int SL) { return 32 * SL + 4; }  // floats of a staged pixel
constexpr size_t fwd3_smem(int SL, int NW) {
  return sizeof(float) * kOrd * fwd_row(SL) + NW * (sizeof(float2) + sizeof(unsigned char)) * kOrd;
}

// AXIS0 forward: a CTA takes 32 SL slices, NW views (a warp each) and a run of
// pixel tiles.  A tile is staged as [pixel][slice] (rows of 32 SL + 4 floats:
// the transposing copies of 8 pixels x 4 slices a warp hit 32 banks, a warp
// reads a pixel in 16-byte pieces without conflicts); a warp walks its 256
// pixels in the view's detector order with the open bin and its successor in
// registers, SL slices a lane: one shared read of x, one of the table entry
// (weight, pixel offset) and two operations a slice per pixel.  Entries are
// tested four at a time for a new bin, which about one in ten pixels opens.
// Bound by shared reads (4 bytes an interaction) and issue slots.  SL and NW
// are the plan's.  256^3 x 360 views with two slices a
// lane, two views a warp and a test per entry 3853 us a call, this 1972 us.
template <int SL, int NW>
__global__ void __launch_bounds__(NW * 32, SL == 4 ? 1 : 2) k_p3_ax0_fwd(const Ax0FwdArgs a) {
  if (a.skip && *a.skip != 0.0) return;
  extern __shared__ __align__(16) float smem[];
  constexpr int kRow = fwd_row(SL);
  float* sv = smem;                                               // [kOrd][kRow]
  float2* tab = reinterpret_cast<float2*>(sv + kOrd * kRow);      // [NW][kOrd] weight, byte offset | new bin << 31
  unsigned char* bins = reinterpret_cast<unsigned char*>(tab + NW * kOrd);  // [NW][kOrd] tile-relative bin
  __shared__ int2 tlist[256];                                     // tile origins (j0, k0)
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = blockIdx.x, i0 = blockIdx.y * 32 * SL, v = blockIdx.z * NW + warp;
  bool live = v < a.V;  // warp-uniform
  float2* tabw = tab + warp * kOrd;
  unsigned char* binw = bins + warp * kOrd;
  const uint32_t sv_s = (uint32_t)__cvta_generic_to_shared(sv);

  // this warp's accumulator slices (column c at o + c Spad), zeroed; its view
  // parameters and walk order (entry 32u + lane)
  const bool mine = live && i0 + SL * lane < a.Spad;
  float* o = a.acc_out + ((size_t)g * a.V + (live ? v : 0)) * a.C * a.Spad + i0 + SL * lane;
  FwdVec<SL> zero;
  zero.zero();
  float m11 = 0.f, m12 = 0.f, m13 = 0.f;
  unsigned ord[kOrd / 64];
  if (live) {
    if (mine)
      for (int c = 0; c < a.C; ++c) zero.store(o + (size_t)c * a.Spad);
    const float* m = a.views + (size_t)v * kVT;
    m11 = m[5];
    m12 = m[6];
    m13 = m[7];
    const uint16_t* q = a.order + (size_t)v * kOrd;
#pragma unroll
    for (int u = 0; u < kOrd / 64; ++u) ord[u] = __ldg(q + 64 * u + lane) | (unsigned)__ldg(q + 64 * u + 32 + lane) << 16;
    // a tile's bins are kept in 8 bits (at most 36 for |m| <= 1, which ct_proj3d_views
    // sees to); a view of another table that needs more is left out: zeros
    if (!(15.0f * (fabsf(m11) + fabsf(m12)) <= 250.0f)) {
      if (lane == 0) atomicOr(a.errflag, 1);
      live = false;
    }
  }

  const int per = (a.n_tiles + a.G - 1) / a.G, nrun = min(per, a.n_tiles - g * per);
  const int c8 = lane & 7, s4 = lane >> 3;
  for (int q = 0; q < nrun; ++q) {
    if ((q & 255) == 0) {
      // this group's run of tiles in Z-order, ranks [g per, (g + 1) per)
      for (int e = tid; e < 256 && q + e < nrun; e += NW * 32) {
        const int tiles_j = a.n_tiles / a.tiles_k;
        int tj, tk;
        zorder_decode(zorder_select(g * per + q + e, tiles_j, a.tiles_k), bit_len(tiles_j), bit_len(a.tiles_k), tj, tk);
        tlist[e] = make_int2(tj * kTileJ, tk * kTileK);
      }
      __syncthreads();
    }
    const int2 t0 = tlist[q & 255];
    const int j0 = t0.x, k0 = t0.y;
    // stage: a warp copies 8 pixels of a row x 4 slices per instruction, the
    // slice quads warp, warp + NW, ..
    const bool inside = j0 + kTileJ <= a.NJ && k0 + kTileK <= a.NK;
    for (int sq = warp; sq < 8 * SL; sq += NW) {
      const int s = 4 * sq + s4;
      const float* src = a.vol + ((size_t)min(i0 + s, a.S - 1) * a.NJ + j0) * a.NK + k0 + c8;
      uint32_t d = sv_s + 4u * (uint32_t)(c8 * kRow + s);
      if (inside && i0 + 4 * sq + 4 <= a.S) {  // warp-uniform
#pragma unroll
        for (int j = 0; j < kTileJ; ++j) {
          cp_async4_all(d, src);
          cp_async4_all(d + 4u * 8 * kRow, src + 8);
          src += a.NK;
          d += 4u * kTileK * kRow;
        }
      } else {
        for (int j = 0; j < kTileJ; ++j) {
          const bool row = i0 + s < a.S && j0 + j < a.NJ;
          const bool ok0 = row && k0 + c8 < a.NK, ok1 = row && k0 + c8 + 8 < a.NK;
          cp_async4(d, ok0 ? src : a.vol, ok0);
          cp_async4(d + 4u * 8 * kRow, ok1 ? src + 8 : a.vol, ok1);
          src += a.NK;
          d += 4u * kTileK * kRow;
        }
      }
    }
    // the next tile's accumulator columns towards L2 (all the CTAs' accumulators
    // are larger than it): 8 columns x 4 pieces of the slices an instruction
    if (live && q + 1 < nrun && ((q + 1) & 255) != 0) {
      const int2 t1 = tlist[(q + 1) & 255];
      int lo, hi;
      tile_bins(m11, m12, m13, t1.x, t1.y, lo, hi);
      const float* ahead = o - SL * lane + 8 * SL * s4;
      for (int c = lo + c8; c < hi; c += 8)
        if (c >= 0 && c < a.C && i0 + 8 * SL * s4 < a.Spad)
          asm volatile("prefetch.global.L2 [%0];" ::"l"(ahead + (ptrdiff_t)c * a.Spad));
    }
    // the view's table while the copies run.  The second tap's weight is
    // 1 - w0 = 2 (0.5 - t1) exactly; taps on columns off the detector are
    // accumulated and never written out, so no masks here
    int lo = 0;
    // the accumulator's values of the open bin's column and the next two
    FwdVec<SL> r0 = zero, r1 = zero, r2 = zero;
    auto old_at = [&](int c, const float* at, FwdVec<SL>& r) {
      r = zero;
      if (mine && (unsigned)c < (unsigned)a.C) r = FwdVec<SL>::global(at);
    };
    auto put = [&](int c, float* at, const FwdVec<SL>& r) {
      if (mine && (unsigned)c < (unsigned)a.C) r.store(at);
    };
    if (live) {
      int hi;
      tile_bins(m11, m12, m13, j0, k0, lo, hi);
      old_at(lo, o + (ptrdiff_t)lo * a.Spad, r0);
      old_at(lo + 1, o + (ptrdiff_t)(lo + 1) * a.Spad, r1);
      old_at(lo + 2, o + (ptrdiff_t)(lo + 2) * a.Spad, r2);
      const int nb = hi - lo;
      int last = 0;  // the bin of the entry before this round's first
#pragma unroll
      for (int u = 0; u < kOrd / 32; ++u) {
        const int p = (int)((ord[u / 2] >> (16 * (u & 1))) & 0xffffu);
        const float x1 = (float)(j0 + p / kTileK) + 0.5f, x2 = (float)(k0 + p % kTileK) + 0.5f;
        // Px_1 with M[1][0] = 0: the x0 term is an exact zero
        const float px = fadd(fadd(fmul(m11, x1), fmul(m12, x2)), m13);
        int ul;
        float t1;
        edge3(px, ul, t1);
        const int rel = min(max(ul - lo, 0), nb - 2);  // in range: extremes at corners
        const int before = __shfl_up_sync(0xffffffffu, rel, 1);
        const bool opens = rel != (lane == 0 ? last : before);
        last = __shfl_sync(0xffffffffu, rel, 31);
        tabw[32 * u + lane] = make_float2(fmul(2.0f, t1), __int_as_float(p * kRow * 4 | (opens ? (int)0x80000000 : 0)));
        binw[32 * u + lane] = (unsigned char)rel;
      }
    }
    cp_async_wait_all();
    __syncthreads();

    if (live) {
      // Open bin c - lo: its total is cin + sum w0*x over its own pixels (av);
      // the next bin receives sum (1-w0)*x = sx - av.
      int c = lo;
      float* at = o + (ptrdiff_t)lo * a.Spad;
      FwdVec<SL> cin = zero, av = zero, sx = zero;
      auto open_bin = [&](int nc) {
        put(c, at, r0.plus(cin.plus(av)));
        cin = sx.minus(av);
        if (nc == c + 1) {
          at += a.Spad;
          r0 = r1;
          r1 = r2;
          old_at(c + 3, at + 2 * (ptrdiff_t)a.Spad, r2);
        } else {  // a jump (rare: rounding at near-ties of the order)
          put(c + 1, at + a.Spad, r1.plus(cin));
          at = o + (ptrdiff_t)nc * a.Spad;
          old_at(nc, at, r0);
          old_at(nc + 1, at + a.Spad, r1);
          old_at(nc + 2, at + 2 * (ptrdiff_t)a.Spad, r2);
          cin = zero;
        }
        av = zero;
        sx = zero;
        c = nc;
      };
      const uint32_t xb = sv_s + 4u * SL * (uint32_t)lane;
#pragma unroll 2
      for (int e0 = 0; e0 < kOrd; e0 += kWalkGroup) {
        float2 T[kWalkGroup];
        int any = 0;
#pragma unroll
        for (int u = 0; u < kWalkGroup; ++u) {
          T[u] = tabw[e0 + u];
          any |= __float_as_int(T[u].y);
        }
        FwdVec<SL> x[kWalkGroup];
        if (any >= 0) {  // no new bin among them (warp-uniform)
#pragma unroll
          for (int u = 0; u < kWalkGroup; ++u) x[u] = FwdVec<SL>::shared(xb + (uint32_t)__float_as_int(T[u].y));
#pragma unroll
          for (int u = 0; u < kWalkGroup; ++u) av.add(T[u].x, x[u], sx);
        } else {
#pragma unroll
          for (int u = 0; u < kWalkGroup; ++u)
            x[u] = FwdVec<SL>::shared(xb + (uint32_t)(__float_as_int(T[u].y) & 0x7fffffff));
#pragma unroll
          for (int u = 0; u < kWalkGroup; ++u) {
            if (__float_as_int(T[u].y) < 0) open_bin(lo + binw[e0 + u]);
            av.add(T[u].x, x[u], sx);
          }
        }
      }
      put(c, at, r0.plus(cin.plus(av)));
      put(c + 1, at + a.Spad, r1.plus(sx.minus(av)));
    }
    __syncthreads();
  }
}

constexpr int kMaxGroups = 8;  // AXIS0 forward tile groups (the most a schedule uses)

// proj[v][r][c] = sum_g acc_out[g][v][c][r - row_offset] in group order (0 where
// no slice lands on row r).  32x32 (col, row) tiles through shared memory, the
// groups' values of four columns all loaded before they are added.
__global__ void __launch_bounds__(256) k_p3_ax0_rows(const float* __restrict__ acc, float* __restrict__ proj, int V,
                              int R, int C, int S, int Spad, int G, int row_offset,
                              const double* skip) {
  if (skip && *skip != 0.0) return;
  __shared__ float t[32][33];
  const int c0 = blockIdx.x * 32, r0 = blockIdx.y * 32, v = blockIdx.z;
  const int lx = threadIdx.x, ly = threadIdx.y;  // 32 x 8
  const int i = r0 + lx - row_offset;
  const bool slice = i >= 0 && i < S;
  float s[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int gg = 0; gg < kMaxGroups; gg += 4) {
    if (gg >= G) break;
    float x[4][4];
#pragma unroll
    for (int h = 0; h < 4; ++h)
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int c = c0 + ly + 8 * q;
        x[h][q] = slice && c < C && gg + h < G ? __ldcs(acc + (((size_t)(gg + h) * V + v) * C + c) * Spad + i) : 0.f;
      }
#pragma unroll
    for (int h = 0; h < 4; ++h)
#pragma unroll
      for (int q = 0; q < 4; ++q) s[q] += x[h][q];
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) t[ly + 8 * q][lx] = s[q];
  __syncthreads();
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int rl = ly + 8 * q, r = r0 + rl, c = c0 + lx;
    if (r < R && c < C) proj[((size_t)v * R + r) * C + c] = t[lx][rl];
  }
}

// ---------------------------------------------------------------------------
// AXIS0 adjoint.  A CTA owns 16 x 16 pixels and 32 SL slices, a warp 4 x 4 of
// the pixels with SL slices a lane: 16 SL accumulators in registers.  The
// views' detector windows are staged as [column][slice] (rows of 32 SL + 4
// floats: the transposing copies of 8 columns x 4 slices a warp hit 32 banks,
// a warp reads a row in 16-byte pieces without conflicts), kAdjViews views per
// barrier, the next ones copied meanwhile.  A pixel takes the rows of its two
// columns for all its slices.  Even rows live in one set of registers and odd
// rows in another, each reloaded only when a pixel needs another row, and the
// 4 x 4 pixels are visited back and forth along the axis whose step on the
// detector is the smaller: about half of the pixels load one row, some 2 bytes
// of shared reads per interaction instead of the 8 of one (y[c], y[c+1]) pair
// each, which bound the version before (lane = pixel, 32 slices of
// accumulators).  Weights and row offsets come from a table that a warp makes
// for its pixels, half a warp per view.  256^3 x 360 views: 2258 -> 1494 us (two view
// splits), of issue slots (19 a pixel and view) and shared reads alike.
// ---------------------------------------------------------------------------
constexpr int kAdjTile = 16;   // tile edge (pixels)
constexpr int kAdjCols = 40;   // staged columns: 15 (|m11| + |m12|) + 6 for |m| <= 1, whole copies of 8
constexpr int kAdjViews = 4;   // views per barrier
constexpr int kAdjWarps = 16;
constexpr int kAdjChunk3 = 512;  // views whose windows are laid out at once

struct Ax0AdjArgs {
  const float* proj;  // (V, R, C)
  float* out;         // (S, NJ, NK), or split partials
  const float* views;
  int S, NJ, NK, V, R, C, row_offset;
  int tiles_k, nsg;   // tiles along axis 2, slice groups
  int per_split;
  size_t split_stride;
  int* errflag;
  const double* skip;
};

__host__ __device__ constexpr int adj_row(int SL) { return 32 * SL + 4; }  // floats of a staged column
constexpr size_t adj3_smem(int SL) {
  return sizeof(float) * 2 * kAdjViews * kAdjCols * adj_row(SL) +
         (sizeof(float2) + sizeof(unsigned)) * kAdjWarps * kAdjViews * 16 + (sizeof(float4) + sizeof(int)) * kAdjChunk3;
}

// Window [lo, lo + nb) of detector columns that the tile at (j0, k0) reads in
// one view: every operation of the rounded Px is monotone in each pixel index,
// so the extremes are at corners (one column spare below, two above).
__device__ __forceinline__ void adj_window(float m11, float m12, float m13, int j0, int k0,
                                           int& lo, int& nb) {
  const float ja = (float)j0 + 0.5f, jb = (float)(j0 + kAdjTile - 1) + 0.5f;
  const float ka = (float)k0 + 0.5f, kb = (float)(k0 + kAdjTile - 1) + 0.5f;
  const float a0 = fmul(m11, ja), a1 = fmul(m11, jb), b0 = fmul(m12, ka), b1 = fmul(m12, kb);
  lo = (int)floorf(fadd(fminf(a0, a1) + fminf(b0, b1), m13) - 0.25f) - 1;
  nb = (int)floorf(fadd(fmaxf(a0, a1) + fmaxf(b0, b1), m13) - 0.25f) + 3 - lo;
}

// SL floats a lane of a staged column.
template <int SL>
struct AdjVec {
  float p[SL];
  // the row at `at`, when it is not the one held
  __device__ __forceinline__ void reload(uint32_t at, uint32_t held) {
    if constexpr (SL == 4)
      asm volatile("{\n.reg .pred p;\nsetp.ne.u32 p, %4, %5;\n@p ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];\n}"
                   : "+f"(p[0]), "+f"(p[1]), "+f"(p[2]), "+f"(p[3])
                   : "r"(at), "r"(held));
    else if constexpr (SL == 2)
      asm volatile("{\n.reg .pred p;\nsetp.ne.u32 p, %2, %3;\n@p ld.shared.v2.f32 {%0, %1}, [%2];\n}"
                   : "+f"(p[0]), "+f"(p[1])
                   : "r"(at), "r"(held));
    else
      asm volatile("{\n.reg .pred p;\nsetp.ne.u32 p, %1, %2;\n@p ld.shared.f32 %0, [%1];\n}"
                   : "+f"(p[0])
                   : "r"(at), "r"(held));
  }
  __device__ __forceinline__ void fma(float w, const AdjVec& y) {
#pragma unroll
    for (int i = 0; i < SL; ++i) p[i] = fmaf(w, y.p[i], p[i]);
  }
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int i = 0; i < SL; ++i) p[i] = 0.0f;
  }
  __device__ __forceinline__ void store(float* o) const {
#pragma unroll
    for (int i = 0; i < SL; ++i) o[i] = p[i];
  }
};

// Position t of a visit of the 4 x 4 pixels: back and forth along axis 2
// (COL = false) or axis 1; returns 4 (axis-1 offset) + (axis-2 offset).
template <bool COL>
__host__ __device__ constexpr int visit(int t) {
  const int o = t >> 2, i = (o & 1) ? 3 - (t & 3) : (t & 3);
  return COL ? 4 * i + o : 4 * o + i;
}

template <int SL, bool COL>
__device__ __forceinline__ void adj_view(const float2* wt, const uint2* ot, uint32_t base, AdjVec<SL> (&acc)[16]) {
  AdjVec<SL> ye, yo;
  ye.zero();
  yo.zero();
  uint32_t he = 0xffffffffu, ho = 0xffffffffu;
#pragma unroll
  for (int t = 0; t < 16; t += 2) {
    const uint2 o = ot[t / 2];  // two pixels: offset of the even row, of the odd row (16 bits each)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const float2 w = wt[t + h];  // their weights
      const uint32_t oh = h ? o.y : o.x;
      const uint32_t ae = base + (oh & 0xffffu), ao = base + (oh >> 16);
      ye.reload(ae, he);
      yo.reload(ao, ho);
      he = ae;
      ho = ao;
      AdjVec<SL>& a = acc[visit<COL>(t + h)];
      a.fma(w.x, ye);
      a.fma(w.y, yo);
    }
  }
}

// grid = (tiles, slice groups x splits), block = 512.
template <int SL>
__global__ void __launch_bounds__(kAdjWarps * 32, 1) k_p3_ax0_adj(const Ax0AdjArgs a) {
  if (a.skip && *a.skip != 0.0) return;
  extern __shared__ __align__(16) float smem[];
  constexpr int kRow = adj_row(SL), kBuf = kAdjViews * kAdjCols * kRow;
  float2* wtab = reinterpret_cast<float2*>(smem + 2 * kBuf);  // [warp][view][16] weight of the even row, of the odd row
  unsigned* otab = reinterpret_cast<unsigned*>(wtab + kAdjWarps * kAdjViews * 16);  // [warp][view][16] byte offsets
  float4* vtab = reinterpret_cast<float4*>(otab + kAdjWarps * kAdjViews * 16);  // M[1][1..3], first column
  int* ntab = reinterpret_cast<int*>(vtab + kAdjChunk3);                // columns
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int j0 = (blockIdx.x / a.tiles_k) * kAdjTile, k0 = (blockIdx.x % a.tiles_k) * kAdjTile;
  const int sg = blockIdx.y % a.nsg, split = blockIdx.y / a.nsg;
  const int i0 = sg * 32 * SL;
  const int vs = split * a.per_split, ve = min(a.V, vs + a.per_split);
  const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(smem);

  // staging: lane = 8 columns x 4 slices; a warp takes the slice quads
  // warp, warp + 16, ..
  const int c8 = lane & 7, s4 = lane >> 3;
  constexpr int kQuads = (8 * SL + kAdjWarps - 1) / kAdjWarps;
  const bool has = 8 * SL >= kAdjWarps || 4 * warp < 32 * SL;
  bool rows_ok = true;
  bool row_ok[kQuads];
  const float* row[kQuads];
#pragma unroll
  for (int q = 0; q < kQuads; ++q) {
    const int s = 4 * (warp + kAdjWarps * q) + s4, r = i0 + s + a.row_offset;
    row_ok[q] = has && i0 + s < a.S && r >= 0 && r < a.R;
    rows_ok = rows_ok && row_ok[q];
    row[q] = a.proj + (size_t)(row_ok[q] ? r : 0) * a.C + c8;
  }
  rows_ok = __all_sync(0xffffffffu, rows_ok);
  const uint32_t dst0 = sbase + 4u * (uint32_t)(c8 * kRow + 4 * warp + s4);
  auto stage = [&](int v, int slot, int lo, int nb) {
    const uint32_t d = dst0 + 4u * (uint32_t)(slot * kAdjCols * kRow);
    const ptrdiff_t off = (ptrdiff_t)v * a.R * a.C + lo;
    if (rows_ok && lo >= 0 && lo + 8 * ((nb + 7) / 8) <= a.C) {  // warp-uniform: every copy reads
#pragma unroll
      for (int q = 0; q < kQuads; ++q) {
        const float* src = row[q] + off;
#pragma unroll
        for (int g = 0; g < kAdjCols / 8; ++g)
          if (8 * g < nb) cp_async4_all(d + 4u * (uint32_t)(8 * g * kRow + 4 * kAdjWarps * q), src + 8 * g);
      }
    } else if (has) {
#pragma unroll
      for (int q = 0; q < kQuads; ++q) {
#pragma unroll
        for (int g = 0; g < kAdjCols / 8; ++g)
          if (8 * g < nb) {
            const bool ok = row_ok[q] && (unsigned)(lo + 8 * g + c8) < (unsigned)a.C;
            cp_async4(d + 4u * (uint32_t)(8 * g * kRow + 4 * kAdjWarps * q), ok ? row[q] + off + 8 * g : a.proj, ok);
          }
      }
    }
  };

  AdjVec<SL> acc[16];
#pragma unroll
  for (int p = 0; p < 16; ++p) acc[p].zero();
  const int jw = j0 + 4 * (warp >> 2), kw = k0 + 4 * (warp & 3);
  float2* wt = wtab + warp * kAdjViews * 16;
  unsigned* ot = otab + warp * kAdjViews * 16;

  for (int vc = vs; vc < ve; vc += kAdjChunk3) {
    const int nc = min(kAdjChunk3, ve - vc);
    for (int u = tid; u < nc; u += kAdjWarps * 32) {
      const float* m = a.views + (size_t)(vc + u) * kVT;
      int lo, nb;
      adj_window(m[5], m[6], m[7], j0, k0, lo, nb);
      if (nb > kAdjCols) atomicOr(a.errflag, 2);  // cannot happen for |m| <= 1
      vtab[u] = make_float4(m[5], m[6], m[7], __int_as_float(lo));
      ntab[u] = min(nb, kAdjCols);
    }
    __syncthreads();
    auto stage_batch = [&](int c, int buf) {
#pragma unroll
      for (int u = 0; u < kAdjViews; ++u)
        if (c + u < nc) stage(vc + c + u, buf * kAdjViews + u, __float_as_int(vtab[c + u].w), ntab[c + u]);
    };
    stage_batch(0, 0);
    cp_async_wait_all();
    __syncthreads();
    int buf = 0;
    for (int c = 0; c < nc; c += kAdjViews, buf ^= 1) {
      if (c + kAdjViews < nc) stage_batch(c + kAdjViews, buf ^ 1);
      const int nv = min(kAdjViews, nc - c);
      // weights and rows of the warp's pixels in visiting order, two views at
      // a time (half a warp each)
#pragma unroll
      for (int u = 0; u < kAdjViews; u += 2) {
        const int vu = u + (lane >> 4), t = lane & 15;
        if (vu < nv) {
          const float4 m = vtab[c + vu];
          const int p = fabsf(m.y) > fabsf(m.x) ? visit<true>(t) : visit<false>(t);
          const float x1 = (float)(jw + (p >> 2)) + 0.5f, x2 = (float)(kw + (p & 3)) + 0.5f;
          const float px = fadd(fadd(fmul(m.x, x1), fmul(m.y, x2)), m.z);
          int ul;
          float t1;
          edge3(px, ul, t1);
          // columns off the detector are staged as zeros; inside the window
          // by the corner bound
          const int rel = min(max(ul - __float_as_int(m.w), 0), ntab[c + vu] - 2), odd = rel & 1;
          const float w0 = fmul(2.0f, t1), w1 = fmul(2.0f, fsub(0.5f, t1));
          wt[16 * vu + t] = make_float2(odd ? w1 : w0, odd ? w0 : w1);
          ot[16 * vu + t] = (unsigned)((rel + odd) * kRow * 4) | (unsigned)((rel + 1 - odd) * kRow * 4) << 16;
        }
      }
      __syncwarp();
      const uint32_t vb = sbase + 4u * (uint32_t)(buf * kBuf) + 4u * SL * (uint32_t)lane;
#pragma unroll 1
      for (int u = 0; u < nv; ++u) {
        const float4 m = vtab[c + u];
        const uint32_t base = vb + 4u * (uint32_t)(u * kAdjCols * kRow);
        if (fabsf(m.y) > fabsf(m.x))
          adj_view<SL, true>(wt + 16 * u, reinterpret_cast<const uint2*>(ot + 16 * u), base, acc);
        else
          adj_view<SL, false>(wt + 16 * u, reinterpret_cast<const uint2*>(ot + 16 * u), base, acc);
      }
      cp_async_wait_all();
      __syncthreads();
    }
  }
  // the accumulators through shared memory, [pixel][slice], so that the rows
  // along axis 2 are written whole
#pragma unroll
  for (int p = 0; p < 16; ++p) {
    const int pix = (4 * (warp >> 2) + (p >> 2)) * kAdjTile + 4 * (warp & 3) + (p & 3);
    acc[p].store(smem + pix * kRow + SL * lane);
  }
  __syncthreads();
  float* out = a.out + (size_t)split * a.split_stride;
  for (int e = tid; e < 32 * SL * kAdjTile * kAdjTile; e += kAdjWarps * 32) {
    const int k = e & 15, j = (e >> 4) & 15, s = e >> 8;
    if (i0 + s < a.S && j0 + j < a.NJ && k0 + k < a.NK)
      out[((size_t)(i0 + s) * a.NJ + j0 + j) * a.NK + k0 + k] = smem[(j * kAdjTile + k) * kRow + s];
  }
}

// ---------------------------------------------------------------------------
// GENERAL forward, the march: one detector pixel per thread.  Taps are found
// plane by plane along the ray's dominant axis; an exact test on the rounded ul
// decides membership, so each output has one owner.  SOME: only the views of
// `plan` that the window kernels (proj3d_gen.cuh) leave out, by few blocks a view, as most find
// it taken; else every view, a pixel per thread (the loop over pixels costs 3-7 %:
// 64^3 voxels of three pixels, 30 views, 1154 -> 1102 us).
// ---------------------------------------------------------------------------
// x range [lo, hi] of voxel centres along one axis allowed by the detector
// window [wlo, whi] on one detector axis, given Px = beta + mq * x.
__device__ __forceinline__ void narrow(float beta, float mq, float wlo, float whi, float& lo,
                                       float& hi) {
  if (fabsf(mq) > 1e-20f) {
    const float u = (wlo - beta) / mq, w = (whi - beta) / mq;
    lo = fmaxf(lo, fminf(u, w));
    hi = fminf(hi, fmaxf(u, w));
  } else if (beta < wlo || beta > whi) {
    lo = 1.0f;
    hi = 0.0f;
  }
}

template <bool SOME>
__global__ void __launch_bounds__(256) k_p3_gen_march(const float* __restrict__ vol,
                                                      float* __restrict__ proj,
                                                      const float* __restrict__ views, int n0,
                                                      int n1, int n2, int R, int C,
                                                      const GenView* __restrict__ plan,
                                                      const double* skip) {
  if (skip && *skip != 0.0) return;
  const int v = blockIdx.y;
  if (SOME && plan[v].ok) return;
  const float* m = views + (size_t)v * kVT;
  float mm[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) mm[q] = m[q];
  const int ax = (int)m[8];
  // the other two axes, ascending: p = ax==0 ? 1 : 0, q = ax==2 ? 1 : 2
  auto pick = [ax](float a0, float a1, float a2, int which) {
    // which: 0 = the marching axis, 1 = p, 2 = q
    const int k = which == 0 ? ax : (which == 1 ? (ax == 0 ? 1 : 0) : (ax == 2 ? 1 : 2));
    return k == 0 ? a0 : (k == 1 ? a1 : a2);
  };
  const float na_f = pick((float)n0, (float)n1, (float)n2, 0);
  const int na = (int)na_f, np = (int)pick((float)n0, (float)n1, (float)n2, 1),
            nq = (int)pick((float)n0, (float)n1, (float)n2, 2);
  const float ma0 = pick(mm[0], mm[1], mm[2], 0), mp0 = pick(mm[0], mm[1], mm[2], 1),
              mq0 = pick(mm[0], mm[1], mm[2], 2);
  const float ma1 = pick(mm[4], mm[5], mm[6], 0), mp1 = pick(mm[4], mm[5], mm[6], 1),
              mq1 = pick(mm[4], mm[5], mm[6], 2);
  // voxel strides of the marching, p and q axes
  const size_t sa = ax == 0 ? (size_t)n1 * n2 : (ax == 1 ? (size_t)n2 : 1);
  const size_t sp = ax == 0 ? (size_t)n2 : (size_t)n1 * n2;
  const size_t sq = ax == 2 ? (size_t)n2 : 1;
  const int first = blockIdx.x * blockDim.x + threadIdx.x;
  if (!SOME && first >= R * C) return;
  for (int pix = first; pix < R * C; pix += gridDim.x * blockDim.x) {
    const int r = pix / C, c = pix - (pix / C) * C;
    // taps reaching (r, c) come from voxels with floor(left) in {r-1, r} x
    // {c-1, c}: Px in [r-0.75, r+1.25) x [c-0.75, c+1.25); widened by a margin
    // far above the rounding of the range arithmetic (the exact test decides)
    const float mg = 0.05f;
    const float w0lo = (float)r - 0.75f - mg, w0hi = (float)r + 1.25f + mg;
    const float w1lo = (float)c - 0.75f - mg, w1hi = (float)c + 1.25f + mg;
    // |x_p - centre_p| <= e_p from the 2x2 system of the (p, q) plane
    const float det = mp0 * mq1 - mq0 * mp1;
    const float h0 = 0.5f * (w0hi - w0lo), h1 = 0.5f * (w1hi - w1lo);
    const float ep = (fabsf(mq1) * h0 + fabsf(mq0) * h1) / fabsf(det);
    float acc = 0.f;
    for (int ia = 0; ia < na; ++ia) {
      const float xa = (float)ia + 0.5f;
      const float al0 = ma0 * xa + mm[3], al1 = ma1 * xa + mm[7];
      const float cr0 = 0.5f * (w0lo + w0hi) - al0, cr1 = 0.5f * (w1lo + w1hi) - al1;
      const float cp = (mq1 * cr0 - mq0 * cr1) / det;
      const float plo = fmaxf(0.5f, cp - ep - mg), phi = fminf((float)np - 0.5f, cp + ep + mg);
      if (!(plo <= phi)) continue;
      const int ip0 = max(0, (int)ceilf(plo - 0.5f)), ip1 = min(np - 1, (int)floorf(phi - 0.5f));
      for (int ip = ip0; ip <= ip1; ++ip) {
        const float xp = (float)ip + 0.5f;
        float qlo = 0.5f, qhi = (float)nq - 0.5f;
        narrow(al0 + mp0 * xp, mq0, w0lo, w0hi, qlo, qhi);
        narrow(al1 + mp1 * xp, mq1, w1lo, w1hi, qlo, qhi);
        if (!(qlo <= qhi)) continue;
        const int iq0 = max(0, (int)ceilf(qlo - 0.5f - mg)), iq1 = min(nq - 1, (int)floorf(qhi - 0.5f + mg));
        for (int iq = iq0; iq <= iq1; ++iq) {
          const int i0 = ax == 0 ? ia : ip;
          const int i1 = ax == 0 ? ip : (ax == 1 ? ia : iq);
          const int i2 = ax == 2 ? ia : iq;
          const float x0 = (float)i0 + 0.5f, x1 = (float)i1 + 0.5f, x2 = (float)i2 + 0.5f;
          int u0, u1;
          float t0, t1;
          edge3(px3(mm[0], mm[1], mm[2], mm[3], x0, x1, x2), u0, t0);
          edge3(px3(mm[4], mm[5], mm[6], mm[7], x0, x1, x2), u1, t1);
          const int d0 = r - u0, d1 = c - u1;
          if ((unsigned)d0 > 1u || (unsigned)d1 > 1u) continue;
          const float f0 = d0 ? fsub(0.5f, t0) : t0;
          const float f1 = d1 ? fsub(0.5f, t1) : t1;
          const float w = fmul(fmul(f0, f1), 4.0f);
          acc = fmaf(w, __ldg(vol + ia * sa + ip * sp + iq * sq), acc);
        }
      }
    }
    proj[((size_t)v * R + r) * C + c] = acc;
    if (!SOME) break;
  }
}

// out[e] = sum over the view splits, in split order.  A stream of nsplit + 1
// volumes: W = 4 elements an access where the volume's size and both arrays allow
// it, four splits loaded before they are added (2 splits of 256^3: 71.6 us with
// single elements, 26.1 us; the back projection 1541 -> 1501 us).
template <int W>
__global__ void __launch_bounds__(256) k_p3_sum_splits(const float* __restrict__ part, float* __restrict__ out,
                                                       size_t n, int nsplit) {
  constexpr int kAhead = 4;
  for (size_t e = W * ((size_t)blockIdx.x * 256 + threadIdx.x); e < n; e += W * (size_t)gridDim.x * 256) {
    float acc[W] = {};
    for (int k = 0; k < nsplit; k += kAhead) {
      float v[kAhead][W];
#pragma unroll
      for (int u = 0; u < kAhead; ++u) {
        if (k + u >= nsplit) break;
        const float* q = part + (size_t)(k + u) * n + e;
        if constexpr (W == 4) {
          const float4 f = __ldcs(reinterpret_cast<const float4*>(q));
          v[u][0] = f.x, v[u][1] = f.y, v[u][2] = f.z, v[u][3] = f.w;
        } else {
          v[u][0] = __ldcs(q);
        }
      }
#pragma unroll
      for (int u = 0; u < kAhead; ++u) {
        if (k + u >= nsplit) break;
#pragma unroll
        for (int j = 0; j < W; ++j) acc[j] += v[u][j];
      }
    }
    if constexpr (W == 4)
      *reinterpret_cast<float4*>(out + e) = make_float4(acc[0], acc[1], acc[2], acc[3]);
    else
      out[e] = acc[0];
  }
}

}  // namespace

// ---------------------------------------------------------------------------
// Host planning and launchers
// ---------------------------------------------------------------------------

ct_status proj3d_check(const ct_geom3d* g, const char* who) {
  if (!g) return fail(CT_ERR_INVALID_ARG, "%s: null geometry", who);
  for (int q = 0; q < 3; ++q)
    if (g->shape[q] <= 0) return fail(CT_ERR_SHAPE, "%s: shape[%d]=%d", who, q, g->shape[q]);
  if (g->det_shape[0] <= 0 || g->det_shape[1] <= 0)
    return fail(CT_ERR_SHAPE, "%s: det_shape=(%d, %d)", who, g->det_shape[0], g->det_shape[1]);
  if (g->n_views <= 0) return fail(CT_ERR_SHAPE, "%s: n_views=%d", who, g->n_views);
  if (!g->views) return fail(CT_ERR_INVALID_ARG, "%s: null view table", who);
  if (g->kind != CT_PROJ3D_GENERAL && g->kind != CT_PROJ3D_AXIS0)
    return fail(CT_ERR_INVALID_ARG, "%s: kind=%d", who, g->kind);
  if (g->kind == CT_PROJ3D_AXIS0 && !g->order)
    return fail(CT_ERR_INVALID_ARG, "%s: AXIS0 geometry without an order table", who);
  const double n = (double)g->shape[0] * g->shape[1] * g->shape[2];
  if (n > 2147483647.0 || (double)g->det_shape[0] * g->det_shape[1] > 2147483647.0)
    return fail(CT_ERR_UNSUPPORTED, "%s: volume or detector above 2^31 elements", who);
  return CT_OK;
}

// Most adjoint view splits the tuner tries.
constexpr int kMaxSplits3d = 4;
constexpr size_t kGenScratch = 96u << 20;       // bytes of GENERAL forward tiles per launch
constexpr size_t kGenScratchView = 1024u << 20;  // the most that one view's tiles may take (or the volume's size)

// Windows of a view of a GENERAL forward (a bound over the marching axes; 0: no
// windows, the march), segments of its planes until two warps a slot are there, and
// the bytes of one view's tiles.  Flat volumes thousands of voxels wide have so many windows that their
// tiles would outgrow the volume itself: those march.
struct GenTiles {
  int nwin = 0, nseg = 1;
  size_t per_view = 0;
};
GenTiles gen_tiles(const int32_t* n, int V) {
  GenTiles t;
  double nwin = 0;
  for (int ax = 0; ax < 3; ++ax) {
    const long na = n[ax], np = n[ax == 0 ? 1 : 0], nq = n[ax == 2 ? 1 : 2];
    nwin = std::max(nwin, (double)((np + na) / kWin + 2) * (double)((nq + na) / kWin + 2));
  }
  const size_t most = std::max(kGenScratchView, sizeof(float) * (size_t)n[0] * n[1] * n[2]);
  if (nwin * sizeof(float) * kTilePix > (double)most) return t;
  t.nwin = (int)nwin;
  const long warps = std::max(1L, t.nwin / 4L * V), target = 40L * std::max(1, sm_count());
  t.nseg = (int)std::min<long>(std::max(1L, (target + warps - 1) / warps),
                               std::max(1, std::min({n[0], n[1], n[2]}) / 8));
  const size_t one = sizeof(float) * (size_t)t.nwin * kTilePix;
  t.nseg = (int)std::min<size_t>(t.nseg, std::max<size_t>(1, most / one));
  t.per_view = one * t.nseg;
  return t;
}

// The AXIS0 span bounds need max |M[1][1]| and |M[1][2]|; ct_proj3d_views
// guarantees both <= 1, so the bounds are fixed.
Proj3dPlan proj3d_plan_sched(const ct_geom3d* g, Sched3d sc) {
  Proj3dPlan p;
  const int S = g->shape[0], NJ = g->shape[1], NK = g->shape[2], V = g->n_views;
  const int C = g->det_shape[1];
  const int sms = std::max(1, sm_count());
  int ns = 1, ns_max = 1;
  // adjoint scratch below which a call (old_ns splits) and its tuning (the
  // splits that it tries) have always been refused
  auto least_scratch = [&](int old_ns, int tried) {
    const size_t one = sizeof(float) * (size_t)S * NJ * NK;
    const int eff = sc.ns > 0 ? std::min(sc.ns, ns_max) : old_ns;
    const int per = (V + eff - 1) / eff, split = (V + per - 1) / per, tune = std::max(old_ns, tried);
    p.adj_least = split > 1 ? round_up((size_t)split * one, 256) : 0;
    p.adj_tune = tune > 1 ? round_up((size_t)tune * one, 256) : 0;
  };
  if (g->kind == CT_PROJ3D_AXIS0) {
    p.Spad = (S + kFwdPad - 1) / kFwdPad * kFwdPad;
    p.tiles_k = (NK + kTileK - 1) / kTileK;
    p.n_tiles = p.tiles_k * ((NJ + kTileJ - 1) / kTileJ);
    const int g_max = std::min(kMaxGroups, p.n_tiles);
    // forward: slices a lane, warps a CTA and tile groups by the time of the
    // busiest SM, in units of one view's walk of a tile with four slices a lane:
    // 0.66 and 0.5 for two and one, a tile's copies, which nothing overlaps,
    // about a quarter a slice of the lane, slower below 16 warps an SM (0.7 of
    // the rate at 8, 1.15 at 32); fitted to 256^3 x 360, 128^3 x 180, 64^3 x 90
    // and unequal sides
    auto fwd_cost = [&](int sl, int nw, int G) {
      const long ctas = (long)((S + 32 * sl - 1) / (32 * sl)) * ((V + nw - 1) / nw) * G;
      const double rounds = std::ceil((double)ctas / sms);
      const int fit = sl == 4 ? 1 : std::min((int)(220 * 1024 / fwd3_smem(sl, nw)), nw == 16 ? 2 : 20 / nw);
      const double warps = nw * std::min((double)fit, rounds);
      const double walk = sl == 4 ? 1.0 : (sl == 2 ? 0.66 : 0.5);
      return rounds * ((p.n_tiles + G - 1) / G) * (nw * walk + 0.25 * sl) / std::min(1.15, std::pow(warps / 16.0, 0.55)) +
             0.02 * (double)V * p.n_tiles * S / 128 / sms * G;  // the groups' sum
    };
    auto fwd_best = [&](int G, Proj3dPlan& q) {
      double best = 1e300;
      for (int sl = 4; sl >= 1; sl /= 2)
        for (int nw = 16; nw >= 4; nw /= 2) {
          const double c = fwd_cost(sl, nw, G);
          if (c < 0.98 * best) {
            best = c;
            q.fwd_sl = sl;
            q.fwd_nw = nw;
          }
        }
      return best;
    };
    p.G = std::min(std::max(sc.G, 1), g_max);
    if (sc.G <= 0) {
      double best = 1e300;
      for (int G = 1; G <= g_max; ++G) {
        const double c = fwd_best(G, p);
        if (c < 0.98 * best) {
          best = c;
          p.G = G;
        }
      }
    }
    fwd_best(p.G, p);
    // the groups that a call has always needed scratch for (64 slices and 16
    // views a CTA, two CTAs an SM)
    int old_G = std::min(std::max(sc.G, 1), g_max);
    if (sc.G <= 0) {
      const long base = (long)(p.Spad / 64) * ((V + 15) / 16), slots = 2L * sms;
      double best = -1.0;
      for (int G = 1; G <= g_max; ++G) {
        const double waves = (double)(base * G) / (double)slots;
        const double score = std::min(1.0, waves) * waves / std::ceil(waves);
        if (score > best + 1e-9) {
          best = score;
          old_G = G;
        }
      }
    }
    const size_t group = sizeof(float) * (size_t)V * C * p.Spad;
    p.fwd_least = round_up(group * old_G, 256);
    p.fwd_bytes = round_up(group * p.G, 256);
    p.fwd_ws_bytes = round_up(group * g_max, 256);
    // adjoint: slices a lane (SL) and view splits by the time of the busiest SM,
    // in units of a CTA's view: 1 at SL = 4, 0.62 and 0.42 at 2 and 1 (the
    // per-pixel work is shared by fewer slices); a split costs a pass over
    // its partial volume
    const long tiles = (long)((NK + kAdjTile - 1) / kAdjTile) * ((NJ + kAdjTile - 1) / kAdjTile);
    auto cost = [&](int sl, int k) {
      const long ctas = tiles * ((S + 32 * sl - 1) / (32 * sl));
      return std::ceil((double)ctas * k / sms) * (sl == 4 ? 1.0 : (sl == 2 ? 0.62 : 0.42)) / k * (k > 1 ? 1.0 + 4.0 * (k + 0.5) / V : 1.0);
    };
    auto lanes = [&](int k) { return cost(4, k) <= std::min(cost(2, k), cost(1, k)) ? 4 : (cost(2, k) <= cost(1, k) ? 2 : 1); };
    const int most = std::max(1, V / (2 * kAdjViews));
    ns_max = std::max(1, V / 16);
    // the scratch that a call has always needed (32 x 16 pixel tiles of 32 slices)
    const long old_ctas = (long)((NK + 31) / 32) * ((NJ + 15) / 16) * (p.Spad / 32);
    const int old_ns = std::min(old_ctas < 304 ? (int)((304 + old_ctas - 1) / old_ctas) : 1, ns_max);
    // and no fewer splits than those, so that no sum gets longer (134 x 200 x 72, 64
    // views: one split instead of two has 1.7 times the error against 64 bits)
    double least = 1e300;
    for (int k = std::min({16, most, old_ns}); k <= std::min(16, most); ++k) {
      const double c = cost(lanes(k), k);
      if (c < 0.98 * least) {
        least = c;
        ns = k;
      }
    }
    p.adj_sl = lanes(sc.ns > 0 ? std::min(sc.ns, most) : ns);
    least_scratch(old_ns, std::min(kMaxSplits3d, ns_max));
    ns_max = most;
  } else {
    ns_max = std::max(1, V / 8);
    // the scratch that a call has always needed (a voxel per thread, four CTAs
    // of 256 an SM); one with no more runs the splits that fit (ct_proj3d_adj)
    const long old_ctas = (long)(((double)S * NJ * NK + 255) / 256);
    const int old_ns = std::min(old_ctas < 4L * sms ? (int)((4L * sms + old_ctas - 1) / old_ctas) : 1, ns_max);
    least_scratch(old_ns, std::min(kMaxSplits3d, ns_max));
    // Bricks, or a voxel per thread where there are too few bricks to keep the SMs
    // busy, and the view splits, by the us of the busiest SM: a view costs a brick
    // 1.2, each further brick beside it (three an SM) 0.55; a voxel's chain 0.28 a view, or
    // the rate of 4e-6 a voxel and view; splits a pass over the partial volumes.  Within
    // 10 % of the best measured choice for volumes of 8^3 to 128^3 with 3 to 180
    // views (16^3, 6 views: 9.6 us in bricks, 2.5 us by voxels; 40^3, 20 views 15.9 and 8.5;
    // 64^3, 20 views 13.6 and 24.0; 4 x 256 x 256, 8 views 17.2 and 11.7).  Bricks need
    // a lead: voxels of more than a pixel, which only the device sees, cost them up
    // to three times as much.
    ns_max = std::max(1, V / 2);
    const double voxels = (double)S * NJ * NK;
    const long bricks = (long)((S + kBrick - 1) / kBrick) * ((NJ + kBrick - 1) / kBrick) * ((NK + kBrick - 1) / kBrick);
    auto split_us = [&](int k) { return k > 1 ? 2.0 + 7e-7 * voxels * (k + 1) : 0.0; };
    auto brick_us = [&](int k) {
      const long c = (bricks * k + sms - 1) / sms, part = c % 3;
      return ((V + k - 1) / k) * ((c / 3) * 2.3 + (part ? 0.65 + 0.55 * part : 0.0)) + split_us(k);
    };
    auto voxel_us = [&](int k) { return std::max(0.28 * ((V + k - 1) / k), 4e-6 * voxels * V) + split_us(k); };
    // no fewer splits than fill the SMs' three CTAs or a call has always had, at eight
    // views or more each, so that no sum gets longer
    int first = 1;
    double least = 1e300;
    for (int k = 1; k <= 16; ++k) {
      const double rounds = std::ceil((double)bricks * k / (3.0 * sms)) / k * (1.0 + 0.02 * (k - 1));
      if (rounds < 0.98 * least) {
        least = rounds;
        first = k;
      }
    }
    first = std::max(old_ns, std::min(first, std::max(1, V / 8)));
    int nb = first, nv = first;
    for (int k = first + 1; k <= std::min(16, ns_max); ++k)
      if (brick_us(k) < 0.98 * brick_us(nb)) nb = k;
    for (int k = first + 1; k <= std::min(16, V / 4); ++k)
      if (voxel_us(k) < 0.98 * voxel_us(nv)) nv = k;
    ns = voxel_us(nv) < 1.25 * brick_us(nb) ? nv : nb;  // also the scratch that is asked for, whatever the schedule
    if (sc.ns > 0) nb = nv = std::min(sc.ns, ns_max);
    p.adj_voxels = voxel_us(nv) < 1.25 * brick_us(nb);
    // forward: views per launch until the tiles of a launch pass kGenScratch (they
    // are read back from L2); the turned volume last, so that a call can go without it
    const GenTiles t = gen_tiles(g->shape, V);
    p.nwin = t.nwin;
    p.nseg = t.nseg;
    if (p.nwin > 0) {
      p.gen_views = (int)std::max<size_t>(1, std::min<size_t>(std::min(V, 65535), kGenScratch / t.per_view));
      p.gen_plan = round_up(sizeof(GenView) * (size_t)V, 256);
      p.gen_tiles = round_up((size_t)p.gen_views * t.per_view, 256);
      p.gen_turn = round_up(sizeof(float) * (size_t)S * NJ * NK, 256);
      p.fwd_bytes = p.fwd_ws_bytes = p.gen_plan + p.gen_tiles + p.gen_turn;
    }
  }
  ns = std::min(ns, ns_max);
  const int ns_ws = std::max(ns, std::min(kMaxSplits3d, ns_max));
  if (sc.ns > 0) ns = std::min(sc.ns, ns_max);
  p.per_split = (V + ns - 1) / ns;
  p.nsplit = (V + p.per_split - 1) / p.per_split;
  p.adj_bytes = p.nsplit > 1 ? round_up(sizeof(float) * (size_t)p.nsplit * S * NJ * NK, 256) : 0;
  p.adj_ws_bytes = ns_ws > 1 ? round_up(sizeof(float) * (size_t)ns_ws * S * NJ * NK, 256) : 0;
  p.adj_ws_bytes = std::max(p.adj_ws_bytes, std::max(p.adj_bytes, std::max(p.adj_least, p.adj_tune)));
  return p;
}

ct_status sum_splits(const float* part, float* out, size_t n, int nsplit, cudaStream_t s) {
  const int vec = quad_ok(n, part, out);
  const size_t per = vec ? 1024 : 256;
  const int blocks = (int)std::min<size_t>((n + per - 1) / per, 16 * 1024);
  (vec ? k_p3_sum_splits<4> : k_p3_sum_splits<1>)<<<blocks, 256, 0, s>>>(part, out, n, nsplit);
  return launch_check("k_p3_sum_splits");
}

// Schedules recorded by ct_proj3d_autotune, keyed by the geometry's sizes
// and kind.
using Sched3dKey = std::tuple<int, int, int, int, int, int, int>;
struct Sched3dVal {
  Sched3d s;
  float fwd_us = 0.0f, adj_us = 0.0f;
};
std::mutex g_sched3_mu;
std::map<Sched3dKey, Sched3dVal> g_sched3;

Sched3dKey sched3_key(const ct_geom3d* g) {
  return Sched3dKey(g->shape[0], g->shape[1], g->shape[2], g->n_views, g->det_shape[0], g->det_shape[1], g->kind);
}

bool sched3_lookup(const ct_geom3d* g, Sched3dVal& out) {
  std::lock_guard<std::mutex> lk(g_sched3_mu);
  const auto it = g_sched3.find(sched3_key(g));
  if (it == g_sched3.end()) return false;
  out = it->second;
  return true;
}

Proj3dPlan proj3d_plan(const ct_geom3d* g, int batch) {
  (void)batch;  // one volume per launch; a batch runs the same plan per volume
  Sched3dVal v;
  return proj3d_plan_sched(g, sched3_lookup(g, v) ? v.s : Sched3d{});
}

ct_status need_ws(const char* who, size_t need, void* ws, size_t bytes) {
  if (need == 0) return CT_OK;
  if (!ws || bytes < need || !aligned(ws, 256))
    return fail(CT_ERR_WORKSPACE, "%s: need %zu bytes (256-B aligned), got %zu", who, need, bytes);
  return CT_OK;
}

// f(kernel, shared bytes, slices of a CTA) of the plan's AXIS0 forward.
template <class F>
void with_fwd(const Proj3dPlan& p, F&& f) {
  auto by_warps = [&](auto sl) {
    constexpr int SL = decltype(sl)::value;
    if (p.fwd_nw == 16)
      f(k_p3_ax0_fwd<SL, 16>, fwd3_smem(SL, 16), 32 * SL);
    else if (p.fwd_nw == 8)
      f(k_p3_ax0_fwd<SL, 8>, fwd3_smem(SL, 8), 32 * SL);
    else
      f(k_p3_ax0_fwd<SL, 4>, fwd3_smem(SL, 4), 32 * SL);
  };
  if (p.fwd_sl == 4)
    by_warps(std::integral_constant<int, 4>());
  else if (p.fwd_sl == 2)
    by_warps(std::integral_constant<int, 2>());
  else
    by_warps(std::integral_constant<int, 1>());
}

// The kernels' dynamic shared memory limits, raised once per device (any plan
// of a geometry may follow).
ct_status proj3d_prepare(const ct_geom3d* g, const Proj3dPlan& p) {
  (void)g;
  (void)p;
  if (!errflag3_ptr()) return fail(CT_ERR_CUDA, "proj3d: error-word address unavailable");
  static std::atomic<uint64_t> done{0};
  int dev = 0;
  ct_status st = cuda_check(cudaGetDevice(&dev), "current device");
  if (st != CT_OK) return st;
  const uint64_t bit = dev < 64 ? 1ull << dev : 0;
  if (done.load(std::memory_order_acquire) & bit) return CT_OK;
  auto raise = [&](auto* kernel, size_t bytes, const char* what) {
    if (st == CT_OK)
      st = cuda_check(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes), what);
  };
  raise(k_p3_gen_windows, sizeof(float4) * kGenWarps * kSlots, "k_p3_gen_windows smem attribute");
  raise(k_p3_ax0_adj<4>, adj3_smem(4), "k_p3_ax0_adj smem attribute");
  raise(k_p3_ax0_adj<2>, adj3_smem(2), "k_p3_ax0_adj smem attribute");
  raise(k_p3_ax0_adj<1>, adj3_smem(1), "k_p3_ax0_adj smem attribute");
  Proj3dPlan each;
  for (each.fwd_sl = 1; each.fwd_sl <= 4; each.fwd_sl *= 2)
    for (each.fwd_nw = 4; each.fwd_nw <= 16; each.fwd_nw *= 2)
      with_fwd(each, [&](auto* kernel, size_t bytes, int) { raise(kernel, bytes, "k_p3_ax0_fwd smem attribute"); });
  if (st == CT_OK) done.fetch_or(bit, std::memory_order_release);
  return st;
}

ct_status proj3d_fwd_launch(const ct_geom3d* g, const Proj3dPlan& p, const float* vol, float* proj,
                            void* ws, cudaStream_t s, const double* skip) {
  const int S = g->shape[0], NJ = g->shape[1], NK = g->shape[2], V = g->n_views;
  const int R = g->det_shape[0], C = g->det_shape[1];
  if (g->kind == CT_PROJ3D_AXIS0) {
    Ax0FwdArgs a;
    a.vol = vol;
    a.acc_out = static_cast<float*>(ws);
    a.views = g->views;
    a.order = g->order;
    a.S = S;
    a.NJ = NJ;
    a.NK = NK;
    a.V = V;
    a.C = C;
    a.Spad = p.Spad;
    a.tiles_k = p.tiles_k;
    a.n_tiles = p.n_tiles;
    a.G = p.G;
    a.errflag = errflag3_ptr();
    a.skip = skip;
    with_fwd(p, [&](auto* kernel, size_t bytes, int slices) {
      const dim3 grid(p.G, (S + slices - 1) / slices, (V + p.fwd_nw - 1) / p.fwd_nw);
      kernel<<<grid, p.fwd_nw * 32, bytes, s>>>(a);
    });
    ct_status st = launch_check("k_p3_ax0_fwd");
    if (st != CT_OK) return st;
    dim3 g2((C + 31) / 32, (R + 31) / 32, V);
    k_p3_ax0_rows<<<g2, dim3(32, 8), 0, s>>>(a.acc_out, proj, V, R, C, S, p.Spad, p.G,
                                             g->row_offset, skip);
    return launch_check("k_p3_ax0_rows");
  }
  GenView* plan = p.nwin > 0 ? static_cast<GenView*>(ws) : nullptr;
  if (plan) {
    GenFwdArgs a;
    float* turned = p.gen_turn ? reinterpret_cast<float*>(static_cast<char*>(ws) + p.gen_plan + p.gen_tiles) : nullptr;
    a.vol = vol;
    a.vol_t = turned;
    a.plan = plan;
    a.part = reinterpret_cast<float*>(static_cast<char*>(ws) + p.gen_plan);
    a.proj = proj;
    a.n0 = S;
    a.n1 = NJ;
    a.n2 = NK;
    a.R = R;
    a.C = C;
    a.nwin = p.nwin;
    a.nseg = p.nseg;
    a.skip = skip;
    const unsigned turn_blocks = !turned ? 0 : (unsigned)((S * (long)NJ + 31) / 32) * (unsigned)((NK + 31) / 32);
    k_p3_gen_setup<<<(V + 7) / 8 + turn_blocks, 256, 0, s>>>(g->views, plan, vol, turned, S, NJ, NK, V, p.nwin, skip);
    ct_status st = launch_check("k_p3_gen_setup");
    if (st != CT_OK) return st;
    for (a.v0 = 0; a.v0 < V; a.v0 += p.gen_views) {
      const int nv = std::min(p.gen_views, V - a.v0);
      const dim3 gw((unsigned)(((long)p.nwin * p.nseg + kGenWarps - 1) / kGenWarps), nv);
      k_p3_gen_windows<<<gw, kGenWarps * 32, sizeof(float4) * kGenWarps * kSlots, s>>>(a);
      st = launch_check("k_p3_gen_windows");
      if (st != CT_OK) return st;
      const dim3 gg((unsigned)((C + 31) / 32) * (unsigned)((R + kGatherWarps - 1) / kGatherWarps), nv);
      k_p3_gen_gather<<<gg, kGatherWarps * 32, 0, s>>>(a);
      st = launch_check("k_p3_gen_gather");
      if (st != CT_OK) return st;
    }
  }
  const int full = (int)(((long)R * C + 255) / 256);
  dim3 grid(plan ? std::min(full, std::max(16, 16 * sm_count() / V)) : full, V);
  (plan ? k_p3_gen_march<true> : k_p3_gen_march<false>)<<<grid, 256, 0, s>>>(vol, proj, g->views, S, NJ, NK, R, C, plan, skip);
  return launch_check("k_p3_gen_march");
}

ct_status proj3d_adj_launch(const ct_geom3d* g, const Proj3dPlan& p, const float* proj, float* out,
                            float* part, cudaStream_t s, const double* skip) {
  const int S = g->shape[0], NJ = g->shape[1], NK = g->shape[2], V = g->n_views;
  const int R = g->det_shape[0], C = g->det_shape[1];
  const size_t vol_n = (size_t)S * NJ * NK;
  float* dst = p.nsplit > 1 ? part : out;
  if (g->kind == CT_PROJ3D_AXIS0) {
    Ax0AdjArgs a;
    a.proj = proj;
    a.out = dst;
    a.views = g->views;
    a.S = S;
    a.NJ = NJ;
    a.NK = NK;
    a.V = V;
    a.R = R;
    a.C = C;
    a.row_offset = g->row_offset;
    a.tiles_k = (NK + kAdjTile - 1) / kAdjTile;
    a.nsg = (S + 32 * p.adj_sl - 1) / (32 * p.adj_sl);
    a.per_split = p.per_split;
    a.split_stride = vol_n;
    a.errflag = errflag3_ptr();
    a.skip = skip;
    const dim3 grid((unsigned)a.tiles_k * ((NJ + kAdjTile - 1) / kAdjTile), a.nsg * p.nsplit);
    if (p.adj_sl == 4)
      k_p3_ax0_adj<4><<<grid, kAdjWarps * 32, adj3_smem(4), s>>>(a);
    else if (p.adj_sl == 2)
      k_p3_ax0_adj<2><<<grid, kAdjWarps * 32, adj3_smem(2), s>>>(a);
    else
      k_p3_ax0_adj<1><<<grid, kAdjWarps * 32, adj3_smem(1), s>>>(a);
    return launch_check("k_p3_ax0_adj");
  }
  if (p.adj_voxels) {
    k_p3_gen_adj_voxels<<<dim3((unsigned)((vol_n + 255) / 256), p.nsplit), 256, 0, s>>>(
        proj, dst, g->views, S, NJ, NK, V, R, C, p.per_split, vol_n, skip);
    return launch_check("k_p3_gen_adj_voxels");
  }
  const dim3 grid((unsigned)((NK + kBrick - 1) / kBrick) * ((NJ + kBrick - 1) / kBrick) * ((S + kBrick - 1) / kBrick), p.nsplit);
  k_p3_gen_adj<<<grid, 256, 0, s>>>(proj, dst, g->views, S, NJ, NK, V, R, C, p.per_split, vol_n,
                                    skip);
  return launch_check("k_p3_gen_adj");
}

}  // namespace ct

extern "C" {

ct_status ct_proj3d_views(const float* matrices, int32_t n_views, const int32_t* shape,
                          const int32_t* det_shape, float* views_out, uint16_t* order_out,
                          int32_t* kind_out, int32_t* row_offset_out) {
  using ct::fail;
  if (!matrices || !shape || !det_shape || !views_out || !kind_out || !row_offset_out)
    return fail(CT_ERR_INVALID_ARG, "ct_proj3d_views: null argument");
  if (n_views <= 0) return fail(CT_ERR_SHAPE, "ct_proj3d_views: n_views=%d", n_views);
  for (int q = 0; q < 3; ++q)
    if (shape[q] <= 0) return fail(CT_ERR_SHAPE, "ct_proj3d_views: shape[%d]=%d", q, shape[q]);
  if (det_shape[0] <= 0 || det_shape[1] <= 0)
    return fail(CT_ERR_SHAPE, "ct_proj3d_views: det_shape=(%d, %d)", det_shape[0], det_shape[1]);
  for (int v = 0; v < n_views; ++v) {
    const float* m = matrices + (size_t)v * 8;
    float* t = views_out + (size_t)v * CT_VIEW3D_STRIDE;
    for (int q = 0; q < 8; ++q) {
      if (!std::isfinite(m[q]))
        return fail(CT_ERR_NONFINITE, "ct_proj3d_views: matrix %d has a non-finite entry", v);
      t[q] = m[q];
    }
    const double d[3] = {(double)m[1] * m[6] - (double)m[2] * m[5],
                         (double)m[2] * m[4] - (double)m[0] * m[6],
                         (double)m[0] * m[5] - (double)m[1] * m[4]};
    int ax = 0;
    for (int q = 1; q < 3; ++q)
      if (std::fabs(d[q]) > std::fabs(d[ax])) ax = q;
    const double n0 = std::sqrt((double)m[0] * m[0] + (double)m[1] * m[1] + (double)m[2] * m[2]);
    const double n1 = std::sqrt((double)m[4] * m[4] + (double)m[5] * m[5] + (double)m[6] * m[6]);
    if (!(std::fabs(d[ax]) > 1e-6 * n0 * n1))
      return fail(CT_ERR_UNSUPPORTED,
                  "ct_proj3d_views: matrix %d maps the volume onto a line (parallel rows)", v);
    t[8] = (float)ax;
    t[9] = t[10] = t[11] = 0.0f;
  }
  // AXIS0: rows of axis 0 only, shared by all views, each slice on one row
  // with to_next 0.5 (float32 arithmetic as the reference's; the zero terms
  // of Px_0 are exact)
  bool ax0 = order_out != nullptr;
  int32_t off = 0;
  for (int v = 0; ax0 && v < n_views; ++v) {
    const float* m = matrices + (size_t)v * 8;
    ax0 = m[1] == 0.0f && m[2] == 0.0f && m[4] == 0.0f && std::fabs(m[5]) <= 1.0f &&
          std::fabs(m[6]) <= 1.0f;
    // every view must put slice i on row i + off with to_next 0.5 (the
    // translation may differ between views by amounts below one ulp)
    for (int i = 0; ax0 && i < shape[0]; ++i) {
      const float x0 = (float)i + 0.5f;
      const float px = m[0] * x0 + m[3];  // two roundings; host code is not contracted
      const float left = px - 0.25f;
      const float tn = std::fmin(std::ceil(left) - left, 0.5f);
      const int ul = (int)std::floor(left);
      if (v == 0 && i == 0) off = ul;
      ax0 = tn == 0.5f && ul == i + off;
    }
  }
  *kind_out = ax0 ? CT_PROJ3D_AXIS0 : CT_PROJ3D_GENERAL;
  *row_offset_out = ax0 ? off : 0;
  if (ax0) {
    std::vector<std::pair<double, int>> key(CT_PROJ3D_ORDER);
    for (int v = 0; v < n_views; ++v) {
      const float* m = matrices + (size_t)v * 8;
      for (int p = 0; p < CT_PROJ3D_ORDER; ++p)
        key[p] = {(double)m[5] * (p / ct::kTileK) + (double)m[6] * (p % ct::kTileK), p};
      std::stable_sort(key.begin(), key.end(),
                       [](const std::pair<double, int>& a, const std::pair<double, int>& b) {
                         return a.first < b.first;
                       });
      for (int p = 0; p < CT_PROJ3D_ORDER; ++p)
        order_out[(size_t)v * CT_PROJ3D_ORDER + p] = (uint16_t)key[p].second;
    }
  }
  return CT_OK;
}

ct_status ct_proj3d_window_views(const float* views, int32_t n_views, const int32_t* shape, int32_t* taken_out) {
  if (!views || !shape || !taken_out) return ct::fail(CT_ERR_INVALID_ARG, "ct_proj3d_window_views: null argument");
  if (n_views <= 0) return ct::fail(CT_ERR_SHAPE, "ct_proj3d_window_views: n_views=%d", n_views);
  for (int q = 0; q < 3; ++q)
    if (shape[q] <= 0) return ct::fail(CT_ERR_SHAPE, "ct_proj3d_window_views: shape[%d]=%d", q, shape[q]);
  const int nwin = ct::gen_tiles(shape, n_views).nwin;
  for (int v = 0; v < n_views; ++v) {
    const float* m = views + (size_t)v * CT_VIEW3D_STRIDE;
    if (!(m[8] == 0.0f || m[8] == 1.0f || m[8] == 2.0f))
      return ct::fail(CT_ERR_INVALID_ARG, "ct_proj3d_window_views: view %d is not of ct_proj3d_views", v);
    taken_out[v] = !ct::gen_view_fits(m, shape[0], shape[1], shape[2], nwin) ? 0 : (m[8] == 2.0f ? 2 : 1);
  }
  return CT_OK;
}

ct_status ct_proj3d_workspace(const ct_geom3d* g, int32_t batch, size_t* fwd_bytes,
                              size_t* adj_bytes) {
  ct_status st = ct::proj3d_check(g, "ct_proj3d_workspace");
  if (st != CT_OK) return st;
  if (batch <= 0) return ct::fail(CT_ERR_INVALID_ARG, "ct_proj3d_workspace: batch=%d", batch);
  const ct::Proj3dPlan p = ct::proj3d_plan(g, batch);
  if (fwd_bytes) *fwd_bytes = p.fwd_ws_bytes;  // fit any schedule the autotuner may record
  if (adj_bytes) *adj_bytes = p.adj_ws_bytes;
  return CT_OK;
}

ct_status ct_proj3d_fwd(const ct_geom3d* g, const float* vol, float* proj, int32_t batch,
                        void* workspace, size_t workspace_bytes, ct_stream_t stream) {
  using namespace ct;
  ct_status st = proj3d_check(g, "ct_proj3d_fwd");
  if (st != CT_OK) return st;
  if (!vol || !proj) return fail(CT_ERR_INVALID_ARG, "ct_proj3d_fwd: null array");
  if (batch <= 0) return fail(CT_ERR_INVALID_ARG, "ct_proj3d_fwd: batch=%d", batch);
  Proj3dPlan p = proj3d_plan(g, batch);
  if (g->kind == CT_PROJ3D_AXIS0) {
    st = need_ws("ct_proj3d_fwd", p.fwd_least, workspace, workspace_bytes);
    if (st == CT_OK && workspace_bytes < p.fwd_bytes) {  // the groups that fit
      const size_t group = sizeof(float) * (size_t)g->n_views * g->det_shape[1] * p.Spad;
      Sched3d fewer;
      fewer.G = (int)std::max<size_t>(1, workspace_bytes / group);
      fewer.ns = p.nsplit;
      p = proj3d_plan_sched(g, fewer);
    }
  } else if (workspace_bytes < p.fwd_bytes - p.gen_turn || !aligned(workspace, 256)) {
    workspace = nullptr;  // GENERAL runs without scratch, slower
  } else if (workspace_bytes < p.fwd_bytes) {
    p.gen_turn = 0;  // views that march along axis 2 without their copy of the volume, slower
  }
  if (st != CT_OK) return st;
  st = proj3d_prepare(g, p);
  if (st != CT_OK) return st;
  const size_t vol_n = (size_t)g->shape[0] * g->shape[1] * g->shape[2];
  const size_t proj_n = (size_t)g->n_views * g->det_shape[0] * g->det_shape[1];
  for (int b = 0; b < batch; ++b) {
    st = proj3d_fwd_launch(g, p, vol + b * vol_n, proj + b * proj_n, workspace, as_stream(stream),
                           nullptr);
    if (st != CT_OK) return st;
  }
  return CT_OK;
}

ct_status ct_proj3d_adj(const ct_geom3d* g, const float* proj, float* vol, int32_t batch,
                        void* workspace, size_t workspace_bytes, ct_stream_t stream) {
  using namespace ct;
  ct_status st = proj3d_check(g, "ct_proj3d_adj");
  if (st != CT_OK) return st;
  if (!vol || !proj) return fail(CT_ERR_INVALID_ARG, "ct_proj3d_adj: null array");
  if (batch <= 0) return fail(CT_ERR_INVALID_ARG, "ct_proj3d_adj: batch=%d", batch);
  Proj3dPlan p = proj3d_plan(g, batch);
  st = need_ws("ct_proj3d_adj", p.adj_least, workspace, workspace_bytes);
  if (st != CT_OK) return st;
  if (p.nsplit > 1 && (!workspace || workspace_bytes < p.adj_bytes || !aligned(workspace, 256))) {
    // as many splits as the scratch given holds
    const size_t one = sizeof(float) * (size_t)g->shape[0] * g->shape[1] * g->shape[2];
    const bool use = workspace && aligned(workspace, 256);
    const int ns = std::max(1, (int)std::min<size_t>(p.nsplit, use ? workspace_bytes / one : 1));
    p.per_split = (g->n_views + ns - 1) / ns;
    p.nsplit = (g->n_views + p.per_split - 1) / p.per_split;
  }
  st = proj3d_prepare(g, p);
  if (st != CT_OK) return st;
  cudaStream_t s = as_stream(stream);
  const size_t vol_n = (size_t)g->shape[0] * g->shape[1] * g->shape[2];
  const size_t proj_n = (size_t)g->n_views * g->det_shape[0] * g->det_shape[1];
  float* part = static_cast<float*>(workspace);
  for (int b = 0; b < batch; ++b) {
    st = proj3d_adj_launch(g, p, proj + b * proj_n, vol + b * vol_n, part, s, nullptr);
    if (st != CT_OK) return st;
    if (p.nsplit > 1) {
      st = sum_splits(part, vol + b * vol_n, vol_n, p.nsplit, s);
      if (st != CT_OK) return st;
    }
  }
  return CT_OK;
}

ct_status ct_proj3d_autotune(const ct_geom3d* g, float* vol, float* proj, void* workspace,
                             size_t workspace_bytes, int32_t reps, ct_stream_t stream,
                             ct_proj3d_schedule* chosen) {
  using namespace ct;
  const char* who = "ct_proj3d_autotune";
  ct_status st = proj3d_check(g, who);
  if (st != CT_OK) return st;
  if (!vol || !proj) return fail(CT_ERR_INVALID_ARG, "%s: null array", who);
  if (reps <= 0) return fail(CT_ERR_INVALID_ARG, "%s: reps=%d", who, reps);
  cudaStream_t s = as_stream(stream);
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  st = cuda_check(cudaStreamIsCapturing(s, &cap), "stream capture query");
  if (st != CT_OK) return st;
  if (cap != cudaStreamCaptureStatusNone) return fail(CT_ERR_INVALID_ARG, "%s: cannot measure inside a stream capture", who);
  const Proj3dPlan p0 = proj3d_plan_sched(g, Sched3d{});
  // GENERAL tunes the adjoint alone
  const size_t need = g->kind == CT_PROJ3D_AXIS0 ? std::max(p0.fwd_ws_bytes, p0.adj_tune) : p0.adj_tune;
  st = need_ws(who, need, workspace, workspace_bytes);
  if (st != CT_OK) return st;
  st = proj3d_prepare(g, p0);
  if (st != CT_OK) return st;
  const size_t vol_n = (size_t)g->shape[0] * g->shape[1] * g->shape[2];
  float* part = static_cast<float*>(workspace);

  auto timed = [&](auto&& fn, float& us) {
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    ct_status r = cuda_check(cudaEventCreate(&e0), "autotune event");
    if (r == CT_OK) r = cuda_check(cudaEventCreate(&e1), "autotune event");
    if (r == CT_OK) r = fn();
    if (r == CT_OK) r = cuda_check(cudaEventRecord(e0, s), "autotune event record");
    for (int k = 0; k < reps && r == CT_OK; ++k) r = fn();
    if (r == CT_OK) r = cuda_check(cudaEventRecord(e1, s), "autotune event record");
    if (r == CT_OK) r = cuda_check(cudaEventSynchronize(e1), "autotune event sync");
    float ms = 0.0f;
    if (r == CT_OK) r = cuda_check(cudaEventElapsedTime(&ms, e0, e1), "autotune elapsed time");
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
    us = 1000.0f * ms / (float)reps;
    return r;
  };

  // Ties (within kTie of the fastest) go to the smaller count: both counts set
  // a summation order, so the choice should not flip between runs on noise.
  constexpr float kTie = 1.03f;
  auto pick = [&](const std::vector<std::pair<int, float>>& cand, int& val, float& us) {
    float fastest = cand.front().second;
    for (const auto& c : cand) fastest = std::min(fastest, c.second);
    for (const auto& c : cand)
      if (c.second <= kTie * fastest) {
        val = c.first;
        us = c.second;
        return;
      }
  };
  Sched3d best;
  float best_f = 0.0f, best_a = 0.0f;
  if (g->kind == CT_PROJ3D_AXIS0) {
    std::vector<std::pair<int, float>> cand;
    for (int G = 1; G <= std::min(kMaxGroups, p0.n_tiles); ++G) {
      const Proj3dPlan p = proj3d_plan_sched(g, Sched3d{G, 0});
      float us = 0.0f;
      st = timed([&] { return proj3d_fwd_launch(g, p, vol, proj, workspace, s, nullptr); }, us);
      if (st != CT_OK) return st;
      cand.emplace_back(p.G, us);
    }
    pick(cand, best.G, best_f);
  }
  {
    // 1, 2 and 4 view splits and the planner's own count, of those what the scratch
    // given holds (a call may always have had less than the counts of now need)
    const size_t scratch = workspace && aligned(workspace, 256) ? workspace_bytes : 0;
    auto time_adj = [&](int ns, float& us) {
      const Proj3dPlan p = proj3d_plan_sched(g, Sched3d{0, ns});
      return timed(
          [&] {
            ct_status r = proj3d_adj_launch(g, p, proj, vol, part, s, nullptr);
            if (r != CT_OK || p.nsplit == 1) return r;
            return sum_splits(part, vol, vol_n, p.nsplit, s);
          },
          us);
    };
    std::vector<std::pair<int, float>> cand;
    int last = 0;
    for (int ns = 1; ns <= kMaxSplits3d; ns *= 2) {
      const Proj3dPlan p = proj3d_plan_sched(g, Sched3d{0, ns});
      if (p.nsplit == last || p.adj_bytes > scratch) continue;
      last = p.nsplit;
      float us = 0.0f;
      st = time_adj(ns, us);
      if (st != CT_OK) return st;
      cand.emplace_back(p.nsplit, us);
    }
    // 64 x 96 x 80 x 48 views: 16.7 us with 4 splits, 15.7 us with the planner's 5, in some
    // runs 10 % apart over a few samples: a lead of 20 %
    st = tuned_splits(cand, 1.20f, p0.adj_bytes <= scratch, time_adj, best.ns, best_a);
    if (st != CT_OK) return st;
  }
  {
    std::lock_guard<std::mutex> lk(g_sched3_mu);
    g_sched3[sched3_key(g)] = Sched3dVal{best, best_f, best_a};
  }
  if (chosen) {
    const Proj3dPlan p = proj3d_plan_sched(g, best);
    chosen->tile_groups = g->kind == CT_PROJ3D_AXIS0 ? p.G : 0;
    chosen->adj_splits = p.nsplit;
    chosen->fwd_us = best_f;
    chosen->adj_us = best_a;
    chosen->tuned = 1;
  }
  return CT_OK;
}

ct_status ct_proj3d_schedule_get(const ct_geom3d* g, ct_proj3d_schedule* out) {
  using namespace ct;
  ct_status st = proj3d_check(g, "ct_proj3d_schedule_get");
  if (st != CT_OK) return st;
  if (!out) return fail(CT_ERR_INVALID_ARG, "ct_proj3d_schedule_get: null output");
  Sched3dVal v{};
  const bool tuned = sched3_lookup(g, v);
  const Proj3dPlan p = proj3d_plan_sched(g, tuned ? v.s : Sched3d{});
  out->tile_groups = g->kind == CT_PROJ3D_AXIS0 ? p.G : 0;
  out->adj_splits = p.nsplit;
  out->fwd_us = tuned ? v.fwd_us : 0.0f;
  out->adj_us = tuned ? v.adj_us : 0.0f;
  out->tuned = tuned ? 1 : 0;
  return CT_OK;
}

void ct_proj3d_schedule_clear(void) {
  std::lock_guard<std::mutex> lk(ct::g_sched3_mu);
  ct::g_sched3.clear();
}

// Diagnostic: returns (and clears) the 3D projector's internal check word.
int ct_proj3d_errflag(void) {
  int v = 0;
  if (cudaMemcpyFromSymbol(&v, ct::g_proj3d_err, sizeof(int)) != cudaSuccess) return -1;
  if (v != 0) {  // clear only a set word (no copy on the common path)
    const int zero = 0;
    cudaMemcpyToSymbol(ct::g_proj3d_err, &zero, sizeof(int));
  }
  return v;
}

}  // extern "C"
