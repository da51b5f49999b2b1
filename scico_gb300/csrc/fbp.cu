// Ramp filter of XRayTransform2D.fbp (scico/linop/xray/_xray2d.py:158-221).
//
// Each sinogram row y[0..N) is convolved with the ramp filter of Kak &
// Slaney eq. (61) at tau = 1 -- h(0) = 1/4, h(n) = -1/(pi^2 n^2) for odd n,
// 0 for even n != 0, taps n = -(N-1)/2 .. N-1-(N-1)/2 -- and cropped to the N
// samples aligned with the input:  out[i] = sum_n h(n) y[i - n].  The
// reference evaluates this linear convolution with zero-padded FFTs of
// length 2N-1; here it is summed directly (only the centre and odd taps are
// non-zero), which is exact up to float32 rounding and deterministic.
//
// k_fbp_rows: a CTA filters one row.  An output of one parity meets samples of
// the other parity only, so the row is split by parity in shared memory, and a
// thread takes kR = 8 outputs of its parity, consecutive there: their inputs
// slide by one sample a tap, so eight taps on both sides cost 16 loads and two
// tap loads for 128 multiply-adds.  Zeros around the row stand for the tests
// of its ends.  A row of 9 floats per 8 samples keeps the threads (8 samples
// apart) on different banks.  Bound by FFMA issue and, at a few hundred rows,
// by having only some 7 warps an SM.  fbp of 501^2 from 360 rows of 709: 98 us
// a pass with one output and one pair of tests per tap, the taps in float64
// (43.6 us of it this kernel) and the mask in three elementwise kernels; 55 us now.
#include <math.h>

#include <algorithm>

#include "common.cuh"

namespace {

constexpr int kR = 8;               // outputs per thread, taps per step
constexpr int kFbpMaxThreads = 512;

// Position of sample k of a parity array (k + base >= 0, base a multiple of 8).
__host__ __device__ constexpr int fbp_pos(int kb) { return kb + (kb >> 3); }

struct FbpPlan {
  int N;
  int taps;        // odd taps m = 1, 3, .. on both sides: min(hi, off)
  int extra;       // 1 when the left side has one more odd tap (hi odd, hi > off)
  int groups;      // threads per parity: groups of kR outputs
  int base;        // samples of zeros before a parity array (a multiple of 8)
  int len;         // floats of one parity array in shared memory
};

// -1 / (pi^2 m^2) rounded to float32, by float pairs: 1/pi^2 and m^2 as two
// floats each, one correction of the quotient by its remainder (exact in an
// FMA).  The same floats as the float64 quotient for every odd m below 25600;
// float64 divisions, at this GPU's rate for them, took as long as the sums.
__device__ __forceinline__ float ramp_tap(int m) {
  const float ch = 0.10132118f, cl = 4.9729154e-10f;
  const unsigned mm = (unsigned)m * (unsigned)m;
  const float mh = (float)mm, ml = (float)(int)(mm - (unsigned)mh);
  const float q = __fdiv_rn(ch, mh);
  const float r = __fmaf_rn(-q, ml, __fadd_rn(__fmaf_rn(-q, mh, ch), cl));
  return -__fadd_rn(q, __fdiv_rn(r, mh));
}

__global__ void __launch_bounds__(kFbpMaxThreads) k_fbp_rows(const float* __restrict__ y, float* __restrict__ out,
                                                             const FbpPlan p) {
  extern __shared__ __align__(16) float sm[];
  // S[0]: odd samples, S[0][k] = y[2k + 1], read by even outputs; S[1]: even
  // samples one further, S[1][k] = y[2k + 2], read by odd outputs.  Output k of
  // either parity then meets S[k - 1 - t] and S[k + t] with tap m = 2t + 1.
  float* taps = sm + 2 * p.len;
  const float* src = y + (size_t)blockIdx.x * p.N;
  for (int e = threadIdx.x; e < 2 * p.len; e += blockDim.x) sm[e] = 0.0f;
  for (int t = threadIdx.x; t < p.taps + p.extra; t += blockDim.x) taps[t] = ramp_tap(2 * t + 1);
  __syncthreads();
  for (int i = threadIdx.x; i < p.N; i += blockDim.x) {
    const int odd = i & 1, k = odd ? i >> 1 : (i >> 1) - 1;
    // positions hold k + 1, so that a thread's left neighbours start a row
    sm[(odd ? 0 : p.len) + fbp_pos(k + 1 + p.base)] = src[i];
  }
  __syncthreads();
  for (int t = threadIdx.x; t < 2 * p.groups; t += blockDim.x) {
    const int par = t >= p.groups ? 1 : 0, g = t - par * p.groups;
    const float* S = sm + par * p.len;
    const float* O = sm + (1 - par) * p.len;  // the outputs' own samples
    const int row = 9 * (g + p.base / 8);     // row of k + 1 = 8g

    float acc[kR];
#pragma unroll
    for (int j = 0; j < kR; ++j) {
      // y[2k + par], k = 8g + j: odd sample k of S[0], or even sample k - 1 of S[1]
      const int kk = 8 * g + j + p.base + (par ? 1 : 0);
      acc[j] = 0.25f * O[fbp_pos(kk)];
    }
    float lc[kR], rc[kR], ln[kR], rn[kR];
#pragma unroll
    for (int u = 0; u < kR; ++u) {
      lc[u] = S[row + u];                          // k = 8g - 1 + u
      rc[u] = S[row + (u < 7 ? u + 1 : u + 2)];    // k = 8g + u
    }
    int t0 = 0;
    for (; t0 + kR <= p.taps; t0 += kR) {
      const float* L = S + row - 9 * (t0 / 8 + 1);
      const float* R = S + row + 9 * (t0 / 8 + 1);
#pragma unroll
      for (int u = 0; u < kR; ++u) {
        ln[u] = L[u];
        rn[u] = R[u < 7 ? u + 1 : u + 2];
      }
      const float4 ha = *reinterpret_cast<const float4*>(taps + t0), hb = *reinterpret_cast<const float4*>(taps + t0 + 4);
      const float h[kR] = {ha.x, ha.y, ha.z, ha.w, hb.x, hb.y, hb.z, hb.w};
#pragma unroll
      for (int s = 0; s < kR; ++s)
#pragma unroll
        for (int j = 0; j < kR; ++j) {
          acc[j] = fmaf(h[s], j >= s ? lc[j - s] : ln[kR + j - s], acc[j]);
          acc[j] = fmaf(h[s], j + s < kR ? rc[j + s] : rn[j + s - kR], acc[j]);
        }
#pragma unroll
      for (int u = 0; u < kR; ++u) {
        lc[u] = ln[u];
        rc[u] = rn[u];
      }
    }
    for (; t0 < p.taps + p.extra; ++t0) {
      const float h = taps[t0];
      const bool right = t0 < p.taps;
#pragma unroll
      for (int j = 0; j < kR; ++j) {
        acc[j] = fmaf(h, S[fbp_pos(8 * g + j - t0 + p.base)], acc[j]);
        if (right) acc[j] = fmaf(h, S[fbp_pos(8 * g + j + t0 + 1 + p.base)], acc[j]);
      }
    }
    float* o = out + (size_t)blockIdx.x * p.N;
#pragma unroll
    for (int j = 0; j < kR; ++j) {
      const int i = 2 * (8 * g + j) + par;
      if (i < p.N) o[i] = acc[j];
    }
  }
}

FbpPlan fbp_plan(int N) {
  FbpPlan p;
  p.N = N;
  const int off = (N - 1) / 2, hi = N - 1 - off;  // largest offsets left (y[i + m]) and right (y[i - m])
  p.taps = (off + 1) / 2;                         // odd m <= off <= hi
  p.extra = (hi + 1) / 2 - p.taps;                // y[i - m] only, m = hi
  const int half = (N + 1) / 2;
  p.groups = (half + kR - 1) / kR;
  const int reach = (p.taps + p.extra + 2 * kR) / 8 * 8 + 8;
  p.base = reach;
  p.len = (fbp_pos(p.groups * kR + 2 * reach + kR) + 8) / 4 * 4;
  return p;
}

size_t fbp_smem(const FbpPlan& p) { return sizeof(float) * (2 * (size_t)p.len + p.taps + p.extra); }

// Rows too long for the above: the row and its taps alone in shared memory, a
// test of the row's ends for every product.
__global__ void __launch_bounds__(256) k_fbp_long(const float* __restrict__ y, float* __restrict__ out, int N) {
  extern __shared__ __align__(16) float sm[];
  float* row = sm;
  float* taps = sm + N;
  const float* src = y + (size_t)blockIdx.x * N;
  for (int i = threadIdx.x; i < N; i += 256) {
    row[i] = src[i];
    taps[i] = (i & 1) ? ramp_tap(i) : 0.0f;
  }
  __syncthreads();
  const int off = (N - 1) / 2, hi = N - 1 - off;
  for (int i = threadIdx.x; i < N; i += 256) {
    float acc = 0.25f * row[i];
    for (int m = 1; m <= hi; m += 2) {  // hi >= off
      const float t = taps[m];
      if (i - m >= 0) acc = fmaf(t, row[i - m], acc);
      if (m <= off && i + m < N) acc = fmaf(t, row[i + m], acc);
    }
    out[(size_t)blockIdx.x * N + i] = acc;
  }
}

}  // namespace

extern "C" {

ct_status ct_fbp_filter(const float* sino, float* out, int32_t n_rows, int32_t det_count,
                        ct_stream_t stream) {
  if (!sino || !out) return ct::fail(CT_ERR_INVALID_ARG, "ct_fbp_filter: null array");
  if (n_rows <= 0 || det_count <= 0)
    return ct::fail(CT_ERR_SHAPE, "ct_fbp_filter: n_rows=%d det_count=%d", n_rows, det_count);
  // the longest row that the shared-memory copy of it and its taps ever allowed
  if (2 * sizeof(float) * (size_t)det_count > 200u * 1024u)
    return ct::fail(CT_ERR_UNSUPPORTED, "ct_fbp_filter: det_count=%d above %d", det_count,
                    (int)(100u * 1024u / sizeof(float)));
  const FbpPlan p = fbp_plan(det_count);
  const size_t smem = fbp_smem(p);
  if (smem > 200u * 1024u) {  // rows above some 20,000 samples: no room for the zeros around them
    const size_t plain = 2 * sizeof(float) * (size_t)det_count;
    ct_status st = ct::cuda_check(
        cudaFuncSetAttribute(k_fbp_long, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)plain),
        "k_fbp_long smem attribute");
    if (st != CT_OK) return st;
    k_fbp_long<<<n_rows, 256, plain, ct::as_stream(stream)>>>(sino, out, det_count);
    return ct::launch_check("k_fbp_long");
  }
  if (smem > 48u * 1024u) {
    ct_status st = ct::cuda_check(
        cudaFuncSetAttribute(k_fbp_rows, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
        "k_fbp_rows smem attribute");
    if (st != CT_OK) return st;
  }
  const int threads = std::min(kFbpMaxThreads, (2 * p.groups + 31) / 32 * 32);
  k_fbp_rows<<<n_rows, threads, smem, ct::as_stream(stream)>>>(sino, out, p);
  return ct::launch_check("k_fbp_rows");
}

}  // extern "C"
