// Elementwise kernels of the 3-D path around the FFT passes of vol3d_fft.cuh:
// the pyramid's low-pass gather (PrySDdec_onestep.m) and the adjoint of the
// edge replication (MarshalData.m:10-20).
//
// Half spectra are float2 arrays d0 x d1 x pitch holding d2/2 + 1 columns
// (ccsym 'c'); real volumes float arrays, axis 2 contiguous.
#include "fft_core.cuh"
#include "internal.h"
#include "launch.cuh"

namespace nsst {

// ---------------------------------------------------------------------------
// Elementwise volume kernels (grid-stride over one item, blockIdx.y = item)
// ---------------------------------------------------------------------------
#define V3_LOOP(total) \
  for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < (total); idx += (size_t)gridDim.x * blockDim.x)

// Window factor of one axis at parent index p (nr = FFT length of that axis,
// K = last window index, v = window values 0..K); full axes mirror at nr - p,
// the last (half) axis does not.  Returns -1 outside the window's support.
__device__ __forceinline__ float win_at(const float* __restrict__ v, int K, int nr, int p, bool half_axis) {
  if (p <= K) return v[p];
  if (!half_axis && p >= nr - K) return v[nr - p];
  return -1.0f;
}

// PrySDdec_onestep.m:82-108 on half spectra: Lp (small half spectrum, szLp =
// szF/D per axis, last axis szLp/2+1) from X.  Lp is gathered with the
// reference's write order: where the positive and the negative parts of a full
// axis land on the same small index, the negative part (written last by the
// subscripted assignment) wins.
__device__ __forceinline__ int small_to_parent(int s, int K, int nr, int nsmall, bool half_axis) {
  if (!half_axis && s >= nsmall - K) return s + nr - nsmall;  // negative part (written last)
  if (s <= K) return s;
  return -1;
}

__global__ void k_pyr_dec_lp(const float2* __restrict__ Xh, float2* __restrict__ Lp, size_t stride, int d1, int pitch,
                             int s0, int s1, int sh2, int spitch, PyrWin w, float invDN) {
  pdl_sync();
  const float2* X = Xh + blockIdx.y * stride;
  float2* L = Lp + blockIdx.y * stride;
  const size_t total = (size_t)s0 * s1 * sh2;
  V3_LOOP(total) {
    const int z = (int)(idx % sh2);
    const size_t r = idx / sh2;
    const int y = (int)(r % s1), x = (int)(r / s1);
    const int px = small_to_parent(x, w.K[0], w.nr[0], s0, false);
    const int py = small_to_parent(y, w.K[1], w.nr[1], s1, false);
    const int pz = small_to_parent(z, w.K[2], w.nr[2], 2 * (sh2 - 1), true);
    float2 out = make_float2(0.f, 0.f);
    if (px >= 0 && py >= 0 && pz >= 0) {
      const float lf = win_at(w.v0, w.K[0], w.nr[0], px, false) * win_at(w.v1, w.K[1], w.nr[1], py, false) *
                       win_at(w.v2, w.K[2], w.nr[2], pz, true);
      const float2 v = X[((size_t)px * d1 + py) * pitch + pz];
      out = make_float2(v.x * lf * invDN, v.y * lf * invDN);
    }
    L[r * spitch + z] = out;
  }
}

// One axis of the adjoint of the edge replication: out (e with e[axis] reduced to n)
// sums, along `axis`, the source planes that replicate each output plane
// (the last plane collects the padded ones).
__global__ void k_fold_axis(const float* __restrict__ g, size_t g_stride, float* __restrict__ out, size_t o_stride,
                            int e0, int e1, int e2, int axis, int n) {
  pdl_sync();
  const float* src = g + blockIdx.y * g_stride;
  float* dst = out + blockIdx.y * o_stride;
  const int f0 = axis == 0 ? n : e0, f1 = axis == 1 ? n : e1, f2 = axis == 2 ? n : e2;
  const int ext = axis == 0 ? e0 : (axis == 1 ? e1 : e2);
  const size_t step = axis == 0 ? (size_t)e1 * e2 : (axis == 1 ? (size_t)e2 : 1);
  const size_t total = (size_t)f0 * f1 * f2;
  V3_LOOP(total) {
    const int z = (int)(idx % f2);
    const size_t r = idx / f2;
    const int y = (int)(r % f1), x = (int)(r / f1);
    const int c = axis == 0 ? x : (axis == 1 ? y : z);
    const float* s0 = src + ((size_t)x * e1 + y) * e2 + z;
    float sum = s0[0];
    if (c == n - 1)
      for (int k = 1; k < ext - c; k++) sum += s0[k * step];
    dst[idx] = sum;
  }
}

static dim3 v3grid(size_t total, int nitems) {
  return dim3((unsigned)std::min<size_t>((total + 255) / 256, 2048), nitems);
}

cudaError_t launch_pyr_dec_lp(const float2* Xh, float2* Lp, size_t stride, int n, int d1, int pitch, int s0, int s1,
                              int s2, const PyrWin& w, float invDN, cudaStream_t st) {
  const int sh2 = s2 / 2 + 1;
  count_launch();
  launch_pdl(k_pyr_dec_lp, v3grid((size_t)s0 * s1 * sh2, n), 256, 0, st, Xh, Lp, stride, d1, pitch, s0, s1, sh2,
                                                                 v3_pitch(sh2), w, invDN);
  return cudaGetLastError();
}
// Adjoint of the edge replication: g (d0 x d1 x d2) -> out (n0 x n1 x n2), one
// axis at a time through scratch (>= d0 d1 n2 + d0 n1 n2 floats per item).
cudaError_t launch_fold_edge(const float* g, size_t g_stride, float* out, size_t o_stride, float* scratch,
                             size_t s_stride, int n, int n0, int n1, int n2, int d0, int d1, int d2, cudaStream_t st) {
  float* t1 = scratch;                           // d0 x d1 x n2
  float* t2 = scratch + (size_t)d0 * d1 * n2;    // d0 x n1 x n2
  count_launch(3);
  launch_pdl(k_fold_axis, v3grid((size_t)d0 * d1 * n2, n), 256, 0, st, g, g_stride, t1, s_stride, d0, d1, d2, 2, n2);
  launch_pdl(k_fold_axis, v3grid((size_t)d0 * n1 * n2, n), 256, 0, st, t1, s_stride, t2, s_stride, d0, d1, n2, 1, n1);
  launch_pdl(k_fold_axis, v3grid((size_t)n0 * n1 * n2, n), 256, 0, st, t2, s_stride, out, o_stride, d0, n1, n2, 0, n0);
  return cudaGetLastError();
}

}  // namespace nsst
