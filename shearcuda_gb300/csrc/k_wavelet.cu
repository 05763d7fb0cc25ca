// Undecimated (redundant) 2-D wavelet transform and the image-separation
// helpers, for n images per launch.
//
// mrdwt (shearcuda/src/mrdwt_r.h:104-209) filters each level's lowpass along
// rows and then columns with the level's dilation sf = 2^(l-1), periodically;
// mirdwt (mirdwt_r.h:115-219) undoes it columns first.  The filters are
// separable, so a level here runs columns first in both directions, and as one
// kernel: a CTA owns TH rows of one row phase (rows p + sf i of a level only
// meet rows of their own phase) at the full width, filters them down the
// columns from global memory with the taps sliding over registers, keeps the
// two results in shared memory and filters those along the rows.  So a level
// moves each plane once (analysis 1 read, 4 writes; synthesis 4 reads, 1
// write) where separate column and row kernels moved two more, and a column
// step reads (TH + lh - 1) / TH rows per output row instead of lh.
//   analysis   (C_lo, C_hi) = columns of cur; LL, HL = rows of C_lo; LH, HH = rows of C_hi
//   synthesis  x1 = columns of (LL, LH), xh = columns of (HL, HH); x = rows of (x1, xh)
// A level reads its input while other CTAs write its output, so the two must
// not share a buffer.  An analysis level whose input lies in its own output
// planes runs as two kernels instead (launch_rdwt_level_in_place).
#include "internal.h"
#include "launch.cuh"

namespace nsst {

constexpr int kWvThreads = 256;
constexpr int kWvMaxW = 8192;

__device__ __forceinline__ float hard_keep(float v, float t) { return fabsf(v) > t ? v : 0.0f; }
__device__ __forceinline__ float soft(float v, float t) {
  const float r = fabsf(v) - t;  // SoftThresh.m: sign(y) (|y| - t)_+
  return r > 0.0f ? copysignf(r, v) : 0.0f;
}

// LH: the filter length (0: t.lh); TH: rows per CTA; T: its threads; PARTS: of
// `tile`'s columns, not of the whole row.
// Grid: x = row phase (fastest) and group of TH rows of the phase, y = item, z =
// part of the row.
// Taps are applied in ascending order whatever the form.  Two results that take
// the same taps or the same sample share packed FP32 FMAs, which round as two
// single ones.  Bound by issue (71 % of it in the analysis and 50 % in the synthesis
// at 32 images of 256 x 256; HBM 8 and 23 %, the planes stay in L2): 64 registers, so
// that four CTAs share an SM, took the four Symmlet-4 levels there from 93 to 66 us
// (analysis) and 105 to 78 us (synthesis); six CTAs (spills) 87 and 84.  Separate
// column and row kernels measured 133 and 150 us.  With dependent launches a level
// takes 12 and 16 us.
// Columns of a CTA: `out` of the results and `in` of what the row taps reach from
// there, from their first column on (analysis) or up to their last (synthesis);
// both the whole row, or in = out + (lh - 1) sf.
struct WvTile {
  int out, in;
};
__device__ __forceinline__ float2 twice(float v) { return make_float2(v, v); }

template <int LH, int TH, int T, bool PARTS>
__global__ void __launch_bounds__(T, 1024 / T)
    k_rdwt_fwd(const float* __restrict__ cur, size_t s_cur, float* __restrict__ yl, size_t s_yl,
               float* __restrict__ yh, size_t s_yh, int H, int W, int sf, WvTile tile,
               const __grid_constant__ WvTaps t, const float* __restrict__ thr) {
  pdl_sync();
  extern __shared__ float2 sm[];  // [row][column from c0 on] (C_lo, C_hi)
  const int ph = blockIdx.x % sf, i0 = blockIdx.x / sf * TH, item = blockIdx.y, Hp = H / sf;
  const int c0 = PARTS ? blockIdx.z * tile.out : 0, SW = PARTS ? tile.in : W, n_out = PARTS ? min(tile.out, W - c0) : W;
  const size_t HW = (size_t)H * W, rs = (size_t)sf * W;
  const float* x = cur + item * s_cur + (size_t)ph * W;
  for (int s = threadIdx.x; s < SW; s += T) {
    const int c = PARTS && c0 + s >= W ? c0 + s - W : c0 + s;
    float2 lh[TH];  // (lo, hi)
#pragma unroll
    for (int k = 0; k < TH; k++) lh[k] = twice(0.0f);
    if constexpr (LH > 0) {
      int i = i0;
#pragma unroll
      for (int m = 0; m < TH + LH - 1; m++) {
        const float2 v = twice(__ldg(x + i * rs + c));
        if (++i == Hp) i = 0;
#pragma unroll
        for (int k = 0; k < TH; k++)
          if (m - k >= 0 && m - k < LH) lh[k] = __ffma2_rn(make_float2(t.a[m - k], t.b[m - k]), v, lh[k]);
      }
    } else {  // the rows under tap j, rotated by one per tap
      float v[TH];
      int i = i0;
#pragma unroll
      for (int k = 0; k < TH - 1; k++) {
        v[k] = __ldg(x + i * rs + c);
        if (++i == Hp) i = 0;
      }
#pragma unroll TH
      for (int j = 0; j < t.lh; j++) {
        v[TH - 1] = __ldg(x + i * rs + c);
        if (++i == Hp) i = 0;
        const float2 ab = make_float2(t.a[j], t.b[j]);
#pragma unroll
        for (int k = 0; k < TH; k++) lh[k] = __ffma2_rn(ab, twice(v[k]), lh[k]);
#pragma unroll
        for (int k = 0; k < TH - 1; k++) v[k] = v[k + 1];
      }
    }
#pragma unroll
    for (int k = 0; k < TH; k++) sm[k * SW + s] = lh[k];
  }
  __syncthreads();
  const float th = thr ? thr[item] : -1.0f;
  const int lh_n = LH > 0 ? LH : t.lh;
  for (int s = threadIdx.x; s < n_out; s += T) {
    float2 lo[TH], hi[TH];  // (LL, LH), (HL, HH)
#pragma unroll
    for (int k = 0; k < TH; k++) lo[k] = hi[k] = twice(0.0f);
    int ss = s;
#pragma unroll
    for (int j = 0; j < lh_n; j++) {
      const float2 a = twice(t.a[j]), b = twice(t.b[j]);
#pragma unroll
      for (int k = 0; k < TH; k++) {
        const float2 v = sm[k * SW + ss];
        lo[k] = __ffma2_rn(a, v, lo[k]);
        hi[k] = __ffma2_rn(b, v, hi[k]);
      }
      ss += sf;
      if (!PARTS && ss >= W) ss -= W;
    }
#pragma unroll
    for (int k = 0; k < TH; k++) {
      if (i0 + k >= Hp) break;
      const size_t o = (size_t)(ph + (i0 + k) * sf) * W + c0 + s;
      float lv = lo[k].y, hl = hi[k].x, hh = hi[k].y;
      if (th >= 0.0f) {
        hl = hard_keep(hl, th);
        lv = hard_keep(lv, th);
        hh = hard_keep(hh, th);
      }
      yl[item * s_yl + o] = lo[k].x;
      float* d = yh + item * s_yh + o;
      d[0] = lv;
      d[HW] = hl;
      d[2 * HW] = hh;
    }
  }
}

// An analysis level in place, columns and then rows: the column kernel leaves
// (C_lo, C_hi) in the level's HL and LH planes, and the row kernel, one CTA per
// row, holds the row in shared memory while it writes LL (to yl, which may be
// the level's input), LH, HL and HH.  The taps and their order are
// k_rdwt_fwd's, so both forms give the same bits.  Two passes more over memory:
// 24 us a level at 32 images of 256 x 256 and 8 taps, against 12.
__global__ void __launch_bounds__(256) k_rdwt_cols_fwd(const float* __restrict__ cur, size_t s_cur,
                                                       float* __restrict__ yh, size_t s_yh, int H, int W, int sf,
                                                       const __grid_constant__ WvTaps t) {
  pdl_sync();
  const int r = blockIdx.x * 8 + threadIdx.y, c = blockIdx.y * 32 + threadIdx.x, item = blockIdx.z;
  if (c >= W || r >= H) return;
  const float* x = cur + item * s_cur + c;
  float2 acc = twice(0.0f);  // (lo, hi)
  int rr = r;
  for (int j = 0; j < t.lh; j++) {
    acc = __ffma2_rn(make_float2(t.a[j], t.b[j]), twice(__ldg(x + (size_t)rr * W)), acc);
    rr += sf;
    if (rr >= H) rr -= H;
  }
  float* out = yh + item * s_yh + (size_t)r * W + c;
  out[(size_t)H * W] = acc.x;
  out[0] = acc.y;
}

__global__ void __launch_bounds__(kWvThreads) k_rdwt_rows_fwd(float* yl, size_t s_yl, float* yh, size_t s_yh, int H,
                                                              int W, int sf, const __grid_constant__ WvTaps t,
                                                              const float* __restrict__ thr) {
  pdl_sync();
  extern __shared__ float2 sm[];  // [column] (C_lo, C_hi)
  const int r = blockIdx.x, item = blockIdx.y;
  const size_t HW = (size_t)H * W;
  float* p = yh + item * s_yh + (size_t)r * W;
  for (int c = threadIdx.x; c < W; c += kWvThreads) sm[c] = make_float2(p[HW + c], p[c]);
  __syncthreads();
  const float th = thr ? thr[item] : -1.0f;
  float* l = yl + item * s_yl + (size_t)r * W;
  for (int c = threadIdx.x; c < W; c += kWvThreads) {
    float2 lo = twice(0.0f), hi = twice(0.0f);  // (LL, LH), (HL, HH)
    int cc = c;
    for (int j = 0; j < t.lh; j++) {
      const float2 v = sm[cc];
      lo = __ffma2_rn(twice(t.a[j]), v, lo);
      hi = __ffma2_rn(twice(t.b[j]), v, hi);
      cc += sf;
      if (cc >= W) cc -= W;
    }
    float lh = lo.y, hl = hi.x, hh = hi.y;
    if (th >= 0.0f) {
      hl = hard_keep(hl, th);
      lh = hard_keep(lh, th);
      hh = hard_keep(hh, th);
    }
    l[c] = lo.x;
    p[c] = lh;
    p[HW + c] = hl;
    p[2 * HW + c] = hh;
  }
}

template <int LH, int TH, int T, bool PARTS>
__global__ void __launch_bounds__(T, 1024 / T)
    k_rdwt_inv(const float* __restrict__ ll, size_t s_ll, const float* __restrict__ yh, size_t s_yh,
               float* __restrict__ out, size_t s_out, int H, int W, int sf, WvTile tile,
               const __grid_constant__ WvTaps t) {
  pdl_sync();
  extern __shared__ float2 sm[];
  const int ph = blockIdx.x % sf, i0 = blockIdx.x / sf * TH, item = blockIdx.y, Hp = H / sf;
  const int c0 = PARTS ? blockIdx.z * tile.out : 0, SW = PARTS ? tile.in : W, n_out = PARTS ? min(tile.out, W - c0) : W;
  const int off = PARTS ? tile.in - tile.out : 0;
  float2 *s1 = sm, *sh = sm + TH / 2 * SW;  // [row pair][column from c0 - off on]: x1, xh of rows 2 q and 2 q + 1
  const size_t HW = (size_t)H * W, rs = (size_t)sf * W;
  const float* p = ll + item * s_ll + (size_t)ph * W;
  const float* q = yh + item * s_yh + (size_t)ph * W;
  for (int s = threadIdx.x; s < SW; s += T) {
    int c = c0 - off + s;
    if (PARTS && c < 0) c += W;
    if (PARTS && c >= W) c -= W;
    float2 x[TH];  // (x1, xh)
#pragma unroll
    for (int k = 0; k < TH; k++) x[k] = twice(0.0f);
    if constexpr (LH > 0) {
      int i = (i0 + TH - 1) % Hp;  // input row of output row i0 + k at tap t: i0 + k - t
#pragma unroll
      for (int m = 0; m < TH + LH - 1; m++) {
        const size_t o = i * rs + c;
        const float2 v = make_float2(__ldg(p + o), __ldg(q + HW + o));           // LL, HL
        const float2 w = make_float2(__ldg(q + o), __ldg(q + 2 * HW + o));       // LH, HH
        if (--i < 0) i = Hp - 1;
#pragma unroll
        for (int k = 0; k < TH; k++) {
          const int tt = m - (TH - 1) + k;
          if (tt >= 0 && tt < LH) x[k] = __ffma2_rn(twice(t.b[tt]), w, __ffma2_rn(twice(t.a[tt]), v, x[k]));
        }
      }
    } else {  // the rows under tap tt, rotated by one per tap
      float2 v[TH], w[TH];  // (LL, HL), (LH, HH)
      auto row = [&](int k, int i) {
        const size_t o = i * rs + c;
        v[k] = make_float2(__ldg(p + o), __ldg(q + HW + o));
        w[k] = make_float2(__ldg(q + o), __ldg(q + 2 * HW + o));
      };
      int i = i0;
#pragma unroll
      for (int k = 1; k < TH; k++) {
        if (++i == Hp) i = 0;
        row(k, i);
      }
      i = i0;
#pragma unroll TH
      for (int tt = 0; tt < t.lh; tt++) {
        row(0, i);
        if (--i < 0) i = Hp - 1;
        const float2 a = twice(t.a[tt]), b = twice(t.b[tt]);
#pragma unroll
        for (int k = 0; k < TH; k++) x[k] = __ffma2_rn(b, w[k], __ffma2_rn(a, v[k], x[k]));
#pragma unroll
        for (int k = TH - 1; k > 0; k--) v[k] = v[k - 1], w[k] = w[k - 1];
      }
    }
#pragma unroll
    for (int k = 0; k < TH; k += 2) {
      s1[k / 2 * SW + s] = make_float2(x[k].x, x[k + 1].x);
      sh[k / 2 * SW + s] = make_float2(x[k].y, x[k + 1].y);
    }
  }
  __syncthreads();
  const int lh_n = LH > 0 ? LH : t.lh;
  for (int s = threadIdx.x; s < n_out; s += T) {
    float2 acc[TH / 2];
#pragma unroll
    for (int k = 0; k < TH / 2; k++) acc[k] = twice(0.0f);
    int ss = s + off;
#pragma unroll
    for (int j = 0; j < lh_n; j++) {
      const float2 a = twice(t.a[j]), b = twice(t.b[j]);
#pragma unroll
      for (int k = 0; k < TH / 2; k++) acc[k] = __ffma2_rn(b, sh[k * SW + ss], __ffma2_rn(a, s1[k * SW + ss], acc[k]));
      ss -= sf;
      if (!PARTS && ss < 0) ss += W;
    }
#pragma unroll
    for (int k = 0; k < TH; k++)
      if (i0 + k < Hp)
        out[item * s_out + (size_t)(ph + (i0 + k) * sf) * W + c0 + s] = k & 1 ? acc[k / 2].y : acc[k / 2].x;
  }
}

// ----------------------------------------------------- TV correction (Haar)
// y = mirdwt(LL, soft(yh, gamma)) with (LL, yh) = mrdwt(x) at one level and
// the Haar pair (analysis lo = a x[c] + a x[c+1], hi = a x[c] - a x[c+1];
// synthesis x = a/2 (lo[c] + lo[c-1]) + a/2 (hi[c] - hi[c-1]), a = 1/sqrt 2):
// an output pixel reads the 3 x 3 neighbourhood x[r-1..r+1][c-1..c+1].
//
// A warp walks kTvRows rows of 31 output columns (lane 0 holds the column to
// their left): each lane computes its column's coefficients once per row, the
// row above's stay in registers and the left column's column synthesis comes
// from the next lane.  With one output per thread the four coefficient sets of
// every output, their soft thresholds and the tile's periodic indices were the
// time (instruction issue; 32 x 256^2: 26 -> 11 us).
constexpr int kTvRows = 8, kTvWarps = 8, kTvCols = 31;
__global__ void __launch_bounds__(32 * kTvWarps)
    k_tv_haar(const float* __restrict__ x, float* __restrict__ y, size_t stride, int H, int W, WvTaps ta, WvTaps ts,
              float gamma) {
  pdl_sync();
  const int lane = threadIdx.x, c0 = blockIdx.x * kTvCols, item = blockIdx.z;
  const int r0 = (blockIdx.y * kTvWarps + threadIdx.y) * kTvRows;
  if (r0 >= H) return;  // whole warps
  const int c = (c0 + lane - 1 + W) % W, c1 = c + 1 == W ? 0 : c + 1;  // periodic
  const float* xi = x + item * stride;
  auto row = [&](int r, float& l, float& h) {  // rows first (mrdwt_r.h:157-177)
    const float u = __ldg(xi + (size_t)r * W + c), v = __ldg(xi + (size_t)r * W + c1);
    l = ta.a[0] * u + ta.a[1] * v;
    h = ta.b[0] * u + ta.b[1] * v;
  };
  int r = r0 ? r0 - 1 : H - 1;
  float l0, h0;
  row(r, l0, h0);
  float LLp = 0.f, LHp = 0.f, HLp = 0.f, HHp = 0.f;  // the row above's coefficients
#pragma unroll
  for (int k = -1; k < kTvRows; k++) {
    if (r0 + k >= H) break;
    r = r + 1 == H ? 0 : r + 1;
    float l1, h1;
    row(r, l1, h1);
    // then columns (:180-206)
    const float LL = ta.a[0] * l0 + ta.a[1] * l1;
    const float LH = soft(ta.b[0] * l0 + ta.b[1] * l1, gamma);
    const float HL = soft(ta.a[0] * h0 + ta.a[1] * h1, gamma);
    const float HH = soft(ta.b[0] * h0 + ta.b[1] * h1, gamma);
    if (k >= 0) {
      // columns (mirdwt_r.h:163-189): x1 = a LL + b LH, xh = a HL + b HH over rows r, r-1
      const float x1 = ts.a[0] * LL + ts.b[0] * LH + ts.a[1] * LLp + ts.b[1] * LHp;
      const float xh = ts.a[0] * HL + ts.b[0] * HH + ts.a[1] * HLp + ts.b[1] * HHp;
      // rows (:192-213) over columns c, c-1
      const float x1l = __shfl_up_sync(0xffffffffu, x1, 1), xhl = __shfl_up_sync(0xffffffffu, xh, 1);
      if (lane > 0 && c0 + lane - 1 < W)
        y[item * stride + (size_t)(r0 + k) * W + c] = ts.a[0] * x1 + ts.b[0] * xh + ts.a[1] * x1l + ts.b[1] * xhl;
    }
    l0 = l1, h0 = h1;
    LLp = LL, LHp = LH, HLp = HL, HHp = HH;
  }
}

// ---------------------------------------------------- decimated HH (FP64)
struct DTaps {
  double b[kMaxQmf];
  int lh;
};
__global__ void __launch_bounds__(256) k_dwt_hh(const float* __restrict__ xb, size_t stride, int H, int W, DTaps t,
                                                double* __restrict__ hhb) {
  pdl_sync();
  const int l = blockIdx.x * 32 + threadIdx.x, k = blockIdx.y * 8 + threadIdx.y;
  if (l >= W / 2 || k >= H / 2) return;
  const float* x = xb + blockIdx.z * stride;
  double* hh = hhb + (size_t)blockIdx.z * (H / 2) * (W / 2);
  double acc = 0.0;
  int rr = 2 * k;
  for (int i = 0; i < t.lh; i++) {
    double row = 0.0;
    int cc = 2 * l;
    const float* xr = x + (size_t)rr * W;
    for (int j = 0; j < t.lh; j++) {
      row = fma(t.b[j], (double)__ldg(xr + cc), row);
      if (++cc >= W) cc -= W;
    }
    acc = fma(t.b[i], row, acc);
    if (++rr >= H) rr -= H;
  }
  hh[(size_t)k * (W / 2) + l] = acc;
}

// ------------------------------------------------------------- separation
__global__ void k_sep_residual(const float* __restrict__ img, const float* __restrict__ p1,
                               const float* __restrict__ p2, float* __restrict__ ra1, float* __restrict__ ra2,
                               size_t n) {
  pdl_sync();
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const float a = p1[i], b = p2[i];
    const float r = (img[i] - a) - b;  // GPUminus twice (separate.m:146-148)
    ra1[i] = a + r;
    ra2[i] = b + r;
  }
}

// ----------------------------------------------------------------- launchers
bool rdwt_width_supported(int W) { return W >= 2 && W <= kWvMaxW; }

constexpr size_t kWvTwoCtas = 110 * 1024;  // shared memory of a CTA of which two fit an SM
constexpr int kWvLong = kWvTwoCtas / (4 * sizeof(float2));  // longest row of which four fit there
static int fill() { return 2 * sm_count(); }                // CTAs that fill the GPU

// Columns per CTA.  The whole row, whose columns are filtered once, as a rule.
// Parts of it where it is longer than kWvLong, so that more than two rows share
// the taps' rows (1024 x 8192, 8 taps: 60 and 104 us -> 56 and 83, 20 taps 145 and
// 225 -> 94 and 149), and where the whole rows are too few CTAs (64 x 8192, 20
// taps: 34 and 46 -> 16 and 16); up to a quarter of a part shared with the next.
static WvTile rdwt_tile(int n, int H, int W, int sf, int lh) {
  const int halo = (lh - 1) * sf;
  const long groups = (long)n * sf * ((H / sf + 1) / 2);
  WvTile t{W, W};
  if (W <= kWvLong && groups >= fill()) return t;
  for (int in : {1024, 512, 256}) {
    if (in >= W || halo > in / 4) continue;
    t = {in - halo, in};
    if (groups * ((W + t.out - 1) / t.out) >= fill()) break;
  }
  return t;
}
// Rows per CTA: as many as share the taps' rows (8, 4 or 2) while two CTAs fit
// an SM and the grid fills the GPU; 2 where the row or the grid is small.
static int rdwt_rows(int n, int H, int W, int sf, WvTile t) {
  for (int th : {8, 4})
    if (th * t.in * sizeof(float2) <= kWvTwoCtas &&
        (long)n * sf * ((H / sf + th - 1) / th) * ((W + t.out - 1) / t.out) >= fill())
      return th;
  return 2;
}

// The shared memory opted into is the most that the kernel is ever launched
// with: the attribute is the function's, and a launch of another width in another
// thread may come between a smaller one's setting and its launch.
template <auto Kernel, class... Args>
static cudaError_t launch_rdwt(int th, int threads, int n, int H, int W, int sf, WvTile t, cudaStream_t st,
                               Args... args) {
  const size_t sm = th * t.in * sizeof(float2);
  if (sm > 48 * 1024) {
    const size_t most = th > 2 ? kWvTwoCtas : 2 * kWvMaxW * sizeof(float2);
    const cudaError_t e = cudaFuncSetAttribute(Kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
    if (e != cudaSuccess) return e;
  }
  count_launch();
  launch_pdl(Kernel, dim3((unsigned)(sf * ((H / sf + th - 1) / th)), (unsigned)n, (unsigned)((W + t.out - 1) / t.out)),
             threads, sm, st, args...);
  return cudaGetLastError();
}

// The lengths of the Haar, Daubechies, Symmlet, Coiflet-1..3 and Beylkin filters
// are compiled in.  The others (Coiflet-4 and -5, Vaidyanathan, Battle, a caller's
// own) take the taps from a loop, with the rows under a tap rotating through
// registers: 2048^2, four levels, 24 taps 331 and 384 us (analysis, synthesis);
// with every output row's samples read anew 430 and 592.
#define NSST_RDWT_LENS(X) X(2) X(4) X(6) X(8) X(10) X(12) X(14) X(16) X(18) X(20)

cudaError_t launch_rdwt_level(const WvPlanes& P, int n, int H, int W, int sf, const WvTaps& t, const float* thr,
                              cudaStream_t st) {
  if (!rdwt_width_supported(W) || t.lh < 1 || t.lh > kMaxQmf || n < 1 || n > 65535) return cudaErrorInvalidValue;
  const WvTile tile = rdwt_tile(n, H, W, sf, t.lh);
#define GO(l, h, T, parts)                                                                                                  \
  launch_rdwt<k_rdwt_fwd<l, h, T, parts>>(h, T, n, H, W, sf, tile, st, P.cur, P.s_cur, P.yl, P.s_yl, P.yh, P.s_yh, H, W, sf, tile, t, thr)
#define ROWS(l, parts)                                 \
  switch (rdwt_rows(n, H, W, sf, tile)) {              \
    case 8: return GO(l, 8, kWvThreads, parts);        \
    case 4: return GO(l, 4, kWvThreads, parts);        \
    default: return GO(l, 2, kWvThreads, parts);       \
  }
#define CASE(l) \
  case l: ROWS(l, false)
  if (tile.in < W) ROWS(0, true)
  if (W > kWvLong) return GO(0, 2, 4 * kWvThreads, false);
  switch (t.lh) {
    NSST_RDWT_LENS(CASE)
    default:
      ROWS(0, false)
  }
#undef CASE
#undef ROWS
#undef GO
}

cudaError_t launch_rdwt_level_in_place(const WvPlanes& P, int n, int H, int W, int sf, const WvTaps& t,
                                       const float* thr, cudaStream_t st) {
  if (!rdwt_width_supported(W) || t.lh < 1 || t.lh > kMaxQmf || n < 1 || n > 65535) return cudaErrorInvalidValue;
  const size_t sm = (size_t)W * sizeof(float2);
  if (sm > 48 * 1024) {
    const cudaError_t e =
        cudaFuncSetAttribute(k_rdwt_rows_fwd, cudaFuncAttributeMaxDynamicSharedMemorySize, kWvMaxW * sizeof(float2));
    if (e != cudaSuccess) return e;
  }
  count_launch(2);
  launch_pdl(k_rdwt_cols_fwd, dim3((H + 7) / 8, (W + 31) / 32, n), dim3(32, 8), 0, st, P.cur, P.s_cur, P.yh, P.s_yh, H,
             W, sf, t);
  launch_pdl(k_rdwt_rows_fwd, dim3(H, n), kWvThreads, sm, st, P.yl, P.s_yl, P.yh, P.s_yh, H, W, sf, t, thr);
  return cudaGetLastError();
}

cudaError_t launch_irdwt_level(const float* ll, size_t s_ll, const float* yh, size_t s_yh, float* x, size_t s_x, int n,
                               int H, int W, int sf, const WvTaps& t, cudaStream_t st) {
  if (!rdwt_width_supported(W) || t.lh < 1 || t.lh > kMaxQmf || n < 1 || n > 65535) return cudaErrorInvalidValue;
  const WvTile tile = rdwt_tile(n, H, W, sf, t.lh);
#define GO(l, h, T, parts) launch_rdwt<k_rdwt_inv<l, h, T, parts>>(h, T, n, H, W, sf, tile, st, ll, s_ll, yh, s_yh, x, s_x, H, W, sf, tile, t)
#define ROWS(l, parts)                                 \
  switch (rdwt_rows(n, H, W, sf, tile)) {              \
    case 8: return GO(l, 8, kWvThreads, parts);        \
    case 4: return GO(l, 4, kWvThreads, parts);        \
    default: return GO(l, 2, kWvThreads, parts);       \
  }
#define CASE(l) \
  case l: ROWS(l, false)
  if (tile.in < W) ROWS(0, true)
  if (W > kWvLong) return GO(0, 2, 4 * kWvThreads, false);
  switch (t.lh) {
    NSST_RDWT_LENS(CASE)
    default:
      ROWS(0, false)
  }
#undef CASE
#undef ROWS
#undef GO
}

cudaError_t launch_tv_haar(const float* x, float* y, size_t stride, int n, int H, int W, float a, float gamma,
                           cudaStream_t st) {
  if (n < 1 || n > 65535) return cudaErrorInvalidValue;
  const std::vector<double> haar = {(double)a, (double)a};
  const WvTaps ta = analysis_taps(haar), ts = synthesis_taps(haar);
  count_launch();
  const int rows = kTvRows * kTvWarps;
  launch_pdl(k_tv_haar, dim3((W + kTvCols - 1) / kTvCols, (H + rows - 1) / rows, n), dim3(32, kTvWarps), 0, st, 
      x, y, stride, H, W, ta, ts, gamma);
  return cudaGetLastError();
}

cudaError_t launch_dwt_hh(const float* x, size_t stride, int n, int H, int W, const double* b, int lh, double* hh,
                          cudaStream_t st) {
  if (lh < 1 || lh > kMaxQmf || n < 1 || n > 65535) return cudaErrorInvalidValue;
  DTaps t{};
  t.lh = lh;
  for (int i = 0; i < lh; i++) t.b[i] = b[i];
  count_launch();
  launch_pdl(k_dwt_hh, dim3((W / 2 + 31) / 32, (H / 2 + 7) / 8, n), dim3(32, 8), 0, st, x, stride, H, W, t, hh);
  return cudaGetLastError();
}

cudaError_t launch_sep_residual(const float* img, const float* p1, const float* p2, float* ra1, float* ra2,
                                size_t n, cudaStream_t st) {
  const int blocks = (int)std::min<size_t>((n + 255) / 256, 152 * 8);
  count_launch();
  launch_pdl(k_sep_residual, blocks, 256, 0, st, img, p1, p2, ra1, ra2, n);
  return cudaGetLastError();
}

}  // namespace nsst
