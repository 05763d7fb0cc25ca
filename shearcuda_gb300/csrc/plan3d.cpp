// 3-D NSST plan and the C ABI of the volume path declared in include/nsst.h.
//
// The reference runs this path as MATLAB glue around cuFFT
// (shearcuda3d/DenoiseDemo/main.m:80-145, ShDecThRec_cuda.cpp:178-335): every
// call builds cuFFT plans, re-transforms every directional filter, and pads
// and crops through three temporary arrays per band.  Here the plan owns,
// once: the FP64-built Meyer filters' convolution spectra in FP32 on the
// device, the pyramid windows, the twiddle tables, and every work buffer for
// a batch of volumes; an execute call is a fixed sequence of launches on the
// caller's stream over all volumes of the batch at once.
//
// Pipeline of one level of the directional stage (convnfft.m:79-201, 'same'):
//   Y = FFT3(zero-pad(BP_l, Lc))            once per level, half spectrum
//   W = F_a .* Y + i F_b .* Y               two real filters per complex IFFT
//   IFFT3(W); real part -> band a, imaginary part -> band b, cropped at
//   offset ceil((24-1)/2) = 12; hard threshold and band sum (ShRec.m:11-24).
// All band pairs of a level go through each of the inverse's three passes in
// one launch (in chunks, where the plan's work buffer does not hold them all).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>
#include <mutex>
#include <random>
#include <memory>
#include <thread>

#include "internal.h"

using namespace nsst;

namespace {

constexpr int kCube = 24;          // Meyer filter support (GetMeyerBasedFilter.m:18)
constexpr int kSameOff = 12;       // convnfft 'same' offset: ceil((24 - 1) / 2)
constexpr int kMaxGrid = 192;      // largest padded grid per dimension
constexpr int kCtasPerSm = 8;      // CTAs per SM that keep a pass's loads in flight
// Band pairs in flight per level: the work buffer holds as many as fit here (at least one; one,
// if the device has no room for more).
constexpr size_t kPairBytes = (size_t)1 << 30;
// The 2^a 3^b lengths: the grids of NSST3_GRID_FAST, and the convolution lengths that nsst3_level_dims reports.
const int kFftLens[] = {16, 24, 32, 48, 64, 72, 96, 128, 144, 192, 216, 256};
constexpr int kMaxLen = 256;

bool is_fft_len(int n) {
  for (int v : kFftLens)
    if (v == n) return true;
  return false;
}
// Smallest supported circular-convolution length for the 'same' part of a
// linear convolution of m samples with the 24-tap filter: outputs 12 .. m+11
// alias no wrapped tap once N >= m + 12 (taps reach 23 back and 11 ahead of
// the kept range), so the full m + 23 is not needed.
int conv_len(int m) {
  for (int v : kFftLens)
    if (v >= m + kSameOff) return v;
  return -1;
}
// The length the transforms run at: the shortest compiled one, with factors 5
// and 7 beside 2 and 3 (and 11 and 17 where the padded grids have them anyway).
// A level costs its convolution volume, so 156 -> 160 instead of 192, 108
// instead of 128 and 76 -> 80 instead of 96 are 0.58, 0.60 and 0.58 of it.
int run_len(int m) {
  for (int v = m + kSameOff; v <= kMaxLen; v++)
    if (const V3Ops* o = v3_ops(v); o && o->conv) return v;
  return -1;
}
// What a grid may have as a level size is what the pyramid is compiled for.
bool is_pyr_len(int n) {
  const V3Ops* o = v3_ops(n);
  return o && o->pyr;
}

nsst_status fail3(nsst_status s, const std::string& msg) {
  set_error(msg);
  return s;
}
nsst_status cuda_fail3(cudaError_t e, const char* what) {
  set_error(std::string(what) + ": " + cudaGetErrorString(e));
  return e == cudaErrorMemoryAllocation ? NSST_ERR_OUT_OF_MEMORY : NSST_ERR_CUDA;
}
#define V3_CUDA(call)                                    \
  do {                                                   \
    cudaError_t _e = (call);                             \
    if (_e != cudaSuccess) return cuda_fail3(_e, #call); \
  } while (0)
#define V3_TRY(call)              \
  do {                            \
    nsst_status _s = (call);      \
    if (_s != NSST_OK) return _s; \
  } while (0)

// PyrNDDec_mm.m:58-74: w, tbw and D of each level for a pyramid mode
bool pyr_params(double mode, int L, double* w, double* tbw, double* D) {
  double w0, w1, t0, t1, d0, d1;
  if (mode == 1.0) {
    w0 = 0.5, w1 = 0.25, t0 = 1.0 / 6, t1 = 1.0 / 12, d0 = 1.0, d1 = 2.0;
  } else if (mode == 1.5) {
    w0 = 0.5, w1 = 3.0 / 8, t0 = 1.0 / 7, t1 = 1.0 / 9, d0 = 1.5, d1 = 2.0;
  } else if (mode == 2.0) {
    w0 = w1 = 1.0 / 3, t0 = t1 = 1.0 / 7, d0 = d1 = 2.0;
  } else {
    return false;
  }
  for (int l = 0; l < L; l++) {
    w[l] = l ? w1 : w0;
    tbw[l] = l ? t1 : t0;
    D[l] = l ? d1 : d0;
  }
  return true;
}

// Level sizes of a grid g: g, g/D0, g/D0/D1, ...; false if one is not an
// integer 2^a 3^b transform length or its convolution length is missing.
bool level_sizes(int g, int L, const double* D, int* out) {
  double v = g;
  out[0] = g;
  if (!is_fft_len(g) || !is_pyr_len(g) || run_len(g) < 0) return false;
  for (int l = 0; l < L; l++) {
    v /= D[l];
    const int iv = (int)std::lround(v);
    if (std::fabs(v - iv) > 1e-9 || !is_fft_len(iv) || !is_pyr_len(iv) || iv % 8) return false;
    if (l + 1 < L && run_len(iv) < 0) return false;
    out[l + 1] = iv;
  }
  return true;
}

// The grid of MarshalData.m:3-22 (the reference's any-size demo,
// mainAnySize.m:51): every dimension gains d - rem(n, d) planes, d = 3 2^(L-1)
// (divFactor [3 6 12 24] of the level count), so that Pyr_mode 1.5's level
// sizes g, g/1.5, g/3, ... are integers.  Its level sizes need transform
// lengths with other prime factors (132 = 3 * 4 * 11, 204 = 3 * 4 * 17).  The
// largest compiled one is 216, for sides up to 215 on one or two levels.
int marshal_grid(int n, int L) {
  const int d = 3 << (L - 1);
  return n + d - n % d;
}
bool marshal_sizes(int g, int L, const double* D, int* out, int* missing) {
  double v = g;
  out[0] = g;
  *missing = 0;
  if (!is_pyr_len(g) || run_len(g) < 0) {
    *missing = g;
    return false;
  }
  for (int l = 0; l < L; l++) {
    v /= D[l];
    const int iv = (int)std::lround(v);
    if (std::fabs(v - iv) > 1e-9 || !is_pyr_len(iv) || (l + 1 < L && run_len(iv) < 0)) {
      *missing = iv;
      return false;
    }
    out[l + 1] = iv;
  }
  return true;
}

// Smallest supported grid >= n for which every level size works.
int grid_size(int n, int L, const double* D) {
  int tmp[NSST_MAX_LEVELS + 1];
  for (int g : kFftLens)
    if (g >= n && g <= kMaxGrid && level_sizes(g, L, D, tmp)) return g;
  return -1;
}

// row pitch of the keep bits along the box's last dimension: a multiple of 8,
// so that the eight sequences of a pass group fill whole bytes
int mask_pitch(int m2) { return (m2 + 7) / 8 * 8; }

int host_threads3() {
  unsigned n = std::thread::hardware_concurrency();
  return n == 0 ? 4 : (int)std::min(n, 16u);
}

size_t align_up3(size_t v, size_t a) { return (v + a - 1) / a * a; }
size_t mask_band_bytes(const int* m) { return align_up3((size_t)m[0] * m[1] * mask_pitch(m[2]) / 8, 256); }

}  // namespace

struct nsst3_plan {
  nsst3_config cfg{};
  int n[3] = {0, 0, 0};  // volume dims
  int g[3] = {0, 0, 0};  // padded grid
  int L = 0, B = 1, nbands = 0, device = 0;
  double w[NSST_MAX_LEVELS], tbw[NSST_MAX_LEVELS], D[NSST_MAX_LEVELS];

  struct Level {
    int m[3] = {0, 0, 0};   // band-pass dims (level L: lowpass)
    int lc[3] = {0, 0, 0};  // convolution transform lengths (levels < L)
    int nd = 0, nb = 0, first_band = 0;
    size_t bp_off = 0;      // floats, in the sub-band layout
    size_t xh_off = 0;      // float2, in one volume's half-spectrum block
    size_t spec_off = 0;    // float2, first band's spectrum
    int K[3] = {0, 0, 0};   // window support of the decomposition step (levels < L)
    size_t win_off[3] = {0, 0, 0};
    size_t vol() const { return (size_t)m[0] * m[1] * m[2]; }
    size_t half() const { return (size_t)m[0] * m[1] * v3_pitch(m[2] / 2 + 1); }
    size_t conv() const { return (size_t)lc[0] * lc[1] * lc[2]; }
    // one band pair's partly inverted spectrum: the box's z kept
    size_t pair() const { return (size_t)lc[0] * lc[1] * v3_pitch(m[2]); }
    int npairs() const { return (nb + 1) / 2; }
  };
  std::vector<Level> lev;  // L + 1 entries
  std::vector<int> band_level, band_cone, band_l2, band_l1;

  size_t bp_floats = 0;    // sub-band layout per volume
  size_t vol_elems = 0;    // voxels of the grid
  size_t xh_elems = 0;     // half spectra of every level per item
  size_t conv_elems = 0;   // largest convolution spectrum
  size_t wk_elems = 0;     // band-pair work buffer (all items)
  size_t in_elems = 0;     // n0 n1 n2

  char* arena = nullptr;
  size_t arena_bytes = 0;
  float2* spec = nullptr;
  float* win = nullptr;
  float2* tw = nullptr;
  std::map<int, size_t> tw_off;  // transform length -> offset (float2) in tw
  float2* xh = nullptr;
  float2* Y = nullptr;
  float2* Wk = nullptr;
  float* bp = nullptr;
  float* rbp = nullptr;
  float* th = nullptr;

  // differentiation: keep bits of every band of the last thresholded forward
  uint8_t* mask = nullptr;
  size_t mask_bytes = 0;            // per item
  std::vector<size_t> mask_off;     // per band, in bytes (bit k = voxel k of the band, linear order)
  int masks_valid_n = 0;            // items covered by the stored masks (0 = none)

  std::vector<double> scalars;
  bool has_scalars = false;
  std::vector<float> th_host;
  std::mutex mu;

  const float2* twid(int len) const { return tw + tw_off.at(len); }
};

namespace {

// Strides of a line pass along `axis` (1 or 0) in an array d0 x d1 x pitch.
void set_axis(V3Cols& P, int axis, int d1, int pitch) {
  P.in_a = P.out_a = axis == 1 ? d1 * pitch : pitch;
  P.in_i = P.out_i = axis == 1 ? pitch : d1 * pitch;
}
// A pass along `axis` of n items in place on v (d0 x d1 x pitch, item stride
// `stride`): lines (a < an, z < zn), elements [in] loaded, [out] stored, both
// ranges kept at the start of the line.
struct Range {
  int lo, n;
};
V3Cols line_pass(int axis, float2* v, size_t stride, int d1, int pitch, int n, int an, int zn, Range in, Range out) {
  V3Cols P;
  P.in = v;
  P.out = v;
  P.items = n, P.an = an, P.zn = zn;
  P.in_item = P.out_item = stride;
  set_axis(P, axis, d1, pitch);
  P.in_lo = in.lo, P.in_n = in.n, P.out_lo = out.lo, P.out_n = out.n;
  return P;
}
nsst_status run_cols(nsst3_plan* p, int len, int dir, int ld, int st_mode, const V3Cols& P, int npairs,
                     cudaStream_t st) {
  V3_CUDA(v3_ops(len)->cols(dir, ld, st_mode, P, p->twid(len), npairs, st));
  return NSST_OK;
}

// Forward FFT of n real volumes m (item stride rstride floats, dims src[3];
// beyond them zero or, edge, the last sample repeated) on a grid d: half
// spectra d0 x d1 x pitch(d2/2 + 1) in h.  rec: the axis-0 pass merges the next
// level's half spectrum (ST_REC fields set by the caller in *rec).
nsst_status fft3_real(nsst3_plan* p, const float* x, size_t rstride, const int* src, bool edge, const int* m,
                      float2* h, size_t stride, const int* d, int n, cudaStream_t st, const V3Cols* rec = nullptr) {
  const int H = d[2] / 2 + 1, pitch = v3_pitch(H);
  V3Real R;
  R.src = x;
  R.spec = h;
  R.r_stride = rstride, R.spec_stride = stride;
  R.rows0 = m[0], R.rows1 = m[1];
  R.n0 = src[0], R.n1 = src[1], R.n2 = src[2];
  R.s1 = d[1], R.pitch = pitch, R.line = d[2], R.edge = edge;
  V3_CUDA(v3_ops(d[2])->real(-1, R, p->twid(d[2]), n, st));
  V3_TRY(run_cols(p, d[1], -1, V3_LD_CPLX, V3_ST_CPLX,
                  line_pass(1, h, stride, d[1], pitch, n, m[0], H, {0, m[1]}, {0, d[1]}), 1, st));
  V3Cols P = line_pass(0, h, stride, d[1], pitch, n, d[1], H, {0, m[0]}, {0, d[0]});
  if (rec) {
    P.win = rec->win;
    P.lp = rec->lp;
    P.s0 = rec->s0, P.s1 = rec->s1, P.s2p = rec->s2p;
    P.scale = rec->scale;
  }
  return run_cols(p, d[0], -1, V3_LD_CPLX, rec ? V3_ST_REC : V3_ST_CPLX, P, 1, st);
}

// Inverse FFT of half spectra in h (grid d, destroyed) whose first out[k]
// samples per axis, times scale, go to the real volumes x.  hp: the axis-0
// pass first applies the level's high-pass window.
nsst_status ifft3_real(nsst3_plan* p, float2* h, size_t stride, const int* d, float* x, size_t rstride,
                       const int* out, float scale, int n, cudaStream_t st, const PyrWin* hp = nullptr) {
  const int H = d[2] / 2 + 1, pitch = v3_pitch(H);
  V3Cols P = line_pass(0, h, stride, d[1], pitch, n, d[1], H, {0, d[0]}, {0, out[0]});
  if (hp) P.win = *hp;
  V3_TRY(run_cols(p, d[0], +1, hp ? V3_LD_HP : V3_LD_CPLX, V3_ST_CPLX, P, 1, st));
  V3_TRY(run_cols(p, d[1], +1, V3_LD_CPLX, V3_ST_CPLX,
                  line_pass(1, h, stride, d[1], pitch, n, out[0], H, {0, d[1]}, {0, out[1]}), 1, st));
  V3Real R;
  R.dst = x;
  R.spec = h;
  R.r_stride = rstride, R.spec_stride = stride;
  R.rows0 = out[0], R.rows1 = out[1], R.n2 = out[2];
  R.s1 = d[1], R.pitch = pitch, R.line = d[2];
  R.scale = scale;
  V3_CUDA(v3_ops(d[2])->real(+1, R, p->twid(d[2]), n, st));
  return NSST_OK;
}

PyrWin level_window(const nsst3_plan* p, int l) {
  const nsst3_plan::Level& a = p->lev[l];
  PyrWin w;
  for (int k = 0; k < 3; k++) {
    w.K[k] = a.K[k];
    w.nr[k] = a.m[k];
  }
  w.v0 = p->win + a.win_off[0];
  w.v1 = p->win + a.win_off[1];
  w.v2 = p->win + a.win_off[2];
  return w;
}

// PyrNDDec_mm.m:20-109 (OutD 'S') for n volumes x (dims in[3], padded to the
// grid by edge replication, or by zeros for the adjoint) into the sub-band
// layout bp (item stride bp_floats).
nsst_status run_pyr_dec(nsst3_plan* p, const float* x, const int* in, float* bp, int n, cudaStream_t st,
                        bool zero_pad = false) {
  const size_t xs = (size_t)in[0] * in[1] * in[2];
  V3_TRY(fft3_real(p, x, xs, in, !zero_pad, p->g, p->xh + p->lev[0].xh_off, p->xh_elems, p->g, n, st));
  for (int l = 0; l <= p->L; l++) {
    const nsst3_plan::Level& a = p->lev[l];
    PyrWin win;
    if (l < p->L) {
      // PrySDdec_onestep.m:82-125: Lp into the next level's block; Hp in the inverse's first pass
      const nsst3_plan::Level& b = p->lev[l + 1];
      win = level_window(p, l);
      V3_CUDA(launch_pyr_dec_lp(p->xh + a.xh_off, p->xh + b.xh_off, p->xh_elems, n, a.m[1], v3_pitch(a.m[2] / 2 + 1),
                                b.m[0], b.m[1], b.m[2], win, (float)(1.0 / std::pow(p->D[l], 1.5)), st));
    }
    // subs{l} = real(ifftn(ccsym(Hp, 3, 'e')))   (lowpass: the last Lp)
    V3_TRY(ifft3_real(p, p->xh + a.xh_off, p->xh_elems, a.m, bp + a.bp_off, p->bp_floats, a.m,
                      (float)(1.0 / (double)a.vol()), n, st, l < p->L ? &win : nullptr));
  }
  return NSST_OK;
}

// PyrNDRec_mm.m:20-95 (InD 'S'): bp -> x (dims out[3], the grid cropped).
nsst_status run_pyr_rec(nsst3_plan* p, const float* bp, float* x, const int* out, int n, cudaStream_t st) {
  for (int l = p->L; l >= 0; l--) {
    const nsst3_plan::Level& a = p->lev[l];
    V3Cols rec;
    if (l < p->L) {  // PrySDrec_onestep.m:96-119
      const nsst3_plan::Level& b = p->lev[l + 1];
      rec.win = level_window(p, l);
      rec.lp = p->xh + b.xh_off;
      rec.s0 = b.m[0], rec.s1 = b.m[1], rec.s2p = v3_pitch(b.m[2] / 2 + 1);
      rec.scale = (float)std::pow(p->D[l], 1.5);
    }
    // ccsym(fftn(subs{l}), 3, 'c')
    V3_TRY(fft3_real(p, bp + a.bp_off, p->bp_floats, a.m, false, a.m, p->xh + a.xh_off, p->xh_elems, a.m, n, st,
                     l < p->L ? &rec : nullptr));
  }
  const nsst3_plan::Level& l0 = p->lev[0];
  return ifft3_real(p, p->xh + l0.xh_off, p->xh_elems, p->g, x, (size_t)out[0] * out[1] * out[2], out,
                    (float)(1.0 / (double)l0.vol()), n, st);
}

// Pairs of a level that one pass over the work buffer takes for n items.
int pair_chunk(const nsst3_plan* p, const nsst3_plan::Level& a, int n) {
  return (int)std::max<size_t>(1, std::min<size_t>(a.npairs(), p->wk_elems / (a.pair() * n)));
}
// The passes whose CTAs loop over the chunk's pairs (what the pairs share is
// then read once) split them over the grid until it fills the GPU.
int pair_shares(int ctas, int pairs) {
  return std::min(pairs, std::max(1, (sm_count() * kCtasPerSm + ctas - 1) / ctas));
}
// Keep bits of the level's bands from band k on.
void set_masks(const nsst3_plan* p, V3Cols& P, int l, int k) {
  const nsst3_plan::Level& a = p->lev[l];
  P.m_r2 = mask_pitch(a.m[2]);
  P.m_band = mask_band_bytes(a.m);
  P.m_stride = p->mask_bytes;
  P.mask = p->mask + p->mask_off[a.first_band] + (size_t)k * P.m_band;
}
V3Pair pair_pass(const nsst3_plan* p, const nsst3_plan::Level& a, int k0, int pairs, int n) {
  V3Pair P;
  P.spec = p->spec + a.spec_off + (size_t)k0 * a.conv();
  P.W = p->Wk;
  P.w_item = a.pair();
  P.w_pair = a.pair() * n;
  P.N0 = a.lc[0], P.N1 = a.lc[1];
  P.wpitch = v3_pitch(a.m[2]);
  P.z_lo = kSameOff, P.z_n = a.m[2];
  P.pairs = pairs, P.items = n;
  return P;
}
// The chunk's pass along axis 1 in the work buffer, in place.
V3Cols pair_cols(const nsst3_plan* p, const nsst3_plan::Level& a, int n, Range in, Range out) {
  V3Cols P = line_pass(1, p->Wk, a.pair(), a.lc[1], v3_pitch(a.m[2]), n, a.lc[0], a.m[2], in, out);
  P.in_pair = P.out_pair = a.pair() * n;
  return P;
}

// Directional stage of one level.  Y = FFT3(zero-pad(bp_l)) once; per band
// pair, W = IFFT3(Y .* C) with C = F_a + i F_b, cut to the 'same' box at
// offset 12.  acc != NULL: hard threshold (th, or none when th is NULL) and
// band sum into acc (sub-band layout, level l region, item stride
// bp_floats), with keep bits when record_masks.  acc == NULL: band
// coefficients into coeffs (nb volumes of the level per item).
nsst_status run_sh_level(nsst3_plan* p, const float* bp, int l, float* acc, const float* th, float* coeffs, int n,
                         cudaStream_t st, bool record_masks = false) {
  const nsst3_plan::Level& a = p->lev[l];
  const int* N = a.lc;
  const int* m = a.m;
  const int wp = v3_pitch(m[2]);
  V3_TRY(fft3_real(p, bp + a.bp_off, p->bp_floats, m, false, m, p->Y, p->conv_elems, N, n, st));
  const int chunk = pair_chunk(p, a, n);
  for (int k0 = 0; k0 < a.npairs(); k0 += chunk) {
    const int pairs = std::min(chunk, a.npairs() - k0);
    // z rows: the product, stored only where the box needs it
    V3Pair P1 = pair_pass(p, a, k0, pairs, n);
    P1.Y = p->Y;
    P1.y_item = p->conv_elems;
    P1.pitch = v3_pitch(N[2] / 2 + 1);
    V3_CUDA(v3_ops(N[2])->pair(+1, P1, p->twid(N[2]), pair_shares((N[0] * N[1] + 7) / 8 * n, pairs), st));
    V3_TRY(run_cols(p, N[1], +1, V3_LD_CPLX, V3_ST_CPLX, pair_cols(p, a, n, {0, N[1]}, {kSameOff, m[1]}), pairs, st));
    V3Cols P3 = line_pass(0, p->Wk, a.pair(), N[1], wp, n, m[1], m[2], {0, N[0]}, {kSameOff, m[0]});
    P3.in_pair = a.pair() * n;
    P3.pairs = pairs;
    P3.nbands = a.nb - 2 * k0;
    P3.scale = (float)(1.0 / (double)a.conv());
    P3.r1 = m[1], P3.r2 = m[2];
    if (acc) {
      P3.rdst = acc + a.bp_off;
      P3.r_stride = p->bp_floats;
      P3.th = th ? th + a.first_band + 2 * k0 : nullptr;
      P3.nb_item = p->nbands;
      P3.first = k0 == 0;
      if (record_masks) set_masks(p, P3, l, 2 * k0);
      V3_TRY(run_cols(p, N[0], +1, V3_LD_CPLX, V3_ST_THRESH, P3, 1, st));
    } else {
      P3.rdst = coeffs + (size_t)(2 * k0) * a.vol();
      P3.r_stride = (size_t)a.nb * a.vol();
      P3.band_stride = a.vol();
      V3_TRY(run_cols(p, N[0], +1, V3_LD_CPLX, V3_ST_PAIR, P3, pair_shares(m[1] * ((m[2] + 7) / 8) * n, pairs), st));
    }
  }
  return NSST_OK;
}

// th[i * nbands + b] = T[level(b)] * sigma_i * scalars[b]  (ThresholdShCoeff.m:7)
nsst_status upload_th(nsst3_plan* p, int n, const double* sigma, const double* T, const double* scalars,
                      cudaStream_t st) {
  if (!sigma || !T) return fail3(NSST_ERR_INVALID_ARG, "sigma and T are required");
  if (!scalars) {
    if (!p->has_scalars) return fail3(NSST_ERR_INVALID_ARG, "no band scalars given or stored in the plan");
    scalars = p->scalars.data();
  }
  p->th_host.resize((size_t)n * p->nbands);
  for (int i = 0; i < n; i++)
    for (int b = 0; b < p->nbands; b++)
      p->th_host[(size_t)i * p->nbands + b] = (float)(T[p->band_level[b]] * sigma[i] * scalars[b]);
  // pageable source: the copy is staged before the call returns
  V3_CUDA(cudaMemcpyAsync(p->th, p->th_host.data(), p->th_host.size() * sizeof(float), cudaMemcpyHostToDevice, st));
  return NSST_OK;
}

// ShDecThRec_cuda: rec (sub-band layout) = per level sum of thresholded
// bands; lowpass copied from bp.
nsst_status run_dec_thresh_rec(nsst3_plan* p, const float* bp, float* rec, int n, const float* th, cudaStream_t st,
                               bool record_masks = false) {
  for (int l = 0; l < p->L; l++) V3_TRY(run_sh_level(p, bp, l, rec, th, nullptr, n, st, record_masks));
  // the layout's alignment gaps read as zero
  for (const nsst3_plan::Level& a : p->lev) {
    const size_t gap = align_up3(a.vol(), 64) - a.vol();
    if (gap)
      V3_CUDA(cudaMemset2DAsync(rec + a.bp_off + a.vol(), p->bp_floats * sizeof(float), 0, gap * sizeof(float), n, st));
  }
  const nsst3_plan::Level& lp = p->lev[p->L];
  V3_CUDA(cudaMemcpy2DAsync(rec + lp.bp_off, p->bp_floats * sizeof(float), bp + lp.bp_off,
                            p->bp_floats * sizeof(float), lp.vol() * sizeof(float), n, cudaMemcpyDeviceToDevice, st));
  return NSST_OK;
}

nsst_status check_call(nsst3_plan* p, int n, const void* a, const void* b) {
  if (!p) return fail3(NSST_ERR_INVALID_ARG, "NULL plan");
  if (n < 1 || n > p->B) return fail3(NSST_ERR_INVALID_ARG, "n must be in [1, batch capacity]");
  if (!a || !b) return fail3(NSST_ERR_INVALID_ARG, "NULL buffer");
  if (((uintptr_t)a & 3) || ((uintptr_t)b & 3)) return fail3(NSST_ERR_INVALID_ARG, "buffers must be 4-byte aligned");
  if (cudaSetDevice(p->device) != cudaSuccess) return fail3(NSST_ERR_CUDA, "cudaSetDevice failed");
  return NSST_OK;
}

}  // namespace

extern "C" {

int nsst3_meyer_filters(int nlevels, const int* num_dirs, double* out) {
  if (nlevels < 1 || nlevels > NSST_MAX_LEVELS || !num_dirs) return -1;
  int count = 0;
  for (int l = 0; l < nlevels; l++) {
    const int nd = num_dirs[l];
    if (nd < 2 || nd > 12 || kCube % nd) return -1;
    count += 3 * nd * nd;
  }
  if (out) {
    std::vector<double> f = meyer_filters_3d(kCube, nlevels, num_dirs);
    std::memcpy(out, f.data(), f.size() * sizeof(double));
  }
  return count;
}

nsst_status nsst3_plan_create(const nsst3_config* cfg, int n0, int n1, int n2, int batch, nsst3_plan** out) {
  if (!out) return fail3(NSST_ERR_INVALID_ARG, "NULL output pointer");
  *out = nullptr;
  if (!cfg) return fail3(NSST_ERR_INVALID_ARG, "config is NULL");
  if (cfg->nlevels < 1 || cfg->nlevels > 4) return fail3(NSST_ERR_INVALID_ARG, "nlevels must be in [1, 4]");
  if (batch < 1) return fail3(NSST_ERR_INVALID_ARG, "batch must be >= 1");
  if (nsst3_meyer_filters(cfg->nlevels, cfg->num_dirs, nullptr) < 0)
    return fail3(NSST_ERR_INVALID_ARG, "num_dirs must divide 24 and lie in [2, 12]");
  auto p = std::make_unique<nsst3_plan>();
  p->cfg = *cfg;
  p->L = cfg->nlevels;
  p->B = batch;
  if (!pyr_params(cfg->pyr_mode, p->L, p->w, p->tbw, p->D))
    return fail3(NSST_ERR_INVALID_ARG, "pyr_mode must be 1, 1.5 or 2");
  const int dims[3] = {n0, n1, n2};
  int sizes[3][NSST_MAX_LEVELS + 1];
  if (cfg->grid != NSST3_GRID_FAST && cfg->grid != NSST3_GRID_MARSHAL)
    return fail3(NSST_ERR_INVALID_ARG, "grid must be NSST3_GRID_FAST or NSST3_GRID_MARSHAL");
  if (cfg->grid == NSST3_GRID_MARSHAL && cfg->pyr_mode != 1.5)
    return fail3(NSST_ERR_INVALID_ARG, "NSST3_GRID_MARSHAL pads for Pyr_mode 1.5 (MarshalData.m's divFactor)");
  for (int k = 0; k < 3; k++) {
    if (dims[k] < 1) return fail3(NSST_ERR_INVALID_ARG, "volume dims must be positive");
    p->n[k] = dims[k];
    if (cfg->grid == NSST3_GRID_MARSHAL) {
      p->g[k] = marshal_grid(dims[k], p->L);
      int miss = 0;
      if (!marshal_sizes(p->g[k], p->L, p->D, sizes[k], &miss))
        return fail3(NSST_ERR_UNSUPPORTED_SIZE,
                     "MarshalData grid " + std::to_string(p->g[k]) + " of dimension " + std::to_string(dims[k]) +
                         " needs transform length " + std::to_string(miss) +
                         ", not compiled (level sizes of the 132 and 204 grids and the 2^a 3^b lengths up to 216 are)");
    } else {
      p->g[k] = grid_size(dims[k], p->L, p->D);
      if (p->g[k] < 0 || !level_sizes(p->g[k], p->L, p->D, sizes[k]))
        return fail3(NSST_ERR_UNSUPPORTED_SIZE, "volume dimension too large for this pyramid (grid <= 192)");
    }
  }
  V3_CUDA(cudaGetDevice(&p->device));
  p->in_elems = (size_t)n0 * n1 * n2;

  // level geometry, band tables and layout offsets
  p->lev.resize(p->L + 1);
  size_t bp_off = 0, xh_off = 0, spec_off = 0, win_off = 0;
  for (int l = 0; l <= p->L; l++) {
    nsst3_plan::Level& a = p->lev[l];
    for (int k = 0; k < 3; k++) a.m[k] = sizes[k][l];
    a.bp_off = bp_off;
    bp_off += align_up3(a.vol(), 64);
    a.xh_off = xh_off;
    xh_off += align_up3(a.half(), 32);
    if (l == p->L) break;
    for (int k = 0; k < 3; k++) a.lc[k] = run_len(a.m[k]);
    a.nd = cfg->num_dirs[l];
    a.nb = 3 * a.nd * a.nd;
    a.first_band = p->nbands;
    for (int c = 0; c < 3; c++)
      for (int l2 = 0; l2 < a.nd; l2++)
        for (int l1 = 0; l1 < a.nd; l1++) {
          p->band_level.push_back(l);
          p->band_cone.push_back(c);
          p->band_l2.push_back(l2);
          p->band_l1.push_back(l1);
        }
    p->nbands += a.nb;
    a.spec_off = spec_off;
    spec_off += (size_t)((a.nb + 1) / 2) * a.conv();  // one spectrum F_a + i F_b per band pair
    p->conv_elems = std::max(p->conv_elems, a.conv());
  }
  size_t wk_least = 0;
  for (int l = 0; l < p->L; l++) {
    const nsst3_plan::Level& a = p->lev[l];
    const size_t one = a.pair() * batch;
    const size_t fit = std::max<size_t>(1, kPairBytes / (one * sizeof(float2)));
    // the backward's half spectra of S and its fold scratch live there too
    wk_least = std::max({wk_least, one, (size_t)a.m[0] * a.lc[1] * v3_pitch(a.lc[2] / 2 + 1) * batch});
    p->wk_elems = std::max({p->wk_elems, wk_least, one * std::min<size_t>(a.npairs(), fit)});
  }
  p->bp_floats = bp_off;
  p->xh_elems = xh_off;
  p->vol_elems = (size_t)p->g[0] * p->g[1] * p->g[2];

  // pyramid windows (PrySDdec_onestep.m:48-82), FP64 -> FP32
  std::vector<float> win_host;
  for (int l = 0; l < p->L; l++) {
    nsst3_plan::Level& a = p->lev[l];
    for (int k = 0; k < 3; k++) {
      std::vector<double> v;
      pyr_window_1d(a.m[k], p->w[l], p->tbw[l], &a.K[k], &v);
      // the window must fit the level's half spectrum and the next level's
      // grid (full axes: both halves; half axis: its non-negative part)
      const int small = p->lev[l + 1].m[k];
      if (a.K[k] >= a.m[k] / 2 + 1 || (k < 2 && a.K[k] >= small) || (k == 2 && a.K[k] >= small / 2 + 1))
        return fail3(NSST_ERR_UNSUPPORTED_SIZE, "pyramid window wider than the level");
      a.win_off[k] = win_off;
      for (double d : v) win_host.push_back((float)d);
      win_off += v.size();
    }
  }
  // twiddle tables of every transform length in use
  std::vector<float2> tw_host;
  auto add_tw = [&](int len) {
    if (p->tw_off.count(len)) return;
    p->tw_off[len] = tw_host.size();
    std::vector<float2> t = twiddle_table(len);
    tw_host.insert(tw_host.end(), t.begin(), t.end());
  };
  for (int l = 0; l <= p->L; l++)
    for (int k = 0; k < 3; k++) {
      add_tw(p->lev[l].m[k]);
      if (l < p->L) add_tw(p->lev[l].lc[k]);
      const V3Ops *om = v3_ops(p->lev[l].m[k]), *oc = l < p->L ? v3_ops(p->lev[l].lc[k]) : nullptr;
      if (!om || !om->pyr || (l < p->L && (!oc || !oc->conv)))
        return fail3(NSST_ERR_UNSUPPORTED_SIZE, "volume transform length not compiled");
    }
  for (auto& kv : p->tw_off) {
    cudaError_t e = v3_ops(kv.first)->prepare();
    if (e != cudaSuccess) return cuda_fail3(e, "volume pass set-up");
  }

  // one device arena
  const size_t B = (size_t)batch;
  size_t off = 0;
  auto take = [&](size_t bytes) {
    size_t o = off;
    off = align_up3(off + bytes, 256);
    return o;
  };
  const size_t o_spec = take(spec_off * sizeof(float2));
  const size_t o_win = take(win_host.size() * sizeof(float));
  const size_t o_tw = take(tw_host.size() * sizeof(float2));
  const size_t o_xh = take(B * p->xh_elems * sizeof(float2));
  const size_t o_y = take(B * p->conv_elems * sizeof(float2));
  const size_t o_bp = take(B * p->bp_floats * sizeof(float));
  const size_t o_rbp = take(B * p->bp_floats * sizeof(float));
  const size_t o_th = take(B * p->nbands * sizeof(float));
  const size_t o_w = off;  // last: its size depends on the room there is
  void* arena = nullptr;
  take(p->wk_elems * sizeof(float2));
  cudaError_t e = dev_alloc(&arena, off);
  if (e == cudaErrorMemoryAllocation && wk_least < p->wk_elems) {
    (void)cudaGetLastError();
    p->wk_elems = wk_least;
    off = o_w;
    take(p->wk_elems * sizeof(float2));
    e = dev_alloc(&arena, off);
  }
  if (e != cudaSuccess) return cuda_fail3(e, "plan arena");
  p->arena = (char*)arena;
  p->arena_bytes = off;
  p->spec = (float2*)(p->arena + o_spec);
  p->win = (float*)(p->arena + o_win);
  p->tw = (float2*)(p->arena + o_tw);
  p->xh = (float2*)(p->arena + o_xh);
  p->Y = (float2*)(p->arena + o_y);
  p->Wk = (float2*)(p->arena + o_w);
  p->bp = (float*)(p->arena + o_bp);
  p->rbp = (float*)(p->arena + o_rbp);
  p->th = (float*)(p->arena + o_th);
  nsst3_plan* raw = p.get();
  auto cleanup = [&](nsst_status s) {
    cudaFree(raw->arena);
    raw->arena = nullptr;
    return s;
  };
  if ((e = cudaMemcpy(p->win, win_host.data(), win_host.size() * sizeof(float), cudaMemcpyHostToDevice)) ||
      (e = cudaMemcpy(p->tw, tw_host.data(), tw_host.size() * sizeof(float2), cudaMemcpyHostToDevice)))
    return cleanup(cuda_fail3(e, "plan tables"));

  // Meyer filters (FP64) and the convolution spectra of each band pair,
  // C = F_a + i F_b, FP64 on host worker threads, converted to FP32 and
  // uploaded as each is finished.
  const std::vector<double> filt = meyer_filters_3d(kCube, p->L, cfg->num_dirs);
  const size_t f3 = (size_t)kCube * kCube * kCube;
  std::vector<int> pair_a;  // first band of every pair
  for (int l = 0; l < p->L; l++)
    for (int k = 0; k < p->lev[l].nb; k += 2) pair_a.push_back(p->lev[l].first_band + k);
  const int npairs = (int)pair_a.size();
  const int nthreads = std::min(host_threads3(), npairs);
  std::vector<cudaError_t> terr(nthreads, cudaSuccess);
  std::vector<std::thread> workers;
  for (int t = 0; t < nthreads; t++) {
    workers.emplace_back([&, t]() {
      if (cudaSetDevice(raw->device) != cudaSuccess) {
        terr[t] = cudaErrorInvalidDevice;
        return;
      }
      std::vector<cd> Sa, Sb;
      std::vector<float2> s32;
      for (int q = t; q < npairs; q += nthreads) {
        const int b = pair_a[q];
        const nsst3_plan::Level& a = raw->lev[raw->band_level[b]];
        const bool has_b = b + 1 < a.first_band + a.nb;
        filter_spectrum_3d(filt.data() + (size_t)b * f3, kCube, a.lc[0], a.lc[1], a.lc[2], &Sa);
        if (has_b) filter_spectrum_3d(filt.data() + (size_t)(b + 1) * f3, kCube, a.lc[0], a.lc[1], a.lc[2], &Sb);
        s32.resize(Sa.size());
        for (size_t i = 0; i < Sa.size(); i++) {
          cd c = Sa[i];
          if (has_b) c += cd(0, 1) * Sb[i];
          s32[i] = make_float2((float)c.real(), (float)c.imag());
        }
        const size_t dst = a.spec_off + (size_t)((b - a.first_band) / 2) * a.conv();
        cudaError_t ce = cudaMemcpy(raw->spec + dst, s32.data(), s32.size() * sizeof(float2), cudaMemcpyHostToDevice);
        if (ce != cudaSuccess) {
          terr[t] = ce;
          return;
        }
      }
    });
  }
  for (auto& w : workers) w.join();
  for (cudaError_t te : terr)
    if (te != cudaSuccess) return cleanup(cuda_fail3(te, "filter spectra upload"));
  *out = p.release();
  return NSST_OK;
}

nsst_status nsst3_plan_destroy(nsst3_plan* p) {
  if (!p) return NSST_OK;
  {
    std::lock_guard<std::mutex> lk(p->mu);
    cudaSetDevice(p->device);
    if (p->arena) cudaFree(p->arena);
    if (p->mask) cudaFree(p->mask);
    p->arena = nullptr;
    p->mask = nullptr;
  }
  delete p;
  return NSST_OK;
}

int nsst3_num_bands(const nsst3_plan* p) { return p ? p->nbands : 0; }
size_t nsst3_subband_floats(const nsst3_plan* p) { return p ? p->bp_floats : 0; }
size_t nsst3_plan_device_bytes(const nsst3_plan* p) { return p ? p->arena_bytes : 0; }

nsst_status nsst3_level_dims(const nsst3_plan* p, int level, int* dims, int* conv) {
  if (!p) return fail3(NSST_ERR_INVALID_ARG, "NULL plan");
  if (level < -1 || level > p->L) return fail3(NSST_ERR_INVALID_ARG, "level out of range");
  for (int k = 0; k < 3; k++) {
    if (dims) dims[k] = level < 0 ? p->g[k] : p->lev[level].m[k];
    if (conv) conv[k] = (level < 0 || level == p->L) ? 0 : conv_len(p->lev[level].m[k]);
  }
  return NSST_OK;
}

nsst_status nsst3_band_info(const nsst3_plan* p, int b, int* info) {
  if (!p || !info) return fail3(NSST_ERR_INVALID_ARG, "NULL argument");
  if (b < 0 || b >= p->nbands) return fail3(NSST_ERR_INVALID_ARG, "band out of range");
  info[0] = p->band_level[b];
  info[1] = p->band_cone[b];
  info[2] = p->band_l2[b];
  info[3] = p->band_l1[b];
  return NSST_OK;
}

nsst_status nsst3_plan_set_scalars(nsst3_plan* p, const double* s) {
  if (!p || !s) return fail3(NSST_ERR_INVALID_ARG, "NULL argument");
  p->scalars.assign(s, s + p->nbands);
  p->has_scalars = true;
  return NSST_OK;
}

}  // extern "C"

extern "C" {

nsst_status nsst3_pyr_dec(nsst3_plan* p, const float* x, float* bp, int n, void* stream) {
  V3_TRY(check_call(p, n, x, bp));
  std::lock_guard<std::mutex> lk(p->mu);
  return run_pyr_dec(p, x, p->n, bp, n, (cudaStream_t)stream);
}

nsst_status nsst3_pyr_rec(nsst3_plan* p, const float* bp, float* x, int n, void* stream) {
  V3_TRY(check_call(p, n, bp, x));
  std::lock_guard<std::mutex> lk(p->mu);
  return run_pyr_rec(p, bp, x, p->n, n, (cudaStream_t)stream);
}

nsst_status nsst3_sh_dec(nsst3_plan* p, const float* bp, int level, float* coeffs, int n, void* stream) {
  V3_TRY(check_call(p, n, bp, coeffs));
  if (level < 0 || level >= p->L) return fail3(NSST_ERR_INVALID_ARG, "level must be a band-pass level");
  std::lock_guard<std::mutex> lk(p->mu);
  return run_sh_level(p, bp, level, nullptr, nullptr, coeffs, n, (cudaStream_t)stream);
}

nsst_status nsst3_sh_dec_thresh_rec(nsst3_plan* p, const float* bp, float* rec_bp, int n, const double* sigma,
                                    const double* T, const double* scalars, void* stream) {
  V3_TRY(check_call(p, n, bp, rec_bp));
  if (bp == rec_bp) return fail3(NSST_ERR_INVALID_ARG, "bp and rec_bp must not alias");
  std::lock_guard<std::mutex> lk(p->mu);
  const cudaStream_t st = (cudaStream_t)stream;
  V3_TRY(upload_th(p, n, sigma, T, scalars, st));
  return run_dec_thresh_rec(p, bp, rec_bp, n, p->th, st);
}

nsst_status nsst3_denoise_batch(nsst3_plan* p, const float* x, float* out, int n, const double* sigma,
                                const double* T, const double* scalars, void* stream) {
  V3_TRY(check_call(p, n, x, out));
  std::lock_guard<std::mutex> lk(p->mu);
  const cudaStream_t st = (cudaStream_t)stream;
  V3_TRY(upload_th(p, n, sigma, T, scalars, st));
  V3_TRY(run_pyr_dec(p, x, p->n, p->bp, n, st));
  p->masks_valid_n = 0;
  V3_TRY(run_dec_thresh_rec(p, p->bp, p->rbp, n, p->th, st, p->mask != nullptr));
  if (p->mask) p->masks_valid_n = n;
  return run_pyr_rec(p, p->rbp, out, p->n, n, st);
}

nsst_status nsst3_compute_scalars(nsst3_plan* p, uint64_t seed, double* out) {
  if (!p) return fail3(NSST_ERR_INVALID_ARG, "NULL plan");
  if (cudaSetDevice(p->device) != cudaSuccess) return fail3(NSST_ERR_CUDA, "cudaSetDevice failed");
  std::lock_guard<std::mutex> lk(p->mu);
  const size_t G = p->vol_elems;
  // seeded N(0,1) grid volume in FP64 (Box-Muller over a 64-bit Mersenne twister)
  std::mt19937_64 gen(seed);
  std::vector<float> noise(G);
  for (size_t i = 0; i < G; i += 2) {
    double u1 = ((gen() >> 11) + 0.5) * (1.0 / 9007199254740992.0);
    double u2 = ((gen() >> 11) + 0.5) * (1.0 / 9007199254740992.0);
    double r = std::sqrt(-2.0 * std::log(u1));
    noise[i] = (float)(r * std::cos(2 * M_PI * u2));
    if (i + 1 < G) noise[i + 1] = (float)(r * std::sin(2 * M_PI * u2));
  }
  size_t maxc = 0;
  for (int l = 0; l < p->L; l++) maxc = std::max(maxc, (size_t)p->lev[l].nb * p->lev[l].vol());
  float *dx = nullptr, *dc = nullptr;
  cudaError_t e = dev_alloc((void**)&dx, G * sizeof(float));
  if (e != cudaSuccess) return cuda_fail3(e, "scalar scratch");
  e = dev_alloc((void**)&dc, maxc * sizeof(float));
  if (e != cudaSuccess) {
    cudaFree(dx);
    return cuda_fail3(e, "scalar scratch");
  }
  std::vector<double> sc(p->nbands);
  nsst_status s = NSST_OK;
  std::vector<float> coeffs(maxc);
  e = cudaMemcpy(dx, noise.data(), G * sizeof(float), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) s = run_pyr_dec(p, dx, p->g, p->bp, 1, nullptr);
  for (int l = 0; l < p->L && e == cudaSuccess && s == NSST_OK; l++) {
    const nsst3_plan::Level& a = p->lev[l];
    s = run_sh_level(p, p->bp, l, nullptr, nullptr, dc, 1, nullptr);
    if (s != NSST_OK) break;
    e = cudaMemcpy(coeffs.data(), dc, (size_t)a.nb * a.vol() * sizeof(float), cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) break;
    // MAD / 0.6745 per band (NsstScalars.m:11-15), FP64, bands in parallel
    const int nt = std::min(host_threads3(), a.nb);
    std::vector<std::thread> th;
    for (int t = 0; t < nt; t++)
      th.emplace_back([&, t]() {
        std::vector<double> v(a.vol());
        auto median = [](std::vector<double>& x) {
          size_t m = x.size(), h = m / 2;
          std::nth_element(x.begin(), x.begin() + h, x.end());
          double hi = x[h];
          if (m % 2) return hi;
          double lo = *std::max_element(x.begin(), x.begin() + h);
          return 0.5 * (lo + hi);
        };
        for (int k = t; k < a.nb; k += nt) {
          const float* c = coeffs.data() + (size_t)k * a.vol();
          for (size_t i = 0; i < v.size(); i++) v[i] = c[i];
          const double med = median(v);
          for (size_t i = 0; i < v.size(); i++) v[i] = std::fabs((double)c[i] - med);
          sc[a.first_band + k] = median(v) / 0.6745;
        }
      });
    for (auto& t : th) t.join();
  }
  cudaFree(dx);
  cudaFree(dc);
  if (e != cudaSuccess) return cuda_fail3(e, "compute scalars");
  if (s != NSST_OK) return s;
  p->scalars = sc;
  p->has_scalars = true;
  if (out) std::copy(sc.begin(), sc.end(), out);
  return NSST_OK;
}

}  // extern "C"

// ---------------------------------------------------------------------------
// Differentiation of the 3-D denoise.  The hard threshold's subgradient keeps
// the forward pass's masks; the band-pass pyramid is a Parseval frame, so the
// adjoint of the decomposition is the reconstruction and vice versa; the
// adjoint of each 'same' convolution is a correlation (the conjugate filter
// spectrum) of the masked gradient placed back at offset 12.
// ---------------------------------------------------------------------------
extern "C" {

nsst_status nsst3_plan_enable_grad(nsst3_plan* p) {
  if (!p) return fail3(NSST_ERR_INVALID_ARG, "NULL plan");
  if (p->mask) return NSST_OK;
  if (cudaSetDevice(p->device) != cudaSuccess) return fail3(NSST_ERR_CUDA, "cudaSetDevice failed");
  std::lock_guard<std::mutex> lk(p->mu);
  p->mask_off.assign(p->nbands, 0);
  size_t bytes = 0;
  for (int b = 0; b < p->nbands; b++) {
    p->mask_off[b] = bytes;
    const nsst3_plan::Level& lv = p->lev[p->band_level[b]];
    bytes += mask_band_bytes(lv.m);
  }
  p->mask_bytes = bytes;
  void* m = nullptr;
  cudaError_t e = dev_alloc(&m, (size_t)p->B * bytes);
  if (e != cudaSuccess) return cuda_fail3(e, "mask buffer");
  p->mask = (uint8_t*)m;
  p->masks_valid_n = 0;
  return NSST_OK;
}

nsst_status nsst3_denoise_backward(nsst3_plan* p, const float* gy, float* gx, int n, void* stream) {
  V3_TRY(check_call(p, n, gy, gx));
  std::lock_guard<std::mutex> lk(p->mu);
  if (!p->mask) return fail3(NSST_ERR_INVALID_ARG, "gradients are not enabled on this plan");
  if (p->masks_valid_n != n)
    return fail3(NSST_ERR_INVALID_ARG, "no forward nsst3_denoise_batch of these n volumes since grad was enabled");
  const cudaStream_t st = (cudaStream_t)stream;
  // u = pyr_dec(zero-pad(gy)): the adjoint of crop + pyr_rec
  V3_TRY(run_pyr_dec(p, gy, p->n, p->rbp, n, st, true));
  // per level: bp_bar_l = sum_b corr(mask_b * u_l, f_b).  Per band pair,
  // Z = FFT3(place(mask_a u + i mask_b u)) from the box outwards (the zero
  // outside the box is never read), then S (+)= conj(C) .* Z in the last
  // pass; one inverse transform of S per level, cut to the box at 0.
  for (int l = 0; l < p->L; l++) {
    const nsst3_plan::Level& a = p->lev[l];
    const int* N = a.lc;
    const int* m = a.m;
    const int wp = v3_pitch(m[2]);
    const size_t cs = p->conv_elems;
    const int chunk = pair_chunk(p, a, n);
    for (int k0 = 0; k0 < a.npairs(); k0 += chunk) {
      const int pairs = std::min(chunk, a.npairs() - k0);
      V3Cols P1 = line_pass(0, p->Wk, a.pair(), N[1], wp, n, m[1], m[2], {kSameOff, m[0]}, {0, N[0]});
      P1.out_pair = a.pair() * n;
      P1.pairs = pairs;
      P1.nbands = a.nb - 2 * k0;
      P1.r1 = m[1], P1.r2 = m[2];
      P1.rsrc = p->rbp + a.bp_off;
      P1.r_stride = p->bp_floats;
      set_masks(p, P1, l, 2 * k0);
      V3_TRY(run_cols(p, N[0], -1, V3_LD_MASKED, V3_ST_CPLX, P1, pair_shares(m[1] * ((m[2] + 7) / 8) * n, pairs), st));
      V3_TRY(run_cols(p, N[1], -1, V3_LD_CPLX, V3_ST_CPLX, pair_cols(p, a, n, {kSameOff, m[1]}, {0, N[1]}), pairs, st));
      V3Pair P3 = pair_pass(p, a, k0, pairs, n);
      P3.S = p->Y;
      P3.s_item = cs;
      P3.first = k0 == 0;
      V3_CUDA(v3_ops(N[2])->pair(-1, P3, p->twid(N[2]), 1, st));
    }
    // the real part of S's inverse: that of its Hermitian part, on half spectra in the work buffer
    const int H = N[2] / 2 + 1, hp = v3_pitch(H);
    const size_t hs = (size_t)m[0] * N[1] * hp;
    V3Cols P = line_pass(0, p->Wk, hs, N[1], hp, n, N[1], H, {0, N[0]}, {0, m[0]});
    P.in = p->Y;
    P.in_item = cs;
    P.in_a = N[2], P.in_i = N[1] * N[2];
    P.sym_a = N[1], P.sym_z = N[2];
    V3_TRY(run_cols(p, N[0], +1, V3_LD_SYM, V3_ST_CPLX, P, 1, st));
    V3_TRY(run_cols(p, N[1], +1, V3_LD_CPLX, V3_ST_CPLX,
                    line_pass(1, p->Wk, hs, N[1], hp, n, m[0], H, {0, N[1]}, {0, m[1]}), 1, st));
    V3Real R;
    R.dst = p->bp + a.bp_off;
    R.spec = p->Wk;
    R.r_stride = p->bp_floats, R.spec_stride = hs;
    R.rows0 = m[0], R.rows1 = m[1], R.n2 = m[2];
    R.s1 = N[1], R.pitch = hp, R.line = N[2];
    R.scale = (float)(1.0 / (double)a.conv());
    V3_CUDA(v3_ops(N[2])->real(+1, R, p->twid(N[2]), n, st));
  }
  // the lowpass passes through unchanged
  const nsst3_plan::Level& lp = p->lev[p->L];
  V3_CUDA(cudaMemcpy2DAsync(p->bp + lp.bp_off, p->bp_floats * sizeof(float), p->rbp + lp.bp_off,
                            p->bp_floats * sizeof(float), lp.vol() * sizeof(float), n, cudaMemcpyDeviceToDevice, st));
  // pyr_rec (the adjoint of pyr_dec) to the full grid, then fold the edge padding
  V3_TRY(run_pyr_rec(p, p->bp, p->rbp, p->g, n, st));
  V3_CUDA(launch_fold_edge(p->rbp, p->vol_elems, gx, p->in_elems, (float*)p->Wk, 2 * p->vol_elems, n, p->n[0],
                           p->n[1], p->n[2], p->g[0], p->g[1], p->g[2], st));
  return NSST_OK;
}

}  // extern "C"
