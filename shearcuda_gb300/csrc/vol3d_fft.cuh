// FFT passes of the 3-D path: one pass transforms every line of a batch of
// volumes along one axis, with the work next to the transform fused into its
// loads and stores.
//
// A line of N = R1 R2 points is two register DFTs around one exchange through
// shared memory: thread (line s, j < R2) loads x[j + R2 r] (r < R1) from
// global memory straight into registers, takes the R1-point DFT, multiplies by
// W_N^(j k1) and writes row (k1, j) of the exchange; thread (line s, k1 < R1)
// reads the R2 values of row k1, takes the R2-point DFT and holds X[k1 + R1
// k2], which it stores straight from registers.  A CTA owns 8 lines and
// 8 max(R1, R2) threads (in whole warps), one butterfly per thread and stage.  What bounded the
// three- and four-pass shared-memory form of these passes was instruction
// issue (about 105 instructions per point: staging, then a shared-memory round
// trip, twiddles and index arithmetic per radix), not HBM (2.8-3.7 TB/s);
// two stages with the largest radices that fit in registers need about half.
//
// Real volumes are transformed as real: two real lines share one complex
// transform along axis 2, and axes 1 and 0 then see only the half spectrum
// (N/2 + 1 columns, rows padded to a multiple of four complex values).
//
// The directional stage multiplies one volume's spectrum by many filters: the
// band pairs of a level run inside a launch (grid z or a loop in the CTA), so a
// level costs three launches however many directions it has, the spectrum is
// read once per group of pairs and the band sum is kept in registers.
#pragma once
#include <cstdint>

#include "fft_core.cuh"
#include "internal.h"
#include "launch.cuh"

namespace nsst {

constexpr int kLines = 8;  // lines per CTA: 64-byte rows along z on the strided axes
// Shared memory share of the SM's L1 the passes run under: half, which holds
// their resident CTAs' exchanges and leaves the rest to the twiddles and the
// rows that several CTAs touch (4 x 128^3, us: 25 % 2225, 33 % 1657, 42 % 1645,
// 50 % 1572, 60 % 1587, 75 % 1628, 100 % 1873; left to the driver, which picks
// it per kernel, 1895).
constexpr int kV3Carveout = 50;

// Radices per length.  The larger second: every thread of a CTA then loads.
template <int N>
struct V3Radix;
#define V3_RADIX(n, a, b)                       \
  template <>                                   \
  struct V3Radix<n> {                           \
    static_assert((a) * (b) == (n), "radices"); \
    static constexpr int R1 = a, R2 = b;        \
  };
V3_RADIX(16, 4, 4)
V3_RADIX(22, 2, 11)
V3_RADIX(24, 4, 6)
V3_RADIX(32, 4, 8)
V3_RADIX(34, 2, 17)
V3_RADIX(44, 4, 11)
V3_RADIX(48, 6, 8)
V3_RADIX(56, 7, 8)
V3_RADIX(60, 6, 10)
V3_RADIX(64, 8, 8)
V3_RADIX(68, 4, 17)
V3_RADIX(72, 8, 9)
V3_RADIX(80, 8, 10)
V3_RADIX(88, 8, 11)
V3_RADIX(96, 8, 12)
V3_RADIX(100, 10, 10)
V3_RADIX(108, 9, 12)
V3_RADIX(128, 8, 16)
V3_RADIX(132, 11, 12)
V3_RADIX(136, 8, 17)
V3_RADIX(140, 10, 14)
V3_RADIX(144, 12, 12)
V3_RADIX(160, 10, 16)
V3_RADIX(192, 12, 16)
V3_RADIX(204, 12, 17)
V3_RADIX(216, 12, 18)
V3_RADIX(256, 16, 16)
#undef V3_RADIX

template <int N>
struct V3Cfg {
  static constexpr int R1 = V3Radix<N>::R1, R2 = V3Radix<N>::R2;
  static constexpr int T = (kLines * (R1 > R2 ? R1 : R2) + 31) / 32 * 32;
  // exchange rows (k1, j): an odd row length spreads the readers' rows (one per k1) over the banks
  static constexpr int P2 = R2 | 1;
  // strided axes: element (k1, j) of line s at (k1 P2 + j) 8 + s
  static constexpr int EX = R1 * P2 * kLines;
  // axis 2: line s starts at s SZ; SZ = R2 (mod 16) continues the writers' j across lines
  static constexpr int SZ = (R1 * P2 + 15) / 16 * 16 + R2 % 16;
  static constexpr int EXZ = SZ * kLines;
};

// Launch bound for at most `regs` registers a thread.
constexpr int v3_min_ctas(int threads, int regs) { return 65536 / (threads * regs); }
// Column passes that loop over the band pairs in the CTA.
constexpr bool v3_loops(int ld, int st) { return ld == V3_LD_MASKED || st == V3_ST_THRESH || st == V3_ST_PAIR; }

// First stage: load, R1-point DFTs, twiddles, exchange write at ex[row(k1, j)].
template <int N, int DIR, class Ld, class Row>
__device__ __forceinline__ void v3_stage1(float2* ex, const float2* __restrict__ tw, int j, const Ld& ld, const Row& row) {
  constexpr int R1 = V3Cfg<N>::R1, R2 = V3Cfg<N>::R2;
  float2 v[R1];
#pragma unroll
  for (int r = 0; r < R1; r++) v[r] = ld(r, j + R2 * r);
  Dft<R1, DIR>::run(v);
#pragma unroll
  for (int k1 = 0; k1 < R1; k1++) ex[row(k1, j)] = k1 ? tw_mul<DIR>(v[k1], tw, j * k1) : v[0];
}
// Second stage: exchange read, R2-point DFT, u[k2] = X[k1 + R1 k2].
template <int N, int DIR, class Row>
__device__ __forceinline__ void v3_stage2(const float2* ex, int k1, float2 (&u)[V3Cfg<N>::R2], const Row& row) {
  constexpr int R2 = V3Cfg<N>::R2;
#pragma unroll
  for (int q = 0; q < R2; q++) u[q] = ex[row(k1, q)];
  Dft<R2, DIR>::run(u);
}

// The pyramid's separable low-pass value at (x, y, z) of a half spectrum, or
// -1 outside the window's support (full axes mirror at nr - p, the half axis
// does not); PrySDdec_onestep.m:48-82.
__device__ __forceinline__ float v3_win(const float* __restrict__ v, int K, int nr, int p, bool half_axis) {
  if (p <= K) return __ldg(v + p);
  if (!half_axis && p >= nr - K) return __ldg(v + nr - p);
  return -1.0f;
}

// ---------------------------------------------------------------------------
// Axes 1 and 0: 8 lines adjacent along z.
// ---------------------------------------------------------------------------
// CTA x: line group (a, 8 z) and item, item fastest; y: band pair, or, for the
// loads and stores that loop over the pairs, the share of them.  G: thread
// groups of a CTA that take every G-th pair of a band sum.
template <int N, int DIR, int LD, int ST, int G = 1>
__global__ void __launch_bounds__(V3Cfg<N>::T * G, v3_loops(LD, ST) ? v3_min_ctas(V3Cfg<N>::T * G, 96) : 1)
    k_v3_cols(const V3Cols P, const float2* __restrict__ tw) {
  pdl_sync();
  using C = V3Cfg<N>;
  constexpr int R1 = C::R1, R2 = C::R2;
  constexpr bool kLoop = v3_loops(LD, ST);
  __shared__ float2 ex[kLoop && G == 1 ? 2 : G][C::EX];
  const int grp = G > 1 ? threadIdx.x / C::T : 0, tid = threadIdx.x - grp * C::T;
  const int item = blockIdx.x % P.items, g = blockIdx.x / P.items;
  const int zg = (P.zn + kLines - 1) / kLines;
  const int a = g / zg, z = (g % zg) * kLines + (tid & (kLines - 1));
  const int j = tid / kLines;
  const bool zin = z < P.zn;
  auto row = [&](int k1, int q) { return (k1 * C::P2 + q) * kLines + (tid & (kLines - 1)); };
  const size_t ibase = (size_t)item * P.in_item + (size_t)a * P.in_a + z;
  const size_t obase = (size_t)item * P.out_item + (size_t)a * P.out_a + z;

  if constexpr (!kLoop) {
    const float2* in = P.in + ibase + blockIdx.y * P.in_pair;
    float2* out = P.out + obase + blockIdx.y * P.out_pair;
    if (j < R2) {
      // window factors of this line's fixed coordinates (axis 0: y = a, z)
      float wyz = -1.f;
      if constexpr (LD == V3_LD_HP)
        if (zin) {
          const float b = v3_win(P.win.v1, P.win.K[1], P.win.nr[1], a, false);
          const float c = v3_win(P.win.v2, P.win.K[2], P.win.nr[2], z, true);
          wyz = b >= 0.f && c >= 0.f ? b * c : -1.f;
        }
      // the Hermitian mirror line of (a, z) in the full spectrum: (-a, -z)
      const float2* mir = nullptr;
      if constexpr (LD == V3_LD_SYM)
        mir = P.in + (size_t)item * P.in_item + (size_t)(a ? P.sym_a - a : 0) * P.in_a + (z ? P.sym_z - z : 0);
      auto ld = [&](int, int n) -> float2 {
        float2 v = make_float2(0.f, 0.f);
        if (!zin || n < P.in_lo || n >= P.in_lo + P.in_n) return v;
        v = in[(n - P.in_lo) * P.in_i];
        if constexpr (LD == V3_LD_HP) {
          // PrySDdec_onestep.m:110-125: Hp = sqrt(1 - Lf^2) X on the window's support
          const float w = v3_win(P.win.v0, P.win.K[0], P.win.nr[0], n, false);
          if (wyz >= 0.f && w >= 0.f) {
            const float lf = w * wyz;
            v = cscale(v, sqrtf(fmaxf(1.0f - lf * lf, 0.0f)));
          }
        }
        if constexpr (LD == V3_LD_SYM) {
          // the Hermitian part, whose transform is the real part of the transform
          const float2 m = mir[(n ? N - n : 0) * P.in_i];
          v = make_float2(0.5f * (v.x + m.x), 0.5f * (v.y - m.y));
        }
        return v;
      };
      v3_stage1<N, DIR>(ex[0], tw, j, ld, row);
    }
    __syncthreads();
    if (j < R1) {
      float2 u[R2];
      v3_stage2<N, DIR>(ex[0], j, u, row);
      if (!zin) return;
      float wyz = -1.f;
      const float2* lp = nullptr;
      if constexpr (ST == V3_ST_REC) {
        const float b = v3_win(P.win.v1, P.win.K[1], P.win.nr[1], a, false);
        const float c = v3_win(P.win.v2, P.win.K[2], P.win.nr[2], z, true);
        wyz = b >= 0.f && c >= 0.f ? b * c : -1.f;
        const int sy = a <= P.win.K[1] ? a : a - P.win.nr[1] + P.s1;
        lp = P.lp + (size_t)item * P.in_item + (size_t)sy * P.s2p + z;
      }
#pragma unroll
      for (int k2 = 0; k2 < R2; k2++) {
        const int n = j + R1 * k2;
        if (n < P.out_lo || n >= P.out_lo + P.out_n) continue;
        float2 v = u[k2];
        if constexpr (ST == V3_ST_REC) {
          // PrySDrec_onestep.m:96-119: sqrt(1 - Lf^2) Hp + Lf D^(N/2) Lp on the window's support
          const float w = v3_win(P.win.v0, P.win.K[0], P.win.nr[0], n, false);
          if (wyz >= 0.f && w >= 0.f) {
            const float lf = w * wyz, s = sqrtf(fmaxf(1.0f - lf * lf, 0.0f));
            const int sx = n <= P.win.K[0] ? n : n - P.win.nr[0] + P.s0;
            const float2 l = lp[(size_t)sx * P.s1 * P.s2p];
            v = make_float2(s * v.x + lf * P.scale * l.x, s * v.y + lf * P.scale * l.y);
          }
        }
        out[(n - P.out_lo) * P.out_i] = v;
      }
    }
    return;
  }

  // ------- launches that loop over the band pairs of the chunk -------
  // box offset of this line: real element i of the line at rbase + i r_i
  const size_t rbase = (size_t)item * P.r_stride + (size_t)a * P.r2 + z;
  const int r_i = P.r1 * P.r2;
  if constexpr (LD == V3_LD_MASKED) {
    // u of the line, once; per pair the two bands' keep bits select it
    float u0[R1];
    if (j < R2) {
#pragma unroll
      for (int r = 0; r < R1; r++) {
        const int n = j + R2 * r - P.in_lo;
        u0[r] = zin && n >= 0 && n < P.in_n ? P.rsrc[rbase + (size_t)n * r_i] : 0.f;
      }
    }
    int it = 0;
    for (int k = blockIdx.y; k < P.pairs; k += gridDim.y, it ^= 1) {
      const uint8_t* ma = P.mask + item * P.m_stride + (size_t)(2 * k) * P.m_band;
      const uint8_t* mb = 2 * k + 1 < P.nbands ? ma + P.m_band : nullptr;
      const unsigned bit = 1u << (z & 7);
      if (j < R2) {
        auto ld = [&](int r, int nn) -> float2 {
          const int n = nn - P.in_lo;
          float2 v = make_float2(0.f, 0.f);
          if (zin && n >= 0 && n < P.in_n) {
            const size_t b = (((size_t)n * P.r1 + a) * P.m_r2 + z) >> 3;
            v.x = ma[b] & bit ? u0[r] : 0.f;
            if (mb) v.y = mb[b] & bit ? u0[r] : 0.f;
          }
          return v;
        };
        v3_stage1<N, DIR>(ex[it], tw, j, ld, row);
      }
      __syncthreads();
      if (j < R1) {
        float2 u[R2];
        v3_stage2<N, DIR>(ex[it], j, u, row);
        float2* out = P.out + obase + (size_t)k * P.out_pair;
        if (zin) {
#pragma unroll
          for (int k2 = 0; k2 < R2; k2++) {
            const int n = j + R1 * k2;
            if (n >= P.out_lo && n < P.out_lo + P.out_n) out[(n - P.out_lo) * P.out_i] = u[k2];
          }
        }
      }
    }
  } else {
    const unsigned members = __ballot_sync(0xffffffffu, j < R1);
    // The band sum adds the pairs in their order whatever the chunks and groups
    // are, so that a batch and its volumes one by one give the same bits.
    float acc[R2];
#pragma unroll
    for (int k2 = 0; k2 < R2; k2++) {
      const int n = j + R1 * k2 - P.out_lo;
      acc[k2] = ST == V3_ST_THRESH && !P.first && grp == 0 && j < R1 && zin && n >= 0 && n < P.out_n
                    ? P.rdst[rbase + (size_t)n * r_i]
                    : 0.f;
    }
    float* part = reinterpret_cast<float*>(ex[grp]);  // G > 1: the group's summands of this round
    int it = 0;
    for (int k0 = blockIdx.y * G; k0 < P.pairs; k0 += gridDim.y * G) {
      const int k = k0 + grp;
      const bool live = G == 1 || k < P.pairs;
      float2* x = ex[G == 1 ? it : grp];
      const float2* in = P.in + ibase + (size_t)k * P.in_pair;
      if (live && j < R2) {
        auto ld = [&](int, int n) -> float2 {
          return zin && n >= P.in_lo && n < P.in_lo + P.in_n ? in[(n - P.in_lo) * P.in_i] : make_float2(0.f, 0.f);
        };
        v3_stage1<N, DIR>(x, tw, j, ld, row);
      }
      __syncthreads();
      float2 u[R2];
      if (live && j < R1) {
        v3_stage2<N, DIR>(x, j, u, row);
        const bool has_b = 2 * k + 1 < P.nbands;
        float ta = -1.f, tb = -1.f;
        if constexpr (ST == V3_ST_THRESH)
          if (P.th) {
            ta = __ldg(P.th + (size_t)item * P.nb_item + 2 * k);
            if (has_b) tb = __ldg(P.th + (size_t)item * P.nb_item + 2 * k + 1);
          }
#pragma unroll
        for (int k2 = 0; k2 < R2; k2++) {
          const int n = j + R1 * k2 - P.out_lo;
          const bool st = zin && n >= 0 && n < P.out_n;
          const float ca = u[k2].x * P.scale, cb = has_b ? u[k2].y * P.scale : 0.f;
          if constexpr (ST == V3_ST_THRESH) {
            // ThresholdShCoeff.m:7 zeroes |c| <= t
            const bool ka = st && !(fabsf(ca) <= ta), kb = st && has_b && !(fabsf(cb) <= tb);
            u[k2].x = (ka ? ca : 0.f) + (kb ? cb : 0.f);
            if (grp == 0) acc[k2] += u[k2].x;
            if (P.mask) {  // uniform across the grid; the eight lanes of a line group give one byte
              const unsigned ba = __ballot_sync(members, ka), bb = __ballot_sync(members, kb);
              if (n >= 0 && n < P.out_n && (tid & 7) == 0) {
                uint8_t* b = P.mask + item * P.m_stride + (size_t)(2 * k) * P.m_band +
                             ((((size_t)n * P.r1 + a) * P.m_r2 + z) >> 3);
                *b = (uint8_t)(ba >> (tid & 24));
                if (has_b) b[P.m_band] = (uint8_t)(bb >> (tid & 24));
              }
            }
          } else if (st) {
            float* c = P.rdst + rbase + (size_t)n * r_i + (size_t)(2 * k) * P.band_stride;
            c[0] = ca;
            if (has_b) c[P.band_stride] = cb;
          }
        }
      }
      if constexpr (G > 1) {
        __syncthreads();  // every thread has read its group's exchange
        if (grp > 0 && live && j < R1) {
#pragma unroll
          for (int k2 = 0; k2 < R2; k2++) part[k2 * (R1 * kLines) + tid] = u[k2].x;
        }
        __syncthreads();
        if (grp == 0 && j < R1) {
          for (int q = 1; q < G && k0 + q < P.pairs; q++) {
            const float* pq = reinterpret_cast<const float*>(ex[q]);
#pragma unroll
            for (int k2 = 0; k2 < R2; k2++) acc[k2] += pq[k2 * (R1 * kLines) + tid];
          }
        }
        __syncthreads();
      }
      it ^= 1;
    }
    if constexpr (ST == V3_ST_THRESH) {
      if (grp == 0 && j < R1 && zin) {
#pragma unroll
        for (int k2 = 0; k2 < R2; k2++) {
          const int n = j + R1 * k2 - P.out_lo;
          if (n < 0 || n >= P.out_n) continue;
          float* d = P.rdst + rbase + (size_t)n * r_i;
          *d = acc[k2];
        }
      }
    }
  }
}

// ---------------------------------------------------------------------------
// Axis 2: 8 lines of consecutive rows.
// ---------------------------------------------------------------------------
// Real rows -> half spectra: rows 2 s and 2 s + 1 are the real and imaginary
// part of complex line s; X[k], X[N - k] separate into the two rows' spectra.
template <int N>
__global__ void __launch_bounds__(V3Cfg<N>::T) k_v3_real_fwd(const V3Real P, const float2* __restrict__ tw) {
  pdl_sync();
  using C = V3Cfg<N>;
  constexpr int R1 = C::R1, R2 = C::R2, H = N / 2 + 1, NP = N + 1;
  __shared__ float2 ex[C::EXZ];
  __shared__ float2 xs[kLines * NP];
  const int rows = P.rows0 * P.rows1, row0 = blockIdx.x * 2 * kLines;
  const float* src = P.src + blockIdx.y * P.r_stride;
  float2* dst = P.spec + blockIdx.y * P.spec_stride;
  auto at = [&](int s) { return [s](int k1, int q) { return s * C::SZ + k1 * C::P2 + q; }; };
  {
    const int j = threadIdx.x % R2, s = threadIdx.x / R2;
    if (s < kLines) {
      // source row of line row r: edge rows repeat the last one of the volume
      auto src_row = [&](int r) -> const float* {
        if (r >= rows) return nullptr;
        int x = r / P.rows1, y = r % P.rows1;
        if (x >= P.n0 || y >= P.n1) {
          if (!P.edge) return nullptr;
          x = min(x, P.n0 - 1), y = min(y, P.n1 - 1);
        }
        return src + ((size_t)x * P.n1 + y) * P.n2;
      };
      const float *ra = src_row(row0 + 2 * s), *rb = src_row(row0 + 2 * s + 1);
      auto ld = [&](int, int n) -> float2 {
        if (n >= P.n2) {
          if (!P.edge || n >= P.line) return make_float2(0.f, 0.f);
          n = P.n2 - 1;
        }
        return make_float2(ra ? __ldg(ra + n) : 0.f, rb ? __ldg(rb + n) : 0.f);
      };
      v3_stage1<N, -1>(ex, tw, j, ld, at(s));
    }
  }
  __syncthreads();
  {
    const int k1 = threadIdx.x % R1, s = threadIdx.x / R1;
    if (s < kLines) {
      float2 u[R2];
      v3_stage2<N, -1>(ex, k1, u, at(s));
#pragma unroll
      for (int k2 = 0; k2 < R2; k2++) xs[s * NP + k1 + R1 * k2] = u[k2];
    }
  }
  __syncthreads();
  for (int e = threadIdx.x; e < kLines * H; e += C::T) {
    const int s = e / H, k = e - s * H, r = row0 + 2 * s;
    if (r >= rows) break;
    const float2 p = xs[s * NP + k], q = xs[s * NP + (k ? N - k : 0)];
    const int x = r / P.rows1, y = r % P.rows1;
    dst[((size_t)x * P.s1 + y) * P.pitch + k] = make_float2(0.5f * (p.x + q.x), 0.5f * (p.y - q.y));
    if (r + 1 < rows) {
      const int x1 = (r + 1) / P.rows1, y1 = (r + 1) % P.rows1;
      dst[((size_t)x1 * P.s1 + y1) * P.pitch + k] = make_float2(0.5f * (p.y + q.y), 0.5f * (q.x - p.x));
    }
  }
}

// Half spectra -> real rows (times scale), two per complex line: X = A + i B
// with A[N - k] = conj(A[k]) and the imaginary parts at 0 and N/2 dropped.
template <int N>
__global__ void __launch_bounds__(V3Cfg<N>::T) k_v3_real_inv(const V3Real P, const float2* __restrict__ tw) {
  pdl_sync();
  using C = V3Cfg<N>;
  constexpr int R1 = C::R1, R2 = C::R2;
  __shared__ float2 ex[C::EXZ];
  const int rows = P.rows0 * P.rows1, row0 = blockIdx.x * 2 * kLines;
  const float2* spec = P.spec + blockIdx.y * P.spec_stride;
  float* dst = P.dst + blockIdx.y * P.r_stride;
  auto at = [&](int s) { return [s](int k1, int q) { return s * C::SZ + k1 * C::P2 + q; }; };
  {
    const int j = threadIdx.x % R2, s = threadIdx.x / R2;
    if (s < kLines) {
      auto spec_row = [&](int r) -> const float2* {
        return r < rows ? spec + ((size_t)(r / P.rows1) * P.s1 + r % P.rows1) * P.pitch : nullptr;
      };
      const float2 *ra = spec_row(row0 + 2 * s), *rb = spec_row(row0 + 2 * s + 1);
      auto ld = [&](int, int n) -> float2 {
        const int m = 2 * n > N ? N - n : n;
        float2 A = ra ? ra[m] : make_float2(0.f, 0.f), B = rb ? rb[m] : make_float2(0.f, 0.f);
        if (m == 0 || 2 * m == N) A.y = B.y = 0.f;
        if (m != n) A.y = -A.y, B.y = -B.y;
        return make_float2(A.x - B.y, A.y + B.x);
      };
      v3_stage1<N, +1>(ex, tw, j, ld, at(s));
    }
  }
  __syncthreads();
  const int k1 = threadIdx.x % R1, s = threadIdx.x / R1;
  const int r = row0 + 2 * s;
  if (s >= kLines || r >= rows) return;
  float2 u[R2];
  v3_stage2<N, +1>(ex, k1, u, at(s));
  float* da = dst + (size_t)r * P.n2;  // output rows are contiguous: rows0 x rows1 x n2
#pragma unroll
  for (int k2 = 0; k2 < R2; k2++) {
    const int n = k1 + R1 * k2;
    if (n < P.n2) {
      da[n] = u[k2].x * P.scale;
      if (r + 1 < rows) da[P.n2 + n] = u[k2].y * P.scale;
    }
  }
}

// Directional analysis along z: per band pair of the chunk Y .* C, inverse
// transform, the box's z kept.  Y is read once for all pairs (its upper half
// is the conjugate mirror of the stored half).  CTA x: 8 rows and item, item
// fastest, so the items share each filter row through L2; y: share of the pairs.
template <int N>
__global__ void __launch_bounds__(V3Cfg<N>::T, v3_min_ctas(V3Cfg<N>::T, 112)) k_v3_pair_inv(const V3Pair P, const float2* __restrict__ tw) {
  pdl_sync();
  using C = V3Cfg<N>;
  constexpr int R1 = C::R1, R2 = C::R2;
  __shared__ float2 ex[2][C::EXZ];
  const int item = blockIdx.x % P.items, row0 = blockIdx.x / P.items * kLines;
  const int rows = P.N0 * P.N1;
  auto at = [&](int s) { return [s](int k1, int q) { return s * C::SZ + k1 * C::P2 + q; }; };
  const int j = threadIdx.x % R2, s1 = threadIdx.x / R2;
  const bool l1 = s1 < kLines && row0 + s1 < rows;
  const int k1 = threadIdx.x % R1, s2 = threadIdx.x / R1;
  const bool l2 = s2 < kLines && row0 + s2 < rows;
  float2 y[R1];
  const float2* spec = nullptr;
  if (l1) {
    const int r = row0 + s1, x0 = r / P.N1, x1 = r % P.N1;
    const float2* lo = P.Y + (size_t)item * P.y_item + (size_t)r * P.pitch;
    const float2* hi = P.Y + (size_t)item * P.y_item +
                       ((size_t)(x0 ? P.N0 - x0 : 0) * P.N1 + (x1 ? P.N1 - x1 : 0)) * P.pitch;
#pragma unroll
    for (int q = 0; q < R1; q++) {
      const int n = j + R2 * q;
      y[q] = 2 * n > N ? cconj(hi[N - n]) : lo[n];
    }
    spec = P.spec + (size_t)r * N + j;
  }
  // the next pair's filter row is loaded while this pair's second stage runs
  float2 c[R1];
  auto fetch = [&](int k) {
    if (l1 && k < P.pairs) {
#pragma unroll
      for (int q = 0; q < R1; q++) c[q] = __ldg(spec + (size_t)k * rows * N + R2 * q);
    }
  };
  fetch(blockIdx.y);
  int it = 0;
  for (int k = blockIdx.y; k < P.pairs; k += gridDim.y, it ^= 1) {
    if (l1) v3_stage1<N, +1>(ex[it], tw, j, [&](int q, int) { return cmul(y[q], c[q]); }, at(s1));
    fetch(k + gridDim.y);
    __syncthreads();
    if (l2) {
      float2 u[R2];
      v3_stage2<N, +1>(ex[it], k1, u, at(s2));
      float2* w = P.W + (size_t)k * P.w_pair + (size_t)item * P.w_item + (size_t)(row0 + s2) * P.wpitch;
#pragma unroll
      for (int k2 = 0; k2 < R2; k2++) {
        const int n = k1 + R1 * k2 - P.z_lo;
        if (n >= 0 && n < P.z_n) w[n] = u[k2];
      }
    }
  }
}

// Its adjoint: per band pair of the chunk the box's z, forward transform,
// S (+)= conj(C) .* Z summed over the pairs in registers.
template <int N>
__global__ void __launch_bounds__(V3Cfg<N>::T, v3_min_ctas(V3Cfg<N>::T, 128)) k_v3_pair_fwd(const V3Pair P, const float2* __restrict__ tw) {
  pdl_sync();
  using C = V3Cfg<N>;
  constexpr int R1 = C::R1, R2 = C::R2;
  __shared__ float2 ex[2][C::EXZ];
  const int item = blockIdx.x % P.items, row0 = blockIdx.x / P.items * kLines;
  const int rows = P.N0 * P.N1;
  auto at = [&](int s) { return [s](int k1, int q) { return s * C::SZ + k1 * C::P2 + q; }; };
  const int j = threadIdx.x % R2, s1 = threadIdx.x / R2;
  const bool l1 = s1 < kLines && row0 + s1 < rows;
  const int k1 = threadIdx.x % R1, s2 = threadIdx.x / R1;
  const bool l2 = s2 < kLines && row0 + s2 < rows;
  float2 acc[R2];
#pragma unroll
  for (int k2 = 0; k2 < R2; k2++)
    acc[k2] = l2 && !P.first ? P.S[(size_t)item * P.s_item + (size_t)(row0 + s2) * N + k1 + R1 * k2] : make_float2(0.f, 0.f);
  // the next pair's row is loaded while this pair's second stage runs
  float2 v[R1];
  auto fetch = [&](int k) {
    if (l1 && k < P.pairs) {
      const float2* w = P.W + (size_t)k * P.w_pair + (size_t)item * P.w_item + (size_t)(row0 + s1) * P.wpitch;
#pragma unroll
      for (int q = 0; q < R1; q++) {
        const int n = j + R2 * q - P.z_lo;
        v[q] = n >= 0 && n < P.z_n ? w[n] : make_float2(0.f, 0.f);
      }
    }
  };
  fetch(0);
  for (int k = 0; k < P.pairs; k++) {
    if (l1) v3_stage1<N, -1>(ex[k & 1], tw, j, [&](int q, int) { return v[q]; }, at(s1));
    fetch(k + 1);
    __syncthreads();
    if (l2) {
      float2 u[R2];
      v3_stage2<N, -1>(ex[k & 1], k1, u, at(s2));
      const float2* c = P.spec + (size_t)k * rows * N + (size_t)(row0 + s2) * N + k1;
#pragma unroll
      for (int k2 = 0; k2 < R2; k2++) acc[k2] = cadd(acc[k2], cmulc(u[k2], __ldg(c + R1 * k2)));
    }
  }
  if (!l2) return;
  float2* S = P.S + (size_t)item * P.s_item + (size_t)(row0 + s2) * N + k1;
#pragma unroll
  for (int k2 = 0; k2 < R2; k2++) S[R1 * k2] = acc[k2];
}

// ---------------------------------------------------------------------------
// Launchers of one length.
// ---------------------------------------------------------------------------
template <int N, bool PYR, bool CONV>
struct V3Launch {
  static constexpr int T = V3Cfg<N>::T;
  static cudaError_t real(int dir, const V3Real& P, const float2* tw, int items, cudaStream_t st) {
    const dim3 grid((unsigned)((P.rows0 * P.rows1 + 2 * kLines - 1) / (2 * kLines)), (unsigned)items);
    count_launch();
    if (dir < 0)
      launch_pdl(k_v3_real_fwd<N>, grid, T, 0, st, P, tw);
    else
      launch_pdl(k_v3_real_inv<N>, grid, T, 0, st, P, tw);
    return cudaGetLastError();
  }
  static cudaError_t cols(int dir, int ld, int st_mode, const V3Cols& P, const float2* tw, int npairs, cudaStream_t st) {
    const dim3 grid((unsigned)(P.an * ((P.zn + kLines - 1) / kLines) * P.items), (unsigned)npairs);
    count_launch();
    // A band sum over few lines: its CTAs' chain of pairs is the time, so four
    // groups of threads share it; with more CTAs the groups only wait for one another.
    if constexpr (CONV && N <= 108)
      if (st_mode == V3_ST_THRESH && P.pairs >= 4 && grid.x <= (unsigned)(2 * sm_count())) {
        launch_pdl(k_v3_cols<N, 1, V3_LD_CPLX, V3_ST_THRESH, 4>, grid, 4 * T, 0, st, P, tw);
        return cudaGetLastError();
      }
#define V3_COLS(cond, d, l, s)                          \
  if constexpr (cond)                                   \
    if (dir == d && ld == l && st_mode == s) {          \
      launch_pdl(k_v3_cols<N, d, l, s>, grid, T, 0, st, P, tw); \
      return cudaGetLastError();                        \
    }
    V3_COLS(true, -1, V3_LD_CPLX, V3_ST_CPLX)
    V3_COLS(true, 1, V3_LD_CPLX, V3_ST_CPLX)
    V3_COLS(PYR, 1, V3_LD_HP, V3_ST_CPLX)
    V3_COLS(PYR, -1, V3_LD_CPLX, V3_ST_REC)
    V3_COLS(CONV, 1, V3_LD_SYM, V3_ST_CPLX)
    V3_COLS(CONV, -1, V3_LD_MASKED, V3_ST_CPLX)
    V3_COLS(CONV, 1, V3_LD_CPLX, V3_ST_THRESH)
    V3_COLS(CONV, 1, V3_LD_CPLX, V3_ST_PAIR)
#undef V3_COLS
    return cudaErrorInvalidValue;
  }
  static cudaError_t pair(int dir, const V3Pair& P, const float2* tw, int shares, cudaStream_t st) {
    if constexpr (CONV) {
      const dim3 grid((unsigned)((P.N0 * P.N1 + kLines - 1) / kLines * P.items), (unsigned)shares);
      count_launch();
      if (dir > 0)
        launch_pdl(k_v3_pair_inv<N>, grid, T, 0, st, P, tw);
      else
        launch_pdl(k_v3_pair_fwd<N>, grid, T, 0, st, P, tw);
      return cudaGetLastError();
    }
    return cudaErrorInvalidValue;
  }
  // One shared-memory carve-out for every pass: with dependent launches the
  // SMs do not drain between kernels, and a kernel placed under another's
  // carve-out would keep the occupancy that it allows.
  static cudaError_t prepare() {
    cudaError_t e = cudaSuccess;
    auto one = [&](auto kernel) {
      if (e == cudaSuccess)
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, kV3Carveout);
    };
    one(k_v3_real_fwd<N>);
    one(k_v3_real_inv<N>);
    one(k_v3_cols<N, -1, V3_LD_CPLX, V3_ST_CPLX>);
    one(k_v3_cols<N, 1, V3_LD_CPLX, V3_ST_CPLX>);
    if constexpr (PYR) {
      one(k_v3_cols<N, 1, V3_LD_HP, V3_ST_CPLX>);
      one(k_v3_cols<N, -1, V3_LD_CPLX, V3_ST_REC>);
    }
    if constexpr (CONV) {
      one(k_v3_cols<N, 1, V3_LD_SYM, V3_ST_CPLX>);
      one(k_v3_cols<N, -1, V3_LD_MASKED, V3_ST_CPLX>);
      one(k_v3_cols<N, 1, V3_LD_CPLX, V3_ST_THRESH>);
      one(k_v3_cols<N, 1, V3_LD_CPLX, V3_ST_PAIR>);
      one(k_v3_pair_inv<N>);
      one(k_v3_pair_fwd<N>);
      if constexpr (N <= 108) one(k_v3_cols<N, 1, V3_LD_CPLX, V3_ST_THRESH, 4>);
    }
    return e;
  }
  static V3Ops ops() { return {real, cols, pair, prepare, PYR, CONV}; }
};

}  // namespace nsst
