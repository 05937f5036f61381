// FFT convolution (the reference's large-filter path,
// generator/DynamicConvolutionGenerator.scala:322-480 with the expanded shape
// of generator/FFTConvolutionUtils.scala:38-97), hand-written in FP32:
//
//   y = trim( IFFT2( FFT2(expand(x)) * G ) ),   G = FFT2(g) / (Fr * Fc/2)
//
// where expand(x) is the Fr x Fc power-of-two grid holding x with its border
// extension (Zero / Clamp / Cyclic) below/right of the field and, wrapped,
// above/left of it, and g holds the (flipped for convolution) filter centred
// at the origin with cyclic wrap-around.  This equals the direct convolution
// with the same border policy at every output point.
//
// Three kernels per run:
//   fft_rows_r2c   expanded rows (Fc reals packed as N = Fc/2 complex): N-point
//                  FFT, then the even/odd split to the Fc/2 + 1 non-negative
//                  frequencies.  Only the grid rows that hold the field and the
//                  border its outputs can read are transformed (the others are
//                  zero or are never read); the R rows of a dynamic filter go
//                  along in the same launch;
//   fft_cols       blocks of spectrum columns: Fr-point FFT down each
//                  column, times G, inverse FFT (before it, for a dynamic
//                  filter, a launch that makes G: forward FFT and scaling only);
//   fft_rows_c2r   output rows: inverse of the split, N-point inverse FFT,
//                  unpacked and trimmed to the field.
// Each FFT is a Stockham autosort in radix-16 passes (radix 2/4/8 for the
// last): every thread keeps 16 complex values in registers and does one
// 16-point (or 16/R R-point) DFT per pass, so an N-point FFT takes
// ceil(log2 N / 4) passes and one shared-memory exchange fewer: the last pass
// leaves thread tt the elements tt + m T, which are what the first pass of the
// inverse takes and what a column or an output row stores.  Shared-memory
// sequences are padded by one element every 16 so the strided exchanges stay
// free of bank conflicts.  Twiddles are computed in FP64 on the host and stored
// as float2.
#include <cmath>
#include <complex>
#include <vector>

#include "cct_internal.h"
#include "fft_conv.h"
#include "sm100_util.cuh"
#include "tile_common.cuh"

namespace cct {
namespace {

// Threads of a row CTA (as many rows as they hold) and of a column CTA: four
// columns, or more while that leaves fewer than 64 threads; two of 4096 rows, so
// that two CTAs share an SM (2048x2048 clamp: 171 us with one of 1024 threads, 160).
__host__ __device__ constexpr int row_threads(int N) { return N / 16 > 64 ? N / 16 : 64; }
__host__ __device__ constexpr int col_width(int Fr) {
  return Fr == 4096 ? 2 : Fr / 16 * 4 >= 64 ? 4 : 64 / (Fr / 16);
}
// Column threads to keep resident per SM: 1024 (64 registers a thread, a few
// spilled) for columns of more than 1024 rows, 512 and no spills up to that (31x31 cyclic
// or clamp, us a convolution with 1024 / 512: 512x512 20.8 / 18.7, 1024x2048 45.9 / 38.0, 480x640
// 26.6 / 23.7; many CTAs: 16 planes of 1024x1024 152 / 148, 64 of 480x640 275 / 265, 8 of
// 512x4096 clamp 412 / 417; 2048x2048, 1024 against 512, 56.7 / 62.0).
__host__ __device__ constexpr int col_residency(int Fr) { return Fr <= 1024 ? 512 : 1024; }
// Shared-memory stride of a column in complex values: a warp holds 32/CW
// consecutive elements of each of CW columns, so a stride of 32/CW (mod 16)
// spreads its 32 values evenly over the banks.
__host__ __device__ constexpr int col_stride(int Fr) {
  const int base = Fr + Fr / 16, cw = col_width(Fr), want = cw >= 32 ? 1 : 32 / cw;
  return base + ((want - base) % 16 + 16) % 16;
}

__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float2 conjf2(float2 a) { return make_float2(a.x, -a.y); }
__device__ __forceinline__ float2 cscale(float2 a, float s) { return make_float2(a.x * s, a.y * s); }
__device__ __forceinline__ int pad16(int i) { return i + (i >> 4); }

// Spectrum layout of one plane (Fr rows x ld columns, ld a multiple of 4):
// blocks of 4 columns, each block all Fr rows of its 4 columns (32 bytes per
// row).  A row pass reads and writes 32-byte row segments; a column pass
// reads its columns as one contiguous stretch per block.
__host__ __device__ __forceinline__ size_t spec_index(int r, int c, int Fr) {
  return ((size_t)(c >> 2) * Fr + r) * 4 + (c & 3);
}

// multiply by -i (forward transform) or +i (inverse)
template <bool INV>
__device__ __forceinline__ float2 rot(float2 a) {
  return INV ? make_float2(-a.y, a.x) : make_float2(a.y, -a.x);
}
// multiply by exp(-+ 2 pi i j / 16): forward uses the minus sign
template <bool INV>
__device__ __forceinline__ float2 w16(float2 a, float c, float s) {
  return cmul(a, make_float2(c, INV ? s : -s));
}

template <bool INV>
__device__ __forceinline__ void dft2(float2 *v) {
  const float2 a = v[0];
  v[0] = cadd(a, v[1]);
  v[1] = csub(a, v[1]);
}

template <bool INV>
__device__ __forceinline__ void dft4(float2 &a0, float2 &a1, float2 &a2, float2 &a3) {
  const float2 t0 = cadd(a0, a2), t1 = csub(a0, a2), t2 = cadd(a1, a3), t3 = rot<INV>(csub(a1, a3));
  a0 = cadd(t0, t2);
  a2 = csub(t0, t2);
  a1 = cadd(t1, t3);
  a3 = csub(t1, t3);
}

template <bool INV>
__device__ __forceinline__ void dft8(float2 *v) {
  constexpr float h = 0.70710678118654752f;  // cos(pi/4)
  float2 e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6];
  float2 o0 = v[1], o1 = v[3], o2 = v[5], o3 = v[7];
  dft4<INV>(e0, e1, e2, e3);
  dft4<INV>(o0, o1, o2, o3);
  o1 = w16<INV>(o1, h, h);   // W8^1
  o2 = rot<INV>(o2);         // W8^2
  o3 = w16<INV>(o3, -h, h);  // W8^3
  v[0] = cadd(e0, o0);
  v[4] = csub(e0, o0);
  v[1] = cadd(e1, o1);
  v[5] = csub(e1, o1);
  v[2] = cadd(e2, o2);
  v[6] = csub(e2, o2);
  v[3] = cadd(e3, o3);
  v[7] = csub(e3, o3);
}

template <bool INV>
__device__ __forceinline__ void dft16(float2 *v) {
  constexpr float c1 = 0.92387953251128674f, s1 = 0.38268343236508978f;  // cos, sin(pi/8)
  constexpr float h = 0.70710678118654752f;
  // n = 4p + q: 4-point DFTs over p, twiddles W16^(q k1), 4-point DFTs over q
#pragma unroll
  for (int q = 0; q < 4; ++q) dft4<INV>(v[q], v[q + 4], v[q + 8], v[q + 12]);
  v[5] = w16<INV>(v[5], c1, s1);     // q=1 k1=1
  v[9] = w16<INV>(v[9], h, h);       // q=1 k1=2
  v[13] = w16<INV>(v[13], s1, c1);   // q=1 k1=3
  v[6] = w16<INV>(v[6], h, h);       // q=2 k1=1
  v[10] = rot<INV>(v[10]);           // q=2 k1=2
  v[14] = w16<INV>(v[14], -h, h);    // q=2 k1=3
  v[7] = w16<INV>(v[7], s1, c1);     // q=3 k1=1
  v[11] = w16<INV>(v[11], -h, h);    // q=3 k1=2
  v[15] = w16<INV>(v[15], -c1, -s1); // q=3 k1=3 (W16^9)
#pragma unroll
  for (int k1 = 0; k1 < 4; ++k1) dft4<INV>(v[4 * k1], v[4 * k1 + 1], v[4 * k1 + 2], v[4 * k1 + 3]);
  // X[k1 + 4 k2] sits in v[4 k1 + k2]: transpose to natural order
  float2 t[16];
#pragma unroll
  for (int m = 0; m < 16; ++m) t[m] = v[4 * (m & 3) + (m >> 2)];
#pragma unroll
  for (int m = 0; m < 16; ++m) v[m] = t[m];
}

template <int R, bool INV>
__device__ __forceinline__ void dft(float2 *v) {
  if (R == 2) dft2<INV>(v);
  if (R == 4) dft4<INV>(v[0], v[1], v[2], v[3]);
  if (R == 8) dft8<INV>(v);
  if (R == 16) dft16<INV>(v);
}

// One Stockham pass of radix R over an N-point sequence (T = N/16 threads,
// thread tt owns butterflies j = tt + q*T, q < 16/R): twiddles
// w_(Ns R)^(m k) on input m (k = j mod Ns), then the R-point DFT.
template <int R, bool INV>
__device__ __forceinline__ void pass_compute(float2 (&v)[16], int N, int Ns, int T, int tt,
                                             const float2 *__restrict__ tw) {
#pragma unroll
  for (int q = 0; q < 16 / R; ++q) {
    const int j = tt + q * T, k = j & (Ns - 1);
    if (k) {
      // w^m for m < R from two table reads (w and w^4) and at most two
      // products (w^m = (w^4)^a w^b, m = 4a + b), instead of R-1 scattered
      // reads per butterfly
      const int step = N / (Ns * R);
      float2 p[4], p4[4];
      p[0] = make_float2(1.0f, 0.0f);
      p[1] = __ldg(tw + k * step);
      if (R > 2) {
        p[2] = cmul(p[1], p[1]);
        p[3] = cmul(p[2], p[1]);
      }
      if (R > 4) {
        p4[0] = make_float2(1.0f, 0.0f);
        p4[1] = __ldg(tw + 4 * k * step);
        p4[2] = cmul(p4[1], p4[1]);
        p4[3] = cmul(p4[2], p4[1]);
      }
#pragma unroll
      for (int m = 1; m < R; ++m) {
        const float2 w = (m < 4) ? p[m] : ((m & 3) ? cmul(p4[m >> 2], p[m & 3]) : p4[m >> 2]);
        v[q * R + m] = cmul(v[q * R + m], INV ? conjf2(w) : w);
      }
    }
    dft<R, INV>(v + q * R);
  }
}

template <int R>
__device__ __forceinline__ void pass_load(const float2 *s, float2 (&v)[16], int N, int T, int tt) {
#pragma unroll
  for (int q = 0; q < 16 / R; ++q)
#pragma unroll
    for (int m = 0; m < R; ++m) v[q * R + m] = s[pad16(tt + q * T + m * (N / R))];
}

template <int R>
__device__ __forceinline__ void pass_store(float2 *s, const float2 (&v)[16], int Ns, int T, int tt) {
#pragma unroll
  for (int q = 0; q < 16 / R; ++q) {
    const int j = tt + q * T, k = j & (Ns - 1), base = (j - k) * R + k;
#pragma unroll
    for (int m = 0; m < R; ++m) s[pad16(base + m * Ns)] = v[q * R + m];
  }
}

// N-point FFT (N = 2^LOGN >= 16) of the sequence whose elements tt + m T the
// caller holds in v[m]; leaves thread tt the elements tt + m T of the result in
// v[m] (the last pass, of radix R, computes X[tt + T (q + m 16/R)] in v[q R + m]).
// The passes (radix 16, the last 2..16) are fixed at compile time.  Every
// thread of the CTA takes part (the passes synchronise the CTA); SYNC: others
// may still read s when this starts.
template <int LOGN, bool INV, bool SYNC, int NS_LOG = 0>
__device__ __forceinline__ void fft_regs(float2 *s, float2 (&v)[16], int tt, const float2 *__restrict__ tw) {
  constexpr int B = (LOGN - NS_LOG) >= 4 ? 4 : (LOGN - NS_LOG);
  constexpr int R = 1 << B, N = 1 << LOGN, T = N / 16;
  pass_compute<R, INV>(v, N, 1 << NS_LOG, T, tt, tw);
  if constexpr (NS_LOG + B < LOGN) {
    constexpr int R2 = 1 << ((LOGN - NS_LOG - B) >= 4 ? 4 : (LOGN - NS_LOG - B));
    if (SYNC || NS_LOG > 0) __syncthreads();
    pass_store<R>(s, v, 1 << NS_LOG, T, tt);
    __syncthreads();
    pass_load<R2>(s, v, N, T, tt);
    fft_regs<LOGN, INV, SYNC, NS_LOG + B>(s, v, tt, tw);
  } else if constexpr (R < 16) {
    float2 t[16];
#pragma unroll
    for (int q = 0; q < 16 / R; ++q)
#pragma unroll
      for (int m = 0; m < R; ++m) t[q + m * (16 / R)] = v[q * R + m];
#pragma unroll
    for (int m = 0; m < 16; ++m) v[m] = t[m];
  }
}

// Expanded-grid coordinate -> field coordinate (or -1 = zero): positions past
// the field belong to the extension below the field when they are closer to
// it, else to the wrapped extension above it.
__device__ __forceinline__ int expand_index(int p, int n, int F, int border) {
  int v = p;
  if (p >= n) v = (p - n) < (F - p) ? p : p - F;
  return border_index(border, v, n);
}

// Filter tap landing on expanded coordinate `pos` (or -1): g[(r - h) mod F]
// = f[r] for convolution, g[(h - r) mod F] = f[r] for cross-correlation.
__device__ __forceinline__ int filter_index(int pos, int h, int R, int F, bool conv) {
  int r = conv ? pos + h : h - pos;
  if (conv) {
    if (r >= F) r -= F;
  } else {
    if (r < 0) r += F;
  }
  return (r >= 0 && r < R) ? r : -1;
}

// Row pass: row_threads/T sequences of N = Fc/2 complex points per CTA.  The
// first planes * (top + bottom) sequences are the image planes' grid rows,
// expanded with the border, into spec; the rest the rows of the filter planes
// (centred at the origin, flipped for convolution), into rows.
template <int LOGN>
__global__ void __launch_bounds__(row_threads(1 << LOGN), 1024 / row_threads(1 << LOGN))
    fft_rows_r2c(FftParams p, const float *__restrict__ x, const float *__restrict__ f, float2 *__restrict__ spec,
                 float2 *__restrict__ rows, int planes, int fplanes) {
  extern __shared__ __align__(16) float2 fsm[];
  grid_dependency_wait();  // launched with programmatic serialisation
  allow_dependent_launch();
  constexpr int N = 1 << LOGN, T = N / 16, per = row_threads(N) / T;
  const ConvGeom &g = p.g;
  const int sub = threadIdx.x / T, tt = threadIdx.x - sub * T;
  const int held = p.top + p.bottom;
  int gr = blockIdx.x * per + sub;
  const bool image = gr < planes * held;
  if (!image) gr -= planes * held;
  const bool active = image || gr < fplanes * g.R;
  const int per_plane = image ? held : g.R;
  const int pl = gr / per_plane, q = gr - pl * per_plane;
  const int row = image && q >= p.top ? p.Fr - held + q : q;  // grid row, or filter row
  float2 *s = fsm + sub * (N + N / 16);
  float2 v[16];
  if (image) {
    int ip, fp;
    plane_pair(g, pl, 0, &ip, &fp);
    const float *xp = x + (size_t)ip * g.H * g.W;
    const int sr = expand_index(row, g.H, p.Fr, g.border);
    // positions inside the field map to themselves: one 8-byte load per pair
    // (an 8-byte aligned plane of even width keeps every row aligned); the
    // border positions take the expansion rule
    const bool pairs = sr >= 0 && (g.W & 1) == 0 && (reinterpret_cast<uintptr_t>(xp) & 7) == 0;
    const float2 *row2 = reinterpret_cast<const float2 *>(xp + (size_t)(sr < 0 ? 0 : sr) * g.W);
#pragma unroll
    for (int m = 0; m < 16; ++m) {
      const int n = tt + m * T;
      if (pairs && 2 * n + 1 < g.W) {
        v[m] = __ldg(row2 + n);
      } else {
        float e[2];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const int sc = expand_index(2 * n + k, g.W, p.Fc, g.border);
          e[k] = (sr >= 0 && sc >= 0) ? __ldg(xp + (size_t)sr * g.W + sc) : 0.0f;
        }
        v[m] = make_float2(e[0], e[1]);
      }
    }
  } else {
    const float *fp = f + ((size_t)pl * g.R + row) * g.S;
    const bool conv = g.orient == CCT_CONVOLUTION;
#pragma unroll
    for (int m = 0; m < 16; ++m) {
      const int n = tt + m * T;
      float e[2] = {0.0f, 0.0f};
      if (active) {
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const int c = filter_index(2 * n + k, (g.S - 1) / 2, g.S, p.Fc, conv);
          if (c >= 0) e[k] = __ldg(fp + c);
        }
      }
      v[m] = make_float2(e[0], e[1]);
    }
  }
  fft_regs<LOGN, false, false>(s, v, tt, p.tw_n);
  if (LOGN > 4) __syncthreads();  // the last exchange is read
#pragma unroll
  for (int m = 0; m < 16; ++m) s[pad16(tt + m * T)] = v[m];
  __syncthreads();
  if (!active) return;
  // X[k] = E[k] + W^k O[k], E = (Z[k] + conj Z[N-k]) / 2, O = (Z[k] - conj Z[N-k]) / 2i,
  // W = exp(-2 pi i / Fc), k = 0..N
  const int nr = image ? p.Fr : g.R;
  float2 *out = (image ? spec : rows) + (size_t)pl * nr * p.ld;
  auto split = [&](int k, float2 zk, float2 zn) {
    const float2 e = make_float2(0.5f * (zk.x + zn.x), 0.5f * (zk.y + zn.y));
    const float2 dd = make_float2(0.5f * (zk.x - zn.x), 0.5f * (zk.y - zn.y));
    const float2 o = make_float2(dd.y, -dd.x);  // dd / i
    out[spec_index(row, k, nr)] = cadd(e, cmul(__ldg(p.tw_2n + k), o));
  };
#pragma unroll
  for (int m = 0; m < 16; ++m) {
    const int k = tt + m * T;
    split(k, v[m], conjf2(s[pad16(k == 0 ? 0 : N - k)]));
  }
  if (tt == 0) split(N, v[0], conjf2(v[0]));
}

// Column pass over col_width spectrum columns per CTA (c fastest across
// threads, so each warp reads 32-byte row segments).  Bound: instruction issue
// and shared-memory exchanges of one wave of CTAs (2048 rows), their latency
// below that.  With 512 threads for every length, a 512-row grid had 17 CTAs
// whose 16 columns shared two bank offsets (512x512 by 31x31: 69 us, 21 now).
// MODE 0: forward FFT, times G[fplane], inverse FFT, in place in spec: rows that
//         hold the field and its border in, rows of the result out.
// MODE 1: forward FFT and scaling by p.scale of the filters' rows, into spec.
template <int MODE, int LOGR>
__global__ void __launch_bounds__(col_width(1 << LOGR) * (1 << LOGR) / 16,
                                  col_residency(1 << LOGR) / (col_width(1 << LOGR) * (1 << LOGR) / 16))
    fft_cols(FftParams p, float2 *__restrict__ spec, const float2 *__restrict__ G) {
  extern __shared__ __align__(16) float2 fsm[];
  grid_dependency_wait();  // launched with programmatic serialisation
  allow_dependent_launch();
  constexpr int Fr = 1 << LOGR, T = Fr / 16, CW = col_width(Fr);
  const int ncol = p.Fc / 2 + 1;
  const int cblocks = (ncol + CW - 1) / CW;
  const int pl = blockIdx.x / cblocks, c0 = (blockIdx.x - pl * cblocks) * CW;
  const int c = threadIdx.x % CW, tt = threadIdx.x / CW, col = c0 + c;
  const bool active = col < ncol;
  float2 *s = fsm + c * col_stride(Fr);
  float2 *sp = spec + (size_t)pl * Fr * p.ld + spec_index(0, col, Fr);  // row r at sp[4 r]
  float2 v[16];
  if (MODE == 0) {
#pragma unroll
    for (int m = 0; m < 16; ++m) {
      const int r = tt + m * T;
      v[m] = active && (r < p.top || r >= Fr - p.bottom) ? sp[(size_t)r * 4] : make_float2(0.0f, 0.0f);
    }
    fft_regs<LOGR, false, false>(s, v, tt, p.tw_r);
  } else {
    const ConvGeom &g = p.g;
    const float2 *rp = G + (size_t)pl * g.R * p.ld + spec_index(0, col, g.R);
    auto row = [&](int r) {
      const int i = filter_index(r, (g.R - 1) / 2, g.R, Fr, g.orient == CCT_CONVOLUTION);
      return active && i >= 0 ? __ldg(rp + (size_t)i * 4) : make_float2(0.0f, 0.0f);
    };
    if ((g.R - 1) / 2 < T) {
      // the filter's rows lie in the first and the last sixteenth of the grid: a
      // thread's first DFT has two inputs that are not zero, and the compiler
      // drops the arithmetic on the others, whose values it knows.  The same
      // operations as the general case below, so the same bits: a filter with
      // rows of zeros around it gives the field that it gives without them.
      v[0] = row(tt);
#pragma unroll
      for (int m = 1; m < 15; ++m) v[m] = make_float2(0.0f, 0.0f);
      v[15] = row(tt + 15 * T);
      fft_regs<LOGR, false, false>(s, v, tt, p.tw_r);
    } else {
#pragma unroll
      for (int m = 0; m < 16; ++m) v[m] = row(tt + m * T);
      fft_regs<LOGR, false, false>(s, v, tt, p.tw_r);
    }
  }
  if (MODE == 0) {
    int ip, fp;
    plane_pair(p.g, pl, 0, &ip, &fp);
    const float2 *gp = G + (size_t)fp * Fr * p.ld + spec_index(0, col, Fr);
#pragma unroll
    for (int m = 0; m < 16; ++m)
      v[m] = active ? cmul(v[m], __ldg(gp + (size_t)(tt + m * T) * 4)) : make_float2(0.0f, 0.0f);
    fft_regs<LOGR, true, true>(s, v, tt, p.tw_r);
    if (!active) return;
#pragma unroll
    for (int m = 0; m < 16; ++m)
      if (tt + m * T < p.g.OH) sp[(size_t)(tt + m * T) * 4] = v[m];
  } else {
    if (!active) return;
#pragma unroll
    for (int m = 0; m < 16; ++m) sp[(size_t)(tt + m * T) * 4] = cscale(v[m], p.scale);
  }
}

// Inverse row pass: half-spectrum rows -> real rows, trimmed to the output.
template <int LOGN>
__global__ void __launch_bounds__(row_threads(1 << LOGN), 1024 / row_threads(1 << LOGN))
    fft_rows_c2r(FftParams p, const float2 *__restrict__ spec, float *__restrict__ y, int planes) {
  extern __shared__ __align__(16) float2 fsm[];
  grid_dependency_wait();  // launched with programmatic serialisation
  allow_dependent_launch();
  const ConvGeom &g = p.g;
  constexpr int N = 1 << LOGN, T = N / 16, per = row_threads(N) / T;
  const int sub = threadIdx.x / T, tt = threadIdx.x - sub * T;
  const int gr = blockIdx.x * per + sub;
  const bool active = gr < planes * g.OH;
  const int row = gr % g.OH, pl = gr / g.OH;
  float2 *s = fsm + sub * (N + N / 16);
  const float2 *in = spec + (size_t)pl * p.Fr * p.ld;
  // Z[k] = E[k] + i O[k], E = (X[k] + conj X[N-k]) / 2, O = (X[k] - conj X[N-k]) / 2 * conj(W^k)
  float2 v[16];
#pragma unroll
  for (int m = 0; m < 16; ++m) {
    const int k = tt + m * T;
    float2 z = make_float2(0.0f, 0.0f);
    if (active) {
      const float2 xk = __ldg(in + spec_index(row, k, p.Fr)), xn = conjf2(__ldg(in + spec_index(row, N - k, p.Fr)));
      const float2 e = make_float2(0.5f * (xk.x + xn.x), 0.5f * (xk.y + xn.y));
      const float2 dd = make_float2(0.5f * (xk.x - xn.x), 0.5f * (xk.y - xn.y));
      const float2 o = cmul(dd, conjf2(__ldg(p.tw_2n + k)));
      z = make_float2(e.x - o.y, e.y + o.x);  // e + i*o
    }
    v[m] = z;
  }
  fft_regs<LOGN, true, false>(s, v, tt, p.tw_n);
  if (!active) return;
  float *yr = y + ((size_t)pl * g.OH + row) * g.OW;
  if ((g.flags & CCT_FLAG_RELU) != 0) {
#pragma unroll
    for (int m = 0; m < 16; ++m) v[m] = make_float2(fmaxf(v[m].x, 0.0f), fmaxf(v[m].y, 0.0f));
  }
  // an aligned field of even width keeps every output row 8-byte aligned: one
  // pair per store
  const bool pairs = (g.OW & 1) == 0 && (reinterpret_cast<uintptr_t>(y) & 7) == 0;
#pragma unroll
  for (int m = 0; m < 16; ++m) {
    const int j = tt + m * T;
    if (pairs) {
      if (2 * j < g.OW) reinterpret_cast<float2 *>(yr)[j] = v[m];
    } else {
      if (2 * j < g.OW) yr[2 * j] = v[m].x;
      if (2 * j + 1 < g.OW) yr[2 * j + 1] = v[m].y;
    }
  }
}

int ilog2(int v) {
  int l = 0;
  while ((1 << l) < v) ++l;
  return l;
}
int pow2_at_least(int v) { return 1 << ilog2(v); }

// One-dimensional forward FFT of length n in FP64 (iterative radix-2, natural
// order) of v[0], v[stride], ...; w[k] = exp(-2 pi i k / n), k < n/2.
void fft64(std::complex<double> *v, int n, int stride, const std::vector<std::complex<double>> &w,
           std::vector<std::complex<double>> *scratch) {
  std::vector<std::complex<double>> &t = *scratch;
  t.resize(n);
  for (int i = 0; i < n; ++i) t[i] = v[(size_t)i * stride];
  for (int i = 1, j = 0; i < n; ++i) {
    int bit = n >> 1;
    for (; j & bit; bit >>= 1) j ^= bit;
    j ^= bit;
    if (i < j) std::swap(t[i], t[j]);
  }
  for (int len = 2; len <= n; len <<= 1) {
    const int step = n / len;
    for (int i = 0; i < n; i += len)
      for (int k = 0; k < len / 2; ++k) {
        const std::complex<double> u = t[i + k], x = t[i + k + len / 2] * w[(size_t)k * step];
        t[i + k] = u + x;
        t[i + k + len / 2] = u - x;
      }
  }
  for (int i = 0; i < n; ++i) v[(size_t)i * stride] = t[i];
}

std::vector<std::complex<double>> twiddles64(int n) {
  std::vector<std::complex<double>> w(n / 2);
  for (int k = 0; k < n / 2; ++k) w[k] = std::polar(1.0, -2.0 * M_PI * k / n);
  return w;
}

}  // namespace

bool fft_plan(const ConvGeom &g, FftParams *out) {
  if (g.mode != CCT_PLANE_BY_PLANE || g.down != 1 || g.up != 1) return false;
  if (g.border != CCT_BORDER_ZERO && g.border != CCT_BORDER_CLAMP && g.border != CCT_BORDER_CYCLIC)
    return false;
  if (g.H < 2 || g.W < 2) return false;
  FftParams p{};
  p.g = g;
  const int hr = g.R / 2, hc = g.S / 2;  // apron (FFTConvolutionUtils.scala:63-64)
  auto size = [&](int n, int h) {
    switch (g.border) {
      case CCT_BORDER_CLAMP: return pow2_at_least(n + 2 * h);
      case CCT_BORDER_ZERO: return pow2_at_least(n + h);
      default: return (n & (n - 1)) == 0 ? n : pow2_at_least(n + 2 * h);
    }
  };
  p.Fr = size(g.H, hr);
  p.Fc = size(g.W, hc);
  // the register FFTs want at least 16 points per sequence
  if (p.Fc < 32) p.Fc = 32;
  if (p.Fr < 16) p.Fr = 16;
  if (p.Fr > 4096 || p.Fc > 8192) return false;
  if (g.R > p.Fr || g.S > p.Fc) return false;  // no tap may wrap onto another
  // the border extension must fit between the field and its wrapped copy
  if (g.border != CCT_BORDER_ZERO && ((p.Fr > g.H && p.Fr < g.H + 2 * hr) || (p.Fc > g.W && p.Fc < g.W + 2 * hc)))
    return false;
  p.logN = ilog2(p.Fc / 2);
  p.logR = ilog2(p.Fr);
  p.ld = ((p.Fc / 2 + 1) + 3) & ~3;  // whole 4-column blocks (spec_index)
  p.scale = 1.0f / ((float)p.Fr * (float)(p.Fc / 2));
  p.spec_elems = (size_t)g.pout * p.Fr * p.ld;
  p.filter_elems = (size_t)g.pf * p.Fr * p.ld;
  p.row_elems = (size_t)g.pf * g.R * p.ld;
  // a grid larger than the field holds the apron below it and, wrapped, above
  const bool apron = g.border != CCT_BORDER_ZERO && p.Fr > g.H;
  p.top = g.H + (apron ? hr : 0);
  p.bottom = apron ? hr : 0;
  p.tw_elems = (size_t)(p.Fc / 2) + p.Fr + (p.Fc / 2 + 1);
  *out = p;
  return true;
}

void fft_twiddles(const FftParams &p, std::vector<float> *host) {
  host->resize(2 * p.tw_elems);
  float *h = host->data();
  const int N = p.Fc / 2;
  size_t o = 0;
  for (int k = 0; k < N; ++k, ++o) {
    h[2 * o] = (float)std::cos(-2.0 * M_PI * k / N);
    h[2 * o + 1] = (float)std::sin(-2.0 * M_PI * k / N);
  }
  for (int k = 0; k < p.Fr; ++k, ++o) {
    h[2 * o] = (float)std::cos(-2.0 * M_PI * k / p.Fr);
    h[2 * o + 1] = (float)std::sin(-2.0 * M_PI * k / p.Fr);
  }
  for (int k = 0; k <= N; ++k, ++o) {
    h[2 * o] = (float)std::cos(-2.0 * M_PI * k / p.Fc);
    h[2 * o + 1] = (float)std::sin(-2.0 * M_PI * k / p.Fc);
  }
}

void fft_set_tables(FftParams *p, float2 *tw) {
  p->tw_n = tw;
  p->tw_r = tw + p->Fc / 2;
  p->tw_2n = tw + p->Fc / 2 + p->Fr;
}

void fft_static_spectrum(const FftParams &p, const float *host_filter, std::vector<float> *out) {
  const ConvGeom &g = p.g;
  const int Fr = p.Fr, Fc = p.Fc, ld = p.ld;
  const int hr = (g.R - 1) / 2, hc = (g.S - 1) / 2;
  out->assign(2 * p.filter_elems, 0.0f);
  std::vector<std::complex<double>> grid((size_t)Fr * Fc);
  const double scale = 1.0 / ((double)Fr * (double)(Fc / 2));
  const std::vector<std::complex<double>> wc = twiddles64(Fc), wr = twiddles64(Fr);
  std::vector<std::complex<double>> scratch;
  for (int pl = 0; pl < g.pf; ++pl) {
    std::fill(grid.begin(), grid.end(), std::complex<double>(0.0, 0.0));
    const float *f = host_filter + (size_t)pl * g.R * g.S;
    for (int r = 0; r < g.R; ++r)
      for (int s = 0; s < g.S; ++s) {
        int gr, gc;
        if (g.orient == CCT_CONVOLUTION) {
          gr = ((r - hr) % Fr + Fr) % Fr;
          gc = ((s - hc) % Fc + Fc) % Fc;
        } else {
          gr = ((hr - r) % Fr + Fr) % Fr;
          gc = ((hc - s) % Fc + Fc) % Fc;
        }
        grid[(size_t)gr * Fc + gc] += f[(size_t)r * g.S + s];
      }
    for (int r = 0; r < Fr; ++r) fft64(grid.data() + (size_t)r * Fc, Fc, 1, wc, &scratch);
    for (int c = 0; c <= Fc / 2; ++c) fft64(grid.data() + c, Fr, Fc, wr, &scratch);
    float *o = out->data() + 2 * (size_t)pl * Fr * ld;
    for (int r = 0; r < Fr; ++r)
      for (int c = 0; c <= Fc / 2; ++c) {
        const std::complex<double> v = grid[(size_t)r * Fc + c] * scale;
        o[2 * spec_index(r, c, Fr)] = (float)v.real();
        o[2 * spec_index(r, c, Fr) + 1] = (float)v.imag();
      }
  }
}

// Kernel instantiation for the transform length (2^4 .. 2^12 points).
#define CCT_FFT_LOG_SWITCH(LOGV, CALL)                     \
  switch (LOGV) {                                          \
    case 4: { constexpr int L = 4; CALL; } break;          \
    case 5: { constexpr int L = 5; CALL; } break;          \
    case 6: { constexpr int L = 6; CALL; } break;          \
    case 7: { constexpr int L = 7; CALL; } break;          \
    case 8: { constexpr int L = 8; CALL; } break;          \
    case 9: { constexpr int L = 9; CALL; } break;          \
    case 10: { constexpr int L = 10; CALL; } break;        \
    case 11: { constexpr int L = 11; CALL; } break;        \
    case 12: { constexpr int L = 12; CALL; } break;        \
    default: return set_error(CCT_ENOTSUP, "FFT length 2^%d", (int)(LOGV)); \
  }

template <int MODE, int L>
int launch_cols_t(const FftParams &p, float2 *spec, const float2 *G, int planes, cudaStream_t st) {
  constexpr int Fr = 1 << L, cw = col_width(Fr);
  const size_t smem = sizeof(float2) * (size_t)cw * col_stride(Fr);
  int rc = raise_smem_limit(fft_cols<MODE, L>, smem, "cudaFuncSetAttribute(fft)");
  if (rc) return rc;
  const int cblocks = (p.Fc / 2 + 1 + cw - 1) / cw;
  rc = launch_pdl(fft_cols<MODE, L>, dim3(cblocks * planes), dim3(cw * Fr / 16), smem, st, "fft_cols launch", p, spec,
                  G);
  if (!rc) count_launches(1);
  return rc;
}

template <int MODE>
int launch_cols(const FftParams &p, float2 *spec, const float2 *G, int planes, cudaStream_t st) {
  CCT_FFT_LOG_SWITCH(p.logR, return (launch_cols_t<MODE, L>(p, spec, G, planes, st)))
  return CCT_OK;
}

// CTAs and shared memory of a row pass over `rows` sequences of N points.
template <int L>
void row_shape(long long rows, unsigned *blocks, size_t *smem) {
  constexpr int N = 1 << L, per = row_threads(N) / (N / 16);
  *blocks = (unsigned)((rows + per - 1) / per);
  *smem = sizeof(float2) * (size_t)per * (N + N / 16);
}

template <int L>
int launch_r2c_t(const FftParams &p, const float *x, const float *f, float2 *spec, float2 *rows, cudaStream_t st) {
  const int planes = p.g.pout, fplanes = f ? p.g.pf : 0;
  unsigned blocks;
  size_t smem;
  row_shape<L>((long long)planes * (p.top + p.bottom) + (long long)fplanes * p.g.R, &blocks, &smem);
  int rc = raise_smem_limit(fft_rows_r2c<L>, smem, "cudaFuncSetAttribute(fft)");
  if (rc) return rc;
  rc = launch_pdl(fft_rows_r2c<L>, dim3(blocks), dim3(row_threads(1 << L)), smem, st, "fft_rows_r2c launch", p, x, f,
                  spec, rows, planes, fplanes);
  if (!rc) count_launches(1);
  return rc;
}

template <int L>
int launch_c2r_t(const FftParams &p, const float2 *spec, float *y, cudaStream_t st) {
  const int planes = p.g.pout;
  unsigned blocks;
  size_t smem;
  row_shape<L>((long long)planes * p.g.OH, &blocks, &smem);
  int rc = raise_smem_limit(fft_rows_c2r<L>, smem, "cudaFuncSetAttribute(fft)");
  if (rc) return rc;
  rc = launch_pdl(fft_rows_c2r<L>, dim3(blocks), dim3(row_threads(1 << L)), smem, st, "fft_rows_c2r launch", p, spec, y,
                  planes);
  if (!rc) count_launches(1);
  return rc;
}

int launch_fft_conv(const FftParams &p, const float *x, const float *f, float2 *rows, float2 *G, float2 *spec,
                    float *y, cudaStream_t st) {
  int rc = CCT_OK;
  CCT_FFT_LOG_SWITCH(p.logN, rc = (launch_r2c_t<L>(p, x, f, spec, rows, st)))
  if (!rc && f) rc = launch_cols<1>(p, G, rows, p.g.pf, st);
  if (!rc) rc = launch_cols<0>(p, spec, G, p.g.pout, st);
  if (rc) return rc;
  CCT_FFT_LOG_SWITCH(p.logN, rc = (launch_c2r_t<L>(p, spec, y, st)))
  if (rc) return rc;
  return check_cuda(cudaGetLastError(), "fft convolution launch");
}

}  // namespace cct
