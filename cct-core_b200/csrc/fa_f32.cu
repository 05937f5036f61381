// FilterAdjoint (weight gradient) in FP32 for small results:
//   out[B*w + b](r, s) = sum_(i,j) x[b*C + w%C](r + i, s + j) * g'[b*L + w/C](i, j)
// with BorderValid, no sampling (ConvolveHyperKernel.scala:187, 333, 575-590;
// CogFunctionAPI.scala:1480-1511), g' = g flipped for convolveFilterAdjoint.
// The block-reduced form sums the B images of each w in order.
//
// The result planes are tiny (the filter's size) and the reduction is long
// (the whole gradient plane).  A thread owns a (input plane c, result row r)
// and one gradient plane l (fa_rows_kernel, fa_f32_kernel) or four
// (fa_quad_kernel), and keeps the result rows' S outputs in registers while it
// walks the gradient; the image row it needs slides through a register window, so
// an image load feeds S multiply-adds per gradient plane.  Per output the order is the reference's: an fma chain over
// j from 0 per gradient row, row sums added in order, so the result is
// bit-identical to the FP32 oracle.
//
// fa_quad_kernel: the main path, described below.
// fa_rows_kernel (fields too wide for its shared memory, gradients of few rows):
// a CTA serves one image b, kCG input planes and kLG gradient planes.  It
// streams the gradient rows i = 0.. through shared memory together with a ring
// of the OH image rows each step needs (cp.async, the next rows landing while
// the current ones are used), so every image row and gradient row is read from
// L2 once per CTA.
// fa_f32_kernel: the fallback for image rows too wide to stage; one CTA per
// (b, l) with the gradient plane in shared memory and image rows read
// through L1.
// The block-reduced form writes the per-image results to plan workspace and
// a second kernel adds them in image order.
#include "cct_internal.h"
#include "sm100_util.cuh"
#include "tile_common.cuh"

namespace cct {
namespace {

constexpr int kFaThreads = 256;
constexpr int kFaMaxS = 8;
constexpr int kCG = 8, kLG = 8;  // input planes x gradient planes per CTA (fa_rows_kernel)
constexpr size_t kRowsSmemMax = 96 * 1024;

// shared memory of fa_rows_kernel: a ring of OH + 1 image rows per input
// plane and two gradient rows per gradient plane, each row padded to 4 floats
__host__ __device__ inline int fa_row_pitch(int n) { return (n + 3) & ~3; }
__host__ __device__ inline size_t fa_rows_smem(const ConvGeom &g) {
  return sizeof(float) * ((size_t)kCG * (g.OH + 1) * fa_row_pitch(g.W) + (size_t)kLG * 2 * fa_row_pitch(g.S));
}

template <int S>
__global__ void __launch_bounds__(kCG * kLG * kFaMaxS)
    fa_rows_kernel(ConvGeom g, const float *__restrict__ x, const float *__restrict__ f, float *__restrict__ y,
                   int cgroups, int lgroups) {
  extern __shared__ __align__(16) float sm[];
  const int Hg = g.R, Wg = g.S, C = g.n, L = g.groups, B = g.batch, OH = g.OH;
  const int xp_pitch = fa_row_pitch(g.W), gp_pitch = fa_row_pitch(Wg), slots = OH + 1;
  float *xring = sm;                                       // [c][slot][xp_pitch]
  float *grow = sm + (size_t)kCG * slots * xp_pitch;       // [l][2][gp_pitch]
  int bid = blockIdx.x;
  const int cg = bid % cgroups;
  bid /= cgroups;
  const int lg = bid % lgroups, b = bid / lgroups;
  const int c0 = cg * kCG, l0 = lg * kLG;
  const bool conv = g.orient == CCT_CONVOLUTION;
  const int nthreads = blockDim.x;
  // thread -> (l, c, r): r fastest, so neighbouring threads share image rows
  const int r = threadIdx.x % OH, q = threadIdx.x / OH;
  const int cl = q % kCG, ll = q / kCG;
  const bool active = ll < kLG && c0 + cl < C && l0 + ll < L;

  // copies of image row `row` of every input plane of the group into its slot
  auto load_x_row = [&](int row) {
    const int slot = row % slots;
    for (int e = threadIdx.x; e < kCG * g.W; e += nthreads) {
      const int c = e / g.W, col = e - c * g.W;
      const bool ok = c0 + c < C;
      const float *src = x + ((size_t)(b * C + c0 + c) * g.H + row) * g.W + col;
      cp_async_f32(xring + ((size_t)c * slots + slot) * xp_pitch + col, ok ? src : x, ok);
    }
  };
  // gradient row i (flipped for convolution) of every gradient plane into buffer i&1
  auto load_g_row = [&](int i) {
    const int gi = conv ? Hg - 1 - i : i;
    for (int e = threadIdx.x; e < kLG * Wg; e += nthreads) {
      const int l = e / Wg, j = e - l * Wg;
      const bool ok = l0 + l < L;
      const int gj = conv ? Wg - 1 - j : j;
      const float *src = f + ((size_t)(b * L + l0 + l) * Hg + gi) * Wg + gj;
      cp_async_f32(grow + ((size_t)l * 2 + (i & 1)) * gp_pitch + j, ok ? src : f, ok);
    }
  };

  for (int row = 0; row < OH; ++row) load_x_row(row);
  load_g_row(0);
  cp_async_commit();

  float acc[S];
#pragma unroll
  for (int s = 0; s < S; ++s) acc[s] = 0.0f;
  for (int i = 0; i < Hg; ++i) {
    if (i + 1 < Hg) {  // next step's rows land while this step computes
      load_x_row(i + OH);
      load_g_row(i + 1);
      cp_async_commit();
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    __syncthreads();
    if (active) {
      const float *xr = xring + ((size_t)cl * slots + (i + r) % slots) * xp_pitch;
      const float *gr = grow + ((size_t)ll * 2 + (i & 1)) * gp_pitch;
      float win[S], col[S];
#pragma unroll
      for (int s = 0; s < S; ++s) {
        col[s] = 0.0f;
        win[s] = xr[s];
      }
      for (int j = 0; j < Wg; ++j) {
        const float w = gr[j];
#pragma unroll
        for (int s = 0; s < S; ++s) col[s] = __fmaf_rn(win[s], w, col[s]);
#pragma unroll
        for (int s = 0; s + 1 < S; ++s) win[s] = win[s + 1];
        win[S - 1] = xr[min(j + S, g.W - 1)];  // the last step's value is never used
      }
#pragma unroll
      for (int s = 0; s < S; ++s) acc[s] = __fadd_rn(acc[s], col[s]);
    }
    __syncthreads();  // the ring slot and gradient buffer are refilled next step
  }
  if (!active) return;
  float *yp = y + ((size_t)B * ((l0 + ll) * C + c0 + cl) + b) * OH * g.OW + (size_t)r * g.OW;
  const bool relu = (g.flags & CCT_FLAG_RELU) != 0;
#pragma unroll
  for (int s = 0; s < S; ++s) yp[s] = relu ? fmaxf(acc[s], 0.0f) : acc[s];
}

// fa_quad_kernel (the main path): a lane owns one (input plane, result row)
// and four gradient planes, so an image value feeds 4 S multiply-adds and a
// float4 of the four planes' gradients comes as one broadcast read; a warp
// owns a gradient row i of the step, NW warps the step's rows.  Row sums
// meet in shared memory and are added in row order by the thread that keeps
// the output, so splitting the rows over warps does not change the order.
// Gradient planes l, l+1 advance together in packed fma.rn.f32x2 (each lane
// the scalar RN operation).
//
// Bound: the FP32 pipe (2 S packed multiply-adds per gradient column; half busy,
// the 16 warps that shared memory leaves an SM wait on their chains): 0.20 ms for
// the weight gradient of the B=16, C=32, K=64, 64x64, 5x5 layer.  fa_rows_kernel
// read an image and a gradient value from shared memory per S multiply-adds: L1
// 91 % busy, 0.62 ms.
// NW gradient rows per step, one per warp: 4, or 8 or 16 where the grid leaves
// SMs idle and the steps' latency is what the launch waits for.
constexpr int kQL = 4;                   // gradient planes per CTA
constexpr size_t kQuadSmemMax = 220 * 1024;

// input planes a warp's 32 consecutive (plane, row) pairs can touch
__host__ __device__ inline int quad_planes(const ConvGeom &g) {
  const int n = (32 + g.OH - 2) / g.OH + 1;
  return n < g.n ? n : g.n;
}
__host__ __device__ inline int quad_ring(int OH, int NW) { return 2 * NW + OH - 1; }
// row pitch: whole float4s past the last window, an odd number of them so that
// neighbouring ring rows start on different banks
__host__ __device__ inline int quad_pitch(const ConvGeom &g) {
  const int n4 = (g.S + 3) / 4 + (g.OW + 6) / 4;
  return 4 * (n4 | 1);
}
inline size_t quad_smem(const ConvGeom &g, int NW) {
  return sizeof(float) * ((size_t)quad_planes(g) * quad_ring(g.OH, NW) * quad_pitch(g) +
                          2 * (size_t)NW * kQL * ((g.S + 3) & ~3) + (size_t)NW * kQL * g.OW * 32);
}

template <int S, int NW>
__global__ void __launch_bounds__(NW * 32)
    fa_quad_kernel(ConvGeom g, const float *__restrict__ x, const float *__restrict__ f, float *__restrict__ y,
                   int mgroups, int lgroups) {
  extern __shared__ __align__(16) float sm[];
  grid_dependency_wait();  // launched with programmatic serialisation: nothing global before this
  constexpr int NT = NW * 32, NV = (S + 6) / 4, OUTS = kQL * S * 32, NO = (OUTS + NT - 1) / NT;
  const int Hg = g.R, Wg = g.S, C = g.n, L = g.groups, B = g.batch, OH = g.OH, W = g.W;
  const int pitch = quad_pitch(g), ring = quad_ring(OH, NW), gcols = (Wg + 3) & ~3;
  float *xr = sm;                                                       // [plane][ring][pitch]
  float *gr = xr + (size_t)quad_planes(g) * ring * pitch;              // [2][row][column][plane]
  float *sums = gr + 2 * NW * kQL * gcols;                          // [row][(plane, s)][lane]
  int bid = blockIdx.x;
  const int m0 = (bid % mgroups) * 32;
  bid /= mgroups;
  const int l0 = (bid % lgroups) * kQL, b = bid / lgroups;
  const int c0 = m0 / OH, nc = min(C, (m0 + 31) / OH + 1) - c0, nl = min(kQL, L - l0);
  const bool conv = g.orient == CCT_CONVOLUTION;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m = min(m0 + lane, C * OH - 1), cl = m / OH - c0, r = m - (m / OH) * OH;
  const bool wide = (W & 3) == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0;

  // One image row of every plane of the group into its ring slot (a warp).
  const float *xg = x + (size_t)(b * C + c0) * g.H * W;
  const int cstride = ring * pitch, lane4 = 4 * lane;
  auto load_x = [&](int row, int slot) {
    const float *src = xg + (size_t)row * W + (wide ? lane4 : lane);
    float *dst = xr + slot * pitch + (wide ? lane4 : lane);
    const size_t page = (size_t)g.H * W;
    for (int c = 0; c < nc; ++c, src += page, dst += cstride) {
      if (wide) {
        for (int col = 0; col + lane4 < W; col += 128) cp_async_16(dst + col, src + col, true);
      } else {
        for (int col = 0; col + lane < W; col += 32) cp_async_f32(dst + col, src + col, true);
      }
    }
  };
  // This warp's gradient row i (flipped for convolution) of the four planes,
  // a column's planes adjacent.
  const float *fg = f + (size_t)(b * L + l0) * Hg * Wg;
  const size_t gpage = (size_t)Hg * Wg;
  const int jstep = conv ? -32 : 32;
  auto load_g = [&](int i, float *buf) {
    const float *src = fg + (size_t)(conv ? Hg - 1 - i : i) * Wg + (conv ? Wg - 1 - lane : lane);
    float *dst = buf + (size_t)warp * gcols * kQL + lane * kQL;
    for (int j = lane; j < Wg; j += 32, src += jstep, dst += 32 * kQL)
#pragma unroll
      for (int l = 0; l < kQL; ++l) cp_async_f32(dst + l, l < nl ? src + l * gpage : f, l < nl);
  };

  const int steps = (Hg + NW - 1) / NW;
  for (int row = warp; row < min(NW, Hg) + OH - 1; row += NW) load_x(row, row);
  if (warp < Hg) load_g(warp, gr);
  cp_async_commit();

  // ring slots of the row this lane reads at step k (i0 + warp + r) and of the
  // row this warp loads for the next step (i0 + NW + OH - 1 + warp)
  int rslot = (warp + r) % ring, lslot = (NW + OH - 1 + warp) % ring;
  float acc[NO];
#pragma unroll
  for (int o = 0; o < NO; ++o) acc[o] = 0.0f;
  for (int k = 0; k < steps; ++k) {
    const int i0 = k * NW, rows = min(NW, Hg - i0);
    cp_async_wait<0>();
    __syncthreads();  // this step's rows have landed; the last step's sums are added
    if (i0 + NW + warp < Hg) {
      load_x(i0 + NW + OH - 1 + warp, lslot);
      load_g(i0 + NW + warp, gr + ((k + 1) & 1) * NW * kQL * gcols);
    }
    cp_async_commit();
    if (warp < rows) {
      const float4 *xp = reinterpret_cast<const float4 *>(xr + (size_t)cl * cstride + rslot * pitch);
      const float4 *gp = reinterpret_cast<const float4 *>(gr + ((k & 1) * NW + warp) * kQL * gcols);
      float2 cs[S][2];
#pragma unroll
      for (int s = 0; s < S; ++s) cs[s][0] = cs[s][1] = make_float2(0.0f, 0.0f);
      // the image values of columns 4 q .. 4 (q + NV) - 1, each twice (the
      // packed form's operand), float4 number n at place n mod NV: NV quads of
      // columns are unrolled, so that the window never moves
      float2 win[4 * NV];
      auto put = [&](int e, const float4 v) {
        win[4 * e + 0] = make_float2(v.x, v.x);
        win[4 * e + 1] = make_float2(v.y, v.y);
        win[4 * e + 2] = make_float2(v.z, v.z);
        win[4 * e + 3] = make_float2(v.w, v.w);
      };
      auto tap = [&](int first, const float4 v) {  // one gradient column
        const float2 g0 = make_float2(v.x, v.y), g1 = make_float2(v.z, v.w);
#pragma unroll
        for (int s = 0; s < S; ++s) {
          const float2 xv = win[(first + s) % (4 * NV)];
          cs[s][0] = __ffma2_rn(xv, g0, cs[s][0]);
          cs[s][1] = __ffma2_rn(xv, g1, cs[s][1]);
        }
      };
#pragma unroll
      for (int e = 0; e < NV; ++e) put(e, xp[e]);
      const int quads = Wg / 4, rest = Wg - 4 * quads;
      // a quad's gradients, and the image values it brings in, are read while the
      // quad before it is multiplied
      float4 gq[4];
#pragma unroll
      for (int jj = 0; jj < 4; ++jj) gq[jj] = gp[jj];
      auto quad = [&](int q, int u) {
        const float4 nx = xp[q + NV];
        float4 gn[4];
#pragma unroll
        for (int jj = 0; jj < 4; ++jj) gn[jj] = gp[4 * (q + 1) + jj];  // past the last column: not used
#pragma unroll
        for (int jj = 0; jj < 4; ++jj) tap(4 * u + jj, gq[jj]);
        put(u, nx);
#pragma unroll
        for (int jj = 0; jj < 4; ++jj) gq[jj] = gn[jj];
      };
      auto tail = [&](int u) {
#pragma unroll
        for (int jj = 0; jj < 3; ++jj)
          if (jj < rest) tap(4 * u + jj, gq[jj]);
      };
      int q = 0;
#pragma unroll 1
      for (; q + NV <= quads; q += NV) {
#pragma unroll
        for (int u = 0; u < NV; ++u) quad(q + u, u);
      }
#pragma unroll
      for (int u = 0; u < NV; ++u) {
        if (q + u < quads)
          quad(q + u, u);
        else if (q + u == quads)
          tail(u);
      }
      float *out = sums + (size_t)warp * OUTS + lane;
#pragma unroll
      for (int s = 0; s < S; ++s) {
        out[(0 * S + s) * 32] = cs[s][0].x;
        out[(1 * S + s) * 32] = cs[s][0].y;
        out[(2 * S + s) * 32] = cs[s][1].x;
        out[(3 * S + s) * 32] = cs[s][1].y;
      }
    }
    rslot += NW;
    if (rslot >= ring) rslot -= ring;
    lslot += NW;
    if (lslot >= ring) lslot -= ring;
    __syncthreads();
#pragma unroll
    for (int o = 0; o < NO; ++o) {
      const int q = o * NT + threadIdx.x;
      if (OUTS % NT == 0 || q < OUTS) {
#pragma unroll 4
        for (int i = 0; i < rows; ++i) acc[o] = __fadd_rn(acc[o], sums[i * OUTS + q]);
      }
    }
  }
  allow_dependent_launch();
  const bool relu = (g.flags & CCT_FLAG_RELU) != 0;
#pragma unroll
  for (int o = 0; o < NO; ++o) {
    const int q = o * NT + threadIdx.x, l = q / (32 * S), s = (q >> 5) - l * S, mm = m0 + (q & 31);
    if ((OUTS % NT == 0 || q < OUTS) && l < nl && mm < C * OH) {
      const int c = mm / OH, rr = mm - c * OH;
      float *yp = y + ((size_t)B * ((size_t)(l0 + l) * C + c) + b) * OH * S + (size_t)rr * S;
      yp[s] = relu ? fmaxf(acc[o], 0.0f) : acc[o];
    }
  }
}

template <int S>
__global__ void __launch_bounds__(kFaThreads)
    fa_f32_kernel(ConvGeom g, const float *__restrict__ x, const float *__restrict__ f, float *__restrict__ y,
                  int cgroups) {
  extern __shared__ __align__(16) float gs[];
  const int Hg = g.R, Wg = g.S;  // the gradient plane is the "filter"
  const int C = g.n, L = g.groups, B = g.batch;
  int bid = blockIdx.x;
  const int cg = bid % cgroups;
  bid /= cgroups;
  const int l = bid % L, b = bid / L;
  const int per = blockDim.x / g.OH;  // input planes per CTA
  const int c = cg * per + threadIdx.x / g.OH, r = threadIdx.x % g.OH;
  const bool conv = g.orient == CCT_CONVOLUTION;
  const float *gp = f + (size_t)(b * L + l) * Hg * Wg;
  for (int i = threadIdx.x; i < Hg * Wg; i += blockDim.x)
    gs[i] = __ldg(gp + (conv ? Hg * Wg - 1 - i : i));
  __syncthreads();
  if (threadIdx.x >= per * g.OH || c >= C) return;
  const float *xp = x + (size_t)(b * C + c) * g.H * g.W + (size_t)r * g.W;
  float acc[S];
#pragma unroll
  for (int s = 0; s < S; ++s) acc[s] = 0.0f;
  for (int i = 0; i < Hg; ++i) {
    const float *xr = xp + (size_t)i * g.W;
    const float *gr = gs + i * Wg;
    float win[S], col[S];
#pragma unroll
    for (int s = 0; s < S; ++s) {
      col[s] = 0.0f;
      win[s] = s < g.OW ? __ldg(xr + s) : 0.0f;
    }
    for (int j = 0; j < Wg; ++j) {
      const float w = gr[j];
#pragma unroll
      for (int s = 0; s < S; ++s) col[s] = __fmaf_rn(win[s], w, col[s]);
      // slide: win[s] = x(r + i, j + 1 + s)
#pragma unroll
      for (int s = 0; s + 1 < S; ++s) win[s] = win[s + 1];
      const int nx = j + S;
      win[S - 1] = nx < g.W ? __ldg(xr + nx) : 0.0f;
    }
#pragma unroll
    for (int s = 0; s < S; ++s) acc[s] = __fadd_rn(acc[s], col[s]);
  }
  // output plane B*w + b, w = l*C + c
  float *yp = y + ((size_t)B * (l * C + c) + b) * g.OH * g.OW + (size_t)r * g.OW;
  const bool relu = (g.flags & CCT_FLAG_RELU) != 0;
#pragma unroll
  for (int s = 0; s < S; ++s)
    if (s < g.OW) yp[s] = relu ? fmaxf(acc[s], 0.0f) : acc[s];
}

// out[w] = sum_b part[B*w + b], images in order (acc from 0).  Bound: the latency
// of its loads, so eight images' values are read before they are added.
__global__ void __launch_bounds__(256) fa_reduce_kernel(const float *__restrict__ part, float *__restrict__ y, int B,
                                                        long long planes, int plane_elems, bool relu) {
  grid_dependency_wait();  // launched with programmatic serialisation: nothing global before this
  allow_dependent_launch();
  const long long n = planes * plane_elems;
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < n;
       e += (long long)gridDim.x * blockDim.x) {
    const long long w = e / plane_elems, q = e - w * plane_elems;
    const float *pp = part + (size_t)w * B * plane_elems + q;
    float acc = 0.0f;
    int b = 0;
    for (; b + 8 <= B; b += 8) {
      float v[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = pp[(size_t)(b + i) * plane_elems];
#pragma unroll
      for (int i = 0; i < 8; ++i) acc = __fadd_rn(acc, v[i]);
    }
    for (; b < B; ++b) acc = __fadd_rn(acc, pp[(size_t)b * plane_elems]);
    y[e] = relu ? fmaxf(acc, 0.0f) : acc;
  }
}

}  // namespace

bool fa_f32_supported(const ConvGeom &g) {
  if (g.mode != CCT_FILTER_ADJOINT && g.mode != CCT_FILTER_ADJOINT_BLOCK_REDUCE_SUM) return false;
  if (g.border != CCT_BORDER_VALID || g.down != 1 || g.up != 1 || g.fup != 1) return false;
  if (g.OW > kFaMaxS || g.OH > kFaThreads) return false;
  return (size_t)g.R * g.S * sizeof(float) <= 96 * 1024;
}

size_t fa_workspace_bytes(const ConvGeom &g) {
  if (g.mode != CCT_FILTER_ADJOINT_BLOCK_REDUCE_SUM || g.batch == 1) return 0;
  return (size_t)g.batch * g.n * g.groups * g.OH * g.OW * sizeof(float);
}

int launch_fa_f32(const ConvGeom &g, const float *x, const float *f, float *y, float *work, cudaStream_t st) {
  const bool reduce = g.mode == CCT_FILTER_ADJOINT_BLOCK_REDUCE_SUM && g.batch > 1;
  float *dst = reduce ? work : y;
  if (reduce && !work) return set_error(CCT_EINVAL, "FilterAdjoint block reduce needs plan workspace");
  const int per = kFaThreads / g.OH;
  const int cgroups = (g.n + per - 1) / per;
  const size_t smem = (size_t)g.R * g.S * sizeof(float);
  const long long blocks = (long long)g.batch * g.groups * cgroups;
  if (blocks > 0x7fffffffLL) return set_error(CCT_ENOTSUP, "FilterAdjoint grid too large");
  ConvGeom q = g;
  if (reduce) q.flags &= ~CCT_FLAG_RELU;  // ReLU applies to the reduced sum
  const size_t rsmem = fa_rows_smem(g);
  const long long mgroups = ((long long)g.n * g.OH + 31) / 32, qlgroups = (g.groups + kQL - 1) / kQL;
  const long long qblocks = g.batch * qlgroups * mgroups;
  // up to 400 CTAs: as many rows per step as shared memory holds (us with 16 /
  // 4: 96 CTAs of a 3x3 64 -> 64 layer on 64x64 26 / 63, 160 of a 5x5 32 -> 32
  // on 4x 48x48 39 / 47, 384 of a 3x3 64 -> 64 on 4x 32x32 28 / 32; 1280 of a
  // 5x5 32 -> 64 on 16x 64x64 248 / 224)
  const int nw = qblocks > 400 ? 4 : quad_smem(g, 16) <= kQuadSmemMax ? 16 : quad_smem(g, 8) <= kQuadSmemMax ? 8 : 4;
  const size_t qsmem = quad_smem(g, nw);
  // Gradients of one to three rows leave most of a step's warps idle and its sums'
  // exchange in the open: fa_rows_kernel is the faster one for narrow results, once the
  // grid is more than a wave of latency (us, quad / rows: 1x1 on 16x 38 -> 64 with 5x5
  // results 13.2 / 11.0, 1x4 on 8x 38 -> 26 with 3x3 6.7 / 4.8, 1x8 on 64 -> 64 with 1x1 5.9 / 4.3,
  // 2x2 on 8x 38 -> 26 with 5x5 9.2 / 7.6; but 8x8 results 5.9 / 10.8, 2x2 on 8 -> 8 with 5x5
  // 4.1 / 6.5).
  const bool flat = g.OW <= 5 && g.R <= (g.OW <= 3 ? 3 : 2) && (qblocks >= 150 || (g.R == 1 && g.OW <= 3)) &&
                    rsmem <= kRowsSmemMax;
  if (!flat && g.OH <= kFaMaxS && qsmem <= kQuadSmemMax && qblocks <= 0x7fffffffLL &&
      (long long)g.n * g.OH < (1 << 30)) {
#define CCT_FA_QUAD_CASE(SS)                                                                                  \
  case SS: {                                                                                                  \
    const auto kern = nw == 16 ? fa_quad_kernel<SS, 16> : nw == 8 ? fa_quad_kernel<SS, 8> : fa_quad_kernel<SS, 4>; \
    int rc = raise_smem_limit(kern, qsmem, "cudaFuncSetAttribute(fa quad)");                                  \
    if (rc) return rc;                                                                                        \
    rc = launch_pdl(kern, dim3((unsigned)qblocks), dim3(nw * 32), qsmem, st,                              \
                        "fa_quad_kernel launch", q, x, f, dst, (int)mgroups, (int)qlgroups);                  \
    if (rc) return rc;                                                                                        \
    break;                                                                                                    \
  }
    switch (g.OW) {
      CCT_FA_QUAD_CASE(1) CCT_FA_QUAD_CASE(2) CCT_FA_QUAD_CASE(3) CCT_FA_QUAD_CASE(4)
      CCT_FA_QUAD_CASE(5) CCT_FA_QUAD_CASE(6) CCT_FA_QUAD_CASE(7) CCT_FA_QUAD_CASE(8)
      default: return set_error(CCT_ENOTSUP, "FilterAdjoint result width %d", g.OW);
    }
#undef CCT_FA_QUAD_CASE
    count_launches(1);
  } else if (g.OH <= kFaMaxS && rsmem <= kRowsSmemMax) {
    const int cgroups = (g.n + kCG - 1) / kCG, lgroups = (g.groups + kLG - 1) / kLG;
    const long long rblocks = (long long)g.batch * lgroups * cgroups;
    if (rblocks > 0x7fffffffLL) return set_error(CCT_ENOTSUP, "FilterAdjoint grid too large");
    const int threads = kCG * kLG * g.OH;
#define CCT_FA_ROWS_CASE(SS)                                                                            \
  case SS: {                                                                                            \
    int rc = raise_smem_limit(fa_rows_kernel<SS>, rsmem, "cudaFuncSetAttribute(fa rows)");              \
    if (rc) return rc;                                                                                  \
    fa_rows_kernel<SS><<<(unsigned)rblocks, threads, rsmem, st>>>(q, x, f, dst, cgroups, lgroups);      \
    break;                                                                                              \
  }
    switch (g.OW) {
      CCT_FA_ROWS_CASE(1) CCT_FA_ROWS_CASE(2) CCT_FA_ROWS_CASE(3) CCT_FA_ROWS_CASE(4)
      CCT_FA_ROWS_CASE(5) CCT_FA_ROWS_CASE(6) CCT_FA_ROWS_CASE(7) CCT_FA_ROWS_CASE(8)
      default: return set_error(CCT_ENOTSUP, "FilterAdjoint result width %d", g.OW);
    }
#undef CCT_FA_ROWS_CASE
    count_launches(1);
  } else {
#define CCT_FA_CASE(SS)                                                                               \
  case SS: {                                                                                          \
    int rc = raise_smem_limit(fa_f32_kernel<SS>, smem, "cudaFuncSetAttribute(fa)");                   \
    if (rc) return rc;                                                                                \
    fa_f32_kernel<SS><<<(unsigned)blocks, per * g.OH, smem, st>>>(q, x, f, dst, cgroups);             \
    break;                                                                                            \
  }
  switch (g.OW) {
    CCT_FA_CASE(1) CCT_FA_CASE(2) CCT_FA_CASE(3) CCT_FA_CASE(4)
    CCT_FA_CASE(5) CCT_FA_CASE(6) CCT_FA_CASE(7) CCT_FA_CASE(8)
    default: return set_error(CCT_ENOTSUP, "FilterAdjoint result width %d", g.OW);
  }
#undef CCT_FA_CASE
    count_launches(1);
  }
  if (reduce) {
    const long long planes = (long long)g.n * g.groups;
    const long long n = planes * g.OH * g.OW;
    const int rblocks = (int)std::min<long long>((n + 255) / 256, 148LL * 8);
    int rc = launch_pdl(fa_reduce_kernel, dim3(rblocks), dim3(256), 0, st, "fa_reduce_kernel launch", work, y, g.batch,
                        planes, g.OH * g.OW, (g.flags & CCT_FLAG_RELU) != 0);
    if (rc) return rc;
    count_launches(1);
  }
  return check_cuda(cudaGetLastError(), "FilterAdjoint launch");
}

}  // namespace cct
