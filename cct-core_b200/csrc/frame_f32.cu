// Fused filter-bank convolution in FP32 on the CUDA cores:
//   ProjectFrameBlockReduceSum      y[b*K+k] = sum_c xcorr(x[b*N+c], f[k*N+c])
//   BackProjectFrameBlockReduceSum  y[b*L+l] = sum_n conv (x[b*N+n], f[n*L+l])
// (ConvolveHyperKernel.scala:153-199, 319-340, 574-645, fused by
// ProjectFrameTensorReduceSumOptimizer.scala:75-170).
//
// One CTA owns a 32x16 output tile of one image for a block of 4 or 16 output
// planes.  It walks the N input planes in order; each plane's halo tile and
// the filters' taps for that plane are staged in shared memory with cp.async,
// in three buffers, so the next two planes load while this one computes and
// one barrier per plane suffices.
// A thread holds 4 adjacent outputs x 4 or 8 output planes.  Summation order
// per output matches the reference (per-row fma chain, row sum, plane sum), so
// results are bit-identical to the FP32 CPU restatement.
//
// Bound: the FP32 pipe, R*S packed multiply-adds and R adds per output pair
// (75 % busy on the B=16, C=32, K=64, 64x64, 5x5 layer: 0.165 ms, 41 TFLOP/s;
// 0.269 ms with the staging's index arithmetic repeated for every plane).
//
// The same kernel without the reduce (REDUCE = false) serves the unfused
// modes ProjectFrame / BackProjectFrame (CogFunctionAPI.scala:1370-1377,
// 1425-1432), whose output plane b*F + k*N + c is input plane c of image b
// correlated with one filter: each input plane's tile feeds the 16 filters
// of the block and every result (per-row fma chain, row sum) is stored to
// its own plane.
#include "cct_internal.h"
#include "sm100_util.cuh"
#include "tile_common.cuh"

namespace cct {
namespace {

constexpr int kU = 4;        // adjacent outputs per thread
constexpr int kSX = 8, kSY = 16;  // spatial threads per group
constexpr int kTW = kSX * kU, kTH = kSY;  // 32 x 16 output tile

// KT output planes per thread, KG groups of threads: KT * KG output planes per
// CTA.
template <int R, int S, int DOWN, int KT, int KG>
struct FrameTile {
  static constexpr int KB = KT * KG, THREADS = kSX * kSY * KG;
  static constexpr int IN_COLS = (kTW - 1) * DOWN + S;
  static constexpr int IN_ROWS = (kTH - 1) * DOWN + R;
  static constexpr int PITCH = (IN_COLS + 3) & ~3;
  static constexpr int TILE = IN_ROWS * PITCH;
  // [tap][plane], a tap every 4 or 20 floats: the taps a warp copies fall on 8
  // different banks, and a tap's planes stay 16-byte aligned
  static constexpr int FP = KB == 4 ? 4 : KB + 4;
  static constexpr int FILT = R * S * FP;
  static constexpr int STAGE = TILE + FILT;
  static constexpr int STAGES = 3;
  static constexpr size_t SMEM = sizeof(float) * STAGES * STAGE;
  // elements a thread copies per plane
  static constexpr int NT = (IN_ROWS * IN_COLS + THREADS - 1) / THREADS, NF = (R * S * KB + THREADS - 1) / THREADS;
};

template <int R, int S, int DOWN, bool REDUCE, int KT, int KG>
__global__ void __launch_bounds__(kSX * kSY * KG, KT == 8 ? 2 : 4)
    frame_f32_kernel(ConvGeom g, const float *__restrict__ x,
                     const float *__restrict__ f, float *__restrict__ y,
                     int tiles_x, int tiles_y, int kblocks, int tchunk) {
  grid_dependency_wait();  // launched with programmatic serialisation: nothing global before this
  using T = FrameTile<R, S, DOWN, KT, KG>;
  constexpr int kKT = KT, kKB = T::KB, kThreads = T::THREADS;
  constexpr int E = (kU - 1) * DOWN + S;
  constexpr int E4 = (E + 3) / 4;
  static_assert((kU * DOWN) % 4 == 0, "16-byte aligned thread origin");
  extern __shared__ __align__(16) float smem[];

  int bid = blockIdx.x;
  const int tx_i = bid % tiles_x;
  bid /= tiles_x;
  const int ty_i = bid % tiles_y;
  bid /= tiles_y;
  const int kb = bid % kblocks;
  bid /= kblocks;
  // unfused modes: the input planes are split into chunks of tchunk, one per
  // CTA (their outputs are independent); reduced modes: one chunk of all
  const int nchunks = REDUCE ? 1 : (g.n + tchunk - 1) / tchunk;
  const int t0 = REDUCE ? 0 : (bid % nchunks) * tchunk;
  const int b = bid / nchunks;
  const int k0 = kb * kKB;
  const int kcount = min(kKB, g.groups - k0);

  const int tid = threadIdx.x;
  const int grp = tid / (kSX * kSY);
  const int sp = tid % (kSX * kSY);
  const int tx = sp % kSX, ty = sp / kSX;
  const int out_r0 = ty_i * kTH, out_c0 = tx_i * kTW;
  const int org_r = out_r0 * DOWN - g.low_r;
  const int org_c = out_c0 * DOWN - g.low_c;
  const int plane = g.H * g.W;
  const bool conv = g.orient == CCT_CONVOLUTION;

  // What a thread copies is the same for every input plane but for the plane's
  // address, so the border mapping and the tap order are worked out once (done
  // per plane, they were two fifths of the instructions).
  int t_src[T::NT];  // offset in the input plane, -1 reads zero
#pragma unroll
  for (int e = 0; e < T::NT; ++e) {
    const int i = tid + e * kThreads, tr = i / T::IN_COLS, tc = i - tr * T::IN_COLS;
    const int sr = border_index(g.border, org_r + tr, g.H), sc = border_index(g.border, org_c + tc, g.W);
    t_src[e] = (sr >= 0 && sc >= 0) ? sr * g.W + sc : -1;
  }
  // filter plane of (output plane k, input plane t): k*N + t, or t*K + k for
  // the back-projected forms (plane_pair)
  const bool back = g.mode == CCT_BACK_PROJECT_FRAME || g.mode == CCT_BACK_PROJECT_FRAME_BLOCK_REDUCE_SUM;
  const size_t f_step = back ? (size_t)g.groups * (R * S) : (size_t)(R * S);
  int f_src[T::NF];  // from the block's first filter plane
#pragma unroll
  for (int e = 0; e < T::NF; ++e) {
    const int i = tid + e * kThreads, kk = i / (R * S), tap = i - kk * (R * S);
    f_src[e] = min(kk, kcount - 1) * (back ? 1 : g.n) * (R * S) + (conv ? R * S - 1 - tap : tap);
  }
  const float *ft0 = f + (back ? (size_t)t0 * g.groups + k0 : (size_t)k0 * g.n + t0) * (R * S);
  const float *xt = x + (size_t)(b * g.n + t0) * plane;
  // Stage loader of input-plane term t (called in order).
  auto issue = [&](int t) {
    float *tile = smem + (t % T::STAGES) * T::STAGE;
    float *ft = tile + T::TILE;
#pragma unroll
    for (int e = 0; e < T::NT; ++e) {
      const int i = tid + e * kThreads;
      if (i < T::IN_ROWS * T::IN_COLS) {
        const int tr = i / T::IN_COLS, tc = i - tr * T::IN_COLS;
        cp_async_f32(tile + tr * T::PITCH + tc, t_src[e] >= 0 ? xt + t_src[e] : x, t_src[e] >= 0);
      }
    }
    const float *fp = ft0;
    ft0 += f_step;
#pragma unroll
    for (int e = 0; e < T::NF; ++e) {
      const int i = tid + e * kThreads;
      if (i < R * S * kKB) {
        const int kk = i / (R * S), tap = i - kk * (R * S);
        cp_async_f32(ft + tap * T::FP + kk, fp + f_src[e], kk < kcount);
      }
    }
    xt += plane;
    cp_async_commit();
  };

  // Output planes k, k+1 advance together in packed fma.rn.f32x2 / add.rn.f32x2
  // (each lane the same RN operation as the scalar form, so the order and
  // the result per output are unchanged).
  constexpr int kP = kKT / 2;
  float2 acc[kU][kP];
#pragma unroll
  for (int u = 0; u < kU; ++u)
#pragma unroll
    for (int k = 0; k < kP; ++k) acc[u][k] = make_float2(0.0f, 0.0f);

  const int nterms = REDUCE ? g.terms : min(tchunk, g.n - t0);
  const bool relu = (g.flags & CCT_FLAG_RELU) != 0;
  const size_t opage = (size_t)g.OH * g.OW;
  const int row = out_r0 + ty;
  auto next = [&](int t) {  // an empty group past the last plane
    if (t < nterms)
      issue(t);
    else
      cp_async_commit();
  };
  next(0);
  next(1);
  for (int t = 0; t < nterms; ++t) {
    cp_async_wait<1>();
    __syncthreads();  // plane t has landed, and every thread is done with plane t - 1
    next(t + 2);
    const float *tile = smem + (t % T::STAGES) * T::STAGE;
    const float *ft = tile + T::TILE + grp * kKT;
    const float *base = tile + (ty * DOWN) * T::PITCH + tx * kU * DOWN;

    float2 rs[kU][kP];
#pragma unroll
    for (int u = 0; u < kU; ++u)
#pragma unroll
      for (int k = 0; k < kP; ++k) rs[u][k] = make_float2(0.0f, 0.0f);

#pragma unroll
    for (int r = 0; r < R; ++r) {
      float vals[E4 * 4];
#pragma unroll
      for (int e = 0; e < E4; ++e) {
        const float4 q = *reinterpret_cast<const float4 *>(base + r * T::PITCH + 4 * e);
        vals[4 * e + 0] = q.x;
        vals[4 * e + 1] = q.y;
        vals[4 * e + 2] = q.z;
        vals[4 * e + 3] = q.w;
      }
      float2 cs[kU][kP];
#pragma unroll
      for (int s = 0; s < S; ++s) {
        float2 w[kP];
#pragma unroll
        for (int k4 = 0; k4 < kKT / 4; ++k4) {
          const float4 q = *reinterpret_cast<const float4 *>(ft + (r * S + s) * T::FP + 4 * k4);
          w[2 * k4 + 0] = make_float2(q.x, q.y);
          w[2 * k4 + 1] = make_float2(q.z, q.w);
        }
#pragma unroll
        for (int u = 0; u < kU; ++u) {
          const float xv = vals[u * DOWN + s];
          const float2 x2 = make_float2(xv, xv);
#pragma unroll
          for (int k = 0; k < kP; ++k)
            cs[u][k] = __ffma2_rn(x2, w[k], s == 0 ? make_float2(0.0f, 0.0f) : cs[u][k]);
        }
      }
#pragma unroll
      for (int u = 0; u < kU; ++u)
#pragma unroll
        for (int k = 0; k < kP; ++k) rs[u][k] = __fadd2_rn(rs[u][k], cs[u][k]);
    }
    if (REDUCE) {
#pragma unroll
      for (int u = 0; u < kU; ++u)
#pragma unroll
        for (int k = 0; k < kP; ++k) acc[u][k] = (t == 0) ? rs[u][k] : __fadd2_rn(acc[u][k], rs[u][k]);
    } else if (row < g.OH) {
      // this input plane's result for each filter of the block: its own plane
      const int col0 = out_c0 + tx * kU;
      const bool vec = (g.OW & 3) == 0 && col0 + kU <= g.OW;
#pragma unroll
      for (int k = 0; k < kKT; ++k) {
        const int kk = grp * kKT + k;
        if (kk >= kcount) break;
        float *ys = y + (size_t)(b * g.pf + (k0 + kk) * g.n + t0 + t) * opage + (size_t)row * g.OW;
        float v[kU];
#pragma unroll
        for (int u = 0; u < kU; ++u) {
          const float a = (k & 1) ? rs[u][k >> 1].y : rs[u][k >> 1].x;
          v[u] = relu ? fmaxf(a, 0.0f) : a;
        }
        if (vec) {
          *reinterpret_cast<float4 *>(ys + col0) = make_float4(v[0], v[1], v[2], v[3]);
        } else {
#pragma unroll
          for (int u = 0; u < kU; ++u)
            if (col0 + u < g.OW) ys[col0 + u] = v[u];
        }
      }
    }
  }

  if constexpr (REDUCE) {
    if (row >= g.OH) return;
#pragma unroll
    for (int k = 0; k < kKT; ++k) {
      const int kk = grp * kKT + k;
      if (kk >= kcount) break;
      float *ys = y + (size_t)(b * g.groups + k0 + kk) * opage + (size_t)row * g.OW;
#pragma unroll
      for (int u = 0; u < kU; ++u) {
        const int col = out_c0 + tx * kU + u;
        const float a = (k & 1) ? acc[u][k >> 1].y : acc[u][k >> 1].x;
        if (col < g.OW) ys[col] = relu ? fmaxf(a, 0.0f) : a;
      }
    }
  }
}

template <int R, int S, int DOWN, bool REDUCE, int KT, int KG>
int launch_k(const ConvGeom &g, const float *x, const float *f, float *y, cudaStream_t st) {
  using T = FrameTile<R, S, DOWN, KT, KG>;
  const int tiles_x = (g.OW + kTW - 1) / kTW, tiles_y = (g.OH + kTH - 1) / kTH;
  const int kblocks = (g.groups + T::KB - 1) / T::KB;
  const int tchunk = REDUCE ? g.terms : 4;  // unfused: 4 input planes per CTA
  const int nchunks = REDUCE ? 1 : (g.n + tchunk - 1) / tchunk;
  const long long blocks = (long long)tiles_x * tiles_y * kblocks * nchunks * g.batch;
  if (blocks > 0x7fffffffLL) return set_error(CCT_ENOTSUP, "frame grid too large");
  const auto kern = frame_f32_kernel<R, S, DOWN, REDUCE, KT, KG>;
  int rc = raise_smem_limit(kern, T::SMEM, "cudaFuncSetAttribute(frame_f32)");
  if (rc) return rc;
  rc = launch_pdl(kern, dim3((unsigned)blocks), dim3(T::THREADS), T::SMEM, st,
                            "frame_f32_kernel launch", g, x, f, y, tiles_x, tiles_y, kblocks, tchunk);
  if (!rc) count_launches(1);
  return rc;
}

template <int R, int S, int DOWN>
int launch(const ConvGeom &g, const float *x, const float *f, float *y, cudaStream_t st) {
  if (g.mode != CCT_PROJECT_FRAME_BLOCK_REDUCE_SUM && g.mode != CCT_BACK_PROJECT_FRAME_BLOCK_REDUCE_SUM)
    return launch_k<R, S, DOWN, false, 8, 2>(g, x, f, y, st);
  // 16 output planes per CTA re-use a staged tile four times as often, which
  // pays for filters of up to 3x3 while that grid fills the SMs; larger filters
  // are bound by the multiply-adds either way, and four times the CTAs spread
  // better (us, 16 / 4 planes per CTA: 3x3 32 -> 64 planes on 16x 64x64, 512 CTAs
  // 83 / 93; 3x3 32 -> 16 on 64x 32x32, 128 CTAs 26 / 30; 3x3 64 -> 64 on 8x 32x32,
  // 64 CTAs 48 / 32; 5x5 32 -> 64 on 16x 64x64 169 / 165; 7x7 309 / 285; 5x5
  // 32 -> 32 on 4x 48x48 49 / 29).
  const long long blocks16 = (long long)((g.OW + kTW - 1) / kTW) * ((g.OH + kTH - 1) / kTH) * g.batch *
                             ((g.groups + 15) / 16);
  const bool full16 = (g.groups + 15) / 16 * 16 * 4 <= g.groups * 5;  // at most a fifth of the planes idle
  // DownsampleOutput(2) stages four times the field per output, so there every size takes 16
  // planes, 1x1 from 40 CTAs on (us, 16 / 4, clamp: 1x1 10 -> 47 planes on 16x 40x14 14 / 31; 5x5
  // 23 -> 117 on 16x 48x34 96 / 166; 7x7 8 -> 143 on 8x 40x80 61 / 101; at 192 CTAs and zero
  // borders about even: 5x5 25 -> 44 on 16x 40x114 82 / 70).
  if constexpr (R <= 3 || DOWN == 2) {
    if (blocks16 >= (R == 1 && DOWN == 2 ? 40 : 128) && full16) return launch_k<R, S, DOWN, true, 8, 2>(g, x, f, y, st);
  }
  return launch_k<R, S, DOWN, true, 4, 1>(g, x, f, y, st);
}

}  // namespace

bool frame_f32_supported(const ConvGeom &g) {
  if (g.mode != CCT_PROJECT_FRAME_BLOCK_REDUCE_SUM && g.mode != CCT_BACK_PROJECT_FRAME_BLOCK_REDUCE_SUM &&
      g.mode != CCT_PROJECT_FRAME && g.mode != CCT_BACK_PROJECT_FRAME)
    return false;
  if (g.up != 1) return false;
  if (g.R != g.S) return false;
  // a block's filter offsets and a plane's element offsets are 32-bit
  if (16LL * g.n * g.R * g.S > 0x7fffffffLL || (long long)g.H * g.W > 0x7fffffffLL) return false;
  if (g.down != 1 && g.down != 2) return false;
  return g.R == 1 || g.R == 3 || g.R == 5 || g.R == 7 || g.R == 9;
}

int launch_frame_f32(const ConvGeom &g, const float *x, const float *f, float *y,
                     cudaStream_t st) {
#define CCT_FRAME_CASE(RR, DD) \
  if (g.R == RR && g.down == DD) return launch<RR, RR, DD>(g, x, f, y, st);
  CCT_FRAME_CASE(1, 1) CCT_FRAME_CASE(3, 1) CCT_FRAME_CASE(5, 1) CCT_FRAME_CASE(7, 1) CCT_FRAME_CASE(9, 1)
  CCT_FRAME_CASE(1, 2) CCT_FRAME_CASE(3, 2) CCT_FRAME_CASE(5, 2) CCT_FRAME_CASE(7, 2) CCT_FRAME_CASE(9, 2)
#undef CCT_FRAME_CASE
  return set_error(CCT_ENOTSUP, "frame FP32 kernel: unsupported filter %dx%d step %d", g.R, g.S,
                   g.down);
}

}  // namespace cct
