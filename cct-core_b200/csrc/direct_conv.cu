// Direct (stencil) field convolution: one output plane per CTA column of
// tiles, halo tile staged in shared memory, register-blocked outputs.
//
// Every output follows the summation order of the reference's generated
// OpenCL (ConvolveHyperKernel.scala:509-521 and :593-603): for each filter
// row a fused multiply-add chain over the filter columns starting from 0
// (`columnSum`), added into `rowSum`; frame reductions add `rowSum` of each
// input plane in increasing plane order.  The explicit __fmaf_rn/__fadd_rn
// keep nvcc from contracting the adds, so results are bit-identical to the
// CPU restatement of that order.
#include <algorithm>

#include "cct_internal.h"
#include "sm100_util.cuh"
#include "stencil.cuh"
#include "tile_common.cuh"

namespace cct {
namespace {

constexpr int kThreads = 256;
constexpr int kTX = 16, kTY = 16;  // thread grid of the square and the generic kernel

// ---------------------------------------------------------------------------
// Small square filters (weights in registers), down-sampling 1 or 2, every
// border and width.  A CTA of 128 threads computes 64 columns x 8 V rows; a
// thread owns 4 adjacent columns x V rows, so a staged row it reads (float4,
// lanes contiguous) feeds up to R output rows.
//
// Bound: FP32 issue (R*S multiply-adds and R adds per output) for 7x7, HBM
// below that.  Overlap of staging and arithmetic comes from the 4-5 CTAs an SM
// holds.  V = 8 amortises the R-1 extra rows and the staging; planes whose
// V = 8 grid would not give every SM a CTA take V = 2.
constexpr int kSmThreads = 128, kSmU = 4, kSmTX = 16, kSmTY = 8;
constexpr int kSmTW = kSmTX * kSmU;

// First staged column relative to the output's centred window, for 16-byte
// staging (TileStage): the columns before it that round the origin down.
__host__ __device__ constexpr int vec_off(int S, bool VEC) { return VEC ? (4 - ((S - 1) / 2) % 4) % 4 : 0; }

template <int R, int S, int DOWN, int V, bool VEC>
__global__ void __launch_bounds__(kSmThreads, R == 7 ? 3 : 4)
    direct_small_kernel(ConvGeom g, const float *__restrict__ x, const float *__restrict__ f,
                        float *__restrict__ y, int tiles_x, int tiles_y) {
  constexpr int U = kSmU, TW = kSmTW, TH = kSmTY * V, OFF = vec_off(S, VEC);
  constexpr int IN_COLS = VEC ? (OFF + (TW - 1) * DOWN + S + 3) & ~3 : (TW - 1) * DOWN + S;
  constexpr int IN_ROWS = (TH - 1) * DOWN + R;
  constexpr int PITCH = (IN_COLS + 3) & ~3;
  constexpr int E = OFF + (U - 1) * DOWN + S;
  constexpr int E4 = (E + 3) / 4;
  // the thread's last float4 may read past the last staged row
  constexpr int SLACK = 4 * E4 + (TW - U) * DOWN > PITCH ? 4 * E4 + (TW - U) * DOWN - PITCH : 0;
  __shared__ __align__(16) float tile[IN_ROWS * PITCH + SLACK];
  grid_dependency_wait();  // launched with programmatic serialisation: nothing global before this

  int bid = blockIdx.x;
  const int tx_i = bid % tiles_x;
  bid /= tiles_x;
  const int ty_i = bid % tiles_y;
  const int o = bid / tiles_y;
  const int tx = threadIdx.x % kSmTX, ty = threadIdx.x / kSmTX;
  const int out_r0 = ty_i * TH, out_c0 = tx_i * TW;
  const int org_r = out_r0 * DOWN - g.low_r;
  const int rows = min(TH, g.OH - out_r0);  // output rows of this tile
  const TileStage<IN_COLS, PITCH, kSmThreads, VEC> stage(g, out_c0 * DOWN - g.low_c - OFF,
                                                         OFF + (min(TW, g.OW - out_c0) - 1) * DOWN + S);

  float acc[V][U];
  for (int t = 0; t < g.terms; ++t) {
    int ip, fp;
    plane_pair(g, o, t, &ip, &fp);
    const float *fs = f + (size_t)fp * (R * S);
    if (t > 0) __syncthreads();
    stage.copy(tile, x + (size_t)ip * g.H * g.W, g, org_r, (rows - 1) * DOWN + R);
    cp_async_commit();
    float w[R][S];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int s = 0; s < S; ++s)
        w[r][s] = __ldg(fs + (g.orient == CCT_CONVOLUTION ? (R - 1 - r) * S + (S - 1 - s) : r * S + s));
    cp_async_wait<0>();
    __syncthreads();

    if (ty * V < rows) {
      float rs[V][U];
#pragma unroll
      for (int v = 0; v < V; ++v)
#pragma unroll
        for (int u = 0; u < U; ++u) rs[v][u] = 0.0f;
      const float *base = tile + (ty * V * DOWN) * PITCH + tx * U * DOWN;
#pragma unroll
      for (int tr = 0; tr < (V - 1) * DOWN + R; ++tr) {
        float vals[E4 * 4];
#pragma unroll
        for (int e = 0; e < E4; ++e) {
          const float4 q = *reinterpret_cast<const float4 *>(base + tr * PITCH + 4 * e);
          vals[4 * e + 0] = q.x;
          vals[4 * e + 1] = q.y;
          vals[4 * e + 2] = q.z;
          vals[4 * e + 3] = q.w;
        }
#pragma unroll
        for (int v = 0; v < V; ++v) {
          const int r = tr - v * DOWN;
          if (r >= 0 && r < R) {
#pragma unroll
            for (int u = 0; u < U; ++u) {
              float cs = 0.0f;
#pragma unroll
              for (int s = 0; s < S; ++s) cs = __fmaf_rn(vals[OFF + u * DOWN + s], w[r][s], cs);
              rs[v][u] = __fadd_rn(rs[v][u], cs);
            }
          }
        }
      }
#pragma unroll
      for (int v = 0; v < V; ++v)
#pragma unroll
        for (int u = 0; u < U; ++u) acc[v][u] = (t == 0) ? rs[v][u] : __fadd_rn(acc[v][u], rs[v][u]);
    }
  }
  allow_dependent_launch();

  float *ys = y + (size_t)o * g.OH * g.OW;
  if ((g.flags & CCT_FLAG_RELU) != 0) {
#pragma unroll
    for (int v = 0; v < V; ++v)
#pragma unroll
      for (int u = 0; u < U; ++u) acc[v][u] = fmaxf(acc[v][u], 0.0f);
  }
  if ((g.OW & 3) == 0 && (reinterpret_cast<uintptr_t>(y) & 15) == 0) {
    const int col = out_c0 + tx * U;
    if (col >= g.OW) return;
#pragma unroll
    for (int v = 0; v < V; ++v)
      if (ty * V + v < rows)
        *reinterpret_cast<float4 *>(ys + (size_t)(out_r0 + ty * V + v) * g.OW + col) =
            make_float4(acc[v][0], acc[v][1], acc[v][2], acc[v][3]);
    return;
  }
  // Rows that are not 16-byte aligned: through the tile (a row of it holds at
  // least 64 floats), so that a warp stores 32 adjacent values at a time.
  __syncthreads();
#pragma unroll
  for (int v = 0; v < V; ++v)
    *reinterpret_cast<float4 *>(tile + (ty * V + v) * TW + tx * U) =
        make_float4(acc[v][0], acc[v][1], acc[v][2], acc[v][3]);
  __syncwarp();
  const int w0 = (threadIdx.x >> 5) * 2 * V;  // a warp's lanes are two rows of threads
  if (w0 < rows)
    store_rows64(ys + (size_t)(out_r0 + w0) * g.OW + out_c0, g.OW, tile + w0 * TW, TW, min(2 * V, rows - w0),
               min(TW, g.OW - out_c0), threadIdx.x & 31);
}

// ---------------------------------------------------------------------------
// Wide filters: S odd, 3..63, any R, no sampling, one term.  Weights come from
// shared memory as broadcast float4s, so a thread owns 8 adjacent columns: a
// weight load feeds 32 multiply-adds and the row of 8 + S - 1 inputs it holds
// in registers feeds V output rows (one input per multiply-add came from
// shared memory before: 1.6 TFLOP/s on 480x640 with sixteen 11x11 filters).
// Bound: FP32 issue, R*S multiply-adds and R adds per output.
// A warp's 8-lane float4 phases cover 4 column groups x 2 rows of threads; V
// odd and a pitch of 4 (mod 8) floats put them on different banks.  Seven CTAs an
// SM up to 9 columns (732x64 by sixty-four 9x9 filters 16.6 us, 18.3 with six).
constexpr int kWdThreads = 128, kWdU = 8, kWdTX = 8, kWdTY = 16;
constexpr int kWdTW = kWdTX * kWdU;

__host__ __device__ constexpr int wide_pitch(int S) {
  const int c = (kWdTW + S - 1 + 3) & ~3;
  return (c & 7) == 4 ? c : c + 4;
}
// floats: the tile (which also holds the finished 64-wide rows) and the weights
inline size_t wide_smem(int R, int S, int V) {
  return sizeof(float) * ((size_t)(kWdTY * V + R - 1) * wide_pitch(S) + (size_t)R * ((S + 3) & ~3));
}

template <int S, int V>
__global__ void __launch_bounds__(kWdThreads, V == 1 ? 8 : S > 9 ? 6 : 7)
    direct_wide_kernel(ConvGeom g, const float *__restrict__ x, const float *__restrict__ f,
                       float *__restrict__ y, int tiles_x, int tiles_y) {
  constexpr int U = kWdU, TW = kWdTW, TH = kWdTY * V, PITCH = wide_pitch(S), SP = (S + 3) & ~3;
  constexpr int E4 = (U + S - 1 + 3) / 4;
  static_assert((V & 1) == 1, "odd V: rows of threads on different banks");
  static_assert(4 * E4 + TW - U <= PITCH, "a thread's loads stay inside its row");
  extern __shared__ __align__(16) float smem[];
  grid_dependency_wait();  // launched with programmatic serialisation: nothing global before this
  const int R = g.R;
  float *tile = smem, *wf = smem + (TH + R - 1) * PITCH;

  int bid = blockIdx.x;
  const int tx_i = bid % tiles_x;
  bid /= tiles_x;
  const int ty_i = bid % tiles_y;
  const int o = bid / tiles_y;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tx = (lane & 3) | ((lane >> 1) & 4), ty = warp * 4 + (((lane >> 2) & 1) | ((lane >> 3) & 2));
  const int out_r0 = ty_i * TH, out_c0 = tx_i * TW;
  const int rows = min(TH, g.OH - out_r0);
  int ip, fp;
  plane_pair(g, o, 0, &ip, &fp);
  {
    const TileStage<TW + S - 1, PITCH, kWdThreads, false> stage(g, out_c0 - g.low_c,
                                                                   min(TW, g.OW - out_c0) + S - 1);
    stage.copy(tile, x + (size_t)ip * g.H * g.W, g, out_r0 - g.low_r, rows + R - 1);
    cp_async_commit();
  }
  const float *fs = f + (size_t)fp * R * S;
  for (int i = threadIdx.x; i < R * S; i += kWdThreads) {
    const int r = i / S, s = i - r * S;
    wf[r * SP + s] = __ldg(fs + (g.orient == CCT_CONVOLUTION ? R * S - 1 - i : i));
  }
  cp_async_wait<0>();
  __syncthreads();

  float rs[V][U];
#pragma unroll
  for (int v = 0; v < V; ++v)
#pragma unroll
    for (int u = 0; u < U; ++u) rs[v][u] = 0.0f;
  if (warp * 4 * V < rows) {
    const float *base = tile + (ty * V) * PITCH + tx * U;
#pragma unroll 1
    for (int tr = 0; tr < V - 1 + R; ++tr) {
      float vals[E4 * 4];
#pragma unroll
      for (int e = 0; e < E4; ++e) {
        const float4 q = *reinterpret_cast<const float4 *>(base + tr * PITCH + 4 * e);
        vals[4 * e + 0] = q.x;
        vals[4 * e + 1] = q.y;
        vals[4 * e + 2] = q.z;
        vals[4 * e + 3] = q.w;
      }
#pragma unroll
      for (int v = 0; v < V; ++v) {
        const int r = tr - v;
        if (r >= 0 && r < R) {  // the same for every thread
          const float *wr = wf + r * SP;
          float cs[U];
#pragma unroll
          for (int s4 = 0; s4 < SP; s4 += 4) {
            const float4 q = *reinterpret_cast<const float4 *>(wr + s4);
            const float w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const int s = s4 + k;
              if (s < S) {
#pragma unroll
                for (int u = 0; u < U; ++u) cs[u] = __fmaf_rn(vals[u + s], w[k], s == 0 ? 0.0f : cs[u]);
              }
            }
          }
#pragma unroll
          for (int u = 0; u < U; ++u) rs[v][u] = __fadd_rn(rs[v][u], cs[u]);
        }
      }
    }
  }
  allow_dependent_launch();
  const bool relu = (g.flags & CCT_FLAG_RELU) != 0;
  __syncthreads();  // the tile is read: it now takes the finished rows
#pragma unroll
  for (int v = 0; v < V; ++v) {
    if (relu) {
#pragma unroll
      for (int u = 0; u < U; ++u) rs[v][u] = fmaxf(rs[v][u], 0.0f);
    }
#pragma unroll
    for (int e = 0; e < U / 4; ++e)
      *reinterpret_cast<float4 *>(tile + (ty * V + v) * PITCH + tx * U + 4 * e) =
          make_float4(rs[v][4 * e], rs[v][4 * e + 1], rs[v][4 * e + 2], rs[v][4 * e + 3]);
  }
  __syncwarp();
  const int w0 = warp * 4 * V;
  if (w0 < rows)
    store_rows64(y + (size_t)o * g.OH * g.OW + (size_t)(out_r0 + w0) * g.OW + out_c0, g.OW, tile + w0 * PITCH, PITCH,
               min(4 * V, rows - w0), min(TW, g.OW - out_c0), lane);
}

// ---------------------------------------------------------------------------
// UpsampleInput by UP (2 or 3), R x R filters centred on the output.  Output
// (UP I + p, UP J + q) takes only the taps that land on field values: rows
// r = UP d - p + low for d = DMIN..DMAX (columns likewise), reading field row
// I + d.  A thread owns 4 field columns x V field rows and computes all UP^2
// phases of them from one register window, in the reference's tap order
// (ConvolveHyperKernel.scala:405-436 visits exactly those taps); a quarter
// (ninth) of the multiply-adds of running the zero-inserted grid.
// Bound: HBM (UP^2 floats written per float read); rows leave through shared
// memory so that a warp's stores are contiguous.
template <int R, int UP, int V>
struct UpTile {
  static constexpr int LOW = (R - 1) / 2;
  static constexpr int DMIN = -(LOW / UP), DMAX = (UP - 1 + LOW) / UP, D = DMAX - DMIN;
  static constexpr int TW = kSmTW, TH = kSmTY * V;              // field positions per CTA
  static constexpr int IN_ROWS = TH + D, IN_COLS = TW + D;
  static constexpr int E4 = (kSmU + D + 3) / 4;
  static constexpr int PITCH = TW - kSmU + 4 * E4;
  static constexpr int OUT_PITCH = TW * UP, OUT_ROWS = UP;       // one field row of a warp at a time
};

template <int R, int UP, int V>
__global__ void __launch_bounds__(kSmThreads, R == 9 ? 2 : R == 7 || UP == 3 ? 3 : 4)
    direct_up_kernel(ConvGeom g, const float *__restrict__ x, const float *__restrict__ f, float *__restrict__ y,
                     int tiles_x, int tiles_y) {
  using T = UpTile<R, UP, V>;
  constexpr int U = kSmU, LOW = T::LOW;
  __shared__ __align__(16) float tile[T::IN_ROWS * T::PITCH];
  __shared__ __align__(16) float out[kSmTY][T::OUT_ROWS * T::OUT_PITCH];
  grid_dependency_wait();  // launched with programmatic serialisation: nothing global before this

  int bid = blockIdx.x;
  const int tx_i = bid % tiles_x;
  bid /= tiles_x;
  const int ty_i = bid % tiles_y;
  const int o = bid / tiles_y;
  const int tx = threadIdx.x % kSmTX, ty = threadIdx.x / kSmTX;
  const int r0 = ty_i * T::TH, c0 = tx_i * T::TW;
  const int rows = min(T::TH, g.H - r0), cols = min(T::TW, g.W - c0);
  const TileStage<T::IN_COLS, T::PITCH, kSmThreads, false> stage(g, c0 + T::DMIN, cols + T::D);

  float acc[V][UP][UP][U];
  for (int t = 0; t < g.terms; ++t) {
    int ip, fp;
    plane_pair(g, o, t, &ip, &fp);
    const float *fs = f + (size_t)fp * (R * R);
    if (t > 0) __syncthreads();
    stage.copy(tile, x + (size_t)ip * g.H * g.W, g, r0 + T::DMIN, rows + T::D);
    cp_async_commit();
    float w[R][R];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int s = 0; s < R; ++s)
        w[r][s] = __ldg(fs + (g.orient == CCT_CONVOLUTION ? (R - 1 - r) * R + (R - 1 - s) : r * R + s));
    cp_async_wait<0>();
    __syncthreads();
    if (ty * V >= rows) continue;

    float rs[V][UP][UP][U];
#pragma unroll
    for (int v = 0; v < V; ++v)
#pragma unroll
      for (int p = 0; p < UP; ++p)
#pragma unroll
        for (int q = 0; q < UP; ++q)
#pragma unroll
          for (int u = 0; u < U; ++u) rs[v][p][q][u] = 0.0f;
    const float *base = tile + (ty * V) * T::PITCH + tx * U;
#pragma unroll
    for (int tr = 0; tr < V + T::D; ++tr) {
      float vals[4 * T::E4];
#pragma unroll
      for (int e = 0; e < T::E4; ++e) {
        const float4 q = *reinterpret_cast<const float4 *>(base + tr * T::PITCH + 4 * e);
        vals[4 * e + 0] = q.x;
        vals[4 * e + 1] = q.y;
        vals[4 * e + 2] = q.z;
        vals[4 * e + 3] = q.w;
      }
#pragma unroll
      for (int v = 0; v < V; ++v)
#pragma unroll
        for (int p = 0; p < UP; ++p) {
          const int r = UP * (tr - v + T::DMIN) - p + LOW;
          if (tr - v >= 0 && tr - v <= T::D && r >= 0 && r < R) {
#pragma unroll
            for (int q = 0; q < UP; ++q)
#pragma unroll
              for (int u = 0; u < U; ++u) {
                float cs = 0.0f;
#pragma unroll
                for (int d = 0; d <= T::D; ++d) {
                  const int s = UP * (d + T::DMIN) - q + LOW;
                  if (s >= 0 && s < R) cs = __fmaf_rn(vals[u + d], w[r][s], cs);
                }
                rs[v][p][q][u] = __fadd_rn(rs[v][p][q][u], cs);
              }
          }
        }
    }
#pragma unroll
    for (int v = 0; v < V; ++v)
#pragma unroll
      for (int p = 0; p < UP; ++p)
#pragma unroll
        for (int q = 0; q < UP; ++q)
#pragma unroll
          for (int u = 0; u < U; ++u)
            acc[v][p][q][u] = (t == 0) ? rs[v][p][q][u] : __fadd_rn(acc[v][p][q][u], rs[v][p][q][u]);
  }
  allow_dependent_launch();

  // One field row of each row of threads at a time: its UP output rows are
  // laid out in shared memory by the 16 threads that own it (half a warp) and
  // stored by them, 16 adjacent values at a time or float4s.
  const bool relu = (g.flags & CCT_FLAG_RELU) != 0;
  const bool vec = (g.OW & 3) == 0 && (reinterpret_cast<uintptr_t>(y) & 15) == 0;
  float *mine = out[ty];
#pragma unroll
  for (int v = 0; v < V; ++v) {
    __syncwarp();
#pragma unroll
    for (int p = 0; p < UP; ++p) {
      float line[U * UP];
#pragma unroll
      for (int q = 0; q < UP; ++q)
#pragma unroll
        for (int u = 0; u < U; ++u) line[u * UP + q] = relu ? fmaxf(acc[v][p][q][u], 0.0f) : acc[v][p][q][u];
#pragma unroll
      for (int e = 0; e < UP; ++e)
        *reinterpret_cast<float4 *>(mine + p * T::OUT_PITCH + tx * U * UP + 4 * e) =
            make_float4(line[4 * e], line[4 * e + 1], line[4 * e + 2], line[4 * e + 3]);
    }
    __syncwarp();
    if (ty * V + v < rows) {
      float *dst = y + (size_t)o * g.OH * g.OW + (size_t)(r0 + ty * V + v) * UP * g.OW + c0 * UP;
      for (int p = 0; p < UP; ++p) {
        if (vec) {
          for (int c = tx; c < cols * UP / 4; c += kSmTX)
            reinterpret_cast<float4 *>(dst + (size_t)p * g.OW)[c] =
                reinterpret_cast<const float4 *>(mine + p * T::OUT_PITCH)[c];
        } else {
          for (int c = tx; c < cols * UP; c += kSmTX) dst[(size_t)p * g.OW + c] = mine[p * T::OUT_PITCH + c];
        }
      }
    }
  }
}

// ---------------------------------------------------------------------------
// Squares over a zero-inserted grid that direct_up_kernel does not take
// (UpsampleInput by 4 and more, BorderFull and BorderValid, 1x1): weights in
// registers, 64 x 64 outputs a CTA, 4 x 4 a thread, the grid staged as it stands.
// Bound: the staging, a division and a border mapping per staged value, which
// is why 256 threads share a tile: 128 with twice the outputs took 1.2 to 2 times
// as long, the general kernel below up to 2.7 (7x7 step 5, 569x620: 81 us here,
// 119, 216).
template <int R>
__global__ void __launch_bounds__(kThreads)
    direct_square_kernel(ConvGeom g, const float *__restrict__ x, const float *__restrict__ f,
                         float *__restrict__ y, int tiles_x, int tiles_y) {
  grid_dependency_wait();  // launched with programmatic serialisation: nothing global before this
  constexpr int S = R, U = 4, V = 4, TW = kTX * U, TH = kTY * V;
  constexpr int IN_COLS = TW - 1 + S;
  constexpr int IN_ROWS = TH - 1 + R;
  constexpr int PITCH = (IN_COLS + 3) & ~3;
  constexpr int E = U - 1 + S;  // values per tile row per thread
  constexpr int E4 = (E + 3) / 4;
  __shared__ __align__(16) float tile[IN_ROWS * PITCH];

  int bid = blockIdx.x;
  const int tx_i = bid % tiles_x;
  bid /= tiles_x;
  const int ty_i = bid % tiles_y;
  const int o = bid / tiles_y;
  const int tx = threadIdx.x % kTX, ty = threadIdx.x / kTX;
  const int out_r0 = ty_i * TH, out_c0 = tx_i * TW;
  const int org_r = out_r0 - g.low_r;
  const int org_c = out_c0 - g.low_c;

  float acc[V][U];
#pragma unroll
  for (int v = 0; v < V; ++v)
#pragma unroll
    for (int u = 0; u < U; ++u) acc[v][u] = 0.0f;

  for (int t = 0; t < g.terms; ++t) {
    int ip, fp;
    plane_pair(g, o, t, &ip, &fp);
    const float *xs = x + (size_t)ip * g.H * g.W;
    const float *fs = f + (size_t)fp * (R * S);
    float w[R][S];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int s = 0; s < S; ++s)
        w[r][s] = __ldg(fs + (g.orient == CCT_CONVOLUTION ? (R - 1 - r) * S + (S - 1 - s) : r * S + s));
    if (t > 0) __syncthreads();
    load_tile(tile, PITCH, IN_ROWS, IN_COLS, xs, g, org_r, org_c);
    __syncthreads();

    float rs[V][U];
#pragma unroll
    for (int v = 0; v < V; ++v)
#pragma unroll
      for (int u = 0; u < U; ++u) rs[v][u] = 0.0f;

    const float *base = tile + (ty * V) * PITCH + tx * U;
#pragma unroll
    for (int tr = 0; tr < V - 1 + R; ++tr) {
      float vals[E4 * 4];
#pragma unroll
      for (int e = 0; e < E4; ++e) {
        const float4 q = *reinterpret_cast<const float4 *>(base + tr * PITCH + 4 * e);
        vals[4 * e + 0] = q.x;
        vals[4 * e + 1] = q.y;
        vals[4 * e + 2] = q.z;
        vals[4 * e + 3] = q.w;
      }
#pragma unroll
      for (int v = 0; v < V; ++v) {
        const int r = tr - v;
        if (r >= 0 && r < R) {
#pragma unroll
          for (int u = 0; u < U; ++u) {
            float cs = 0.0f;
#pragma unroll
            for (int s = 0; s < S; ++s) cs = __fmaf_rn(vals[u + s], w[r][s], cs);
            rs[v][u] = __fadd_rn(rs[v][u], cs);
          }
        }
      }
    }
#pragma unroll
    for (int v = 0; v < V; ++v)
#pragma unroll
      for (int u = 0; u < U; ++u)
        acc[v][u] = (t == 0) ? rs[v][u] : __fadd_rn(acc[v][u], rs[v][u]);
  }

  float *ys = y + (size_t)o * g.OH * g.OW;
  const bool relu = (g.flags & CCT_FLAG_RELU) != 0;
#pragma unroll
  for (int v = 0; v < V; ++v) {
    const int row = out_r0 + ty * V + v;
    if (row >= g.OH) continue;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int col = out_c0 + tx * U + u;
      if (col < g.OW) ys[(size_t)row * g.OW + col] = relu ? fmaxf(acc[v][u], 0.0f) : acc[v][u];
    }
  }
}

// Any filter size and down-sampling step: filter staged in shared memory,
// four outputs along a row per thread.
constexpr int kGU = 4;                       // outputs per thread (columns)
constexpr int kGTW = kTX * kGU, kGTH = kTY;  // 64 x 16 output tile

__global__ void __launch_bounds__(kThreads)
    direct_generic_kernel(ConvGeom g, const float *__restrict__ x,
                          const float *__restrict__ f, float *__restrict__ y,
                          int tiles_x, int tiles_y, int in_rows, int in_cols,
                          int pitch) {
  grid_dependency_wait();  // launched with programmatic serialisation: nothing global before this
  extern __shared__ __align__(16) float smem[];
  float *tile = smem;
  float *wf = smem + in_rows * pitch;

  int bid = blockIdx.x;
  const int tx_i = bid % tiles_x;
  bid /= tiles_x;
  const int ty_i = bid % tiles_y;
  const int o = bid / tiles_y;
  const int tx = threadIdx.x % kTX, ty = threadIdx.x / kTX;
  const int out_r0 = ty_i * kGTH, out_c0 = tx_i * kGTW;
  const int org_r = out_r0 * g.down - g.low_r;
  const int org_c = out_c0 * g.down - g.low_c;
  const int R = g.R, S = g.S, D = g.down;

  float acc[kGU];
#pragma unroll
  for (int u = 0; u < kGU; ++u) acc[u] = 0.0f;

  for (int t = 0; t < g.terms; ++t) {
    int ip, fp;
    plane_pair(g, o, t, &ip, &fp);
    const float *xs = x + (size_t)ip * g.H * g.W;
    const float *fs = f + (size_t)fp * g.fr * g.fs;
    if (t > 0) __syncthreads();
    // Tap (r, s) of the R x S filter as applied: flipped for convolution, and
    // for an upsampled FilterAdjoint gradient the zero-inserted lattice
    // (stored taps at multiples of fup).
    for (int i = threadIdx.x; i < R * S; i += blockDim.x) {
      const int r = i / S, s = i - r * S;
      const int er = g.orient == CCT_CONVOLUTION ? R - 1 - r : r;
      const int es = g.orient == CCT_CONVOLUTION ? S - 1 - s : s;
      float v = 0.0f;
      if (er % g.fup == 0 && es % g.fup == 0) v = __ldg(fs + (er / g.fup) * g.fs + es / g.fup);
      wf[i] = v;
    }
    load_tile(tile, pitch, in_rows, in_cols, xs, g, org_r, org_c);
    __syncthreads();

    float rs[kGU];
#pragma unroll
    for (int u = 0; u < kGU; ++u) rs[u] = 0.0f;
    const float *base = tile + (ty * D) * pitch + tx * kGU * D;
    for (int r = 0; r < R; ++r) {
      const float *row = base + r * pitch;
      const float *wr = wf + r * S;
      float cs[kGU];
#pragma unroll
      for (int u = 0; u < kGU; ++u) cs[u] = 0.0f;
      for (int s = 0; s < S; ++s) {
        const float w = wr[s];
#pragma unroll
        for (int u = 0; u < kGU; ++u) cs[u] = __fmaf_rn(row[u * D + s], w, cs[u]);
      }
#pragma unroll
      for (int u = 0; u < kGU; ++u) rs[u] = __fadd_rn(rs[u], cs[u]);
    }
#pragma unroll
    for (int u = 0; u < kGU; ++u) acc[u] = (t == 0) ? rs[u] : __fadd_rn(acc[u], rs[u]);
  }

  const int row = out_r0 + ty;
  if (row < g.OH) {
    float *ys = y + (size_t)o * g.OH * g.OW + (size_t)row * g.OW;
    const bool relu = (g.flags & CCT_FLAG_RELU) != 0;
#pragma unroll
    for (int u = 0; u < kGU; ++u) {
      const int col = out_c0 + tx * kGU + u;
      if (col < g.OW) ys[col] = relu ? fmaxf(acc[u], 0.0f) : acc[u];
    }
  }
}

// Grid of one CTA per (tile, output plane).
int tile_grid(const ConvGeom &g, int h, int w, int th, int tw, int *tiles_x, int *tiles_y, long long *blocks) {
  *tiles_x = (w + tw - 1) / tw;
  *tiles_y = (h + th - 1) / th;
  *blocks = (long long)*tiles_x * *tiles_y * g.pout;
  if (*blocks > 0x7fffffffLL) return set_error(CCT_ENOTSUP, "direct convolution grid too large");
  return CCT_OK;
}

// Tall tiles once their grid gives each of 148 SMs a CTA; shorter ones spread
// a small field over more SMs.
constexpr long long kTallTiles = 148;

template <int R, int DOWN, int V, bool VEC>
int launch_small_v(const ConvGeom &g, const float *x, const float *f, float *y, cudaStream_t st, long long min_blocks) {
  int tx, ty;
  long long blocks;
  int rc = tile_grid(g, g.OH, g.OW, kSmTY * V, kSmTW, &tx, &ty, &blocks);
  if (rc) return rc;
  if (blocks < min_blocks) return 1;  // a shorter tile is wanted
  rc = launch_pdl(direct_small_kernel<R, R, DOWN, V, VEC>, dim3((unsigned)blocks), dim3(kSmThreads), 0, st,
                  "direct_small_kernel launch", g, x, f, y, tx, ty);
  if (!rc) count_launches(1);
  return rc;
}

template <int R, int DOWN>
int launch_small(const ConvGeom &g, const float *x, const float *f, float *y, cudaStream_t st, bool vec) {
  constexpr int V = DOWN == 1 ? 8 : 4;
  // 16-byte staging: aligned rows and a centred filter (Zero, Clamp, Cyclic)
  if (vec) {
    const int rc = launch_small_v<R, DOWN, V, true>(g, x, f, y, st, kTallTiles);
    return rc == 1 ? launch_small_v<R, DOWN, 2, true>(g, x, f, y, st, 0) : rc;
  }
  const int rc = launch_small_v<R, DOWN, V, false>(g, x, f, y, st, kTallTiles);
  return rc == 1 ? launch_small_v<R, DOWN, 2, false>(g, x, f, y, st, 0) : rc;
}

template <int S, int V>
int launch_wide_v(const ConvGeom &g, const float *x, const float *f, float *y, cudaStream_t st, long long min_blocks) {
  int tx, ty;
  long long blocks;
  int rc = tile_grid(g, g.OH, g.OW, kWdTY * V, kWdTW, &tx, &ty, &blocks);
  if (rc) return rc;
  if (blocks < min_blocks) return 1;  // a shorter tile is wanted
  const size_t smem = wide_smem(g.R, S, V);
  rc = raise_smem_limit(direct_wide_kernel<S, V>, smem, "cudaFuncSetAttribute(direct_wide)");
  if (rc) return rc;
  rc = launch_pdl(direct_wide_kernel<S, V>, dim3((unsigned)blocks), dim3(kWdThreads), smem, st,
                  "direct_wide_kernel launch", g, x, f, y, tx, ty);
  if (!rc) count_launches(1);
  return rc;
}

template <int S>
int launch_wide(const ConvGeom &g, const float *x, const float *f, float *y, cudaStream_t st) {
  // 3 rows per thread once that gives two CTAs per SM (480x640 by 11x11, us for
  // V = 3 / 1: one plane 6.3 / 5.2, two 8.7 / 7.3, four 10.7 / 11.7, sixteen
  // 32.4 / 36.0); from 25 columns on the input rows' halo outweighs it (31x31,
  // four planes: 59.7 / 53.6).
  if constexpr (S < 25) {
    const int rc = launch_wide_v<S, 3>(g, x, f, y, st, 2 * 148);
    if (rc != 1) return rc;
  }
  return launch_wide_v<S, 1>(g, x, f, y, st, 0);
}

template <int R, int UP, int V>
int launch_up_v(const ConvGeom &g, const float *x, const float *f, float *y, cudaStream_t st, long long min_blocks) {
  int tx, ty;
  long long blocks;
  int rc = tile_grid(g, g.H, g.W, kSmTY * V, kSmTW, &tx, &ty, &blocks);
  if (rc) return rc;
  if (blocks < min_blocks) return 1;
  rc = launch_pdl(direct_up_kernel<R, UP, V>, dim3((unsigned)blocks), dim3(kSmThreads), 0, st,
                  "direct_up_kernel launch", g, x, f, y, tx, ty);
  if (!rc) count_launches(1);
  return rc;
}

template <int R, int UP>
int launch_up(const ConvGeom &g, const float *x, const float *f, float *y, cudaStream_t st) {
  if constexpr (UP == 2 && R < 9) {
    const int rc = launch_up_v<R, UP, 2>(g, x, f, y, st, kTallTiles);
    if (rc != 1) return rc;
  }
  return launch_up_v<R, UP, 1>(g, x, f, y, st, 0);
}

template <int R>
int launch_square(const ConvGeom &g, const float *x, const float *f, float *y, cudaStream_t st) {
  int tx, ty;
  long long blocks;
  int rc = tile_grid(g, g.OH, g.OW, kTY * 4, kTX * 4, &tx, &ty, &blocks);
  if (rc) return rc;
  // Small grids are better off in the general kernel's quarter tiles, longer the
  // smaller the filter (up-sampled by 4, us here / there: 1x1 at 400 tiles 13.2 / 12.0,
  // 800 22.9 / 20.8, 1000 24.3 / 25.1; 3x3 at 296 17.6 / 16.0, 400 18.9 / 19.4; 5x5 at 180
  // 18.4 / 16.1, 296 18.7 / 23.5; 7x7 at 80 17.9 / 17.1, 120 18.1 / 20.6).
  // So are grids that waste the lower part of their squares, where quarters do not (1x1
  // up 3, fields of 6x56, 64 rows against 32: 917 / 561 us; 3x3 up 2 BorderFull, 8x9, the
  // same 44 / 35; but 111x11, 256 against 224: 140 / 185, and 7x7 up 3 BorderFull, 5x91, 64
  // against 32: 529 / 771).
  const int tall = (g.OH + 63) / 64 * 64, flat = (g.OH + 15) / 16 * 16;
  if (tall * 10LL > flat * (R == 1 ? 15LL : R == 3 ? 16 : R == 5 ? 19 : 22)) return 1;
  if (blocks < (R == 1 ? 900 : R == 3 ? 360 : R == 5 ? 220 : 88)) return 1;
  rc = launch_pdl(direct_square_kernel<R>, dim3((unsigned)blocks), dim3(kThreads), 0, st,
                  "direct_square_kernel launch", g, x, f, y, tx, ty);
  if (!rc) count_launches(1);
  return rc;
}

int launch_generic(const ConvGeom &g, const float *x, const float *f, float *y,
                   cudaStream_t st) {
  const int tiles_x = (g.OW + kGTW - 1) / kGTW, tiles_y = (g.OH + kGTH - 1) / kGTH;
  const int in_rows = (kGTH - 1) * g.down + g.R;
  const int in_cols = (kGTW - 1) * g.down + g.S;
  const int pitch = (in_cols + 3) & ~3;
  const size_t smem = sizeof(float) * ((size_t)in_rows * pitch + (size_t)g.R * g.S);
  int dev = 0, max_smem = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (smem > (size_t)max_smem)
    return set_error(CCT_ENOTSUP, "filter %dx%d with step %d needs %zu bytes of shared memory (max %d)",
                     g.R, g.S, g.down, smem, max_smem);
  int rc = raise_smem_limit(direct_generic_kernel, smem, "cudaFuncSetAttribute(direct_generic)");
  if (rc) return rc;
  const long long blocks = (long long)tiles_x * tiles_y * g.pout;
  if (blocks > 0x7fffffffLL) return set_error(CCT_ENOTSUP, "direct convolution grid too large");
  rc = launch_pdl(direct_generic_kernel, dim3((unsigned)blocks), dim3(kThreads), smem, st,
                            "direct_generic_kernel launch", g, x, f, y, tiles_x, tiles_y, in_rows, in_cols, pitch);
  if (!rc) count_launches(1);
  return rc;
}

}  // namespace

int launch_direct(const ConvGeom &g, const float *x, const float *f, float *y,
                  cudaStream_t st) {
  if (g.fup != 1) return launch_generic(g, x, f, y, st);
  // Odd widths without sampling: weights in shared memory, unless an aligned
  // field of a small filter can stage 16 bytes at a time (5x5 clamp, 256 planes
  // of 256x256: 44 us there, 48 here; 64 planes of 301x403, which cannot: 31 /
  // 28, 7x7: 44 / 35).  R <= 64 keeps tile and weights under 70 KB.
  const bool vec = (g.W & 3) == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0 &&
                   g.border != CCT_BORDER_VALID && g.border != CCT_BORDER_FULL;
  if (g.up == 1 && g.down == 1 && g.terms == 1 && g.R <= 64 && !(vec && g.R == g.S && g.R <= 5)) {
#define CCT_WIDE_CASE(SS) case SS: return launch_wide<SS>(g, x, f, y, st);
    switch (g.S) {
      CCT_WIDE_CASE(3) CCT_WIDE_CASE(5) CCT_WIDE_CASE(7) CCT_WIDE_CASE(9) CCT_WIDE_CASE(11) CCT_WIDE_CASE(13)
      CCT_WIDE_CASE(15) CCT_WIDE_CASE(17) CCT_WIDE_CASE(19) CCT_WIDE_CASE(21) CCT_WIDE_CASE(23) CCT_WIDE_CASE(25)
      CCT_WIDE_CASE(27) CCT_WIDE_CASE(29) CCT_WIDE_CASE(31) CCT_WIDE_CASE(33) CCT_WIDE_CASE(35) CCT_WIDE_CASE(37)
      CCT_WIDE_CASE(39) CCT_WIDE_CASE(41) CCT_WIDE_CASE(43) CCT_WIDE_CASE(45) CCT_WIDE_CASE(47) CCT_WIDE_CASE(49)
      CCT_WIDE_CASE(51) CCT_WIDE_CASE(53) CCT_WIDE_CASE(55) CCT_WIDE_CASE(57) CCT_WIDE_CASE(59) CCT_WIDE_CASE(61)
      CCT_WIDE_CASE(63)
      default: break;
    }
#undef CCT_WIDE_CASE
  }
  if (g.up == 1 && g.R == g.S && (g.down == 1 || g.down == 2)) {
#define CCT_SMALL_CASE(RR) \
  case RR: return g.down == 1 ? launch_small<RR, 1>(g, x, f, y, st, vec) : launch_small<RR, 2>(g, x, f, y, st, vec);
    switch (g.R) {
      CCT_SMALL_CASE(1) CCT_SMALL_CASE(3) CCT_SMALL_CASE(5) CCT_SMALL_CASE(7)
      default: break;
    }
#undef CCT_SMALL_CASE
  }
  // centred filters (BorderZero, BorderCyclic; BorderClamp does not up-sample)
  if ((g.up == 2 || g.up == 3) && g.down == 1 && g.R == g.S &&
      (g.border == CCT_BORDER_ZERO || g.border == CCT_BORDER_CYCLIC)) {
#define CCT_UP_CASE(RR) \
  case RR: return g.up == 2 ? launch_up<RR, 2>(g, x, f, y, st) : launch_up<RR, 3>(g, x, f, y, st);
    switch (g.R) {
      CCT_UP_CASE(3) CCT_UP_CASE(5) CCT_UP_CASE(7)
      case 9:
        if (g.up == 2) return launch_up<9, 2>(g, x, f, y, st);
        break;
      default: break;
    }
#undef CCT_UP_CASE
  }
  if (g.up != 1 && g.down == 1 && g.R == g.S) {
    int rc = 1;
#define CCT_SQUARE_CASE(RR) case RR: rc = launch_square<RR>(g, x, f, y, st); break;
    switch (g.R) {
      CCT_SQUARE_CASE(1) CCT_SQUARE_CASE(3) CCT_SQUARE_CASE(5) CCT_SQUARE_CASE(7)
      default: break;
    }
    if (rc != 1) return rc;
#undef CCT_SQUARE_CASE
  }
  return launch_generic(g, x, f, y, st);
}

}  // namespace cct
