// Separable convolution: a rows pass then a columns pass
// (ConvolveRows2DHyperKernel.scala:66-160, ConvolveColumns2DHyperKernel.scala).
// Each output is a fused multiply-add chain from 0 over the 1-D filter taps,
// the order of the reference's `sum += localImage[..] * filter` loop.
// Short filters run both passes fused per output tile: under BorderZero on
// large fields whose width is a multiple of 4 floats the halo tiles arrive by
// TMA (separable_tma, up to 9 taps), otherwise threads stage them
// (separable_tile, up to 15 + 31 taps; separable_fused, up to about 33); long
// filters run one thread per output per pass, through a scratch field.
#include <algorithm>
#include <atomic>

#include "cct_internal.h"
#include "sm100_util.cuh"
#include "stencil.cuh"
#include "tile_common.cuh"
#include "tile_ring.cuh"

namespace cct {
namespace {

constexpr int kThreads = 256;

// dir 0: along columns of a row (rows pass); dir 1: along rows (columns pass).
template <int DIR>
__global__ void __launch_bounds__(kThreads)
    separable_pass(int rows, int cols, int planes, const float *__restrict__ x,
                   const float *__restrict__ filt, int len, int border, int orient,
                   float *__restrict__ y) {
  __shared__ float wf[1024];
  for (int i = threadIdx.x; i < len; i += blockDim.x)
    wf[i] = filt[orient == CCT_CONVOLUTION ? len - 1 - i : i];
  __syncthreads();
  const long long total = (long long)rows * cols * planes;
  const int halo = (len - 1) / 2;
  for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    const int c = (int)(idx % cols);
    const long long rp = idx / cols;
    const int r = (int)(rp % rows);
    const float *xp = x + (rp / rows) * (long long)rows * cols;
    float sum = 0.0f;
    if (DIR == 0) {
      const float *line = xp + (size_t)r * cols;
      for (int k = 0; k < len; ++k) {
        const int j = border_index(border, c - halo + k, cols);
        sum = __fmaf_rn(j < 0 ? 0.0f : __ldg(line + j), wf[k], sum);
      }
    } else {
      for (int k = 0; k < len; ++k) {
        const int i = border_index(border, r - halo + k, rows);
        sum = __fmaf_rn(i < 0 ? 0.0f : __ldg(xp + (size_t)i * cols + c), wf[k], sum);
      }
    }
    y[idx] = sum;
  }
}

// Both passes fused per 32 x 64 output tile: the image rows the columns
// pass needs (border-mapped) are staged in shared memory with their
// border-mapped column halo, the rows pass fills an intermediate tile of
// those rows, and the columns pass reads it.  Each intermediate value is the
// same fma chain as in the two-pass form, so the result is bit-identical to
// it while the image is read and the result written once.
constexpr int kSTH = 32, kSTW = 64;

__global__ void __launch_bounds__(kThreads)
    separable_fused(int rows, int cols, int planes, const float *__restrict__ x,
                    const float *__restrict__ rf, int rlen, const float *__restrict__ cf, int clen,
                    int border, int orient, float *__restrict__ y, int tiles_x, int tiles_y) {
  extern __shared__ __align__(16) float sm[];
  const int hr = (rlen - 1) / 2, hc = (clen - 1) / 2;
  const int IR = kSTH + clen - 1, IC = kSTW + rlen - 1;  // staged image rows x columns
  float *wr = sm, *wc = sm + rlen;
  float *img = wc + clen;                // IR x IC
  float *mid = img + (size_t)IR * IC;    // IR x kSTW (rows pass)
  const bool conv = orient == CCT_CONVOLUTION;
  for (int i = threadIdx.x; i < rlen; i += blockDim.x) wr[i] = rf[conv ? rlen - 1 - i : i];
  for (int i = threadIdx.x; i < clen; i += blockDim.x) wc[i] = cf[conv ? clen - 1 - i : i];
  int bid = blockIdx.x;
  const int tx = bid % tiles_x;
  bid /= tiles_x;
  const int ty = bid % tiles_y, pl = bid / tiles_y;
  const int r0 = ty * kSTH, c0 = tx * kSTW;
  const float *xp = x + (size_t)pl * rows * cols;
  // image rows r0-hc .. r0+kSTH+hc-1, mapped by the border (the intermediate
  // field's border), columns c0-hr .. c0+kSTW+hr-1 mapped likewise; one warp
  // per staged row, lanes along it
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
  const bool inside_c = c0 - hr >= 0 && c0 - hr + IC <= cols;
  for (int ir = warp; ir < IR; ir += nwarps) {
    const int sr = border_index(border, r0 - hc + ir, rows);
    float *dst = img + (size_t)ir * IC;
    if (sr < 0) {
      for (int ic = lane; ic < IC; ic += 32) dst[ic] = 0.0f;
    } else if (inside_c) {
      const float *src = xp + (size_t)sr * cols + (c0 - hr);
      for (int ic = lane; ic < IC; ic += 32) dst[ic] = __ldg(src + ic);
    } else {
      const float *src = xp + (size_t)sr * cols;
      for (int ic = lane; ic < IC; ic += 32) {
        const int sc = border_index(border, c0 - hr + ic, cols);
        dst[ic] = sc >= 0 ? __ldg(src + sc) : 0.0f;
      }
    }
  }
  __syncthreads();
  // rows pass: intermediate of every staged row (zero rows stay zero: the
  // intermediate field is zero outside under BorderZero)
  for (int e = threadIdx.x; e < IR * kSTW; e += blockDim.x) {
    const int ir = e / kSTW, j = e - ir * kSTW;
    const float *line = img + (size_t)ir * IC + j;
    float sum = 0.0f;
#pragma unroll 4
    for (int k = 0; k < rlen; ++k) sum = __fmaf_rn(line[k], wr[k], sum);
    mid[e] = sum;
  }
  __syncthreads();
  // columns pass
  float *yp = y + (size_t)pl * rows * cols;
  for (int e = threadIdx.x; e < kSTH * kSTW; e += blockDim.x) {
    const int i = e / kSTW, j = e - i * kSTW;
    const int r = r0 + i, c = c0 + j;
    if (r >= rows || c >= cols) continue;
    const float *col = mid + (size_t)i * kSTW + j;
    float sum = 0.0f;
#pragma unroll 4
    for (int k = 0; k < clen; ++k) sum = __fmaf_rn(col[(size_t)k * kSTW], wc[k], sum);
    yp[(size_t)r * cols + c] = sum;
  }
}

// Row filters of up to 15 taps (compiled), column filters of up to 31, every
// border and width.  A CTA of 128 threads computes 64 columns x 8 V rows: the
// halo is staged with the columns mapped once per tile (TileStage), the rows
// pass slides a register window along 8 columns of a staged row, and the columns
// pass keeps 4 columns x V rows per thread, so a row-filtered value is read once
// per V outputs.  Each value is the same fma chain as in the two-pass form.
// Bound: FP32 issue and staging latency.  The forms it replaces mapped every
// staged element by the border, and past 9 taps read shared memory per tap:
// 1080x1920 x3, 7 + 7 clamp 31 us, 720x1280 x3, 15 + 15 35 us; 21.4 and 14.0 here.
constexpr int kTlThreads = 128, kTlW = 64, kTlMid = kTlW + 4, kTlMaxR = 15, kTlMaxC = 31;
__host__ __device__ constexpr int tile_pitch(int RL) {
  const int c = (kTlW + RL - 1 + 3) & ~3;
  return (c & 7) == 4 ? c : c + 4;  // 4 (mod 8): two rows of a float4 phase on different banks
}
inline size_t tile_smem(int RL, int clen, int V) {
  return sizeof(float) * ((size_t)(8 * V + clen - 1) * (tile_pitch(RL) + kTlMid) + kTlMaxC + 1);
}

template <int RL, int V>
__global__ void __launch_bounds__(kTlThreads, V == 8 ? 5 : 8)
    separable_tile(int rows, int cols, const float *__restrict__ x, const float *__restrict__ rf,
                   const float *__restrict__ cf, int clen, int border, int orient, float *__restrict__ y, int tiles_x,
                   int tiles_y) {
  constexpr int TH = 8 * V, PITCH = tile_pitch(RL), U = 8, E4 = (U + RL - 1 + 3) / 4;
  static_assert(4 * E4 + kTlW - U <= PITCH, "a thread's loads stay inside its row");
  extern __shared__ __align__(16) float sm[];
  const int IR = TH + clen - 1;
  float *img = sm, *mid = sm + IR * PITCH, *wc = mid + IR * kTlMid;
  grid_dependency_wait();  // launched with programmatic serialisation: nothing global before this
  const bool conv = orient == CCT_CONVOLUTION;
  int bid = blockIdx.x;
  const int tx_i = bid % tiles_x;
  bid /= tiles_x;
  const int ty_i = bid % tiles_y, pl = bid / tiles_y;
  const int r0 = ty_i * TH, c0 = tx_i * kTlW, out_rows = min(TH, rows - r0), need = out_rows + clen - 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  ConvGeom g;  // what the staging reads
  g.H = rows;
  g.W = cols;
  g.border = border;
  {
    const TileStage<kTlW + RL - 1, PITCH, kTlThreads, false> stage(g, c0 - (RL - 1) / 2,
                                                                       min(kTlW, cols - c0) + RL - 1);
    stage.copy(img, x + (size_t)pl * rows * cols, g, r0 - (clen - 1) / 2, need);
    cp_async_commit();
  }
  float wr[RL];
#pragma unroll
  for (int k = 0; k < RL; ++k) wr[k] = __ldg(rf + (conv ? RL - 1 - k : k));
  if (threadIdx.x < clen) wc[threadIdx.x] = __ldg(cf + (conv ? clen - 1 - (int)threadIdx.x : (int)threadIdx.x));
  cp_async_wait<0>();
  __syncthreads();
  {
    // a float4 phase of 8 lanes covers 4 column blocks x 2 rows
    const int cb = (lane & 3) | ((lane >> 1) & 4), rsub = ((lane >> 2) & 1) | ((lane >> 3) & 2);
    for (int r = warp * 4 + rsub; r < need; r += 16) {
      const float *line = img + r * PITCH + cb * U;
      float win[4 * E4];
#pragma unroll
      for (int e = 0; e < E4; ++e) {
        const float4 q = *reinterpret_cast<const float4 *>(line + 4 * e);
        win[4 * e + 0] = q.x;
        win[4 * e + 1] = q.y;
        win[4 * e + 2] = q.z;
        win[4 * e + 3] = q.w;
      }
      float h[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        float sum = 0.0f;
#pragma unroll
        for (int k = 0; k < RL; ++k) sum = __fmaf_rn(win[u + k], wr[k], sum);
        h[u] = sum;
      }
      float4 *dst = reinterpret_cast<float4 *>(mid + r * kTlMid + cb * U);
      dst[0] = make_float4(h[0], h[1], h[2], h[3]);
      dst[1] = make_float4(h[4], h[5], h[6], h[7]);
    }
  }
  __syncthreads();
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  float acc[V][4];
#pragma unroll
  for (int v = 0; v < V; ++v)
#pragma unroll
    for (int u = 0; u < 4; ++u) acc[v][u] = 0.0f;
  if (ty * V < out_rows) {
    const float *base = mid + ty * V * kTlMid + tx * 4;
    for (int tr = 0; tr < V - 1 + clen; ++tr) {
      const float4 q = *reinterpret_cast<const float4 *>(base + tr * kTlMid);
#pragma unroll
      for (int v = 0; v < V; ++v) {
        const int k = tr - v;
        if (k >= 0 && k < clen) {  // the same for every thread
          const float w = wc[k];
          acc[v][0] = __fmaf_rn(q.x, w, acc[v][0]);
          acc[v][1] = __fmaf_rn(q.y, w, acc[v][1]);
          acc[v][2] = __fmaf_rn(q.z, w, acc[v][2]);
          acc[v][3] = __fmaf_rn(q.w, w, acc[v][3]);
        }
      }
    }
  }
  allow_dependent_launch();
  float *yp = y + (size_t)pl * rows * cols + (size_t)r0 * cols + c0;
  if ((cols & 3) == 0 && (reinterpret_cast<uintptr_t>(y) & 15) == 0) {
    if (c0 + tx * 4 >= cols) return;
#pragma unroll
    for (int v = 0; v < V; ++v)
      if (ty * V + v < out_rows)
        *reinterpret_cast<float4 *>(yp + (size_t)(ty * V + v) * cols + tx * 4) =
            make_float4(acc[v][0], acc[v][1], acc[v][2], acc[v][3]);
    return;
  }
  // rows that are not 16-byte aligned leave through the image's tile, which the
  // rows pass has read: a warp stores 32 adjacent values at a time
#pragma unroll
  for (int v = 0; v < V; ++v)
    *reinterpret_cast<float4 *>(img + (ty * V + v) * kTlW + tx * 4) =
        make_float4(acc[v][0], acc[v][1], acc[v][2], acc[v][3]);
  __syncwarp();
  const int w0 = warp * 2 * V;
  if (w0 < out_rows)
    store_rows64(yp + (size_t)w0 * cols, cols, img + w0 * kTlW, kTlW, min(2 * V, out_rows - w0), min(kTlW, cols - c0),
                 lane);
}

template <int RL, int V>
int launch_tile_v(int rows, int cols, int planes, const float *x, const float *rf, const float *cf, int clen,
                  int border, int orient, float *y, cudaStream_t st, long long min_blocks) {
  const int tx = (cols + kTlW - 1) / kTlW, ty = (rows + 8 * V - 1) / (8 * V);
  const long long blocks = (long long)tx * ty * planes;
  if (blocks < min_blocks) return 1;  // a shorter tile is wanted
  if (blocks > 0x7fffffffLL) return set_error(CCT_ENOTSUP, "separable: grid too large");
  const size_t smem = tile_smem(RL, clen, V);
  int rc = raise_smem_limit(separable_tile<RL, V>, smem, "cudaFuncSetAttribute(separable_tile)");
  if (rc) return rc;
  rc = launch_pdl(separable_tile<RL, V>, dim3((unsigned)blocks), dim3(kTlThreads), smem, st,
                            "separable launch", rows, cols, x, rf, cf, clen, border, orient, y, tx, ty);
  if (!rc) count_launches(1);
  return rc;
}

// The tile form for a row filter of 1, 3, .. 15 taps; tall tiles once they give
// each of 148 SMs two CTAs.
int launch_tile(int rows, int cols, int planes, const float *x, const float *rf, int rlen, const float *cf, int clen,
                int border, int orient, float *y, cudaStream_t st) {
#define CCT_TILE_CASE(RL)                                                                                          \
  case RL: {                                                                                                       \
    const int rc = launch_tile_v<RL, 8>(rows, cols, planes, x, rf, cf, clen, border, orient, y, st, 2 * 148);      \
    return rc == 1 ? launch_tile_v<RL, 2>(rows, cols, planes, x, rf, cf, clen, border, orient, y, st, 0) : rc;     \
  }
  switch (rlen) {
    CCT_TILE_CASE(1) CCT_TILE_CASE(3) CCT_TILE_CASE(5) CCT_TILE_CASE(7)
    CCT_TILE_CASE(9) CCT_TILE_CASE(11) CCT_TILE_CASE(13) CCT_TILE_CASE(15)
    default: return set_error(CCT_ENOTSUP, "separable: row filter of %d taps", rlen);
  }
#undef CCT_TILE_CASE
}

// BorderZero with TMA staging: persistent CTAs walk their output tiles and a
// loading warp keeps kSepStages halo tiles in flight (3-D TMA loads
// completing on mbarriers; TMA's out-of-bounds zero fill is BorderZero, for
// the image and for the intermediate field alike).  The box's x origin is
// rounded down to a multiple of 4 floats and the kernel indexes from the
// remainder OFF.  A thread owns 4 columns x 8 rows of output: for each staged
// row it forms the 4 row-filtered values (an fma chain from 0 over the row
// taps) and feeds each to the column chains of the outputs that use that
// row, in tap order, so every output is the same fma chain of the same
// values as in the two-pass form.
// Tiles of 128 x 64 or 64 x 128 (columns x rows), whichever covers the field with
// less padding, the wide ones on a tie (eight planes of 1080x1920, 9 + 9 taps:
// 28.4 us against 31.0).
constexpr int kSepU = 4, kSepV = 8, kSepStages = 2;
template <bool WIDE>
struct SepShape {
  static constexpr int TW = WIDE ? 128 : 64, TH = WIDE ? 64 : 128, TX = TW / kSepU;
  static long long padded(int rows, int cols) {
    return (long long)((cols + TW - 1) / TW) * TW * ((rows + TH - 1) / TH) * TH;
  }
};

template <int RL, int CL, int OFF, bool WIDE>
struct SepTma {
  static constexpr int kSepTW = SepShape<WIDE>::TW, kSepTH = SepShape<WIDE>::TH;
  static constexpr int hr = (RL - 1) / 2, hc = (CL - 1) / 2;
  static constexpr int IN_ROWS = kSepTH + CL - 1;
  static constexpr int BOX_C = (kSepTW + RL - 1 + OFF + 3) & ~3;
  static constexpr int STAGE = ((IN_ROWS * BOX_C) + 31) & ~31;  // floats, 128-byte multiple
  static constexpr uint32_t BYTES = IN_ROWS * BOX_C * 4;
  static constexpr size_t SMEM = (size_t)kSepStages * STAGE * 4;
};

template <int RL, int CL, int OFF, bool WIDE>
__global__ void __launch_bounds__(kThreads + 32)
    separable_tma(const __grid_constant__ CUtensorMap xmap, int rows, int cols, const float *__restrict__ rf,
                  const float *__restrict__ cf, int orient, float *__restrict__ y, int tiles_x, int tiles_y,
                  int total, unsigned *err) {
  using T = SepTma<RL, CL, OFF, WIDE>;
  constexpr int kSepTW = T::kSepTW, kSepTH = T::kSepTH, kSepTX = SepShape<WIDE>::TX;
  constexpr int E = kSepU - 1 + RL;  // staged values a thread reads per row, from OFF
  constexpr int E4 = (OFF + E + 3) / 4;
  extern __shared__ __align__(128) float smem[];
  __shared__ TileRing<kSepStages, kThreads / 32> ring;
  const int tid = threadIdx.x;
  ring.init();
  __syncthreads();
  grid_dependency_wait();  // launched with programmatic serialisation: global memory only after this
  allow_dependent_launch();  // persistent: every CTA is resident already
  auto decode = [&](int i, int &pl, int &tyi, int &txi) {
    txi = i % tiles_x;
    const int q = i / tiles_x;
    tyi = q % tiles_y;
    pl = q / tiles_y;
  };
  if (tid >= kThreads) {  // the loading warp (one lane)
    if (tid == kThreads)
      ring.produce(total, err, [&](int i, int s, uint64_t *full) {
        int pl, tyi, txi;
        decode(i, pl, tyi, txi);
        mbar_arrive_expect_tx(full, T::BYTES);
        tma_load_3d(smem + s * T::STAGE, &xmap, full, txi * kSepTW - T::hr - OFF, tyi * kSepTH - T::hc, pl);
      });
    return;
  }
  const int tx = tid % kSepTX, ty = tid / kSepTX;
  float wr[RL], wc[CL];
  const bool conv = orient == CCT_CONVOLUTION;
#pragma unroll
  for (int k = 0; k < RL; ++k) wr[k] = __ldg(rf + (conv ? RL - 1 - k : k));
#pragma unroll
  for (int k = 0; k < CL; ++k) wc[k] = __ldg(cf + (conv ? CL - 1 - k : k));
  const size_t page = (size_t)rows * cols;

  int j = 0;
  for (int i = blockIdx.x; i < total; i += gridDim.x, ++j) {
    const int s = j % kSepStages;
    int pl, tyi, txi;
    decode(i, pl, tyi, txi);
    if (!ring.wait_full(j, err)) return;
    const float *base = smem + s * T::STAGE + (ty * kSepV) * T::BOX_C + tx * kSepU;
    float acc[kSepV][kSepU];
#pragma unroll
    for (int v = 0; v < kSepV; ++v)
#pragma unroll
      for (int u = 0; u < kSepU; ++u) acc[v][u] = 0.0f;
#pragma unroll
    for (int tr = 0; tr < kSepV + CL - 1; ++tr) {
      float vals[E4 * 4];
#pragma unroll
      for (int e = 0; e < E4; ++e) {
        const float4 q = *reinterpret_cast<const float4 *>(base + tr * T::BOX_C + 4 * e);
        vals[4 * e + 0] = q.x;
        vals[4 * e + 1] = q.y;
        vals[4 * e + 2] = q.z;
        vals[4 * e + 3] = q.w;
      }
      float h[kSepU];
#pragma unroll
      for (int u = 0; u < kSepU; ++u) {
        float sum = 0.0f;
#pragma unroll
        for (int k = 0; k < RL; ++k) sum = __fmaf_rn(vals[OFF + u + k], wr[k], sum);
        h[u] = sum;
      }
#pragma unroll
      for (int v = 0; v < kSepV; ++v) {
        const int k = tr - v;
        if (k >= 0 && k < CL) {
#pragma unroll
          for (int u = 0; u < kSepU; ++u) acc[v][u] = __fmaf_rn(h[u], wc[k], acc[v][u]);
        }
      }
    }
    ring.release(s);  // this warp is done with the stage
    // the field width is a multiple of 4, so a thread's 4 columns are all in
    // or all out
    const int col0 = txi * kSepTW + tx * kSepU;
    if (col0 < cols) {
      float *yp = y + (size_t)pl * page + col0;
#pragma unroll
      for (int v = 0; v < kSepV; ++v) {
        const int row = tyi * kSepTH + ty * kSepV + v;
        if (row < rows)
          *reinterpret_cast<float4 *>(yp + (size_t)row * cols) = make_float4(acc[v][0], acc[v][1], acc[v][2],
                                                                             acc[v][3]);
      }
    }
  }
}

template <int RL, int CL, int OFF, bool WIDE>
int launch_tma_t(int rows, int cols, int planes, const float *x, const float *rf, const float *cf, int orient,
                 float *y, cudaStream_t st) {
  using T = SepTma<RL, CL, OFF, WIDE>;
  const int tiles_x = (cols + T::kSepTW - 1) / T::kSepTW, tiles_y = (rows + T::kSepTH - 1) / T::kSepTH;
  const long long total = (long long)tiles_x * tiles_y * planes;
  if (total > 0x7fffffffLL) return set_error(CCT_ENOTSUP, "separable: grid too large");
  CUtensorMap map;
  int rc = encode_tensor_map_3d(&map, x, cols, rows, planes, T::BOX_C, T::IN_ROWS);
  if (rc) return rc;
  auto kern = separable_tma<RL, CL, OFF, WIDE>;
  int dev = 0;
  rc = check_cuda(cudaGetDevice(&dev), "cudaGetDevice");
  if (rc) return rc;
  // per instance: devices whose function attributes and grid size are set
  static std::atomic<unsigned long long> ready{0};
  static int grid_cap[64];
  if (dev >= 64) return set_error(CCT_ENOTSUP, "separable: device ordinal %d", dev);
  if (!(ready.load() >> dev & 1ull)) {
    rc = check_cuda(cudaFuncSetAttribute((const void *)kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)T::SMEM),
                    "cudaFuncSetAttribute(separable_tma)");
    int sms = 0, per_sm = 0;
    if (!rc) rc = check_cuda(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev), "SM count");
    if (!rc)
      rc = check_cuda(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kThreads + 32, T::SMEM),
                      "separable occupancy");
    if (rc) return rc;
    grid_cap[dev] = sms * (per_sm > 0 ? per_sm : 1);
    ready.fetch_or(1ull << dev);
  }
  const int grid = (int)(total < grid_cap[dev] ? total : grid_cap[dev]);
  const int rc2 = launch_pdl(kern, dim3(grid), dim3(kThreads + 32), T::SMEM, st, "separable_tma launch", map, rows, cols,
                             rf, cf, orient, y, tiles_x, tiles_y, (int)total, device_error_word());
  if (!rc2) count_launches(1);
  return rc2;
}

// Row lengths 1..9 (odd) with their x-offset remainder, column lengths 1..9
// (odd); -1 if not covered, else the launch status.
int launch_tma_small(int rows, int cols, int planes, const float *x, const float *rf, int rlen, const float *cf,
                     int clen, int orient, float *y, cudaStream_t st) {
  const bool wide = SepShape<true>::padded(rows, cols) <= SepShape<false>::padded(rows, cols);
#define CCT_SEPT_C(RL, CL, OFF) \
  if (rlen == RL && clen == CL)                                                                      \
    return wide ? launch_tma_t<RL, CL, OFF, true>(rows, cols, planes, x, rf, cf, orient, y, st)       \
                : launch_tma_t<RL, CL, OFF, false>(rows, cols, planes, x, rf, cf, orient, y, st);
#define CCT_SEPT_R(RL, OFF) \
  CCT_SEPT_C(RL, 1, OFF) CCT_SEPT_C(RL, 3, OFF) CCT_SEPT_C(RL, 5, OFF) CCT_SEPT_C(RL, 7, OFF) CCT_SEPT_C(RL, 9, OFF)
  // OFF = (-(RL - 1) / 2) mod 4
  CCT_SEPT_R(1, 0) CCT_SEPT_R(3, 3) CCT_SEPT_R(5, 2) CCT_SEPT_R(7, 1) CCT_SEPT_R(9, 0)
#undef CCT_SEPT_R
#undef CCT_SEPT_C
  return -1;
}

size_t separable_fused_smem(int rlen, int clen) {
  const size_t IR = kSTH + clen - 1, IC = kSTW + rlen - 1;
  return sizeof(float) * (rlen + clen + IR * IC + IR * kSTW);
}

}  // namespace

int launch_separable(int rows, int cols, int planes, const float *x, const float *rf,
                     int rlen, const float *cf, int clen, int border, int orient,
                     float *tmp, float *y, cudaStream_t st) {
  if (rows < 1 || cols < 1 || planes < 1)
    return set_error(CCT_EINVAL, "separable: field sizes must be positive");
  if (border != CCT_BORDER_ZERO && border != CCT_BORDER_CLAMP && border != CCT_BORDER_CYCLIC)
    return set_error(CCT_EINVAL, "separable: unsupported border policy %d", border);
  if (rlen < 1 || clen < 1 || rlen % 2 == 0 || clen % 2 == 0)
    return set_error(CCT_EINVAL, "separable: row and column filters must be of odd size");
  if (rlen > 1024 || clen > 1024)
    return set_error(CCT_ENOTSUP, "separable: filters longer than 1024 taps");
  if (orient != CCT_CONVOLUTION && orient != CCT_CROSS_CORRELATION)
    return set_error(CCT_EINVAL, "separable: bad orientation");
  const size_t fsmem = separable_fused_smem(rlen, clen);
  if (fsmem <= 96 * 1024) {
    const int tiles_x = (cols + kSTW - 1) / kSTW, tiles_y = (rows + kSTH - 1) / kSTH;
    const long long blocks = (long long)tiles_x * tiles_y * planes;
    // Fewer than 96 TMA tiles leave most SMs idle; the smaller tiles below do not
    // (us: one plane of 512x512, 5 + 5, 32 tiles 3.4 / 2.7; 768x768, 72 tiles 3.5 /
    // 3.3; 1024x1024, 128 tiles 3.7 / 4.4).
    // Fields that fill less than half of a TMA tile but fit one 64 x 64 tile's columns
    // and rows are staged as far as they reach there, which pays for flat ones and
    // for the most taps (us, TMA / small: 3000 of 8x20, 3 + 3 17.3 / 11.8; 1000 of 32x32, 3 +
    // 3 8.8 / 8.7, 9 + 9 15.6 / 10.9; 1024 of 60x64, 9 + 9 16.3 / 14.3, but 3 + 3 9.6 / 12.3, 5 + 5
    // 11.0 / 12.4).
    const long long pad = std::min(SepShape<true>::padded(rows, cols), SepShape<false>::padded(rows, cols));
    const long long small = (long long)((rows + 63) / 64 * 64) * ((cols + 63) / 64 * 64);
    const bool wasted = 2 * small <= pad && (rows <= 32 || rlen + clen >= 18);
    if (border == CCT_BORDER_ZERO && !wasted && (cols & 3) == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0 &&
        (reinterpret_cast<uintptr_t>(y) & 15) == 0 && pad / (64 * 128) * planes >= 96) {
      const int rc = launch_tma_small(rows, cols, planes, x, rf, rlen, cf, clen, orient, y, st);
      if (rc >= 0) return rc;
    }
    if (rlen <= kTlMaxR && clen <= kTlMaxC)
      return launch_tile(rows, cols, planes, x, rf, rlen, cf, clen, border, orient, y, st);
    if (blocks <= 0x7fffffffLL) {
      int rc = raise_smem_limit(separable_fused, fsmem, "cudaFuncSetAttribute(separable)");
      if (rc) return rc;
      separable_fused<<<(unsigned)blocks, kThreads, fsmem, st>>>(rows, cols, planes, x, rf, rlen, cf, clen,
                                                                 border, orient, y, tiles_x, tiles_y);
      count_launches(1);
      return check_cuda(cudaGetLastError(), "separable launch");
    }
  }
  // long filters: the two passes through the caller's scratch field
  const long long total = (long long)rows * cols * planes;
  const long long want = (total + kThreads - 1) / kThreads;
  const int blocks = (int)(want < 148LL * 64 ? want : 148LL * 64);
  separable_pass<0><<<blocks, kThreads, 0, st>>>(rows, cols, planes, x, rf, rlen, border, orient, tmp);
  separable_pass<1><<<blocks, kThreads, 0, st>>>(rows, cols, planes, tmp, cf, clen, border, orient, y);
  count_launches(2);
  return check_cuda(cudaGetLastError(), "separable launch");
}

}  // namespace cct
