// Device pieces of the register-window stencils: border-mapped tile staging
// with 4-byte cp.async, and the output store through shared memory.
#pragma once

#include "cct_internal.h"
#include "tile_common.cuh"

namespace cct {

// border_index with the division of the cyclic border only outside the field.
__device__ __forceinline__ int stencil_index(int border, int v, int n) {
  if (v >= 0 && v < n) return v;
  return border_index(border, v, n);
}

// Copies rows x COLS border-mapped values whose corner is (org_r, org_c) into
// tile[row * PITCH + col]; of a row, only the first `need` columns are read from the
// field (102 x 8 outputs of a clamped 3x3 DownsampleOutput(2), 361 planes: 44 us
// reading whole rows, 13 so).  A thread owns fixed columns of every row it copies,
// so a column is mapped by the border once per tile and an element costs an
// add and a copy.  (Mapping every element, the way load_tile does, took most
// of the ~195 instructions per output of a 7x7 clamped stencil.)
//
// VEC = false: any width; a warp per row, lanes along it, 4-byte copies.
// VEC = true: rows of a 16-byte aligned field whose width is a multiple of 4,
// org_c a multiple of 4 and COLS too: 16-byte copies of 4-column chunks, which
// lie inside the field or outside it as a whole (a cyclic chunk wraps whole; a
// clamped one repeats one value).
template <int COLS, int PITCH, int THREADS, bool VEC>
struct TileStage;

template <int COLS, int PITCH, int THREADS>
struct TileStage<COLS, PITCH, THREADS, false> {
  static constexpr int KC = (COLS + 31) / 32, STEP = THREADS / 32;
  int sc[KC];    // source column of this lane's k-th column (0 where it reads zero)
  bool in[KC];   // the column is needed, and not outside a border that reads zero

  __device__ __forceinline__ TileStage(const ConvGeom &g, int org_c, int need) {
#pragma unroll
    for (int k = 0; k < KC; ++k) {
      const int col = (int)(threadIdx.x & 31) + 32 * k, c = stencil_index(g.border, org_c + col, g.W);
      in[k] = c >= 0 && col < need;
      sc[k] = c < 0 ? 0 : c;
    }
  }
  __device__ __forceinline__ void row(float *d, const float *s, bool ok) const {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int k = 0; k < KC; ++k)
      if (32 * (k + 1) <= COLS || lane + 32 * k < COLS) cp_async_f32(d + 32 * k, s + sc[k], ok && in[k]);
  }
  __device__ __forceinline__ void copy(float *tile, const float *__restrict__ src, const ConvGeom &g, int org_r,
                                       int rows) const {
    int tr = threadIdx.x >> 5;
    float *d = tile + tr * PITCH + (threadIdx.x & 31);
    if (org_r >= 0 && org_r + rows <= g.H) {
      const float *s = src + (size_t)(org_r + tr) * g.W;
      const size_t step = (size_t)STEP * g.W;
#pragma unroll 2
      for (; tr < rows; tr += STEP, d += STEP * PITCH, s += step) row(d, s, true);
    } else {
      for (; tr < rows; tr += STEP, d += STEP * PITCH) {
        const int sr = stencil_index(g.border, org_r + tr, g.H);
        row(d, src + (size_t)(sr < 0 ? 0 : sr) * g.W, sr >= 0);
      }
    }
  }
};

template <int COLS, int PITCH, int THREADS>
struct TileStage<COLS, PITCH, THREADS, true> {
  static_assert(COLS % 4 == 0 && PITCH % 4 == 0, "whole 16-byte chunks");
  static constexpr int CH = COLS / 4, STEP = THREADS / CH;  // chunks per row, rows per round
  static_assert(STEP >= 1, "a round covers a row");
  int sc, r0, c0;
  bool in, splat;

  __device__ __forceinline__ TileStage(const ConvGeom &g, int org_c, int need) {
    r0 = threadIdx.x / CH;
    c0 = 4 * (threadIdx.x - r0 * CH);
    const int c = org_c + c0, m = stencil_index(g.border, c, g.W);
    // a chunk past the right edge clamps to the last column, past the left
    // edge to the first: its four values are that one
    splat = g.border == CCT_BORDER_CLAMP && m != c;
    in = m >= 0;
    sc = m < 0 ? 0 : m;
    if (r0 >= STEP || c0 >= need) r0 = 1 << 30;  // idle
  }
  __device__ __forceinline__ void chunk(float *d, const float *s, bool ok) const {
    if (splat) {
#pragma unroll
      for (int k = 0; k < 4; ++k) cp_async_f32(d + k, s, ok);
    } else {
      cp_async_16(d, s, ok && in);
    }
  }
  __device__ __forceinline__ void copy(float *tile, const float *__restrict__ src, const ConvGeom &g, int org_r,
                                       int rows) const {
    int tr = r0;
    if (tr >= rows) return;
    float *d = tile + tr * PITCH + c0;
    if (org_r >= 0 && org_r + rows <= g.H) {
      const float *s = src + (size_t)(org_r + tr) * g.W + sc;
      const size_t step = (size_t)STEP * g.W;
#pragma unroll 2
      for (; tr < rows; tr += STEP, d += STEP * PITCH, s += step) chunk(d, s, true);
    } else {
      for (; tr < rows; tr += STEP, d += STEP * PITCH) {
        const int sr = stencil_index(g.border, org_r + tr, g.H);
        chunk(d, src + (size_t)(sr < 0 ? 0 : sr) * g.W + sc, sr >= 0);
      }
    }
  }
};

// Stores `rows` rows of `cols` <= 64 finished values (shared memory, row pitch
// `pitch` floats) to dst rows of stride `stride`, one warp, lanes along a row:
// coalesced whatever the field's width or alignment.
__device__ __forceinline__ void store_rows64(float *dst, size_t stride, const float *src, int pitch, int rows, int cols,
                                             int lane) {
  const bool a = lane < cols, b = lane + 32 < cols;
  dst += lane;
  src += lane;
#pragma unroll 4
  for (int r = 0; r < rows; ++r, dst += stride, src += pitch) {
    if (a) dst[0] = src[0];
    if (b) dst[32] = src[32];
  }
}

}  // namespace cct
