// Fused filter-bank convolution on the tcgen05 tensor cores, split BF16:
// ProjectFrameBlockReduceSum / BackProjectFrameBlockReduceSum
// (ConvolveHyperKernel.scala:153-199, 319-340, 574-645), every border policy
// (:235-317), DownsampleOutput(1, 2) (:205-223), UpsampleInput(2-4)
// (:206-212, 405-459, as one sub-filter per output phase), any field width.
// A block of filters fills the MMAs in one of four forms (bank_tc.h).  The plain one
// takes 64 filters, with the layout and the zero rows described here.  Banks of at
// most 32 filters put two taps of a filter row into each MMA (paired taps: tap b's
// sums are read one grid position to the right).  The wide forms, 128 filters or 64
// filters x two taps, keep big and small sums in separate accumulator columns and have
// no zero rows (below block_term).
//
// GEMM view, per image b and block of filters:
//   D[filter k][position p] = sum over (plane c, tap t) F[k][c, t] * X[c][p + off(t)]
// M = the filter block, N = a tile of output positions, reduction = planes x
// taps.  Positions live on a padded output grid of pitch P = BW + (S-1)/step
// columns (a band of BW output columns plus the tap reach): the input value a
// position reads at tap t then sits at a fixed offset off(t) from the
// position on the same grid, so the B operand of tap t is a contiguous run of
// the halo in shared memory and the tensor core reads it through a shifted
// descriptor -- no per-tap copies.  Grid columns past the band's outputs are
// computed and discarded ((S-1)/P of the work).  DownsampleOutput(2) holds
// the input as its four polyphase components, each a stride-1 grid.
//
// Split precision.  x = xh + xl (+ xm) and f likewise, each term bf16.  In the plain
// form the filter operand of one MMA is 128 rows: rows 0-63 ("big") multiply into the
// hi*hi sum only, rows 64-127 ("small") into the correction products:
//   2 terms (BF16X3): [Fh; Fl] x Xh  and  [0; Fh] x Xl
//                     -> big hh, small lh + hl
//   3 terms (BF16X6): [Fh; Fm] x Xh, [0; Fh] x Xm, [0; Fh] x Xl, [0; Fl] x Xh,
//                     [0; Fm] x Xm
//                     -> big hh, small mh + hm + hl + lh + mm
// The big rows never receive a small addend: the tensor core's FP32
// accumulation drops the bits of an addend below the accumulator's last
// place, and measured that way its error grows with the number of MMAs
// accumulated, so only hh goes into the big sum and zero rows (which add
// exactly 0) fill the big half of the other MMAs.  For long reductions the
// accumulator is also promoted: every seg_stages stages the epilogue adds it
// into an FP32 running sum (RN, CUDA cores) and the next MMA starts it
// afresh, which bounds the accumulation error by the segment length; the
// wide forms' small sums every few segments.  The epilogue adds each filter's big and
// small sums.
//
// Warp roles (one persistent CTA per SM, 640 threads):
//   warps 0-9   converters: for each (tile, plane block) fill a halo buffer:
//               plain loads of the input with the border policy applied
//               (zero, clamp, cyclic), split into bf16 terms, stored in the
//               K-major core-matrix layout [plane group][position][8 planes];
//               two buffers, so the next block is converted while the
//               current one is multiplied.  Then warps 0-7 store half of
//               the CTA's last tile with the epilogue warps.
//   warp 10     MMA issuer (one elected lane): per (tile, plane block, tap):
//               KS k-steps x nmma MMAs, A = filter chunk stage, B = halo.
//   warp 11     loader (one lane): bulk copies of the pre-packed filter
//               chunks (nb, plane block, tap) into a ring of stages, one copy
//               per stage of several taps.
//   warps 12-19 epilogue, two per tensor-memory lane quarter (alternate
//               column halves): promotion adds, then per 16-column chunk the
//               warps holding one filter block's parts write them to shared
//               memory, and each adds the parts of a share of the filters,
//               applies ReLU and stores.
// Every wait is bounded: on a timeout the CTA records it in the device error
// word, lets its copies and MMAs land, frees tensor memory and exits.
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>

#include "bank_tc.h"
#include "sm100_util.cuh"

namespace cct {
namespace {

constexpr int kConvWarps = 10;  // ten: a 536-position halo takes two rounds of loads, not three
constexpr int kConvThreads = 32 * kConvWarps;
constexpr int kMmaWarp = kConvWarps;
constexpr int kLoadWarp = kConvWarps + 1;
constexpr int kEpiWarp0 = kConvWarps + 2;
constexpr int kEpiWarps = 8;
constexpr int kThreads = 32 * (kEpiWarp0 + kEpiWarps);
constexpr int kMaxStages = 8;
constexpr int kPackThreads = 128;
constexpr uint32_t kAccCols = 256;  // one accumulator (N <= 256 fp32 columns)
// Epilogue exchange: eight part tiles of 32 filters x 16 positions, a filter's
// four float4s permuted by its number (xch_quad) so that eight filters' float4s
// of one position, and two filters' rows, cover all banks.
constexpr int kXchPitch = 16;
__device__ __forceinline__ int xch_quad(int filter, int quad) { return quad ^ ((filter >> 1) & 3); }
constexpr int kXchFloats = 32 * kXchPitch;
constexpr size_t kXchBytes = 8 * kXchFloats * sizeof(float);

// Filter chunk row blocks (64 rows each) and the MMAs over them.
// Block contents: -1 zero, else the split term (0 hi, 1 mid / lo for 2 terms, 2 lo).
__host__ __device__ constexpr int block_term(int terms, int blk) {
  return terms == 2 ? (blk == 0 ? -1 : blk - 1)                          // Z Fh Fl
                    : (blk == 0 || blk == 3 || blk == 5 ? -1             // Z Fh Fm Z Fl Z Fm
                                                        : (blk == 1 ? 0 : blk == 2 ? 1 : blk == 4 ? 2 : 1));
}
// Paired taps (banks of at most 32 filters): a chunk of 32-row blocks
// [0 0 Fh_a Fh_b Fl_a Fl_b] for taps a and b = a + 1 of one filter row, the
// same 192 rows and MMAs as an unpaired two-term chunk: [Fh_a; Fh_b; Fl_a;
// Fl_b] x Xh and [0; 0; Fh_a; Fh_b] x Xl.
// The wide forms (bank_tc.h) need no zero rows: a chunk is each split term's 128 rows, an
// accumulator is 128 columns of big sums and 128 of small ones (N <= 128), and
// every MMA's rows are all live: 6 MMAs of N = 128 do 128 x 128 outputs where the
// plain form's 5 of N = 256 do 64 x 256 (three terms; 3 against 2 for two).
__host__ __device__ constexpr bool pairs_taps(int form) { return form == kPair || form == kWidePair; }
__host__ __device__ constexpr bool wide_form(int form) { return form >= kWide; }
// Parts of a filter's sum in different rows (warps): big and small, tap a and tap b.
__host__ __device__ constexpr int form_parts(int form) { return form == kPair ? 4 : form == kWide ? 1 : 2; }

template <int TERMS, bool WIDE>
struct MmaList;
template <>
struct MmaList<2, false> {
  static constexpr int n = 2;
  __device__ static int arow(int m) { return m == 0 ? 64 : 0; }  // [Fh; Fl], [0; Fh] (paired: at tap a's offset)
  __device__ static int bterm(int m) { return m; }               // Xh, Xl
};
template <>
struct MmaList<3, false> {
  static constexpr int n = 5;
  // [Fh; Fm] x Xh, [0; Fh] x Xm, [0; Fh] x Xl, [0; Fl] x Xh, [0; Fm] x Xm
  __device__ static int arow(int m) { return m == 0 ? 64 : m == 3 ? 192 : m == 4 ? 320 : 0; }
  __device__ static int bterm(int m) { return m == 0 || m == 3 ? 0 : m == 2 ? 2 : 1; }
};
// Wide: MMA 0 into the big columns, the others into the small ones.
template <>
struct MmaList<2, true> {
  static constexpr int n = 3;
  // Fh x Xh; Fl x Xh, Fh x Xl
  __device__ static int arow(int m) { return m == 1 ? 128 : 0; }
  __device__ static int bterm(int m) { return m == 2 ? 1 : 0; }
};
template <>
struct MmaList<3, true> {
  static constexpr int n = 6;
  // Fh x Xh; Fm x Xh, Fl x Xh, Fh x Xm, Fm x Xm, Fh x Xl
  __device__ static int arow(int m) { return m == 1 || m == 4 ? 128 : m == 2 ? 256 : 0; }
  __device__ static int bterm(int m) { return m < 3 ? 0 : m < 5 ? 1 : 2; }
};

struct Bars {
  uint64_t full[kMaxStages], empty[kMaxStages];  // filter chunk stages
  uint64_t hfull[2], hempty[2];                  // halo buffers
  uint64_t dfull[2], dempty[2];                  // accumulators (one per segment in flight)
  uint64_t drain;                                // MMA warp: every MMA retired
  uint32_t tmem_slot;
  int abort_flag;
};

// Border policy of the input (ConvolveHyperKernel.scala:235-317): maps
// (iy, ix) into the field, or returns false for a zero.
__device__ __forceinline__ bool border_map(const ConvGeom &g, int iy, int ix, int &ry, int &rx) {
  if (g.border == CCT_BORDER_CLAMP) {
    ry = min(max(iy, 0), g.H - 1);
    rx = min(max(ix, 0), g.W - 1);
    return true;
  }
  if (g.border == CCT_BORDER_CYCLIC) {
    ry = ((iy % g.H) + g.H) % g.H;
    rx = ((ix % g.W) + g.W) % g.W;
    return true;
  }
  ry = iy;
  rx = ix;
  return iy >= 0 && iy < g.H && ix >= 0 && ix < g.W;
}

struct Item {
  int b, ph, band, tile, nb;
};
__device__ __forceinline__ Item decode(const BankParams &p, int i) {
  Item it;
  it.nb = i % p.nblocks;
  int rest = i / p.nblocks;
  it.tile = rest % p.tiles_band;
  rest /= p.tiles_band;
  it.band = rest % p.nbands;
  rest /= p.nbands;
  it.ph = rest % p.nph_out;
  it.b = rest / p.nph_out;
  return it;
}

// Reduction units of a work item: ts taps per filter row of its (sub-)filter,
// nu units, nst stages per plane block, and the first packed chunk of its
// filter block.  Every role derives its loop bounds from here.
struct ItemUnits {
  int ts, nu, nst;
  size_t chunk0;
};
template <int FORM>
__device__ __forceinline__ ItemUnits item_units(const BankParams &p, const Item &it) {
  ItemUnits r;
  int rows;
  if (p.up > 1) {
    const int rho = it.ph / p.up;
    rows = p.up_rq[rho];
    r.ts = p.up_sq[it.ph - rho * p.up];
  } else {
    rows = p.g.R;
    r.ts = p.g.S;
  }
  r.nu = rows * (pairs_taps(FORM) ? (r.ts + 1) / 2 : r.ts);
  r.nst = p.hblocks > 1 ? p.nst : (r.nu + p.T - 1) / p.T;
  r.chunk0 = (size_t)p.up_choff[it.ph] + (size_t)it.nb * p.NCB * r.nu;
  return r;
}

// One halo block: a plane block of every input phase with every unit, or
// (hblocks > 1, DownsampleOutput(2)) of one phase with the units that read it.
struct Block {
  int cb, u0, u1;
};
__device__ __forceinline__ Block block_of(const BankParams &p, const ItemUnits &iu, int blk) {
  Block r;
  r.cb = blk / p.hblocks;
  r.u0 = 0;
  r.u1 = iu.nu;
  if (p.hblocks > 1) {
    const int ph = blk - r.cb * p.hblocks;
    r.u0 = p.ph_u0[ph];
    r.u1 = p.ph_u0[ph + 1];
  }
  return r;
}

// Split 8*KG planes of one halo position into bf16 terms and store them as
// KG core-matrix rows (16 bytes per term).  src points at the position in
// the first plane; `cvalid` planes exist (the rest are zero).  All 8*KG loads
// are issued before the first store, so a converter thread keeps that many
// reads in flight.
template <int KG>
__device__ __forceinline__ void load_kgroups(const float *src, size_t plane, bool in, int cvalid, float (&v)[8 * KG]) {
#pragma unroll
  for (int j = 0; j < 8 * KG; ++j) v[j] = (in && j < cvalid) ? __ldg(src + j * plane) : 0.0f;
}

template <int TERMS, int KG>
__device__ __forceinline__ void store_kgroups(const float (&v)[8 * KG], uint8_t *dst, uint32_t kg_stride,
                                              uint32_t part_bytes) {
#pragma unroll
  for (int k = 0; k < KG; ++k) {
    uint8_t *d = dst + k * kg_stride;
    const float *w = v + 8 * k;
    if (TERMS == 2) {
      uint32_t hi[4], lo[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) split_bf16x2(w[2 * j], w[2 * j + 1], hi[j], lo[j]);
      *reinterpret_cast<uint4 *>(d) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
      *reinterpret_cast<uint4 *>(d + part_bytes) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
    } else {
      uint32_t hi[4], mi[4], lo[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) split3_bf16x2(w[2 * j], w[2 * j + 1], hi[j], mi[j], lo[j]);
      *reinterpret_cast<uint4 *>(d) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
      *reinterpret_cast<uint4 *>(d + part_bytes) = make_uint4(mi[0], mi[1], mi[2], mi[3]);
      *reinterpret_cast<uint4 *>(d + 2 * (size_t)part_bytes) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
    }
  }
}

template <int TERMS, int KG>
__device__ __forceinline__ void convert_kgroups(const float *src, size_t plane, bool in, int cvalid,
                                                uint8_t *dst, uint32_t kg_stride, uint32_t part_bytes) {
  float v[8 * KG];
  load_kgroups<KG>(src, plane, in, cvalid, v);
  store_kgroups<TERMS, KG>(v, dst, kg_stride, part_bytes);
}

// A barrier over the G warps of a group (one warp: none but itself).
template <int G>
__device__ __forceinline__ void group_sync(int bar_id) {
  if (G == 1)
    __syncwarp();
  else
    named_sync(bar_id, 32 * G);
}
template <int G>
__device__ __forceinline__ bool group_sync_or(int bar_id, bool pred) {
  return G == 1 ? __any_sync(0xffffffffu, pred) != 0 : named_sync_or(bar_id, 32 * G, pred);
}
// Where a warp's lane quarter stands: its group, and its part in it.
template <int FORM>
__device__ __forceinline__ void group_of(int quarter, int half, int &grp, int &part) {
  grp = FORM == kPair ? half : FORM == kWide ? quarter * 2 + half : (quarter & 1) * 2 + half;
  part = FORM == kPair ? quarter : FORM == kWide ? 0 : (quarter < 2 ? 0 : 1);
}

// Final accumulator of work item `it` (S in tensor-memory columns at `sc`,
// plus the running sum at `rc` unless `first`), columns [cbeg, cbeg + ncol):
// the group of G warps holding one block of 32 filters' parts (this warp's
// lane quarter `quarter`, part `part`) writes each 16-column chunk into its
// own [filter][position] tile, and after a barrier each adds the parts of its
// share of the filters (a half, or a quarter) and stores them, so no warp
// waits on another's stores.  `release` (or null): arrived on once this
// warp's last accumulator load is done.
template <int TERMS, int FORM>
__device__ __forceinline__ void store_tile_columns(const BankParams &p, const Item &it, uint32_t sc, uint32_t rc,
                                                   bool first, int cbeg, int ncol, float *tiles, int bar_id,
                                                   int quarter, int part, int lane, uint64_t *release) {
  const ConvGeom &g = p.g;
  constexpr int G = form_parts(FORM);  // parts (warps) per group
  // tap b's rows: their sums sit one position to the right
  const bool shifted = FORM == kPair ? (quarter & 1) != 0 : FORM == kWidePair ? quarter >= 2 : false;
  const bool relu = (g.flags & CCT_FLAG_RELU) != 0;
  const size_t opl = (size_t)g.OH * g.OW;
  const int limit = pairs_taps(FORM) ? p.tile_adv : p.N;  // columns of the tile with complete sums
  const int p0 = it.tile * p.tile_adv;
  // grid position (Y, X) of band `band` -> output (up*Y + rho, up*(band*BW + X) + kap)
  const int rho = it.ph / p.up, kap = it.ph - rho * p.up;
  const int ohv = (g.OH - rho + p.up - 1) / p.up;                                 // valid grid rows
  const int bw = min(p.BW, (g.OW - kap + p.up - 1) / p.up - it.band * p.BW);     // valid columns of the band
  const size_t ors = (size_t)p.up * g.OW;                                          // output row stride of a grid row
  // the group's 32 filters
  const int fb = it.nb * p.fblock + (FORM == kPair ? 0 : FORM == kWide ? quarter * 32 : (quarter & 1) * 32);
  float *ybase0 = p.y + (size_t)it.b * g.groups * opl + (size_t)rho * g.OW + (size_t)it.band * p.BW * p.up + kap +
                  (size_t)fb * opl;
  // The next chunk's accumulator load is in flight while a chunk is combined
  // and stored (18 warps: 96 registers a thread at most; three-term and
  // paired kernels have none to spare and load each chunk when they reach it).
  uint32_t n16[16], ne = 0;
  auto issue = [&](int c) {
    tmem_ld16(sc + c, n16);
    // paired taps: tap b's rows also need column c + 16
    if (shifted && c + 16 < p.N) tmem_ld1(sc + c + 16, ne);
  };
  constexpr bool kAhead = TERMS == 2 && FORM == kPlain;
  if (kAhead) issue(cbeg);
  for (int c = cbeg; c < cbeg + ncol; c += 16) {
    if (!kAhead) issue(c);
    tc_wait_ld();
    const bool ext = shifted && c + 16 < p.N;
    uint32_t s16[16], r16[16], e1 = ne, e2 = 0;
#pragma unroll
    for (int t = 0; t < 16; ++t) s16[t] = n16[t];
    if (!first) {
      tmem_ld16(rc + c, r16);
      if (ext) tmem_ld1(rc + c + 16, e2);
      tc_wait_ld();
    }
    float v[17];
#pragma unroll
    for (int t = 0; t < 16; ++t) v[t] = __uint_as_float(s16[t]) + (first ? 0.0f : __uint_as_float(r16[t]));
    v[16] = ext ? __uint_as_float(e1) + (first ? 0.0f : __uint_as_float(e2)) : 0.0f;
    if (wide_form(FORM)) {  // the small sums, in columns of their own
      tmem_ld16(sc + kAccCols / 2 + c, s16);
      if (ext) tmem_ld1(sc + kAccCols / 2 + c + 16, e1);
      tc_wait_ld();
#pragma unroll
      for (int t = 0; t < 16; ++t) v[t] += __uint_as_float(s16[t]);
      if (ext) v[16] += __uint_as_float(e1);
    }
    if (release && c + 16 >= cbeg + ncol) {  // the accumulator is read: release it
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(release);
    }
    {
      float4 *mine = reinterpret_cast<float4 *>(tiles + part * kXchFloats + lane * kXchPitch);
#pragma unroll
      for (int k = 0; k < 4; ++k)
        mine[xch_quad(lane, k)] = shifted ? make_float4(v[4 * k + 1], v[4 * k + 2], v[4 * k + 3], v[4 * k + 4])
                                          : make_float4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
    }
    if (kAhead && c + 16 < cbeg + ncol) issue(c + 16);
    group_sync<G>(bar_id);  // every part of the chunk is in place
    // this warp's share: the parts of its filters, all loaded before the
    // barrier that lets the group overwrite the tiles
    float w[16];
    int t0, fl;
    if (p.vec4) {
      // lane -> (filter 8*i + lane/4, positions 4*(lane%4) .. +3), i in the share
      t0 = 4 * (lane & 3);
      fl = lane >> 2;
#pragma unroll
      for (int k = 0; k < 4 / G; ++k)
#pragma unroll
        for (int q = 0; q < G; ++q) {
          const int f = 8 * (part * (4 / G) + k) + fl;
          const float4 r = reinterpret_cast<const float4 *>(tiles + q * kXchFloats + f * kXchPitch)[xch_quad(f, lane & 3)];
          w[(k * G + q) * 4 + 0] = r.x;
          w[(k * G + q) * 4 + 1] = r.y;
          w[(k * G + q) * 4 + 2] = r.z;
          w[(k * G + q) * 4 + 3] = r.w;
        }
    } else {
      // lane -> (filter 2*i + lane/16, position lane%16), i in the share
      t0 = lane & 15;
      fl = lane >> 4;
#pragma unroll
      for (int k = 0; k < 16 / G; ++k)
#pragma unroll
        for (int q = 0; q < G; ++q) {
          const int f = 2 * (part * (16 / G) + k) + fl;
          w[k * G + q] = tiles[q * kXchFloats + f * kXchPitch + 4 * xch_quad(f, t0 >> 2) + (t0 & 3)];
        }
    }
    group_sync<G>(bar_id);  // the tiles may be rewritten
    const int Gp = p0 + c + t0;
    const int Y = Gp / p.P, X = Gp - Y * p.P;
    const bool ok = Y < ohv && X < bw && c + t0 < limit;
    if (p.vec4) {
      float *yo = ybase0 + (size_t)Y * ors + X;  // up == 1 here
#pragma unroll
      for (int k = 0; k < 4 / G; ++k) {
        const int f = 8 * (part * (4 / G) + k) + fl;
        float o[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          float acc = w[(k * G) * 4 + e];
#pragma unroll
          for (int q = 1; q < G; ++q) acc = acc + w[(k * G + q) * 4 + e];  // parts in order
          o[e] = relu ? fmaxf(acc, 0.0f) : acc;
        }
        if (ok && fb + f < g.groups)
          *reinterpret_cast<float4 *>(yo + (size_t)f * opl) = make_float4(o[0], o[1], o[2], o[3]);
      }
    } else {
      float *yo = ybase0 + (size_t)Y * ors + (size_t)X * p.up;
#pragma unroll
      for (int k = 0; k < 16 / G; ++k) {
        const int f = 2 * (part * (16 / G) + k) + fl;
        float acc = w[k * G];
#pragma unroll
        for (int q = 1; q < G; ++q) acc = acc + w[k * G + q];  // parts in order
        if (relu) acc = fmaxf(acc, 0.0f);
        if (ok && fb + f < g.groups) yo[(size_t)f * opl] = acc;
      }
    }
  }
}

// The last tile of a CTA is stored by the converter warps as well as the
// epilogue warps (each taking a quarter of the columns): by then the
// converters have nothing left to fill.  Only when every item is one
// accumulation segment (the converters then wait on the last item's
// accumulator phase in order) and a quarter of a tile is whole chunks.
__device__ __forceinline__ bool helpers_store_last(const BankParams &p) { return !p.promote && p.N % 64 == 0; }

// CB16: 16-plane blocks (the converters pair their (phase, position) items);
// a separate instance, so the other plane blocks' code is unchanged.
template <int TERMS, int FORM, bool CB16>
__global__ void __launch_bounds__(kThreads, 1) bank_tc_kernel(const __grid_constant__ BankParams p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ Bars bars;
  // epilogue exchange: 4 groups of 2 part tiles, (paired taps) 2 groups of 4, or (128
  // filters) 8 groups of 1
  __shared__ __align__(16) float xch[8 * kXchFloats];
  __shared__ uint32_t unit_boff[kBankMaxTaps];  // MMA warp: B operand offset of each unit
  const ConvGeom &g = p.g;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint8_t *halo = smem;                                 // 2 x halo_bytes
  uint8_t *stage = smem + 2 * (size_t)p.halo_bytes;     // stages x stage_bytes

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(&bars.full[s], 1);   // loader expect_tx
      mbar_init(&bars.empty[s], 1);  // MMA commit
    }
    for (int h = 0; h < 2; ++h) {
      mbar_init(&bars.hfull[h], kConvWarps);  // one arrival per converter warp
      mbar_init(&bars.hempty[h], 1);          // MMA commit
      mbar_init(&bars.dfull[h], 1);           // MMA commit
      mbar_init(&bars.dempty[h], kEpiWarps);  // one arrival per epilogue warp
    }
    mbar_init(&bars.drain, 1);
    bars.abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == kMmaWarp) tmem_alloc(&bars.tmem_slot, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = bars.tmem_slot;
  // Nothing above touches global memory, so it may overlap the previous
  // kernel in the stream (programmatic serialisation).  When that kernel is
  // this launch's own filter pack, only the packed operand is still being
  // written: the pack waited for every earlier grid before it let this one
  // start, so the input is complete and the output no longer read, and only
  // the loader (which reads the packed operand) waits here.
  if (!p.after_pack) grid_dependency_wait();
  allow_dependent_launch();

  volatile int *abort_flag = &bars.abort_flag;

  if (warp < kConvWarps) {
    // ------------------------------------------------------------ converters
    const int nkg = p.CB / 8;                   // 2, 4 or 8 core-matrix columns
    const uint32_t kgs = (uint32_t)p.L * 16;     // bytes between them
    const size_t plane = (size_t)g.H * g.W;
    uint32_t hb = 0;
    bool failed = false;
    for (int i = blockIdx.x; i < p.total && !failed; i += gridDim.x) {
      const Item it = decode(p, i);
      const int p0 = it.tile * p.tile_adv;
      // strided input row / column of halo position 0
      const int rho = it.ph / p.up, kap = it.ph - rho * p.up;
      const int row0 = p.up > 1 ? p.up_sr[rho] : p.sr_min;
      const int col0 = it.band * p.BW + (p.up > 1 ? p.up_sc[kap] : p.sc_min);
      const float *xb = p.x + (size_t)it.b * g.n * plane;
      for (int blk = 0; blk < p.NCB * p.hblocks; ++blk, ++hb) {
        const int cb = blk / p.hblocks;
        const int ph0 = p.hblocks > 1 ? blk - cb * p.hblocks : 0, nph = p.hblocks > 1 ? 1 : p.nphase;  // its phases
        const int buf = hb & 1;
        if (*abort_flag || !mbar_wait(&bars.hempty[buf], ((hb >> 1) & 1) ^ 1, p.err)) {
          failed = true;
          break;
        }
        uint8_t *hbase = halo + (size_t)buf * p.halo_bytes;
        const int cv = g.n - cb * p.CB;  // planes of this block that exist
        const float *xc = xb + (size_t)cb * p.CB * plane;
        if constexpr (CB16) {
          // 16-plane blocks: the (phase, position) items two at a time, both
          // items' loads issued before either is converted, so a thread has
          // as many loads in flight as with a 32-plane position
          const int total = nph * p.L;
          for (int it = threadIdx.x; it < total; it += 2 * kConvThreads) {
            const float *src[2];
            bool in[2];
            uint8_t *dst[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const int item = min(it + e * kConvThreads, total - 1);
              const int ph = item / p.L, q = item - ph * p.L;
              const int G = p0 + q;
              const int Y = G / p.P, X = G - Y * p.P;
              const int iy = g.down * (Y + row0) + p.phase_r[ph0 + ph];
              const int ix = g.down * (col0 + X) + p.phase_c[ph0 + ph];
              int ry, rx;
              in[e] = border_map(g, iy, ix, ry, rx);
              src[e] = in[e] ? xc + (size_t)ry * g.W + rx : xc;
              dst[e] = hbase + (size_t)ph * TERMS * p.part_bytes + (size_t)q * 16;
            }
            float va[16], vb[16];
            load_kgroups<2>(src[0], plane, in[0], cv, va);
            load_kgroups<2>(src[1], plane, in[1], cv, vb);
            store_kgroups<TERMS, 2>(va, dst[0], kgs, p.part_bytes);
            if (it + kConvThreads < total) store_kgroups<TERMS, 2>(vb, dst[1], kgs, p.part_bytes);
          }
        } else {
          for (int ph = 0; ph < nph; ++ph) {
            uint8_t *hph = hbase + (size_t)ph * TERMS * p.part_bytes;
            for (int q = threadIdx.x; q < p.L; q += kConvThreads) {
              const int G = p0 + q;
              const int Y = G / p.P, X = G - Y * p.P;
              const int iy = g.down * (Y + row0) + p.phase_r[ph0 + ph];
              const int ix = g.down * (col0 + X) + p.phase_c[ph0 + ph];
              int ry, rx;
              const bool in = border_map(g, iy, ix, ry, rx);
              const float *src = in ? xc + (size_t)ry * g.W + rx : xc;
              uint8_t *dst = hph + (size_t)q * 16;
              int kg = 0;
              for (; kg + 4 <= nkg; kg += 4)
                convert_kgroups<TERMS, 4>(src + (size_t)kg * 8 * plane, plane, in, cv - kg * 8, dst + (size_t)kg * kgs,
                                          kgs, p.part_bytes);
              for (; kg < nkg; kg += 2)
                convert_kgroups<TERMS, 2>(src + (size_t)kg * 8 * plane, plane, in, cv - kg * 8, dst + (size_t)kg * kgs,
                                          kgs, p.part_bytes);
            }
          }
        }
        // the tensor core reads the halo through the async proxy
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars.hfull[buf]);
      }
    }
    if (failed) *abort_flag = 1;
    if (helpers_store_last(p) && blockIdx.x < p.total && warp < 8) {
      // The CTA's last tile, upper half of the columns: wait for its
      // accumulator (one segment per item, so the phases of each buffer are
      // waited in order), then store through tiles in the halo, which no MMA
      // reads any more.
      constexpr int G = form_parts(FORM);
      int i_last = blockIdx.x, nitems = 0;
      for (int i = blockIdx.x; i < p.total; i += gridDim.x, ++nitems) i_last = i;
      const uint32_t u = (uint32_t)nitems - 1;  // the last item's segment (one per item)
      const int bi = (int)(u & 1);
      const uint32_t use = u >> 1;
      const int quarter = warp & 3, chalf = warp >> 2;  // converter warps 0-7: lane quarter, column quarter
      int grp, part;
      group_of<FORM>(quarter, chalf, grp, part);
      const int bar_id = 6 + grp;  // epilogue groups use 2-5 (groups of one warp none)
      // every converter warp comes here, failed or not, so both (or all
      // four) warps of a group reach the barrier; they agree to skip if any
      // of them failed or the wait gives up
      bool bad = failed || *abort_flag != 0;
      if (!bad) bad = !mbar_wait(&bars.dfull[bi], use & 1, p.err);
      bad = group_sync_or<G>(bar_id, bad);
      if (!bad) {
        tc_fence_after();
        const uint32_t sc = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)bi * kAccCols;
        float *tiles = reinterpret_cast<float *>(halo) + grp * G * kXchFloats;
        const int ncol = p.N / 4;
        store_tile_columns<TERMS, FORM>(p, decode(p, i_last), sc, sc, true, p.N / 2 + chalf * ncol, ncol, tiles,
                                        bar_id, quarter, part, lane, nullptr);
      } else {
        *abort_flag = 1;
      }
    }
  } else if (warp == kMmaWarp) {
    // ------------------------------------------------------------ MMA issuer
    using ML = MmaList<TERMS, wide_form(FORM)>;
    const uint32_t idesc = idesc_bf16_f32(128, p.N);
    // Operand descriptors are a template (layout, strides) plus the address
    // in 16-byte units; shared-memory addresses stay below 256 KB, so the
    // address field never carries into the stride fields.
    const uint64_t a_tmpl = smem_desc_kmajor(0, 128, (uint32_t)p.CB * 16);
    const uint64_t b_tmpl = smem_desc_kmajor(0, (uint32_t)p.L * 16, 128);
    const uint32_t stage0 = smem_u32(stage) >> 4, halo0 = smem_u32(halo) >> 4;
    const uint32_t chunk16 = p.chunk_bytes >> 4, part16 = p.part_bytes >> 4, stage16 = p.stage_bytes >> 4;
    const uint32_t kstep_b16 = 2u * p.L;              // B: two plane groups of L positions
    const uint32_t row16 = (uint32_t)p.CB / 8;        // A: one filter row (CB bf16) in 16-byte units
    // The issuing thread's own latency bounds the stage rate, so the loop
    // keeps to 32-bit descriptor words (the address field never carries into
    // the stride fields), per-MMA operand offsets in registers, the B offset
    // of each unit in a shared table, and stage / phase counters without
    // divisions.
    const uint32_t a_hi = (uint32_t)(a_tmpl >> 32), b_hi = (uint32_t)(b_tmpl >> 32);
    const uint32_t a_lo0 = (uint32_t)a_tmpl + stage0, b_lo0 = (uint32_t)b_tmpl + halo0;
    uint32_t aoff[ML::n], boff[ML::n];
#pragma unroll
    for (int m = 0; m < ML::n; ++m) {
      aoff[m] = (uint32_t)ML::arow(m) * row16;
      boff[m] = (uint32_t)ML::bterm(m) * part16;
    }
    int s = 0;             // stage slot
    uint32_t sph = 0;      // parity of the slot's current fill
    uint32_t hb = 0, u = 0;
    int table_key = -1;    // (sub-filter width, units) the unit table holds
    bool failed = false;
    for (int i = blockIdx.x; i < p.total && !failed; i += gridDim.x) {
      const ItemUnits iu = item_units<FORM>(p, decode(p, i));
      if (iu.ts * 1024 + iu.nu != table_key) {
        // (re)written whenever the sub-filter width or the unit count changes
        // (output phases of UpsampleInput), so every unit k < nu has its entry
        // B offset of each unit (paired: of its first tap), in 16-byte units
        const int hs = pairs_taps(FORM) ? (iu.ts + 1) / 2 : iu.ts;  // units per filter row
        for (int k = lane; k < iu.nu; k += 32) {
          const int tap = p.hblocks > 1 ? p.unit_tap[k] : (k / hs) * p.tstride + (pairs_taps(FORM) ? 2 : 1) * (k % hs);
          unit_boff[k] = (uint32_t)p.tap_phase[tap] * TERMS * part16 + (uint32_t)p.tap_off[tap];
        }
        __syncwarp();
        table_key = iu.ts * 1024 + iu.nu;
      }
      const int tstages = p.NCB * iu.nst;
      int seg_left = 0, done = 0, bi = 0, small_left = 0;
      // first: the next MMA starts a segment's (big) sum; first_small, wide forms:
      // it starts the small sums, which stay in their columns for small_segs
      // segments (plan_form says why)
      bool first = false, first_small = true;
      for (int blk = 0; blk < p.NCB * p.hblocks && !failed; ++blk, ++hb) {
        const Block bk = block_of(p, iu, blk);
        const int buf = hb & 1;
        failed = __any_sync(0xffffffffu, *abort_flag || !mbar_wait(&bars.hfull[buf], (hb >> 1) & 1, p.err));
        if (failed) break;
        tc_fence_after();
        const uint32_t hlo = b_lo0 + (uint32_t)buf * (p.halo_bytes >> 4);
        for (int u0 = bk.u0; u0 < bk.u1; u0 += p.T) {
          if (seg_left == 0) {
            // a new accumulation segment: wait until its accumulator is free
            bi = p.promote ? 0 : (int)(u & 1);
            const uint32_t use = p.promote ? u : (u >> 1);
            failed = __any_sync(0xffffffffu, !mbar_wait(&bars.dempty[bi], (use & 1) ^ 1, p.err));
            if (failed) break;
            tc_fence_after();
            seg_left = min(p.seg_stages, tstages - done);
            first = true;
            if (wide_form(FORM)) {
              if (small_left == 0) {
                small_left = p.small_segs;
                first_small = true;
              }
              --small_left;
            }
          }
          failed = __any_sync(0xffffffffu, !mbar_wait(&bars.full[s], sph, p.err));
          if (failed) break;
          tc_fence_after();
          if (elect_one()) {
            const uint32_t dt = tmem + (uint32_t)bi * kAccCols;
            const int u1 = min(bk.u1, u0 + p.T);
            uint32_t alo = a_lo0 + (uint32_t)s * stage16;
            for (int k = u0; k < u1; ++k, alo += chunk16) {
              const uint32_t blo = hlo + unit_boff[k];
              for (int j = 0; j < p.KS; ++j) {
#pragma unroll
                for (int m = 0; m < ML::n; ++m) {
                  const bool small = wide_form(FORM) && m > 0;
                  mma_bf16_ss(dt + (small ? kAccCols / 2 : 0u), desc_word(a_hi, alo + aoff[m] + 16u * j),
                              desc_word(b_hi, blo + boff[m] + (uint32_t)j * kstep_b16), idesc,
                              (m == 0 && first) || (m == 1 && wide_form(FORM) && first_small) ? 0u : 1u);
                }
                first = first_small = false;
              }
            }
            tc_commit(&bars.empty[s]);  // the stage may be refilled once these MMAs are done
          }
          __syncwarp();
          if (++s == p.stages) {
            s = 0;
            sph ^= 1u;
          }
          first = first_small = false;
          ++done;
          if (--seg_left == 0) {
            if (elect_one()) tc_commit(&bars.dfull[bi]);
            __syncwarp();
            ++u;
          }
        }
        if (failed) break;
        if (elect_one()) tc_commit(&bars.hempty[buf]);  // the halo buffer may be refilled
        __syncwarp();
      }
    }
    if (failed) *abort_flag = 1;
    // Every MMA issued retires before tensor and shared memory are released.
    if (elect_one()) tc_commit(&bars.drain);
    __syncwarp();
    mbar_wait(&bars.drain, 0, p.err);
  } else if (warp == kLoadWarp) {
    // ------------------------------------------------------------ loader
    // A bulk copy costs its issuing thread a few hundred cycles whatever its
    // size, so each stage (T consecutive taps of one plane block, contiguous
    // in the packed operand) is one copy.
    if (lane == 0) {
      if (p.after_pack) grid_dependency_wait();
      uint32_t q = 0;     // stages issued
      int s = 0;          // stage slot
      uint32_t sph = 0;   // parity of the slot's current fill
      bool ok = true;
      for (int i = blockIdx.x; ok && i < p.total && !*abort_flag; i += gridDim.x) {
        const ItemUnits iu = item_units<FORM>(p, decode(p, i));
        const uint8_t *src = p.bpack + iu.chunk0 * p.chunk_bytes;
        for (int blk = 0; ok && blk < p.NCB * p.hblocks; ++blk) {
          const Block bk = block_of(p, iu, blk);
          for (int u0 = bk.u0; u0 < bk.u1; u0 += p.T, ++q) {
            if (!mbar_wait(&bars.empty[s], sph ^ 1u, p.err)) {
              ok = false;
              break;
            }
            const uint32_t bytes = (uint32_t)min(p.T, bk.u1 - u0) * p.chunk_bytes;
            mbar_arrive_expect_tx(&bars.full[s], bytes);
            bulk_load(stage + (size_t)s * p.stage_bytes, src + ((size_t)bk.cb * iu.nu + u0) * p.chunk_bytes, bytes,
                      &bars.full[s]);
            if (++s == p.stages) {
              s = 0;
              sph ^= 1u;
            }
          }
        }
      }
      if (!ok) *abort_flag = 1;
      if (*abort_flag) {
        // copies still in flight land before shared memory is released
        for (uint32_t qq = q > (uint32_t)p.stages ? q - p.stages : 0; qq < q; ++qq)
          mbar_wait(&bars.full[qq % p.stages], (qq / p.stages) & 1, p.err);
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue
    // Lane quarters: rows 0-63 hold hi*hi sums, rows 64-127 corrections; with
    // paired taps the quarters are tap a's hi*hi, tap b's hi*hi, a's and b's
    // corrections, tap b's one grid position to the right.  The warps holding
    // the parts of one block of 32 filters for the same columns form a group
    // (two warps, or with paired taps four): store_tile_columns.
    constexpr int G = form_parts(FORM);   // parts (warps) per group
    const int ew = warp - kEpiWarp0;
    const int quarter = warp & 3;         // tensor-memory lanes this warp may access
    const int half = ew >> 2;             // column half
    int grp, part;                        // this warp's part, and its share of filters
    group_of<FORM>(quarter, half, grp, part);
    const int bar_id = 2 + grp;
    const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
    float *tiles = xch + grp * G * kXchFloats;  // the group's part tiles, [part][filter][16]
    const bool helped = helpers_store_last(p);
    uint32_t u = 0;
    bool failed = false;
    for (int i = blockIdx.x; i < p.total && !failed; i += gridDim.x) {
      const Item it = decode(p, i);
      const ItemUnits iu = item_units<FORM>(p, it);
      const int nseg = (p.NCB * iu.nst + p.seg_stages - 1) / p.seg_stages;  // accumulation segments
      // the CTA's last tile: the converters store the upper half of the columns
      const bool last_item = i + (int)gridDim.x >= p.total;
      const int ncol = (helped && last_item) ? p.N / 4 : p.N / 2;
      const int cbeg = half * ncol;
      for (int seg = 0; seg < nseg; ++seg, ++u) {
        const int bi = p.promote ? 0 : (int)(u & 1);
        const uint32_t use = p.promote ? u : (u >> 1);
        bool bad = *abort_flag != 0 || !mbar_wait(&bars.dfull[bi], use & 1, p.err);
        bad = group_sync_or<G>(bar_id, bad);  // the group agrees
        if (bad) {
          failed = true;
          break;
        }
        tc_fence_after();
        const uint32_t sc = tmem + lane_base + (uint32_t)bi * kAccCols;
        const uint32_t rc = tmem + lane_base + kAccCols;  // running sum (promotion)
        const bool first = seg == 0, last = seg == nseg - 1;
        if (!last) {
          // promotion: R (+)= S, FP32 round to nearest, over the warp's column half;
          // the small sums of a wide form with it where their segments end
          const bool small = wide_form(FORM) && (seg + 1) % p.small_segs == 0;
          for (int c = half * (p.N / 2); c < (half + 1) * (p.N / 2); c += 16) {
            uint32_t s16[16], r16[16];
            tmem_ld16(sc + c, s16);
            if (!first) tmem_ld16(rc + c, r16);
            tc_wait_ld();
            if (!first) {
#pragma unroll
              for (int t = 0; t < 16; ++t) s16[t] = __float_as_uint(__uint_as_float(s16[t]) + __uint_as_float(r16[t]));
            }
            if (small) {
              tmem_ld16(sc + kAccCols / 2 + c, r16);
              tc_wait_ld();
#pragma unroll
              for (int t = 0; t < 16; ++t) s16[t] = __float_as_uint(__uint_as_float(s16[t]) + __uint_as_float(r16[t]));
            }
            tmem_st16(rc + c, s16);
          }
          tc_wait_st();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&bars.dempty[bi]);
          continue;
        }
        // last segment: out = S (+ R) for every part of each filter
        store_tile_columns<TERMS, FORM>(p, it, sc, rc, first, cbeg, ncol, tiles, bar_id, quarter, part, lane,
                                        &bars.dempty[bi]);
      }
    }
    if (failed) *abort_flag = 1;
  }

  // ---------------------------------------------------------------- teardown
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == kMmaWarp) tmem_dealloc(tmem, 512);
}

// Pack the filter bank into per-chunk operand images: chunk (output phase,
// nb, cb, unit) = arows x CB bf16, column ci = plane cb*CB + ci, the filter
// value of the tap (flipped for convolution).  A chunk is blocks of SR source
// rows (64, wide forms 128), each the rows' values in one split term, or zero,
// as block_term() lists them (wide: the terms in order).  A source row is a
// filter nb*fblock + n of the unit's tap, or, in the pairing forms, the first
// half of the rows are tap a of the unit's filters and the second half tap a + 1
// (0 past the filter row's end).  With UpsampleInput the taps of a unit are those
// of its phase's sub-filter.  Layout: core matrices of 8 rows x 8 columns (128
// bytes), row groups SBO = CB*16 bytes apart, column groups LBO = 128 bytes
// apart.  Rows or columns past the real counts are 0.
//
// One thread per 8 planes of one source row: 8 loads in flight, then one
// 16-byte store for each block (loading the values again for every block, from
// one CTA per SM, took 147 us for a 3x3 512 -> 512 bank; 20 us now).  The
// launch is one CTA of 128 threads per SM: at 32 registers a thread its four
// warps fit in the registers a filter-bank CTA leaves free on each SM
// sub-partition, so with programmatic serialisation it is resident before the
// previous launch ends and runs the moment that launch is done (measured: 1.6 /
// 2.3 us less per forward / backward launch than one thread per value in
// 256-thread CTAs).
template <int FORM>
__global__ void __launch_bounds__(kPackThreads, 16) bank_pack_kernel(const __grid_constant__ BankParams p,
                                                                     const float *__restrict__ f,
                                                                     uint8_t *__restrict__ out) {
  constexpr int SR = wide_form(FORM) ? 128 : 64;
  const ConvGeom &g = p.g;
  const int CB8 = p.CB / 8, nblk = p.arows / SR;
  // every (phase, block, plane block, unit) slot of the largest phase; the
  // units a phase lacks are skipped.  Below 2^31 (checked at launch).
  const int total = p.nph_out * p.nblocks * p.NCB * p.nunits * SR * CB8;
  // the previous kernel (the last launch that read the packed operand) must
  // be done before it is rewritten; the consuming kernel may be scheduled now
  grid_dependency_wait();
  allow_dependent_launch();
  for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += gridDim.x * blockDim.x) {
    const int c8 = idx % CB8;
    int rest = idx / CB8;
    const int row = rest % SR;
    rest /= SR;
    const int unit = rest % p.nunits;
    rest /= p.nunits;
    const int cb = rest % p.NCB;
    rest /= p.NCB;
    const int nb = rest % p.nblocks;
    Item it{};
    it.ph = rest / p.nblocks;
    it.nb = nb;
    const ItemUnits iu = item_units<FORM>(p, it);
    if (unit >= iu.nu) continue;
    const int hs = pairs_taps(FORM) ? (iu.ts + 1) / 2 : iu.ts;
    const int k = nb * p.fblock + (pairs_taps(FORM) ? row % (SR / 2) : row);
    const int uo = p.hblocks > 1 ? p.unit_tap[unit] : unit;  // units in filter order
    const int ss = pairs_taps(FORM) ? 2 * (uo % hs) + row / (SR / 2) : uo % hs;
    const int rr = uo / hs;
    int r = rr, s = ss;
    if (p.up > 1) {
      const int rho = it.ph / p.up;
      r = p.up_r0[rho] + p.up * rr;
      s = p.up_s0[it.ph - rho * p.up] + p.up * ss;
    }
    const bool live = ss < iu.ts && r < g.R && s < g.S && k < g.groups;
    const int src = g.orient == CCT_CONVOLUTION ? (g.R - 1 - r) * g.S + (g.S - 1 - s) : r * g.S + s;
    // filter plane of (filter k, plane c), as plane_pair gives it: k*n + c
    // for projectFrame, c*groups + k for backProjectFrame
    const bool fwd = g.mode == CCT_PROJECT_FRAME_BLOCK_REDUCE_SUM;
    const int c0 = cb * p.CB + c8 * 8;
    const size_t taps = (size_t)g.R * g.S;
    const size_t fstride = fwd ? taps : (size_t)g.groups * taps;
    const float *fp = f + (fwd ? (size_t)k * g.n + c0 : (size_t)c0 * g.groups + k) * taps + src;
    float a[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) a[e] = (live && c0 + e < g.n) ? __ldg(fp + (size_t)e * fstride) : 0.0f;
    const size_t chunk = iu.chunk0 + (size_t)cb * iu.nu + unit;
    uint8_t *dst = out + chunk * ((size_t)p.arows * p.CB * 2) +
                   (uint32_t)((row >> 3) * (p.CB * 16) + c8 * 128 + (row & 7) * 16);
    for (int b = 0; b < nblk; ++b, dst += (size_t)SR * p.CB * 2) {
      const int term = wide_form(FORM) ? b : block_term(p.terms, b);
      uint32_t w[4];
#pragma unroll
      for (int e = 0; e < 8; e += 2) {
        float v[2];
#pragma unroll
        for (int d = 0; d < 2; ++d) {
          const float x = a[e + d];
          const float h = __bfloat162float(__float2bfloat16_rn(x));
          if (term < 0) {
            v[d] = 0.0f;
          } else if (term == 0) {
            v[d] = h;
          } else if (p.terms == 2) {
            v[d] = x - h;  // rounded to bf16 below
          } else {
            const float m = __bfloat162float(__float2bfloat16_rn(x - h));
            v[d] = term == 1 ? m : (x - h) - m;
          }
        }
        const __nv_bfloat162 b2 = __floats2bfloat162_rn(v[0], v[1]);  // v[0] in the low half
        w[e / 2] = *reinterpret_cast<const uint32_t *>(&b2);
      }
      *reinterpret_cast<uint4 *>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
    }
  }
}

template <int TERMS, int FORM, bool CB16>
int launch_terms(const BankParams &p, cudaStream_t st) {
  auto kern = bank_tc_kernel<TERMS, FORM, CB16>;
  int rc = raise_smem_limit(kern, p.smem_bytes, "cudaFuncSetAttribute(bank_tc)");
  if (rc) return rc;
  rc = launch_pdl(kern, dim3(p.grid), dim3(kThreads), p.smem_bytes, st, "bank_tc_kernel launch", p);
  if (rc) return rc;
  count_launches(1);
  return check_cuda(cudaGetLastError(), "bank_tc_kernel launch");
}

int floor_div(int a, int b) { return a >= 0 ? a / b : -((-a + b - 1) / b); }
int pos_mod(int a, int b) { return ((a % b) + b) % b; }

}  // namespace

namespace {

// The plan of one form, or false where the form or the kernel does not take the
// shape.  *cost: modelled MMA cycles of the longest-running CTA.
// split: one input phase per halo block.
bool plan_form(const ConvGeom &g, int terms, int form, bool split, int sms, BankParams *out, double *cost_out) {
  if (g.mode != CCT_PROJECT_FRAME_BLOCK_REDUCE_SUM && g.mode != CCT_BACK_PROJECT_FRAME_BLOCK_REDUCE_SUM)
    return false;
  if (terms != 2 && terms != 3) return false;
  if (g.fup != 1 || g.down < 1 || g.down > 2 || g.up < 1 || g.up > kBankMaxUp) return false;
  if (g.up > 1 && (g.down != 1 || g.border == CCT_BORDER_CLAMP)) return false;
  const int RS = g.R * g.S;
  if (RS > kBankMaxTaps || g.n < 1 || g.groups < 1) return false;
  BankParams p{};
  p.g = g;
  p.terms = terms;
  const int d = g.down, u = g.up;
  p.up = u;
  p.nph_out = u * u;
  int dr, dc;  // reach of the (sub-)filter on the grid, rows and columns
  int rq_max = 1, sq_max = 1;
  if (u > 1) {
    // UpsampleInput (ConvolveHyperKernel.scala:206-212, 405-459): output row
    // i = u*I + rho takes filter rows r with (rho - low_r + r) % u == 0, that
    // is r = r0 + u*rr, reading input row I + (rho - low_r + r0)/u + rr.
    // Phases without such rows keep one zero sub-filter row, so every phase
    // writes its outputs.
    for (int ph = 0; ph < u; ++ph) {
      const int r0 = pos_mod(g.low_r - ph, u), s0 = pos_mod(g.low_c - ph, u);
      p.up_r0[ph] = r0;
      p.up_s0[ph] = s0;
      p.up_rq[ph] = std::max(1, r0 < g.R ? (g.R - 1 - r0) / u + 1 : 0);
      p.up_sq[ph] = std::max(1, s0 < g.S ? (g.S - 1 - s0) / u + 1 : 0);
      p.up_sr[ph] = floor_div(ph - g.low_r + r0, u);
      p.up_sc[ph] = floor_div(ph - g.low_c + s0, u);
      rq_max = std::max(rq_max, p.up_rq[ph]);
      sq_max = std::max(sq_max, p.up_sq[ph]);
    }
    dr = rq_max - 1;
    dc = sq_max - 1;
    p.OHq = (g.OH + u - 1) / u;
    p.OWq = (g.OW + u - 1) / u;
    p.nphase = 1;
    p.tstride = sq_max;
  } else {
    // row / column shifts in strided units and the input phases the taps read
    p.sr_min = floor_div(-g.low_r, d);
    p.sc_min = floor_div(-g.low_c, d);
    dr = floor_div(g.R - 1 - g.low_r, d) - p.sr_min;
    dc = floor_div(g.S - 1 - g.low_c, d) - p.sc_min;
    p.OHq = g.OH;
    p.OWq = g.OW;
    p.tstride = g.S;
    rq_max = g.R;
    sq_max = g.S;
  }
  if (rq_max * p.tstride > kBankMaxTaps) return false;
  // paired taps: stride-1 grids only, where tap a + 1 reads one grid position
  // past tap a
  p.form = form;
  p.pair = pairs_taps(form) ? 1 : 0;
  if (p.pair && (d != 1 || sq_max < 2)) return false;
  if (form == kPair && (terms != 2 || g.groups > 32)) return false;
  if (form == kWidePair && terms != 3) return false;  // in two terms it won 19 of 30000 random shapes
  p.fblock = form == kPair ? 32 : form == kWide ? 128 : 64;
  p.nblocks = (g.groups + p.fblock - 1) / p.fblock;
  // units per phase: sub-filter rows x (columns, or column pairs)
  auto units_of = [&](int rows, int cols) { return rows * (p.pair ? (cols + 1) / 2 : cols); };
  p.nunits = 0;
  for (int ph = 0; ph < p.nph_out; ++ph) {
    const int nu = u > 1 ? units_of(p.up_rq[ph / u], p.up_sq[ph % u]) : units_of(g.R, g.S);
    p.nunits = std::max(p.nunits, nu);
  }
  const bool wide = wide_form(form);
  p.nmma = wide ? (terms == 2 ? 3 : 6) : (terms == 2 ? 2 : 5);
  p.arows = wide ? 128 * terms : (terms == 2 ? 192 : 448);
  const size_t xch_bytes = kXchBytes;
  const int NU = p.nunits;
  int phase_of[2][2] = {{-1, -1}, {-1, -1}};
  if (u > 1) {
    phase_of[0][0] = 0;
  } else {
    for (int r = 0; r < g.R; ++r)
      for (int s = 0; s < g.S; ++s) {
        const int pr = pos_mod(r - g.low_r, d), pc = pos_mod(s - g.low_c, d);
        if (phase_of[pr][pc] < 0) {
          phase_of[pr][pc] = p.nphase;
          p.phase_r[p.nphase] = pr;
          p.phase_c[p.nphase] = pc;
          ++p.nphase;
        }
      }
  }
  if (split && p.nphase == 1) return false;
  p.hblocks = split ? p.nphase : 1;
  const int NUP = (NU + p.hblocks - 1) / p.hblocks;  // units of a halo block, about
  // Band width BW, tile size N (positions) and plane block CB, by a cost
  // model: an M=128, 16-deep MMA over N positions takes N/2 tensor cycles and
  // reads 4 KB of filter plus 32*N bytes of halo from shared memory at about
  // 128 B per cycle, so its time is max(N/2, 32 + N/4) cycles; each tile also
  // pays a fixed hand-off (about 8 cycles per k-step).  Grid columns past a
  // band's outputs are paid for too, and the work items (image, band, tile,
  // filter block) run in waves of one per SM.  The
  // plan needs two halo buffers, at least three filter stages and the
  // epilogue's exchange buffers in shared memory; among equal costs the
  // larger plane block wins (fewer halo hand-offs).
  // dynamic shared memory: 227 KB per CTA less the static barriers and exchange buffers
  const size_t budget = 225 * 1024;
  // epilogue cycles a position: 64 filters (3 -> 64 planes on 8x 224x224); more where it adds
  // shifted taps, or stores 128 filters from columns of big and small sums (1.2 to 1.7
  // times per position over eight layers of 1 to 18 planes, us in 128s / in 64s: 9 -> 145
  // planes, 5x5 up 4 on 2x 104x36, three terms 113 / 98; 17 -> 106, 1x3 up 2 on 16x 22x123
  // 65 / 87; 8 -> 87, 3x3 on 16x 109x23, two terms 23 / 28)
  const double epilogue = p.pair ? 80.0 : form == kWide ? 72.0 : 50.0;
  const int cmax = ((g.n + 15) / 16) * 16;
  bool found = false;
  double best_cost = 0.0, best_waves = 0.0;
  int best_cb = 0;
  for (int bw : {p.OWq, 512, 256, 192, 128, 96, 64, 48, 32}) {
    if (bw > p.OWq || (bw == p.OWq && bw > 1024)) continue;
    const int nbands = (p.OWq + bw - 1) / bw;
    const int BW = (p.OWq + nbands - 1) / nbands;  // balanced bands
    // A pitch of whole float4s lets the epilogue store four outputs at a time, where
    // the columns it adds are at most 1 in 18 (3x3, us without / with: 32 -> 64 planes
    // on 16x 64x64 24.2 / 20.5, pitch 66 -> 68; 128 -> 256 on 56x56 58.5 / 54.2, 58 ->
    // 60; 512 -> 512 on 28x28, 30 -> 32, 114 / 123).
    const int P4 = (BW + dc + 3) & ~3;
    const bool pad = u == 1 && BW % 4 == 0 && g.OW % 4 == 0 && (P4 - BW - dc) * 18 <= BW + dc;
    const int P = pad ? P4 : BW + dc;
    const long long npos = (long long)p.OHq * P;
    for (int N : {256, 224, 192, 160, 128, 96, 64}) {
      if (wide && N > 128) continue;  // big and small sums share the accumulator's columns
      const int adv = p.pair ? N - 4 : N;  // paired: the last 4 positions of a tile lack tap b's sums
      const long long tiles = (npos + adv - 1) / adv;
      const int L = ((N + dr * P + dc) + 7) & ~7;
      for (int CB : {64, 32, 16}) {
        if (CB > cmax && CB != 16) continue;
        const size_t part = (size_t)L * CB * 2;
        const size_t halo = (((size_t)(split ? 1 : p.nphase) * terms * part) + 127) & ~(size_t)127;
        const size_t chunk = (size_t)p.arows * CB * 2;
        // Units per stage: each stage hand-off (the MMA thread's wait and
        // commit, the loader's refill) costs ~400 cycles of the issuing
        // thread's latency whatever the stage holds, so a stage takes as many
        // units as fit, up to ~2000 cycles of MMAs, in three stages; two
        // stages do when a stage holds at least ~1500 cycles of MMAs, enough
        // to cover the refill of the other (measured: 12 MMAs of N = 256 in
        // two stages beat 8 in three).
        const double tap_cycles = (CB / 16) * p.nmma * std::max(0.5 * N, 32.0 + 0.25 * N);
        auto fits = [&](int t, int st) { return 2 * halo + (size_t)st * t * chunk + xch_bytes <= budget; };
        auto ok_stages = [&](int t) { return fits(t, 3) || (fits(t, 2) && t * tap_cycles >= 1500.0); };
        int T = std::min(NUP, std::max(1, (int)(2000.0 / tap_cycles)));
        while (T > 1 && !ok_stages(T)) --T;
        if (!ok_stages(T) || L * 16 >= (1 << 18)) continue;
        if (T * tap_cycles < 500.0 && T < NUP && CB > 16) continue;  // a smaller plane block keeps stages long
        // work items run in waves over the SMs: a small problem takes smaller
        // tiles to occupy more of them
        const long long items = (long long)g.batch * p.nph_out * nbands * tiles * p.nblocks;
        const double waves = (double)((items + sms - 1) / sms);
        // a stage of less than ~500 cycles of MMAs takes that long all the same (two
        // terms, 3x3 64 -> 64 on 8x 224x224 down 2: 80 us with 256-cycle stages of N =
        // 256, 69 with longer ones of a smaller N), unless the tile has so few that its
        // epilogue takes longer (1x1, 7 -> 9 planes on 20x9: 9.2 us on one tile of 192, 7.2
        // on three of 64)
        double floor = std::max(1.0, 500.0 / (T * tap_cycles));
        if ((double)NU * ((g.n + CB - 1) / CB) * tap_cycles * floor <= epilogue * N) floor = 1.0;
        const double cost = waves * (std::max(0.5 * N, 32.0 + 0.25 * N) + 8.0) * floor;
        if (!found || cost < best_cost * 0.999 || (cost <= best_cost * 1.001 && CB > best_cb)) {
          p.nbands = nbands;
          p.BW = BW;
          p.P = P;
          p.N = N;
          p.CB = CB;
          p.L = L;
          p.part_bytes = (uint32_t)part;
          p.halo_bytes = (uint32_t)halo;
          p.chunk_bytes = (uint32_t)chunk;
          p.T = T;
          p.stage_bytes = (uint32_t)(T * chunk);
          p.stages = (int)std::min<size_t>(6, (budget - 2 * halo - xch_bytes) / p.stage_bytes);
          p.tile_adv = adv;
          p.tiles_band = (int)tiles;
          best_cost = cost;
          best_waves = waves;
          best_cb = CB;
          found = true;
        }
        break;  // the largest plane block that fits
      }
    }
  }
  if (!found) return false;
  if (u > 1) {
    // sub-filter tap (rr, ss) of any phase: grid offset rr*P + ss
    for (int rr = 0; rr < rq_max; ++rr)
      for (int ss = 0; ss < sq_max; ++ss) {
        p.tap_phase[rr * p.tstride + ss] = 0;
        p.tap_off[rr * p.tstride + ss] = rr * p.P + ss;
      }
  } else {
    for (int tap = 0; tap < RS; ++tap) {
      const int r = tap / g.S, s = tap % g.S;
      const int ar = r - g.low_r, ac = s - g.low_c;
      p.tap_phase[tap] = split ? 0 : phase_of[pos_mod(ar, d)][pos_mod(ac, d)];
      p.tap_off[tap] = (floor_div(ar, d) - p.sr_min) * p.P + (floor_div(ac, d) - p.sc_min);
    }
  }
  p.NCB = (g.n + p.CB - 1) / p.CB;
  if (split) {  // units ordered by the phase they read
    int k = 0;
    p.nst = 0;
    for (int ph = 0; ph < p.nphase; ++ph) {
      p.ph_u0[ph] = k;
      for (int tap = 0; tap < RS; ++tap)
        if (phase_of[pos_mod(tap / g.S - g.low_r, d)][pos_mod(tap % g.S - g.low_c, d)] == ph) p.unit_tap[k++] = tap;
      p.nst += (k - p.ph_u0[ph] + p.T - 1) / p.T;
    }
    p.ph_u0[p.nphase] = k;
  }
  p.KS = p.CB / 16;
  if (!split) p.nst = (NU + p.T - 1) / p.T;
  const int tstages = p.NCB * p.nst;
  // Promotion: the hi*hi accumulator takes at most 64 k-steps (1024 terms of
  // the reduction) before it is added into the FP32 running sum.
  const int kmax = 64;
  p.promote = p.NCB * NU * p.KS > kmax ? 1 : 0;
  p.seg_stages = p.promote ? std::max(1, kmax / (p.T * p.KS)) : tstages;
  if (p.promote) {
    // as many segments as that takes, of equal length: the error of a segment grows
    // with its length (1.46e-8 of the result per k-step of three terms), so 48 + 48 + 48
    // loses less than 64 + 64 + 16 (256 -> 192 planes, 3x3: 7.0e-7 against 9.3e-7 RMS)
    const int nseg = (tstages + p.seg_stages - 1) / p.seg_stages;
    p.seg_stages = (tstages + nseg - 1) / nseg;
  }
  // The small sums of the wide forms are a 2^-8 part of the result and could take 2^8
  // times the MMAs of a segment for the same error; they are promoted within 2^4 times,
  // every 1280 MMAs at most (0.3 % of the error; left in the accumulator for the
  // whole of 6400 k-steps they raised it by a quarter).
  p.small_segs = std::max(1, 1280 / (p.seg_stages * p.T * p.KS * (p.nmma - 1)));
  // float4 stores: groups of 4 grid positions (p0, N and tile_adv are multiples of 4)
  // never straddle a grid row or the band's last output column, and land on
  // 16-byte aligned outputs
  // (up-sampled outputs are strided: scalar stores)
  p.vec4 = (u == 1 && p.P % 4 == 0 && p.BW % 4 == 0 && g.OW % 4 == 0 && p.N % 4 == 0) ? 1 : 0;
  const long long total = (long long)g.batch * p.nph_out * p.nbands * p.tiles_band * p.nblocks;
  if (total < 1 || total > 0x7fffffffLL) return false;
  p.total = (int)total;
  p.grid = std::min(p.total, sms);
  p.sms = sms;
  p.smem_bytes = 2 * (size_t)p.halo_bytes + (size_t)p.stages * p.stage_bytes;
  // packed chunks: each output phase's filter blocks, plane blocks and units
  size_t chunks = 0;
  for (int ph = 0; ph < p.nph_out; ++ph) {
    p.up_choff[ph] = (int)chunks;
    const int nu = u > 1 ? units_of(p.up_rq[ph / u], p.up_sq[ph % u]) : NU;
    chunks += (size_t)p.nblocks * p.NCB * nu;
  }
  p.pack_bytes = chunks * p.chunk_bytes;
  *out = p;
  // A tile takes its MMAs or its epilogue, whichever is longer.
  double units = 0.0;
  for (int ph = 0; ph < p.nph_out; ++ph)
    units += u > 1 ? units_of(p.up_rq[ph / u], p.up_sq[ph % u]) : NU;
  const double mmas = best_cost / best_waves * p.NCB * p.KS * p.nmma * units / p.nph_out;
  *cost_out = best_waves * std::max(mmas, epilogue * p.N);
  return true;
}

}  // namespace

bool bank_tc_plan(const ConvGeom &g, int terms, int sms, BankParams *out) {
  // Banks of at most 32 filters would leave half of each 128-row MMA empty: two
  // taps of a filter row share it instead where they can.
  BankParams p{}, w{};
  double cost = 0.0, wcost = 0.0;
  const bool paired = terms == 2 && plan_form(g, terms, kPair, false, sms, &p, &cost);
  const bool ok = paired || plan_form(g, terms, kPlain, false, sms, &p, &cost);
  if (!ok) return false;
  p.pack_limit = p.pack_bytes;
  // The wide forms where the model says they take fewer MMA cycles: 128 filters
  // (from 0.95: 256 -> 512 planes on 8x 28x28, three terms 134 -> 94 us, two terms
  // 70 -> 62), or 64 filters x two taps, whose smaller tiles convert and store more
  // per position (from 0.78: three terms, 5x5 64 -> 32 planes on 16x 64x64, 0.74,
  // 96 -> 85 us; 3x3 64 -> 64 on 8x 112x112, 0.83, 60 / 69 us).  Never a larger
  // packed operand: whoever holds a fixed scratch for it keeps what it takes.
  const int form = paired ? -1 : g.groups > 64 ? kWide : kWidePair;
  if (form >= 0 && plan_form(g, terms, form, false, sms, &w, &wcost) && wcost < (form == kWide ? 0.95 : 0.78) * cost &&
      w.pack_bytes <= p.pack_bytes) {
    w.pack_limit = p.pack_bytes;
    p = w;
    cost = wcost;
  }
  // One input phase per halo block, where that lets a three-term DownsampleOutput(2)
  // layer have longer stages: all four phases often leave room for one tap of 16
  // planes (3x3 64 -> 64 on 8x 224x224: 129 us, 92 split; 7x7 32 -> 32 on 4x 64x64: 47 /
  // 33).  At equal stages it loses (256 -> 256 on 56x56: 59 / 62), and in two terms,
  // whose phases of one tap convert for longer than they multiply (80 / 96, 41 / 46).
  if (terms == 3 && plan_form(g, terms, p.form, true, sms, &w, &wcost) && wcost < 0.97 * cost &&
      w.pack_bytes <= p.pack_limit) {
    w.pack_limit = p.pack_limit;
    p = w;
  }
  *out = p;
  return true;
}

int launch_bank_pack(const BankParams &p, const float *f, uint8_t *packed, cudaStream_t st) {
  const long long total = (long long)p.nph_out * p.nblocks * p.NCB * p.nunits * (wide_form(p.form) ? 128 : 64) * (p.CB / 8);
  if (total > 0x7fffffffLL) return set_error(CCT_ENOTSUP, "packed filter operand too large");
  // One CTA per SM (more would wait for the filter-bank CTAs to leave) while a
  // thread then packs one or two rows; a larger bank takes up to 16 (dynamic filter,
  // one / more, us by rows per thread: 1.1, 7x7 96 -> 32 planes on 2x 45x85 31.9 / 41.8;
  // 1.4, 5x5 64 -> 128 on 8x 40x40 28.4 / 27.6; 1.5, 7x7 128 -> 32 39.3 / 50.9; 2.9, 3x3 192 ->
  // 192 on 8x 28x28 47.1 / 43.4; 3.9, 256 -> 256 65.2 / 51.1).
  const long long ctas = (total + kPackThreads - 1) / kPackThreads;
  const int blocks = (int)std::min<long long>(ctas, ctas > 2LL * p.sms ? 16LL * p.sms : p.sms);
  const auto kern = p.form == kPair       ? bank_pack_kernel<kPair>
                    : p.form == kWide     ? bank_pack_kernel<kWide>
                    : p.form == kWidePair ? bank_pack_kernel<kWidePair>
                                          : bank_pack_kernel<kPlain>;
  const int rc = launch_pdl(kern, dim3(blocks), dim3(kPackThreads), 0, st, "bank_pack_kernel launch", p, f, packed);
  if (rc) return rc;
  count_launches(1);
  return check_cuda(cudaGetLastError(), "bank_pack_kernel launch");
}

int launch_bank_tc(const BankParams &p, const float *x, float *y, const uint8_t *packed, unsigned *err,
                   cudaStream_t st, bool after_pack) {
  BankParams q = p;
  q.after_pack = after_pack ? 1 : 0;
  q.x = x;
  q.y = y;
  if ((reinterpret_cast<uintptr_t>(y) & 15) != 0) q.vec4 = 0;  // float4 stores need a 16-byte aligned output
  q.bpack = packed;
  q.err = err;
  const bool cb16 = p.CB == 16;
#define CCT_BANK_CASE(TT, FF) \
  if (p.terms == TT && p.form == FF) return cb16 ? launch_terms<TT, FF, true>(q, st) : launch_terms<TT, FF, false>(q, st);
  CCT_BANK_CASE(2, kPlain) CCT_BANK_CASE(2, kPair) CCT_BANK_CASE(2, kWide)
  CCT_BANK_CASE(3, kPlain) CCT_BANK_CASE(3, kWide) CCT_BANK_CASE(3, kWidePair)
#undef CCT_BANK_CASE
  return set_error(CCT_ENOTSUP, "filter-bank kernel: no form %d of %d terms", p.form, p.terms);
}

}  // namespace cct

namespace cct {

bool frame_tc_choose(const ConvGeom &g, int precision, int sms, FrameTcChoice *out) {
  FrameTcChoice c{};
  BankParams bp{};
  const bool bank_ok = bank_tc_plan(g, precision == CCT_PREC_BF16X6 ? 3 : 2, sms, &bp);
  if (bank_ok && (bp.form == kPair || g.groups > 32 || precision != CCT_PREC_BF16X3)) {
    c.bank = true;
    c.bp = bp;
    c.pack_bytes = bp.pack_bytes;
  } else if (precision == CCT_PREC_BF16X3 && frame_tc_plan(g, sms, &c.tp)) {
    c.bank = false;
    c.pack_bytes = c.tp.pack_bytes;
  } else if (bank_ok) {
    c.bank = true;
    c.bp = bp;
    c.pack_bytes = bp.pack_bytes;
  } else {
    return false;
  }
  *out = c;
  return true;
}

int frame_tc_pack(const FrameTcChoice &c, const float *f, uint8_t *packed, cudaStream_t st) {
  return c.bank ? launch_bank_pack(c.bp, f, packed, st) : launch_pack_filters(c.tp, f, packed, st);
}

int frame_tc_run(const FrameTcChoice &c, const float *x, float *y, const uint8_t *packed, unsigned *err,
                 cudaStream_t st, bool after_pack) {
  if (c.bank) return launch_bank_tc(c.bp, x, y, packed, err, st, after_pack);
  if ((reinterpret_cast<uintptr_t>(x) & 15) != 0)
    return set_error(CCT_EINVAL, "image pointer must be 16-byte aligned for the tensor-core path");
  return launch_frame_tc(c.tp, x, y, packed, err, st);
}

}  // namespace cct
