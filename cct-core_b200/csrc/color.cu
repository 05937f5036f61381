// Colour-field convolution (generator/DynamicConvolutionGenerator.scala:
// 89-106): a ColorField is an RGBA UNORM_INT8 image (OpenCLBuffer.scala:
// 135-136).  The reference splits it into red, green and blue scalar planes
// (ColorPlaneHyperKernel: byte / 255), convolves each with the scalar filter
// through the ordinary convolution triage, and merges the three results into
// a colour field (CreateColorFieldHyperKernel: (r, g, b, 1) written to the
// UNORM_INT8 image, i.e. saturate(v * 255) rounded half to even).
//
// Here a colour plan wraps one plane plan over the three planes (one
// launch, the filter shared) between an unpack and a pack kernel.  Small square
// filters without sampling that the plane plan would run directly take one
// kernel from bytes to bytes instead.
#include <cuda_runtime.h>

#include <new>

#include "cct_internal.h"
#include "sm100_util.cuh"
#include "stencil.cuh"

namespace cct {
namespace {

__global__ void color_unpack_kernel(long long n, const uchar4 *__restrict__ rgba, float *__restrict__ planes) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const uchar4 v = rgba[i];
    planes[i] = (float)v.x / 255.0f;
    planes[n + i] = (float)v.y / 255.0f;
    planes[2 * n + i] = (float)v.z / 255.0f;
  }
}

__device__ __forceinline__ unsigned char to_unorm8(float v) {
  const float s = v * 255.0f;
  // fmaxf/fminf return the number for a NaN operand, so NaN saturates to 0
  return (unsigned char)__float2uint_rn(fminf(fmaxf(s, 0.0f), 255.0f));
}

__global__ void color_pack_kernel(long long n, const float *__restrict__ planes, uchar4 *__restrict__ rgba) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    rgba[i] = make_uchar4(to_unorm8(planes[i]), to_unorm8(planes[n + i]), to_unorm8(planes[2 * n + i]), 255);
}

// Bytes to bytes: a CTA of 128 threads stages the halo of 64 columns x 8 V rows
// as three float planes (byte / 255 from a table of the 256 quotients) and runs
// the plane stencil on each, in the plane kernels' summation order, so the bytes
// are those of the unpack, convolve and pack launches.
// Bound: FP32 issue (three times R*S multiply-adds and R adds per pixel).  The
// three launches moved six float planes through memory besides: 1080x1920, 5x5
// clamp, 34.9 us against 17.8.
constexpr int kCT = 128, kCU = 4, kCTX = 16, kCTY = 8, kCTW = kCTX * kCU;

template <int R, int V>
__global__ void __launch_bounds__(kCT, R == 7 ? 4 : 5)
    color_stencil_kernel(ConvGeom g, const uchar4 *__restrict__ x, const float *__restrict__ f, uchar4 *__restrict__ y,
                         int tiles_x) {
  constexpr int TH = kCTY * V, COLS = kCTW + R - 1, ROWS = TH + R - 1, PITCH = (COLS + 3) & ~3;
  constexpr int E4 = (kCU + R - 1 + 3) / 4, PAGE = ROWS * PITCH, KC = (COLS + 31) / 32, NW = kCT / 32, RD = 2;
  static_assert(4 * E4 + kCTW - kCU <= PITCH, "a thread's loads stay inside its row");
  extern __shared__ __align__(16) float tile[];  // [channel][row][PITCH]
  __shared__ float unorm[256];
  for (int i = threadIdx.x; i < 256; i += kCT) unorm[i] = (float)i / 255.0f;
  grid_dependency_wait();  // launched with programmatic serialisation: nothing global before this

  const int tx_i = blockIdx.x % tiles_x, ty_i = blockIdx.x / tiles_x;
  const int tx = threadIdx.x % kCTX, ty = threadIdx.x / kCTX, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int r0 = ty_i * TH, c0 = tx_i * kCTW, rows = min(TH, g.OH - r0);
  float w[R][R];
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int s = 0; s < R; ++s)
      w[r][s] = __ldg(f + (g.orient == CCT_CONVOLUTION ? (R - 1 - r) * R + (R - 1 - s) : r * R + s));
  int sc[KC];
#pragma unroll
  for (int k = 0; k < KC; ++k) sc[k] = stencil_index(g.border, c0 - g.low_c + lane + 32 * k, g.W);
  __syncthreads();  // the table

  // two rows a round: their loads are in flight together
  const int need = rows + R - 1;
  for (int tr = warp; tr < need; tr += RD * NW) {
    uchar4 v[RD][KC];
    bool ok[RD][KC];
#pragma unroll
    for (int h = 0; h < RD; ++h) {
      const int t = tr + h * NW, sr = t < need ? stencil_index(g.border, r0 - g.low_r + t, g.H) : -1;
      const uchar4 *row = x + (size_t)(sr < 0 ? 0 : sr) * g.W;
#pragma unroll
      for (int k = 0; k < KC; ++k) {
        ok[h][k] = sr >= 0 && sc[k] >= 0 && lane + 32 * k < COLS;
        v[h][k] = ok[h][k] ? __ldg(row + sc[k]) : make_uchar4(0, 0, 0, 0);
      }
    }
#pragma unroll
    for (int h = 0; h < RD; ++h)
      if (tr + h * NW < need) {
        float *d = tile + (tr + h * NW) * PITCH + lane;
#pragma unroll
        for (int k = 0; k < KC; ++k)
          if (lane + 32 * k < COLS) {  // what reads zero is byte 0: 0 / 255 is 0
            d[32 * k] = unorm[v[h][k].x];
            d[32 * k + PAGE] = unorm[v[h][k].y];
            d[32 * k + 2 * PAGE] = unorm[v[h][k].z];
          }
      }
  }
  __syncthreads();
  allow_dependent_launch();
  if (ty * V >= rows) return;

  unsigned out[V][kCU];
#pragma unroll
  for (int v = 0; v < V; ++v)
#pragma unroll
    for (int u = 0; u < kCU; ++u) out[v][u] = 255u << 24;
#pragma unroll 1
  for (int ch = 0; ch < 3; ++ch) {
    const float *base = tile + ch * PAGE + (ty * V) * PITCH + tx * kCU;
    float rs[V][kCU];
#pragma unroll
    for (int v = 0; v < V; ++v)
#pragma unroll
      for (int u = 0; u < kCU; ++u) rs[v][u] = 0.0f;
#pragma unroll
    for (int tr = 0; tr < V - 1 + R; ++tr) {
      float vals[4 * E4];
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
          for (int u = 0; u < kCU; ++u) {
            float cs = 0.0f;
#pragma unroll
            for (int s = 0; s < R; ++s) cs = __fmaf_rn(vals[u + s], w[r][s], cs);
            rs[v][u] = __fadd_rn(rs[v][u], cs);
          }
        }
      }
    }
#pragma unroll
    for (int v = 0; v < V; ++v)
#pragma unroll
      for (int u = 0; u < kCU; ++u) out[v][u] |= (unsigned)to_unorm8(rs[v][u]) << (8 * ch);
  }
  const int col = c0 + tx * kCU;
  const bool vec = (g.OW & 3) == 0 && (reinterpret_cast<uintptr_t>(y) & 15) == 0;
#pragma unroll
  for (int v = 0; v < V; ++v)
    if (ty * V + v < rows && col < g.OW) {
      unsigned *dst = reinterpret_cast<unsigned *>(y) + (size_t)(r0 + ty * V + v) * g.OW + col;
      if (vec) {
        *reinterpret_cast<uint4 *>(dst) = make_uint4(out[v][0], out[v][1], out[v][2], out[v][3]);
      } else {
#pragma unroll
        for (int u = 0; u < kCU; ++u)
          if (col + u < g.OW) dst[u] = out[v][u];
      }
    }
}

template <int R, int V>
int launch_color(const ConvGeom &g, const uchar4 *x, const float *f, uchar4 *y, cudaStream_t st) {
  constexpr int PITCH = (kCTW + R - 1 + 3) & ~3;
  constexpr size_t smem = sizeof(float) * 3 * (kCTY * V + R - 1) * PITCH;
  static_assert(smem <= 48 * 1024 - 1024, "the default shared memory limit");
  const int tiles_x = (g.OW + kCTW - 1) / kCTW, tiles_y = (g.OH + kCTY * V - 1) / (kCTY * V);
  const long long blocks = (long long)tiles_x * tiles_y;
  if (blocks > 0x7fffffffLL) return set_error(CCT_ENOTSUP, "colour convolution grid too large");
  const int rc = launch_pdl(color_stencil_kernel<R, V>, dim3((unsigned)blocks), dim3(kCT), smem, st,
                            "color_stencil_kernel launch", g, x, f, y, tiles_x);
  if (!rc) count_launches(1);
  return rc;
}

// Square filters of 1, 3, 5 or 7 without sampling.
bool color_fused(const ConvGeom &g) {
  return g.up == 1 && g.down == 1 && g.R == g.S && (g.R == 1 || g.R == 3 || g.R == 5 || g.R == 7);
}
int launch_color_fused(const ConvGeom &g, const uchar4 *x, const float *f, uchar4 *y, cudaStream_t st) {
  // 16-row tiles once they give each of 148 SMs two CTAs, else 8-row ones
  // (5x5, us with V = 4 / 2 / 1: 1080x1920 19.5 / 17.8 / 21.9, 400x500 - / 5.0 /
  // 4.5, 120x160 - / 4.2 / 3.2)
  const long long tall = (long long)((g.OW + kCTW - 1) / kCTW) * ((g.OH + 15) / 16);
#define CCT_COLOR_CASE(RR) \
  case RR: return tall >= 2 * 148 ? launch_color<RR, 2>(g, x, f, y, st) : launch_color<RR, 1>(g, x, f, y, st);
  switch (g.R) {
    CCT_COLOR_CASE(1) CCT_COLOR_CASE(3) CCT_COLOR_CASE(5) CCT_COLOR_CASE(7)
    default: return set_error(CCT_ENOTSUP, "colour stencil: filter %d", g.R);
  }
#undef CCT_COLOR_CASE
}

unsigned grid_for(long long n) {
  const long long b = (n + 255) / 256;
  return (unsigned)(b < 148LL * 16 ? (b < 1 ? 1 : b) : 148LL * 16);
}

}  // namespace
}  // namespace cct

using namespace cct;

struct cct_color_plan {
  cct_conv_plan *planes;  // the plane plan over red, green, blue
  bool fused;             // one kernel from bytes to bytes
  ConvGeom g;
  uchar4 *copy;           // fused: a copy of the image, read where the output overlaps it
  float *in, *out;        // 3 planes each (not fused)
  long long n_in, n_out;  // pixels per plane
};

extern "C" {

int cct_color_plan_create(const cct_conv_desc *desc, cct_color_plan **out) {
  if (!out) return set_error(CCT_EINVAL, "null plan output");
  *out = nullptr;
  if (!desc) return set_error(CCT_EINVAL, "null descriptor");
  if (desc->struct_size != (int32_t)sizeof(cct_conv_desc))
    return set_error(CCT_EINVAL, "descriptor struct_size %d != %d", desc->struct_size, (int)sizeof(cct_conv_desc));
  if (desc->image_planes > 1)
    return set_error(CCT_EINVAL, "colour convolution: the image is one colour field (image_planes 0 or 1)");
  if (desc->filter_planes > 1)
    return set_error(CCT_EINVAL, "colour convolution needs a scalar filter");
  if (desc->vector_mode != CCT_PLANE_BY_PLANE)
    return set_error(CCT_EINVAL, "colour convolution is plane by plane (projections need a real image input)");
  if (desc->precision != CCT_PREC_FP32) return set_error(CCT_EINVAL, "colour convolution runs in FP32");
  cct_conv_desc d = *desc;
  d.image_planes = 3;
  d.filter_planes = 0;
  int32_t orows = 0, ocols = 0;
  int rc = cct_conv_output_shape(&d, &orows, &ocols, nullptr);
  if (rc) return rc;
  cct_color_plan *p = new (std::nothrow) cct_color_plan();
  if (!p) return set_error(CCT_ENOMEM, "plan allocation failed");
  rc = cct_conv_plan_create(&d, &p->planes);
  p->n_in = (long long)d.image_rows * d.image_cols;
  p->n_out = (long long)orows * ocols;
  if (!rc) rc = resolve_geom(&d, &p->g);
  int32_t algo = -1;
  if (!rc) rc = cct_conv_plan_algo(p->planes, &algo);
  if (!rc) plan_fft_whole_grid(p->planes);
  p->fused = !rc && algo == 0 && color_fused(p->g);
  if (p->fused) {
    rc = check_cuda(cudaMalloc(&p->copy, p->n_in * sizeof(uchar4)), "cudaMalloc(colour image copy)");
    if (rc) {
      cct_color_plan_destroy(p);
      return rc;
    }
    *out = p;
    return CCT_OK;
  }
  if (!rc) rc = check_cuda(cudaMalloc(&p->in, 3 * p->n_in * sizeof(float)), "cudaMalloc(colour planes)");
  if (!rc) rc = check_cuda(cudaMalloc(&p->out, 3 * p->n_out * sizeof(float)), "cudaMalloc(colour planes)");
  if (rc) {
    cct_color_plan_destroy(p);
    return rc;
  }
  *out = p;
  return CCT_OK;
}

int cct_color_plan_destroy(cct_color_plan *p) {
  if (!p) return CCT_OK;
  cct_conv_plan_destroy(p->planes);
  cudaFree(p->copy);
  cudaFree(p->in);
  cudaFree(p->out);
  delete p;
  return CCT_OK;
}

int cct_color_plan_set_static_filter(cct_color_plan *p, const float *host_filter) {
  if (!p) return set_error(CCT_EINVAL, "null plan");
  return cct_conv_plan_set_static_filter(p->planes, host_filter);
}

int cct_color_run(const cct_color_plan *p, const uint8_t *image, const float *filter, uint8_t *out, void *stream) {
  if (!p) return set_error(CCT_EINVAL, "null plan");
  if (!image || !out) return set_error(CCT_EINVAL, "null image or output pointer");
  if ((reinterpret_cast<uintptr_t>(image) & 3) != 0 || (reinterpret_cast<uintptr_t>(out) & 3) != 0)
    return set_error(CCT_EINVAL, "colour fields must be 4-byte aligned");
  cudaStream_t st = (cudaStream_t)stream;
  if (p->fused) {
    cct_conv_desc desc;
    const float *dev_filter = nullptr;
    size_t elems = 0;
    int device = 0;
    int rc = plan_record_parts(p->planes, &desc, &dev_filter, &elems, &device);
    if (rc) return rc;
    if (!filter) filter = dev_filter;
    if (!filter) return set_error(CCT_EINVAL, "null image, filter or output pointer");
    const uchar4 *x = reinterpret_cast<const uchar4 *>(image);
    // A CTA reads the halo of its tile while others store theirs: an image that
    // the output overlaps is read from a copy.
    if (image < out + 4 * p->n_out && out < image + 4 * p->n_in) {
      rc = check_cuda(cudaMemcpyAsync(p->copy, x, p->n_in * sizeof(uchar4), cudaMemcpyDeviceToDevice, st),
                      "colour image copy");
      if (rc) return rc;
      x = p->copy;
    }
    return launch_color_fused(p->g, x, filter, reinterpret_cast<uchar4 *>(out), st);
  }
  color_unpack_kernel<<<grid_for(p->n_in), 256, 0, st>>>(p->n_in, reinterpret_cast<const uchar4 *>(image), p->in);
  count_launches(1);
  int rc = check_cuda(cudaGetLastError(), "colour unpack launch");
  if (rc) return rc;
  rc = cct_conv_run(p->planes, p->in, filter, p->out, stream);
  if (rc) return rc;
  color_pack_kernel<<<grid_for(p->n_out), 256, 0, st>>>(p->n_out, p->out, reinterpret_cast<uchar4 *>(out));
  count_launches(1);
  return check_cuda(cudaGetLastError(), "colour pack launch");
}

}  // extern "C"
