// smvs_pyramid.cu — the coarse-to-fine image pyramid on the GPU.
//
// The reference runs its PatchMatch passes per pyramid level on images it
// rescales on the host (PatchMatchController::ProcessProblem,
// patch_match_controller.cc:4407-4410 and 4610, Image::Rescale,
// src/mvs/image.cc:44-70, through FreeImage's bilinear filter), and carries
// depth and normal maps between levels by DepthMap::Rescale / NormalMap::
// Rescale (src/mvs/depth_map.cc:32-55, src/mvs/normal_map.cc:27-72), i.e.
// InterpolateImage -> ResampleImageBilinear (src/util/mat.cc:18-58, 129-137)
// followed by a re-normalisation of the normals. This unit does both on the
// device:
// * RescaleImageKernel: separable resampling with the bilinear (triangle)
//   filter widened by the inverse scale when minifying (the published
//   algorithm of FreeImage's FILTER_BILINEAR rescale; FreeImage itself is a
//   third-party library that is not part of the reference tree), weights
//   normalised over the pixels inside the image, result rounded to an
//   integer grey level 0..255 like the 8-bit bitmap.
// * ResampleMapKernel: ResampleImageBilinear exactly (same float expressions,
//   constant-0 border), for the depth map and each normal slice, then the
//   normal re-normalisation. This unit is compiled without FMA contraction
//   and with IEEE division and square root, so its results equal the C
//   restatement in the oracle bit for bit.
#include <cmath>

#include <cuda_runtime.h>

#include "../../include/smvs.h"

extern "C" void smvs_internal_set_error(const char* msg);

namespace {

constexpr int kBlockX = 32, kBlockY = 8;

// The image filter gives a thread four outputs from this many outputs of the row
// pass on, where it still fills the GPU: 3000x2000 halved takes 26 us against 36 us
// with one each (cold L2, both launches), 1500x1000 15 against 17, 750x500 13
// against 11.
constexpr size_t kRescaleFour = 500000;

// The filter's tap range and centre for output pixel `o` of `n` input pixels;
// `support` is the triangle's half-width in input pixels, `fscale` its inverse.
__device__ __forceinline__ float Taps(int o, int n, float scale, float support, int* i0, int* i1) {
  const float c = ((float)o + 0.5f) / scale;
  *i0 = max((int)floorf(c - support), 0);
  *i1 = min((int)ceilf(c + support), n - 1);
  return c;
}

// One pass of the separable image filter over rows (axis 0 = along x).
// out[y][x] = sum_i w_i in[y][i] / sum_i w_i for the input pixels i whose
// centres lie within the filter support around the output pixel's centre.
// The weights depend on x alone: a thread computes each once for kRows rows,
// whose loads are independent of one another. Bound by its instructions (75 % of
// the issue slots; the weight took half of them with one row a thread):
// 3000x2000 to 1500x2000 takes 15 us (18.7 us before), its bytes 6 us.
template <int kRows>
__global__ void __launch_bounds__(kBlockX* kBlockY) ResampleRowsKernel(const float* __restrict__ in, int w, int h,
                                                                       float* __restrict__ out, int ow, float scale,
                                                                       float support, float fscale) {
  const int x = blockIdx.x * kBlockX + threadIdx.x;
  const int y0 = (blockIdx.y * kBlockY + threadIdx.y) * kRows;
  if (x >= ow || y0 >= h) return;
  int i0, i1;
  const float c = Taps(x, w, scale, support, &i0, &i1);
  float acc[kRows], wsum = 0.f;
#pragma unroll
  for (int k = 0; k < kRows; ++k) acc[k] = 0.f;
  const float* row = in + (size_t)y0 * w;
  for (int i = i0; i <= i1; ++i) {
    const float wt = 1.0f - fabsf(((float)i + 0.5f) - c) * fscale;
    if (wt <= 0.f) continue;
#pragma unroll
    for (int k = 0; k < kRows; ++k)
      if (y0 + k < h) acc[k] += wt * __ldg(row + (size_t)k * w + i);
    wsum += wt;
  }
#pragma unroll
  for (int k = 0; k < kRows; ++k)
    if (y0 + k < h) out[(size_t)(y0 + k) * ow + x] = wsum > 0.f ? acc[k] / wsum : 0.f;
}

// The same filter along y; rounds to an integer grey level. The weights depend
// on y alone: a thread computes each once for kCols columns, a warp apart.
// 1500x2000 to 1500x1000: 9.4 us (11.7 us before), its bytes 3 us.
template <int kCols>
__global__ void __launch_bounds__(kBlockX* kBlockY) ResampleColsKernel(const float* __restrict__ in, int w, int h,
                                                                       float* __restrict__ out, int oh, float scale,
                                                                       float support, float fscale) {
  const int x0 = blockIdx.x * (kBlockX * kCols) + threadIdx.x;
  const int y = blockIdx.y * kBlockY + threadIdx.y;
  if (x0 >= w || y >= oh) return;
  int i0, i1;
  const float c = Taps(y, h, scale, support, &i0, &i1);
  float acc[kCols], wsum = 0.f;
#pragma unroll
  for (int k = 0; k < kCols; ++k) acc[k] = 0.f;
  for (int i = i0; i <= i1; ++i) {
    const float wt = 1.0f - fabsf(((float)i + 0.5f) - c) * fscale;
    if (wt <= 0.f) continue;
    const float* row = in + (size_t)i * w + x0;
#pragma unroll
    for (int k = 0; k < kCols; ++k)
      if (x0 + k * kBlockX < w) acc[k] += wt * __ldg(row + k * kBlockX);
    wsum += wt;
  }
#pragma unroll
  for (int k = 0; k < kCols; ++k) {
    if (x0 + k * kBlockX >= w) continue;
    const float v = wsum > 0.f ? acc[k] / wsum : 0.f;
    out[(size_t)y * w + x0 + k * kBlockX] = fminf(255.f, fmaxf(0.f, rintf(v)));
  }
}

// ResampleImageBilinear (mat.cc:18-58) of the depth map and (or) the normal
// map's three planes, then the re-normalisation of NormalMap::Rescale
// (normal_map.cc:57-72). A thread takes one column over kRows output rows: the
// column's position and weights are computed once, and an input row's
// horizontal interpolation serves every output row that lies between it and a
// neighbour. Bound by its instructions (85 % of the issue slots), a third of them
// the IEEE root and divisions of the normal. Depth and normal 1500x1000 to
// 3000x2000: 39 us (49 + 90 us before, a launch each), its bytes 18 us.
template <bool kDepth, bool kNormal, int kRows>
__global__ void __launch_bounds__(kBlockX* kBlockY)
    ResampleMapKernel(const float* __restrict__ depth, const float* __restrict__ normal, int rows, int cols,
                      float* __restrict__ out_depth, float* __restrict__ out_normal, int new_rows, int new_cols) {
  constexpr int kPlanes = (kDepth ? 1 : 0) + (kNormal ? 3 : 0);
  const int c = blockIdx.x * kBlockX + threadIdx.x;
  const int r0 = (blockIdx.y * kBlockY + threadIdx.y) * kRows;
  if (c >= new_cols || r0 >= new_rows) return;
  const float scale_r = (float)rows / (float)new_rows;
  const float scale_c = (float)cols / (float)new_cols;
  const float c_i = ((float)c + 0.5f) * scale_c - 0.5f;
  const int c_i_min = (int)floorf(c_i);
  const int c_i_max = c_i_min + 1;
  const float d_c_min = c_i - (float)c_i_min;
  const float d_c_max = (float)c_i_max - c_i;
  const bool in_min = c_i_min >= 0 && c_i_min < cols, in_max = c_i_max >= 0 && c_i_max < cols;
  const size_t in_plane = (size_t)rows * cols, out_plane = (size_t)new_rows * new_cols;
  const float* src[kPlanes];
#pragma unroll
  for (int p = 0; p < kPlanes; ++p)
    src[p] = (kDepth && p == 0 ? depth : normal + (p - (kDepth ? 1 : 0)) * in_plane) + c_i_min;
  // An input row between its columns; 0 outside the map.
  auto across = [&](int row, float (&v)[kPlanes]) {
    const bool inside = row >= 0 && row < rows;
    const size_t at = (size_t)(inside ? row : 0) * cols;
#pragma unroll
    for (int p = 0; p < kPlanes; ++p) {
      const float a = inside && in_min ? __ldg(src[p] + at) : 0.0f;
      const float b = inside && in_max ? __ldg(src[p] + at + 1) : 0.0f;
      v[p] = d_c_max * a + d_c_min * b;
    }
  };
  float value1[kPlanes], value2[kPlanes];
  int have = -2;  // the input row of value1; none (rows start at -1)
#pragma unroll
  for (int k = 0; k < kRows; ++k) {
    const int r = r0 + k;
    if (r >= new_rows) return;
    const float r_i = ((float)r + 0.5f) * scale_r - 0.5f;
    const int r_i_min = (int)floorf(r_i);
    const int r_i_max = r_i_min + 1;
    const float d_r_min = r_i - (float)r_i_min;
    const float d_r_max = (float)r_i_max - r_i;
    if (k == 0 || r_i_min != have) {
      if (k > 0 && r_i_min == have + 1) {
#pragma unroll
        for (int p = 0; p < kPlanes; ++p) value1[p] = value2[p];
      } else {
        across(r_i_min, value1);
      }
      across(r_i_max, value2);
      have = r_i_min;
    }
    float v[kPlanes];
#pragma unroll
    for (int p = 0; p < kPlanes; ++p) v[p] = d_r_max * value1[p] + d_r_min * value2[p];
    const size_t o = (size_t)r * new_cols + c;
    if (kDepth) out_depth[o] = v[0];
    if (kNormal) {
      float* n = v + (kDepth ? 1 : 0);
      const float sq = (n[0] * n[0] + n[1] * n[1]) + n[2] * n[2];
      if (sq > 0.f) {
        const float len = sqrtf(sq);
        n[0] = n[0] / len; n[1] = n[1] / len; n[2] = n[2] / len;
      }
#pragma unroll
      for (int p = 0; p < 3; ++p) out_normal[p * out_plane + o] = n[p];
    }
  }
}

int Blocks(int n, int per_block) { return (n + per_block - 1) / per_block; }

template <int kPer>
void LaunchRescale(const float* in, int w, int h, float* tmp, float* out, int ow, int oh, cudaStream_t s) {
  const dim3 blk(kBlockX, kBlockY);
  const float sx = (float)ow / (float)w, sy = (float)oh / (float)h;
  ResampleRowsKernel<kPer><<<dim3(Blocks(ow, kBlockX), Blocks(h, kBlockY * kPer)), blk, 0, s>>>(
      in, w, h, tmp, ow, sx, sx < 1.0f ? 1.0f / sx : 1.0f, std::fmin(sx, 1.0f));
  ResampleColsKernel<kPer><<<dim3(Blocks(ow, kBlockX * kPer), Blocks(oh, kBlockY)), blk, 0, s>>>(
      tmp, ow, h, out, oh, sy, sy < 1.0f ? 1.0f / sy : 1.0f, std::fmin(sy, 1.0f));
}

template <int kRows>
void LaunchResample(const float* depth, const float* normal, int w, int h, float* out_depth, float* out_normal, int ow,
                    int oh, cudaStream_t s) {
  const dim3 blk(kBlockX, kBlockY), grd(Blocks(ow, kBlockX), Blocks(oh, kBlockY * kRows));
  auto kernel = depth && normal ? ResampleMapKernel<true, true, kRows>
                : depth         ? ResampleMapKernel<true, false, kRows>
                                : ResampleMapKernel<false, true, kRows>;
  kernel<<<grd, blk, 0, s>>>(depth, normal, h, w, out_depth, out_normal, oh, ow);
}

int Fail(int code, const char* msg) {
  smvs_internal_set_error(msg);
  return code;
}

}  // namespace

extern "C" {

int smvs_pyramid_level_size(int width, int height, int level, int* out_width, int* out_height, float* factor) {
  if (width <= 0 || height <= 0 || level < 0 || !out_width || !out_height)
    return Fail(SMVS_EINVAL, "smvs_pyramid_level_size: bad arguments");
  // patch_match_controller.cc:4407-4410: 1 / 2^level, but never below 320
  // pixels on the longer side; image.cc:51-52: rounded sizes.
  float f = 1.0f / std::pow(2.0f, (float)level);
  const float max_size = (float)(width > height ? width : height);
  const float min_size = std::min(320.f, max_size);
  f = std::max(f, min_size / max_size);
  *out_width = (int)std::round(width * f);
  *out_height = (int)std::round(height * f);
  if (factor) *factor = f;
  return SMVS_OK;
}

int smvs_rescale_image(const float* in, int width, int height, float* out, int out_width, int out_height,
                       void* scratch, void* stream) {
  if (!in || !out || !scratch || width <= 0 || height <= 0 || out_width <= 0 || out_height <= 0)
    return Fail(SMVS_EINVAL, "smvs_rescale_image: bad arguments");
  cudaStream_t s = (cudaStream_t)stream;
  float* tmp = static_cast<float*>(scratch);  // out_width x height
  if ((size_t)out_width * height < kRescaleFour)
    LaunchRescale<1>(in, width, height, tmp, out, out_width, out_height, s);
  else
    LaunchRescale<4>(in, width, height, tmp, out, out_width, out_height, s);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return Fail(SMVS_ECUDA, cudaGetErrorString(e));
  return SMVS_OK;
}

int smvs_resample_maps(const float* depth, const float* normal, int width, int height, float* out_depth,
                       float* out_normal, int out_width, int out_height, void* stream) {
  if ((!depth && !normal) || (depth && !out_depth) || (normal && !out_normal) || width <= 0 || height <= 0 ||
      out_width <= 0 || out_height <= 0)
    return Fail(SMVS_EINVAL, "smvs_resample_maps: bad arguments");
  cudaStream_t s = (cudaStream_t)stream;
  // Normals that go where the depth map lies wait until it has been read.
  const char *n0 = reinterpret_cast<const char*>(out_normal), *d0 = reinterpret_cast<const char*>(depth);
  if (depth && normal && d0 < n0 + 12 * (size_t)out_width * out_height && n0 < d0 + 4 * (size_t)width * height) {
    const int st = smvs_resample_maps(depth, nullptr, width, height, out_depth, nullptr, out_width, out_height, stream);
    return st ? st
              : smvs_resample_maps(nullptr, normal, width, height, nullptr, out_normal, out_width, out_height, stream);
  }
  // Rows share their input only where the map grows: 1500x1000 to 3000x2000 takes
  // 42 us with four rows a thread, 58 with one; the way back 36 and 30 (cold L2).
  if (out_height <= height)
    LaunchResample<1>(depth, normal, width, height, out_depth, out_normal, out_width, out_height, s);
  else
    LaunchResample<4>(depth, normal, width, height, out_depth, out_normal, out_width, out_height, s);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return Fail(SMVS_ECUDA, cudaGetErrorString(e));
  return SMVS_OK;
}

}  // extern "C"
