// Resampling around the hook chain: pz_resample.
//
// Two host steps surround a prescaler in mpv and decide what it shows:
//   * a pass's //!OFFSET (ravu-r3.hook:424 "-0.5 -0.5"; nnedi3-nns16-win8x4.hook:95
//     "0 -0.5" and :185 "-0.5 0") announces a pixel shift of its
//     output, which the host folds into its next scaling pass;
//   * a NATIVE hook (compute/ravu-r2-yuv.hook:15) sees the planes merged at
//     luma size, i.e. subsampled chroma already upscaled by --cscale
//     (README.md:50-56).
// Both are one separable interpolation per plane:
//   out(x, y) = sum_i sum_j k(u - i) k(v - j) in(clamp(i), clamp(j)),
//   u = sx * x + ox,  v = sy * y + oy,
// with texel centres at integer coordinates and clamp-to-edge borders.
// k is the bilinear tent or the Catmull-Rom cubic (Keys' cubic convolution
// kernel with a = -1/2).  resample_kernel computes one output texel per thread
// from its 2x2 or 4x4 input footprint through L1, at any scale; shifts (sx = sy =
// 1, the //!OFFSET correction) go by 4 x 4 blocks (shift_kernel).
#include "../../include/prescale.h"
#include "kernels.h"
#include "model.h"
#include "ravu_tiles.cuh"

namespace pz {
namespace {

// Planes of one size (grid z) through one resampling.
constexpr int kMaxPlanes = 4;
struct ResampleArgs {
  const void* in[kMaxPlanes];
  void* out[kMaxPlanes];
  int in_pitch[kMaxPlanes], out_pitch[kMaxPlanes];
  int in_w, in_h;
  int out_w, out_h;
  float sx, ox, sy, oy;
};

// Catmull-Rom weights of the 4 taps floor(u)-1 .. floor(u)+2 at fraction t.
__device__ __forceinline__ void cubic_weights(float t, float (&w)[4]) {
  const float t2 = t * t, t3 = t2 * t;
  w[0] = 0.5f * (-t3 + 2.0f * t2 - t);
  w[1] = 0.5f * (3.0f * t3 - 5.0f * t2 + 2.0f);
  w[2] = 0.5f * (-3.0f * t3 + 4.0f * t2 + t);
  w[3] = 0.5f * (t3 - t2);
}

__device__ __forceinline__ void st_quad(float* p, const float (&v)[4]) {
  *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
}
__device__ __forceinline__ void st_quad(__half* p, const float (&v)[4]) {
  const __half2 a = __floats2half2_rn(v[0], v[1]), b = __floats2half2_rn(v[2], v[3]);
  *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
}

// The weights of the taps around position u = fmaf(s, x, o), and floor(u).
template <int TAPS>
__device__ __forceinline__ int tap_weights(float s, int x, float o, float (&w)[TAPS]) {
  const float u = fmaf(s, (float)x, o), f = floorf(u);
  if constexpr (TAPS == 2) {
    w[0] = 1.0f - (u - f);
    w[1] = u - f;
  } else {
    cubic_weights(u - f, w);
  }
  return (int)f;
}

template <int TAPS, typename T>
__device__ __forceinline__ float resample_one(const ResampleArgs& a, int x, int y) {
  const T* in = static_cast<const T*>(a.in[blockIdx.z]);
  const int pitch = a.in_pitch[blockIdx.z];
  float wx[TAPS], wy[TAPS];
  const int iu = tap_weights<TAPS>(a.sx, x, a.ox, wx), iv = tap_weights<TAPS>(a.sy, y, a.oy, wy);
  constexpr int K0 = TAPS == 2 ? 0 : -1;
  int cx[TAPS];
#pragma unroll
  for (int i = 0; i < TAPS; i++) cx[i] = clampi(iu + K0 + i, 0, a.in_w - 1);
  float acc = 0.0f;
#pragma unroll
  for (int j = 0; j < TAPS; j++) {
    const T* row = in + (size_t)clampi(iv + K0 + j, 0, a.in_h - 1) * pitch;
    float r = 0.0f;
#pragma unroll
    for (int i = 0; i < TAPS; i++) r += wx[i] * ldp(row + cx[i]);
    acc += wy[j] * r;
  }
  return acc;
}

template <int TAPS, typename T>
__global__ void __launch_bounds__(256) resample_kernel(const __grid_constant__ ResampleArgs a) {
  const int x = blockIdx.x * 32 + (threadIdx.x & 31);
  const int y = blockIdx.y * 8 + (threadIdx.x >> 5);
  if (x >= a.out_w || y >= a.out_h) return;
  stp(static_cast<T*>(a.out[blockIdx.z]) + (size_t)y * a.out_pitch[blockIdx.z] + x, resample_one<TAPS, T>(a, x, y));
}

// Shifts: one thread per 4 x 4 block of outputs.  Neighbouring outputs share
// all but one input column and row, so a block reads TAPS + 3 input rows in
// quads, filters each row once for its 4 columns and adds it to the output
// rows that it reaches: the sums of resample_one in their order, at a sixth of
// its instructions (one texel a thread, 207 instructions a texel, issue-bound at
// 8 % of the copy bandwidth).  OFF: column of the first tap within its quad,
// (floor(ox) + first tap) mod 4, the same for every thread.  A block whose
// positions do not step by whole texels (the rounding of x + ox far from 0) goes
// texel by texel.  3840x2160 FP16, planes in L2 / from memory: Catmull-Rom 20.6 / 28.9
// us (one texel a thread 61.6 / 61.7), bilinear 12.2 / 18.3 (26.8 / 30.9); 2560x1440
// Catmull-Rom 10.6 (28.9).
template <int TAPS, int OFF, typename T>
__global__ void __launch_bounds__(256) shift_kernel(const __grid_constant__ ResampleArgs a) {
  constexpr int K0 = TAPS == 2 ? 0 : -1, QUADS = (OFF + TAPS + 3 + 3) / 4;
  const int X = (blockIdx.x * 32 + (threadIdx.x & 31)) * 4, Y = (blockIdx.y * 8 + (threadIdx.x >> 5)) * 4;
  if (X >= a.out_w || Y >= a.out_h) return;
  const int in_pitch = a.in_pitch[blockIdx.z], out_pitch = a.out_pitch[blockIdx.z];
  T* out = static_cast<T*>(a.out[blockIdx.z]) + (size_t)Y * out_pitch + X;
  const int nx = min(4, a.out_w - X), ny = min(4, a.out_h - Y);
  float wx[4][TAPS], wy[4][TAPS];
  int iu[4], iv[4];
#pragma unroll
  for (int k = 0; k < 4; k++) {
    iu[k] = tap_weights<TAPS>(a.sx, X + k, a.ox, wx[k]);
    iv[k] = tap_weights<TAPS>(a.sy, Y + k, a.oy, wy[k]);
  }
  const int c0 = iu[0] + K0 - OFF;  // a quad's first column
  bool whole = (c0 & 3) == 0;
#pragma unroll
  for (int k = 1; k < 4; k++) whole = whole && iu[k] == iu[0] + k && iv[k] == iv[0] + k;
  if (!whole) {
    for (int j = 0; j < ny; j++)
      for (int i = 0; i < nx; i++) stp(out + (size_t)j * out_pitch + i, resample_one<TAPS, T>(a, X + i, Y + j));
    return;
  }
  const T* in = static_cast<const T*>(a.in[blockIdx.z]);
  const bool aligned = quads_aligned(in, in_pitch);
  float acc[4][4];
#pragma unroll
  for (int j = 0; j < 4; j++)
#pragma unroll
    for (int i = 0; i < 4; i++) acc[j][i] = 0.0f;
#pragma unroll
  for (int row = 0; row < TAPS + 3; row++) {
    const T* src = in + (size_t)clampi(iv[0] + K0 + row, 0, a.in_h - 1) * in_pitch;
    float v[QUADS * 4];
#pragma unroll
    for (int q = 0; q < QUADS; q++) {
      Quad<T> t;
      load_quad(t, src, c0 + 4 * q, a.in_w, aligned);
      const float4 f = t.get();
      v[4 * q] = f.x;
      v[4 * q + 1] = f.y;
      v[4 * q + 2] = f.z;
      v[4 * q + 3] = f.w;
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
      float r = 0.0f;
#pragma unroll
      for (int t = 0; t < TAPS; t++) r += wx[i][t] * v[OFF + i + t];
#pragma unroll
      for (int j = 0; j < 4; j++)
        if (row - j >= 0 && row - j < TAPS) acc[j][i] += wy[j][row - j] * r;
    }
  }
  const bool quads = nx == 4 && quads_aligned(static_cast<const T*>(a.out[blockIdx.z]), out_pitch);
#pragma unroll
  for (int j = 0; j < 4; j++) {
    if (j >= ny) break;
    T* o = out + (size_t)j * out_pitch;
    if (quads) {
      st_quad(o, acc[j]);
    } else {
      for (int i = 0; i < nx; i++) stp(o + i, i == 0 ? acc[j][0] : (i == 1 ? acc[j][1] : (i == 2 ? acc[j][2] : acc[j][3])));
    }
  }
}

template <int TAPS, typename T>
void launch_resample(const ResampleArgs& a, int planes, cudaStream_t s) {
  if (a.sx != 1.0f || a.sy != 1.0f) {
    resample_kernel<TAPS, T><<<dim3((a.out_w + 31) / 32, (a.out_h + 7) / 8, planes), 256, 0, s>>>(a);
    return;
  }
  const dim3 grid((a.out_w + 127) / 128, (a.out_h + 31) / 32, planes);
  switch (((int)floorf(a.ox) + (TAPS == 2 ? 0 : -1)) & 3) {
    case 0: shift_kernel<TAPS, 0, T><<<grid, 256, 0, s>>>(a); break;
    case 1: shift_kernel<TAPS, 1, T><<<grid, 256, 0, s>>>(a); break;
    case 2: shift_kernel<TAPS, 2, T><<<grid, 256, 0, s>>>(a); break;
    default: shift_kernel<TAPS, 3, T><<<grid, 256, 0, s>>>(a);
  }
}

int check_rs_plane(const pz_plane* p, const char* what) {
  if (!p || !p->data) return set_error(PZ_EINVAL, "%s: null plane", what);
  if (p->width <= 0 || p->height <= 0 || p->pitch < p->width)
    return set_error(PZ_EINVAL, "%s: bad size %dx%d pitch %d", what, p->width, p->height, p->pitch);
  if (p->dtype != PZ_F32 && p->dtype != PZ_F16) return set_error(PZ_EINVAL, "%s: unknown dtype %d", what, p->dtype);
  if (reinterpret_cast<uintptr_t>(p->data) % (p->dtype == PZ_F32 ? 4 : 2))
    return set_error(PZ_EINVAL, "%s: misaligned base", what);
  return PZ_OK;
}

}  // namespace
}  // namespace pz

extern "C" int pz_resample(const pz_plane* in, pz_plane* out, float sx, float ox, float sy, float oy, int filter,
                           void* stream) {
  return pz_resample_planes(in, out, 1, sx, ox, sy, oy, filter, stream);
}

extern "C" int pz_resample_planes(const pz_plane* in, pz_plane* out, int n_planes, float sx, float ox, float sy,
                                  float oy, int filter, void* stream) {
  if (n_planes < 1 || n_planes > pz::kMaxPlanes)
    return pz::set_error(PZ_EINVAL, "%d planes: 1 to %d", n_planes, pz::kMaxPlanes);
  pz::ResampleArgs a{};
  for (int c = 0; c < n_planes; c++) {
    int rc;
    if ((rc = pz::check_rs_plane(in ? in + c : nullptr, "in")) || (rc = pz::check_rs_plane(out ? out + c : nullptr, "out")))
      return rc;
    if (in[c].dtype != out[c].dtype) return pz::set_error(PZ_EINVAL, "input and output dtypes differ");
    if (in[c].width != in->width || in[c].height != in->height || out[c].width != out->width ||
        out[c].height != out->height || in[c].dtype != in->dtype)
      return pz::set_error(PZ_EINVAL, "the planes of one call share sizes and dtype");
    a.in[c] = in[c].data;
    a.out[c] = out[c].data;
    a.in_pitch[c] = in[c].pitch;
    a.out_pitch[c] = out[c].pitch;
  }
  if (filter != PZ_FILTER_BILINEAR && filter != PZ_FILTER_CATMULL_ROM)
    return pz::set_error(PZ_EINVAL, "unknown filter %d", filter);
  // every sample position must stay a finite float well inside int range
  const float lim = 1.0e7f;
  const float ux0 = ox, ux1 = sx * (float)(out->width - 1) + ox;
  const float vy0 = oy, vy1 = sy * (float)(out->height - 1) + oy;
  if (!(fabsf(ux0) < lim && fabsf(ux1) < lim && fabsf(vy0) < lim && fabsf(vy1) < lim))
    return pz::set_error(PZ_EINVAL, "sample positions out of range");
  a.in_w = in->width;
  a.in_h = in->height;
  a.out_w = out->width;
  a.out_h = out->height;
  a.sx = sx;
  a.ox = ox;
  a.sy = sy;
  a.oy = oy;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const bool f16 = in->dtype == PZ_F16;
  if (filter == PZ_FILTER_BILINEAR)
    f16 ? pz::launch_resample<2, __half>(a, n_planes, s) : pz::launch_resample<2, float>(a, n_planes, s);
  else
    f16 ? pz::launch_resample<4, __half>(a, n_planes, s) : pz::launch_resample<4, float>(a, n_planes, s);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return pz::set_error(PZ_EIO, "resample launch: %s", cudaGetErrorString(e));
  return PZ_OK;
}
