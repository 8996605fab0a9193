// C ABI of libprescale.so (declared in include/prescale.h): model upload,
// argument checking, dispatch to the kernels, thread-local error messages.
#include <cuda.h>

#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <new>
#include <string>
#include <vector>

#include "../../include/prescale.h"
#include "async.cuh"
#include "kernels.h"
#include "model.h"
#include "ravu_tiles.cuh"

namespace {

thread_local std::string g_err;

int fail(int code, const char* fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof buf, fmt, ap);
  va_end(ap);
  g_err = buf;
  return code;
}

int cuda_fail(cudaError_t e, const char* what) {
  return fail(PZ_EIO, "%s: %s", what, cudaGetErrorString(e));
}

template <typename T>
int upload(T** dst, const void* src, size_t bytes) {
  cudaError_t e = cudaMalloc(reinterpret_cast<void**>(dst), bytes);
  if (e != cudaSuccess) return cuda_fail(e, "cudaMalloc");
  e = cudaMemcpy(*dst, src, bytes, cudaMemcpyHostToDevice);
  if (e != cudaSuccess) return cuda_fail(e, "cudaMemcpy");
  return PZ_OK;
}

// The device-side error word every kernel reports into (first failure wins,
// see kErr* in common.cuh).  A file-scope __device__ variable: nothing is
// allocated for it, so the first launch on a device may come inside stream
// capture.  Host code looks its device address up once per device.
__device__ int g_device_err;

constexpr int kMaxDevices = 64;
std::mutex g_err_mu;
int* g_err_words[kMaxDevices];  // device address of g_device_err, per device

size_t dtype_size(int dt) { return dt == PZ_F32 ? 4 : 2; }

// A bounded wait that nothing ever completes: the mbarrier is initialised for
// one arrival and never arrived at, no copy or MMA is issued.  The wait gives
// up after `limit_ns` and reports kErrWaitTimeout like every kernel does.
__global__ void wait_selftest_kernel(int* err, unsigned long long limit_ns) {
  __shared__ __align__(8) unsigned long long mbar;
  const uint32_t mb = pz::smem_u32(&mbar);
  if (threadIdx.x == 0) pz::mbar_init(mb, 1);
  __syncthreads();
  if (!__syncthreads_and(pz::mbar_wait_bounded(mb, 0u, limit_ns)) && threadIdx.x == 0)
    atomicCAS(err, 0, pz::kErrWaitTimeout);
}

size_t zoom_table_size(const pz_model* m, int W, int H, int OW, int OH, pz::FastDiv* px, pz::FastDiv* py) {
  return pz::zoom_table_bytes(m->radius, m->ar != 0.0f, m->lut_rows / 9, W, H, OW, OH, px, py);
}

// `pairs`: the plane is written with 2-wide vector stores, so its base and
// pitch must keep every even column 2-element aligned.
int check_plane(const pz_plane& p, const char* what, int idx, bool pairs) {
  if (!p.data) return fail(PZ_EINVAL, "%s[%d]: null data", what, idx);
  if (p.width <= 0 || p.height <= 0) return fail(PZ_EINVAL, "%s[%d]: bad size %dx%d", what, idx, p.width, p.height);
  if (p.pitch < p.width) return fail(PZ_EINVAL, "%s[%d]: pitch %d < width %d", what, idx, p.pitch, p.width);
  if (p.dtype != PZ_F32 && p.dtype != PZ_F16) return fail(PZ_EINVAL, "%s[%d]: unknown dtype %d", what, idx, p.dtype);
  const size_t es = dtype_size(p.dtype);
  if ((reinterpret_cast<uintptr_t>(p.data) % es) != 0)
    return fail(PZ_EINVAL, "%s[%d]: data not aligned to its element size", what, idx);
  if (pairs && ((reinterpret_cast<uintptr_t>(p.data) % (2 * es)) != 0 || (p.pitch % 2) != 0))
    return fail(PZ_EINVAL, "%s[%d]: this output is written in pixel pairs; base and pitch must be 2-element aligned",
                what, idx);
  return PZ_OK;
}

constexpr double kLog2e = 1.4426950408889634;

// The tensor-core operands B [2*nns][KP] of an NNEDI3 model, chunk-major:
// chunk c of NC neurons (nnedi3_tc_chunk) is NC softmax-branch rows followed by
// NC Elliott-branch rows.  Row = [weights (T taps), sum of the
// weights, the bias in pieces, 0...]; against A rows [x_hat, mean*invstd, 1, 1,
// 1, 0...] the MMA yields the whole pre-activation <x,w>*invstd + b.  Softmax
// rows are scaled by log2(e) so the epilogue takes exp2 directly.  Stored as
// no-swizzle K-major core matrices (8 rows x 8 halves; K-neighbours 64 halves
// apart, 8-row groups 8*KP apart).
//   wts_h  FP16 values (the fast form)
//   wts_s  two FP16 pieces of each value, [hi][lo]: hi = fp16(v), lo =
//          fp16(v - hi), v scaled by the power of two that brings the largest
//          magnitude to 2^13..2^14.  Every value down to 2^-16 of the largest
//          then keeps 22 bits or more, and a smaller one an absolute error of
//          2^-39 of the largest.  Not made (the CUDA cores run the model)
//          when a value is not finite or the power lies outside 2^-8..2^30,
//          so that the blend's product of two denominators, of at most 2^31
//          each, and its reciprocal stay within FP32's normal range.  Whether its
//          numerators may leave FP32's range (nn_tc_kernel marks such pixels) is
//          bounded here: a window's x_hat has norm sqrt(T) and no mean, and its
//          mean term is at most 60000, so that a pre-activation is at most
//          sqrt(T) |w - mean(w)| + 60000 |sum w| + |bias|.
//
// One block per row (the softmax or Elliott branch of a neuron), one thread per
// element; `up`: the power of two, 0: no pieces.  On the device, where its three
// conversions a value cost nothing: nns256 8x6 loads in 0.19 ms, in 0.70 with
// them on the host.
__global__ void operand_kernel(const float* wts, const float* bias, int T, int KP, int nch, int ncs, double up,
                               __half* h, __half* s) {
  const int r = blockIdx.x, t = threadIdx.x;
  const size_t piece = (size_t)gridDim.x * KP;
  const float* w = wts + (size_t)r * T;
  const double scale = r % 2 == 0 ? kLog2e : 1.0;
  double x = 0.0;
  if (t < T) x = w[t];
  if (t == T)
    for (int i = 0; i < T; i++) x += w[i];
  if (t > T && t <= T + 3) x = bias[r];
  x *= scale;
  auto at = [&](int nc) {
    const int k = r / 2, row = k / nc * 2 * nc + r % 2 * nc + k % nc;
    return (size_t)(row >> 3) * 8 * KP + (t >> 3) * 64 + (row & 7) * 8 + (t & 7);
  };
  // piece j of v: the FP16 value of what the pieces before it leave
  auto take = [](double v, int j) {
    __half p = __float2half_rn((float)v);
    for (; j > 0; j--) {
      v -= (double)__half2float(p);
      p = __float2half_rn((float)v);
    }
    return p;
  };
  const int j = t > T ? t - T - 1 : 0;  // a bias has an element for each of its pieces
  h[at(nch)] = j < 2 ? take(x, j) : __float2half_rn(0.0f);
  if (up > 0.0) {
    s[at(ncs)] = j < 3 ? take(x * up, j) : __float2half_rn(0.0f);
    s[piece + at(ncs)] = t <= T ? take(x * up, 1) : __float2half_rn(0.0f);
  }
}

// The operands from the FP32 weights and biases that the model already holds on
// the device (w, bias: on the host).
int upload_operands(pz_model* m, const std::vector<float>& w, const std::vector<float>& bias) {
  const int n = m->nns, T = m->win_w * m->win_h;
  const int KP = (T + 4 + 15) / 16 * 16;  // taps, mean term, three bias pieces, padded to a K step
  double top = 0.0, most[2] = {0.0, 0.0};  // largest pre-activation per branch (softmax: log2 units)
  bool finite = true;
  for (int r = 0; r < 2 * n; r++) {
    const float* row = &w[(size_t)r * T];
    const double scale = r % 2 == 0 ? kLog2e : 1.0;
    double sum = 0.0, squares = 0.0, largest = std::fabs(bias[r]);
    for (int t = 0; t < T; t++) {
      const double x = row[t];
      sum += x;
      squares += x * x;
      largest = std::max(largest, std::fabs(x));
    }
    largest = std::max(largest, std::fabs(sum));
    const double norm = std::sqrt(std::max(squares - sum * sum / T, 0.0));
    most[r % 2] = std::max(most[r % 2], (std::sqrt((double)T) * norm + 60000.0 * std::fabs(sum) + std::fabs(bias[r])) * scale);
    finite = finite && std::isfinite(squares + sum + bias[r]);
    top = std::max(top, largest * scale);
  }
  const int exp2 = top > 0.0 && finite ? 13 - std::ilogb(top) : 0;
  const bool split = finite && exp2 >= -8 && exp2 <= 30;
  const size_t piece = (size_t)2 * n * KP * sizeof(__half);
  cudaError_t e = cudaMalloc(reinterpret_cast<void**>(&m->d_wts_h), piece);
  if (e == cudaSuccess && split) e = cudaMalloc(reinterpret_cast<void**>(&m->d_wts_s), 2 * piece);
  if (e != cudaSuccess) return cuda_fail(e, "cudaMalloc");
  operand_kernel<<<2 * n, KP>>>(m->d_wts, m->d_bias, T, KP, pz::nnedi3_tc_chunk(n, m->win_h, false),
                                pz::nnedi3_tc_chunk(n, m->win_h, true), split ? std::ldexp(1.0, exp2) : 0.0, m->d_wts_h,
                                m->d_wts_s);
  if ((e = cudaGetLastError()) != cudaSuccess || (e = cudaStreamSynchronize(nullptr)) != cudaSuccess)
    return cuda_fail(e, "NNEDI3 operands");
  if (split) {
    m->split_one = (float)std::ldexp(1.0, exp2);
    // e s (1 + |s|) at the square of the scale, over all neurons, with room for
    // the roundings; and one e of at least 2^-89
    const double top2 = most[0] + 2.0 * (exp2 + std::log2(1.0 + most[1])) + std::log2((double)n);
    m->may_mark = !(top2 < 126.0 && most[0] < 89.0);
  }
  return PZ_OK;
}

}  // namespace

namespace pz {
// Tensor map of one plane for 2-D TMA boxes of box_w x box_h texels.  False
// when the plane cannot be described (base or row pitch not 16-byte aligned,
// plane smaller than a box, driver entry point missing): callers then use
// clamped loads.
bool encode_plane_map(CUtensorMap* map, const void* base, int W, int H, int pitch, int dtype, int box_w,
                      int box_h) {
  typedef CUresult (*EncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                               const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                               CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
  static EncodeFn encode = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      encode = reinterpret_cast<EncodeFn>(fn);
  });
  const size_t es = dtype == PZ_F32 ? 4 : 2;
  if (!encode || W < box_w || H < box_h || box_w > 256 || box_h > 256) return false;
  if (reinterpret_cast<uintptr_t>(base) % 16 || ((size_t)pitch * es) % 16) return false;
  const cuuint64_t dims[2] = {(cuuint64_t)W, (cuuint64_t)H};
  const cuuint64_t strides[1] = {(cuuint64_t)pitch * es};
  const cuuint32_t box[2] = {(cuuint32_t)box_w, (cuuint32_t)box_h};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult r = encode(map, dtype == PZ_F32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16,
                            2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                            CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

int set_error(int code, const char* fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof buf, fmt, ap);
  va_end(ap);
  g_err = buf;
  return code;
}

int* device_error_word() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return nullptr;
  std::lock_guard<std::mutex> lk(g_err_mu);
  if (!g_err_words[dev]) {
    void* w = nullptr;
    if (cudaGetSymbolAddress(&w, g_device_err) != cudaSuccess) return nullptr;
    g_err_words[dev] = static_cast<int*>(w);
  }
  return g_err_words[dev];
}

int check_opts(const pz_opts* o, int dtype) {
  if (o && (o->precision < PZ_PREC_FP32 || o->precision > PZ_PREC_MPV))
    return set_error(PZ_EINVAL, "unknown precision %d", o->precision);
  if (o && o->precision == PZ_PREC_MPV && dtype != PZ_F16)
    return set_error(PZ_EINVAL, "the mpv form takes FP16 planes (the host's textures are rgba16f)");
  if (o && (o->staging < 0 || o->staging > 1))
    return set_error(PZ_EINVAL, "staging %d: 0 (clamped loads) or 1 (TMA boxes)", o->staging);
  if (o && o->tile_rows != 0 && o->tile_rows != 4 && o->tile_rows != 8 && o->tile_rows != 16)
    return set_error(PZ_EINVAL, "tile_rows %d: 0 (default), 4, 8 or 16", o->tile_rows);
  return PZ_OK;
}
}  // namespace pz

extern "C" {

int pz_version(void) { return PZ_ABI_VERSION; }

const char* pz_last_error(void) { return g_err.c_str(); }

int pz_model_create(const pz_model_desc* d, pz_model** out) {
  if (!d || !out) return fail(PZ_EINVAL, "null argument");
  *out = nullptr;
  pz_model* m = new (std::nothrow) pz_model();
  if (!m) return fail(PZ_ENOMEM, "host allocation failed");
  cudaGetDevice(&m->device);
  m->family = d->family;
  m->radius = d->radius;
  m->channels = d->channels;
  m->ar = d->ar_strength;
  int rc = PZ_OK;
  if (d->family == PZ_NNEDI3) {
    if (d->nns <= 0 || d->nns % 8 || d->win_w != 8 || (d->win_h != 4 && d->win_h != 6) || !d->weights_a ||
        !d->weights_b || !d->bias_a || !d->bias_b) {
      delete m;
      return fail(PZ_EINVAL, "bad NNEDI3 description (nns %d, window %dx%d)", d->nns, d->win_w, d->win_h);
    }
    m->nns = d->nns;
    m->win_w = d->win_w;
    m->win_h = d->win_h;
    const int T = d->win_w * d->win_h, n = d->nns;
    std::vector<float> w((size_t)n * 2 * T), cs((size_t)n * 2), bias((size_t)n * 2);
    for (int k = 0; k < n; k++) {
      double sa = 0, sb = 0;
      for (int t = 0; t < T; t++) {
        float a = d->weights_a[(size_t)t * n + k], b = d->weights_b[(size_t)t * n + k];
        w[((size_t)k * 2 + 0) * T + t] = a;
        w[((size_t)k * 2 + 1) * T + t] = b;
        sa += a;
        sb += b;
      }
      cs[2 * k] = (float)sa;
      cs[2 * k + 1] = (float)sb;
      bias[2 * k] = d->bias_a[k];
      bias[2 * k + 1] = d->bias_b[k];
    }
    if ((rc = upload(&m->d_wts, w.data(), w.size() * 4)) || (rc = upload(&m->d_cs, cs.data(), cs.size() * 4)) ||
        (rc = upload(&m->d_bias, bias.data(), bias.size() * 4)) ||
        (pz::nnedi3_tc_supported(n, d->win_h) && (rc = upload_operands(m, w, bias)))) {
      pz_model_destroy(m);
      return rc;
    }
    *out = m;
    return PZ_OK;
  }
  if (d->family < PZ_RAVU_LITE || d->family > PZ_RAVU_3X) {
    delete m;
    return fail(PZ_EINVAL, "unknown family %d", d->family);
  }
  const int maxr = d->family == PZ_RAVU_ZOOM ? 3 : 4;
  if (d->radius < 2 || d->radius > maxr) {
    delete m;
    return fail(PZ_ENOTSUP, "radius %d not supported for family %d", d->radius, d->family);
  }
  if (d->channels < PZ_LUMA || d->channels > PZ_RGB || (d->family == PZ_RAVU_LITE && d->channels != PZ_LUMA)) {
    delete m;
    return fail(PZ_EINVAL, "bad channels %d for family %d", d->channels, d->family);
  }
  if (!d->lut || d->lut_rows <= 0 || d->lut_cols <= 0 || !d->grad_weights || d->n_grad <= 0 || d->n_grad > 36) {
    delete m;
    return fail(PZ_EINVAL, "bad LUT / gradient description");
  }
  const int n = d->family == PZ_RAVU_LITE || d->family == PZ_RAVU_3X ? 2 * d->radius - 1 : 2 * d->radius;
  const int pts = n <= 4 ? n * n : (n - 2) * (n - 2);
  if (d->n_grad != pts) {
    delete m;
    return fail(PZ_EINVAL, "%d gradient weights, window needs %d", d->n_grad, pts);
  }
  pz::KeyParams& kp = m->kp;
  {
    // gradient points in kernel order (px outer, py inner); where both
    // stencils of a point share one scale c, gwf = gw c^2
    const bool four = d->family == PZ_RAVU || d->family == PZ_RAVU_ZOOM;
    const int p0 = n <= 4 ? 0 : 1, p1 = n <= 4 ? n : n - 1;
    const double scale2[3] = {1.0, 0.25, 1.0 / 144.0};  // c^2 per stencil kind
    int i = 0;
    for (int px = p0; px < p1; px++)
      for (int py = p0; py < p1; py++, i++) {
        const int kx = pz::stencil_kind(n, four, px), ky = pz::stencil_kind(n, four, py);
        kp.gw[i] = (float)d->grad_weights[i];
        kp.gwf[i] = kx == ky ? (float)((double)kp.gw[i] * scale2[kx]) : kp.gw[i];
      }
  }
  kp.log2_mode = d->strength_log2;
  if (kp.log2_mode) {
    kp.log2_scale = d->strength_scale;
    kp.log2_max = d->strength_max;
    kp.n_strength = d->strength_max + 1;
  } else {
    if (d->n_strength_thr != 2 && d->n_strength_thr != 3) {
      delete m;
      return fail(PZ_EINVAL, "need 2 or 3 strength thresholds");
    }
    kp.n_thr = d->n_strength_thr;
    for (int i = 0; i < kp.n_thr; i++) kp.thr[i] = d->strength_thr[i];
    kp.n_strength = kp.n_thr + 1;
  }
  kp.coh0 = d->coherence_thr[0];
  kp.coh1 = d->coherence_thr[1];
  kp.rows = 24 * kp.n_strength * 3;
  const int want_rows = d->family == PZ_RAVU_ZOOM ? kp.rows * 9 : kp.rows;
  if (d->lut_rows != want_rows) {
    delete m;
    return fail(PZ_EINVAL, "LUT has %d rows, key layout needs %d", d->lut_rows, want_rows);
  }
  const int S = n * n;
  int need_cols = 0;
  switch (d->family) {
    case PZ_RAVU_LITE: need_cols = (S + 1) / 2; break;
    case PZ_RAVU: need_cols = (S / 2 + 3) / 4; break;
    case PZ_RAVU_3X: need_cols = 2 * ((S + 1) / 2); break;
    case PZ_RAVU_ZOOM: need_cols = 9 * ((S / 2 + 3) / 4); break;
  }
  if (d->lut_cols != need_cols) {
    delete m;
    return fail(PZ_EINVAL, "LUT has %d columns, radius %d needs %d", d->lut_cols, d->radius, need_cols);
  }
  if (d->family == PZ_RAVU_ZOOM && (d->ar_strength != 0.0f) != (d->lut_ar != nullptr)) {
    delete m;
    return fail(PZ_EINVAL, "ravu-zoom anti-ringing needs the _ar LUT and a strength");
  }
  m->lut_rows = d->lut_rows;
  // ravu-zoom's tables are held by LUT point (zoom_texel_at, ravu_tiles.cuh),
  // the others by rows.  ravu's FP32 rows are padded to an odd texel count: a warp
  // gathers texel q of 32 rows at once, and the file's 8 texels a row at r4 (128
  // bytes) put all of them in one of L1's 8 16-byte banks, its 2 at r2 in 4 (the
  // others' counts are odd): 1080p ravu-r4 131 us, 209 unpadded; ravu-r4-yuv 204,
  // 279; ravu-r2 58.1, 58.4.  FP16 rows are padded to an even count,
  // so that texel pairs are 16-byte loads.
  const bool zoom = d->family == PZ_RAVU_ZOOM;
  const int nb = need_cols / 9;
  m->lut_h_pitch = zoom ? 9 * ((nb + 1) & ~1) : (d->lut_cols + 1) & ~1;
  m->lut_pitch = d->family == PZ_RAVU ? d->lut_cols | 1 : d->lut_cols;
  const size_t rows = d->lut_rows, cols = d->lut_cols, bytes = rows * m->lut_pitch * 16;
  // FP32 rows as they are stored: the file's own where the pitch is (ravu-zoom's
  // FP32 order is the file's)
  std::vector<float> room;
  auto padded = [&](const float* src) {
    if ((size_t)m->lut_pitch == cols) return src;
    room.assign(bytes / 4, 0.0f);
    for (size_t y = 0; y < rows; y++) std::memcpy(&room[y * m->lut_pitch * 4], src + y * cols * 4, cols * 16);
    return (const float*)room.data();
  };
  // every value rounded to FP16 (round to nearest even), as FP32 and as halves
  std::vector<float> rounded(rows * cols * 4);
  std::vector<__half> halves(rows * cols * 4);
  auto round16 = [&](const float* src) {
    for (size_t i = 0; i < halves.size(); i++) {
      halves[i] = __float2half_rn(src[i]);
      rounded[i] = __half2float(halves[i]);
    }
    return (const float*)rounded.data();
  };
  if ((rc = upload(&m->d_lut, padded(d->lut), bytes)) || (rc = upload(&m->d_lut16, padded(round16(d->lut)), bytes))) {
    pz_model_destroy(m);
    return rc;
  }
  std::vector<__half> luth(rows * m->lut_h_pitch * 4, __float2half_rn(0.0f));
  for (size_t y = 0; y < rows; y++) {
    const __half* src = &halves[y * cols * 4];
    if (!zoom) {
      std::memcpy(&luth[y * m->lut_h_pitch * 4], src, cols * 8);
      continue;
    }
    for (uint32_t t = 0, c = 0; c < cols; t++)
      for (uint32_t x = 0; x < 9; x++, c++) {
        const size_t at = d->radius == 2 ? pz::zoom_texel_at<2, true>(y, x, t) : pz::zoom_texel_at<3, true>(y, x, t);
        std::memcpy(&luth[at * 4], src + c * 4, 8);
      }
  }
  if ((rc = upload(&m->d_lut_h, luth.data(), luth.size() * 2)) ||
      (d->lut_ar && ((rc = upload(&m->d_lut_ar, padded(d->lut_ar), bytes)) ||
                     (rc = upload(&m->d_lut_ar16, padded(round16(d->lut_ar)), bytes))))) {
    pz_model_destroy(m);
    return rc;
  }
  *out = m;
  return PZ_OK;
}

void pz_model_destroy(pz_model* m) {
  if (!m) return;
  cudaFree(m->d_lut);
  cudaFree(m->d_lut_ar);
  cudaFree(m->d_lut16);
  cudaFree(m->d_lut_ar16);
  cudaFree(m->d_lut_h);
  cudaFree(m->d_wts);
  cudaFree(m->d_cs);
  cudaFree(m->d_bias);
  cudaFree(m->d_wts_h);
  cudaFree(m->d_wts_s);
  delete m;
}

static int nn_axes(const pz_opts* o) {
  int ax = o ? o->nnedi3_axes : 0;
  return ax == 0 ? 3 : ax;
}

int pz_query(const pz_model* m, int in_w, int in_h, int dtype, const pz_opts* o, pz_query_result* r) {
  if (!m || !r) return fail(PZ_EINVAL, "null argument");
  if (in_w <= 0 || in_h <= 0) return fail(PZ_EINVAL, "bad input size %dx%d", in_w, in_h);
  if (dtype != PZ_F32 && dtype != PZ_F16) return fail(PZ_EINVAL, "unknown dtype %d", dtype);
  r->family = m->family;
  r->n_planes = m->channels == PZ_LUMA ? 1 : 3;
  r->scratch_bytes = 0;
  switch (m->family) {
    case PZ_RAVU_3X:
      r->out_width = 3 * in_w;
      r->out_height = 3 * in_h;
      break;
    case PZ_RAVU_ZOOM:
      if (!o || o->out_width <= in_w || o->out_height <= in_h)
        return fail(PZ_EINVAL, "ravu-zoom needs opts->out_width/out_height above the input size");
      r->out_width = o->out_width;
      r->out_height = o->out_height;
      break;
    case PZ_NNEDI3: {
      const int ax = nn_axes(o);
      r->out_width = (ax & 2) ? 2 * in_w : in_w;
      r->out_height = (ax & 1) ? 2 * in_h : in_h;
      if (ax == 3) r->scratch_bytes = (size_t)2 * in_h * in_w * dtype_size(dtype);
      break;
    }
    default:
      r->out_width = 2 * in_w;
      r->out_height = 2 * in_h;
      if (m->family == PZ_RAVU) r->scratch_bytes = pz::lattice_scratch_bytes(m, in_w, in_h);
  }
  return PZ_OK;
}

size_t pz_scratch_bytes(const pz_model* m, const pz_plane* in, const pz_opts* o) {
  if (!m || !in) return 0;
  if (m->family == PZ_RAVU) return pz::lattice_scratch_bytes(m, in->width, in->height);
  if (m->family != PZ_NNEDI3 || nn_axes(o) != 3) return 0;
  return (size_t)2 * in->height * in->width * dtype_size(in->dtype);
}

size_t pz_scratch_wanted(const pz_model* m, int in_w, int in_h, int dtype, const pz_opts* o) {
  pz_query_result q;
  if (pz_query(m, in_w, in_h, dtype, o, &q)) return 0;
  if (m->family != PZ_RAVU_ZOOM || o->staging) return q.scratch_bytes;
  pz::FastDiv px, py;
  return zoom_table_size(m, in_w, in_h, q.out_width, q.out_height, &px, &py);
}

// ravu-zoom's phase table (ravu_zoom.cu) and a call's scratch.
enum ZoomTable {
  kNoTable,      // the scratch is not to be written by a ravu-zoom
  kMakeTable,    // it takes the table, if there is room
  kTableFilled,  // a call before on this stream, with the same sizes and options, has left the table there
};

// pz_run on `frames` frames whose planes lie in_frame / out_frame elements apart
// (more than one: scratch for each given, plain loads, no keys).
static int run_frame(const pz_model* m, const pz_plane* in, int n_in, pz_plane* out, int n_out, const pz_opts* o,
                     void* stream, ZoomTable table, int frames = 1, long long in_frame = 0, long long out_frame = 0) {
  if (!m || !in || !out) return fail(PZ_EINVAL, "null argument");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int C = m->channels == PZ_LUMA ? 1 : 3;
  if (n_in != C || n_out != C) return fail(PZ_EINVAL, "model needs %d planes, got %d in / %d out", C, n_in, n_out);
  int rc;
  const bool pairs = m->family == PZ_RAVU_LITE || m->family == PZ_RAVU || (m->family == PZ_NNEDI3 && (nn_axes(o) & 2));
  for (int c = 0; c < C; c++) {
    if ((rc = check_plane(in[c], "in", c, false)) || (rc = check_plane(out[c], "out", c, pairs))) return rc;
    if (in[c].width != in[0].width || in[c].height != in[0].height)
      return fail(PZ_EINVAL, "input planes differ in size");
    if (in[c].dtype != in[0].dtype || out[c].dtype != in[0].dtype)
      return fail(PZ_EINVAL, "all planes must share one dtype");
    if (out[c].width != out[0].width || out[c].height != out[0].height)
      return fail(PZ_EINVAL, "output planes differ in size");
  }
  const int W = in[0].width, H = in[0].height, dt = in[0].dtype;
  if ((rc = pz::check_opts(o, dt))) return rc;
  int* err = pz::device_error_word();
  if (!err) return fail(PZ_EIO, "device error word: cudaGetSymbolAddress failed");
  int OW = 2 * W, OH = 2 * H;
  if (m->family == PZ_RAVU_3X) {
    OW = 3 * W;
    OH = 3 * H;
  } else if (m->family == PZ_RAVU_ZOOM) {
    if (!o) return fail(PZ_EINVAL, "ravu-zoom needs opts->out_width/out_height");
    OW = o->out_width;
    OH = o->out_height;
    if (OW <= W || OH <= H)
      return fail(PZ_EINVAL, "ravu-zoom upscales only (//!WHEN in < out): %dx%d -> %dx%d", W, H, OW, OH);
  } else if (m->family == PZ_NNEDI3) {
    const int ax = nn_axes(o);
    OW = (ax & 2) ? 2 * W : W;
    OH = (ax & 1) ? 2 * H : H;
  }
  if (out[0].width != OW || out[0].height != OH)
    return fail(PZ_EINVAL, "output must be %dx%d, got %dx%d", OW, OH, out[0].width, out[0].height);

  if (m->family == PZ_NNEDI3) {
    const int ax = nn_axes(o);
    const int precision = o ? o->precision : PZ_PREC_FP32;
    pz::NnArgs a = pz::nn_args(m, err);
    void* tmp = nullptr;
    bool own_tmp = false;
    if (ax == 3) {
      const size_t need = (size_t)2 * H * W * dtype_size(dt);
      if (o && o->scratch) {
        if (o->scratch_bytes < need) return fail(PZ_EINVAL, "scratch %zu bytes < %zu needed", o->scratch_bytes, need);
        tmp = o->scratch;
      } else {
        cudaError_t e = cudaMallocAsync(&tmp, need, s);
        if (e != cudaSuccess) return cuda_fail(e, "cudaMallocAsync(scratch)");
        own_tmp = true;
      }
    }
    auto pass = [&](bool xpass, const void* src, int sw, int sh, int spitch, long long sframe, void* dst, int dpitch,
                    long long dframe) {
      a.in = src;
      a.in_pitch = spitch;
      a.out = dst;
      a.out_pitch = dpitch;
      a.W = sw;
      a.H = sh;
      a.frames = frames;
      a.in_frame = sframe;
      a.out_frame = dframe;
      a.after = src == tmp && tmp;
      return pz::launch_nnedi3(m, a, precision, xpass, dt, s);
    };
    rc = 0;
    if (ax == 3) {
      const long long doubled = 2LL * H * W;
      rc = pass(false, in[0].data, W, H, in[0].pitch, in_frame, tmp, W, doubled);
      if (!rc) rc = pass(true, tmp, W, 2 * H, W, doubled, out[0].data, out[0].pitch, out_frame);
    } else {
      rc = pass(ax != 1, in[0].data, W, H, in[0].pitch, in_frame, out[0].data, out[0].pitch, out_frame);
    }
    if (own_tmp) cudaFreeAsync(tmp, s);
    if (rc) return fail(rc, "NNEDI3 launch configuration not supported");
  } else {
    pz::RavuArgs a{};
    for (int c = 0; c < C; c++) {
      a.in[c] = in[c].data;
      a.in_pitch[c] = in[c].pitch;
      a.out[c] = out[c].data;
      a.out_pitch[c] = out[c].pitch;
    }
    a.W = W;
    a.H = H;
    a.OW = OW;
    a.OH = OH;
    a.frames = frames;
    a.in_frame = in_frame;
    a.out_frame = out_frame;
    pz::select_lut(m, o ? o->precision : PZ_PREC_FP32, &a);
    a.ar = m->ar;
    a.keys = o ? o->keys : nullptr;
    a.err = err;
    a.staging = o ? o->staging : 0;
    a.tile_rows = o && o->tile_rows ? o->tile_rows : pz::default_tile_rows(m);
    a.kp = m->kp;
    bool own_i11 = false;
    if (m->family == PZ_RAVU) {  // the int11 plane between the two lattice launches
      const size_t need = pz::lattice_scratch_bytes(m, W, H);
      if (o && o->scratch) {
        if (o->scratch_bytes < need) return fail(PZ_EINVAL, "scratch %zu bytes < %zu needed", o->scratch_bytes, need);
        if (reinterpret_cast<uintptr_t>(o->scratch) % 4) return fail(PZ_EINVAL, "scratch not 4-byte aligned");
        a.i11 = static_cast<float*>(o->scratch);
      } else {
        void* tmp = nullptr;
        cudaError_t e = cudaMallocAsync(&tmp, need, s);
        if (e != cudaSuccess) return cuda_fail(e, "cudaMallocAsync(scratch)");
        a.i11 = static_cast<float*>(tmp);
        own_i11 = true;
      }
    }
    switch (m->family) {
      case PZ_RAVU_LITE: rc = pz::launch_lite(a, m->radius, m->ar != 0.0f, dt, s); break;
      case PZ_RAVU_3X: rc = pz::launch_3x(a, m->radius, m->channels, dt, s); break;
      case PZ_RAVU: rc = pz::launch_lattice(a, m->radius, m->channels, dt, s); break;
      case PZ_RAVU_ZOOM:
        pz::zoom_divisors(&a);
        // with scratch for it, the weights of a scale of few phases are formed once
        if (table != kNoTable && o->scratch && !a.staging && reinterpret_cast<uintptr_t>(o->scratch) % 16 == 0) {
          const size_t need = zoom_table_size(m, W, H, OW, OH, &a.zpx, &a.zpy);
          if (need && o->scratch_bytes >= need) {
            if (!o->tile_rows) a.tile_rows = 4;
            a.ztab = static_cast<const float4*>(o->scratch);
            if (table == kMakeTable) pz::launch_zoom_table(a, m->radius, m->ar != 0.0f, s);
            a.after = table == kMakeTable;
          }
        }
        rc = pz::launch_zoom(a, m->radius, m->channels, m->ar != 0.0f, dt, s); break;
      default: rc = PZ_EINVAL;
    }
    if (own_i11) cudaFreeAsync(a.i11, s);
    if (rc) return fail(rc, "no kernel for family %d radius %d", m->family, m->radius);
  }
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "kernel launch");
  return PZ_OK;
}

int pz_run(const pz_model* m, const pz_plane* in, int n_in, pz_plane* out, int n_out, const pz_opts* o, void* stream) {
  return run_frame(m, in, n_in, out, n_out, o, stream, kNoTable);
}

int pz_run_with_scratch(const pz_model* m, const pz_plane* in, int n_in, pz_plane* out, int n_out, const pz_opts* opts,
                        void* scratch, size_t scratch_bytes, void* stream) {
  pz_opts o{};
  if (opts) o = *opts;
  o.scratch = scratch;
  o.scratch_bytes = scratch ? scratch_bytes : 0;
  return run_frame(m, in, n_in, out, n_out, &o, stream, kMakeTable);
}

int pz_run_frames(const pz_model* m, const void* in, long long in_frame, long long in_plane, int in_pitch, void* out,
                  long long out_frame, long long out_plane, int out_pitch, int n_frames, int width, int height,
                  int dtype, const pz_opts* opts, void* scratch, size_t scratch_bytes, void* stream) {
  if (n_frames <= 0) return fail(PZ_EINVAL, "n_frames %d", n_frames);
  if (n_frames > 1 && opts && opts->keys) return fail(PZ_EINVAL, "opts->keys holds the keys of one frame, not of %d", n_frames);
  pz_query_result q;
  if (const int rc = pz_query(m, width, height, dtype, opts, &q)) return rc;
  if (!in || !out) return fail(PZ_EINVAL, "null planes");
  pz_opts o{};
  if (opts) o = *opts;
  if (!scratch) scratch_bytes = 0;  // no room, whatever the caller counted
  o.scratch = scratch;
  o.scratch_bytes = scratch_bytes;
  const long long es = (long long)dtype_size(dtype);
  // all frames in one launch per pass (at most 1024: the tile numbers of one
  // launch stay far below 2^31, its grid within bounds) where each has scratch of its own
  const bool together = !o.staging && out_frame % 2 == 0 && q.scratch_bytes * (size_t)n_frames <= scratch_bytes;
  const int step = together ? 1024 : 1;
  for (int f = 0; f < n_frames; f += step) {
    pz_plane pin[3], pout[3];
    for (int c = 0; c < q.n_planes; c++) {
      char* i = static_cast<char*>(const_cast<void*>(in)) + (f * in_frame + c * in_plane) * es;
      char* d = static_cast<char*>(out) + (f * out_frame + c * out_plane) * es;
      pin[c] = {i, width, height, in_pitch, dtype};
      pout[c] = {d, q.out_width, q.out_height, out_pitch, dtype};
    }
    const int n = n_frames - f < step ? n_frames - f : step;
    if (const int rc = run_frame(m, pin, q.n_planes, pout, q.n_planes, &o, stream, f > 0 ? kTableFilled : kMakeTable, n,
                                 in_frame, out_frame))
      return rc;
  }
  return PZ_OK;
}

int pz_check_device_error(void* cuda_stream) {
  cudaStream_t s = static_cast<cudaStream_t>(cuda_stream);
  int* w = pz::device_error_word();
  if (!w) return fail(PZ_EIO, "device error word: cudaGetSymbolAddress failed");
  cudaError_t e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return cuda_fail(e, "cudaStreamSynchronize");
  int code = 0;
  e = cudaMemcpy(&code, w, sizeof(int), cudaMemcpyDeviceToHost);
  if (e != cudaSuccess) return cuda_fail(e, "reading the device error word");
  if (code == pz::kErrNone) return PZ_OK;
  const int zero = 0;
  e = cudaMemcpy(w, &zero, sizeof(int), cudaMemcpyHostToDevice);
  if (e != cudaSuccess) return cuda_fail(e, "clearing the device error word");
  switch (code) {
    case pz::kErrWaitTimeout:
      return fail(PZ_ETIMEDOUT, "a bounded device-side wait ran out; the tiles of that launch were not written");
    case pz::kErrTileOverflow:
      return fail(PZ_EIO, "a ravu-zoom tile needed more input than its staging area (downscale?)");
    default:
      return fail(PZ_EIO, "device error code %d", code);
  }
}

int pz_selftest_wait(long long limit_ns, void* cuda_stream) {
  if (limit_ns < 0) return fail(PZ_EINVAL, "negative wait limit");
  int* w = pz::device_error_word();
  if (!w) return fail(PZ_EIO, "device error word: cudaGetSymbolAddress failed");
  wait_selftest_kernel<<<1, 32, 0, static_cast<cudaStream_t>(cuda_stream)>>>(w, (unsigned long long)limit_ns);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "kernel launch");
  return PZ_OK;
}

}  // extern "C"
