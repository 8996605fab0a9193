// Internal layout of pz_model (opaque in the public C ABI) and the
// thread-local error setter shared by the entry points.
#pragma once
#include <cuda_fp16.h>

#include "../../include/prescale.h"
#include "kernels.h"

struct pz_model {
  int family = 0, radius = 0, channels = 0;
  float ar = 0.0f;
  float4* d_lut = nullptr;
  float4* d_lut_ar = nullptr;
  float4* d_lut16 = nullptr;     // the LUTs with every value rounded to FP16
  float4* d_lut_ar16 = nullptr;
  __half* d_lut_h = nullptr;     // the LUT as FP16 texels (fast form), rows padded
  int lut_h_pitch = 0;           // to an even texel count (16-byte texel pairs)
  int lut_rows = 0, lut_pitch = 0;  // keys (ravu-zoom: key * 9 rows); FP32 texels per stored row
  pz::KeyParams kp{};
  int nns = 0, win_w = 0, win_h = 0;
  float* d_wts = nullptr;   // [nns][2][T]
  float* d_cs = nullptr;    // [nns][2]
  float* d_bias = nullptr;  // [nns][2]
  __half* d_wts_h = nullptr;
  __half* d_wts_s = nullptr;  // split operand of the plain FP32 form (null: CUDA cores)
  float split_one = 1.0f;     // the power of two it is scaled by
  bool may_mark = true;       // may its pixels leave the split blend's range?
  int device = 0;
};

namespace pz {
// Record `msg` for pz_last_error() on the calling thread; returns `code`.
int set_error(int code, const char* fmt, ...);

// Device address of the error word the kernels report into (one per device,
// a __device__ variable: nothing is allocated); null if the lookup failed.
// pz_check_device_error reads and clears it.
int* device_error_word();

// pz_run's checks of the options: opts->precision against the plane dtype,
// opts->tile_rows (PZ_OK or PZ_EINVAL with the message set).
int check_opts(const pz_opts* o, int dtype);

// Does the fast form read this model's LUT as FP16 texels?  The lite, 3x and
// zoom programs gather a whole LUT row (or four bilinear texels per block)
// per pixel and are bound by those L1 gathers; FP16 halves them.  The ravu
// lattice reads 5-8 texels per key and keeps FP32, and so does ravu-zoom-ar's
// anti-ringing LUT: most of its values lie below FP16's normal range.
inline bool fast_half_lut(const pz_model* m, int precision) {
  return precision == PZ_PREC_FAST &&
         (m->family == PZ_RAVU_LITE || m->family == PZ_RAVU_3X || m->family == PZ_RAVU_ZOOM);
}

// The LUTs and LUT sampling of a precision form: the mpv form reads the
// FP16-rounded copies and quantises zoom bilinear fractions to 1/256; the
// fast form reads FP16 texels where fast_half_lut says so.
inline void select_lut(const pz_model* m, int precision, RavuArgs* a) {
  const bool mpv = precision == PZ_PREC_MPV;
  a->lut = mpv ? m->d_lut16 : m->d_lut;
  a->lut_ar = mpv ? m->d_lut_ar16 : m->d_lut_ar;
  a->lut_rows = m->lut_rows;
  a->lut_pitch = m->lut_pitch;
  a->lut_frac = mpv ? 256.0f : 0.0f;
  const bool h = fast_half_lut(m, precision);
  a->lut_h = h ? reinterpret_cast<const uint2*>(m->d_lut_h) : nullptr;
  a->lut_h_pitch = m->lut_h_pitch;
  // the host's int11 texture is rgba16f: the mpv form rounds int11 to FP16,
  // the other forms keep it FP32 between the two lattice launches
  a->i11_half = mpv ? 1 : 0;
}

// Tile height of a model's per-frame launches when the caller asks for none,
// the fastest on GB300 at 480p-1080p (1080p, fast form, 4 / 8 / 16 rows:
// ravu-lite-r3 31.3 / 30.0 / 31.3 us, ravu-lite-ar-r4 72.4 / 71.3 / 79.5, ravu-3x-r3
// 44.1 / 43.2 / 45.6, ravu-r2 58.1 / 54.2 / 54.2, ravu-r3 74.9 / 74.6 / 78.6, ravu-r4
// 116.4 / 114.3 / 118.4, ravu-r3-yuv 121.9 / 117.8 / 128.1, ravu-r4-yuv 210.6 /
// 198.0 / 188.7; ravu-zoom at 1.5x, 4 / 8: r2 85.8 / 85.7, r3 FP32 334 / 283).
inline int default_tile_rows(const pz_model* m) {
  if (m->family == PZ_RAVU && m->radius == 4 && m->channels != PZ_LUMA) return 16;
  return m->family == PZ_RAVU_ZOOM && m->radius == 2 ? 4 : 8;
}

// The neurons of an NNEDI3 model, as the doubling passes take them.
inline NnArgs nn_args(const pz_model* m, int* err) {
  NnArgs a{};
  a.nns = m->nns;
  a.win_h = m->win_h;
  a.wts = m->d_wts;
  a.cs = m->d_cs;
  a.bias = m->d_bias;
  a.wts_h = m->d_wts_h;
  a.wts_s = m->d_wts_s;
  a.split_one = m->split_one;
  a.split_unit = 1.0f / m->split_one;
  a.err = err;
  return a;
}

// One doubling pass in the form `precision` asks for.  The fast form runs
// its neurons on the tensor cores in FP16; every other form keeps FP32 values
// and runs them there as two FP16 pieces each.  1080p to 2160p, FP32 planes,
// split against CUDA cores: nns128 8x6 441 against 4919 us, nns16 8x4 176
// against 491 us; 160x90 nns32 8x4 the same (both are the two launches).  The
// error against 64 bits is 0.5-0.65x the CUDA cores' for every nns and window
// with weights that sum to zero, as the files' do (nns128 8x6 at 640x360: 8.5e-8
// against 1.46e-7 relative); with Elliott weights 130 times as large it is 0.75-1.1x
// (largest error 1.8e-6 against 4.3e-7, nns32 8x4), with logits of 60 0.9-1.5x.  Models of other
// shapes, or with weights that the pieces cannot hold, stay on the CUDA cores;
// and so do single pixels of models whose pre-activations may leave the split
// blend's range (may_mark), by a second launch that looks for them.
inline int launch_nnedi3(const pz_model* m, const NnArgs& a, int precision, bool xpass, int dtype, cudaStream_t s) {
  if (nnedi3_tc_supported(a.nns, a.win_h)) {
    if (precision == PZ_PREC_FAST) return launch_nnedi3_tc(a, xpass, dtype, s);
    if (a.wts_s) {
      const int rc = launch_nnedi3_split(a, xpass, dtype, s);
      return rc || !m->may_mark ? rc : launch_nnedi3_marked(a, xpass, dtype, s);
    }
  }
  return launch_nnedi3_simt(a, xpass, dtype, s);
}

// Scratch of a ravu lattice chain: the int11 plane, FP32 [channels][H][W].
inline size_t lattice_scratch_bytes(const pz_model* m, int W, int H) {
  return (size_t)(m->channels == PZ_LUMA ? 1 : 3) * W * H * sizeof(float);
}
}  // namespace pz
