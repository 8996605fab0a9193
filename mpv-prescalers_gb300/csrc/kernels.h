// Host-side launch interface of the prescaler kernels (internal; the public
// C ABI is include/prescale.h).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "common.cuh"

namespace pz {

// Launches `kern`; `after`: its prerequisite is the launch just before it on the
// stream, whose CTAs have all begun when this one's may (pdl_trigger, pdl_wait): its
// CTAs fill the SMs that the other's last wave leaves idle and run up to their wait.
// One after the other / overlapped: ravu-r3 854x480 26.9 / 24.2 us, 1080p 74.6 / 73.9,
// ravu-r3-yuv 720p 60.1 / 57.2, ravu-zoom-r2 720p to 1080p (its phase table first)
// 33.1 / 31.6, nnedi3-nns64-win8x4 FP32 854x480 63.9 / 62.1.
template <class... P, class... A>
void launch_kernel(void (*kern)(P...), dim3 grid, int threads, size_t smem, cudaStream_t s, bool after, const A&... a) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c{};
  c.gridDim = grid;
  c.blockDim = dim3(threads);
  c.dynamicSmemBytes = smem;
  c.stream = s;
  c.attrs = &at;
  c.numAttrs = after ? 1 : 0;
  cudaLaunchKernelEx(&c, kern, a...);  // errors: cudaGetLastError, as for the other launches
}

enum ChMode : int { kLuma = 0, kYuv = 1, kRgb = 2 };

// One RAVU-family dispatch.  Planes are [H][W] with per-plane pitches.
struct RavuArgs {
  const void* in[3];
  int in_pitch[3];
  void* out[3];
  int out_pitch[3];
  int W, H;          // input size
  int OW, OH;        // output size
  int after;         // launched right after its prerequisite (launch_kernel)
  int frames;        // frames of one launch (0 counts as 1; plain loads only), elements apart:
  long long in_frame, out_frame;
  const float4* lut;     // [lut_rows][lut_pitch] texels
  const float4* lut_ar;  // zoom-ar only
  int lut_rows, lut_pitch;
  float ar;
  int32_t* keys;     // optional raw-key output
  int* err;          // device error word (kErr*)
  int staging;       // 0: clamped loads, 1: TMA boxes for interior tiles
  int tile_rows;     // tile height of the per-frame launches: 4, 8 or 16 rows
  float lut_frac;    // zoom LUT bilinear fraction steps (0: exact FP32)
  const uint2* lut_h;  // fast form: the LUT as FP16 texels (4 halves each), or null
  int lut_h_pitch;     // texels per FP16 LUT row (even)
  int box_w, box_h;    // ravu-zoom TMA staging: the box of this launch's tensor maps (texels x rows)
  const float4* ztab;  // ravu-zoom: every key's weights at every phase of the scale (zoom_table_kernel), or null
  FastDiv zpx, zpy;    // phases per axis: out / gcd(in, out)
  FastDiv zx, zy;      // ravu-zoom: 2 * out per axis (d = 0: positions need 64 bits)
  float* i11;          // ravu lattice: int11 plane, FP32 [C][H][W] (scratch)
  int i11_half;        // round int11 to FP16 before storing it (the mpv form)
  KeyParams kp;
};

// One NNEDI3 doubling pass.  `xpass` doubles columns, otherwise rows.
struct NnArgs {
  const void* in;
  int in_pitch;
  void* out;
  int out_pitch;
  int W, H;                 // size of the pass input
  int after;                // launched right after its prerequisite (launch_kernel; tensor cores)
  int frames;               // frames (of one launch: tensor cores; 0 counts as 1), elements apart:
  long long in_frame, out_frame;
  int nns, win_h;           // window is 8 x win_h (double_y orientation)
  const float* wts;         // [nns][2][T]: A row then B row per neuron (FP32)
  const float* cs;          // [nns][2]: column sums of A and B
  const float* bias;        // [nns][2]
  const __half* wts_h;      // FP16 packed weights for the tensor-core kernel
  const __half* wts_s;      // the same as two FP16 pieces (hi, lo), scaled, or null
  float split_one;          // the power of two that wts_s is scaled by
  float split_unit;         // its inverse
  int* err;                 // device error word
};

int launch_lite(const RavuArgs& a, int radius, bool ar, int dtype, cudaStream_t s);
int launch_3x(const RavuArgs& a, int radius, int chmode, int dtype, cudaStream_t s);
int launch_lattice(const RavuArgs& a, int radius, int chmode, int dtype, cudaStream_t s);
int launch_zoom(const RavuArgs& a, int radius, int chmode, bool ar, int dtype, cudaStream_t s);
// The divisors of ravu-zoom's source positions ((2X + 1) W - OW) / (2 OW).
inline void zoom_divisors(RavuArgs* a) {
  const bool fits = (2ll * a->OW + 1) * a->W < 1ll << 31 && (2ll * a->OH + 1) * a->H < 1ll << 31;
  a->zx = fits ? fast_div(2 * a->OW) : FastDiv{0, 0, 0};
  a->zy = fits ? fast_div(2 * a->OH) : FastDiv{0, 0, 0};
}
// ravu-zoom's weight table for a scale of few phases: its bytes (0: too many
// phases for the frame), and the launch that fills a.ztab.
size_t zoom_table_bytes(int radius, bool ar, int keys, int W, int H, int OW, int OH, FastDiv* px, FastDiv* py);
int launch_zoom_table(const RavuArgs& a, int radius, bool ar, cudaStream_t s);
int launch_nnedi3_simt(const NnArgs& a, bool xpass, int dtype, cudaStream_t s);
// The pixels that launch_nnedi3_split, on the same arguments, has marked.
int launch_nnedi3_marked(const NnArgs& a, bool xpass, int dtype, cudaStream_t s);
int launch_nnedi3_tc(const NnArgs& a, bool xpass, int dtype, cudaStream_t s);
int launch_nnedi3_split(const NnArgs& a, bool xpass, int dtype, cudaStream_t s);
bool nnedi3_tc_supported(int nns, int win_h);
// Neurons per chunk of the tensor-core weight operand (split: of the plain FP32
// form): the host stores B chunk-major, NC softmax rows then NC Elliott rows.
int nnedi3_tc_chunk(int nns, int win_h, bool split);

}  // namespace pz
