// Shared device code for the prescaler kernels (sm_103a).
//
// The arithmetic mirrors the reference shaders expression by expression
// where that matters for the key (the quantised LUT row):
//   structure tensor   ravu-lite-r3.hook:48-76, ravu-r3.hook:58-107
//   eigen/key          ravu-lite-r3.hook:77-88, ravu-r3.hook:108-125
// All key math is FP32; see ravu_key for how each threshold test is evaluated.
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace pz {

// Programmatic dependent launch: a kernel that a later one depends on lets that
// one's CTAs begin once all of its own have (pdl_trigger); the later one waits
// before it reads what the first wrote, until the first is complete and its
// stores are visible (pdl_wait; nothing to wait for in any other launch).
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

constexpr float kFltEps = 1.192092896e-7f;   // the shaders' epsilon literal
constexpr float kPi = 3.141592653589793f;    // the shaders' pi literal

// Key quantisation constants of one model (kernel parameter).
struct KeyParams {
  float gw[36];      // Gaussian weights of the gradient points (geometry order)
  float gwf[36];     // gw * c^2 where both stencils of a point have the same scale c
                     // (1 one-sided, 1/2 central, 1/12 four-tap), else gw
  float thr[3];      // strength thresholds (lite, zoom: 3; 3x: 2)
  int n_thr;
  int log2_mode;     // ravu: strength = clamp(floor(log2(l*scale+eps)), 0, max)
  float log2_scale;
  int log2_max;
  float coh0, coh1;  // coherence thresholds
  int n_strength;    // strength levels
  int rows;          // LUT keys (24 * n_strength * 3)
};

// Device-side error word shared by all kernels: first failure wins.
enum : int { kErrNone = 0, kErrTileOverflow = 1, kErrWaitTimeout = 2, kErrQueue = 3 };

// t / d for 0 <= t < 2^31 by a multiplication, with the divisor fixed on the host
// (Granlund and Montgomery, Division by Invariant Integers using Multiplication,
// 1994, figure 4.1: m' = floor(2^32 (2^s - d) / d) + 1, s = ceil(log2 d); their two
// shifts are one, as the sum fits 32 bits for these t).
struct FastDiv {
  uint32_t m, s, d;
  __device__ __forceinline__ uint32_t operator()(uint32_t t) const { return (__umulhi(t, m) + t) >> s; }
};
inline FastDiv fast_div(uint32_t d) {
  FastDiv f{0, 0, d};
  while ((1ull << f.s) < d) f.s++;
  f.m = (uint32_t)(((1ull << 32) * ((1ull << f.s) - d)) / d + 1);
  return f;
}

// ------------------------------------------------------------- plane I/O --
__device__ __forceinline__ float ldp(const float* p) { return __ldg(p); }
__device__ __forceinline__ float ldp(const __half* p) {
  return __half2float(__ushort_as_half(__ldg(reinterpret_cast<const unsigned short*>(p))));
}
__device__ __forceinline__ void stp(float* p, float v) { *p = v; }
__device__ __forceinline__ void stp(__half* p, float v) { *p = __float2half_rn(v); }
// two horizontally adjacent pixels (p must be 2-element aligned)
__device__ __forceinline__ void stp2(float* p, float a, float b) {
  *reinterpret_cast<float2*>(p) = make_float2(a, b);
}
__device__ __forceinline__ void stp2(__half* p, float a, float b) {
  *reinterpret_cast<__half2*>(p) = __floats2half2_rn(a, b);
}

__device__ __forceinline__ int clampi(int v, int lo, int hi) { return v < lo ? lo : (v > hi ? hi : v); }
__device__ __forceinline__ float clampf(float v, float lo, float hi) { return fminf(fmaxf(v, lo), hi); }
// GLSL mod(): x - y * floor(x / y)
__device__ __forceinline__ float gl_mod(float x, float y) { return x - y * floorf(x / y); }

// --------------------------------------------------- structure tensor -----
// Gradient stencil at grid position p along one axis of an N-tap window:
// one-sided at the border, central /2 inside, and (FOUR: ravu, ravu-zoom)
// (-s[p+2] + 8 s[p+1] - 8 s[p-1] + s[p-2]) / 12 where both exist.
// stencil_kind: 0 one-sided, 1 central, 2 four-tap (also used on the host
// to scale the weights of KeyParams::gwf).
__host__ __device__ constexpr int stencil_kind(int n, bool four, int p) {
  return (p == 0 || p == n - 1) ? 0 : ((four && p >= 2 && p <= n - 3) ? 2 : 1);
}

// The stencil without its scale (1, 1/2, 1/12).
template <int N, bool FOUR, class G>
__device__ __forceinline__ float deriv_unscaled(const G& s, int p) {
  if (p == 0) return s(1) - s(0);
  if (p == N - 1) return s(N - 1) - s(N - 2);
  if (FOUR && p >= 2 && p <= N - 3) return -s(p + 2) + 8.0f * s(p + 1) - 8.0f * s(p - 1) + s(p - 2);
  return s(p + 1) - s(p - 1);
}

template <int N, bool FOUR, class G>
__device__ __forceinline__ float deriv(const G& s, int p) {
  if (p == 0) return s(1) - s(0);
  if (p == N - 1) return s(N - 1) - s(N - 2);
  if (FOUR && p >= 2 && p <= N - 3)
    return (-s(p + 2) + 8.0f * s(p + 1) - 8.0f * s(p - 1) + s(p - 2)) * (1.0f / 12.0f);
  return (s(p + 1) - s(p - 1)) * 0.5f;
}

// Gaussian-weighted sum of (gx^2, gx gy, gy^2) over the gradient points:
// the whole window when N <= 4, else the window minus a one-tap border.
// `get(kx, ky)` returns the key input at window grid (kx, ky).  a and d
// accumulate as one FP32x2 pair, a += gx (gx w), d += gy (gy w), b += (gx w) gy
// (three instructions per point instead of six), and where
// both stencils of a point share one scale c the scale moves into the weight
// (gwf = gw c^2: the unscaled differences are used).  Each term then rounds
// a few times differently from the shader's gx * gx * w, far inside the
// key's FP32 boundary budget.
template <int N, bool FOUR, class Get>
__device__ __forceinline__ void structure_tensor(const Get& get, const KeyParams& kp, float& a,
                                                 float& b, float& d) {
  constexpr int P0 = N <= 4 ? 0 : 1;
  constexpr int P1 = N <= 4 ? N : N - 1;
  float2 ad = make_float2(0.0f, 0.0f);
  b = 0.0f;
  int i = 0;
#pragma unroll
  for (int px = P0; px < P1; px++) {
#pragma unroll
    for (int py = P0; py < P1; py++) {
      const bool fold = stencil_kind(N, FOUR, px) == stencil_kind(N, FOUR, py);
      auto sx = [&](int q) { return get(q, py); };
      auto sy = [&](int q) { return get(px, q); };
      const float gx = fold ? deriv_unscaled<N, FOUR>(sx, px) : deriv<N, FOUR>(sx, px);
      const float gy = fold ? deriv_unscaled<N, FOUR>(sy, py) : deriv<N, FOUR>(sy, py);
      const float w = fold ? kp.gwf[i] : kp.gw[i];
      i++;
      const float2 g2 = make_float2(gx, gy);
      const float2 gw2 = __fmul2_rn(g2, make_float2(w, w));
      ad = __ffma2_rn(g2, gw2, ad);
      b = fmaf(gw2.x, gy, b);
    }
  }
  a = ad.x;
  d = ad.y;
}

// The structure tensors of E windows of one lattice that a thread evaluates
// together: window e covers grid (X, Y) in [Off::x(e), +N) x [Off::y(e), +N),
// and `get(X, Y)` returns the key input at lattice point (X, Y).  The points run
// in lattice order, so that a derivative that several windows share (the same
// stencil at the same point) is formed once; each window's own sums see their
// terms in the order and (PACKED) rounding of structure_tensor; else each lane
// rounds as the shader's a += gx * gx * w.
template <int N, bool FOUR, bool PACKED, int E, class Off, class Get>
__device__ __forceinline__ void structure_tensors(const Get& get, const KeyParams& kp, float (&a)[E], float (&b)[E],
                                                  float (&d)[E]) {
  constexpr int P0 = N <= 4 ? 0 : 1;
  constexpr int P1 = N <= 4 ? N : N - 1;
  int x0 = Off::x(0), x1 = x0, y0 = Off::y(0), y1 = y0;
#pragma unroll
  for (int e = 1; e < E; e++) {
    x0 = Off::x(e) < x0 ? Off::x(e) : x0;
    x1 = Off::x(e) > x1 ? Off::x(e) : x1;
    y0 = Off::y(e) < y0 ? Off::y(e) : y0;
    y1 = Off::y(e) > y1 ? Off::y(e) : y1;
  }
  float2 ad[E];
#pragma unroll
  for (int e = 0; e < E; e++) {
    ad[e] = make_float2(0.0f, 0.0f);
    a[e] = b[e] = d[e] = 0.0f;
  }
#pragma unroll
  for (int X = x0 + P0; X < x1 + P1; X++) {
#pragma unroll
    for (int Y = y0 + P0; Y < y1 + P1; Y++) {
#pragma unroll
      for (int e = 0; e < E; e++) {
        const int px = X - Off::x(e), py = Y - Off::y(e);
        if (px < P0 || px >= P1 || py < P0 || py >= P1) continue;
        const int i = (px - P0) * (P1 - P0) + py - P0;
        const bool fold = PACKED && stencil_kind(N, FOUR, px) == stencil_kind(N, FOUR, py);
        auto sx = [&](int q) { return get(q + Off::x(e), Y); };
        auto sy = [&](int q) { return get(X, q + Off::y(e)); };
        const float gx = fold ? deriv_unscaled<N, FOUR>(sx, px) : deriv<N, FOUR>(sx, px);
        const float gy = fold ? deriv_unscaled<N, FOUR>(sy, py) : deriv<N, FOUR>(sy, py);
        const float w = fold ? kp.gwf[i] : kp.gw[i];
        if constexpr (PACKED) {
          const float gxw = __fmul_rn(gx, w), gyw = __fmul_rn(gy, w);
          ad[e] = __ffma2_rn(make_float2(gx, gy), make_float2(gxw, gyw), ad[e]);
          b[e] = fmaf(gxw, gy, b[e]);
        } else {
          a[e] += gx * gx * w;
          b[e] += gx * gy * w;
          d[e] += gy * gy * w;
        }
      }
    }
  }
  if constexpr (PACKED) {
#pragma unroll
    for (int e = 0; e < E; e++) {
      a[e] = ad[e].x;
      d[e] = ad[e].y;
    }
  }
}

__device__ __forceinline__ float sqrt_approx(float x) {
  float r;
  // NaN for x < 0, as in GLSL.  Subnormal arguments count as zero: they mean
  // eigenvalues below 2^-102, where every gate of ravu_key is closed anyway
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// floor(24 * theta / pi) with theta = mod(atan(y, x) + pi, pi) in [0, pi),
// without the arctangent: the direction is folded into [0, pi/4] (opposite
// signs: theta above pi/2, turned back by pi/2; then a mirror about the
// diagonal) and the sector boundaries k*pi/24 at or below it are counted in
// three comparisons of y with tan(k*pi/24) * x (k = 4; then 2 or 6; then 1, 3 or
// 5).  Only directions within FP32 rounding of a boundary can land in the
// neighbouring sector (the oracle's boundary keys); NaN components fail every
// comparison: sector 0, or 12 for x < 0.
__device__ __forceinline__ int angle_sector(float x, float y) {
  const bool turn = ((x < 0.0f) != (y < 0.0f)) && y != 0.0f;
  const float u = fabsf(turn ? y : x), v = fabsf(turn ? x : y);
  const bool mirror = v > u;
  const float c = mirror ? v : u, s = mirror ? u : v;
  const bool p = s >= 0.577350269f * c;
  const bool q = s >= (p ? 1.0f : 0.267949192f) * c;
  const bool r = s >= (p ? 0.767326988f : (q ? 0.414213562f : 0.131652498f)) * c;
  int k = (p ? 4 : 0) + (q ? (p ? 1 : 2) : 0) + (r ? 1 : 0);
  if (mirror) k = 11 - k;
  return turn ? k + 12 : k;
}

// Eigen analysis + quantisation -> raw key (not clamped to the LUT).
// ravu-lite-r3.hook:77-88 (strength thresholds), ravu-r3.hook:121-125 (log2).
//
// The quantised outputs equal the shader's; only the way each threshold test
// is evaluated changes, so results can differ only where a quantity lies
// within FP32 rounding of a threshold (the oracle's boundary keys):
//   * angle: the sector by comparisons with tan(k*pi/24) (angle_sector)
//     instead of floor(atan(.) * 24 / pi);
//   * coherence: mu >= c  <=>  (sqrtL1 - sqrtL2) >= c * (sqrtL1 + sqrtL2),
//     no division; NaN (L2 < 0) still fails every test -> 0, and the
//     sqrtL1 + sqrtL2 < eps gate still forces 0;
//   * log2 strength: floor(log2(v)) is the unbiased exponent of v (> 0).
__device__ __forceinline__ int ravu_key(float a, float b, float d, const KeyParams& kp) {
  float T = a + d, D = a * d - b * b;
  float delta = sqrt_approx(fmaxf(T * T * 0.25f - D, 0.0f));
  float L1 = T * 0.5f + delta, L2 = T * 0.5f - delta;
  float sqrtL1 = sqrt_approx(L1), sqrtL2 = sqrt_approx(L2);
  const int angle = fabsf(b) < kFltEps ? 0 : angle_sector(b, L1 - a);
  float lambda = sqrtL1;
  int strength;
  if (kp.log2_mode) {
    const float v = lambda * kp.log2_scale + kFltEps;
    strength = clampi((__float_as_int(v) >> 23) - 127, 0, kp.log2_max);
  } else if (kp.n_thr == 3) {
    strength = lambda >= kp.thr[1] ? (lambda >= kp.thr[2] ? 3 : 2) : (lambda >= kp.thr[0] ? 1 : 0);
  } else {
    strength = lambda >= kp.thr[1] ? 2 : (lambda >= kp.thr[0] ? 1 : 0);
  }
  const float ssum = sqrtL1 + sqrtL2, sdif = sqrtL1 - sqrtL2;
  int coherence = 0;
  if (!(ssum < kFltEps)) coherence = sdif >= kp.coh1 * ssum ? 2 : (sdif >= kp.coh0 * ssum ? 1 : 0);
  return (angle * kp.n_strength + strength) * 3 + coherence;
}

// Anti-ringing powers of one value as an FP32x2 pair: (0.1 + v)^32 and
// (1.1 - v)^32 by five squarings (ravu-lite-ar-r3.hook:91-98); each lane rounds
// as a scalar FMUL would.
__device__ __forceinline__ float2 ar_pow32(float v) {
  float2 q = __ffma2_rn(make_float2(v, v), make_float2(1.0f, -1.0f), make_float2(0.1f, 1.1f));
#pragma unroll
  for (int i = 0; i < 5; i++) q = __fmul2_rn(q, q);
  return q;
}

// The clamp of one output: mix(res, clamp(res, lo, hi), s).  The shaders bound
// res by lo = 1.1 - sum g l^33 / sum g l^32 and hi = sum g h^33 / sum g h^32 -
// 0.1 with h = 0.1 + v, l = 1.1 - v; both are means of v itself, weighted by
// g l^32 and g h^32, and are taken as such: sums = (sum g h^32, sum g l^32),
// means = (sum g h^32 v, sum g l^32 v).
// The quotients are approximate (__fdividef, about 2 ulp, the precision a
// shader's division has): they only move the clamp bounds, by < 3e-7.  Both
// operands are scaled by 2^24 first, so that a subnormal denominator
// (positive weights summing below ~1e-6) still has a finite reciprocal; for
// every other denominator the scaling changes no bit of the quotient.
__device__ __forceinline__ float ar_quot(float n, float d) {
  return __fdividef(n * 16777216.0f, d * 16777216.0f);
}
__device__ __forceinline__ float ar_finish(float res, float2 sums, float2 means, float s) {
  const float hib = ar_quot(means.x, sums.x), lob = ar_quot(means.y, sums.y);
  const float c = fminf(fmaxf(res, lob), hib);
  return res * (1.0f - s) + c * s;
}

// Rec.709 luma of an RGB sample (ravu-r2-rgb.hook:21 color_primary).
__device__ __forceinline__ float rgb_luma(float r, float g, float b) {
  return r * 0.2126f + g * 0.7152f + b * 0.0722f;
}

}  // namespace pz
