// RAVU tile programs: one CTA computes one tile of 32 x TR pixels.
//
// Each program is a struct with the shared-memory bytes it needs and a
// device `run(p, x0, y0, smem)` that stages the tile (plus its radius halo)
// and computes it.  The per-model kernels (ravu_lite.cu, ravu_lattice.cu,
// ravu_zoom.cu) launch one CTA per tile; the persistent batch kernel
// (batch.cu) feeds many programs of many frames to the same CTAs.
//
// References (per program):
//   LiteTile    compute/ravu-lite-ar-r3.hook:15-171, ravu-lite-r3.hook:15-131
//   ThreeXTile  compute/ravu-3x-r2.hook:15-115
//   Int11Tile   ravu-r3.hook:15-146 (compute/ravu-r3.hook:15-154)
//   LatticeTile ravu-r3.hook:148-437 (compute/ravu-r3.hook:155-430)
//   ZoomTile    ravu-zoom-r2.hook:15-139, compute/ravu-zoom-ar-r2-rgb.hook:15-238
//
// Input tiles are 32 x TR input pixels (zoom: output pixels), TR = 4, 8 or 16
// rows (a template argument of every program; 8 is the reference's own
// workgroup height, compute/ravu-lite-r3.hook:22); thread t handles column
// t % 32 of row t / 32 (zoom; the others: of the P rows from P * (t / 32)).  Out-of-range reads replicate the edge texel (the mpv
// texture border mode).
#pragma once
#include <cstddef>
#include <cstring>

#include "async.cuh"
#include "kernels.h"

namespace pz {

// Tile width in pixels (one warp per tile row); persistent batches run tiles
// of kBatchTileRows rows.
constexpr int kTileW = 32, kBatchTileRows = 8;

// Plane c of frame f.
template <typename T>
__device__ __forceinline__ const T* plane_in(const RavuArgs& p, int c, int f) {
  return static_cast<const T*>(p.in[c]) + f * p.in_frame;
}
template <typename T>
__device__ __forceinline__ T* plane_out(const RavuArgs& p, int c, int f) {
  return static_cast<T*>(p.out[c]) + f * p.out_frame;
}

__host__ __device__ constexpr int cabs(int v) { return v < 0 ? -v : v; }

// The window tiles of the frame-tile programs: 40 columns starting 4 left of
// the tile's own 32, which hold every window up to radius 4 and keep groups of
// 4 columns aligned in the plane (x0 - 4 is a multiple of 4) and in shared
// memory.  Staging moves such quads: one 8- or 16-byte load and one 16-byte
// shared store for 4 texels, where one texel at a time took as many address
// and clamp instructions for each (ravu-r3 at 8-row
// tiles 93.7 to 86.5 us, ravu-lite-ar-r3 64.4 to 56.3 us at 1080p).
// Quads across the frame's left or right edge, and planes whose base or pitch
// is not a multiple of a quad, go texel by texel with clamped columns.
constexpr int kLead = 4, kTilePitch = kTileW + 8;

template <typename T>
struct Quad;
template <>
struct Quad<float> {
  float4 v;
  __device__ __forceinline__ void load(const float* p) { v = __ldg(reinterpret_cast<const float4*>(p)); }
  __device__ __forceinline__ void load_shared(const float* p) { v = *reinterpret_cast<const float4*>(p); }
  __device__ __forceinline__ void load1(const float* p, int a, int b, int c, int d) {
    v = make_float4(__ldg(p + a), __ldg(p + b), __ldg(p + c), __ldg(p + d));
  }
  __device__ __forceinline__ float4 get() const { return v; }
};
template <>
struct Quad<__half> {
  uint2 v;
  __device__ __forceinline__ void load(const __half* p) { v = __ldg(reinterpret_cast<const uint2*>(p)); }
  __device__ __forceinline__ void load_shared(const __half* p) { v = *reinterpret_cast<const uint2*>(p); }
  __device__ __forceinline__ void load1(const __half* p, int a, int b, int c, int d) {
    const unsigned short* q = reinterpret_cast<const unsigned short*>(p);
    v.x = __ldg(q + a) | (uint32_t)__ldg(q + b) << 16;
    v.y = __ldg(q + c) | (uint32_t)__ldg(q + d) << 16;
  }
  __device__ __forceinline__ float4 get() const {
    const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&v.x));
    const float2 b = __half22float2(*reinterpret_cast<const __half2*>(&v.y));
    return make_float4(a.x, a.y, b.x, b.y);
  }
};

// FP32 texels that the launch before may still be writing when this one begins
// (pdl_wait): read with plain loads, not as data constant for the kernel.
struct FreshFloat {
  float v;
};
template <>
struct Quad<FreshFloat> : Quad<float> {
  __device__ __forceinline__ void load(const FreshFloat* p) { v = *reinterpret_cast<const float4*>(p); }
  __device__ __forceinline__ void load1(const FreshFloat* p, int a, int b, int c, int d) {
    v = make_float4(p[a].v, p[b].v, p[c].v, p[d].v);
  }
};

// May a plane be read in quads (at columns that are multiples of 4)?
template <typename T>
__device__ __forceinline__ bool quads_aligned(const T* in, int pitch) {
  return ((reinterpret_cast<uintptr_t>(in) | (uintptr_t)pitch * sizeof(T)) % (4 * sizeof(T))) == 0;
}
// Columns gx .. gx+3 of a row (gx a multiple of 4), replicated past its ends.
template <typename T>
__device__ __forceinline__ void load_quad(Quad<T>& q, const T* row, int gx, int W, bool aligned) {
  if (aligned && gx >= 0 && gx + 3 < W) q.load(row + gx);
  else q.load1(row, clampi(gx, 0, W - 1), clampi(gx + 1, 0, W - 1), clampi(gx + 2, 0, W - 1), clampi(gx + 3, 0, W - 1));
}

// One plane's window tile, rows y0 .. y0+TH-1 and columns x0-4 .. x0+35, in two
// steps, so that the loads of all planes are in flight before the first store.
template <int TH, int NT, typename T>
struct QuadStage {
  static constexpr int kQuads = kTilePitch / 4 * TH, IT = (kQuads + NT - 1) / NT;
  Quad<T> q[IT];
  __device__ __forceinline__ void load(const T* in, int pitch, int W, int H, int x0, int y0) {
    const bool aligned = quads_aligned(in, pitch);
#pragma unroll
    for (int k = 0; k < IT; k++) {
      const int i = threadIdx.x + k * NT;
      if (kQuads % NT == 0 || i < kQuads)
        load_quad(q[k], in + (size_t)clampi(y0 + i / (kTilePitch / 4), 0, H - 1) * pitch,
                  x0 - kLead + i % (kTilePitch / 4) * 4, W, aligned);
    }
  }
  // the same from a box in shared memory whose rows hold bw texels
  __device__ __forceinline__ void load_box(const T* box, int bw) {
    each([&](int k, int i) { q[k].load_shared(box + i / (kTilePitch / 4) * bw + i % (kTilePitch / 4) * 4); });
  }
  template <class F>
  __device__ __forceinline__ void each(const F& f) const {  // f(k, quad number)
#pragma unroll
    for (int k = 0; k < IT; k++)
      if (kQuads % NT == 0 || (int)threadIdx.x + k * NT < kQuads) f(k, threadIdx.x + k * NT);
  }
};

// The window tiles of C planes (`tile`, plane after plane; CM == kRgb: the
// Rec.709 luma, the key input, as one more).
template <int CM, int TH, int NT, typename T>
struct TileStage {
  static constexpr int C = CM == kLuma ? 1 : 3;
  QuadStage<TH, NT, T> s[C];
  template <class In>
  __device__ __forceinline__ void load(const In& in, int W, int H, int x0, int y0) {  // in(c, &pitch): plane c
#pragma unroll
    for (int c = 0; c < C; c++) {
      int pitch;
      const T* base = in(c, pitch);
      s[c].load(base, pitch, W, H, x0, y0);
    }
  }
  // POW: beside the values of a luma tile, `pow` gets every texel's
  // anti-ringing powers
  template <bool POW = false>
  __device__ __forceinline__ void store(float* tile, float4* pow = nullptr) const {
    float4* t4 = reinterpret_cast<float4*>(tile);
    s[0].each([&](int k, int i) {
      float4 v[C];
#pragma unroll
      for (int c = 0; c < C; c++) {
        v[c] = s[c].q[k].get();
        t4[c * (kTilePitch / 4 * TH) + i] = v[c];
      }
      if constexpr (CM == kRgb)
        t4[C * (kTilePitch / 4 * TH) + i] =
            make_float4(rgb_luma(v[0].x, v[1].x, v[2].x), rgb_luma(v[0].y, v[1].y, v[2].y),
                        rgb_luma(v[0].z, v[1].z, v[2].z), rgb_luma(v[0].w, v[1].w, v[2].w));
      if constexpr (POW) {
        const float2 a = ar_pow32(v[0].x), b = ar_pow32(v[0].y), c = ar_pow32(v[0].z), d = ar_pow32(v[0].w);
        pow[2 * i] = make_float4(a.x, a.y, b.x, b.y);
        pow[2 * i + 1] = make_float4(c.x, c.y, d.x, d.y);
      }
    });
  }
};

// ---------------------------------------------------------- TMA staging ---
// Interior tiles (window fully inside the plane) can be staged by TMA: one
// 2-D box per plane lands in shared memory, then one pass converts it to the
// float tile the programs read.  Border tiles keep the clamped loads above,
// because TMA fills out-of-range texels with zeros, not the edge value.  The
// box starts at the tile origin rounded down to 8 columns, so its x
// coordinate is 16-byte aligned for FP32 and FP16 planes.
struct TmaMaps {
  CUtensorMap map[3];
};

struct TmaCtx {
  const CUtensorMap* map;  // one per plane (kernel parameter or global memory); null: clamped loads
  uint32_t mbar;           // shared mbarrier (count 1)
  unsigned char* raw;      // landing area, 128-byte aligned
  uint32_t phase;          // parity of the mbarrier's next completion (flips per TMA-staged tile)
  int dead;                // a wait timed out: this CTA stages by clamped loads from now on
};

template <int TW>
__host__ __device__ constexpr int tma_box_w() {
  return (TW + 7 + 7) & ~7;  // up to 7 lead columns from rounding the start down
}
template <int TW, int TH, typename T>
__host__ __device__ constexpr uint32_t tma_plane_bytes() {
  return ((uint32_t)tma_box_w<TW>() * TH * sizeof(T) + 127u) & ~127u;
}

__device__ __forceinline__ float lds_f(const float* p) { return *p; }
__device__ __forceinline__ float lds_f(const __half* p) { return __half2float(*p); }

// A bw x bh box per plane at (bx, by) (bx a multiple of 8) into the landing
// area (plane stride pb bytes), issued by thread 0.
template <int CM, typename T>
__device__ __forceinline__ void tma_issue_box(TmaCtx* t, int bx, int by, int bw, int bh, uint32_t pb) {
  constexpr int C = CM == kLuma ? 1 : 3;
  if (threadIdx.x == 0) {
    mbar_arrive_expect_tx(t->mbar, (uint32_t)C * bw * bh * sizeof(T));
#pragma unroll
    for (int c = 0; c < C; c++) tma_load_2d(t->raw + c * pb, &t->map[c], bx, by, t->mbar);
  }
}
// Wait for the boxes.  False when the copy did not complete within the wait
// bound (error word set, the tile abandoned and TMA off for the rest of the
// CTA).  The outcome is made uniform across the CTA, so every thread takes the
// same path through the tile's barriers.
__device__ __forceinline__ bool tma_wait_box(const RavuArgs& p, TmaCtx* t) {
  if (!__syncthreads_and(mbar_wait_bounded(t->mbar, t->phase))) {
    if (threadIdx.x == 0 && p.err) atomicCAS(p.err, 0, kErrWaitTimeout);
    t->dead = 1;
    return false;
  }
  t->phase ^= 1u;
  return true;
}

// A CTA whose TMA wait timed out may still have that copy in flight into its
// landing area: before the CTA exits, thread 0 waits (bounded again) for the
// outstanding phase, so the copy never lands in shared memory that another
// CTA owns.  Nothing else touches the landing area or the mbarrier once the
// CTA is marked dead.
__device__ __forceinline__ void tma_drain(const TmaCtx* t) {
  if (t && t->dead && threadIdx.x == 0) (void)mbar_wait_bounded(t->mbar, t->phase);
}

// Stage the window tile of the frame whose own columns start at x0 (rows y0 ..
// y0+TH-1): interior tiles from a TMA box per plane where the launch has maps,
// the others by quads; `also` (its load, then its store) is more staging whose
// loads overlap with the tile's.  Returns false only when a TMA wait timed out
// (the tile is abandoned).
struct NoStage {
  __device__ __forceinline__ void load() {}
  __device__ __forceinline__ void store() {}
};
template <int CM, int TH, int NT, typename T, bool POW = false, class Also = NoStage>
__device__ __forceinline__ bool stage_frame(const RavuArgs& p, TmaCtx* t, int f, int x0, int y0, float* tile,
                                            Also&& also = NoStage(), float4* pow = nullptr) {
  TileStage<CM, TH, NT, T> st;
  constexpr int C = CM == kLuma ? 1 : 3, BW = tma_box_w<kTilePitch>();
  const int wx = x0 - kLead;
  if (t && t->map && !t->dead && wx >= 0 && y0 >= 0 && wx + kTilePitch <= p.W && y0 + TH <= p.H) {
    constexpr uint32_t pb = tma_plane_bytes<kTilePitch, TH, T>();
    const int bx = wx & ~7;
    tma_issue_box<CM, T>(t, bx, y0, BW, TH, pb);
    also.load();
    if (!tma_wait_box(p, t)) return false;
    // x0 is a multiple of 32, so the window starts 4 columns into the box: a
    // quad's place in shared memory
#pragma unroll
    for (int c = 0; c < C; c++)
      st.s[c].load_box(reinterpret_cast<const T*>(t->raw + c * pb) + (wx - bx), BW);
  } else {
    st.load([&](int c, int& pitch) { pitch = p.in_pitch[c]; return plane_in<T>(p, c, f); }, p.W, p.H, x0, y0);
    also.load();
  }
  st.template store<POW>(tile, pow);
  also.store();
  return true;
}

// Two adjacent FP32 texels i, i+1 (i even, row pitch even) as one 32-byte load.
__device__ __forceinline__ void lut_pair_f32(const float4* f, size_t i, float4& a, float4& b) {
  asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
      : "l"(f + i));
}

// Two adjacent FP16 texels i, i+1 (i even) as one 16-byte load.
__device__ __forceinline__ void lut_pair_h16(const uint2* h, size_t i, float4& a, float4& b) {
  const uint4 q = __ldg(reinterpret_cast<const uint4*>(h + i));
  const float2 a01 = __half22float2(*reinterpret_cast<const __half2*>(&q.x));
  const float2 a23 = __half22float2(*reinterpret_cast<const __half2*>(&q.y));
  const float2 b01 = __half22float2(*reinterpret_cast<const __half2*>(&q.z));
  const float2 b23 = __half22float2(*reinterpret_cast<const __half2*>(&q.w));
  a = make_float4(a01.x, a01.y, a23.x, a23.y);
  b = make_float4(b01.x, b01.y, b23.x, b23.y);
}

// Windows of a thread's P pixels, one below the other.
struct OffDown {
  __host__ __device__ static constexpr int x(int) { return 0; }
  __host__ __device__ static constexpr int y(int e) { return e; }
};

// ------------------------------------------------------------ ravu-lite ---
// Does lite LUT column c take part in the anti-ringing sums?  r2: every
// tap; r3/r4: the 13-tap diamond |dx|+|dy| <= 2 (ravu-lite-ar-r3.hook:93-170).
template <int R>
__host__ __device__ constexpr bool lite_ar_col(int c) {
  return R == 2 || cabs(c / (2 * R - 1) - (R - 1)) + cabs(c % (2 * R - 1) - (R - 1)) <= 2;
}

template <int R, bool AR, typename T, bool H16 = false, int TR = 8>
struct LiteTile {
  static constexpr int N = 2 * R - 1, S = N * N, HALO = R - 1;
  // two pixels of a column per thread, keys first: shared loads and derivatives
  // of the two windows (1080p at 8 rows, one / two / four pixels a thread:
  // ravu-lite-r4 fast 61.0 / 53.3 / 53.1 us, -ar-r3 54.1 / 49.6 / 50.0, -ar-r4 76.7 /
  // 71.3 / 78.6, r3 FP32 48.7 / 46.6 / 46.6).  Bound by L1 (80-93 %): a 16-byte
  // gather from 32 LUT rows takes 12-13 wavefronts.
  static constexpr int P = 2;
  static constexpr int kRows = TR, kThreads = kTileW * TR / P;
  static constexpr bool kOutputTiles = false;
  static constexpr int TW = kTilePitch, TH = TR + N - 1;
  // the value tile and (AR) each texel's two 32nd powers, formed while staging
  // and read as 8 bytes a tap (1080p, 4-row tiles: r3 fast 54.1 us, formed per tap
  // 57.0; r4 fast 74.9 and 76.0; r2 39.8 and 41.8).  With FP32 texels, whose
  // gathers already fill L1, r3 and r4 lose by it (57.0 us without, 61.0 with; 93
  // and 102) and form them per tap
  static constexpr bool kTable = AR && (H16 || R == 2);
  static constexpr size_t smem_bytes = (size_t)TW * TH * (kTable ? 12 : 4);

  static constexpr int kPlanes = 1;
  static constexpr bool kTma = true;
  static constexpr int kMaxRegs = 0;  // any cap costs 1-5 % (64 and 80 measured)
  // ravu-lite-ar-r2 / -r3 measured 2-5 % slower with the packed structure
  // tensor (register allocation of the anti-ringing sums)
  static constexpr bool kPackedTensor = !(R <= 3 && AR);
  using Elem = T;

  __device__ static void run(const RavuArgs& p, int f, int x0, int y0, float* smem, TmaCtx* tma = nullptr) {
    float* tile = smem;
    float* pow = tile + TW * TH;
    if (!stage_frame<kLuma, TH, kThreads, T, kTable>(p, tma, f, x0, y0 - HALO, tile, NoStage(), reinterpret_cast<float4*>(pow)))
      return;
    __syncthreads();
    const int tx = threadIdx.x % kTileW, ty = threadIdx.x / kTileW * P;
    const int gx = x0 + tx, gy = y0 + ty;
    if (gx >= p.W || gy >= p.H) return;
    const int at = ty * TW + tx + kLead - HALO;
    float a[P], b[P], d[P];
    structure_tensors<N, false, kPackedTensor, P, OffDown>([&](int X, int Y) { return tile[at + Y * TW + X]; }, p.kp, a,
                                                           b, d);
    size_t rows[P];
#pragma unroll
    for (int e = 0; e < P; e++) {
      const int key = ravu_key(a[e], b[e], d[e], p.kp);
      if (p.keys && gy + e < p.H) p.keys[(size_t)(gy + e) * p.W + gx] = key;
      rows[e] = (size_t)min(max(key, 0), p.lut_rows - 1) * (H16 ? p.lut_h_pitch : p.lut_pitch);
    }
#pragma unroll
    for (int e = 0; e < P; e++)
      if (gy + e < p.H) 
        filter(p, f, rows[e], tile + at + e * TW, reinterpret_cast<const float2*>(pow) + at + e * TW, gx, gy + e);
  }

  // one pixel's four outputs: its LUT row, its window and (kTable) powers
  __device__ static __forceinline__ void filter(const RavuArgs& p, int f, size_t row, const float* base,
                                                const float2* pbase, int gx, int gy) {
    auto get = [&](int kx, int ky) { return base[ky * TW + kx]; };
    float4 w_next;  // H16: the odd texel of the pair loaded at the even one
    static_assert(S / 2 % 2 == 0, "texel pairs start at even columns");
    // FP32x2 sums: P = sum va*w, Q = sum vb*w, res = P + Q.wzyx; the
    // anti-ringing sums of output k (ar_finish): G = sums, M = means
    float2 P01 = make_float2(0.f, 0.f), P23 = P01, Q01 = P01, Q23 = P01;
    float2 G[4], M[4];
#pragma unroll
    for (int k = 0; k < 4; k++) G[k] = M[k] = P01;
    // one AR tap: value v at window tap t, its weights g[k] (mirrored: g[3-k])
    auto ar_tap = [&](float v, int t, const float (&g)[4], bool mirrored) {
      const float2 h = kTable ? pbase[t % N * TW + t / N] : ar_pow32(v), hv = __fmul2_rn(h, make_float2(v, v));
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const float gk = g[mirrored ? 3 - k : k];
        G[k] = __ffma2_rn(h, make_float2(gk, gk), G[k]);
        M[k] = __ffma2_rn(hv, make_float2(gk, gk), M[k]);
      }
    };
#pragma unroll
    for (int c = 0; c <= S / 2; c++) {
      float4 w;
      if constexpr (H16) {
        if (c % 2 == 0) lut_pair_h16(p.lut_h, row + c, w, w_next);
        else w = w_next;
      } else {
        w = __ldg(p.lut + row + c);
      }
      const float va = get(c / N, c % N), vb = get((S - 1 - c) / N, (S - 1 - c) % N);
      const float2 w01 = make_float2(w.x, w.y), w23 = make_float2(w.z, w.w);
      const float2 a2 = make_float2(va, va), b2 = make_float2(vb, vb);
      P01 = __ffma2_rn(a2, w01, P01);
      P23 = __ffma2_rn(a2, w23, P23);
      if (c < S / 2) {  // the centre tap is its own mirror
        Q01 = __ffma2_rn(b2, w01, Q01);
        Q23 = __ffma2_rn(b2, w23, Q23);
      }
      if (AR && lite_ar_col<R>(c)) {
        const float g[4] = {fmaxf(w.x, 0.f), fmaxf(w.y, 0.f), fmaxf(w.z, 0.f), fmaxf(w.w, 0.f)};
        ar_tap(va, c, g, false);
        if (c < S / 2) ar_tap(vb, S - 1 - c, g, true);
      }
    }
    float4 res = make_float4(P01.x + Q23.y, P01.y + Q23.x, P23.x + Q01.y, P23.y + Q01.x);
    if (AR) {  // no [0,1] clamp after anti-ringing (compute/ravu-lite-ar-r3.hook:166)
      res.x = ar_finish(res.x, G[0], M[0], p.ar);
      res.y = ar_finish(res.y, G[1], M[1], p.ar);
      res.z = ar_finish(res.z, G[2], M[2], p.ar);
      res.w = ar_finish(res.w, G[3], M[3], p.ar);
    } else {
      res.x = clampf(res.x, 0.f, 1.f); res.y = clampf(res.y, 0.f, 1.f);
      res.z = clampf(res.z, 0.f, 1.f); res.w = clampf(res.w, 0.f, 1.f);
    }
    // res[0..3] -> offsets (0,0), (0,1), (1,0), (1,1)  (compute/ravu-lite-r3.hook:101-104)
    T* out = plane_out<T>(p, 0, f);
    const int op = p.out_pitch[0];
    stp2(out + (size_t)(2 * gy) * op + 2 * gx, res.x, res.z);
    stp2(out + (size_t)(2 * gy + 1) * op + 2 * gx, res.y, res.w);
  }
};

// --------------------------------------------------------------- ravu-3x --
template <int R, int CM, typename T, bool H16 = false, int TR = 8>
struct ThreeXTile {
  static constexpr int N = 2 * R - 1, S = N * N, HALO = R - 1;
  // two pixels of a column per thread, as in LiteTile (1080p at 8 rows, one / two /
  // four pixels a thread: r3 fast 47.3 / 43.2 / 44.0 us, r4 FP32 128.0 / 108.5 /
  // 110.7, r3-rgb fast 93.0 / 84.5 / 91.5)
  static constexpr int P = 2;
  static constexpr int kRows = TR, kThreads = kTileW * TR / P;
  static constexpr bool kOutputTiles = false;
  static constexpr int TW = kTilePitch, TH = TR + N - 1;
  static constexpr int C = CM == kLuma ? 1 : 3;
  static constexpr size_t smem_bytes = (size_t)(C + (CM == kRgb ? 1 : 0)) * TW * TH * 4;
  static constexpr int kPlanes = C;
  static constexpr bool kTma = true;
  static constexpr int kMaxRegs = 0;  // the compiler's own allocation
  using Elem = T;

  __device__ static void run(const RavuArgs& p, int f, int x0, int y0, float* smem, TmaCtx* tma = nullptr) {
    float* tile = smem;
    if (!stage_frame<CM, TH, kThreads, T>(p, tma, f, x0, y0 - HALO, tile)) return;
    __syncthreads();
    const int tx = threadIdx.x % kTileW, ty = threadIdx.x / kTileW * P;
    const int gx = x0 + tx, gy = y0 + ty;
    if (gx >= p.W || gy >= p.H) return;
    const float* base = tile + ty * TW + tx + kLead - HALO;
    const float* lbase = base + (CM == kRgb ? C * TW * TH : 0);
    float a[P], b[P], d[P];
    structure_tensors<N, false, true, P, OffDown>([&](int X, int Y) { return lbase[Y * TW + X]; }, p.kp, a, b, d);
    // 3x rows hold 2 * ceil(S / 2) texels: even, so the FP32 texel pairs are
    // 32-byte aligned without padding (1.2x over two 16-byte loads)
    size_t rows[P];
#pragma unroll
    for (int e = 0; e < P; e++) {
      const int key = ravu_key(a[e], b[e], d[e], p.kp);
      if (p.keys && gy + e < p.H) p.keys[(size_t)(gy + e) * p.W + gx] = key;
      rows[e] = (size_t)min(max(key, 0), p.lut_rows - 1) * (H16 ? p.lut_h_pitch : p.lut_pitch);
    }
#pragma unroll
    for (int e = 0; e < P; e++)
      if (gy + e < p.H) filter(p, f, rows[e], base + e * TW, gx, gy + e);
  }

  // one pixel's 3 x 3 outputs: its LUT row and its windows
  __device__ static __forceinline__ void filter(const RavuArgs& p, int f, size_t row, const float* base, int gx,
                                                int gy) {
    auto val = [&](int c, int t) { return base[c * TW * TH + t % N * TW + t / N]; };
    // res0 += a*w0 + b*w1.wzyx; res1 += a*w1 + b*w0.wzyx, as FP32x2 sums
    // P0 = sum a*w0, P1 = sum a*w1, Q0 = sum b*w0, Q1 = sum b*w1 (pairs .xy, .zw)
    float2 P0[C][2], P1[C][2], Q0[C][2], Q1[C][2];
#pragma unroll
    for (int c = 0; c < C; c++)
#pragma unroll
      for (int h = 0; h < 2; h++) P0[c][h] = P1[c][h] = Q0[c][h] = Q1[c][h] = make_float2(0.f, 0.f);
#pragma unroll
    for (int t = 0; t < S / 2; t++) {
      float4 w0, w1;
      if constexpr (H16) lut_pair_h16(p.lut_h, row + 2 * t, w0, w1);
      else lut_pair_f32(p.lut, row + 2 * t, w0, w1);
      const float2 w0a = make_float2(w0.x, w0.y), w0b = make_float2(w0.z, w0.w);
      const float2 w1a = make_float2(w1.x, w1.y), w1b = make_float2(w1.z, w1.w);
#pragma unroll
      for (int c = 0; c < C; c++) {
        const float va = val(c, t), vb = val(c, S - 1 - t);
        const float2 a2 = make_float2(va, va), b2 = make_float2(vb, vb);
        P0[c][0] = __ffma2_rn(a2, w0a, P0[c][0]);
        P0[c][1] = __ffma2_rn(a2, w0b, P0[c][1]);
        P1[c][0] = __ffma2_rn(a2, w1a, P1[c][0]);
        P1[c][1] = __ffma2_rn(a2, w1b, P1[c][1]);
        Q0[c][0] = __ffma2_rn(b2, w0a, Q0[c][0]);
        Q0[c][1] = __ffma2_rn(b2, w0b, Q0[c][1]);
        Q1[c][0] = __ffma2_rn(b2, w1a, Q1[c][0]);
        Q1[c][1] = __ffma2_rn(b2, w1b, Q1[c][1]);
      }
    }
    constexpr int tc = S / 2;
    float4 w0, w1;
    if constexpr (H16) lut_pair_h16(p.lut_h, row + 2 * tc, w0, w1);
    else lut_pair_f32(p.lut, row + 2 * tc, w0, w1);
    float4 r0[C], r1[C];
#pragma unroll
    for (int c = 0; c < C; c++) {
      const float v = val(c, tc);
      const float2 v2 = make_float2(v, v);
      P0[c][0] = __ffma2_rn(v2, make_float2(w0.x, w0.y), P0[c][0]);
      P0[c][1] = __ffma2_rn(v2, make_float2(w0.z, w0.w), P0[c][1]);
      P1[c][0] = __ffma2_rn(v2, make_float2(w1.x, w1.y), P1[c][0]);
      P1[c][1] = __ffma2_rn(v2, make_float2(w1.z, w1.w), P1[c][1]);
      // r0 = P0 + Q1.wzyx, r1 = P1 + Q0.wzyx
      r0[c] = make_float4(P0[c][0].x + Q1[c][1].y, P0[c][0].y + Q1[c][1].x, P0[c][1].x + Q1[c][0].y,
                          P0[c][1].y + Q1[c][0].x);
      r1[c] = make_float4(P1[c][0].x + Q0[c][1].y, P1[c][0].y + Q0[c][1].x, P1[c][1].x + Q0[c][0].y,
                          P1[c][1].y + Q0[c][0].x);
      const float4 a0 = make_float4(clampf(r0[c].x, 0.f, 1.f), clampf(r0[c].y, 0.f, 1.f),
                                    clampf(r0[c].z, 0.f, 1.f), clampf(r0[c].w, 0.f, 1.f));
      const float4 a1 = make_float4(clampf(r1[c].x, 0.f, 1.f), clampf(r1[c].y, 0.f, 1.f),
                                    clampf(r1[c].z, 0.f, 1.f), clampf(r1[c].w, 0.f, 1.f));
      // imageStore(gid*3 + (dx,dy)): res0 -> (0,0),(0,1),(0,2),(1,0); centre (1,1);
      // res1 -> (1,2),(2,0),(2,1),(2,2)   (compute/ravu-3x-r2.hook:106-114)
      T* o = plane_out<T>(p, c, f);
      const size_t op = p.out_pitch[c];
      T* r = o + (size_t)(3 * gy) * op + 3 * gx;
      stp(r, a0.x); stp(r + 1, a0.w); stp(r + 2, a1.y);
      r += op;
      stp(r, a0.y); stp(r + 1, v); stp(r + 2, a1.z);
      r += op;
      stp(r, a0.z); stp(r + 1, a1.x); stp(r + 2, a1.w);
    }
  }
};

// ------------------------------------------------------ ravu lattice -----

// int11: the keyed filter over the input window (ravu-r3.hook:15-146):
// res[c] = sum over the S/2 mirrored tap pairs of (x_i + x_{S-1-i}) * w_i, the
// weights w_i packed 4 to a texel, even and odd i in the lanes of an FP32x2 sum.
// A thread computes P pixels of one column, whose windows overlap in all but
// one row each: loads, derivatives and staging are shared (33 shared loads and
// stores a pixel at r3, from 73).  Each thread stores its int11 values into the
// compact FP32 int11 plane (p.i11, [C][H][W]): one coalesced 4-byte store per
// pixel and channel.  The lattice program below writes every output pixel.
// Bound by issue (70 %) and by L1 (74 %), half of it the gathers of LUT rows.
// 1080p, r3 luma: 26 us (34.4 us with one pixel a thread and texel staging).
template <int R, int CM, typename T, int TR = 8>
struct Int11Tile {
  static constexpr int N = 2 * R, S = N * N, HALO = R - 1;
  static constexpr int C = CM == kLuma ? 1 : 3;
  static constexpr int P = 4;
  static constexpr int kRows = TR, kThreads = kTileW * TR / P;
  static constexpr bool kOutputTiles = false;
  static constexpr int TW = kTilePitch, TH = TR + N - 1;
  static constexpr size_t smem_bytes = (size_t)(C + (CM == kRgb ? 1 : 0)) * TW * TH * 4;
  static constexpr int kPlanes = C;
  static constexpr bool kTma = true;
  // r3 luma at 56 registers (of 66) is 1 % faster; the others lose by any cap
  static constexpr int kMaxRegs = R == 3 && CM == kLuma ? 56 : 0;
  using Elem = T;

  __device__ static void run(const RavuArgs& p, int f, int x0, int y0, float* smem, TmaCtx* tma = nullptr) {
    pdl_trigger();  // the lattice launch
    float* tile = smem;
    if (!stage_frame<CM, TH, kThreads, T>(p, tma, f, x0, y0 - HALO, tile)) return;
    __syncthreads();
    const int tx = threadIdx.x % kTileW, ty = threadIdx.x / kTileW * P;
    const int gx = x0 + tx, gy = y0 + ty;
    if (gx >= p.W || gy >= p.H) return;
    const float* base = tile + ty * TW + tx + kLead - HALO;
    const float* lbase = base + (CM == kRgb ? C * TW * TH : 0);
    float a[P], b[P], d[P];
    structure_tensors<N, true, true, P, OffDown>([&](int X, int Y) { return lbase[Y * TW + X]; }, p.kp, a, b, d);
    const float4* L[P];
#pragma unroll
    for (int e = 0; e < P; e++) {
      const int key = ravu_key(a[e], b[e], d[e], p.kp);
      if (p.keys && gy + e < p.H) p.keys[(size_t)(gy + e) * p.W + gx] = key;
      L[e] = p.lut + (size_t)min(max(key, 0), p.lut_rows - 1) * p.lut_pitch;
    }
    if (C > 1 || R == 4) asm volatile("" ::: "memory");  // no window value stays in a register from here
    float2 acc[P][C];
    float4 w4[P];
#pragma unroll
    for (int e = 0; e < P; e++)
#pragma unroll
      for (int c = 0; c < C; c++) acc[e][c] = make_float2(0.0f, 0.0f);
#pragma unroll
    for (int i = 0; i < S / 2; i += 2) {
      const int X = i / N, Y = i % N;
#pragma unroll
      for (int e = 0; e < P; e++) {
        if (i % 4 == 0) w4[e] = __ldg(L[e] + i / 4);
        const float2 w2 = i % 4 == 0 ? make_float2(w4[e].x, w4[e].y) : make_float2(w4[e].z, w4[e].w);
#pragma unroll
        for (int c = 0; c < C; c++) {
          auto v = [&](int x, int y) { return base[c * TW * TH + (y + e) * TW + x]; };
          const float2 s2 = make_float2(v(X, Y) + v(N - 1 - X, N - 1 - Y), v(X, Y + 1) + v(N - 1 - X, N - 2 - Y));
          acc[e][c] = __ffma2_rn(s2, w2, acc[e][c]);
        }
      }
    }
    const size_t plane = (size_t)p.W * p.H;
#pragma unroll
    for (int e = 0; e < P; e++) {
      if (gy + e >= p.H) break;
#pragma unroll
      for (int c = 0; c < C; c++) {
        float v = clampf(acc[e][c].x + acc[e][c].y, 0.f, 1.f);
        if (p.i11_half) v = __half2float(__float2half_rn(v));
        p.i11[(f * C + c) * plane + (size_t)(gy + e) * p.W + gx] = v;
      }
    }
  }
};

// The two lattice passes read windows turned by 45 degrees (s = kx+ky-(N-1),
// d = ky-kx; ravu-r3.hook:155-189 int10, :289-323 int01) of the lattice that
// interleaves input and int11 pixels.  int01's window is int10's one step back
// along kx, so both are windows of one lattice (X, Y): int10 at X = kx, int01
// at X = kx - 1.
// The windows of the pixel below lie one step back along X and one on along Y.
struct OffLattice {
  __host__ __device__ static constexpr int x(int e) { return -(e % 2) - e / 2; }
  __host__ __device__ static constexpr int y(int e) { return e / 2; }
};
// Where lattice point (X, Y) lies: 0 = input, 1 = int11, at offset (dx, dy).
template <int N>
__host__ __device__ constexpr int lat_src(int X, int Y) {
  return (X + Y - (N - 1)) % 2 != 0 ? 0 : 1;
}
template <int N>
__host__ __device__ constexpr int lat_dx(int X, int Y) {
  return lat_src<N>(X, Y) == 0 ? (X + Y - (N - 1) + 1) / 2 : (X + Y - (N - 1)) / 2;
}
template <int N>
__host__ __device__ constexpr int lat_dy(int X, int Y) {
  return lat_src<N>(X, Y) == 0 ? (Y - X) / 2 : (Y - X - 1) / 2;
}

// int10 + int01: both lattice filters per input pixel (ravu-r3.hook:148-437).
// The input tile and the int11 tile (from the FP32 int11 plane, clamped to
// its edge: the clamp-to-edge of the int11 texture) are staged; each thread
// evaluates both windows of P = 2 pixels, one below the other.  The keys of all
// four windows come first: they share most loads and derivatives.  A pixel's
// filters then load every lattice value once for its two windows, and a tap is
// one lane of an FP32x2 product with its weight (no sums of mirrored taps first:
// the two windows mirror differently).  The thread holds all four samples of an
// output 2x2 block -- input (0,0), int10 (1,0), int01 (0,1), int11 (1,1) -- and
// writes them as two pixel-pair rows.
// Bound by issue (69 %) and by L1 (76-80 %).  1080p, both passes together at 8
// rows, one / two pixels a thread: ravu-r2 56.2 / 54.2 us, ravu-r3 78.7 (4 rows) /
// 74.6 (100.9 with each window by itself and texel staging), ravu-r4 131 / 114
// (266), ravu-r3-yuv 125 / 118 (153), ravu-r4-yuv 204 / 198, 189 at 16 rows (330).
template <int R, int CM, typename T, int TR = 8>
struct LatticeTile {
  static constexpr int N = 2 * R, S = N * N;
  static constexpr int P = 2;
  static constexpr int kRows = TR, kThreads = kTileW * TR / P;
  static constexpr bool kOutputTiles = false;
  static constexpr int TW = kTilePitch, TH = TR + N - 1;
  static constexpr int C = CM == kLuma ? 1 : 3;
  static constexpr int PL = C + (CM == kRgb ? 1 : 0);  // planes per tile set
  static constexpr size_t smem_bytes = (size_t)2 * PL * TW * TH * 4;
  static constexpr int kPlanes = C;
  static constexpr bool kTma = true;
  // r4 luma at 80 registers (of 100) is 2 % faster; the others lose by any cap
  // (r4-yuv at 80: 207 against 198 us, at 64: 259)
  static constexpr int kMaxRegs = R == 4 && CM == kLuma ? 80 : 0;
  using Elem = T;

  __device__ static void run(const RavuArgs& p, int f, int x0, int y0, float* smem, TmaCtx* tma = nullptr) {
    float* tin = smem;                      // input, rows y0-(R-1) ..
    float* t11 = smem + PL * TW * TH;       // int11, rows y0-R ..
    const size_t plane = (size_t)p.W * p.H;
    struct {
      TileStage<CM, TH, kThreads, FreshFloat> st;
      const RavuArgs& p;
      float* t11;
      int f, x0, y0;
      __device__ __forceinline__ void load() {
        pdl_wait();  // the input tile's loads are in flight
        st.load([&](int c, int& pitch) {
          pitch = p.W;
          return reinterpret_cast<const FreshFloat*>(p.i11) + (size_t)(f * C + c) * p.W * p.H;
        }, p.W, p.H, x0, y0);
      }
      __device__ __forceinline__ void store() { st.store(t11); }
    } i11{{}, p, t11, f, x0, y0 - R};
    if (!stage_frame<CM, TH, kThreads, T>(p, tma, f, x0, y0 - (R - 1), tin, i11)) return;
    __syncthreads();
    const int tx = threadIdx.x % kTileW, ty = threadIdx.x / kTileW * P;
    const int gx = x0 + tx, gy = y0 + ty;
    if (gx >= p.W || gy >= p.H) return;
    const float* bin = tin + (ty + R - 1) * TW + tx + kLead;
    const float* b11 = t11 + (ty + R) * TW + tx + kLead;
    auto point = [&](int c, int X, int Y, int down) {
      return (lat_src<N>(X, Y) == 0 ? bin : b11)[c * TW * TH + (lat_dy<N>(X, Y) + down) * TW + lat_dx<N>(X, Y)];
    };
    float a[2 * P], b[2 * P], d[2 * P];
    structure_tensors<N, true, true, 2 * P, OffLattice>(
        [&](int X, int Y) { return point(CM == kRgb ? C : 0, X, Y, 0); }, p.kp, a, b, d);  // rgb: the luma tile is plane C
    const float4* rows[2 * P];
#pragma unroll
    for (int e = 0; e < 2 * P; e++) {
      const int key = ravu_key(a[e], b[e], d[e], p.kp);
      if (p.keys && gy + e / 2 < p.H) p.keys[(size_t)(1 + e % 2) * plane + (size_t)(gy + e / 2) * p.W + gx] = key;
      rows[e] = p.lut + (size_t)min(max(key, 0), p.lut_rows - 1) * p.lut_pitch;
    }
    if (C > 1 || R == 4) asm volatile("" ::: "memory");  // no window value stays in a register from here
#pragma unroll
    for (int down = 0; down < P; down++) {
      if (gy + down >= p.H) break;
      auto val = [&](int c, int X, int Y) { return point(c, X, Y, down); };
      float4 w[2][(S / 2 + 3) / 4];
#pragma unroll
      for (int e = 0; e < 2; e++)
#pragma unroll
        for (int q = 0; q < (S / 2 + 3) / 4; q++) w[e][q] = __ldg(rows[2 * down + e] + q);
      // weights i, i+1 (i even) of window e as a pair
      auto wpair = [&](int e, int i) {
        const float4& q = w[e][i / 4];
        return i % 4 == 0 ? make_float2(q.x, q.y) : make_float2(q.z, q.w);
      };
#pragma unroll
      for (int c = 0; c < C; c++) {
        float2 acc[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
        for (int X = -1; X < N; X++) {
#pragma unroll
          for (int Y = 0; Y < N; Y += 2) {
            const float v0 = val(c, X, Y), v1 = val(c, X, Y + 1);
#pragma unroll
            for (int e = 0; e < 2; e++) {
              const int i = (X + e) * N + Y;  // taps i, i+1 of window e; the upper half mirrors the lower
              if (i < 0 || i >= S) continue;
              if (i < S / 2) acc[e] = __ffma2_rn(make_float2(v0, v1), wpair(e, i), acc[e]);
              else acc[e] = __ffma2_rn(make_float2(v1, v0), wpair(e, S - 2 - i), acc[e]);
            }
          }
        }
        T* o = plane_out<T>(p, c, f) + (size_t)(2 * (gy + down)) * p.out_pitch[c] + 2 * gx;
        // row 2i: input, int10; row 2i+1: int01, int11 (ravu-r3.hook:424-437)
        stp2(o, bin[c * TW * TH + down * TW], clampf(acc[0].x + acc[0].y, 0.f, 1.f));
        stp2(o + p.out_pitch[c], clampf(acc[1].x + acc[1].y, 0.f, 1.f), b11[c * TW * TH + down * TW]);
      }
    }
  }
};

// ------------------------------------------------------------ ravu-zoom ---
struct ZoomPos {
  int i;    // floor(pos - 0.5)
  float s;  // fract(pos - 0.5)
};

// pos - 0.5 = ((2X+1) W - OW) / (2 OW), taken exactly (centre-aligned map);
// `d`: 2 OW, or d.d = 0 where the numerator needs 64 bits.
__device__ __forceinline__ ZoomPos zoom_pos(int X, int W, int OW, const FastDiv& d) {
  if (d.d) {
    const int num = (2 * X + 1) * W - OW;  // > -2 OW: W < OW
    const int q = num < 0 ? -1 : (int)d(num);
    return {q, (float)(num - q * (int)d.d) / (float)(int)d.d};
  }
  const long long num = (2LL * X + 1) * W - OW;
  const long long den = 2LL * OW;
  const long long q = num >= 0 ? num / den : -((-num + den - 1) / den);
  return {(int)q, (float)(num - q * den) / (float)den};
}

// Texels (4 weights) of a key's half window at each of ravu-zoom's 9 x 9 LUT
// points, and where texel t of point (row key * 9 + jy, jx) lies:
//   FP32  as in the file, 9 neighbouring points' texels t side by side (144
//         bytes): lanes with one key and different phases share a line
//   FP16  by points, the point's texels side by side and padded to an even count,
//         so that they come as 16-byte pairs
// ravu-zoom-r2 / -r3, 1080p to 1.5x: FP16 by points 85 / 171 us against 132 / 217 us
// as in the file; FP32 by points 121 / 330 us against 135 / 283 us as in the file.
template <int R>
__host__ __device__ constexpr int zoom_texels() {
  return (2 * R * R + 3) / 4;
}
template <int R, bool H16>
__host__ __device__ constexpr uint32_t zoom_texel_at(uint32_t row, uint32_t jx, uint32_t t) {
  return H16 ? (row * 9 + jx) * ((zoom_texels<R>() + 1) & ~1) + t : (row * zoom_texels<R>() + t) * 9 + jx;
}

// The bilinear (FILTER LINEAR) position of one sub-position in a key's 9 x 9
// points: x = 8 sx, y = key * 9 + 8 sy (LUTPOS(x, 9) / (blocks, 288),
// ravu-zoom-r2.hook:23-31); rows clamp to the table's edge.  With q > 0 the
// fractions are rounded to multiples of 1/q, as a texture unit's fixed-point
// filter weights are (q = 256: 8 fractional bits).
struct ZoomLut {
  uint32_t row[2], col[2];  // rows floor(y), floor(y) + 1; columns floor(x), and the next (at most the
                            // last one, whose weight is then 0)
  float w[4];               // weights of (0, 0), (1, 0), (0, 1), (1, 1) (column, row)
  __device__ __forceinline__ ZoomLut() {}
  __device__ __forceinline__ ZoomLut(int rows, int key, float sx, float sy, float q) {
    const float fx8 = 8.0f * sx, fy8 = 8.0f * sy;
    const float x0f = floorf(fx8), y0f = floorf(fy8);
    float fx = fx8 - x0f, fy = fy8 - y0f;
    if (q > 0.0f) {
      fx = rintf(fx * q) / q;
      fy = rintf(fy * q) / q;
    }
    col[0] = min((int)x0f, 8);
    col[1] = min(col[0] + 1, 8u);
    row[0] = clampi(key * 9 + (int)y0f, 0, rows - 1);
    row[1] = min((int)row[0] + 1, rows - 1);
    const float gx = 1.0f - fx, gy = 1.0f - fy;
    w[0] = gx * gy;
    w[1] = fx * gy;
    w[2] = gx * fy;
    w[3] = fx * fy;
  }
  // Texels 2t, 2t+1 of the interpolated point as FP32x2 pairs.
  template <int R, bool H16>
  __device__ __forceinline__ void texels(const float4* f, const uint2* h, int t, float2 (&out)[4]) const {
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const uint32_t y = row[k / 2], x = col[k % 2];
      float4 a, b = make_float4(0.f, 0.f, 0.f, 0.f);
      if constexpr (H16) {
        lut_pair_h16(h, zoom_texel_at<R, true>(y, x, 2 * t), a, b);
      } else {
        a = __ldg(f + zoom_texel_at<R, false>(y, x, 2 * t));
        if (2 * t + 1 < zoom_texels<R>()) b = __ldg(f + zoom_texel_at<R, false>(y, x, 2 * t + 1));
      }
      const float2 w2 = make_float2(w[k], w[k]);
      const float2 v[4] = {make_float2(a.x, a.y), make_float2(a.z, a.w), make_float2(b.x, b.y), make_float2(b.z, b.w)};
#pragma unroll
      for (int j = 0; j < 4; j++) out[j] = k == 0 ? __fmul2_rn(v[j], w2) : __ffma2_rn(v[j], w2, out[j]);
    }
  }
};

// float4 of an entry of the phase table: the weights of the two half windows,
// then (AR) the anti-ringing weights' two, padded to an odd count: a warp's loads
// gather from 32 entries at once, and at an even stride they meet in few of L1's
// 8 16-byte banks (1080p to 1.5x: ravu-zoom-ar-r2 97 us, 158 at 8 float4;
// ravu-zoom-r2 62 us, 76 at 4).
template <int R, bool AR>
__host__ __device__ constexpr uint32_t zoom_entry() {
  return zoom_texels<R>() * (AR ? 4 : 2) + 1;
}

// The weights of every key at every phase of a scale whose output positions
// repeat after few pixels (1.5x: 3 x 3 phases; 2.25x: 9 x 9), [key][phase y]
// [phase x][entry]: the same bilinear fetches as a pixel's own, once per launch
// instead of once per pixel.  One thread per entry and texel pair.
template <int R, bool AR, bool H16>
__global__ void zoom_table_kernel(const __grid_constant__ RavuArgs p, float4* out) {
  constexpr int NB = zoom_texels<R>(), NT2 = (NB + 1) / 2, PER = NT2 * (AR ? 4 : 2);
  pdl_trigger();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int phases = (int)(p.zpx.d * p.zpy.d), n = p.lut_rows / 9 * phases;
  if (i >= n * PER) return;
  const int entry = i / PER, t = i % PER % NT2, part = i % PER / NT2;  // part: halves, then the AR halves
  const int key = entry / phases, phase = entry % phases, py = p.zpx(phase), px = phase - py * (int)p.zpx.d;
  float sx = zoom_pos(px, p.W, p.OW, p.zx).s, sy = zoom_pos(py, p.H, p.OH, p.zy).s;
  if (part & 1) {
    sx = 1.0f - sx;
    sy = 1.0f - sy;
  }
  const ZoomLut l(p.lut_rows, key, sx, sy, p.lut_frac);
  float2 w[4];
  if (part < 2) l.texels<R, H16>(p.lut, p.lut_h, t, w);
  else l.texels<R, false>(p.lut_ar, nullptr, t, w);
  float4* o = out + (size_t)entry * zoom_entry<R, AR>() + part * NB + 2 * t;
  o[0] = make_float4(w[0].x, w[0].y, w[1].x, w[1].y);
  if (2 * t + 1 < NB) o[1] = make_float4(w[2].x, w[2].y, w[3].x, w[3].y);
}

// One thread per OUTPUT pixel; the tile is 32 x TR output pixels and stages the
// input rectangle they touch (at most (32+N+1) x (TR+N+1) when upscaling;
// its origin follows from the tile's source positions, as the compute
// shader's rect, compute/ravu-zoom-ar-r2.hook:28-37): by quads of columns from
// the multiple of 4 at or left of the rectangle, or (TMA staging, interior
// rectangles) from one TMA box per plane whose size the host fits to the
// launch's scale factor (tma_box_of), converting just the rectangle.
// Bound by L1, where the gathers of LUT texels go (86 %; 16-40 loads a pixel).
// 1080p to 1.5x, without / with the phase table: ravu-zoom-r2 86 / 62 us fast (132
// with a load per texel, scalar blends and texel staging), r3 FP32 283 / 111 us
// (290), ravu-zoom-ar-r2-rgb fast 274 / 165 us (302).
// TAB: the weights come from the launch's phase table, at the same bits.
template <int R, int CM, bool AR, typename T, bool H16 = false, int TR = 8, bool TAB = false>
struct ZoomTile {
  static constexpr int N = 2 * R, S = N * N, LO = R - 1;
  static constexpr int kRows = TR, kThreads = kTileW * TR;
  static constexpr bool kOutputTiles = true;
  static constexpr int RW = kTileW + N + 1, RH = TR + N + 1;
  static constexpr int RP = (RW + 3 + 3) & ~3;  // row pitch: up to 3 lead columns
  static constexpr int C = CM == kLuma ? 1 : 3;
  static constexpr int PL = C + (CM == kRgb ? 1 : 0);
  static constexpr int NT2 = (zoom_texels<R>() + 1) / 2;  // texel pairs of a LUT point
  // input rectangle planes, then the powers of the first CT channels: with the
  // phase table's weights and three channels, forming all powers per tap keeps
  // the FMA pipe 75 % busy, L1 58 %; two channels' powers from shared memory, once
  // per texel, balance them (1080p to 1.5x: 0 / 1 / 2 / 3 channels 187 / 177 / 171 /
  // 179 us; to 2.25x 412 / 397 / 397 / 428; luma at 1.75x 73 / 78)
  static constexpr int CT = AR && TAB && C == 3 ? 2 : 0;
  static constexpr size_t smem_bytes = (size_t)(PL + 2 * CT) * RP * RH * 4;

  static constexpr int kPlanes = C;
  static constexpr bool kTma = !TAB;  // the table goes with plain loads
  // anti-ringing on FP32 texels: 4-8 % faster at 80 registers (of 96-126); any
  // cap costs the other programs
  static constexpr int kMaxRegs = AR && !H16 && !TAB ? 80 : 0;
  // the largest TMA box: the largest rectangle plus up to 7 lead columns
  static constexpr int kBoxMaxW = (RW + 7 + 7) & ~7, kBoxMaxH = RH;
  using Elem = T;

  // one staged texel: its values, its luma (RGB)
  __device__ static __forceinline__ void put(float* tile, int at, const float (&v)[C]) {
#pragma unroll
    for (int c = 0; c < C; c++) tile[c * RP * RH + at] = v[c];
    if constexpr (CM == kRgb) tile[C * RP * RH + at] = rgb_luma(v[0], v[1], v[2]);
  }

  __device__ static void run(const RavuArgs& p, int f, int X0, int Y0, float* smem, TmaCtx* tma = nullptr) {
    float* tile = smem;
    float2* pow = reinterpret_cast<float2*>(smem + PL * RP * RH);
    // exact source positions: lane l of every warp takes column X0 + l and row
    // Y0 + min(l, TR - 1); the tile's corners and the warp's own row come by shuffles
    // (no barrier; as 64-bit divisions shared through memory they held every tile
    // up: ravu-zoom-ar-r2-rgb at 1.5x 171 us, now 165; -ar-r2 at 2.25x 252, now 223)
    const int lane = threadIdx.x % kTileW, warp = threadIdx.x / kTileW;
    const int X = X0 + lane, Y = Y0 + warp, oy = min(Y0 + min(lane, TR - 1), p.OH - 1);
    ZoomPos px = zoom_pos(min(X, p.OW - 1), p.W, p.OW, p.zx), rows = zoom_pos(oy, p.H, p.OH, p.zy);
    const ZoomPos py = {__shfl_sync(~0u, rows.i, warp), __shfl_sync(~0u, rows.s, warp)};
    const int rx = __shfl_sync(~0u, px.i, 0) - LO, ry = __shfl_sync(~0u, rows.i, 0) - LO;
    const int rw = __shfl_sync(~0u, px.i, 31) + R - rx + 1, rh = __shfl_sync(~0u, rows.i, 31) + R - ry + 1;
    if (rw > RW || rh > RH) {  // only reachable when downscaling, which the host rejects
      if (threadIdx.x == 0 && p.err) atomicCAS(p.err, 0, kErrTileOverflow);
      return;
    }
    const int off = rx & 3;  // the rectangle's first column in the tile
    // every operand of these tests is uniform across the CTA
    if (tma && tma->map && !tma->dead && rx >= 0 && ry >= 0 && rx + rw <= p.W && ry + rh <= p.H &&
        (rx & 7) + rw <= p.box_w && rh <= p.box_h) {
      const uint32_t pb = ((uint32_t)p.box_w * p.box_h * sizeof(T) + 127u) & ~127u;
      tma_issue_box<CM, T>(tma, rx & ~7, ry, p.box_w, p.box_h, pb);
      if (!tma_wait_box(p, tma)) return;
      for (int i = threadIdx.x; i < rw * rh; i += kThreads) {
        const int ty = i / rw, tx = i % rw;
        float v[C];
#pragma unroll
        for (int c = 0; c < C; c++)
          v[c] = lds_f(reinterpret_cast<const T*>(tma->raw + c * pb) + ty * p.box_w + tx + (rx & 7));
        put(tile, ty * RP + tx + off, v);
      }
    } else {
      // loads of all planes first, then values, powers and luma
      constexpr int QW = RP / 4, IT = (QW * RH + kThreads - 1) / kThreads;
      Quad<T> q[C][IT];
      auto each = [&](auto f) {
#pragma unroll
        for (int k = 0; k < IT; k++) {
          const int i = threadIdx.x + k * kThreads, ty = i / QW, tx = i % QW * 4;
          if (ty < rh && tx < off + rw) f(k, ty, tx);
        }
      };
#pragma unroll
      for (int c = 0; c < C; c++) {
        const T* in = plane_in<T>(p, c, f);
        const int pitch = p.in_pitch[c];
        const bool aligned = quads_aligned(in, pitch);
        each([&](int k, int ty, int tx) {
          load_quad(q[c][k], in + (size_t)clampi(ry + ty, 0, p.H - 1) * pitch, rx - off + tx, p.W, aligned);
        });
      }
      each([&](int k, int ty, int tx) {
        float4 v[C];
#pragma unroll
        for (int c = 0; c < C; c++) v[c] = q[c][k].get();
        float4* t4 = reinterpret_cast<float4*>(tile + ty * RP + tx);
#pragma unroll
        for (int c = 0; c < C; c++) {
          t4[c * (RP * RH / 4)] = v[c];
          if (c < CT) {
            const float2 a = ar_pow32(v[c].x), b = ar_pow32(v[c].y), e = ar_pow32(v[c].z), d = ar_pow32(v[c].w);
            float4* p4 = reinterpret_cast<float4*>(pow + c * RP * RH + ty * RP + tx);
            p4[0] = make_float4(a.x, a.y, b.x, b.y);
            p4[1] = make_float4(e.x, e.y, d.x, d.y);
          }
        }
        if constexpr (CM == kRgb)
          t4[C * (RP * RH / 4)] = make_float4(rgb_luma(v[0].x, v[1].x, v[2].x), rgb_luma(v[0].y, v[1].y, v[2].y),
                                              rgb_luma(v[0].z, v[1].z, v[2].z), rgb_luma(v[0].w, v[1].w, v[2].w));
      });
    }
    __syncthreads();
    if (X >= p.OW || Y >= p.OH) return;
    const int at = (py.i - LO - ry) * RP + px.i - LO - rx + off;  // window origin in the tile
    const float* base = tile + at;
    auto val = [&](int c, int k) { return base[c * RP * RH + k % N * RP + k / N]; };
    auto lum = [&](int kx, int ky) { return base[(CM == kRgb ? C * RP * RH : 0) + ky * RP + kx]; };
    float a, b, d;
    structure_tensor<N, true>(lum, p.kp, a, b, d);
    const int key = ravu_key(a, b, d, p.kp);  // no +0.5 row centring (ravu-zoom-r2.hook:124)
    if (p.keys) p.keys[(size_t)Y * p.OW + X] = key;
    // the weights of taps 8t .. 8t+7 of a half window (0: from the front, 1: the
    // mirrored taps from the back; +2: anti-ringing) as pairs
    constexpr int NB = zoom_texels<R>();
    const float4* entry = nullptr;
    ZoomLut ls, li;
    if constexpr (TAB) {
      const int phx = X - (int)(p.zpx(X) * p.zpx.d), phy = Y - (int)(p.zpy(Y) * p.zpy.d);
      const int k = clampi(key, 0, p.lut_rows / 9 - 1) * (int)p.zpy.d + phy;
      pdl_wait();
      entry = p.ztab + ((size_t)k * p.zpx.d + phx) * zoom_entry<R, AR>();
    } else {
      ls = ZoomLut(p.lut_rows, key, px.s, py.s, p.lut_frac);
      li = ZoomLut(p.lut_rows, key, 1.0f - px.s, 1.0f - py.s, p.lut_frac);
    }
    auto weights = [&](int part, int t, float2 (&w)[4]) {
      if constexpr (TAB) {
        const float4 a = entry[part * NB + 2 * t];  // written by a launch this one may overlap
        const float4 b = 2 * t + 1 < NB ? entry[part * NB + 2 * t + 1] : a;
        w[0] = make_float2(a.x, a.y);
        w[1] = make_float2(a.z, a.w);
        w[2] = make_float2(b.x, b.y);
        w[3] = make_float2(b.z, b.w);
      } else {
        const ZoomLut& l = part & 1 ? li : ls;
        if (part < 2) l.texels<R, H16>(p.lut, p.lut_h, t, w);
        else l.texels<R, false>(p.lut_ar, nullptr, t, w);
      }
    };
    // taps i, i+1 in the lanes of res; anti-ringing sums per channel (ar_finish)
    float2 res[C], G[C], M[C];
#pragma unroll
    for (int c = 0; c < C; c++) res[c] = G[c] = M[c] = make_float2(0.0f, 0.0f);
#pragma unroll
    for (int t = 0; t < NT2; t++) {
      float2 ws[4], wi[4], gs[4], gi[4];
      weights(0, t, ws);
      weights(1, t, wi);
      if (AR) {  // the anti-ringing LUT stays FP32 in every form but mpv's (most of
                 // its values lie below FP16's normal range)
        weights(2, t, gs);
        weights(3, t, gi);
      }
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const int i = t * 8 + 2 * j;
        if (i >= S / 2) break;  // S / 2 is even
#pragma unroll
        for (int c = 0; c < C; c++) {
          const float va[2] = {val(c, i), val(c, i + 1)}, vb[2] = {val(c, S - 1 - i), val(c, S - 2 - i)};
          res[c] = __ffma2_rn(make_float2(va[0], va[1]), ws[j], res[c]);
          res[c] = __ffma2_rn(make_float2(vb[0], vb[1]), wi[j], res[c]);
          if constexpr (AR) {
            auto tap = [&](float v, int k, float g) {
              const float2 h = c < CT ? pow[c * RP * RH + at + k % N * RP + k / N] : ar_pow32(v);
              G[c] = __ffma2_rn(h, make_float2(g, g), G[c]);
              M[c] = __ffma2_rn(__fmul2_rn(h, make_float2(v, v)), make_float2(g, g), M[c]);
            };
            tap(va[0], i, gs[j].x);
            tap(va[1], i + 1, gs[j].y);
            tap(vb[0], S - 1 - i, gi[j].x);
            tap(vb[1], S - 2 - i, gi[j].y);
          }
        }
      }
    }
#pragma unroll
    for (int c = 0; c < C; c++) {
      const float r = res[c].x + res[c].y;
      stp(plane_out<T>(p, c, f) + (size_t)Y * p.out_pitch[c] + X,
          AR ? ar_finish(r, G[c], M[c], p.ar) : clampf(r, 0.f, 1.f));
    }
  }
};

// Programs that have a kernel of their own for launches of one frame: with the
// frame's index a constant, the ravu lattice at r4 is scheduled over 125 registers
// instead of 104 (1080p fast: ravu-r4-yuv 190 / 199 us, -rgb 193 / 203, luma 112.9 /
// 114.3).  The other programs run at one speed either way.
template <class Prog>
struct OneFrame : Prog {};
template <class Prog>
constexpr bool kIsOneFrame = false;
template <class Prog>
constexpr bool kIsOneFrame<OneFrame<Prog>> = true;
template <class Prog>
constexpr bool kHasOneFrame = false;
template <int CM, typename T, int TR>
constexpr bool kHasOneFrame<LatticeTile<4, CM, T, TR>> = true;

// One CTA per tile of a frame (grid z: the frame); with TMA (one frame a
// launch) the frame tile of interior
// tiles comes in by cp.async.bulk.tensor.
template <class Prog, bool TMA>
__device__ __forceinline__ void tile_body(const RavuArgs& p, const TmaMaps& maps) {
  extern __shared__ __align__(128) float4 tile_smem[];
  float* smem = reinterpret_cast<float*>(tile_smem);
  if (TMA) {
    __shared__ __align__(8) unsigned long long mbar;
    if (threadIdx.x == 0) mbar_init(smem_u32(&mbar), 1);
    __syncthreads();
    TmaCtx ctx{maps.map, smem_u32(&mbar),
               reinterpret_cast<unsigned char*>(tile_smem) + ((Prog::smem_bytes + 127) & ~(size_t)127), 0u, 0};
    Prog::run(p, 0, blockIdx.x * kTileW, blockIdx.y * Prog::kRows, smem, &ctx);
    tma_drain(&ctx);
  } else {
    Prog::run(p, kIsOneFrame<Prog> ? 0 : blockIdx.z, blockIdx.x * kTileW, blockIdx.y * Prog::kRows, smem, nullptr);
  }
}

// Programs with kMaxRegs > 0 run under that register cap (the same cap at
// every tile height); the others keep the compiler's own allocation.
template <class Prog, bool TMA>
__global__ void __launch_bounds__(Prog::kThreads) tile_kernel(const __grid_constant__ RavuArgs p,
                                                              const __grid_constant__ TmaMaps maps) {
  tile_body<Prog, TMA>(p, maps);
}
template <class Prog, bool TMA>
__global__ void __maxnreg__(Prog::kMaxRegs) tile_kernel_mr(const __grid_constant__ RavuArgs p,
                                                           const __grid_constant__ TmaMaps maps) {
  tile_body<Prog, TMA>(p, maps);
}

// SMEM: bytes of dynamic shared memory.
template <class Prog, bool TMA, size_t SMEM>
void launch_tile_kernel(dim3 grid, cudaStream_t s, const RavuArgs& a, const TmaMaps& maps) {
  static_assert(SMEM <= 48 * 1024, "tile program needs more than the default shared memory");
  auto kern = [] {
    if constexpr (Prog::kMaxRegs > 0) return tile_kernel_mr<Prog, TMA>;
    else return tile_kernel<Prog, TMA>;
  }();
  launch_kernel(kern, grid, Prog::kThreads, SMEM, s, a.after, a, maps);
}

bool encode_plane_map(CUtensorMap* map, const void* base, int W, int H, int pitch, int dtype, int box_w,
                      int box_h);

// TMA boxes of a program.  The frame-tile programs have one fixed box (the
// tile and its halo plus up to 7 lead columns).  ravu-zoom's box holds the
// largest input rectangle of the launch's scale factor: n consecutive output
// columns span at most floor((n-1) W / OW) + 1 source steps, plus the 2R
// window (rows likewise), capped at the program's largest box; a tile whose
// rectangle does not fit stages by clamped loads.
template <class Prog>
constexpr int tma_box_max_w() {
  if constexpr (Prog::kOutputTiles) return Prog::kBoxMaxW;
  else return tma_box_w<Prog::TW>();
}
template <class Prog>
constexpr int tma_box_max_h() {
  if constexpr (Prog::kOutputTiles) return Prog::kBoxMaxH;
  else return Prog::TH;
}
template <class Prog>
void tma_box_of(const RavuArgs& a, int* bw, int* bh) {
  if constexpr (Prog::kOutputTiles) {
    const int w = (int)((long long)(kTileW - 1) * a.W / a.OW) + 1 + Prog::N;
    const int h = (int)((long long)(Prog::kRows - 1) * a.H / a.OH) + 1 + Prog::N;
    *bw = ((w + 7 + 7) & ~7) < Prog::kBoxMaxW ? ((w + 7 + 7) & ~7) : Prog::kBoxMaxW;
    *bh = h < Prog::kBoxMaxH ? h : Prog::kBoxMaxH;
  } else {
    *bw = tma_box_max_w<Prog>();
    *bh = tma_box_max_h<Prog>();
  }
}
// Shared memory of the landing area: one largest box per plane.
template <class Prog>
constexpr size_t tma_landing_bytes() {
  return (size_t)Prog::kPlanes *
         (((size_t)tma_box_max_w<Prog>() * tma_box_max_h<Prog>() * sizeof(typename Prog::Elem) + 127) & ~(size_t)127);
}
// The maps of a's input planes for Prog's box (recorded in a->box_w / box_h);
// false when a plane cannot be mapped (alignment, a box larger than the plane).
template <class Prog>
bool encode_tma(RavuArgs* a, TmaMaps* maps) {
  int bw, bh;
  tma_box_of<Prog>(*a, &bw, &bh);
  const int dt = sizeof(typename Prog::Elem) == 4 ? 0 : 1;
  for (int c = 0; c < Prog::kPlanes; c++)
    if (!encode_plane_map(&maps->map[c], a->in[c], a->W, a->H, a->in_pitch[c], dt, bw, bh)) return false;
  a->box_w = bw;
  a->box_h = bh;
  return true;
}

// One CTA per tile of the frame (of the output frame for output-tiled
// programs), staged by TMA when the frame asks for it and its planes map.
template <class Prog>
int launch_tiles(const RavuArgs& a, cudaStream_t s) {
  const int fw = Prog::kOutputTiles ? a.OW : a.W, fh = Prog::kOutputTiles ? a.OH : a.H;
  const int tiles_w = (fw + kTileW - 1) / kTileW, tiles_h = (fh + Prog::kRows - 1) / Prog::kRows;
  TmaMaps maps;
  std::memset(&maps, 0, sizeof maps);
  if constexpr (Prog::kTma) {
    RavuArgs b = a;
    if (a.staging == 1 && encode_tma<Prog>(&b, &maps)) {
      constexpr size_t smem = ((Prog::smem_bytes + 127) & ~(size_t)127) + tma_landing_bytes<Prog>();
      launch_tile_kernel<Prog, true, smem>(dim3(tiles_w, tiles_h), s, b, maps);
      return 0;
    }
  }
  if constexpr (kHasOneFrame<Prog>) {
    if (a.frames <= 1) {
      launch_tile_kernel<OneFrame<Prog>, false, Prog::smem_bytes>(dim3(tiles_w, tiles_h), s, a, maps);
      return 0;
    }
  }
  launch_tile_kernel<Prog, false, Prog::smem_bytes>(dim3(tiles_w, tiles_h, a.frames > 0 ? a.frames : 1), s, a, maps);
  return 0;
}

// ------------------------------------------------------ persistent batches ---
// Program ids of a batch job (tile program and form; see batch.cu).
enum ProgId : int {
  kLite0 = 0,      // + (R-2)*2 + AR
  kThreeX0 = 6,    // + (R-2)*3 + CM
  kInt110 = 15,    // + (R-2)*3 + CM
  kLattice0 = 24,  // + (R-2)*3 + CM
  kZoom0 = 33,     // + (R-2)*6 + CM*2 + AR
  kLiteH0 = 45,    // fast form (FP16 LUT texels): as kLite0
  kThreeXH0 = 51,  //   as kThreeX0
  kZoomH0 = 60,    //   as kZoom0
  kNumProgs = 72
};

// One batch job: a frame's arguments, its place in its launch's tile range
// and (has_maps) the TMA maps of its input planes, read by the TMA unit
// from global memory.
struct DevJob {
  RavuArgs a;
  int prog;
  int tiles_w;
  int first_tile;  // prefix sum within its launch group
  int has_maps;
  TmaMaps maps;    // 64-byte aligned (CUtensorMap)
};
// every job's maps start on a 64-byte boundary of the (256-byte aligned) table
static_assert(sizeof(DevJob) % 64 == 0 && offsetof(DevJob, maps) % 64 == 0, "tensor maps must be 64-byte aligned");

// Persistent CTAs of one tile program: claim tile numbers from `counter`
// until `total`; a tile's job is the last whose first tile <= the number
// (binary search over the group's prefix sums); the job's arguments are
// copied to shared memory when the job changes.  Every job of a launch runs
// the same program, so register use and shared memory are the program's own.
template <class Prog>
__device__ __forceinline__ void persistent_body(const DevJob* __restrict__ jobs, int n_jobs, int total,
                                                int* counter) {
  extern __shared__ __align__(128) float4 psmem[];
  float* smem = reinterpret_cast<float*>(psmem);
  __shared__ RavuArgs s_args;
  // TMA staging of interior tiles (jobs with maps; programs with planes):
  // the landing area follows the program's shared memory; the mbarrier is
  // initialised before the first claim barrier, which orders it before use
  __shared__ __align__(8) unsigned long long mbar;
  if (Prog::kPlanes > 0 && threadIdx.x == 0) mbar_init(smem_u32(&mbar), 1);
  TmaCtx ctx{nullptr, smem_u32(&mbar),
             reinterpret_cast<unsigned char*>(psmem) + ((Prog::smem_bytes + 127) & ~(size_t)127), 0u, 0};
  // claim slots alternate between iterations: thread 0 fills slot (i+1)&1
  // while the other threads may still read slot i&1, and cannot get two
  // iterations ahead (the claim barrier of iteration i+1 holds it)
  __shared__ int s_item[2], s_job[2], s_tw[2], s_first[2];
  int loaded = -1;
  // thread 0 claims the next tile while the current one runs
  int next = threadIdx.x == 0 ? atomicAdd(counter, 1) : 0;
  for (int it = 0;; it ^= 1) {
    if (threadIdx.x == 0) {
      const int item = next;
      s_item[it] = item;
      if (item < total) {
        next = atomicAdd(counter, 1);
        int lo = 0, hi = n_jobs - 1;  // last job whose first tile <= item
        while (lo < hi) {
          const int mid = (lo + hi + 1) >> 1;
          if (jobs[mid].first_tile <= item) lo = mid; else hi = mid - 1;
        }
        s_job[it] = lo;
        s_tw[it] = jobs[lo].tiles_w;
        s_first[it] = jobs[lo].first_tile;
      }
    }
    __syncthreads();
    const int item = s_item[it];
    if (item >= total) break;
    const int job = s_job[it], tw = s_tw[it], first = s_first[it];
    if (job != loaded) {  // uniform: every thread reads the same slot
      // every thread is past the previous tile (the claim barrier above), so
      // s_args is free
      loaded = job;
      const int* src = reinterpret_cast<const int*>(&jobs[loaded].a);
      int* dst = reinterpret_cast<int*>(&s_args);
      for (int i = threadIdx.x; i < (int)(sizeof(RavuArgs) / 4); i += Prog::kThreads) dst[i] = src[i];
      ctx.map = jobs[loaded].has_maps ? jobs[loaded].maps.map : nullptr;
      __syncthreads();
    }
    const int t = item - first;
    // No barrier after the tile: the next tile's staging and argument copy
    // come after the next claim barrier, which every thread reaches only
    // when done with this tile.
    Prog::run(s_args, 0, (t % tw) * kTileW, (t / tw) * Prog::kRows, smem, Prog::kPlanes > 0 ? &ctx : nullptr);
  }
  tma_drain(&ctx);
}

template <class Prog>
__global__ void __launch_bounds__(Prog::kThreads) persistent_kernel(const DevJob* __restrict__ jobs, int n_jobs,
                                                                    int total, int* counter) {
  persistent_body<Prog>(jobs, n_jobs, total, counter);
}
template <class Prog>
__global__ void __maxnreg__(Prog::kMaxRegs) persistent_kernel_mr(const DevJob* __restrict__ jobs, int n_jobs,
                                                                 int total, int* counter) {
  persistent_body<Prog>(jobs, n_jobs, total, counter);
}

// Launch, occupancy query and TMA map encoding of one program's persistent
// kernel.
struct PersistentOps {
  void (*launch)(const DevJob* jobs, int n_jobs, int total, int* counter, int grid, cudaStream_t s);
  int (*fit)();                                // resident CTAs per SM
  bool (*encode)(RavuArgs* a, TmaMaps* maps);  // false: the job stages by clamped loads
};

// Shared memory of a persistent CTA: the program's, then (programs with
// planes) the TMA landing area of every plane.
template <class Prog>
constexpr size_t persistent_smem() {
  if constexpr (Prog::kPlanes > 0)
    return ((Prog::smem_bytes + 127) & ~(size_t)127) + tma_landing_bytes<Prog>();
  else
    return Prog::smem_bytes;
}

template <class Prog>
bool persistent_encode(RavuArgs* a, TmaMaps* maps) {
  if constexpr (Prog::kPlanes > 0) return encode_tma<Prog>(a, maps);
  else return false;
}

template <class Prog>
PersistentOps persistent_ops() {
  constexpr size_t kSmem = persistent_smem<Prog>();
  static_assert(kSmem <= 48 * 1024, "persistent tile program needs more than the default shared memory");
  static_assert(Prog::kRows == kBatchTileRows, "persistent batches number tiles of kBatchTileRows rows");
  if constexpr (Prog::kMaxRegs > 0) {
    return {[](const DevJob* j, int n, int total, int* c, int grid, cudaStream_t s) {
              persistent_kernel_mr<Prog><<<grid, Prog::kThreads, kSmem, s>>>(j, n, total, c);
            },
            []() {
              int fit = 0;
              cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, persistent_kernel_mr<Prog>, Prog::kThreads, kSmem);
              return fit;
            },
            persistent_encode<Prog>};
  } else {
    return {[](const DevJob* j, int n, int total, int* c, int grid, cudaStream_t s) {
              persistent_kernel<Prog><<<grid, Prog::kThreads, kSmem, s>>>(j, n, total, c);
            },
            []() {
              int fit = 0;
              cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, persistent_kernel<Prog>, Prog::kThreads, kSmem);
              return fit;
            },
            persistent_encode<Prog>};
  }
}

// The ops of program `prog` for plane dtype `dtype` (0 FP32, 1 FP16), or
// null members when `prog` is not the family's; defined beside the family's
// per-frame launchers.
PersistentOps persistent_ops_lite(int prog, int dtype);     // lite, 3x (ravu_lite.cu)
PersistentOps persistent_ops_lattice(int prog, int dtype);  // int11, lattice (ravu_lattice.cu)
PersistentOps persistent_ops_zoom(int prog, int dtype);     // zoom (ravu_zoom.cu)

}  // namespace pz
