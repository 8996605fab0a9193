// NNEDI3 doubling pass on the 5th-generation tensor cores (tcgen05).
//
// Reference arithmetic: nnedi3-nns16-win8x4.hook:20-50 (normalise the 8xK
// window, nns neuron pairs, exp-weighted Elliott blend); pass geometry as in
// the CUDA-core kernel (nnedi3_simt.cu).
//
// One persistent CTA per SM: NG groups of 4 warps and one MMA-issuing warp
// per group.  The groups share the weight operand B in shared memory (one
// bulk copy per CTA); each works on its own M-tiles of 128 interpolated
// pixels (4 rows x 32 columns, one thread and one TMEM lane per pixel):
//   1. the window tile is staged in shared memory (its loads are in flight
//      while the previous tile's neurons run); each thread normalises its
//      pixel's window, x_hat = (x - mean) * invstd, into one row of A
//      [128 x KP] FP16 (K-major, no-swizzle core matrices: 8 rows x 16 bytes,
//      LBO = 128 B between K-neighbours, SBO = KP*16 B between 8-row groups),
//      followed by mean*invstd and ones, which multiply B's columns of weight
//      sums and biases;
//   2. the group's issuing thread runs tcgen05.mma.kind::f16 (M = 128, N = 64,
//      K = 16) for 32-neuron chunks into two alternating TMEM accumulators (or
//      N = 128 for 64-neuron chunks into one: tc_chunk) and commits each to an
//      mbarrier;
//   3. each warp reads its 32 TMEM lanes with tcgen05.ld.32x32b and runs the
//      blend in FP32: e = exp2(s1) (softmax rows of B are in log2 units),
//      wsum += e, vsum += e * s2 / (1 + |s2|).
// Every hand-off is an mbarrier between the warps that need it (A written,
// chunk accumulated, chunk read); the one barrier among a group's warps is
// the window tile's, once per tile.  A is free once the last chunk's MMAs are
// done, so the next tile is normalised before the last chunk is blended: its
// first MMAs run under that blend.
//
// SPLIT (the plain FP32 form): every operand value is two FP16 pieces, hi +
// lo, and a chunk is three products, A_lo B_hi + A_hi B_lo + A_hi B_hi in FP32, the
// small ones first.  The pieces hold 22 bits of a value at least, but a low piece
// ends at FP16's 2^-24: x_hat, whose root mean square is 1, keeps an absolute error
// of 2^-25 below 2^-3 (scaled by 16, which removes that, the error against 64 bits
// is the same); in B, which a power of two of the model's scales, that is 2^-39 of
// the largest value.  A_lo B_lo, at most 2^-22 of a product, is left out.  The
// sums, rounded once a K step instead of once a term, more than make up for it:
// the error against 64 bits is 0.5-0.65x the CUDA cores' (launch_nnedi3).
//
// Bound by issue and latency in the blend (12 packed or scalar instructions
// and 6 MUFU for four neurons) at four warps a scheduler (60 % issue, 37 % MUFU,
// 23 % tensor pipe; 96 registers and 512 TMEM columns allow no fifth group).
// 1080p to 2160p, nns128 8x6: 325 us fast (384 us with scalar sums over neuron
// pairs and rolled chunks; 438 us as four CTAs an SM, each with its own copy of B
// and a CTA barrier per chunk), 441 us split (523 us; 4919 us on the CUDA cores);
// nns256 8x6 at 720p 240 us fast (443 us: two CTAs an SM had room).
//
// Every mbarrier wait is bounded (kWaitNs of %globaltimer).  A wait that runs
// out sets the CTA's abort flag: from then on nobody waits, nothing is stored,
// and the loops run out through the same barriers; before the tensor memory
// is freed, each issuing thread commits once more and waits (bounded) until
// its MMAs have completed, so no MMA can still write the freed columns; the
// failure is reported as kErrWaitTimeout in the device error word.
#include "async.cuh"
#include "kernels.h"

namespace pz {
namespace {

constexpr int kGroup = 128;  // threads per group: 4 warps, one TMEM lane quarter each

// tcgen05 shared-memory matrix descriptor, no swizzle, K-major.
__device__ __forceinline__ uint64_t smem_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);
  d |= (uint64_t)((lbo >> 4) & 0x3FFFu) << 16;
  d |= (uint64_t)((sbo >> 4) & 0x3FFFu) << 32;
  d |= (uint64_t)1 << 46;  // descriptor version for tcgen05
  return d;                // base offset 0, relative LBO, layout 0 = no swizzle
}

// Instruction descriptor, kind::f16: D = F32, A = B = F16, both K-major.
__host__ __device__ constexpr uint32_t instr_desc(int M, int N) {
  return (1u << 4) | (0u << 7) | (0u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void mma_f16(uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem_d),
      "l"(a), "l"(b), "r"(idesc), "r"(acc));
}

__device__ __forceinline__ void mma_commit(uint32_t mbar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar)
               : "memory");
}

// 16 columns of this warp's lanes; the values are valid after tmem_wait16.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]), "=f"(v[8]),
        "=f"(v[9]), "=f"(v[10]), "=f"(v[11]), "=f"(v[12]), "=f"(v[13]), "=f"(v[14]), "=f"(v[15])
      : "r"(taddr));
}

// Wait for this thread's TMEM loads; the operands tie the loaded registers to
// the wait, so that no use of them can be scheduled before it.
__device__ __forceinline__ void tmem_wait16(float (&a)[16], float (&b)[16]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+f"(a[0]), "+f"(a[1]), "+f"(a[2]), "+f"(a[3]), "+f"(a[4]), "+f"(a[5]), "+f"(a[6]), "+f"(a[7]),
                 "+f"(a[8]), "+f"(a[9]), "+f"(a[10]), "+f"(a[11]), "+f"(a[12]), "+f"(a[13]), "+f"(a[14]), "+f"(a[15]),
                 "+f"(b[0]), "+f"(b[1]), "+f"(b[2]), "+f"(b[3])
               :
               : "memory");
  asm volatile("" : "+f"(b[4]), "+f"(b[5]), "+f"(b[6]), "+f"(b[7]), "+f"(b[8]), "+f"(b[9]), "+f"(b[10]), "+f"(b[11]),
                    "+f"(b[12]), "+f"(b[13]), "+f"(b[14]), "+f"(b[15]));
}

__device__ __forceinline__ float exp2f_approx(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

__device__ __forceinline__ float rcp_approx(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ void mbar_arrive(uint32_t mbar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(mbar) : "memory");
}

__device__ __forceinline__ float to_float(float v) { return v; }
__device__ __forceinline__ float to_float(__half v) { return __half2float(v); }

// Barrier among the 128 threads of group g (named barriers 1..4; 0 is the CTA's).
__device__ __forceinline__ void group_sync(int g) {
  asm volatile("bar.sync %0, %1;" ::"r"(g + 1), "n"(kGroup) : "memory");
}

// Neurons per chunk.  Split operands are bound by the MMAs, whose A is read from
// shared memory once per instruction whatever its N: 64 neurons (N = 128) take
// two thirds of the shared-memory time of 32 (N = 64), and then one accumulator
// per group (its MMAs wait for the blend's last read) is all that fits four
// groups.  FP32, chunks of 32 / 64: nns128 8x6 at 1080p 486 / 444 us, nns128 8x4 at
// 720p 183 / 177, nns256 8x4 at 1080p 670 / 603, nns64 8x6 321 / 298; but nns64
// 8x4, with little to multiply, 255 / 266, and nns256 8x6, two groups, at 720p 464 /
// 483.  The fast form, bound by the blend, keeps 32 and two accumulators.
constexpr int tc_chunk(int nns, int wh, bool split) {
  const bool wide = split && (nns == 128 || (nns == 256 && wh == 4) || (nns == 64 && wh == 6));
  return nns < 32 ? nns : (wide ? 64 : 32);
}

// Shape of one instantiation.
template <int WH, int NNS, bool XP, bool SPLIT>
struct TcShape {
  static constexpr int NT = 8 * WH;                   // window taps
  static constexpr int KP = (NT + 4 + 15) / 16 * 16;  // K: taps, mean term, bias pieces, zero pad
  static constexpr int NC = tc_chunk(NNS, WH, SPLIT);     // neurons per chunk
  static constexpr int NBUF = NC == 64 ? 1 : 2;       // chunk buffers per group
  static constexpr int NCH = NNS / NC;                // chunks per tile
  static constexpr int CCOL = 2 * NC;                 // TMEM columns per chunk buffer
  static constexpr int NP = SPLIT ? 2 : 1;            // FP16 pieces per operand value
  static constexpr int DY0 = -(WH / 2 - 1);
  static constexpr int OX0 = XP ? DY0 : -3, OX1 = XP ? WH / 2 : 4;
  static constexpr int OY0 = XP ? -3 : DY0, OY1 = XP ? 4 : WH / 2;
  static constexpr int TW = 32 + OX1 - OX0, TH = 4 + OY1 - OY0;
  static constexpr uint32_t BPIECE = 2 * NNS * KP * 2;  // bytes of one piece of B / of a group's A
  static constexpr uint32_t APIECE = 128 * KP * 2;
  static constexpr uint32_t GROUP_BYTES = NP * APIECE + (TW * TH * 4 + 127) / 128 * 128;
  static constexpr uint32_t kSmemMax = 227 * 1024 - 1024;  // less the static shared memory
  // groups per CTA: four fill the SM's tensor memory (128 columns each, two
  // 32-neuron buffers); fewer where the split operands leave less room
  static constexpr int fit = (int)((kSmemMax - NP * BPIECE) / GROUP_BYTES);
  static constexpr int NG = fit < 4 ? fit : 4;
  static constexpr int THREADS = NG * (kGroup + 32);
  static constexpr uint32_t TCOLS = NG * NBUF * CCOL <= 64 ? 64 : (NG * NBUF * CCOL <= 128 ? 128 : (NG * NBUF * CCOL <= 256 ? 256 : 512));
  static constexpr uint32_t SMEM = NP * BPIECE + NG * GROUP_BYTES;
  static_assert(NNS % NC == 0 && NC % 16 == 0, "neuron count must be a multiple of 16");
  static_assert(NG >= 1 && NG * NBUF * CCOL <= 512, "operands must fit shared and tensor memory");
};

// The tiles of a launch: 32 x 4 pixels, row by row, frame after frame.
struct Tiles {
  FastDiv x, y;  // tiles per row, rows of tiles per frame (a division costs as much as a neuron pair)
  int n;
};

// Neurons are processed in chunks of NC: chunk k's accumulator holds NC
// softmax-branch and NC Elliott-branch columns; the MMA of the next chunk for
// an accumulator is issued as soon as every warp of the group has read it.
// Operand B is stored chunk-major: rows [2*NC*k, 2*NC*k + NC) are the
// softmax weights of neurons k*NC.., the next NC rows their Elliott weights.
template <int WH, int NNS, bool XP, typename T, bool SPLIT>
__global__ void __launch_bounds__(TcShape<WH, NNS, XP, SPLIT>::THREADS, 1) nn_tc_kernel(const __grid_constant__ NnArgs p, const __grid_constant__ Tiles tiles) {
  using S = TcShape<WH, NNS, XP, SPLIT>;
  constexpr int NT = S::NT, KP = S::KP, NC = S::NC, NCH = S::NCH, CCOL = S::CCOL, NG = S::NG, NBUF = S::NBUF;
  constexpr int TW = S::TW, TH = S::TH;
  constexpr uint32_t SBO = KP * 16;  // bytes between 8-row groups (A and B)
  constexpr uint32_t LBO = 128;      // bytes between K-adjacent core matrices

  extern __shared__ __align__(1024) unsigned char smem[];
  unsigned char* sB = smem;  // [NP][2*NNS x KP] f16, then per group [NP][128 x KP] f16 and the window tile
  struct GroupBars {
    unsigned long long afull, full[2], empty[2], drain;
  };
  __shared__ __align__(8) GroupBars bars[NG];
  __shared__ __align__(8) unsigned long long bbar;
  __shared__ uint32_t tmem_base;
  __shared__ int abort_flag;
  volatile int* const aborted = &abort_flag;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    for (int g = 0; g < NG; g++) {
      mbar_init(smem_u32(&bars[g].afull), 4);  // one arrival per warp of the group
      for (int b = 0; b < 2; b++) {
        mbar_init(smem_u32(&bars[g].full[b]), 1);   // tcgen05.commit
        mbar_init(smem_u32(&bars[g].empty[b]), 4);  // one arrival per warp
      }
      mbar_init(smem_u32(&bars[g].drain), 1);
    }
    mbar_init(smem_u32(&bbar), 1);
    abort_flag = 0;
    fence_async_smem();
    // the weight operand, one bulk copy (read by the MMAs only)
    mbar_arrive_expect_tx(smem_u32(&bbar), S::NP * S::BPIECE);
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(sB)),
        "l"(reinterpret_cast<uint64_t>(SPLIT ? p.wts_s : p.wts_h)), "r"(S::NP * S::BPIECE), "r"(smem_u32(&bbar))
        : "memory");
  }
  // the row pass's CTAs may still run (they hold the tensor memory) until here
  pdl_wait();
  pdl_trigger();
  if (warp == 0) {
    __syncwarp();
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base)),
                 "r"(S::TCOLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_base;
  const int ntiles = tiles.n;
  const int stride = NG * gridDim.x;  // tiles go over the SMs first, then over each SM's groups

  // true once the phase has completed; false when the CTA has given up
  auto wait = [&](const unsigned long long* bar, uint32_t parity) {
    const uint32_t mb = smem_u32(bar);
    if (mbar_try(mb, parity)) return true;
    const unsigned long long t0 = globaltimer();
    while (!*aborted) {
      if (mbar_try(mb, parity)) return true;
      if (globaltimer() - t0 > kWaitNs) *aborted = 1;
    }
    return false;
  };

  if (warp >= 4 * NG) {
    // ---- the MMA-issuing warp of group g (one thread)
    const int g = warp - 4 * NG;
    if (lane == 0) {
      GroupBars& B = bars[g];
      constexpr uint32_t IDESC = instr_desc(128, CCOL);
      const uint32_t a_addr = smem_u32(sB + S::NP * S::BPIECE + g * S::GROUP_BYTES), b_addr = smem_u32(sB);
      const uint32_t dcol = tmem + g * NBUF * CCOL;
      bool ok = wait(&bbar, 0u);
      int c = 0, it = 0;  // chunks and tiles issued so far
      for (int t = g * gridDim.x + blockIdx.x; ok && t < ntiles; t += stride, it++) {
        if (!(ok = wait(&B.afull, it & 1))) break;
        for (int k = 0; k < NCH; k++, c++) {
          const int b = c % NBUF, u = c / NBUF;
          if (u > 0 && !(ok = wait(&B.empty[b], (u - 1) & 1))) break;
          tc_fence_after();
          // D[b] = A x B[chunk]^T over the whole K; completion on full[b]
          uint32_t acc = 0;
#pragma unroll
          for (int pr = 0; pr < (SPLIT ? 3 : 1); pr++) {
            const uint32_t ap = a_addr + (SPLIT && pr == 0 ? S::APIECE : 0);
            const uint32_t bp = b_addr + (SPLIT && pr == 1 ? S::BPIECE : 0) + (uint32_t)k * (CCOL / 8) * SBO;
#pragma unroll
            for (int ks = 0; ks < KP / 16; ks++) {
              mma_f16(dcol + b * CCOL, smem_desc(ap + ks * 2 * LBO, LBO, SBO), smem_desc(bp + ks * 2 * LBO, LBO, SBO),
                      IDESC, acc);
              acc = 1;
            }
          }
          mma_commit(smem_u32(&B.full[b]));
        }
      }
      // no MMA may still write tensor memory when it is freed, nor B still land
      mma_commit(smem_u32(&B.drain));
      if (!mbar_wait_bounded(smem_u32(&B.drain), 0u)) *aborted = 1;
      if (g == 0 && !mbar_wait_bounded(smem_u32(&bbar), 0u)) *aborted = 1;
    }
    __syncwarp();
  } else {
    // ---- a group's warps: windows into A, accumulators into pixels
    const int g = warp >> 2, m = tid & (kGroup - 1), py = warp & 3;
    GroupBars& B = bars[g];
    unsigned char* sA = sB + S::NP * S::BPIECE + g * S::GROUP_BYTES;
    float* tile = reinterpret_cast<float*>(sA + S::NP * S::APIECE);
    const T* in = static_cast<const T*>(p.in);
    T* out = static_cast<T*>(p.out);

    // the window tile of a later tile, loaded into registers ahead of use
    constexpr int PF = (TW * TH + kGroup - 1) / kGroup;
    float pre[PF];
    // frame, row and column of tile t
    auto locate = [&](int t, int& f, int& y0) {
      const int row = tiles.x(t);
      f = tiles.y(row);
      y0 = (row - f * (int)tiles.y.d) * 4;
      return (t - row * (int)tiles.x.d) * 32;
    };
    auto prefetch = [&](int t) {
      if (t >= ntiles) return;
      int f, py0;
      const int px0 = locate(t, f, py0);
      const T* src = in + f * p.in_frame;
#pragma unroll
      for (int r = 0; r < PF; r++) {
        const int i = m + r * kGroup;
        if (i < TW * TH) {
          const int ty = i / TW, tx = i % TW;
          const int gx = clampi(px0 + S::OX0 + tx, 0, p.W - 1), gy = clampi(py0 + S::OY0 + ty, 0, p.H - 1);
          pre[r] = to_float(src[(size_t)gy * p.in_pitch + gx]);  // plain loads: pdl_wait
        }
      }
    };
    // a tile's pixel: window mean and standard deviation, the pixel copied through
    struct Pixel {
      float mean, stdv, orig;
    };
    // stage the prefetched window tile and write this thread's row of A.  All
    // warps of the group have read the tile before (their arrivals on afull
    // precede the MMAs whose completion brought this warp here).
    auto normalise = [&]() {
#pragma unroll
      for (int r = 0; r < PF; r++) {
        const int i = m + r * kGroup;
        if (i < TW * TH) tile[i] = pre[r];
      }
      group_sync(g);
      // taps in FP32x2 pairs; 8 independent partial sums (one per window
      // column): no serial chain of NT steps
      Pixel px;
      float2 xv[NT / 2];
#pragma unroll
      for (int t = 0; t < NT; t++) {
        const int dx = t % 8 - 3, dy = t / 8 + S::DY0;
        const int ox = XP ? dy : dx, oy = XP ? dx : dy;
        const float v = tile[(py + oy - S::OY0) * TW + lane + ox - S::OX0];
        if (t % 2 == 0) xv[t / 2].x = v;
        else xv[t / 2].y = v;
      }
      px.orig = tile[(py - S::OY0) * TW + lane - S::OX0];
      float2 ps[4];
#pragma unroll
      for (int c = 0; c < 4; c++) ps[c] = xv[c];
#pragma unroll
      for (int t = 4; t < NT / 2; t++) ps[t % 4] = __fadd2_rn(ps[t % 4], xv[t]);
      auto total = [&]() {
        const float2 q = __fadd2_rn(__fadd2_rn(ps[0], ps[1]), __fadd2_rn(ps[2], ps[3]));
        return q.x + q.y;
      };
      px.mean = total() * (1.0f / NT);
#pragma unroll
      for (int t = 0; t < NT / 2; t++) xv[t] = __fadd2_rn(xv[t], make_float2(-px.mean, -px.mean));
#pragma unroll
      for (int c = 0; c < 4; c++) ps[c] = __fmul2_rn(xv[c], xv[c]);
#pragma unroll
      for (int t = 4; t < NT / 2; t++) ps[t % 4] = __ffma2_rn(xv[t], xv[t], ps[t % 4]);
      const float var = total() * (1.0f / NT);
      const float invstd = var >= kFltEps ? (SPLIT ? 1.0f / sqrtf(var) : rsqrtf(var)) : 0.0f;
      px.stdv = var * invstd;
      // A row: [x_hat (NT), mean * invstd, 1, 1, 1, 0...].  A mean term beyond
      // FP16's range is cut: the output is then clamped whatever the neurons
      // say (|mean| > 22 against a deviation below mean / 60000)
      const float mterm = fminf(fmaxf(px.mean * invstd, -60000.0f), 60000.0f);
      unsigned char* row = sA + (m >> 3) * SBO + (m & 7) * 16;
#pragma unroll
      for (int kc = 0; kc < KP / 8; kc++) {
        __half2 h[4], l[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
          const int t = 8 * kc + 2 * j;
          const float2 v = t < NT ? __fmul2_rn(xv[t < NT ? t / 2 : 0], make_float2(invstd, invstd))
                                  : (t == NT ? make_float2(mterm, 1.0f)
                                             : (t == NT + 2 ? make_float2(1.0f, 1.0f) : make_float2(0.0f, 0.0f)));
          h[j] = __floats2half2_rn(v.x, v.y);
          if (SPLIT) {
            const float2 f = __half22float2(h[j]);
            l[j] = __floats2half2_rn(v.x - f.x, v.y - f.y);
          }
        }
        *reinterpret_cast<uint4*>(row + kc * LBO) = *reinterpret_cast<uint4*>(h);
        if (SPLIT) *reinterpret_cast<uint4*>(row + S::APIECE + kc * LBO) = *reinterpret_cast<uint4*>(l);
      }
      fence_async_smem();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&B.afull));
      return px;
    };

    int t = g * gridDim.x + blockIdx.x;
    Pixel cur{}, nxt{};
    if (t < ntiles) {
      prefetch(t);
      cur = normalise();
      prefetch(t + stride);
    }
    const uint32_t lane_addr = tmem + g * NBUF * CCOL + ((uint32_t)(py * 32) << 16);
    const float one = SPLIT ? p.split_one : 1.0f, unit = SPLIT ? p.split_unit : 1.0f;
    int c = 0;
    for (; t < ntiles; t += stride) {
      float2 wsum = make_float2(0.0f, 0.0f), vsum = wsum;
      // the accumulators in steps of 16 neurons, both branches' columns
      float s1[2][16], s2[2][16];
      constexpr int STEPS = NC / 16;
      // a step's loads are in flight during the arithmetic of the step before,
      // across chunks too but for the tile's last (the next tile is normalised
      // before it); the chunks are unrolled, so that no load in flight crosses a
      // loop's edge.  nns128 8x6 fast, 1080p: rolled 353 us, unrolled 334, and ahead
      // 330.  Split, the MMAs bound it: ahead loses 2 %, and so does unrolling
      // from four chunks on (nns64 8x4 at 480p, two chunks: 67 rolled, 63 unrolled).
      constexpr bool AHEAD = STEPS == 2 && !SPLIT;
      constexpr int UNROLL = SPLIT && NCH > 2 ? 1 : NCH;
      auto load = [&](int b, int q) {
        tmem_ld16(lane_addr + b * CCOL + 16 * q, s1[q & 1]);
        tmem_ld16(lane_addr + b * CCOL + NC + 16 * q, s2[q & 1]);
      };
#pragma unroll UNROLL
      for (int k = 0; k < NCH; k++, c++) {
        const int b = NBUF == 1 ? 0 : (NCH % 2 == 0 ? k & 1 : c & 1);
        if (!AHEAD || k == 0 || k == NCH - 1) {  // not in flight yet
          (void)wait(&B.full[b], (c / NBUF) & 1);
          tc_fence_after();
          if (k == NCH - 1 && t + stride < ntiles) {
            nxt = normalise();
            prefetch(t + 2 * stride);
          }
          load(b, 0);
        }
#pragma unroll
        for (int q = 0; q < STEPS; q++) {
          tmem_wait16(s1[q & 1], s2[q & 1]);
          if (q + 1 < STEPS) {
            load(b, q + 1);
          } else {  // this warp has read buffer b
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&B.empty[b]));
            if (AHEAD && k + 1 < NCH - 1) {
              (void)wait(&B.full[b ^ 1], ((c + 1) >> 1) & 1);
              tc_fence_after();
              load(b ^ 1, 0);
            }
          }
          // sum of e s / (1 + |s|): neurons j and j+2 (and j+1, j+3) share one
          // reciprocal, of the product of their denominators
#pragma unroll
          for (int j = 0; j < 16; j += 4) {
            float2 n[2], d[2];
#pragma unroll
            for (int h = 0; h < 2; h++) {
              const int i = j + 2 * h;
              float2 l = make_float2(s1[q & 1][i], s1[q & 1][i + 1]);
              if (SPLIT) l = __fmul2_rn(l, make_float2(unit, unit));
              const float2 e = make_float2(exp2f_approx(l.x), exp2f_approx(l.y));
              d[h] = make_float2(one + fabsf(s2[q & 1][i]), one + fabsf(s2[q & 1][i + 1]));
              n[h] = __fmul2_rn(e, make_float2(s2[q & 1][i], s2[q & 1][i + 1]));
              wsum = __fadd2_rn(wsum, e);
            }
            const float2 dd = __fmul2_rn(d[0], d[1]);
            const float2 nn = __ffma2_rn(n[0], d[1], __fmul2_rn(n[1], d[0]));
            vsum = __ffma2_rn(nn, make_float2(rcp_approx(dd.x), rcp_approx(dd.y)), vsum);
          }
        }
      }
      int f, gy;
      const int gx = locate(t, f, gy) + lane;
      gy += py;
      T* dst = out + f * p.out_frame;
      if (gx < p.W && gy < p.H && !*aborted) {
        const float ws = wsum.x + wsum.y, vs = vsum.x + vsum.y;
        float v = clampf(cur.mean + 5.0f * vs / ws * cur.stdv, 0.0f, 1.0f);
        // The split blend multiplies e by s (1 + |s|) and the square of its scale
        // before it divides: from logits of about 70 on that is infinite, and stays
        // so or turns to NaN in the sums, where e itself is good to 88; and e is
        // flushed below 2^-126, which 256 neurons may feel where their sum is below
        // 2^-90 (logits below -62).  Such a window's pixel is marked by a NaN, which is
        // stored for no other, and launch_nnedi3_marked takes it in plain FP32.
        // Forming s / (1 + |s|) first and e as the square of 2^(l/2) instead keeps
        // every pixel in range, but costs all of them (nns128 8x6 at 1080p 476 us,
        // 438) and 1 % of accuracy; an FP32 pixel called from here 454 us; the mark 441.
        if (SPLIT && (ws < 0x1p-90f || !(fabsf(vs) < INFINITY)) && fabsf(cur.mean) < INFINITY &&
            fabsf(cur.stdv) < INFINITY)
          v = NAN;
        if (XP) {
          stp2(dst + (size_t)gy * p.out_pitch + 2 * gx, cur.orig, v);
        } else {
          stp(dst + (size_t)(2 * gy) * p.out_pitch + gx, cur.orig);
          stp(dst + (size_t)(2 * gy + 1) * p.out_pitch + gx, v);
        }
      }
      cur = nxt;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (*aborted && tid == 0) atomicCAS(p.err, 0, kErrWaitTimeout);
  if (warp == 0) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(S::TCOLS));
  }
}

template <int WH, int NNS, bool XP, typename T, bool SPLIT>
int launch_one(const NnArgs& a, cudaStream_t s) {
  using S = TcShape<WH, NNS, XP, SPLIT>;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return -95;
  auto kern = nn_tc_kernel<WH, NNS, XP, T, SPLIT>;
  static bool configured[64] = {};  // per instantiation and device
  if (!configured[dev]) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::SMEM) != cudaSuccess)
      return -5;
    configured[dev] = true;
  }
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  Tiles tiles{fast_div((a.W + 31) / 32), fast_div((a.H + 3) / 4), 0};
  tiles.n = (int)(tiles.x.d * tiles.y.d) * (a.frames > 0 ? a.frames : 1);
  launch_kernel(kern, dim3(tiles.n < sms ? tiles.n : sms), S::THREADS, S::SMEM, s, a.after, a, tiles);
  return 0;
}

template <int WH, bool XP, typename T, bool SPLIT>
int dispatch_nns(const NnArgs& a, cudaStream_t s) {
  switch (a.nns) {
    case 16: return launch_one<WH, 16, XP, T, SPLIT>(a, s);
    case 32: return launch_one<WH, 32, XP, T, SPLIT>(a, s);
    case 64: return launch_one<WH, 64, XP, T, SPLIT>(a, s);
    case 128: return launch_one<WH, 128, XP, T, SPLIT>(a, s);
    case 256: return launch_one<WH, 256, XP, T, SPLIT>(a, s);
  }
  return -95;
}

template <typename T, bool SPLIT>
int launch_t(const NnArgs& a, bool xp, cudaStream_t s) {
  if (a.win_h == 4) return xp ? dispatch_nns<4, true, T, SPLIT>(a, s) : dispatch_nns<4, false, T, SPLIT>(a, s);
  if (a.win_h == 6) return xp ? dispatch_nns<6, true, T, SPLIT>(a, s) : dispatch_nns<6, false, T, SPLIT>(a, s);
  return -95;
}

}  // namespace

bool nnedi3_tc_supported(int nns, int win_h) {
  return (nns == 16 || nns == 32 || nns == 64 || nns == 128 || nns == 256) && (win_h == 4 || win_h == 6);
}

int nnedi3_tc_chunk(int nns, int win_h, bool split) { return tc_chunk(nns, win_h, split); }

int launch_nnedi3_tc(const NnArgs& a, bool xpass, int dtype, cudaStream_t s) {
  if (!a.wts_h || !a.err) return -22;
  return dtype == 0 ? launch_t<float, false>(a, xpass, s) : launch_t<__half, false>(a, xpass, s);
}

int launch_nnedi3_split(const NnArgs& a, bool xpass, int dtype, cudaStream_t s) {
  if (!a.wts_s || !a.err) return -22;
  return dtype == 0 ? launch_t<float, true>(a, xpass, s) : launch_t<__half, true>(a, xpass, s);
}

}  // namespace pz
