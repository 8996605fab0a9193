// Per-model launches of the ravu-zoom(-ar) tile program (ravu_tiles.cuh) by
// tile height, and its persistent batch kernels.
#include "ravu_zoom_rows.cuh"

namespace pz {
namespace {

template <typename T>
PersistentOps zoom_ops(int prog) {
#define PZ_Z(id, R, CM, AR, H) \
  case id: return persistent_ops<ZoomTile<R, CM, AR, T, H, kBatchTileRows>>();
  switch (prog) {
    PZ_Z(kZoom0 + 0, 2, kLuma, false, false) PZ_Z(kZoom0 + 1, 2, kLuma, true, false)
    PZ_Z(kZoom0 + 2, 2, kYuv, false, false) PZ_Z(kZoom0 + 3, 2, kYuv, true, false)
    PZ_Z(kZoom0 + 4, 2, kRgb, false, false) PZ_Z(kZoom0 + 5, 2, kRgb, true, false)
    PZ_Z(kZoom0 + 6, 3, kLuma, false, false) PZ_Z(kZoom0 + 7, 3, kLuma, true, false)
    PZ_Z(kZoom0 + 8, 3, kYuv, false, false) PZ_Z(kZoom0 + 9, 3, kYuv, true, false)
    PZ_Z(kZoom0 + 10, 3, kRgb, false, false) PZ_Z(kZoom0 + 11, 3, kRgb, true, false)
    PZ_Z(kZoomH0 + 0, 2, kLuma, false, true) PZ_Z(kZoomH0 + 1, 2, kLuma, true, true)
    PZ_Z(kZoomH0 + 2, 2, kYuv, false, true) PZ_Z(kZoomH0 + 3, 2, kYuv, true, true)
    PZ_Z(kZoomH0 + 4, 2, kRgb, false, true) PZ_Z(kZoomH0 + 5, 2, kRgb, true, true)
    PZ_Z(kZoomH0 + 6, 3, kLuma, false, true) PZ_Z(kZoomH0 + 7, 3, kLuma, true, true)
    PZ_Z(kZoomH0 + 8, 3, kYuv, false, true) PZ_Z(kZoomH0 + 9, 3, kYuv, true, true)
    PZ_Z(kZoomH0 + 10, 3, kRgb, false, true) PZ_Z(kZoomH0 + 11, 3, kRgb, true, true)
  }
#undef PZ_Z
  return {nullptr, nullptr, nullptr};
}

int gcd(int a, int b) {
  while (b) {
    const int t = a % b;
    a = b;
    b = t;
  }
  return a;
}

template <int R, bool AR>
void launch_table(const RavuArgs& a, cudaStream_t s) {
  const int n = a.lut_rows / 9 * (int)(a.zpx.d * a.zpy.d) * ((zoom_texels<R>() + 1) / 2) * (AR ? 4 : 2);
  float4* out = const_cast<float4*>(a.ztab);
  if (a.lut_h) zoom_table_kernel<R, AR, true><<<(n + 127) / 128, 128, 0, s>>>(a, out);
  else zoom_table_kernel<R, AR, false><<<(n + 127) / 128, 128, 0, s>>>(a, out);
}

}  // namespace

// The table pays where it holds fewer entries than the frame has pixels (an
// entry costs about what a pixel saves) and the frame is large enough for one
// more launch (some 4 us).  Gain over weights per pixel, least (ravu-zoom-r2-rgb
// fast) to most (ravu-zoom-ar-r2 FP32), at 720p, 1080p and 2160p outputs, by
// pixels an entry: 8 1.05-1.97x, 18 1.10-2.46x, 32 1.09-2.40x, 72 1.13-2.73x, 3200
// (1.5x) 1.28-2.85x; 1080p to 1.5x ravu-zoom-ar-r2-rgb 187 against 274 us.  Tables
// beyond L2 still pay: ravu-zoom-ar-r3 to 2160p at 8 pixels an entry, 348 MB, 706
// against 1087 us.  But they are scratch of every call: kTableMax leaves every
// output up to 2160p its table and bounds the larger ones', up to 42 bytes a pixel
// (1.4 GB at 7680x4320).  Scales of no simple ratio have as many phases as pixels
// and take none.
constexpr size_t kTableMax = (size_t)512 << 20;

size_t zoom_table_bytes(int radius, bool ar, int keys, int W, int H, int OW, int OH, FastDiv* px,
                        FastDiv* py) {
  *px = fast_div(OW / gcd(W, OW));
  *py = fast_div(OH / gcd(H, OH));
  const long long entries = (long long)keys * px->d * py->d, pixels = (long long)OW * OH;
  if (pixels < 1 << 19 || entries * 8 > pixels) return 0;
  const uint32_t e = radius == 2 ? (ar ? zoom_entry<2, true>() : zoom_entry<2, false>())
                                 : (ar ? zoom_entry<3, true>() : zoom_entry<3, false>());
  const size_t bytes = (size_t)entries * e * sizeof(float4);
  return bytes <= kTableMax ? bytes : 0;
}

int launch_zoom_table(const RavuArgs& a, int radius, bool ar, cudaStream_t s) {
  if (radius == 2) ar ? launch_table<2, true>(a, s) : launch_table<2, false>(a, s);
  else ar ? launch_table<3, true>(a, s) : launch_table<3, false>(a, s);
  return 0;
}

PersistentOps persistent_ops_zoom(int prog, int dtype) {
  return dtype == 0 ? zoom_ops<float>(prog) : zoom_ops<__half>(prog);
}

int launch_zoom(const RavuArgs& a, int radius, int cm, bool ar, int dtype, cudaStream_t s) {
  switch (a.tile_rows) {
    case 4: return launch_zoom_rows<4>(a, radius, cm, ar, dtype, s);
    case 16: return launch_zoom_rows<16>(a, radius, cm, ar, dtype, s);
    default: return launch_zoom_rows<8>(a, radius, cm, ar, dtype, s);
  }
}

}  // namespace pz
