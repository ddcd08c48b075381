// The robust tile kernels of up to 49 samples, their plan hook and dispatch
// (the wider ones instantiate in robust_tile_wide.cu).
#include "robust_tile.cuh"

namespace ndf {

cudaError_t launch_robust_tile_wide(const Plan& p, const float* in, float* out, cudaStream_t s);

// The tile kernel takes float32 windows of up to 128 samples over 1-D to 3-D
// arrays for the MAD, the mode estimators and sigma clipping. Clipping
// multipliers below 1/2 (0 among them) stay with the general kernel: the
// error bounds count on limits of at least half a spread; so does the
// biweight, whose sums need every sample in float64.
bool robust_tile_configure(Plan& p) {
  p.robust_width = 0;
  const RobustArgs& ra = p.robust;
  if (p.dtype != 0 || p.ndim < 1 || p.ndim > 3 || p.r.count < 1 || p.r.count > 128) return false;
  if (ra.kind >= kRobustSigmaMean) {
    auto fits = [](double sigma) { return sigma >= 0.5 && sigma <= 1e6; };
    if (!fits(ra.lower) || !fits(ra.upper) || ra.clip_min_count < 1) return false;
  } else if (ra.kind != kRobustMad && ra.kind != kRobustMode) {
    return false;
  }
  unsigned long long volume = 1;
  for (long long n : p.size) {
    volume *= (unsigned long long)n;
    if (volume > (1ull << 20)) return false;
  }
  plan_setup_tile(p);
  const Geom3& g = p.tile.g;
  Tile& t = p.tile.t;
  // 512 outputs per block share a halo; arrays that would leave SMs without a
  // block take 128. Tiles are 32 columns wide, narrower over arrays of fewer and
  // wider over arrays of few rows: 32 columns over one of 2 or 3 left the MAD
  // slower than one window per thread of the general kernel (5 x 5 x 1 over
  // 400 x 400 x 3: 0.22 ms there, 0.32 in tiles of 32 columns, 0.064 in tiles of 4).
  auto covering = [](long long n, int most) {
    int side = 1;
    while (side < n && side < most) side *= 2;
    return side;
  };
  auto shape = [&](int outputs) {
    t.TW = covering(g.W, 32);
    t.TH = covering(g.H, outputs / t.TW);
    t.TW = covering(g.W, outputs / t.TH);
    t.SW = t.TW + g.kw - 1;
    t.SH = t.TH + g.kh - 1;
    t.tiles_x = (g.W + t.TW - 1) / t.TW;
    t.tiles_y = (g.H + t.TH - 1) / t.TH;
    t.tiles = t.tiles_x * t.tiles_y * g.D;
  };
  shape(512);
  if (t.tiles < 4ll * p.sm_count) shape(128);
  if (t.tiles >= (1ll << 31)) return false;
  // A stack of tiny slices fills few of a block's threads. The general kernel breaks
  // even at about an eighth of them for the MAD (20,000 slices of 4 x 4, 3 x 3 windows:
  // 0.11 ms there, 0.14 in tiles), at a sixteenth for clipping and the mode (there 0.55
  // and 0.24, 0.10 and 0.17 in tiles).
  const long long threads = t.tiles * std::max(t.TW * t.TH, robust_tile::kT);
  if (p.n_out * (ra.kind == kRobustMad ? 7 : 14) < threads) return false;
  static const int widths[] = {9, 16, 25, 32, 49, 64, 81, 128};
  int width = 0;
  for (int w : widths)
    if (width == 0 && p.r.count <= w) width = w;
  p.smem_bytes = tile_select_smem(p, t);
  if (p.smem_bytes + 16 + (size_t)width * robust_tile::kT * sizeof(float) > robust_tile::kRobustTileSmem) return false;
  p.robust_width = width;
  return true;
}

cudaError_t launch_robust_tile(const Plan& p, const float* in, float* out, cudaStream_t s) {
  switch (p.robust_width) {
    case 9: return robust_tile::launch_kind<9>(p, in, out, s);
    case 16: return robust_tile::launch_kind<16>(p, in, out, s);
    case 25: return robust_tile::launch_kind<25>(p, in, out, s);
    case 32: return robust_tile::launch_kind<32>(p, in, out, s);
    case 49: return robust_tile::launch_kind<49>(p, in, out, s);
    default: return launch_robust_tile_wide(p, in, out, s);
  }
}

}  // namespace ndf
