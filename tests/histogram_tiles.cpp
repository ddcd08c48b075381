// Prints the histogram kernel's tile of each window on stdin, as the library's
// host code chooses it (no device): one line "D H W kd kh kw hole double" per
// window, "hole" being the flat position of the one missing tap of a footprint
// (-1: a full box). Reads as "TW TH TZ sdec in_smem smem entries"; TW is 0 where
// the kernel does not take the window. An argument gives the device's SMs (152).
#include <cstdio>
#include <cstdlib>

#include "../ndfiltrs_gb300/csrc/plan.h"

int main(int argc, char** argv) {
  long long D, H, W, hole;
  int kd, kh, kw, wide;
  while (std::scanf("%lld %lld %lld %d %d %d %lld %d", &D, &H, &W, &kd, &kh, &kw, &hole, &wide) == 8) {
    ndf::Plan p;
    p.dtype = wide;
    p.ndim = D > 1 || kd > 1 ? 3 : 2;
    p.sm_count = argc > 1 ? std::atoi(argv[1]) : 152;
    ndf::Geom3& g = p.tile.g;
    g = ndf::Geom3{};
    g.D = D, g.H = H, g.W = W, g.kd = kd, g.kh = kh, g.kw = kw;
    const long long volume = (long long)kd * kh * kw;
    p.r.count = (int)(hole < 0 ? volume : volume - 1);
    if (hole >= 0) {
      p.footprint.assign((size_t)volume, 1);
      p.footprint[(size_t)hole] = 0;
      for (long long i = 0; i < volume; ++i)
        if (i != hole)
          for (int v : {(int)(i / kw / kh), (int)(i / kw % kh), (int)(i % kw)}) p.box_taps.push_back(v);
    }
    p.r.kind = 0;  // median
    if (!ndf::histogram_configure(p)) {
      std::printf("0 0 0 0 0 0 0\n");
      continue;
    }
    std::printf("%d %d %d %d %d %zu %d\n", p.hist_block_w, p.hist_block_h, p.hist_block_d, (int)p.hist_sdec,
                (int)p.hist_in_smem, ndf::histogram_smem(p), p.hist_nf + 2 * p.hist_nv + 2 * p.hist_nh);
  }
}
