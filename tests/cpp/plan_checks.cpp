// Checks of the host-side work plans (capi_internal.h), no GPU needed: the FP64
// fused kernel's tiles and chunks against the best that an exhaustive search
// finds.  Usage: plan_checks <check>; prints "ok" or what is wrong.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>

#include "capi_internal.h"

using namespace mhdint;

static const int kSms = 152;
static int up(int a, int b) { return (a + b - 1) / b; }

// Time of a stage of the FP64 fused kernel, in the time of a warp and plane: one
// CTA on an SM, a plane's time its warps and a fixed part but never below a
// latency, a chunk its planes and 1.6 more, in waves.
static double f64_time(const vlct::StageKind& k, const Window& w, int tx, int ty, int zc) {
  const int nz = zc > 0 && zc < w.len[2] ? up(w.len[2], zc) : 1;
  const int ax = up(w.len[0], up(w.len[0], tx)), ay = up(w.len[1], up(w.len[1], ty));
  const double n = (double)up(w.len[0], ax) * up(w.len[1], ay) * nz;
  const double warps = up((ax + 2) * (ay + 2), 32);
  const double plane = std::max(k.nn ? 5.2 : 6.4, warps + (k.nn ? 1.6 : 2.6));
  return std::ceil(n / kSms) * (up(w.len[2], nz) + 1.6) * plane;
}

static int check_f64_tiles() {
  int bad = 0;
  for (int mhd = 0; mhd < 2; mhd++)
    for (int nn = 0; nn < 2; nn++)
      for (int n : {1, 3, 8, 16, 20, 24, 28, 32, 33, 40}) {
        const vlct::StageKind k = {true, nn != 0, mhd != 0};
        const Window w = {1, {n + 4, n + 4, n + 4}};
        const Decomp d = decompose(k, w, 1, kSms);
        double best = 1e300;
        for (int x = 1; x <= std::min(16, w.len[0]); x++)
          for (int y = 1; y <= std::min(16, w.len[1]); y++)
            for (int zc = 0; zc < w.len[2]; zc++)
              if (k.fits(x, y)) best = std::min(best, f64_time(k, w, x, y, zc));
        const double t = f64_time(k, w, d.tx, d.ty, d.zchunk);
        // the chunk lengths tried are not all there are
        if (!k.fits(d.tx, d.ty) || t > 1.1 * best) {
          std::printf("n %d nn %d: %d x %d, %d planes: %.1f, best %.1f\n", n, nn, d.tx, d.ty,
                      d.zchunk, t, best);
          bad = 1;
        }
      }
  return bad;
}

int main(int argc, char** argv) {
  int bad = 2;
  if (argc > 1 && !std::strcmp(argv[1], "f64_tiles")) bad = check_f64_tiles();
  if (!bad) std::printf("ok\n");
  return bad;
}
