// Checks of the host-side work plans (capi_internal.h), no GPU needed: the FP64
// fused kernel's tiles and chunks against the best that an exhaustive search
// finds, and the search for tiles and chunks against plain loops over all of them.
// Usage: plan_checks <check>; prints "ok" or what is wrong.
#include <algorithm>
#include <chrono>
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

// decompose and fit_tile as plain loops over every extent and chunk length: what the
// library's search must find.
static double cost_of(const vlct::StageKind& k, int tx, int ty) {
  return up((tx + 2) * (ty + 2), 32) + (k.f64 ? (k.nn ? 1.6 : 2.6) : 6.0);
}
static Decomp all_choices(const vlct::StageKind& k, const Window& w, long nblocks) {
  Decomp d;
  const int top = k.f64 ? 16 : 40;
  double best = 1e300;
  for (int y = 1; y <= std::min(top, w.len[1]); y++)
    for (int x = 1; x <= std::min(top, w.len[0]); x++) {
      if (up(w.len[0], up(w.len[0], x)) != x || up(w.len[1], up(w.len[1], y)) != y ||
          !k.fits(x, y))
        continue;
      const int warps = up((x + 2) * (y + 2), 32);
      auto plane = [&](long n) {
        return k.f64 ? std::max(k.nn ? 5.2 : 6.4, cost_of(k, x, y))
                     : std::max(1.0 + 0.02 * warps, 0.35 + 0.065 * (double)n * (up(warps, 4) * 4));
      };
      for (int L : {0, 32, 24, 16, 12, 10, 8, 7, 6, 5, 4, 3, 2, 1}) {
        if (L >= w.len[2]) continue;
        const int nz = L > 0 ? up(w.len[2], L) : 1;
        const long res = (long)k.ctas() * kSms;
        const long n = (long)up(w.len[0], x) * up(w.len[1], y) * nblocks * nz, rest = n % res;
        const double cost = ((double)(n / res) * plane(k.ctas()) +
                             (rest ? plane((rest + kSms - 1) / kSms) : 0.0)) *
                            (up(w.len[2], nz) + (k.f64 ? 1.6 : 2.5));
        if (cost < best * 0.999) {
          best = cost;
          d.tx = x;
          d.ty = y;
          d.zchunk = L;
        }
      }
    }
  return d;
}
static void all_tiles(const vlct::StageKind& k, int lx, int ly, int& tx, int& ty) {
  const int top = k.f64 ? 16 : 40;
  const int mx = std::min(lx, tx > 0 ? std::min(tx, top) : top);
  const int my = std::min(ly, ty > 0 ? std::min(ty, top) : top);
  double best = 1e300;
  for (int x = 1; x <= mx; x++)
    for (int y = 1; y <= my; y++) {
      const int ax = up(lx, up(lx, x)), ay = up(ly, up(ly, y));
      if (!k.fits(ax, ay)) continue;
      const double c = (double)up(lx, ax) * up(ly, ay) * cost_of(k, ax, ay);
      if (c <= best) {
        best = c;
        tx = ax;
        ty = ay;
      }
    }
}
static int check_search() {
  int bad = 0;
  for (int kind = 0; kind < 8; kind++) {
    const vlct::StageKind k = {(kind & 1) != 0, (kind & 2) != 0, (kind & 4) != 0};
    for (int i = 0; i < 400; i++) {
      const unsigned r = 2654435761u * (unsigned)(i + 1);
      const int big = i % 10 == 0 ? 300 : 70;
      const Window w = {1, {1 + (int)(r % big), 1 + (int)(r / 97 % big), 1 + (int)(r / 9409 % big)}};
      const long nb = 1 + (long)(r >> 27);
      const Decomp a = decompose(k, w, nb, kSms), b = all_choices(k, w, nb);
      int tx = i % 3 * 7, ty = i % 5 * 4, ux = tx, uy = ty;
      fit_tile(k, w.len[0], w.len[1], tx, ty);
      all_tiles(k, w.len[0], w.len[1], ux, uy);
      if (a.tx != b.tx || a.ty != b.ty || a.zchunk != b.zchunk || tx != ux || ty != uy) {
        std::printf("kind %d %d x %d x %d, %ld blocks: %d x %d x %d, not %d x %d x %d; %d x %d, not %d x %d\n",
                    kind, w.len[0], w.len[1], w.len[2], nb, a.tx, a.ty, a.zchunk, b.tx, b.ty,
                    b.zchunk, tx, ty, ux, uy);
        bad = 1;
      }
    }
  }
  return bad;
}

// The search of a block's two stages, which a handle's first step at an extent and
// every small batch wait for: at most a tenth of the plain loops' time.
static int check_search_time() {
  int bad = 0;
  for (int f64 = 0; f64 < 2; f64++)
    for (int n : {32, 64, 96}) {
      const vlct::StageKind nn = {f64 != 0, true, true}, plm = {f64 != 0, false, true};
      const Window w0 = {1, {n + 4, n + 4, n + 4}}, w1 = {3, {n, n, n}};
      double t[2] = {1e9, 1e9};
      for (int rep = 0; rep < 200; rep++)
        for (int which = 0; which < 2; which++) {
          const auto t0 = std::chrono::steady_clock::now();
          const Decomp a = which ? all_choices(nn, w0, 1) : decompose(nn, w0, 1, kSms);
          const Decomp b = which ? all_choices(plm, w1, 1) : decompose(plm, w1, 1, kSms);
          const std::chrono::duration<double, std::micro> us = std::chrono::steady_clock::now() - t0;
          if (a.tx + b.tx <= 0) return 1;
          t[which] = std::min(t[which], us.count());
        }
      std::fprintf(stderr, "f64 %d, %d^3: %.1f us, plain loops %.1f us\n", f64, n, t[0], t[1]);
      if (t[0] > 0.25 * t[1]) {
        std::printf("f64 %d, %d^3: %.1f us, plain loops %.1f us\n", f64, n, t[0], t[1]);
        bad = 1;
      }
    }
  return bad;
}

// A z-slab of a split MHD stage solves the x and y faces of two planes more than it
// updates: over all slabs of a block, at most half again as many (or the stage runs
// as the fused kernel), and every plane is updated once, within the workspace.
static int check_slabs() {
  int bad = 0;
  for (int mhd = 0; mhd < 2; mhd++)
    for (int nx : {8, 118, 256, 340, 390, 400, 512, 800, 2000})
      for (int nz : {4, 8, 16, 64, 300}) {
        const int S = 2, lo = S + 1;
        const std::vector<int> m = {nx + 6, nx + 6, nz + 6};
        std::vector<vlct::SplitJob> jobs;
        std::vector<vlct::SplitGroup> groups;
        size_t ws = 0;
        split_plan(m, {}, S, false, mhd != 0, false, jobs, groups, ws);
        int next = lo, planes = 0;
        for (const auto& j : jobs) {
          if (j.za != next) bad = 1;
          next = j.zb;
          planes += j.zb - j.za + 2;
        }
        const int len = m[2] - 2 * lo;
        if ((!jobs.empty() && next != m[2] - lo) || (jobs.empty() && ws != 0)) bad = 1;
        if (mhd && jobs.size() > 1 && planes > 1.5 * len) bad = 1;
        if (mhd && jobs.empty() && nx < 380) bad = 1;  // narrow planes are never refused
        if (bad) {
          std::printf("mhd %d, %d x %d x %d: %zu slabs, %d planes of faces for %d\n", mhd, nx, nx,
                      nz, jobs.size(), planes, len);
          return 1;
        }
      }
  return 0;
}

// The chunks of the timestep's launch: within the work there is, and a grid that is a
// whole number of waves but for a tenth, or as near as eight waves come.
static int check_chunks() {
  for (long nb : {1, 2, 3, 7, 30, 64, 128, 152, 200, 305, 512, 608, 1000, 2000, 100000})
    for (long res : {1, 152, 304, 608})
      for (size_t work : {(size_t)1, (size_t)2744, (size_t)10648, (size_t)343000, (size_t)20000000}) {
        const int c = vlct::wave_chunks(nb, res, work, 512);
        const long most = std::max<long>(1, (long)(work / 512));
        bool ok = c >= 1 && c <= most;
        if (c < most && nb <= 8 * res) {
          double best = 0.0, got = 0.0;
          for (long w = 1; w <= 8; w++) {
            best = std::max(best, (double)(w * res / nb * nb) / (double)(w * res));
            if (w * res >= c * nb) got = std::max(got, (double)(c * nb) / (double)(w * res));
          }
          ok = ok && (got >= 0.9 || got >= best - 1e-9);
        }
        if (!ok) {
          std::printf("%ld blocks, %ld CTAs at once, %zu items: %d chunks\n", nb, res, work, c);
          return 1;
        }
      }
  return 0;
}

int main(int argc, char** argv) {
  int bad = 2;
  if (argc > 1 && !std::strcmp(argv[1], "f64_tiles")) bad = check_f64_tiles();
  if (argc > 1 && !std::strcmp(argv[1], "search")) bad = check_search();
  if (argc > 1 && !std::strcmp(argv[1], "search_time")) bad = check_search_time();
  if (argc > 1 && !std::strcmp(argv[1], "slabs")) bad = check_slabs();
  if (argc > 1 && !std::strcmp(argv[1], "chunks")) bad = check_chunks();
  if (!bad) std::printf("ok\n");
  return bad;
}
