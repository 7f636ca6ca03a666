// FP64 batches and blocks on a GPU with little room: this program's cudaMalloc
// refuses what goes beyond a budget.  Whatever would fit without the split
// stages' workspace is done, and gives the same state bit for bit.
#include <cuda_runtime.h>
#include <dlfcn.h>

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <map>
#include <vector>

#include "mhdvlct_gb300.h"

static size_t g_used = 0, g_budget = ~(size_t)0;
static std::map<void*, size_t> g_sizes;
static std::vector<size_t> g_log;

extern "C" cudaError_t cudaMalloc(void** p, size_t n) {
  static auto real = (cudaError_t(*)(void**, size_t))dlsym(RTLD_NEXT, "cudaMalloc");
  if (g_used + n > g_budget) return cudaErrorMemoryAllocation;
  const cudaError_t e = real(p, n);
  if (e == cudaSuccess) {
    g_sizes[*p] = n;
    g_used += n;
    g_log.push_back(n);
  }
  return e;
}
extern "C" cudaError_t cudaFree(void* p) {
  static auto real = (cudaError_t(*)(void*))dlsym(RTLD_NEXT, "cudaFree");
  auto it = g_sizes.find(p);
  if (it != g_sizes.end()) {
    g_used -= it->second;
    g_sizes.erase(it);
  }
  return real(p);
}

#define CHECK(x)                                                                    \
  do {                                                                              \
    const int rc_ = (int)(x);                                                       \
    if (rc_) {                                                                      \
      std::printf("line %d: %d %s\n", __LINE__, rc_, mhdvlct_last_error_string(h)); \
      std::exit(1);                                                                 \
    }                                                                               \
  } while (0)
#define EXPECT(x)                                  \
  do {                                             \
    if (!(x)) {                                    \
      std::printf("line %d: %s\n", __LINE__, #x);  \
      std::exit(1);                                \
    }                                              \
  } while (0)

static const int kN = 16, kM = kN + 6, kBlocks = 2;
static mhdvlct_handle* h = nullptr;

static mhdvlct_batch* create() {
  int dims[3 * kBlocks];
  double widths[3 * kBlocks];
  for (int i = 0; i < 3 * kBlocks; i++) {
    dims[i] = kN;
    widths[i] = 1.0 / kN;
  }
  mhdvlct_batch* b = nullptr;
  CHECK(mhdvlct_batch_create(h, dims, widths, kBlocks, 3, MHD_DTYPE_F64, &b));
  for (int i = 0; i < kBlocks; i++) {
    MhdBlockView v;
    CHECK(mhdvlct_batch_block_view(b, i, &v));
    unsigned r = 12345u + (unsigned)i;
    auto fill = [&](void* p, size_t n, double base, double amp) {
      std::vector<double> a(n);
      for (double& x : a) {
        r = r * 1664525u + 1013904223u;
        x = base + amp * (r >> 8) / 16777216.0;
      }
      CHECK(cudaMemcpy(p, a.data(), n * sizeof(double), cudaMemcpyHostToDevice));
    };
    const size_t M = (size_t)kM * kM * kM, F = (size_t)(kM + 1) * kM * kM;
    fill(v.density, M, 1.0, 0.3);
    fill(v.total_energy, M, 4.0, 0.3);
    for (int k = 0; k < 3; k++) {
      fill(v.velocity[k], M, 0.0, 0.2);
      fill(v.bfield[k], M, 0.3, 0.0);
      fill(v.bfieldi[k], F, 0.3, 0.0);
    }
  }
  return b;
}
static std::vector<double> step(mhdvlct_batch* b) {
  const double dt[kBlocks] = {1e-3, 2e-3};
  CHECK(mhdvlct_batch_step(b, dt, nullptr));
  CHECK(cudaDeviceSynchronize());
  std::vector<double> out;
  for (int i = 0; i < kBlocks; i++) {
    MhdBlockView v;
    CHECK(mhdvlct_batch_block_view(b, i, &v));
    const size_t M = (size_t)kM * kM * kM;
    for (void* p : {v.density, v.velocity[0], v.velocity[1], v.velocity[2], v.total_energy,
                    v.bfield[0], v.bfield[1], v.bfield[2]}) {
      std::vector<double> a(M);
      CHECK(cudaMemcpy(a.data(), p, M * sizeof(double), cudaMemcpyDeviceToHost));
      for (int z = 3; z < kM - 3; z++)
        for (int y = 3; y < kM - 3; y++)
          out.insert(out.end(), &a[((size_t)z * kM + y) * kM + 3], &a[((size_t)z * kM + y) * kM + kM - 3]);
    }
  }
  return out;
}

int main() {
  MhdVlctParams p;
  char err[256];
  CHECK(mhdvlct_params_parse(
      "Method { mhd_vlct { mhd_choice = \"constrained_transport\"; riemann_solver = \"hlld\";"
      " reconstruct_method = \"plm\"; courant = 0.4; }; }"
      " Physics { fluid_props { eos { gamma = 1.6666666666666667; }"
      " floors { density = 1e-200; pressure = 1e-200; } } }",
      &p, err, sizeof err));
  CHECK(mhdvlct_create(&p, &h));
  CHECK(cudaDeviceSynchronize());
  g_log.clear();
  mhdvlct_batch* b = create();
  const std::vector<size_t> sizes = g_log;
  const size_t all = g_used, ws = *std::max_element(sizes.begin() + 1, sizes.end());
  EXPECT(ws > (size_t)32 * kN * kN * kN * sizeof(double));  // the workspace it is
  const std::vector<double> want = step(b);
  CHECK(mhdvlct_batch_destroy(b));
  EXPECT(g_used == 0);

  // creation in what the rest needs, and in what the workspace fits beside only
  // while the descriptors have not been asked for
  const size_t rest = all - ws;
  for (size_t budget : {rest, rest + ws / 2, all - sizes.back(), all - 1, all}) {
    g_budget = budget;
    b = create();
    EXPECT((g_used == all) == (budget == all));
    EXPECT(step(b) == want);
    // a call that needs more than what is left (a copy of the state), twice
    g_budget = std::max(g_used, all);
    char json[4096];
    CHECK(mhdvlct_batch_autotune(b, 1, json, sizeof json, nullptr));
    CHECK(mhdvlct_batch_autotune(b, 1, json, sizeof json, nullptr));
    g_budget = ~(size_t)0;
    CHECK(mhdvlct_batch_destroy(b));
    EXPECT(g_used == 0);
  }
  // a workspace given back between two steps
  b = create();
  g_budget = g_used;
  char json[4096];
  CHECK(mhdvlct_batch_autotune(b, 1, json, sizeof json, nullptr));
  EXPECT(g_used <= all - ws + 4096);
  EXPECT(step(b) == want);
  g_budget = ~(size_t)0;
  CHECK(mhdvlct_batch_destroy(b));

  // less than the rest is refused, and the next creation is as the first
  g_budget = rest - 1;
  int dims[3 * kBlocks];
  double widths[3 * kBlocks];
  for (int i = 0; i < 3 * kBlocks; i++) {
    dims[i] = kN;
    widths[i] = 1.0 / kN;
  }
  EXPECT(mhdvlct_batch_create(h, dims, widths, kBlocks, 3, MHD_DTYPE_F64, &b) == MHD_ERR_NOMEM);
  EXPECT(g_used == 0);
  g_budget = ~(size_t)0;
  b = create();
  EXPECT(step(b) == want);
  CHECK(mhdvlct_batch_destroy(b));
  CHECK(mhdvlct_destroy(h));
  std::printf("ok\n");
  return 0;
}
