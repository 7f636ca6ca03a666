// vlct_stage.cuh -- one fused VL+CT stage (half or full step) for a set of
// blocks, as a z-marching CUDA kernel.
//
// A CTA owns a column tile [xa, xb) x [ya, yb) of one block and marches up
// the block's z range (or one z-chunk of it).  One thread owns one column of
// the tile and its one-cell halo, (tx + 2) x (ty + 2) of them, for the whole
// march: it loads that column's cells, solves the Riemann problems of the
// faces on the high side of its cell, forms the three edge EMFs there and
// updates its cell.  So a column's positions, windows and addresses are worked
// out once per tile and not once per item; what only the owner reads (the
// cells below and above, the z fluxes, the x-y part of the flux divergence)
// stays in registers; and the shared memory holds one plane of primitives (and
// of slopes) and what neighbours exchange.  Nothing depends on the tile's or
// the block's extents at compile time.  Per z-plane t:
//
//   B  Riemann solves: the z-face at t+1/2, the x- and y-faces of plane t+1
//   |  barrier
//   C  upwinded edge EMFs (E_x, E_y at t+1/2, E_z of plane t); the x-y flux
//      divergence of plane t+1, kept for its update; the next plane's cells
//      (on their way since the start of C, with the start-of-step values that D
//      wants) turned into primitives and published, with the cell-centred E
//   |  barrier
//   D  the constrained-transport face updates around cell (x, y, t) (Bz at
//      t+1, Bx / By at both faces of the cell), the cell update: centred B,
//      flux divergence + dual-energy source, density floor, energy floor /
//      dual-energy sync, store
//   A  (PLM) the x and y slopes of the plane published in C, each formed once
//      and read by both faces of its cell; | barrier
//
// What bounds it: issue slots (53-57% used; FMA, ALU and LSU pipes 24-33%, DRAM
// 10%), with 16 warps an SM, as the Riemann solvers want 128 registers.  Against
// the form it replaced, whose threads took each phase's items in rounds (every
// item's place worked out anew, launch shapes of one block size compiled in, the
// layer around the updated cells in the tiles): HLLD + PLM warp instructions per
// zone 129 -> 98 (half dt), 135 -> 97 (full).  One cycle, before -> after: 256^3
// in blocks of 32^3 6.60 -> 5.65 ms; in blocks of 64^3 with dual energy 11.7 ->
// 5.39 ms; 1000 blocks of 16^3 - 64^3 29.2 -> 12.2 ms; 960 hydro leaves with flux
// correction 7.45 -> 6.00 ms.
//
// The index windows of every quantity are those of the reference's array
// passes (EnzoMHDIntegratorStageCommands::compute_update_stage,
// src/Enzo/hydro-mhd/EnzoMHDIntegratorStageCommands.cpp:102-261, with the
// stale-depth bookkeeping of EnzoMethodMHDVlct::compute, :459-496), so the
// values written are the reference's values wherever the reference defines
// them.  The FP64 instantiation is compiled with --fmad=false and matches the
// reference bit for bit; in the FP32 instantiation the pressure recovery
// (total minus kinetic minus magnetic energy) and the energy floor / sync run
// in float-float (vlct_energy.cuh).  Further instantiations (EXTRA) also
// store the boundary fluxes for flux correction (EXTRA_FC) or, in addition,
// add the gravity source and write the density flux of every updated face
// for the passive scalars' advection (EXTRA_ALL; the scalars themselves are
// advected by passive_kernel, vlct_passive.cuh); the default one compiles
// all of these out.
//
// FP64 runs this kernel only where the split kernels (vlct_split.cuh) cannot or
// should not: the no-allocation step, a GPU too full for their workspace, MHD
// blocks of very wide planes.  FP32, whose arithmetic is 64 times cheaper, always
// does.
#pragma once
#include <type_traits>

#include "vlct_energy.cuh"
#include "vlct_launch.h"
#include "vlct_physics.cuh"
#include "vlct_types.h"

namespace vlct {

// global primitive slot order: rho, Bx, By, Bz, vx, vy, vz, p
enum { Q_RHO = 0, Q_BX = 1, Q_VX = 4, Q_P = 7, NQ = 8 };
// shared flux slots: rho, mom x/y/z, etot, B_(d+1), B_(d+2), eint, vbar
enum { S_RHO = 0, S_MX = 1, S_E = 4, S_BJ = 5, S_BK = 6, S_EINT = 7, S_VBAR = 8 };

__device__ __forceinline__ bool inr(int a, int lo, int hi) {
  return a >= lo && a < hi;
}

// Upwind weight of CT from the sign of the density flux
// (EnzoBfieldMethodCT.cpp:198-213); 1/2 where it is a NaN.
template <class R> __device__ __forceinline__ R upw(R fd) {
  return gt0(fd) ? R(1.0) : (lt0(fd) ? R(0.0) : R(0.5));
}

// compute_edge_<true> (EnzoBfieldMethodCT.cpp:384-457)
template <class R>
__device__ __forceinline__ R edge_emf(R Ej, R Ej_kp1, R Ek, R Ek_jp1, R Wj,
                                      R Wj_kp1, R Wk, R Wk_jp1, R Ec, R Ec_jp1,
                                      R Ec_kp1, R Ec_jkp1) {
  R dEdj_r = Wk_jp1 * (Ec_jp1 + Ej) + (R(1) - Wk_jp1) * (Ec_jkp1 + Ej_kp1);
  R dEdj_l = Wk * (-Ej - Ec) + (R(1) - Wk) * (-Ej_kp1 - Ec_kp1);
  R dEdk_r = Wj_kp1 * (Ec_kp1 - Ek) + (R(1) - Wj_kp1) * (Ec_jkp1 - Ek_jp1);
  R dEdk_l = Wj * (Ek - Ec) + (R(1) - Wj) * (Ek_jp1 - Ec_jp1);
  R Ej_sum = Ej + Ej_kp1;
  Ej_sum *= R(-1);
  R Ek_sum = Ek + Ek_jp1;
  return R(0.25) * (Ej_sum + Ek_sum + (dEdj_l - dEdj_r) + (dEdk_l - dEdk_r));
}
// The same in FP64, where the weights pick their terms instead of multiplying them
// by 1 and 0 (a third of the FP64 operations); the products with 0 are zeros
// wherever what they leave out is finite.
template <>
__device__ __forceinline__ double edge_emf<double>(double Ej, double Ej_kp1, double Ek,
                                                   double Ek_jp1, double Wj, double Wj_kp1,
                                                   double Wk, double Wk_jp1, double Ec,
                                                   double Ec_jp1, double Ec_kp1,
                                                   double Ec_jkp1) {
  // W (a1 +- a2) + (1 - W) (b1 +- b2)
  auto mix = [](double W, double a1, double a2, double b1, double b2, auto minus) -> double {
    constexpr bool M = decltype(minus)::value;
    const int w = __double2hiint(W);  // of 0, 1/2 or 1
    const bool a = w == 0x3ff00000;
    if (w == 0x3fe00000 || !is_finite(a ? b1 : a1) || !is_finite(a ? b2 : a2)) {
      rare_path();
      return W * (M ? a1 - a2 : a1 + a2) + (1.0 - W) * (M ? b1 - b2 : b1 + b2);
    }
    const double x = a ? a1 : b1, y = a ? a2 : b2;
    return M ? x - y : x + y;
  };
  const std::false_type sum{};
  const std::true_type diff{};
  const double dj_r = mix(Wk_jp1, Ec_jp1, Ej, Ec_jkp1, Ej_kp1, sum);
  const double dj_l = mix(Wk, Ej, Ec, Ej_kp1, Ec_kp1, sum);  // minus dEdj_l
  const double dk_r = mix(Wj_kp1, Ec_kp1, Ek, Ec_jkp1, Ek_jp1, diff);
  const double dk_l = mix(Wj, Ek, Ec, Ek_jp1, Ec_jp1, diff);
  return scale2<-2>((((Ek + Ek_jp1) - (Ej + Ej_kp1)) - (dj_l + dj_r)) + (dk_l - dk_r));
}
// The same in FP32, the same value bit for bit (a weight is 0, 1/2 or 1, so its
// products are exact), with the signs of the sums folded in.
template <>
__device__ __forceinline__ float edge_emf<float>(float Ej, float Ej_kp1, float Ek, float Ek_jp1,
                                                 float Wj, float Wj_kp1, float Wk, float Wk_jp1,
                                                 float Ec, float Ec_jp1, float Ec_kp1,
                                                 float Ec_jkp1) {
  auto mix = [](float w, float a, float b) {
    return __fmaf_rn(w, a, __fmul_rn(__fsub_rn(1.0f, w), b));
  };
  const float dj_r = mix(Wk_jp1, Ec_jp1 + Ej, Ec_jkp1 + Ej_kp1);
  const float dj_l = mix(Wk, Ej + Ec, Ej_kp1 + Ec_kp1);  // minus dEdj_l
  const float dk_r = mix(Wj_kp1, Ec_kp1 - Ek, Ec_jkp1 - Ek_jp1);
  const float dk_l = mix(Wj, Ek - Ec, Ek_jp1 - Ec_jp1);
  return 0.25f * ((((Ek + Ek_jp1) - (Ej + Ej_kp1)) - (dj_l + dj_r)) + (dk_l - dk_r));
}

template <class R, int SOLVER, int RECON, bool DE> struct StageCfg {
  static constexpr bool MHD = SOLVER != SOLVER_HLLC;
  static constexpr bool NN = RECON == RECON_NN;
  static constexpr int NF = DE ? 9 : (MHD ? 7 : 5);
};

// Threads of a CTA (and the most columns a tile takes with its halo, one a
// thread) and the CTAs the register allocation leaves room for on an SM.
template <class R, int SOLVER, int RECON> struct StageBounds {
  static constexpr StageKind kind = {sizeof(R) == 8, RECON == RECON_NN, SOLVER != SOLVER_HLLC};
  static constexpr int threads = kind.threads(), min_blocks = kind.ctas();
};
constexpr int kStageRing = StageKind::ring;

// Shared-memory arrays, in elements: of NT each but where a size is given.
template <class R, int SOLVER, int RECON, bool DE> struct StageSmem {
  using C = StageCfg<R, SOLVER, RECON, DE>;
  static constexpr int NT = StageBounds<R, SOLVER, RECON>::threads;
  static constexpr int PQ = NT + (C::NN ? 0 : kStageRing);
  // x / y face fluxes: density and the two transverse B of two planes, the
  // other components of one
  static constexpr int FD = C::MHD ? 3 : 1;            // per plane, two planes
  static constexpr int FS = 4 + (DE ? 2 : 0);          // one plane
  static constexpr int PL = C::NN ? 0 : 1;
  static constexpr int MH = C::MHD ? 1 : 0;
  static constexpr int NEC = C::NN ? 3 : 2;            // planes of E
  static constexpr int NP = C::NN ? 2 : 1;             // planes of primitives
  static constexpr int o_p = 0;
  static constexpr int o_h = o_p + NP * NQ * PQ;            // PLM: x, y slopes
  static constexpr int o_xf = o_h + PL * 2 * (NQ - 1) * NT;
  static constexpr int o_yf = o_xf + (2 * FD + FS) * NT;
  static constexpr int o_zf = o_yf + (2 * FD + FS) * NT;
  static constexpr int o_ec = o_zf + MH * 3 * NT;
  static constexpr int o_ex = o_ec + MH * 3 * NEC * NT;
  static constexpr int o_ey = o_ex + MH * 2 * NT;
  static constexpr int o_ez = o_ey + MH * 2 * NT;
  // the upwind weights of the x and y faces of two planes (the z faces' are in o_zf,
  // in the place of their density flux), formed once and not by each of four edges:
  // right for NaN too at the cost of a shorter form that is not (256^3 box 5.65 ms
  // a cycle with that, 5.66 here; formed by each edge 5.69)
  static constexpr int o_ww = o_ez + MH * NT;
  // a column's own values, kept here across the Riemann solves, which want the
  // registers: PLM's plane t+2 and low z-face state, the z fluxes at t-1/2,
  // the x-y flux divergence of the plane to be updated
  static constexpr int o_w2 = o_ww + MH * 4 * NT;
  static constexpr int o_lz = o_w2 + PL * NQ * NT;
  static constexpr int o_zm = o_lz + PL * NQ * NT;
  static constexpr int o_dx = o_zm + (DE ? 7 : 5) * NT;
  // FP64 NN: what the six faces of a cell take from its density and pressure
  // alone (CellGas), of two planes: formed once a cell and not once a face and
  // side, as the divisions and square roots in it are up to a third of the FP64
  // pipe's work (no-allocation step with NN in both stages, before -> after: HLLE
  // 32^3 624 -> 564 us, 32 x 32 x 16 437 -> 396; HLLC 32^3 325 -> 259)
  static constexpr int NG = C::NN && sizeof(R) == 8 ? CellGas<SOLVER>::N : 0;
  static constexpr int o_cg = o_dx + (DE ? 6 : 5) * NT;
  static constexpr int total = o_cg + 2 * NG * NT;
};
template <class R, int SOLVER, int RECON, bool DE> constexpr size_t stage_smem_bytes() {
  return (size_t)StageSmem<R, SOLVER, RECON, DE>::total * sizeof(R);
}

enum { EXTRA_NONE = 0, EXTRA_FC = 1, EXTRA_ALL = 2 };

// element at a byte offset
template <class R> __device__ __forceinline__ R ldb(const R* p, size_t o) {
  return *reinterpret_cast<const R*>(reinterpret_cast<const char*>(p) + o);
}
template <class R> __device__ __forceinline__ void stb(R* p, size_t o, R v) {
  *reinterpret_cast<R*>(reinterpret_cast<char*>(p) + o) = v;
}

// EXTRA: EXTRA_NONE compiles the optional work out (its run-time checks alone
// cost ~4% of a stage); EXTRA_FC can store the boundary fluxes; EXTRA_ALL
// can also add the gravity source and write the density fluxes that
// passive_kernel advects the passive scalars with.
template <class R, int SOLVER, int RECON, bool DE, int EXTRA>
__global__ void __launch_bounds__(StageBounds<R, SOLVER, RECON>::threads,
                                  StageBounds<R, SOLVER, RECON>::min_blocks)
stage_kernel(const StageBlock<R>* __restrict__ blocks,
             const StageTile* __restrict__ tiles, int ntiles, StageInfo info,
             PhysParams phys) {
  using C = StageCfg<R, SOLVER, RECON, DE>;
  using L = StageSmem<R, SOLVER, RECON, DE>;
  constexpr bool MHD = C::MHD, NN = C::NN;
  constexpr int NT = L::NT, PQ = L::PQ, FD = L::FD;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  R* const sm = reinterpret_cast<R*>(smem_raw);
  const int tid = threadIdx.x;
  const int s = info.s, S = info.S;
  const bool final_stage = info.final_stage != 0;
  // the physical constants in R; in FP32 the values rounded on the host, which
  // need no FP64 conversion on the device
  constexpr bool F32 = std::is_same<R, float>::value;
  const R g = R(phys.gamma_f);  // (FP32)
  (void)g;
  const R theta = F32 ? R(phys.theta_limiter_f) : R(phys.theta_limiter);
  const R dfloor = F32 ? R(phys.density_floor_f) : R(phys.density_floor);
  const R pfloor = F32 ? R(phys.pressure_floor_f) : R(phys.pressure_floor);
  EnergyConsts<R> econ;
  if constexpr (F32)
    econ.init_rounded(phys, DE);
  else
    econ.init(phys, DE);

  __shared__ int s_next;
  // the current tile's block descriptor, copied into shared memory once per
  // tile: read from global memory, its field pointers would be reloaded after
  // every global store (the compiler cannot rule out aliasing)
  __shared__ __align__(16) unsigned long long s_blk_raw[(sizeof(StageBlock<R>) + 7) / 8];
  // the block's flux-correction outputs on a flux-storing final stage, also
  // copied once per tile: read from global memory, every boundary-face store
  // would first wait for its pointer
  constexpr int kFoWords = EXTRA != EXTRA_NONE ? (int)((sizeof(FluxOut<R>) + 7) / 8) : 1;
  __shared__ __align__(16) unsigned long long s_fo_raw[kFoWords];
  // what is the same for all threads of a tile stays in shared memory too: the
  // solves leave no registers for it
  struct Tile {
    R dtdx[3], dt;
    int m0, m1, m2, HP, HQ, za, zb, olo;
    size_t szb, fxzb, fyzb;  // plane strides of the cell, x-face, y-face arrays
    int rowb;                // row stride of the cell arrays
  };
  __shared__ Tile T;
  const StageBlock<R>& B = *reinterpret_cast<const StageBlock<R>*>(s_blk_raw);
  const bool store_fc =
      EXTRA != EXTRA_NONE && final_stage && (info.fc != nullptr || info.block_fc);

  int it = blockIdx.x;
  if (info.queue) {
    if (tid == 0) s_next = atomicAdd(info.queue, 1);
    __syncthreads();
    it = s_next;
  }
  while (it < ntiles) {
    const StageTile tl = tiles[it];
    {
      const unsigned long long* src =
          reinterpret_cast<const unsigned long long*>(blocks + tl.block);
      for (int w = tid; w < (int)((sizeof(StageBlock<R>) + 7) / 8); w += NT)
        s_blk_raw[w] = src[w];
      if (store_fc) {
        const void* fsrc = blocks[tl.block].fc != nullptr ? blocks[tl.block].fc : info.fc;
        const unsigned long long* fw = reinterpret_cast<const unsigned long long*>(fsrc);
        for (int w = tid; w < kFoWords; w += NT) s_fo_raw[w] = fw[w];
      }
    }
    // dt / dx per axis, once per tile (FP64 divisions: one thread)
    if (tid == 0) {
      const StageBlock<R>& Bg = blocks[tl.block];
      const double dt = *Bg.dt * info.dt_factor;
      for (int a = 0; a < 3; a++) T.dtdx[a] = R(dt / Bg.cw[a]);
      T.dt = R(dt);
      T.m0 = Bg.m[0];
      T.m1 = Bg.m[1];
      T.m2 = Bg.m[2];
      T.HP = tl.xb - tl.xa + 2;
      T.HQ = tl.yb - tl.ya + 2;
      T.za = tl.za;
      T.zb = tl.zb;
      T.olo = S + 1;
      T.rowb = T.m0 * (int)sizeof(R);
      T.szb = (size_t)T.rowb * T.m1;
      T.fxzb = (size_t)(T.m0 + 1) * sizeof(R) * T.m1;
      T.fyzb = (size_t)T.rowb * (T.m1 + 1);
    }
    __syncthreads();  // also publishes the descriptor copy

    // ---- the thread's column and what it takes part in
    enum {
      CELL = 1, FX = 2, FY = 4, FZ = 8, EX = 16, EY = 32, EZ = 64, OUT = 128, UX = 256, UY = 512,
      UPD = 1024, RING = 2048, COL = 4096, XHI = 1 << 13, YHI = 1 << 14,
      // face B updated on the low / high side along x, y
      XLO = 1 << 15, XUP = 1 << 16, YLO = 1 << 17, YUP = 1 << 18,
      // first / last column and row of the halo grid
      ILO = 1 << 19, IHI = 1 << 20, JLO = 1 << 21, JHI = 1 << 22
    };
    unsigned fl = 0;
    auto on = [&](unsigned f) { return (fl & f) == f; };
    auto flag = [&](unsigned f, bool v) { fl |= v ? f : 0u; };
    int cb, xb_, rcell = 0;  // byte offsets in a plane: cell and y-face arrays,
                             // x-face arrays, ring
    {
      const int m0 = T.m0, m1 = T.m1, HP = T.HP, HQ = T.HQ;
      const int tx = HP - 2, ty = HQ - 2;
      const int j = tid / HP, i = tid - j * HP;
      const int x = tl.xa - 1 + i, y = tl.ya - 1 + j;
      const bool col = j < HQ;
      const bool iny = inr(y, S, m1 - S), inx = inr(x, S, m0 - S);
      const bool ux = inr(x, S + 1, m0 - S - 1), uy = inr(y, S + 1, m1 - S - 1);
      const bool hx = inr(x, S, m0 - S - 1), hy = inr(y, S, m1 - S - 1);
      const bool out = col && i >= 1 && i <= tx && j >= 1 && j <= ty;
      flag(COL, col);
      flag(CELL, col && inr(x, s, m0 - s) && inr(y, s, m1 - s));
      flag(FX, col && i <= tx && hx && iny);
      flag(FY, col && j <= ty && hy && inx);
      flag(FZ, col && inx && iny);
      flag(EX, col && i >= 1 && i <= tx && j <= ty && ux && hy);
      flag(EY, col && i <= tx && j >= 1 && j <= ty && uy && hx);
      flag(EZ, col && i <= tx && j <= ty && hx && hy);
      flag(OUT, out);
      flag(UX, ux);
      flag(UY, uy);
      flag(UPD, out && ux && uy);
      flag(XLO, inr(x, S + 1, m0 - S));
      flag(XUP, inr(x + 1, S + 1, m0 - S));
      flag(YLO, inr(y, S + 1, m1 - S));
      flag(YUP, inr(y + 1, S + 1, m1 - S));
      flag(XHI, x + 1 == m0 - T.olo);
      flag(YHI, y + 1 == m1 - T.olo);
      cb = y * T.rowb + x * (int)sizeof(R);
      xb_ = cb + y * (int)sizeof(R);
      flag(ILO, i == 0);
      flag(IHI, i == HP - 1);
      flag(JLO, j == 0);
      flag(JHI, j == HQ - 1);
      // PLM: the plane of primitives has a second ring of cells around the
      // halo grid, kept behind it: HP below, HP above, HQ left, HQ right; ring
      // cell k is loaded by thread k
      if (!NN && tid < 2 * (HP + HQ)) {
        const int k = tid < 2 * HP ? tid : tid - 2 * HP;
        const int ri = tid < 2 * HP ? (k < HP ? k : k - HP) : (k < HQ ? -1 : HP);
        const int rj = tid < 2 * HP ? (k < HP ? -1 : HQ) : (k < HQ ? k : k - HQ);
        const int rx = tl.xa - 1 + ri, ry = tl.ya - 1 + rj;
        flag(RING, inr(rx, s, m0 - s) && inr(ry, s, m1 - s));
        rcell = ry * T.rowb + rx * (int)sizeof(R);
      }
    }
    const int t0 = tl.za - 1;
    const int zb = tl.zb;

    R* const s_p0 = sm + L::o_p + tid;
    auto plane_p = [&](int p) { return s_p0 + (NN ? (p & 1) * NQ * PQ : 0); };
    R* const s_w2 = sm + L::o_w2 + tid;
    R* const s_h = sm + L::o_h + tid;
    R* const s_lz = sm + L::o_lz + tid;
    R* const s_zm = sm + L::o_zm + tid;
    R* const s_dx = sm + L::o_dx + tid;
    R* const s_xf = sm + L::o_xf + tid;
    R* const s_yf = sm + L::o_yf + tid;
    R* const s_zf = sm + L::o_zf + tid;
    R* const s_ec = sm + L::o_ec + tid;
    R* const s_ex = sm + L::o_ex + tid;
    R* const s_ey = sm + L::o_ey + tid;
    R* const s_ez = sm + L::o_ez + tid;
    R* const s_ww = sm + L::o_ww + tid;  // x: slots 0, 1 by plane, y: 2, 3
    // flux components in shared memory: plane-buffered ones and single ones
    auto fd = [&](int plane, int k) { return ((plane & 1) * FD + k) * NT; };
    auto fs = [&](int k) { return (2 * FD + k) * NT; };

    // ---- the cell at a byte offset: density, B, v and the energy field, in
    // primitive order; then the energy turned into the pressure
    // (EnzoComputePressure::compute_pressure, EnzoComputePressure.cpp:127-190)
    auto load = [&](size_t at, R* w) {
#pragma unroll
      for (int q = 0; q < NQ; q++)
        w[q] = q == Q_RHO ? ldb(B.cur.c[F_RHO], at)
             : q >= Q_VX && q < Q_P ? ldb(B.cur.c[F_VX + (q - Q_VX)], at)
             : q == Q_P ? ldb(B.cur.c[DE ? F_EINT : F_ETOT], at)
             : MHD ? ldb(B.cur.c[F_BX + (q - Q_BX)], at) : R(0);
    };
    auto prims = [&](R* w) {
      w[Q_P] = DE ? econ.gm1 * w[Q_RHO] * w[Q_P]
                  : pressure_from_etot<R, MHD>(econ, w[Q_RHO], w[Q_P], w[Q_VX], w[Q_VX + 1],
                                               w[Q_VX + 2], w[Q_BX], w[Q_BX + 1], w[Q_BX + 2]);
    };
    auto put = [&](R* dst, int pitch, const R* w) {
#pragma unroll
      for (int q = 0; q < NQ; q++)
        if (MHD || q < Q_BX || q >= Q_VX) dst[q * pitch] = w[q];
    };
    // FP64 NN: the cell's gas quantities, of plane p
    R* const s_cg = sm + L::o_cg + tid;
    auto plane_cg = [&](int p) { return s_cg + (p & 1) * L::NG * NT; };
    auto put_gas = [&](int p, const R* w) {
      if constexpr (L::NG > 0) {
        CellGas<SOLVER> cg;
        cg.init(Gas{phys.gamma, phys.gm1, phys.inv_gm1}, w[Q_RHO], w[Q_P]);
#pragma unroll
        for (int k = 0; k < L::NG; k++) plane_cg(p)[k * NT] = cg.v[k];
      }
    };
    // cell-centred E = -v x B of plane p (EnzoBfieldMethodCT.cpp:267-292)
    auto put_ec = [&](int p, const R* w) {
      if (MHD && on(FZ) && inr(p, S, T.m2 - S)) {
        R* e = s_ec + (p % L::NEC) * 3 * NT;
        const R bx = w[Q_BX], by = w[Q_BX + 1], bz = w[Q_BX + 2];
        const R vx = w[Q_VX], vy = w[Q_VX + 1], vz = w[Q_VX + 2];
        e[0] = (-vy * bz + vz * by);
        e[NT] = (-vz * bx + vx * bz);
        e[2 * NT] = (-vx * by + vy * bx);
      }
    };
    // PLM: half the slopes of the published plane along x (not of Bx) and y
    // (not of By), in the slots that hslot says
    auto hslot = [](int dir, int q) { return dir * (NQ - 1) + (q > Q_BX + dir ? q - 1 : q); };
    auto slopes = [&]() {
      const R* const s_p = s_p0;
      if (on(COL)) {
        const int HP = T.HP, HQ = T.HQ;
        const int j = tid / HP, i = tid - j * HP;
        const int lft = on(ILO) ? NT + 2 * HP + j - tid : -1;
        const int rgt = on(IHI) ? NT + 2 * HP + HQ + j - tid : 1;
        const int dwn = on(JLO) ? NT + i - tid : -HP;
        const int upp = on(JHI) ? NT + HP + i - tid : HP;
#pragma unroll
        for (int q = 0; q < NQ; q++) {
          if (!MHD && q >= Q_BX && q < Q_VX) continue;
          const R* w = s_p + q * PQ;
          const R c = w[0];
          if (q != Q_BX)
            s_h[hslot(0, q) * NT] = half_slope<R, RECON>(w[lft], c, w[rgt], theta);
          if (q != Q_BX + 1)
            s_h[hslot(1, q) * NT] = half_slope<R, RECON>(w[dwn], c, w[upp], theta);
        }
      }
    };

    // ---- column state.  NN: the primitives of planes t and t+1 stay in shared
    // memory.  PLM, at iteration t: w1 the primitives of plane t+1, hz half
    // their z slope; in shared memory the state on the low side of the z-face
    // t+1/2 (s_lz) and plane t+2's primitives (s_w2)
    R w1[NQ], hz[NQ];
    R zp[7];  // z fluxes at t+1/2: rho, mom, E, eint, vbar
    R bz_lo = R(0);
    R p_t = R(0), p_n = R(0);  // floored pressure of plane t, t+1 (dual energy)
#pragma unroll
    for (int q = 0; q < NQ; q++) w1[q] = hz[q] = R(0);
#pragma unroll
    for (int k = 0; k < 7; k++) zp[k] = R(0);

    // ---- prologue: plane t0 published (PLM: and t0 - 1, t0 + 1 held)
    {
      R wa[NQ], wc[NQ];
#pragma unroll
      for (int q = 0; q < NQ; q++) wa[q] = wc[q] = R(0);
      auto have = [&](int p) { return inr(p, s, T.m2 - s); };
      auto fetch = [&](int p, R* w) {
        if (on(CELL) && have(p)) {
          load((size_t)p * T.szb + cb, w);
          prims(w);
        }
      };
      fetch(t0, w1);
      if (on(CELL) && have(t0)) {
        put(plane_p(t0), PQ, w1);
        put_ec(t0, w1);
        put_gas(t0, w1);
      }
      if constexpr (!NN) {
        fetch(t0 - 1, wa);
        fetch(t0 + 1, wc);
        if (on(CELL) && have(t0 + 1)) put(s_w2, NT, wc);
#pragma unroll
        for (int q = 0; q < NQ; q++) hz[q] = half_slope<R, RECON>(wa[q], w1[q], wc[q], theta);
        if (on(RING) && have(t0)) {
          load((size_t)t0 * T.szb + rcell, wa);
          prims(wa);
          put(s_p0 + NT, PQ, wa);
        }
        __syncthreads();
        slopes();
      }
      __syncthreads();
    }

    // face B along x, y (plane t+1) and z (face t+1), loaded ahead of their use
    R bfx = R(0), bfy = R(0), bfz = R(0);
    auto load_bface = [&](int t) {
      if (!MHD) return;
      const int pl = t + 1;
      if (inr(pl, S, T.m2 - S)) {
        if (on(FX)) bfx = ldb(B.cur.f[0], (size_t)pl * T.fxzb + (xb_ + (int)sizeof(R)));
        if (on(FY)) bfy = ldb(B.cur.f[1], (size_t)pl * T.fyzb + (cb + T.rowb));
      }
      if (on(FZ) && inr(t, S, T.m2 - 1 - S)) bfz = ldb(B.cur.f[2], (size_t)pl * T.szb + cb);
    };
    load_bface(t0 - 1);

    for (int t = t0 - 1; t < zb; t++) {
      const bool first = t < t0;  // only the x- and y-faces of plane t0
      const int pl = t + 1;
      // the cells of the plane after next (NN: the next one)
      const int nxt = NN ? t + 2 : t + 3;
      const bool more = t + 1 < zb;
      // ---- B: Riemann solves
      // (EnzoReconstructorNN.cpp:14-49, EnzoReconstructorPLM.hpp:167-345);
      // the longitudinal B is the face's own (EnzoBfieldMethodCT.cpp:122-166)
      FaceFlux<R> F;
      // gl, gr: the gas quantities of the cells at the face (FP64 NN)
      auto solve = [&](auto dir, R bf, auto left, auto right, const R* gl, const R* gr) {
        constexpr int d = decltype(dir)::value, d1 = (d + 1) % 3, d2 = (d + 2) % 3;
        R wl[8], wr[8];
        constexpr int q_of[8] = {Q_RHO, Q_BX + d, Q_BX + d1, Q_BX + d2,
                                 Q_VX + d, Q_VX + d1, Q_VX + d2, Q_P};
#pragma unroll
        for (int k = 0; k < 8; k++) {
          if (k == L_BI) {
            wl[k] = wr[k] = MHD ? bf : R(0);
          } else if (!MHD && (k == L_BJ || k == L_BK)) {
            wl[k] = wr[k] = R(0);
          } else {
            wl[k] = left(q_of[k]);
            wr[k] = right(q_of[k]);
          }
        }
        if (!NN) {
          wl[L_RHO] = smax(wl[L_RHO], dfloor);
          wr[L_RHO] = smax(wr[L_RHO], dfloor);
          wl[L_E] = smax(wl[L_E], pfloor);
          wr[L_E] = smax(wr[L_E], pfloor);
        }
        if constexpr (F32) {
          riemann<SOLVER>(g, wl, wr, F);
        } else {
          const Gas gas = {phys.gamma, phys.gm1, phys.inv_gm1};
          if constexpr (L::NG > 0) {
            CellGas<SOLVER> cl, cr;
#pragma unroll
            for (int k = 0; k < L::NG; k++) {
              cl.v[k] = gl[k * NT];
              cr.v[k] = gr[k * NT];
            }
            riemann<SOLVER>(gas, wl, wr, cl, cr, F);
          } else {
            riemann<SOLVER>(gas, wl, wr, F);
          }
        }
      };
      // boundary fluxes for flux correction (EnzoMethodMHDVlct.cpp:250-330):
      // on the final stage, dt/dx times the flux through the block's active
      // boundary faces, each by the tile (and z-chunk) that owns the cell on
      // its high side, or the last cell along the axis
      auto store_face = [&](int d, int side, size_t at) {
        const FluxOut<R>* fo = reinterpret_cast<const FluxOut<R>*>(s_fo_raw);
        const R sc = T.dtdx[d];
        const R v[6] = {F.f[L_RHO], F.f[L_VI + (3 - d) % 3], F.f[L_VI + (4 - d) % 3],
                        F.f[L_VI + (5 - d) % 3], F.f[L_E], DE ? F.eflux : R(0)};
#pragma unroll
        for (int q = 0; q < 6; q++) {
          R* p = fo->f[d][side][q];
          if (p) p[at] = sc * v[q];
        }
      };
      const int gg = info.fc_g;
      // the column's (and its tile's) place again, only where fluxes are stored
      auto place = [&](int& x, int& y, int& i, int& j) {
        j = tid / T.HP;
        i = tid - j * T.HP;
        x = tl.xa - 1 + i;
        y = tl.ya - 1 + j;
      };
      // x- and y-faces of plane t+1
      auto put_face = [&](R* f, int d) {
        f[fd(pl, 0)] = F.f[L_RHO];
        if (MHD) {
          s_ww[(2 * d + (pl & 1)) * NT] = upw(F.f[L_RHO]);
          f[fd(pl, 1)] = F.f[L_BJ];
          f[fd(pl, 2)] = F.f[L_BK];
        }
        f[fs(0)] = F.f[L_VI + (3 - d) % 3];
        f[fs(1)] = F.f[L_VI + (4 - d) % 3];
        f[fs(2)] = F.f[L_VI + (5 - d) % 3];
        f[fs(3)] = F.f[L_E];
        if (DE) {
          f[fs(4)] = F.eflux;
          f[fs(5)] = F.vbar;
        }
      };
      const bool plane_ok = inr(pl, S, T.m2 - S);
      const R* const s_p = plane_p(pl);
      if (plane_ok && on(FX)) {
        const R* w = s_p + 1;
        solve(std::integral_constant<int, 0>{}, bfx,
              [&](int q) { return NN ? s_p[q * PQ] : w1[q] + s_h[hslot(0, q) * NT]; },
              [&](int q) { return NN ? w[q * PQ] : w[q * PQ] - s_h[hslot(0, q) * NT + 1]; },
              plane_cg(pl), plane_cg(pl) + 1);
        put_face(s_xf, 0);
        if (EXTRA != EXTRA_NONE && store_fc) {
          int x, y, i, j;
          place(x, y, i, j);
          const int side = x == gg - 1 ? 0 : (x == T.m0 - gg - 1 ? 1 : -1);
          if (side >= 0 && (i < T.HP - 2 || on(XHI)) && j >= 1 && j <= tl.yb - tl.ya && inr(y, gg, T.m1 - gg) &&
              pl >= T.za && pl < zb && inr(pl, gg, T.m2 - gg))
            store_face(0, side, (size_t)(pl - gg) * (T.m1 - 2 * gg) + (y - gg));
        }
      }
      if (plane_ok && on(FY)) {
        const R* w = s_p + T.HP;
        const R* h = s_h + T.HP;
        solve(std::integral_constant<int, 1>{}, bfy,
              [&](int q) { return NN ? s_p[q * PQ] : w1[q] + s_h[hslot(1, q) * NT]; },
              [&](int q) { return NN ? w[q * PQ] : w[q * PQ] - h[hslot(1, q) * NT]; },
              plane_cg(pl), plane_cg(pl) + T.HP);
        put_face(s_yf, 1);
        if (EXTRA != EXTRA_NONE && store_fc) {
          int x, y, i, j;
          place(x, y, i, j);
          const int side = y == gg - 1 ? 0 : (y == T.m1 - gg - 1 ? 1 : -1);
          if (side >= 0 && (j < tl.yb - tl.ya || on(YHI)) && i >= 1 && i <= T.HP - 2 && inr(x, gg, T.m0 - gg) &&
              pl >= T.za && pl < zb && inr(pl, gg, T.m2 - gg))
            store_face(1, side, (size_t)(pl - gg) * (T.m0 - 2 * gg) + (x - gg));
        }
      }
      // z-face at t+1/2
      if (!first && on(FZ) && inr(t, S, T.m2 - 1 - S)) {
        solve(std::integral_constant<int, 2>{}, bfz,
              [&](int q) { return NN ? plane_p(t)[q * PQ] : s_lz[q * NT]; },
              [&](int q) { return NN ? s_p[q * PQ] : w1[q] - hz[q]; }, plane_cg(t), plane_cg(pl));
        zp[0] = F.f[L_RHO];
        zp[1] = F.f[L_VJ];
        zp[2] = F.f[L_VK];
        zp[3] = F.f[L_VI];
        zp[4] = F.f[L_E];
        if (DE) {
          zp[5] = F.eflux;
          zp[6] = F.vbar;
        }
        if (MHD) {
          s_zf[0] = upw(F.f[L_RHO]);
          s_zf[NT] = F.f[L_BJ];
          s_zf[2 * NT] = F.f[L_BK];
        }
        if (EXTRA != EXTRA_NONE && store_fc && on(OUT)) {
          const int side = t == gg - 1 ? 0 : (t == T.m2 - gg - 1 ? 1 : -1);
          if (side >= 0 && t >= T.za - 1 && (t < zb - 1 || t + 1 == T.m2 - T.olo)) {
            int x, y, i, j;
            place(x, y, i, j);
            if (inr(x, gg, T.m0 - gg) && inr(y, gg, T.m1 - gg))
              store_face(2, side, (size_t)(y - gg) * (T.m0 - 2 * gg) + (x - gg));
          }
        }
      }
      if constexpr (!NN) {
#pragma unroll
        for (int q = 0; q < NQ; q++)
          if (MHD || q < Q_BX || q >= Q_VX) s_lz[q * NT] = w1[q] + hz[q];
      }
      __syncthreads();

      // ---- C.  First the loads: the next cells, and plane t's start-of-step
      // values for its update in D; their latency passes under the rest of C
      const int HP = T.HP;
      R in[NQ], rin[NQ];
      const bool in_on = more && on(CELL) && inr(nxt, s, T.m2 - s);
      const bool rin_on = !NN && more && on(RING) && inr(t + 2, s, T.m2 - s);
      if (in_on) load((size_t)nxt * T.szb + cb, in);
      if constexpr (!NN) {
        if (rin_on) load((size_t)(t + 2) * T.szb + rcell, rin);
      }
      R base[6], bf[5];  // rho, v, etot, eint; face B: x, x+1, y, y+1, z+1
      if (!first && on(OUT)) {
        const size_t c = (size_t)t * T.szb + cb;
        if (MHD) bf[4] = ldb(B.base.f[2], c + T.szb);
        if (t >= T.za) {  // (plane za - 1 may lie below the block)
          if (MHD) {
            const size_t xo = (size_t)t * T.fxzb + xb_, yo = (size_t)t * T.fyzb + cb;
            bf[0] = ldb(B.base.f[0], xo);
            bf[1] = ldb(B.base.f[0], xo + sizeof(R));
            bf[2] = ldb(B.base.f[1], yo);
            bf[3] = ldb(B.base.f[1], yo + T.rowb);
          }
#pragma unroll
          for (int k = 0; k < 5; k++) base[k] = ldb(B.base.c[F_RHO + k], c);
          if (DE) base[5] = ldb(B.base.c[F_EINT], c);
        }
      }
      // edge EMFs (EnzoBfieldMethodCT.cpp:480-590)
      if (MHD && !first) {
        const R *xf0 = s_xf + fd(t, 0), *xf1 = s_xf + fd(pl, 0);
        const R *yf0 = s_yf + fd(t, 0), *yf1 = s_yf + fd(pl, 0);
        const R *bj = s_zf + NT, *bk = s_zf + 2 * NT;
        const R* ec0 = s_ec + (t % L::NEC) * 3 * NT;
        const R* ec1 = s_ec + (pl % L::NEC) * 3 * NT;
        const bool zt = inr(t, S, T.m2 - S - 1);
        const R *wx = s_ww + (t & 1) * NT, *wy = wx + 2 * NT;
        const R Wx0 = wx[0], Wx1 = s_ww[(pl & 1) * NT], Wy0 = wy[0],
                Wy1 = s_ww[(2 + (pl & 1)) * NT], Wz = s_zf[0];
        if (on(EX) && zt)  // E_x at (x, y+1/2, t+1/2)
          s_ex[(t & 1) * NT] = edge_emf<R>(yf0[NT], yf1[NT], bk[0], bk[HP], Wy0, Wy1, Wz,
                                           s_zf[HP], ec0[0], ec0[HP], ec1[0], ec1[HP]);
        if (on(EY) && zt)  // E_y at (x+1/2, y, t+1/2)
          s_ey[(t & 1) * NT] =
              edge_emf<R>(bj[0], bj[1], xf0[2 * NT], xf1[2 * NT], Wz, s_zf[1], Wx0, Wx1,
                          ec0[NT], ec1[NT], ec0[NT + 1], ec1[NT + 1]);
        if (on(EZ) && inr(t, S + 1, T.m2 - S - 1))  // E_z at (x+1/2, y+1/2, t)
          s_ez[0] = edge_emf<R>(xf0[NT], xf0[NT + HP], yf0[2 * NT], yf0[2 * NT + 1], Wx0,
                                wx[HP], Wy0, wy[1], ec0[2 * NT], ec0[2 * NT + 1],
                                ec0[2 * NT + HP], ec0[2 * NT + HP + 1]);
      }
      // flux divergence of plane t+1 along x, then y
      // (EnzoIntegrationQuanUpdate.cpp:105-147, EnzoSourceInternalEnergy.cpp:16-92);
      // plane t's moves to registers, for its update
      R dxy[6];
      if (on(UPD) && plane_ok) {
#pragma unroll
        for (int k = 0; k < (DE ? 6 : 5); k++) dxy[k] = s_dx[k * NT];
        const R dtdx0 = T.dtdx[0], dtdx1 = T.dtdx[1];
        const R *xr = s_xf + fd(pl, 0), *yr = s_yf + fd(pl, 0);
        R a = R(0.0);
        a -= dtdx0 * (xr[0] - xr[-1]);
        a -= dtdx1 * (yr[0] - *(yr - HP));
        s_dx[0] = a;
#pragma unroll
        for (int k = 0; k < 4; k++) {
          const R *xk = s_xf + fs(k), *yk = s_yf + fs(k);
          a = R(0.0);
          a -= dtdx0 * (xk[0] - xk[-1]);
          a -= dtdx1 * (yk[0] - *(yk - HP));
          s_dx[(1 + k) * NT] = a;
        }
        if (DE) {
          p_n = smax(NN ? s_p[Q_P * PQ] : w1[Q_P], pfloor);
          const R *xe = s_xf + fs(4), *xv = s_xf + fs(5), *ye = s_yf + fs(4), *yv = s_yf + fs(5);
          a = R(0.0);
          a -= dtdx0 * (xe[0] - xe[-1]);
          a -= dtdx0 * p_n * (xv[0] - xv[-1]);
          a -= dtdx1 * (ye[0] - *(ye - HP));
          a -= dtdx1 * p_n * (yv[0] - *(yv - HP));
          s_dx[5 * NT] = a;
        }
        // the passive scalars' advection (passive_kernel) needs the density
        // flux of both faces of every updated cell along each axis: the low
        // faces, and the high ones at the region's edges
        if (EXTRA == EXTRA_ALL && info.npass > 0 && pl >= T.za && pl < zb &&
            inr(pl, S + 1, T.m2 - S - 1)) {
          const size_t c = (size_t)pl * T.szb + cb;
          stb(B.dflux[0], c, xr[-1]);
          stb(B.dflux[1], c, *(yr - HP));
          int x, y, i, j;
          place(x, y, i, j);
          if (x + 1 == T.m0 - S - 1) stb(B.dflux[0], c + sizeof(R), xr[0]);
          if (y + 1 == T.m1 - S - 1) stb(B.dflux[1], c + T.rowb, yr[0]);
        }
      }
      // the next plane's primitives and cell-centred E; plane t+1 is no
      // longer read
      if (more) {
        if constexpr (NN) {
          if (in_on) {
            prims(in);
            put(plane_p(nxt), PQ, in);
            put_ec(nxt, in);
            put_gas(nxt, in);
          }
        } else {
          R w2[NQ];
#pragma unroll
          for (int q = 0; q < NQ; q++)
            w2[q] = (!MHD && q >= Q_BX && q < Q_VX) ? R(0) : s_w2[q * NT];
          if (on(CELL) && inr(t + 2, s, T.m2 - s)) put(s_p0, PQ, w2);
          if (in_on) {
            prims(in);
            put(s_w2, NT, in);
#pragma unroll
            for (int q = 0; q < NQ; q++)
              hz[q] = half_slope<R, RECON>(w1[q], w2[q], in[q], theta);
          }
#pragma unroll
          for (int q = 0; q < NQ; q++) w1[q] = w2[q];
          if (rin_on) {
            prims(rin);
            put(s_p0 + NT, PQ, rin);
          }
        }
        load_bface(t + 1);
      }
      __syncthreads();

      // ---- D: the constrained-transport face updates around cell (x, y, t)
      // (EnzoBfieldMethodCT.cpp:617-687) -- Bz at the face t+1 above it and,
      // when plane t is output, Bx at faces x, x+1 and By at faces y, y+1 --
      // then the cell's update.  A face between two cells of the tile is
      // computed by both (the same expression) and written by the one that
      // owns it: the cell on its high side, or the cell below the block's
      // outermost written face.  A face not updated in this stage keeps its
      // start-of-step value.
      if (on(OUT) && !first) {
        const bool do_plane = t >= T.za;
        const bool in_t = inr(t, S + 1, T.m2 - S - 1);
        const size_t c = (size_t)t * T.szb + cb;
        const R dtdx0 = T.dtdx[0], dtdx1 = T.dtdx[1], dtdx2 = T.dtdx[2];
        R bcx = R(0), bcy = R(0), bcz = R(0);
        if (MHD) {
          const R *ex = s_ex + (t & 1) * NT, *exm = s_ex + ((t - 1) & 1) * NT;
          const R *ey = s_ey + (t & 1) * NT, *eym = s_ey + ((t - 1) & 1) * NT;
          // Bz at face t+1
          R bz_hi = bf[4];
          if (on(UPD) && inr(t + 1, S + 1, T.m2 - S)) {
            const R Ek_term = dtdx0 * (ey[0] - ey[-1]);
            const R Ej_term = dtdx1 * (ex[0] - *(ex - HP));
            bz_hi = bz_hi - Ek_term + Ej_term;
            // the lowest face of a chunk is written by the chunk below it
            if (do_plane || T.za == T.olo) stb(B.out.f[2], c + T.szb, bz_hi);
          }
          if (do_plane) {
            const size_t xo = (size_t)t * T.fxzb + xb_, yo = (size_t)t * T.fyzb + cb;
            // Bx at faces x, x+1: E_z at (kx-1/2, y -+ 1/2), E_y at (kx-1/2, t -+ 1/2)
            R b[2];
#pragma unroll
            for (int k = 0; k < 2; k++) {
              b[k] = bf[k];
              if (on(k == 0 ? XLO : XUP) && on(UY) && in_t) {
                const R Ek_term = dtdx1 * (s_ez[k - 1] - *(s_ez + (k - 1) - HP));
                const R Ej_term = dtdx2 * (ey[k - 1] - eym[k - 1]);
                b[k] = b[k] - Ek_term + Ej_term;
                if (k == 0 || on(XHI)) stb(B.out.f[0], xo + k * sizeof(R), b[k]);
              }
            }
            bcx = R(0.5) * (b[0] + b[1]);
            // By at faces y, y+1: E_x at (x, ky-1/2, t -+ 1/2), E_z at (x -+ 1/2, ky-1/2)
#pragma unroll
            for (int k = 0; k < 2; k++) {
              const size_t o = yo + k * T.rowb;
              b[k] = bf[2 + k];
              if (on(k == 0 ? YLO : YUP) && on(UX) && in_t) {
                const int e = (k - 1) * HP;
                const R Ek_term = dtdx2 * (ex[e] - exm[e]);
                const R Ej_term = dtdx0 * (s_ez[e] - s_ez[e - 1]);
                b[k] = b[k] - Ek_term + Ej_term;
                if (k == 0 || on(YHI)) stb(B.out.f[1], o, b[k]);
              }
            }
            bcy = R(0.5) * (b[0] + b[1]);
            // compute_center_bfield (EnzoBfieldMethodCT.cpp:702-728)
            bcz = R(0.5) * (bz_lo + bz_hi);
            stb(B.out.c[F_BX], c, bcx);
            stb(B.out.c[F_BY], c, bcy);
            stb(B.out.c[F_BZ], c, bcz);
          }
          bz_lo = bz_hi;
        }
        if (do_plane && on(UPD) && in_t) {
          R du[6];
#pragma unroll
          for (int k = 0; k < 5; k++) du[k] = dxy[k] - dtdx2 * (zp[k] - s_zm[k * NT]);
          if (DE) {
            R a = dxy[5];
            a -= dtdx2 * (zp[5] - s_zm[5 * NT]);
            a -= dtdx2 * p_t * (zp[6] - s_zm[6 * NT]);
            du[5] = a;
          }
          const R old_rho = base[0], ovx = base[1], ovy = base[2], ovz = base[3], oet = base[4];
          R eint = DE ? base[5] : R(0);
          // gravity source on the full-dt stage (EnzoSourceGravity.cpp:17-69,
          // EnzoMHDIntegratorStageCommands.cpp:267-297): start-of-step
          // density and velocity
          if (EXTRA == EXTRA_ALL && info.gravity) {
            const R dt = T.dt;
            const R ax = ldb(B.accel[0], c), ay = ldb(B.accel[1], c), az = ldb(B.accel[2], c);
            du[1] += dt * old_rho * ax;
            du[2] += dt * old_rho * ay;
            du[3] += dt * old_rho * az;
            du[4] += dt * old_rho * ((ovx * ax) + (ovy * ay) + (ovz * az));
          }
          // update_quantities (EnzoIntegrationQuanUpdate.cpp:183-231)
          R new_rho = old_rho + du[0];
          new_rho = smax(new_rho, dfloor);
          const R inv_new_rho = R(1.) / new_rho;
          const R vx = (ovx * old_rho + du[1]) * inv_new_rho;
          const R vy = (ovy * old_rho + du[2]) * inv_new_rho;
          const R vz = (ovz * old_rho + du[3]) * inv_new_rho;
          R etot = (oet * old_rho + du[4]) * inv_new_rho;
          if (DE) eint = (eint * old_rho + du[5]) * inv_new_rho;
          // apply_floor_to_energy_and_sync (EnzoPhysicsFluidProps.cpp:162-290)
          energy_floor_sync<MHD, DE>(econ, new_rho, vx, vy, vz, bcx, bcy, bcz, etot, eint);
          stb(B.out.c[F_RHO], c, new_rho);
          stb(B.out.c[F_VX], c, vx);
          stb(B.out.c[F_VY], c, vy);
          stb(B.out.c[F_VZ], c, vz);
          stb(B.out.c[F_ETOT], c, etot);
          if (DE) stb(B.out.c[F_EINT], c, eint);
          if (EXTRA == EXTRA_ALL && info.npass > 0) {
            stb(B.dflux[2], c, s_zm[0]);
            if (t + 1 == T.m2 - S - 1) stb(B.dflux[2], c + T.szb, zp[0]);
          }
        }
#pragma unroll
        for (int k = 0; k < (DE ? 7 : 5); k++) s_zm[k * NT] = zp[k];
      }
      p_t = p_n;
      // ---- A: the slopes of plane t+2, for the next plane's faces, and its
      // cell-centred E (in the buffer of plane t, no longer read)
      if constexpr (!NN) {
        if (more) {
          put_ec(t + 2, w1);
          slopes();
          __syncthreads();
        }
      }
    }
    // next tile: dynamic queue (persistent grid) or static grid stride
    __syncthreads();
    if (info.queue) {
      if (tid == 0) s_next = atomicAdd(info.queue, 1);
      __syncthreads();
      it = s_next;
    } else {
      it += gridDim.x;
    }
  }
}

// On the final stage the reference also recomputes the cell-centred B of the one
// layer of cells around the updated region, from faces of which the stage has
// updated some (EnzoBfieldMethodCT.cpp:702-728).  The stage kernel's tiles cover
// the updated region alone: as columns and planes of its march that layer made
// a 32^3 block 34^3 zones, and 16^3 18^3.  This kernel, on the same tiles after
// it, gives each tile the layer's cells next to it.  It moves nine values a cell
// of the layer: 56 us for 216 blocks of 32^3 (DRAM 36 B a zone).  With it and the
// tiles that fit_tile then takes, the full-dt stage of 512 blocks of 32^3 with
// dual energy takes 2.94 instead of 3.71 ms, and the cycle of the 256^3 box
// without it 5.65 instead of 6.28 ms.
template <class R>
__global__ void __launch_bounds__(128)
ring_bfield_kernel(const StageBlock<R>* __restrict__ blocks, const StageTile* __restrict__ tiles,
                   StageInfo info) {
  const StageTile tl = tiles[blockIdx.x];
  const StageBlock<R>& B = blocks[tl.block];
  const int S = info.S, m0 = B.m[0], m1 = B.m[1], m2 = B.m[2];
  // how far the tile's box reaches into the layer on each side (0 or 1)
  const int xl = tl.xa == S + 1, xh = tl.xb == m0 - S - 1;
  const int yl = tl.ya == S + 1, yh = tl.yb == m1 - S - 1;
  const int zl = tl.za == S + 1, zh = tl.zb == m2 - S - 1;
  const int nx = tl.xb - tl.xa, ny = tl.yb - tl.ya, nz = tl.zb - tl.za;
  const int ex = nx + xl + xh, ey = ny + yl + yh;
  const int cz = (zl + zh) * ex * ey, cy = nz * (yl + yh) * ex, cx = nz * ny * (xl + xh);
  const R *ox = B.out.f[0], *oy = B.out.f[1], *oz = B.out.f[2];
  const R *bx = B.base.f[0], *by = B.base.f[1], *bz = B.base.f[2];
  R *cbx = B.out.c[F_BX], *cby = B.out.c[F_BY], *cbz = B.out.c[F_BZ];
  for (int q = threadIdx.x; q < cz + cy + cx; q += blockDim.x) {
    int x, y, t;
    if (q < cz) {
      const int r = q / ex;
      x = tl.xa - xl + (q - r * ex);
      const int k = r / ey;
      y = tl.ya - yl + (r - k * ey);
      t = zl && k == 0 ? tl.za - 1 : tl.zb;
    } else if (q < cz + cy) {
      const int p = q - cz, r = p / ex;
      x = tl.xa - xl + (p - r * ex);
      const int k = r / nz;
      t = tl.za + (r - k * nz);
      y = yl && k == 0 ? tl.ya - 1 : tl.yb;
    } else {
      const int p = q - cz - cy, r = p / ny;
      y = tl.ya + (p - r * ny);
      const int k = r / nz;
      t = tl.za + (r - k * nz);
      x = xl && k == 0 ? tl.xa - 1 : tl.xb;
    }
    const bool ux = inr(x, S + 1, m0 - S - 1), uy = inr(y, S + 1, m1 - S - 1),
               uz = inr(t, S + 1, m2 - S - 1);
    const size_t c = ((size_t)t * m1 + y) * m0 + x;
    const size_t fx = ((size_t)t * m1 + y) * (m0 + 1) + x;
    const size_t fy = ((size_t)t * (m1 + 1) + y) * m0 + x;
    const size_t szz = (size_t)m0 * m1;
    R v[6];
#pragma unroll
    for (int k = 0; k < 2; k++) {
      v[k] = (uy && uz && inr(x + k, S + 1, m0 - S) ? ox : bx)[fx + k];
      v[2 + k] = (ux && uz && inr(y + k, S + 1, m1 - S) ? oy : by)[fy + (size_t)k * m0];
      v[4 + k] = (ux && uy && inr(t + k, S + 1, m2 - S) ? oz : bz)[c + (size_t)k * szz];
    }
    cbx[c] = R(0.5) * (v[0] + v[1]);
    cby[c] = R(0.5) * (v[2] + v[3]);
    cbz[c] = R(0.5) * (v[4] + v[5]);
  }
}

}  // namespace vlct
