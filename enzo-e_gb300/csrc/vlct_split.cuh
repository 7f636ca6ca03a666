// vlct_split.cuh -- one VL+CT stage as a sequence of small kernels over whole
// blocks: primitives, face fluxes, edge EMFs, update.
//
// The FP64 stages run this way.  GB300's FP64 pipe retires two operations per
// clock and SM (1/64 of FP32), so an FP64 stage costs what it executes on that
// pipe and nothing else: memory traffic, integer work and launches are free
// beside it.  The fused kernel (vlct_stage.cuh) solves the halo faces of every
// tile again; here every face is solved once, the intermediate arrays pass
// through global memory (about 1.3 KB per cell and stage, 3% of the pipe's
// time), and the PLM slope of a cell is formed once per direction: a thread
// marches along a line of faces and carries the state to the left of the next
// face in registers.
//
// The index windows and the order of operations are the fused kernel's (the
// reference's), so the FP64 results are the same bit for bit.
//
// Measured (HLLD + PLM): a 128^3 box of 64 blocks of 32^3, one cycle, 37.9 ms
// with a fused kernel and the reference's own HLLD branches, 14.9 ms here; one
// 32^3 block through the Method (dt, ghosts, step) 981 -> 386 us.  The FP64 pipe
// is 84-86% busy in the flux kernels, which take 85% of the stages' time at 333
// (NN) and 413 (PLM) pipe operations a face, idle lanes included.
//
// Work is cut into jobs: one block, or a z-slab of one, with its slice of the
// workspace.  A launch covers a group of jobs (blockIdx.y), so the workspace
// stays bounded whatever the size of the batch.  MHD blocks of planes too wide
// for slabs of five run the fused kernel (split_plan).
#pragma once
#include "vlct_stage.cuh"

namespace vlct {

// Workspace arrays of one job, in the ghosted block's x and y extents and the
// planes [za - 2, zb + 2): pressure, cell-centred E (3), face fluxes (3 x NF),
// edge EMFs (3), the cells' gas quantities (CellGas: up to 4, NN stages).  A face
// or edge value sits at the cell on its low side.
template <bool MHD, bool DE> struct SplitLayout {
  static constexpr int NF = DE ? 9 : (MHD ? 7 : 5);
  static constexpr int P = 0, EC = 1, F = EC + (MHD ? 3 : 0), EMF = F + 3 * NF,
                       CG = EMF + (MHD ? 3 : 0), N = CG + 4;
  static_assert(N == split_arrays(MHD, DE), "workspace arrays");
};

// one job as the CTAs of a launch see it, set up once per CTA
template <class R> struct SplitCtx {
  int m0, m1, m2, za, zb;
  size_t sy, sz, M;  // strides of a cell array, elements of a workspace array
  R* ws;
  // workspace index of the cell (x, y, z)
  __device__ size_t at(int x, int y, int z) const {
    return (size_t)(z - (za - 2)) * sz + (size_t)y * sy + x;
  }
};
template <class R>
__device__ __forceinline__ SplitCtx<R> split_ctx(const StageBlock<R>& B, const SplitJob& J,
                                                 R* ws) {
  SplitCtx<R> C;
  C.m0 = B.m[0];
  C.m1 = B.m[1];
  C.m2 = B.m[2];
  C.za = J.za;
  C.zb = J.zb;
  C.sy = (size_t)C.m0;
  C.sz = (size_t)C.m0 * C.m1;
  C.M = C.sz * (size_t)(J.zb - J.za + 4);
  C.ws = ws + J.off;
  return C;
}

// ---- primitives: the pressure of every cell the fluxes read, the gas
// quantities that the faces of a cell share in an NN stage, and the cell-centred
// E = -v x B (EnzoComputePressure.cpp:127-190, EnzoBfieldMethodCT.cpp:267-292)
template <class R, int SOLVER, bool NN, bool DE>
__global__ void __launch_bounds__(kSplitThreads)
split_prim_kernel(const StageBlock<R>* __restrict__ blocks, const SplitJob* __restrict__ jobs,
                  R* __restrict__ ws, StageInfo info, PhysParams phys) {
  constexpr bool MHD = SOLVER != SOLVER_HLLC;
  using L = SplitLayout<MHD, DE>;
  const SplitJob J = jobs[blockIdx.y];
  const StageBlock<R>& B = blocks[J.block];
  const SplitCtx<R> C = split_ctx(B, J, ws);
  const int s = info.s, S = info.S;
  const int z0 = max(s, C.za - 2), z1 = min(C.m2 - s, C.zb + 2);
  const int nx = C.m0 - 2 * s, ny = C.m1 - 2 * s;
  EnergyConsts<R> econ;
  econ.init(phys, DE);
  const int n = nx * ny * (z1 - z0);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int r = i / nx, x = s + (i - r * nx);
    const int q = r / ny, y = s + (r - q * ny), z = z0 + q;
    const size_t c = (size_t)z * C.sz + (size_t)y * C.sy + x, w = C.at(x, y, z);
    const R rho = B.cur.c[F_RHO][c];
    R vx = R(0), vy = R(0), vz = R(0), bx = R(0), by = R(0), bz = R(0);
    if (MHD || !DE) {
      vx = B.cur.c[F_VX][c];
      vy = B.cur.c[F_VY][c];
      vz = B.cur.c[F_VZ][c];
    }
    if (MHD) {
      bx = B.cur.c[F_BX][c];
      by = B.cur.c[F_BY][c];
      bz = B.cur.c[F_BZ][c];
    }
    const R e = B.cur.c[DE ? F_EINT : F_ETOT][c];
    const R p = DE ? econ.gm1 * rho * e
                   : pressure_from_etot<R, MHD>(econ, rho, e, vx, vy, vz, bx, by, bz);
    C.ws[L::P * C.M + w] = p;
    if (NN) {
      CellGas<SOLVER> cg;
      cg.init(Gas{phys.gamma, phys.gm1, phys.inv_gm1}, rho, p);
#pragma unroll
      for (int k = 0; k < CellGas<SOLVER>::N; k++) C.ws[(L::CG + k) * C.M + w] = cg.v[k];
    }
    if (MHD && inr(x, S, C.m0 - S) && inr(y, S, C.m1 - S) && inr(z, S, C.m2 - S)) {
      C.ws[(L::EC + 0) * C.M + w] = (-vy * bz + vz * by);
      C.ws[(L::EC + 1) * C.M + w] = (-vz * bx + vx * bz);
      C.ws[(L::EC + 2) * C.M + w] = (-vx * by + vy * bx);
    }
  }
}

// ---- face fluxes along direction blockIdx.z.  A thread takes up to K
// consecutive faces of one line; with PLM it carries each quantity's state on
// the low side of the next face, so a cell's slope is formed once (and once
// more where a line of faces is cut).  K: as many faces as leave the GPU's
// pipes filled (host), with the cut of the line that wastes least (below).
template <class R, int SOLVER, int RECON, bool DE>
__global__ void __launch_bounds__(kSplitThreads)
split_flux_kernel(const StageBlock<R>* __restrict__ blocks, const SplitJob* __restrict__ jobs,
                  R* __restrict__ ws, StageInfo info, PhysParams phys, int kmax) {
  constexpr bool MHD = SOLVER != SOLVER_HLLC;
  constexpr bool NN = RECON == RECON_NN;
  using L = SplitLayout<MHD, DE>;
  const SplitJob J = jobs[blockIdx.y];
  const StageBlock<R>& B = blocks[J.block];
  const SplitCtx<R> C = split_ctx(B, J, ws);
  const int S = info.S, d = blockIdx.z, d1 = (d + 1) % 3, d2 = (d + 2) % 3;
  // faces f (between cells f and f + 1 along d) and the cells across it whose
  // face is needed: with CT one more cell on each side, for the edge EMFs
  const int T = MHD ? S : S + 1;
  int lo[3], hi[3];
  const int m[3] = {C.m0, C.m1, C.m2};
#pragma unroll
  for (int a = 0; a < 3; a++) {
    lo[a] = T;
    hi[a] = m[a] - T;
    if (a == 2) {
      lo[a] = max(lo[a], MHD ? C.za - 1 : C.za);
      hi[a] = min(hi[a], MHD ? C.zb + 1 : C.zb);
    }
    if (a == d) {
      lo[a] = a == 2 ? max(S, C.za - 1) : S;
      hi[a] = a == 2 ? min(m[a] - 1 - S, C.zb) : m[a] - 1 - S;
    }
  }
  const int nf = hi[d] - lo[d];
  if (nf <= 0) return;
  // the faces per thread: of kmax/2 .. kmax (1 for NN) the number that costs a
  // line least, a cut costing about a tenth of a face
  __shared__ int s_k;
  __shared__ const R* s_q[8];
  if (threadIdx.x == 0) {
    int best = 1;
    if (!NN) {
      int cost = 1 << 30;
      for (int k = (kmax + 1) / 2; k <= kmax; k++) {
        const int c = ((nf + k - 1) / k) * (10 * k + 1);
        if (c < cost) {
          cost = c;
          best = k;
        }
      }
    }
    s_k = best;
    s_q[L_RHO] = B.cur.c[F_RHO];
    s_q[L_BI] = nullptr;
    s_q[L_BJ] = MHD ? B.cur.c[F_BX + d1] : nullptr;
    s_q[L_BK] = MHD ? B.cur.c[F_BX + d2] : nullptr;
    s_q[L_VI] = B.cur.c[F_VX + d];
    s_q[L_VJ] = B.cur.c[F_VX + d1];
    s_q[L_VK] = B.cur.c[F_VX + d2];
    // the pressure is indexed like the cell arrays below
    s_q[L_E] = C.ws + L::P * C.M - (size_t)(C.za - 2) * C.sz;
  }
  __syncthreads();
  const int K = s_k, nch = (nf + K - 1) / K;
  // items: (x, other axis, chunk) for d = y, z; (chunk, y, z) for d = x
  const int e0 = d == 0 ? nch : hi[0] - lo[0];
  const int e1 = d == 1 ? hi[2] - lo[2] : hi[1] - lo[1];
  const int e2 = d == 0 ? hi[2] - lo[2] : nch;
  const int n = e0 * e1 * e2;
  const size_t stride = d == 0 ? 1 : (d == 1 ? C.sy : C.sz);
  const R theta = R(phys.theta_limiter);
  const Gas gas = {phys.gamma, phys.gm1, phys.inv_gm1};
  const R dfloor = R(phys.density_floor), pfloor = R(phys.pressure_floor);
  // face B along d: its own strides
  const R* bf = MHD ? B.cur.f[d] : nullptr;
  const size_t by = d == 0 ? (size_t)(C.m0 + 1) : (size_t)C.m0;
  const size_t bz = d == 0 ? by * C.m1 : (d == 1 ? by * (C.m1 + 1) : by * C.m1);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int r = i / e0, i0 = i - r * e0, i2 = r / e1, i1 = r - i2 * e1;
    int p[3];
    int ch;
    if (d == 0) {
      ch = i0;
      p[1] = lo[1] + i1;
      p[2] = lo[2] + i2;
      p[0] = lo[0] + ch * K;
    } else {
      ch = i2;
      p[0] = lo[0] + i0;
      p[1] = d == 1 ? lo[1] + ch * K : lo[1] + i1;
      p[2] = d == 1 ? lo[2] + i1 : lo[2] + ch * K;
    }
    const int cnt = min(K, nf - ch * K);
    size_t c = (size_t)p[2] * C.sz + (size_t)p[1] * C.sy + p[0];
    size_t w = C.at(p[0], p[1], p[2]);
    const R* bface =
        MHD ? bf + ((size_t)p[2] * bz + (size_t)p[1] * by + p[0]) : nullptr;
    const size_t bstep = d == 0 ? 1 : (d == 1 ? by : bz);
    R wl[8], wr[8];
    wl[L_BI] = wr[L_BI] = R(0);
    if (!MHD) wl[L_BJ] = wr[L_BJ] = wl[L_BK] = wr[L_BK] = R(0);
    // PLM: the state on the low side of the first face, from the slope of cell c
    R carry[8];
    if (!NN) {
#pragma unroll
      for (int k = 0; k < 8; k++) {
        if (k == L_BI || (!MHD && (k == L_BJ || k == L_BK))) continue;
        const R* q = s_q[k] + c;
        const R a = *(q - stride), b = q[0], e = q[stride];
        carry[k] = b + half_slope<R, RECON>(a, b, e, theta);
      }
    }
    for (int f = 0; f < cnt; f++) {
#pragma unroll
      for (int k = 0; k < 8; k++) {
        if (k == L_BI || (!MHD && (k == L_BJ || k == L_BK))) continue;
        const R* q = s_q[k] + c;
        if (NN) {
          wl[k] = q[0];
          wr[k] = q[stride];
        } else {
          const R a = q[0], b = q[stride], e = q[2 * stride];
          const R h = half_slope<R, RECON>(a, b, e, theta);
          R lv = carry[k], rv = b - h;
          carry[k] = b + h;
          if (k == L_RHO) {
            lv = smax(lv, dfloor);
            rv = smax(rv, dfloor);
          } else if (k == L_E) {
            lv = smax(lv, pfloor);
            rv = smax(rv, pfloor);
          }
          wl[k] = lv;
          wr[k] = rv;
        }
      }
      if (MHD) {
        bface += bstep;
        wl[L_BI] = wr[L_BI] = *bface;
      }
      FaceFlux<R> F;
      if (NN) {
        CellGas<SOLVER> cl, cr;
        const R* cg = C.ws + (size_t)L::CG * C.M + w;
#pragma unroll
        for (int k = 0; k < CellGas<SOLVER>::N; k++) {
          cl.v[k] = cg[k * C.M];
          cr.v[k] = cg[k * C.M + stride];
        }
        riemann<SOLVER>(gas, wl, wr, cl, cr, F);
      } else {
        riemann<SOLVER>(gas, wl, wr, F);
      }
      R* dst = C.ws + (size_t)(L::F + d * L::NF) * C.M + w;
      dst[S_RHO * C.M] = F.f[L_RHO];
      dst[(S_MX + d) * C.M] = F.f[L_VI];
      dst[(S_MX + d1) * C.M] = F.f[L_VJ];
      dst[(S_MX + d2) * C.M] = F.f[L_VK];
      dst[S_E * C.M] = F.f[L_E];
      if (MHD) {
        dst[S_BJ * C.M] = F.f[L_BJ];
        dst[S_BK * C.M] = F.f[L_BK];
      }
      if (DE) {
        dst[S_EINT * C.M] = F.eflux;
        dst[S_VBAR * C.M] = F.vbar;
      }
      c += stride;
      w += stride;
    }
  }
}

// ---- edge EMFs (EnzoBfieldMethodCT.cpp:480-590): the three edges on the high
// side of each cell
template <class R, bool DE>
__global__ void __launch_bounds__(kSplitThreads)
split_emf_kernel(const StageBlock<R>* __restrict__ blocks, const SplitJob* __restrict__ jobs,
                 R* __restrict__ ws, StageInfo info) {
  using L = SplitLayout<true, DE>;
  const SplitJob J = jobs[blockIdx.y];
  const StageBlock<R>& B = blocks[J.block];
  const SplitCtx<R> C = split_ctx(B, J, ws);
  const int S = info.S;
  const int z0 = max(S, C.za - 1), z1 = min(C.m2 - S - 1, C.zb);
  const int nx = C.m0 - 2 * S - 1, ny = C.m1 - 2 * S - 1;
  const int n = nx * ny * (z1 - z0);
  const R* xf = C.ws + (size_t)(L::F + 0 * L::NF) * C.M;
  const R* yf = C.ws + (size_t)(L::F + 1 * L::NF) * C.M;
  const R* zf = C.ws + (size_t)(L::F + 2 * L::NF) * C.M;
  const R* ec = C.ws + (size_t)L::EC * C.M;
  R* em = C.ws + (size_t)L::EMF * C.M;
  const size_t sy = C.sy, sz = C.sz, M = C.M;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int r = i / nx, x = S + (i - r * nx);
    const int q = r / ny, y = S + (r - q * ny), z = z0 + q;
    const size_t w = C.at(x, y, z);
    const R fx = xf[w], fy = yf[w], fz = zf[w];
    if (x > S) {  // E_x at (x, y+1/2, z+1/2)
      em[w] = edge_emf<R>(yf[S_BJ * M + w], yf[S_BJ * M + w + sz], zf[S_BK * M + w],
                          zf[S_BK * M + w + sy], upw(fy), upw(yf[w + sz]), upw(fz),
                          upw(zf[w + sy]), ec[w], ec[w + sy], ec[w + sz], ec[w + sy + sz]);
    }
    if (y > S) {  // E_y at (x+1/2, y, z+1/2)
      const R* e = ec + M;
      em[M + w] = edge_emf<R>(zf[S_BJ * M + w], zf[S_BJ * M + w + 1], xf[S_BK * M + w],
                              xf[S_BK * M + w + sz], upw(fz), upw(zf[w + 1]), upw(fx),
                              upw(xf[w + sz]), e[w], e[w + sz], e[w + 1], e[w + sz + 1]);
    }
    if (z > S) {  // E_z at (x+1/2, y+1/2, z)
      const R* e = ec + 2 * M;
      em[2 * M + w] = edge_emf<R>(xf[S_BJ * M + w], xf[S_BJ * M + w + sy], yf[S_BK * M + w],
                                  yf[S_BK * M + w + 1], upw(fx), upw(xf[w + sy]), upw(fy),
                                  upw(yf[w + 1]), e[w], e[w + 1], e[w + sy], e[w + sy + 1]);
    }
  }
}

// ---- update: the face B around each output cell, its centred B, the cell's
// conserved update, floors and energy sync, the stored boundary fluxes and the
// density fluxes of the passive scalars (phase D of the fused kernel)
template <class R, bool MHD, bool DE>
__global__ void __launch_bounds__(kSplitThreads)
split_update_kernel(const StageBlock<R>* __restrict__ blocks, const SplitJob* __restrict__ jobs,
                    R* __restrict__ ws, StageInfo info, PhysParams phys) {
  using L = SplitLayout<MHD, DE>;
  __shared__ R s_dtdx[4];
  const SplitJob J = jobs[blockIdx.y];
  const StageBlock<R>& B = blocks[J.block];
  const SplitCtx<R> C = split_ctx(B, J, ws);
  const int S = info.S, m0 = C.m0, m1 = C.m1, m2 = C.m2;
  const int olo = info.final_stage ? S : S + 1;
  const int nx = m0 - 2 * olo, ny = m1 - 2 * olo;
  const int n = nx * ny * (C.zb - C.za);
  if (blockIdx.x * blockDim.x >= n) return;
  if (threadIdx.x < 4) {
    const double dt = *B.dt * info.dt_factor;
    s_dtdx[threadIdx.x] = threadIdx.x < 3 ? R(dt / B.cw[threadIdx.x]) : R(dt);
  }
  __syncthreads();
  const R dtdx[3] = {s_dtdx[0], s_dtdx[1], s_dtdx[2]};
  const R dfloor = R(phys.density_floor), pfloor = R(phys.pressure_floor);
  EnergyConsts<R> econ;
  econ.init(phys, DE);
  const size_t sy = C.sy, sz = C.sz, M = C.M;
  const R* xf = C.ws + (size_t)(L::F + 0 * L::NF) * M;
  const R* yf = C.ws + (size_t)(L::F + 1 * L::NF) * M;
  const R* zf = C.ws + (size_t)(L::F + 2 * L::NF) * M;
  const R* em = C.ws + (size_t)L::EMF * M;
  const FluxOut<R>* fo =
      info.final_stage && (info.fc != nullptr || info.block_fc)
          ? static_cast<const FluxOut<R>*>(B.fc != nullptr ? B.fc : info.fc)
          : nullptr;
  const int gg = info.fc_g;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int r = i / nx, x = olo + (i - r * nx);
    const int q = r / ny, y = olo + (r - q * ny), t = C.za + q;
    const size_t c = (size_t)t * sz + (size_t)y * sy + x, w = C.at(x, y, t);
    const bool in_x = inr(x, S + 1, m0 - S - 1), in_y = inr(y, S + 1, m1 - S - 1),
               in_t = inr(t, S + 1, m2 - S - 1);
    R bc[3] = {R(0), R(0), R(0)};
    if (MHD) {
      // face B on the low (k = 0) and high side along each axis; a face is
      // written by the cell above it, or by the last cell of the window
      // (EnzoBfieldMethodCT.cpp:617-728)
      const R *ex = em, *ey = em + M, *ez = em + 2 * M;
      R v[2];
#pragma unroll
      for (int k = 0; k < 2; k++) {
        const size_t fi = (size_t)t * ((size_t)m1 * (m0 + 1)) + (size_t)y * (m0 + 1) + (x + k);
        v[k] = B.base.f[0][fi];
        if (inr(x + k, S + 1, m0 - S) && in_y && in_t) {
          const size_t e = w + k - 1;
          const R Ek_term = dtdx[1] * (ez[e] - ez[e - sy]);
          const R Ej_term = dtdx[2] * (ey[e] - ey[e - sz]);
          v[k] = v[k] - Ek_term + Ej_term;
          if (k == 0 || x + 1 == m0 - olo) B.out.f[0][fi] = v[k];
        }
      }
      bc[0] = R(0.5) * (v[0] + v[1]);
#pragma unroll
      for (int k = 0; k < 2; k++) {
        const size_t fi = (size_t)t * ((size_t)(m1 + 1) * m0) + (size_t)(y + k) * m0 + x;
        v[k] = B.base.f[1][fi];
        if (inr(y + k, S + 1, m1 - S) && in_x && in_t) {
          const size_t e = w + k * sy - sy;
          const R Ek_term = dtdx[2] * (ex[e] - ex[e - sz]);
          const R Ej_term = dtdx[0] * (ez[e] - ez[e - 1]);
          v[k] = v[k] - Ek_term + Ej_term;
          if (k == 0 || y + 1 == m1 - olo) B.out.f[1][fi] = v[k];
        }
      }
      bc[1] = R(0.5) * (v[0] + v[1]);
#pragma unroll
      for (int k = 0; k < 2; k++) {
        const size_t fi = c + k * sz;
        v[k] = B.base.f[2][fi];
        if (inr(t + k, S + 1, m2 - S) && in_x && in_y) {
          const size_t e = w + k * sz - sz;
          const R Ek_term = dtdx[0] * (ey[e] - ey[e - 1]);
          const R Ej_term = dtdx[1] * (ex[e] - ex[e - sy]);
          v[k] = v[k] - Ek_term + Ej_term;
          if (k == 0 || t + 1 == m2 - olo) B.out.f[2][fi] = v[k];
        }
      }
      bc[2] = R(0.5) * (v[0] + v[1]);
      B.out.c[F_BX][c] = bc[0];
      B.out.c[F_BY][c] = bc[1];
      B.out.c[F_BZ][c] = bc[2];
    }
    if (!in_x || !in_y || !in_t) continue;
    // flux divergence, x then y then z
    // (EnzoIntegrationQuanUpdate.cpp:105-147, EnzoSourceInternalEnergy.cpp:16-92)
    R du[6];
#pragma unroll
    for (int k = 0; k < 5; k++) {
      R a = R(0.0);
      a -= dtdx[0] * (xf[k * M + w] - xf[k * M + w - 1]);
      a -= dtdx[1] * (yf[k * M + w] - yf[k * M + w - sy]);
      a -= dtdx[2] * (zf[k * M + w] - zf[k * M + w - sz]);
      du[k] = a;
    }
    if (DE) {
      const R p = smax(C.ws[L::P * M + w], pfloor);
      R a = R(0.0);
      a -= dtdx[0] * (xf[S_EINT * M + w] - xf[S_EINT * M + w - 1]);
      a -= dtdx[0] * p * (xf[S_VBAR * M + w] - xf[S_VBAR * M + w - 1]);
      a -= dtdx[1] * (yf[S_EINT * M + w] - yf[S_EINT * M + w - sy]);
      a -= dtdx[1] * p * (yf[S_VBAR * M + w] - yf[S_VBAR * M + w - sy]);
      a -= dtdx[2] * (zf[S_EINT * M + w] - zf[S_EINT * M + w - sz]);
      a -= dtdx[2] * p * (zf[S_VBAR * M + w] - zf[S_VBAR * M + w - sz]);
      du[5] = a;
    }
    const R old_rho = B.base.c[F_RHO][c];
    const R ovx = B.base.c[F_VX][c], ovy = B.base.c[F_VY][c], ovz = B.base.c[F_VZ][c];
    // gravity source on the full-dt stage (EnzoSourceGravity.cpp:17-69)
    if (info.gravity) {
      const R dt = s_dtdx[3];
      const R ax = B.accel[0][c], ay = B.accel[1][c], az = B.accel[2][c];
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
    R etot = (B.base.c[F_ETOT][c] * old_rho + du[4]) * inv_new_rho;
    R eint = R(0);
    if (DE) eint = (B.base.c[F_EINT][c] * old_rho + du[5]) * inv_new_rho;
    // apply_floor_to_energy_and_sync (EnzoPhysicsFluidProps.cpp:162-290)
    energy_floor_sync<MHD, DE>(econ, new_rho, vx, vy, vz, bc[0], bc[1], bc[2], etot, eint);
    B.out.c[F_RHO][c] = new_rho;
    B.out.c[F_VX][c] = vx;
    B.out.c[F_VY][c] = vy;
    B.out.c[F_VZ][c] = vz;
    B.out.c[F_ETOT][c] = etot;
    if (DE) B.out.c[F_EINT][c] = eint;
    // the density flux of both faces along each axis, for passive_kernel
    if (info.npass > 0) {
      R* const* D = B.dflux;
      D[0][c] = xf[w - 1];
      D[1][c] = yf[w - sy];
      D[2][c] = zf[w - sz];
      if (x + 1 == m0 - S - 1) D[0][c + 1] = xf[w];
      if (y + 1 == m1 - S - 1) D[1][c + sy] = yf[w];
      if (t + 1 == m2 - S - 1) D[2][c + sz] = zf[w];
    }
    // store_fluxes_for_corrections (EnzoMethodMHDVlct.cpp:250-330): dt/dx times
    // the fluxes through the block's active boundary faces, by the cell inside
    if (fo) {
      const int pos[3] = {x, y, t}, mm[3] = {m0, m1, m2};
      bool act = true;
#pragma unroll
      for (int a = 0; a < 3; a++) act = act && inr(pos[a], gg, mm[a] - gg);
      if (act) {
#pragma unroll
        for (int a = 0; a < 3; a++) {
          const R* f = a == 0 ? xf : (a == 1 ? yf : zf);
          const size_t st = a == 0 ? 1 : (a == 1 ? sy : sz);
          const int ai = a == 0 ? 1 : 0, ao = a == 2 ? 1 : 2;  // inner, outer axis
          const size_t at =
              (size_t)(pos[ao] - gg) * (mm[ai] - 2 * gg) + (size_t)(pos[ai] - gg);
#pragma unroll
          for (int side = 0; side < 2; side++) {
            if (pos[a] != (side == 0 ? gg : mm[a] - gg - 1)) continue;
            const size_t wf = side == 0 ? w - st : w;
#pragma unroll
            for (int k = 0; k < 6; k++) {
              R* p = fo->f[a][side][k];
              if (!p) continue;
              const R v = k == 0 ? f[S_RHO * M + wf]
                        : k <= 3 ? f[(S_MX + k - 1) * M + wf]
                        : k == 4 ? f[S_E * M + wf] : (DE ? f[S_EINT * M + wf] : R(0));
              p[at] = dtdx[a] * v;
            }
          }
        }
      }
    }
  }
}

}  // namespace vlct
