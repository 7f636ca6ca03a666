// vlct_physics.cuh -- device-side physics of the VL+CT step: ideal-gas EOS,
// PLM slope limiters and the HLLE / HLLC / HLLD Riemann solvers.
//
// Every formula keeps the reference's floating-point operation order so that
// the FP64 instantiation (compiled with --fmad=false) reproduces Enzo-E's CPU
// results bit for bit.  The FP32 instantiation uses the same code in float.
// Reference: src/Enzo/fluid-props/EnzoEOSIdeal.hpp,
// src/Enzo/hydro-mhd/toolkit/EnzoReconstructorPLM.hpp,
// src/Enzo/hydro-mhd/riemann/EnzoRiemann{HLL,HLLC,HLLD,Utils}.hpp.
#pragma once
#include <cuda_runtime.h>

namespace vlct {

enum Solver { SOLVER_HLLE = 0, SOLVER_HLLC = 1, SOLVER_HLLD = 2 };
enum Recon { RECON_NN = 0, RECON_PLM = 1, RECON_PLM_ATHENA = 2 };

// Face-frame ordering of the 8 primitives / fluxes (riemann/EnzoRiemannImpl.hpp:
// 40-56, MHDLUT): rho, B_i, B_j, B_k, v_i, v_j, v_k, p (or etot for fluxes).
enum { L_RHO = 0, L_BI = 1, L_BJ = 2, L_BK = 3, L_VI = 4, L_VJ = 5, L_VK = 6,
       L_E = 7 };

// std::min / std::max semantics of the reference (first argument on ties).
template <class R> __device__ __forceinline__ R smin(R a, R b) {
  return (b < a) ? b : a;
}
template <class R> __device__ __forceinline__ R smax(R a, R b) {
  return (a < b) ? b : a;
}
// Sign tests.  For double they read the bit pattern on the integer pipe, as a
// comparison would occupy the narrow FP64 pipe (false for NaN, zeros of either
// sign alike, as the comparisons).
template <class R> __device__ __forceinline__ bool gt0(R x) { return x > R(0); }
template <class R> __device__ __forceinline__ bool lt0(R x) { return x < R(0); }
template <class R> __device__ __forceinline__ bool ge0(R x) { return x >= R(0); }
template <class R> __device__ __forceinline__ bool le0(R x) { return x <= R(0); }
constexpr long long kInfBits = 0x7ff0000000000000LL;
constexpr long long kAbsBits = 0x7fffffffffffffffLL;
// (through a move that the compiler cannot see through: it would turn the
// patterns below back into floating-point comparisons)
__device__ __forceinline__ long long bits_of(double x) {
  long long i;
  asm("mov.b64 %0, %1;" : "=l"(i) : "d"(x));
  return i;
}
__device__ __forceinline__ double abs_i(double x) {
  return __longlong_as_double(bits_of(x) & kAbsBits);
}
template <> __device__ __forceinline__ bool gt0<double>(double x) {
  const long long i = bits_of(x);
  return i > 0 && i <= kInfBits;
}
template <> __device__ __forceinline__ bool lt0<double>(double x) {
  const long long i = bits_of(x), a = i & kAbsBits;
  return i < 0 && a != 0 && a <= kInfBits;
}
template <> __device__ __forceinline__ bool ge0<double>(double x) {
  const long long i = bits_of(x), a = i & kAbsBits;
  return (i >= 0 || a == 0) && a <= kInfBits;
}
template <> __device__ __forceinline__ bool le0<double>(double x) {
  const long long i = bits_of(x), a = i & kAbsBits;
  return (i < 0 || a == 0) && a <= kInfBits;
}
// a < b, the larger and smaller of two with std::max / std::min's choice on
// ties and NaN (below), fmax / fmin's, and products by powers of two and by
// signs, all likewise off the FP64 pipe.
__device__ __forceinline__ bool is_nan(double x) {
  return (bits_of(x) & kAbsBits) > kInfBits;
}
__device__ __forceinline__ bool is_finite(double x) {
  return (bits_of(x) & kAbsBits) < kInfBits;
}
__device__ __forceinline__ bool lt(double a, double b) {
  const long long ia = bits_of(a), ib = bits_of(b);
  // two's-complement order of the sign-magnitude patterns; zeros are equal
  const long long ka = ia ^ ((ia >> 63) & kAbsBits), kb = ib ^ ((ib >> 63) & kAbsBits);
  return ka < kb && ((ia | ib) & kAbsBits) != 0 && !is_nan(a) && !is_nan(b);
}
template <>
__device__ __forceinline__ double smin<double>(double a, double b) {
  return lt(b, a) ? b : a;
}
template <>
__device__ __forceinline__ double smax<double>(double a, double b) {
  return lt(a, b) ? b : a;
}
__device__ __forceinline__ double fmax_i(double a, double b) {
  return is_nan(a) ? b : (lt(a, b) ? b : a);
}
__device__ __forceinline__ double fmin_i(double a, double b) {
  return is_nan(a) ? b : (lt(b, a) ? b : a);
}
// Kept in a branch: without it the compiler would compute the rare case always
// and select.
__device__ __forceinline__ void rare_path() { asm volatile(""); }
// x 2^K: a step of the exponent where x and the product are normal
template <int K> __device__ __forceinline__ double scale2(double x) {
  const int hi = __double2hiint(x), e = (hi >> 20) & 0x7ff;
  if (e >= (K < 0 ? 1 - K : 1) && e <= (K > 0 ? 2046 - K : 2046))
    return __hiloint2double(hi + K * (1 << 20), __double2loint(x));
  if ((bits_of(x) & kAbsBits) == 0) return x;
  rare_path();
  return x * (K < 0 ? 1.0 / (1 << -K) : (double)(1 << K));
}
__device__ __forceinline__ double neg_if(double x, bool n) {
  return n ? __longlong_as_double(bits_of(x) ^ ~kAbsBits) : x;
}
// enzo_utils::min of three values (utils.hpp:82-89)
template <class R> __device__ __forceinline__ R min3(R a, R b, R c) {
  if (a < b) return (c < a) ? c : a;
  return (c < b) ? c : b;
}
template <class R> __device__ __forceinline__ R sqmag(R i, R j, R k) {
  return ((i * i) + ((j * j) + (k * k)));
}

// ---------------------------------------------------------------- EOS ----
template <class R> __device__ __forceinline__ R cs2(R g, R d, R p) {
  return g * p / d;
}
// specific internal energy p / ((gamma-1) rho) (EnzoEOSIdeal.hpp:79-82)
template <class R> __device__ __forceinline__ R specific_eint(R gm1, R d, R p) {
  return p / (gm1 * d);
}
// passive upwinding of the internal energy (EnzoRiemannUtils.hpp:224-249)
template <class R>
__device__ __forceinline__ R eint_flux(R gm1, R dl, R pl, R dr, R pr, R fd) {
  const R el = specific_eint(gm1, dl, pl);
  const R er = specific_eint(gm1, dr, pr);
  const R up = (gt0(fd) ? R(1) : R(0)) * el + (le0(fd) ? R(1) : R(0)) * er;
  return up * fd;
}

// What the FP64 solvers take from a cell's density and pressure alone, divisions
// and square roots: sound speed squared gamma p / rho (HLLC: the sound speed)
// and 1 / rho for the fast speed, sqrt(rho) and p / (gamma - 1) for the Einfeldt
// speeds.  With nearest-neighbour reconstruction a face's states are the cells'
// own, and the six faces of a cell share them.
struct Gas {
  double g, gm1, igm1;  // gamma, gamma - 1, 1 / (gamma - 1)
};
template <int SOLVER> struct CellGas {
  // values kept per cell
  static constexpr int N = SOLVER == SOLVER_HLLD ? 2 : (SOLVER == SOLVER_HLLC ? 3 : 4);
  double v[N];
  __device__ __forceinline__ void init(const Gas& gas, double d, double p) {
    const double c2 = cs2(gas.g, d, p);
    v[0] = SOLVER == SOLVER_HLLC ? sqrt(c2) : c2;
    if (SOLVER == SOLVER_HLLC) {
      v[1] = sqrt(d);
      v[2] = p / gas.gm1;
    } else {
      v[1] = 1.0 / d;
      if (SOLVER == SOLVER_HLLE) {
        v[2 % N] = sqrt(d);
        v[3 % N] = p / gas.gm1;
      }
    }
  }
};
// fast_magnetosonic_speed, generic cos^2 branch (EnzoEOSIdeal.hpp:133-139), from
// gamma p / rho, 1 / rho, B^2 and B_i^2
__device__ __forceinline__ double cfast_of(double c2, double inv_density, double B2, double bi2) {
  const double va2 = B2 * inv_density;
  const double va2_cos2 = bi2 * inv_density;
  const double s = c2 + va2;
  return sqrt(scale2<-1>(va2 + c2 + sqrt(s * s - scale2<2>(c2) * va2_cos2)));
}

// ------------------------------------------------------------ limiters ----
// PLM_EnzoRKLimiter (EnzoReconstructorPLM.hpp:287-302)
template <class R>
__device__ __forceinline__ R limiter_enzo_rk(R vm1, R v, R vp1, R theta) {
  R dv_c = R(0.5) * (vp1 - vm1);
  R dv_l = (v - vm1) * theta;
  R dv_r = (vp1 - v) * theta;
  // sign(dv) in {-1, 0, 1} (the reference's (0 < x) - (x < 0)) as selects,
  // with no integer-to-float conversion
  R sl = (R(0.0) < dv_l) ? R(1.0) : ((dv_l < R(0.0)) ? R(-1.0) : R(0.0));
  R sr = (R(0.0) < dv_r) ? R(1.0) : ((dv_r < R(0.0)) ? R(-1.0) : R(0.0));
  return (R(0.5) * (sl + sr)) * min3(fabs(dv_l), fabs(dv_r), fabs(dv_c));
}
// The same limiter in FP32 with fewer instructions: 0.5 (sgn dl + sgn dr) is
// +-1 when the two one-sided differences share a sign and 0 otherwise (a zero
// difference makes the minimum zero), so the slope is the minimum magnitude
// carrying dl's sign when dl dr > 0, else 0 -- the same value, as sign times
// minimum is exact either way (a product dl dr below the FP32 range flushes
// to 0 under -ftz, as do such differences themselves).
template <>
__device__ __forceinline__ float limiter_enzo_rk<float>(float vm1, float v, float vp1,
                                                        float theta) {
  const float dv_c = 0.5f * (vp1 - vm1);
  const float dv_l = (v - vm1) * theta;
  const float dv_r = (vp1 - v) * theta;
  const float m = fminf(fminf(fabsf(dv_l), fabsf(dv_r)), fabsf(dv_c));
  return (dv_l * dv_r > 0.f) ? copysignf(m, dv_l) : 0.f;
}
// PLM_AthenaLimiter (EnzoReconstructorPLM.hpp:337-345)
template <class R>
__device__ __forceinline__ R limiter_athena(R vm1, R v, R vp1) {
  R dv_l = (v - vm1);
  R dv_r = (vp1 - v);
  R temp = dv_l * dv_r;
  if (temp <= R(0.)) return R(0.);
  return R(2.) * temp / (dv_l + dv_r);
}

// Half the limited slope of a cell: what PLM adds to and takes from the cell's
// value at its two faces.
template <class R, int RECON>
__device__ __forceinline__ R half_slope(R vm1, R v, R vp1, R theta) {
  return (RECON == RECON_PLM ? limiter_enzo_rk(vm1, v, vp1, theta)
                             : limiter_athena(vm1, v, vp1)) * R(0.5);
}
// The theta limiter in FP64, with its sign tests, minimum and halving on the
// integer pipe (the FP64 pipe, which bounds the FP64 stages, keeps five
// operations of about twenty).  Magnitudes of finite doubles order like their
// bit patterns, and halving one that stays normal is a step of its exponent;
// anything else takes limiter_enzo_rk itself.  0.5 (sgn dl + sgn dr) times the
// minimum is the minimum with the common sign, a zero of the sign of the one
// that is not zero, or +0.
template <>
__device__ __forceinline__ double half_slope<double, RECON_PLM>(double vm1, double v,
                                                                double vp1, double theta) {
  const double dv_c = scale2<-1>(vp1 - vm1);
  const double dv_l = (v - vm1) * theta;
  const double dv_r = (vp1 - v) * theta;
  const long long il = bits_of(dv_l), ir = bits_of(dv_r);
  const long long al = il & kAbsBits, ar = ir & kAbsBits,
                  ac = bits_of(dv_c) & kAbsBits;
  long long m = al < ar ? al : ar;
  const long long most = al < ar ? ar : al;
  m = ac < m ? ac : m;
  if ((most < ac ? ac : most) >= kInfBits || (m != 0 && m < 0x0020000000000000LL)) {
    rare_path();
    return limiter_enzo_rk(vm1, v, vp1, theta) * 0.5;
  }
  const bool opposite = al != 0 && ar != 0 && (il ^ ir) < 0;
  const long long sign = (al != 0 ? il : (ar != 0 ? ir : 0)) & ~kAbsBits;
  if (m != 0) m -= 0x0010000000000000LL;
  return opposite ? 0.0 : __longlong_as_double(m | sign);
}

// ------------------------------------------------------ Riemann solvers ----
// Output of one face solve, in the face frame: 8 fluxes (flux[L_BI] == 0),
// the passive internal-energy flux and the interface velocity v_i-bar.
template <class R> struct FaceFlux {
  R f[8];
  R eflux;
  R vbar;
};

// HLLD (riemann/EnzoRiemannHLLD.hpp:40-448).  The flux is that of one side:
// F_L or F_R, plus the jump terms of that side's star states, by the signs of
// the five wave speeds.  So the speeds come first, and only the states that
// the flux of this face is made of are formed: the side's own star state, and
// the other side's only where the double-star state is needed.  Every value
// that is formed is the reference's expression on the same operands, so the
// result is the same bit for bit; on GB300, whose FP64 pipe bounds the FP64
// stages, the operands' selection by integer moves is free.
struct HlldSide {
  double d, u, vj, vk, by, bz, pt, e, sd, sdd, sdm_inv, sdm;  // left or right state
  double st_d, st_inv;                                        // star density and 1 / it
};
struct HlldStar {
  double mx, my, mz, e, by, bz, vb;
};
__device__ __forceinline__ HlldStar hlld_star(const HlldSide& W, double bxi, double bxsq,
                                              double spd2, double ptst, double thr) {
  HlldStar s;
  s.mx = W.st_d * spd2;
  const double den = W.sdd * W.sdm - bxsq;
  if (lt(abs_i(den), thr)) {
    s.my = W.st_d * W.vj;
    s.mz = W.st_d * W.vk;
    s.by = W.by;
    s.bz = W.bz;
  } else {
    double tmp = bxi * (W.sd - W.sdm) / den;
    s.my = W.st_d * (W.vj - W.by * tmp);
    s.mz = W.st_d * (W.vk - W.bz * tmp);
    tmp = (W.d * (W.sd * W.sd) - bxsq) / den;
    s.by = W.by * tmp;
    s.bz = W.bz * tmp;
  }
  s.vb = (s.mx * bxi + (s.my * s.by + s.mz * s.bz)) * W.st_inv;
  s.e = (W.sd * W.e - W.pt * W.u + ptst * spd2 +
         bxi * (W.u * bxi + (W.vj * W.by + W.vk * W.bz) - s.vb)) *
        W.sdm_inv;
  return s;
}

__device__ __forceinline__ void hlld(const Gas& gas, const double* wli, const double* wri,
                                     const CellGas<SOLVER_HLLD>& cl,
                                     const CellGas<SOLVER_HLLD>& cr, FaceFlux<double>& out) {
  const double SMALL = 1.0e-8;
  const double pressure_l = wli[L_E], pressure_r = wri[L_E];
  const double bxi = wli[L_BI];
  const double bxsq = bxi * bxi;
  const double b2l = bxsq + (wli[L_BJ] * wli[L_BJ] + wli[L_BK] * wli[L_BK]);
  const double b2r = bxsq + (wri[L_BJ] * wri[L_BJ] + wri[L_BK] * wri[L_BK]);
  const double pbl = scale2<-1>(b2l), pbr = scale2<-1>(b2r);

  const double cfl = cfast_of(cl.v[0], cl.v[1], b2l, bxsq);
  const double cfr = cfast_of(cr.v[0], cr.v[1], b2r, bxsq);
  const double spd0 = smin(wli[L_VI] - cfl, wri[L_VI] - cfr);
  const double spd4 = smax(wli[L_VI] + cfl, wri[L_VI] + cfr);
  const double uld = wli[L_RHO], urd = wri[L_RHO];
  const double ptl = pressure_l + pbl;
  const double ptr = pressure_r + pbr;
  const double sdl = spd0 - wli[L_VI];
  const double sdr = spd4 - wri[L_VI];
  const double sddl = uld * sdl, sddr = urd * sdr;
  const double spd2 = (sdr * (wri[L_VI] * urd) - sdl * (wli[L_VI] * uld) + (ptl - ptr)) /
                      (sddr - sddl);
  // the reference's order of the cases: F_L (spd0 >= 0), F_R (spd4 <= 0), then
  // left star states for spd2 >= 0 and right ones otherwise
  const bool sup_l = ge0(spd0), outer = sup_l || le0(spd4);
  const bool left = sup_l || (!outer && ge0(spd2));

  HlldSide W;  // the side whose flux this is
  W.d = left ? uld : urd;
  W.u = left ? wli[L_VI] : wri[L_VI];
  W.vj = left ? wli[L_VJ] : wri[L_VJ];
  W.vk = left ? wli[L_VK] : wri[L_VK];
  W.by = left ? wli[L_BJ] : wri[L_BJ];
  W.bz = left ? wli[L_BK] : wri[L_BK];
  W.pt = left ? ptl : ptr;
  W.sd = left ? sdl : sdr;
  W.sdd = left ? sddl : sddr;
  const double mx = W.u * W.d, my = W.vj * W.d, mz = W.vk * W.d;
  {
    const double ke = scale2<-1>(W.d) * (W.u * W.u + (W.vj * W.vj + W.vk * W.vk));
    W.e = (left ? pressure_l : pressure_r) * gas.igm1 + ke + (left ? pbl : pbr);
  }
  double f[7];
  f[0] = mx;
  f[1] = mx * W.u + W.pt - bxsq;
  f[2] = my * W.u - bxi * W.by;
  f[3] = mz * W.u - bxi * W.bz;
  f[4] = W.u * (W.e + W.pt - bxsq) - bxi * (W.vj * W.by + W.vk * W.bz);
  f[5] = W.by * W.u - bxi * W.vj;
  f[6] = W.bz * W.u - bxi * W.vk;

  if (!outer) {
    const double ptstl = ptl + sddl * (spd2 - wli[L_VI]);
    const double ptstr = ptr + sddr * (spd2 - wri[L_VI]);
    const double ptst = scale2<-1>(ptstr + ptstl);
    const double thr = SMALL * ptst;
    const double spdo = left ? spd0 : spd4;  // the side's outermost speed
    W.sdm = spdo - spd2;
    W.sdm_inv = 1.0 / W.sdm;
    W.st_d = W.sdd * W.sdm_inv;
    W.st_inv = 1.0 / W.st_d;
    const double sq = sqrt(W.st_d);
    const double va = abs_i(bxi) / sq;
    const double spdi = spd2 + neg_if(va, left);  // its Alfven speed (spd1 / spd3)
    const bool two = left ? !ge0(spdi) : gt0(spdi);
    const HlldStar st = hlld_star(W, bxi, bxsq, spd2, ptst, thr);
    f[0] = f[0] + spdo * (W.st_d - W.d);
    f[1] = f[1] + spdo * (st.mx - mx);
    f[2] = f[2] + spdo * (st.my - my);
    f[3] = f[3] + spdo * (st.mz - mz);
    f[4] = f[4] + spdo * (st.e - W.e);
    f[5] = f[5] + spdo * (st.by - W.by);
    f[6] = f[6] + spdo * (st.bz - W.bz);
    if (two) {
      double dy = st.my, dz = st.mz, de = st.e, dby = st.by, dbz = st.bz;
      if (!lt(scale2<-1>(bxsq), thr)) {
        HlldSide V;  // the other side
        V.d = left ? urd : uld;
        V.u = left ? wri[L_VI] : wli[L_VI];
        V.vj = left ? wri[L_VJ] : wli[L_VJ];
        V.vk = left ? wri[L_VK] : wli[L_VK];
        V.by = left ? wri[L_BJ] : wli[L_BJ];
        V.bz = left ? wri[L_BK] : wli[L_BK];
        V.sd = left ? sdr : sdl;
        V.sdd = left ? sddr : sddl;
        V.sdm = (left ? spd4 : spd0) - spd2;
        V.sdm_inv = 1.0 / V.sdm;
        V.st_d = V.sdd * V.sdm_inv;
        V.st_inv = 1.0 / V.st_d;
        V.pt = V.e = 0.0;  // its energy is not needed
        const double sqv = sqrt(V.st_d);
        const HlldStar sv = hlld_star(V, bxi, bxsq, spd2, ptst, thr);
        // left and right values, in the reference's expressions; the sign of
        // B_x multiplies by flipping signs
        const double sqrtdl = left ? sq : sqv, sqrtdr = left ? sqv : sq;
        const double invsumd = 1.0 / (sqrtdl + sqrtdr);
        const bool bneg = !gt0(bxi);
        const double vy = st.my * W.st_inv, vz = st.mz * W.st_inv;
        const double oy = sv.my * V.st_inv, oz = sv.mz * V.st_inv;
        const double lvy = left ? vy : oy, rvy = left ? oy : vy;
        const double lvz = left ? vz : oz, rvz = left ? oz : vz;
        const double lby = left ? st.by : sv.by, rby = left ? sv.by : st.by;
        const double lbz = left ? st.bz : sv.bz, rbz = left ? sv.bz : st.bz;
        const double lst_d = left ? W.st_d : V.st_d;
        const double ty =
            invsumd * (sqrtdl * lvy + sqrtdr * rvy + neg_if(rby - lby, bneg));
        const double tz =
            invsumd * (sqrtdl * lvz + sqrtdr * rvz + neg_if(rbz - lbz, bneg));
        const double sqlr = neg_if(sqrtdl * sqrtdr, bneg);
        dby = invsumd * (sqrtdl * rby + sqrtdr * lby + sqlr * (rvy - lvy));
        dbz = invsumd * (sqrtdl * rbz + sqrtdr * lbz + sqlr * (rvz - lvz));
        dy = W.st_d * ty;
        dz = W.st_d * tz;
        // v** . B**, from the left side's values for both sides
        const double vb = spd2 * bxi + ((lst_d * ty) * dby + (lst_d * tz) * dbz) / lst_d;
        const double t = neg_if(sq, bneg) * (st.vb - vb);
        de = st.e + neg_if(t, left);
      }
      // (the density and the normal momentum do not jump there: a zero, but
      // where a value is not finite)
      if (!is_finite(W.st_d) || !is_finite(st.mx) || !is_finite(spdi)) {
        rare_path();
        f[0] = f[0] + spdi * (W.st_d - W.st_d);
        f[1] = f[1] + spdi * (st.mx - st.mx);
      }
      f[2] = f[2] + spdi * (dy - st.my);
      f[3] = f[3] + spdi * (dz - st.mz);
      f[4] = f[4] + spdi * (de - st.e);
      f[5] = f[5] + spdi * (dby - st.by);
      f[6] = f[6] + spdi * (dbz - st.bz);
    }
  }
  out.f[L_RHO] = f[0];
  out.f[L_BI] = 0.0;
  out.f[L_BJ] = f[5];
  out.f[L_BK] = f[6];
  out.f[L_VI] = f[1];
  out.f[L_VJ] = f[2];
  out.f[L_VK] = f[3];
  out.f[L_E] = f[4];
  out.eflux = eint_flux(gas.gm1, wli[L_RHO], pressure_l, wri[L_RHO], pressure_r, f[0]);
  if (gt0(spd0)) {
    out.vbar = wli[L_VI];
  } else if (lt0(spd4)) {
    out.vbar = wri[L_VI];
  } else {
    const bool l = ge0(spd2);
    out.vbar = spd2 * ((l ? sdl : sdr) / ((l ? spd0 : spd4) - spd2));
  }
}

// HLLD in FP32 (EnzoRiemannHLLD.hpp:40-448): the same states, wave speeds
// and flux as the FP64 form, with fewer instructions.  The left and right
// states ride in the two lanes of packed FP32 arithmetic (float2: fadd2 /
// fmul2 / ffma2 on sm_100+), so every side-wise operation is one
// instruction for both sides, down to the flux of each side,
//   F + c1 (U* - U) + c2 (U** - U*),
// with the coefficients chosen in the reference's case order and the same for
// both lanes: one select per component picks the side at the end.  Each shared
// denominator is inverted once (rsqrt for 1/sqrt(rho*)) and multiplied by; a
// division of its own would be eight instructions.  Differences from the FP64
// form lie only in rounding.
namespace packed {
__device__ __forceinline__ float2 f2(float a, float b) { return make_float2(a, b); }
__device__ __forceinline__ float2 s2(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 add(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 mul(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
// a - b as one fused operation: b * -1 + a is exact before its one rounding
__device__ __forceinline__ float2 sub(float2 a, float2 b) {
  return __ffma2_rn(b, make_float2(-1.0f, -1.0f), a);
}
}  // namespace packed

__device__ __forceinline__ void hlld(float g, const float* wli, const float* wri,
                                     FaceFlux<float>& out) {
  using namespace packed;
  const float SMALL = 1.0e-8f;
  const float igm1 = 1.0f / (g - 1.0f);
  const float bxi = wli[L_BI], bxsq = bxi * bxi;
  const float2 BXSQ = s2(bxsq), BXI = s2(bxi), HALF = s2(0.5f);
  const float2 p = f2(wli[L_E], wri[L_E]);
  const float2 d = f2(wli[L_RHO], wri[L_RHO]);
  const float2 u = f2(wli[L_VI], wri[L_VI]);
  const float2 vj = f2(wli[L_VJ], wri[L_VJ]), vk = f2(wli[L_VK], wri[L_VK]);
  const float2 by = f2(wli[L_BJ], wri[L_BJ]), bz = f2(wli[L_BK], wri[L_BK]);
  const float2 inv_d = f2(1.0f / d.x, 1.0f / d.y);
  const float2 bt = fma(by, by, mul(bz, bz));
  const float2 b2 = add(BXSQ, bt);
  const float2 pb = mul(HALF, b2);
  const float2 ke = mul(mul(HALF, d), fma(u, u, fma(vj, vj, mul(vk, vk))));
  const float2 ue = add(fma(p, s2(igm1), ke), pb);
  // fast speeds (EnzoEOSIdeal.hpp:133-139)
  const float2 c2 = mul(mul(s2(g), p), inv_d);
  const float2 va2 = mul(b2, inv_d);
  const float2 vac2 = mul(BXSQ, inv_d);
  const float2 q = add(c2, va2);
  const float2 disc = fma(q, q, mul(mul(s2(-4.0f), c2), vac2));
  const float2 inner = add(q, f2(sqrtf(disc.x), sqrtf(disc.y)));
  const float2 cfh = mul(HALF, inner);
  const float2 cf = f2(sqrtf(cfh.x), sqrtf(cfh.y));
  const float2 um = sub(u, cf), up = add(u, cf);
  const float spd0 = fminf(um.x, um.y);
  const float spd4 = fmaxf(up.x, up.y);
  const float2 pt = add(p, pb);
  // side fluxes: d, mx, my, mz, e, by, bz
  const float2 du = mul(d, u);
  const float2 vbt = fma(vj, by, mul(vk, bz));
  const float2 ptb = sub(pt, BXSQ);
  const float2 F[7] = {du, fma(du, u, ptb), sub(mul(du, vj), mul(BXI, by)),
                       sub(mul(du, vk), mul(BXI, bz)), sub(mul(u, add(ue, ptb)), mul(BXI, vbt)),
                       sub(mul(by, u), mul(BXI, vj)), sub(mul(bz, u), mul(BXI, vk))};
  const float2 S04 = f2(spd0, spd4);
  const float2 sd = sub(S04, u);
  const float2 sdd = mul(sd, d);
  const float2 sddu = mul(sdd, u);
  const float spd2 = (sddu.y - sddu.x + (pt.x - pt.y)) * (1.0f / (sdd.y - sdd.x));
  const float2 SPD2 = s2(spd2);
  const float2 sdm = sub(S04, SPD2);
  const float2 sdm_inv = f2(1.0f / sdm.x, 1.0f / sdm.y);
  const float2 st_d = mul(sdd, sdm_inv);
  const float2 isq = f2(rsqrtf(st_d.x), rsqrtf(st_d.y));
  const float2 sqrtd = mul(st_d, isq);
  const float2 st_d_inv = mul(isq, isq);
  // (the Alfven speeds' roundings are spelled out: near B_x^2 = rho s (s - s_M)
  // one ulp of anything above moves a flux by 1e-4, so results that are to stay
  // the same need every bit the same)
  const float spd1 = __fsub_rn(spd2, __fmul_rn(fabsf(bxi), isq.x));
  const float spd3 = __fmaf_rn(fabsf(bxi), isq.y, spd2);
  const float2 ptw = fma(sdd, sub(SPD2, u), pt);
  const float ptst = 0.5f * (ptw.y + ptw.x);
  // single-star states, both sides at once: d, mx, my, mz, e, by, bz; a
  // side whose |d s (s - s_M) - B_x^2| is below SMALL p* keeps its
  // transverse B and velocity (t1 = 0, t2 = 1)
  const float2 den = sub(mul(sdd, sdm), BXSQ);
  const float thr = SMALL * ptst;
  const bool degl = fabsf(den.x) < thr, degr = fabsf(den.y) < thr;
  const float2 iden = f2(1.0f / den.x, 1.0f / den.y);
  float2 t1 = mul(mul(BXI, sub(sd, sdm)), iden);
  float2 t2 = mul(sub(mul(sdd, sd), BXSQ), iden);
  t1 = f2(degl ? 0.0f : t1.x, degr ? 0.0f : t1.y);
  t2 = f2(degl ? 1.0f : t2.x, degr ? 1.0f : t2.y);
  float2 Us[7];
  Us[0] = st_d;
  Us[1] = mul(st_d, SPD2);
  Us[2] = mul(st_d, sub(vj, mul(by, t1)));
  Us[3] = mul(st_d, sub(vk, mul(bz, t1)));
  Us[5] = mul(by, t2);
  Us[6] = mul(bz, t2);
  const float2 vbst = mul(fma(Us[1], BXI, fma(Us[2], Us[5], mul(Us[3], Us[6]))), st_d_inv);
  const float2 e_num =
      add(fma(SPD2, s2(ptst), sub(mul(sd, ue), mul(pt, u))), mul(BXI, sub(fma(u, BXI, vbt), vbst)));
  Us[4] = mul(e_num, sdm_inv);
  // F = F_side + c1 (U* - U) + c2 (U** - U*), the cases in the reference's
  // order: F_L (spd0 >= 0), F_R (spd4 <= 0), then by the signs of spd1..spd3;
  // both sides at once, so that one select per component picks the side
  const bool outer = spd0 >= 0.0f || spd4 <= 0.0f;
  const bool left = spd0 >= 0.0f || (!(spd4 <= 0.0f) && spd2 >= 0.0f);
  const float c1 = outer ? 0.0f : (left ? spd0 : spd4);
  const float c2v = (outer || 0.5f * bxsq < thr)
                        ? 0.0f
                        : (left ? (spd1 >= 0.0f ? 0.0f : spd1) : (spd3 > 0.0f ? spd3 : 0.0f));
  const float2 C1 = s2(c1);
  const float2 r0 = fma(C1, sub(Us[0], d), F[0]);
  const float2 r1 = fma(C1, sub(Us[1], du), F[1]);
  float2 r2 = fma(C1, sub(Us[2], mul(d, vj)), F[2]);
  float2 r3 = fma(C1, sub(Us[3], mul(d, vk)), F[3]);
  float2 r4 = fma(C1, sub(Us[4], ue), F[4]);
  float2 r5 = fma(C1, sub(Us[5], by), F[5]);
  float2 r6 = fma(C1, sub(Us[6], bz), F[6]);
  if (c2v != 0.0f) {  // the double-star states (U** = U* where B_x^2 / 2 < SMALL p*)
    const float2 C2 = s2(c2v);
    const float invsumd = 1.0f / (sqrtd.x + sqrtd.y);
    const float bxsig = bxi > 0.0f ? 1.0f : -1.0f;
    const float2 vy = mul(Us[2], st_d_inv), vz = mul(Us[3], st_d_inv);
    const float2 wvy = mul(sqrtd, vy), wvz = mul(sqrtd, vz);
    const float ty = invsumd * (wvy.x + wvy.y + bxsig * (Us[5].y - Us[5].x));
    const float tz = invsumd * (wvz.x + wvz.y + bxsig * (Us[6].y - Us[6].x));
    const float2 dmy = mul(Us[0], s2(ty)), dmz = mul(Us[0], s2(tz));
    const float sq = bxsig * sqrtd.x * sqrtd.y;
    const float byd = invsumd * (sqrtd.x * Us[5].y + sqrtd.y * Us[5].x + sq * (vy.y - vy.x));
    const float bzd = invsumd * (sqrtd.x * Us[6].y + sqrtd.y * Us[6].x + sq * (vz.y - vz.x));
    // v** . B** from the left side's values for both (as the scalar form)
    const float tl = spd2 * bxi + (dmy.x * byd + dmz.x * bzd) * st_d_inv.x;
    const float2 sg = mul(sqrtd, f2(-bxsig, bxsig));
    const float2 de = fma(sg, sub(vbst, s2(tl)), Us[4]);
    r2 = fma(C2, sub(dmy, Us[2]), r2);
    r3 = fma(C2, sub(dmz, Us[3]), r3);
    r4 = fma(C2, sub(de, Us[4]), r4);
    r5 = fma(C2, sub(s2(byd), Us[5]), r5);
    r6 = fma(C2, sub(s2(bzd), Us[6]), r6);
  }
  out.f[L_RHO] = left ? r0.x : r0.y;
  out.f[L_VI] = left ? r1.x : r1.y;
  out.f[L_VJ] = left ? r2.x : r2.y;
  out.f[L_VK] = left ? r3.x : r3.y;
  out.f[L_E] = left ? r4.x : r4.y;
  out.f[L_BJ] = left ? r5.x : r5.y;
  out.f[L_BK] = left ? r6.x : r6.y;
  out.f[L_BI] = 0.0f;
  out.eflux = eint_flux(g - 1.0f, d.x, p.x, d.y, p.y, out.f[L_RHO]);
  if (spd0 > 0.0f) out.vbar = u.x;
  else if (spd4 < 0.0f) out.vbar = u.y;
  else out.vbar = spd2 * (spd2 >= 0.0f ? sd.x * sdm_inv.x : sd.y * sdm_inv.y);
}

// Conserved total energy (EnzoRiemannUtils.hpp:48-82); pg: p / (gamma - 1).
// Hydro adds a magnetic energy of zero, which changes no value.
template <bool MHD>
__device__ __forceinline__ double energy_of(const double* w, double pg, double b2) {
  const double ke = scale2<-1>(w[L_RHO]) * sqmag(w[L_VI], w[L_VJ], w[L_VK]);
  return MHD ? pg + ke + scale2<-1>(b2) : pg + ke;
}

// Einfeldt wave speeds with Roe averages (EnzoRiemannHLL.hpp:44-172).  c: sound
// (hydro) or fast (MHD) speeds, sq: sqrt(rho), U: total energies, b2: B^2.
template <bool MHD>
__device__ __forceinline__ void einfeldt(const Gas& gas, const double* wl, const double* wr,
                                         double c_l, double c_r, double sqrtrho_l,
                                         double sqrtrho_r, double El, double Er, double b2l,
                                         double b2r, double* bp, double* bm) {
  const double left_speed = (wl[L_VI] - c_l);
  const double right_speed = (wr[L_VI] + c_r);
  const double inv_tot = 1.0 / (sqrtrho_l + sqrtrho_r);
  const double vi_roe = (sqrtrho_l * wl[L_VI] + sqrtrho_r * wr[L_VI]) * inv_tot;
  const double vj_roe = (sqrtrho_l * wl[L_VJ] + sqrtrho_r * wr[L_VJ]) * inv_tot;
  const double vk_roe = (sqrtrho_l * wl[L_VK] + sqrtrho_r * wr[L_VK]) * inv_tot;
  const double v_roe2 = vi_roe * vi_roe + vj_roe * vj_roe + vk_roe * vk_roe;
  double ptot_l = wl[L_E], ptot_r = wr[L_E];
  if (MHD) {
    ptot_l += scale2<-1>(b2l);
    ptot_r += scale2<-1>(b2r);
  }
  const double h_l = (El + ptot_l) / wl[L_RHO];
  const double h_r = (Er + ptot_r) / wr[L_RHO];
  const double h_roe = (sqrtrho_l * h_l + sqrtrho_r * h_r) * inv_tot;
  double c_roe;
  if (MHD) {  // roe_cfast_ (:134-172)
    const double rho_roe = sqrtrho_l * sqrtrho_r;
    const double bi_roe = wl[L_BI];
    const double bj_roe = (sqrtrho_l * wr[L_BJ] + sqrtrho_r * wl[L_BJ]) * inv_tot;
    const double bk_roe = (sqrtrho_l * wr[L_BK] + sqrtrho_r * wl[L_BK]) * inv_tot;
    const double bi2 = bi_roe * bi_roe;
    const double b_roe2 = bi2 + bj_roe * bj_roe + bk_roe * bk_roe;
    const double gamma_prime = gas.gm1;
    const double gp1 = gamma_prime - 1.;
    const double dbj = wl[L_BJ] - wr[L_BJ];
    const double dbk = wl[L_BK] - wr[L_BK];
    const double x_prime = (scale2<-1>(dbj * dbj + dbk * dbk) * gp1 * inv_tot);
    const double y_prime = (scale2<-1>(gp1 * (wl[L_RHO] + wr[L_RHO])) / rho_roe);
    const double tilde_a2 =
        (gamma_prime * (h_roe - scale2<-1>(v_roe2) - b_roe2 / rho_roe) - x_prime);
    const double tilde_vai2 = bi2 / rho_roe;
    const double tilde_va2 =
        (tilde_vai2 + (gamma_prime - y_prime) * (bj_roe * bj_roe + bk_roe * bk_roe) / rho_roe);
    const double s = tilde_a2 + tilde_va2;
    c_roe = sqrt(scale2<-1>(tilde_a2 + tilde_va2 +
                            sqrt(s * s - scale2<2>(tilde_a2) * tilde_vai2)));
  } else {  // roe_cs_ (:123-130)
    const double temp = h_roe - scale2<-1>(v_roe2);
    c_roe = sqrt(gas.gm1 * smax(temp, 0.));
  }
  *bp = fmax_i(vi_roe + c_roe, right_speed);
  *bm = fmin_i(vi_roe - c_roe, left_speed);
}

// HLLE for MHD (EnzoRiemannHLL.hpp:238-345), physical fluxes as in
// EnzoRiemannUtils.hpp:111-149
__device__ __forceinline__ void hlle(const Gas& gas, const double* wl, const double* wr,
                                     const CellGas<SOLVER_HLLE>& cl,
                                     const CellGas<SOLVER_HLLE>& cr, FaceFlux<double>& out) {
  const double bi2 = wl[L_BI] * wl[L_BI];  // the face's own B_i on both sides
  double Ul[8], Ur[8], Fl[8], Fr[8], b2[2], c[2];
#pragma unroll
  for (int k = 0; k < 2; k++) {
    const double* w = k == 0 ? wl : wr;
    const CellGas<SOLVER_HLLE>& cg = k == 0 ? cl : cr;
    double *U = k == 0 ? Ul : Ur, *F = k == 0 ? Fl : Fr;
    const double vi = w[L_VI], vj = w[L_VJ], vk = w[L_VK];
    const double Bi = w[L_BI], Bj = w[L_BJ], Bk = w[L_BK];
    b2[k] = bi2 + (Bj * Bj + Bk * Bk);
    c[k] = cfast_of(cg.v[0], cg.v[1], b2[k], bi2);
    U[L_RHO] = w[L_RHO];
    U[L_BJ] = Bj;
    U[L_BK] = Bk;
    U[L_VI] = vi * w[L_RHO];
    U[L_VJ] = vj * w[L_RHO];
    U[L_VK] = vk * w[L_RHO];
    U[L_E] = energy_of<true>(w, cg.v[3], b2[k]);
    const double ptot = w[L_E] + scale2<-1>(b2[k]);
    const double mom_i = U[L_VI];
    F[L_RHO] = mom_i;
    F[L_VI] = mom_i * vi - bi2 + ptot;
    F[L_VJ] = mom_i * vj - Bj * Bi;
    F[L_VK] = mom_i * vk - Bk * Bi;
    F[L_E] = ((U[L_E] + ptot) * vi - (Bi * vi + (Bj * vj + Bk * vk)) * Bi);
    F[L_BJ] = Bj * vi - Bi * vj;
    F[L_BK] = Bk * vi - Bi * vk;
  }
  double bp, bm;
  einfeldt<true>(gas, wl, wr, c[0], c[1], cl.v[2], cr.v[2], Ul[L_E], Ur[L_E], b2[0], b2[1], &bp,
                 &bm);
  bp = fmax_i(bp, 0.0);
  bm = fmin_i(bm, 0.0);
  const double inv_speed_diff = 1. / (bp - bm);
#pragma unroll
  for (int k = 0; k < 8; k++) {
    out.f[k] = k == L_BI ? 0.0
                         : ((bp * Fl[k] - bm * Fr[k] + (Ur[k] - Ul[k]) * bp * bm) *
                            inv_speed_diff);
  }
  out.eflux = eint_flux(gas.gm1, wl[L_RHO], wl[L_E], wr[L_RHO], wr[L_E], out.f[L_RHO]);
  out.vbar = (bp * wl[L_VI] - bm * wr[L_VI]) * inv_speed_diff;
}

// HLLC for hydrodynamics (EnzoRiemannHLLC.hpp:34-172).  One of the two sides has
// the weight zero; its products are zero, and left out, where its state is
// finite.
__device__ __forceinline__ void hllc(const Gas& gas, const double* wl, const double* wr,
                                     const CellGas<SOLVER_HLLC>& cl,
                                     const CellGas<SOLVER_HLLC>& cr, FaceFlux<double>& out) {
  const double pl = wl[L_E], pr = wr[L_E];
  const double El = energy_of<false>(wl, cl.v[2], 0.0), Er = energy_of<false>(wr, cr.v[2], 0.0);
  double cs_l, cs_r;
  einfeldt<false>(gas, wl, wr, cl.v[0], cr.v[0], cl.v[1], cr.v[1], El, Er, 0.0, 0.0, &cs_r, &cs_l);
  const double bm = fmin_i(cs_l, 0.0);
  const double bp = fmax_i(cs_r, 0.0);
  const double ul = cs_l - wl[L_VI], ur = cs_r - wr[L_VI];
  const double tl = (pl - ul * wl[L_RHO] * wl[L_VI]);
  const double tr = (pr - ur * wr[L_RHO] * wr[L_VI]);
  const double dl = wl[L_RHO] * ul;
  const double dr = neg_if(wr[L_RHO], true) * ur;
  const double q1 = 1.0 / (dl + dr);
  const double cw = (tr - tl) * q1;
  const double cp = smax((dl * tr + dr * tl) * q1, 0.);
  const bool left = ge0(cw);
  const double den = left ? cw - bm : bp - cw;
  const double sd = neg_if(cw, !left) / den;      // the side's weight
  const double sm = (left ? neg_if(bm, true) : bp) / den;
  // the side's momentum, energy, relative speed and fluxes
  auto side = [&](const double* w, double E, double b, double* f, double& ub) {
    const double mi = w[L_VI] * w[L_RHO];
    ub = w[L_VI] - b;
    f[0] = mi - b * w[L_RHO];
    f[1] = mi * ub + w[L_E];
    f[2] = (w[L_RHO] * w[L_VJ] * ub);
    f[3] = (w[L_RHO] * w[L_VK] * ub);
    f[4] = (E * ub + w[L_E] * w[L_VI]);
  };
  double w[8], f[5], ub;
#pragma unroll
  for (int k = 0; k < 8; k++) w[k] = left ? wl[k] : wr[k];
  side(w, left ? El : Er, left ? bm : bp, f, ub);
#pragma unroll
  for (int k = 0; k < 5; k++) f[k] = sd * f[k];
  ub = sd * ub;
  double o[8];
#pragma unroll
  for (int k = 0; k < 8; k++) o[k] = left ? wr[k] : wl[k];
  const double Eo = left ? Er : El, bo = left ? bp : bm;
  if (!is_finite(o[L_RHO]) || !is_finite(o[L_VI]) || !is_finite(o[L_VJ]) ||
      !is_finite(o[L_VK]) || !is_finite(o[L_E]) || !is_finite(Eo) || !is_finite(bo)) {
    rare_path();
    double fo[5], uo;
    side(o, Eo, bo, fo, uo);
#pragma unroll
    for (int k = 0; k < 5; k++) f[k] += 0.0 * fo[k];
    ub += 0.0 * uo;
  }
  out.f[L_RHO] = f[0];
  out.f[L_VI] = f[1] + (sm * cp);
  out.f[L_VJ] = f[2];
  out.f[L_VK] = f[3];
  out.f[L_E] = f[4] + (sm * cp * cw);
  out.f[L_BI] = out.f[L_BJ] = out.f[L_BK] = 0.0;
  out.eflux = eint_flux(gas.gm1, wl[L_RHO], pl, wr[L_RHO], pr, out.f[L_RHO]);
  out.vbar = ub;
}

// HLLE in FP32 (EnzoRiemannHLL.hpp:44-345): the same states, Einfeldt
// speeds and flux as the FP64 form, the left and right states in the two
// lanes of packed FP32 arithmetic.  Differences from the FP64 form lie only
// in rounding.
__device__ __forceinline__ void hlle(float g, const float* wl, const float* wr,
                                     FaceFlux<float>& out) {
  using namespace packed;
  const float2 HALF = s2(0.5f);
  const float2 p = f2(wl[L_E], wr[L_E]);
  const float2 d = f2(wl[L_RHO], wr[L_RHO]);
  const float2 u = f2(wl[L_VI], wr[L_VI]);
  const float2 vj = f2(wl[L_VJ], wr[L_VJ]), vk = f2(wl[L_VK], wr[L_VK]);
  const float2 bi = f2(wl[L_BI], wr[L_BI]);
  const float2 bj = f2(wl[L_BJ], wr[L_BJ]), bk = f2(wl[L_BK], wr[L_BK]);
  const float2 inv_d = f2(1.0f / d.x, 1.0f / d.y);
  const float gm1 = g - 1.0f;
  // conserved states and physical fluxes (EnzoRiemannUtils.hpp:48-149)
  const float2 mi = mul(u, d), mj = mul(vj, d), mk = mul(vk, d);
  const float2 b2 = fma(bi, bi, fma(bj, bj, mul(bk, bk)));
  const float2 v2 = fma(u, u, fma(vj, vj, mul(vk, vk)));
  const float2 E = add(fma(p, s2(1.0f / gm1), mul(mul(HALF, d), v2)), mul(HALF, b2));
  const float2 pt = fma(HALF, b2, p);
  const float2 vb = fma(bi, u, fma(bj, vj, mul(bk, vk)));
  float2 F[8], U[8];
  U[L_RHO] = d;
  U[L_BI] = bi;
  U[L_BJ] = bj;
  U[L_BK] = bk;
  U[L_VI] = mi;
  U[L_VJ] = mj;
  U[L_VK] = mk;
  U[L_E] = E;
  F[L_RHO] = mi;
  F[L_BI] = s2(0.0f);
  F[L_BJ] = sub(mul(bj, u), mul(bi, vj));
  F[L_BK] = sub(mul(bk, u), mul(bi, vk));
  F[L_VI] = fma(mi, u, sub(pt, mul(bi, bi)));
  F[L_VJ] = sub(mul(mi, vj), mul(bj, bi));
  F[L_VK] = sub(mul(mi, vk), mul(bk, bi));
  F[L_E] = sub(mul(add(E, pt), u), mul(vb, bi));
  // Einfeldt speeds: fast speeds, Roe averages, Roe fast speed
  const float2 c2 = mul(mul(s2(g), p), inv_d);
  const float2 va2 = mul(b2, inv_d);
  const float2 vac2 = mul(mul(bi, bi), inv_d);
  const float2 sfs = add(c2, va2);
  const float2 disc = fma(sfs, sfs, mul(mul(s2(-4.0f), c2), vac2));
  const float2 cfh = mul(HALF, add(sfs, f2(sqrtf(disc.x), sqrtf(disc.y))));
  const float left_speed = u.x - sqrtf(cfh.x), right_speed = u.y + sqrtf(cfh.y);
  const float2 sq = f2(sqrtf(d.x), sqrtf(d.y));
  const float inv_tot = 1.0f / (sq.x + sq.y);
  const float2 su = mul(sq, u), sv = mul(sq, vj), sw = mul(sq, vk);
  const float vi_roe = (su.x + su.y) * inv_tot;
  const float vj_roe = (sv.x + sv.y) * inv_tot;
  const float vk_roe = (sw.x + sw.y) * inv_tot;
  const float v_roe2 = vi_roe * vi_roe + vj_roe * vj_roe + vk_roe * vk_roe;
  const float2 sh = mul(sq, mul(add(E, pt), inv_d));
  const float h_roe = (sh.x + sh.y) * inv_tot;
  const float rho_roe = sq.x * sq.y;
  const float inv_rho_roe = 1.0f / rho_roe;
  const float bi_roe = bi.x;
  const float bj_roe = (sq.x * bj.y + sq.y * bj.x) * inv_tot;
  const float bk_roe = (sq.x * bk.y + sq.y * bk.x) * inv_tot;
  const float bt_roe2 = bj_roe * bj_roe + bk_roe * bk_roe;
  const float b_roe2 = bi_roe * bi_roe + bt_roe2;
  const float dbj = bj.x - bj.y, dbk = bk.x - bk.y;
  const float x_prime = (dbj * dbj + dbk * dbk) * 0.5f * (gm1 - 1.0f) * inv_tot;
  const float y_prime = (gm1 - 1.0f) * (d.x + d.y) * 0.5f * inv_rho_roe;
  const float tilde_a2 = gm1 * (h_roe - 0.5f * v_roe2 - b_roe2 * inv_rho_roe) - x_prime;
  const float tilde_vai2 = bi_roe * bi_roe * inv_rho_roe;
  const float tilde_va2 = tilde_vai2 + (gm1 - y_prime) * bt_roe2 * inv_rho_roe;
  const float sr = tilde_a2 + tilde_va2;
  const float c_roe =
      sqrtf(0.5f * (tilde_a2 + tilde_va2 + sqrtf(sr * sr - 4.0f * tilde_a2 * tilde_vai2)));
  const float bp = fmaxf(fmaxf(vi_roe + c_roe, right_speed), 0.0f);
  const float bm = fminf(fminf(vi_roe - c_roe, left_speed), 0.0f);
  const float inv_speed_diff = 1.0f / (bp - bm);
  const float bpbm = bp * bm;
  const float2 BPM = f2(bp, -bm);
#pragma unroll
  for (int k = 0; k < 8; k++) {
    const float2 t = mul(BPM, F[k]);
    out.f[k] = ((t.x + t.y) + (U[k].y - U[k].x) * bpbm) * inv_speed_diff;
  }
  out.eflux = eint_flux(g - 1.0f, d.x, p.x, d.y, p.y, out.f[L_RHO]);
  out.vbar = (bp * u.x - bm * u.y) * inv_speed_diff;
}

// HLLC in FP32 (EnzoRiemannHLLC.hpp:34-172 with the Einfeldt speeds of
// EnzoRiemannHLL.hpp:44-172): the same states, speeds and flux as the FP64
// form, the left and right states in the two lanes of packed FP32
// arithmetic.  Differences from the FP64 form lie only in rounding.
__device__ __forceinline__ void hllc(float g, const float* wl, const float* wr,
                                     FaceFlux<float>& out) {
  using namespace packed;
  const float2 HALF = s2(0.5f);
  const float2 p = f2(wl[L_E], wr[L_E]);
  const float2 d = f2(wl[L_RHO], wr[L_RHO]);
  const float2 u = f2(wl[L_VI], wr[L_VI]);
  const float2 vj = f2(wl[L_VJ], wr[L_VJ]), vk = f2(wl[L_VK], wr[L_VK]);
  const float2 inv_d = f2(1.0f / d.x, 1.0f / d.y);
  const float gm1 = g - 1.0f;
  // conserved momentum and total energy density
  const float2 mom = mul(u, d);
  const float2 v2 = fma(u, u, fma(vj, vj, mul(vk, vk)));
  const float2 E = fma(p, s2(1.0f / gm1), mul(mul(HALF, d), v2));
  // Einfeldt speeds: sound speeds, Roe averages
  const float2 c2 = mul(mul(s2(g), p), inv_d);
  const float left_speed = u.x - sqrtf(c2.x), right_speed = u.y + sqrtf(c2.y);
  const float2 sq = f2(sqrtf(d.x), sqrtf(d.y));
  const float inv_tot = 1.0f / (sq.x + sq.y);
  const float2 su = mul(sq, u), sv = mul(sq, vj), sw = mul(sq, vk);
  const float vi_roe = (su.x + su.y) * inv_tot;
  const float vj_roe = (sv.x + sv.y) * inv_tot;
  const float vk_roe = (sw.x + sw.y) * inv_tot;
  const float v_roe2 = vi_roe * vi_roe + vj_roe * vj_roe + vk_roe * vk_roe;
  const float2 sh = mul(sq, mul(add(E, p), inv_d));
  const float h_roe = (sh.x + sh.y) * inv_tot;
  const float c_roe = sqrtf(gm1 * smax(h_roe - 0.5f * v_roe2, 0.0f));
  const float cs_r = fmaxf(vi_roe + c_roe, right_speed);
  const float cs_l = fminf(vi_roe - c_roe, left_speed);
  const float bm = fminf(cs_l, 0.0f);
  const float bp = fmaxf(cs_r, 0.0f);
  // contact speed and pressure
  const float2 cu = sub(f2(cs_l, cs_r), u);
  const float2 t = sub(p, mul(cu, mom));
  const float2 dd = mul(d, cu);
  const float dl = dd.x, dr = -dd.y;
  const float q1 = 1.0f / (dl + dr);
  const float cw = (t.y - t.x) * q1;
  const float cp = smax((dl * t.y + dr * t.x) * q1, 0.0f);
  const bool left = cw >= 0.0f;
  const float inv_c = 1.0f / (left ? cw - bm : bp - cw);
  const float sc = fabsf(cw) * inv_c;
  const float sl = left ? sc : 0.0f, sr = left ? 0.0f : sc;
  const float sm = (left ? -bm : bp) * inv_c;
  // side fluxes relative to the outer wave speeds
  const float2 B = f2(bm, bp);
  const float2 ub = sub(u, B);
  const float2 df = sub(mom, mul(B, d));
  const float2 uf = fma(mom, ub, p);
  const float2 vf = mul(mul(d, vj), ub);
  const float2 wf = mul(mul(d, vk), ub);
  const float2 ef = fma(E, ub, mul(p, u));
  const float2 SLR = f2(sl, sr);
  const float2 frho = mul(SLR, df), fu = mul(SLR, uf), fv = mul(SLR, vf), fw = mul(SLR, wf),
               fe = mul(SLR, ef), fvb = mul(SLR, ub);
  out.f[L_RHO] = frho.x + frho.y;
  out.f[L_VI] = (fu.x + fu.y) + sm * cp;
  out.f[L_VJ] = fv.x + fv.y;
  out.f[L_VK] = fw.x + fw.y;
  out.f[L_E] = (fe.x + fe.y) + sm * cp * cw;
  out.f[L_BI] = out.f[L_BJ] = out.f[L_BK] = 0.0f;
  out.eflux = eint_flux(g - 1.0f, d.x, p.x, d.y, p.y, out.f[L_RHO]);
  out.vbar = fvb.x + fvb.y;
}

// The face flux of SOLVER: FP32 from gamma, FP64 from the gas constants and the
// cells' (or face states') own quantities.
template <int SOLVER>
__device__ __forceinline__ void riemann(float g, const float* wl, const float* wr,
                                        FaceFlux<float>& out) {
  if (SOLVER == SOLVER_HLLD) hlld(g, wl, wr, out);
  else if (SOLVER == SOLVER_HLLE) hlle(g, wl, wr, out);
  else hllc(g, wl, wr, out);
}
template <int SOLVER>
__device__ __forceinline__ void riemann(const Gas& gas, const double* wl, const double* wr,
                                        const CellGas<SOLVER>& cl, const CellGas<SOLVER>& cr,
                                        FaceFlux<double>& out) {
  if constexpr (SOLVER == SOLVER_HLLD) hlld(gas, wl, wr, cl, cr, out);
  else if constexpr (SOLVER == SOLVER_HLLE) hlle(gas, wl, wr, cl, cr, out);
  else hllc(gas, wl, wr, cl, cr, out);
}
template <int SOLVER>
__device__ __forceinline__ void riemann(const Gas& gas, const double* wl, const double* wr,
                                        FaceFlux<double>& out) {
  CellGas<SOLVER> cl, cr;
  cl.init(gas, wl[L_RHO], wl[L_E]);
  cr.init(gas, wr[L_RHO], wr[L_E]);
  riemann<SOLVER>(gas, wl, wr, cl, cr, out);
}

}  // namespace vlct
