// rfgpu_kernels.cuh - residual / RK-stage kernels, templated on the working
// precision R of reconstruction, limiter and flux arithmetic.  Included by
// rfgpu_fp64.cu (R = double, built with --fmad=false so every expression
// rounds exactly like the unfused reference expression) and rfgpu_mixed.cu
// (R = float).  On the FP64 path residual accumulation, RK update, EOS and
// time step are FP64 in the reference's operation order; on the mixed path
// they are FP32 with compensation (TwoSum residual sums, a float-float
// conserved state, gather_update_mixed below).
//
// Every kernel walks a tile list (region, first item); a tile is blockDim.x
// consecutive cells / faces / boundary faces of one region, so one launch
// covers one region or a whole batch of regions.  Grids smaller than the tile
// count walk the list persistently.
#pragma once

#include <algorithm>
#include <type_traits>

#include "rfgpu_internal.h"
#include "rfgpu_soft64.cuh"

namespace rfgpu {

template <int N> struct Int { static constexpr int value = N; };

template <typename R> __device__ __forceinline__ R rmin(R a, R b) { return b < a ? b : a; }
template <typename R> __device__ __forceinline__ R rmax(R a, R b) { return b > a ? b : a; }
template <> __device__ __forceinline__ Sd rmin(Sd a, Sd b) { return b < a || unknown(b) ? b : a; }
template <> __device__ __forceinline__ Sd rmax(Sd a, Sd b) { return b > a || unknown(b) ? b : a; }
__device__ __forceinline__ constexpr bool unknown(double) { return false; }
__device__ __forceinline__ double value(double x) { return x; }
__device__ __forceinline__ double value(Sd x) { return x.v; }
__device__ __forceinline__ constexpr bool unknown(float) { return false; }
// max(x, 0) as the reference writes it (0 for NaN)
template <typename R> __device__ __forceinline__ R pos_part(R x) { return x > R(0) ? x : R(0); }
template <> __device__ __forceinline__ Sd pos_part(Sd x) { return x > Sd(0.0) || unknown(x) ? x : Sd(0.0); }

// ---- perfect-gas relations (libfloflu/MixtPerf_*.F90) ----------------------
template <typename R>
__device__ __forceinline__ R eo_dgpuvw(R D, R G, R P, R U, R V, R W) {
  return P / (D * (G - R(1))) + scale<-1>(U * U + V * V + W * W) + R(0);
}

// Physical constants in the working precision: the FP64 values on the FP64
// path, their FP32 copies on the mixed path (no per-thread conversions).
template <typename R> struct PC;
template <> struct PC<double> {
  const Phys &p;
  __device__ double cp() const { return p.refCp; }
  __device__ double g() const { return p.refGamma; }
  __device__ double gc() const { return p.gcRef; }
  __device__ double gvG() const { return p.gvG; }
  __device__ double eps() const { return p.epsentr; }
  __device__ double diss() const { return p.dissFact; }
};
template <> struct PC<Sd> {
  const Phys &p;
  __device__ Sd cp() const { return Sd(p.refCp); }
  __device__ Sd g() const { return Sd(p.refGamma); }
  __device__ Sd gc() const { return Sd(p.gcRef); }
  __device__ Sd gvG() const { return Sd(p.gvG); }
  __device__ Sd eps() const { return Sd(p.epsentr); }
  __device__ Sd diss() const { return Sd(p.dissFact); }
};
template <> struct PC<float> {
  const Phys &p;
  __device__ float cp() const { return p.refCpF; }
  __device__ float g() const { return p.refGammaF; }
  __device__ float gc() const { return p.gcRefF; }
  __device__ float gvG() const { return p.gvGF; }
  __device__ float eps() const { return p.epsentrF; }
  __device__ float diss() const { return p.dissFactF; }
};

// ---- flux functions on reconstructed states ----------------------------------
// Written over a number type: on the FP64 path (R = Sd) the products written
// prod() - those with the normal and the area, of reused factors - are integer
// products and scale<K>() works on the exponent.  More of them (all kinetic
// energies, Roe's averages and waves, HLLC's star states) measured slower:
// 64^3 tets Roe 1.83 -> 1.71 ms but 4,000 cells 22.7 -> 27.1 us, HLLC 1.44 ->
// 1.50 ms; every product: Roe 1.95, HLLC 1.52 ms.

// AUSM+ (modflu/RFLU_ModAUSMFlux.F90:282-367 with the state set-up of :2787-2846)
template <typename R>
__device__ __forceinline__ void ausm_flux(const Phys &ph, const R L[5], const R Rt[5],
                                          R nx, R ny, R nz, R nm, R flx[5]) {
  const PC<R> k{ph};
  const R cp = k.cp(), g = k.g(), gc = k.gc(), fs = R(0);
  R rl = L[0], ul = L[1], vl = L[2], wl = L[3], pl = L[4];
  R rr = Rt[0], ur = Rt[1], vr = Rt[2], wr = Rt[3], pr = Rt[4];
  R tl = pl / (rl * gc);
  R al = sqrt(g * gc * tl);
  R Hl = cp * tl + scale<-1>(ul * ul + vl * vl + wl * wl) + R(0);
  R tr = pr / (rr * gc);
  R ar = sqrt(g * gc * tr);
  R Hr = cp * tr + scale<-1>(ur * ur + vr * vr + wr * wr) + R(0);
  R ql = prod(ul, nx) + prod(vl, ny) + prod(wl, nz) - fs;
  R qr = prod(ur, nx) + prod(vr, ny) + prod(wr, nz) - fs;
  R af = scale<-1>(al + ar);
  R ml = ql / af, mla = fabs(ml);
  R mr = qr / af, mra = fabs(mr);
  R mlp, wtl, mrm, wtr;
  if (mla <= R(1)) {
    mlp = scale<-2>(ml + R(1)) * (ml + R(1)) + scale<-3>(ml * ml - R(1)) * (ml * ml - R(1));
    wtl = scale<-2>(ml + R(1)) * (ml + R(1)) * (R(2) - ml) +
          R(0.1875) * ml * (ml * ml - R(1)) * (ml * ml - R(1));
  } else {
    mlp = scale<-1>(ml + mla);
    wtl = scale<-1>(R(1) + ml / mla);
  }
  if (mra <= R(1)) {
    mrm = -(scale<-2>(mr - R(1)) * (mr - R(1))) - scale<-3>(mr * mr - R(1)) * (mr * mr - R(1));
    wtr = scale<-2>(mr - R(1)) * (mr - R(1)) * (R(2) + mr) -
          R(0.1875) * mr * (mr * mr - R(1)) * (mr * mr - R(1));
  } else {
    mrm = scale<-1>(mr - mra);
    wtr = scale<-1>(R(1) - mr / mra);
  }
  R mf = mlp + mrm, mfa = fabs(mf);
  R mfp = scale<-1>(mf + mfa), mfm = scale<-1>(mf - mfa);
  R pf = wtl * pl + wtr * pr;
  flx[0] = prod((af * (mfp * rl + mfm * rr)), nm);
  flx[1] = prod((af * (prod(mfp * rl, ul) + prod(mfm * rr, ur)) + prod(pf, nx)), nm);
  flx[2] = prod((af * (prod(mfp * rl, vl) + prod(mfm * rr, vr)) + prod(pf, ny)), nm);
  flx[3] = prod((af * (prod(mfp * rl, wl) + prod(mfm * rr, wr)) + prod(pf, nz)), nm);
  flx[4] = prod((af * (prod(mfp * rl, Hl) + prod(mfm * rr, Hr)) + pf * fs), nm);
}

// AUSM+up, RFLU_AUSMPlusUp_FluxFunction2 (modflu/RFLU_ModAUSMPlusUpFlux.F90:
// 469-588) with vFracF = 1 (no particles): AUSM+ split Mach numbers and
// pressures plus the pressure-diffusion (kp, sigma) and velocity-diffusion
// (ku) terms; the routine's blending factor is overwritten with 1, so
// alpha = 3/16.  H and a of both sides come from the caller (they are set up
// differently at first and second order).
template <typename R>
__device__ __forceinline__ void ausmup_flux(R sigma, R kp, R ku, const R L[5], const R Rt[5],
                                            R Hl, R al, R Hr, R ar, R nx, R ny, R nz, R nm,
                                            R flx[5]) {
  const R fs = R(0);
  const R rl = L[0], ul = L[1], vl = L[2], wl = L[3], pl = L[4];
  const R rr = Rt[0], ur = Rt[1], vr = Rt[2], wr = Rt[3], pr = Rt[4];
  R ql = prod(ul, nx) + prod(vl, ny) + prod(wl, nz) - fs;
  R qr = prod(ur, nx) + prod(vr, ny) + prod(wr, nz) - fs;
  R af = scale<-1>(al + ar);
  R ml = ql / af, mla = fabs(ml);
  R mr = qr / af, mra = fabs(mr);
  R mbarsq = scale<-1>(ml * ml + mr * mr);
  const R fa = R(1);
  const R alpha = R(0.1875) * (R(5) * fa * fa - R(4));
  R mlp, wtl, mrm, wtr;
  if (mla <= R(1)) {
    mlp = scale<-2>(ml + R(1)) * (ml + R(1)) + scale<-3>(ml * ml - R(1)) * (ml * ml - R(1));
    wtl = scale<-2>(ml + R(1)) * (ml + R(1)) * (R(2) - ml) +
          alpha * ml * (ml * ml - R(1)) * (ml * ml - R(1));
  } else {
    mlp = scale<-1>(ml + mla);
    wtl = scale<-1>(R(1) + ml / mla);
  }
  if (mra <= R(1)) {
    mrm = -(scale<-2>(mr - R(1)) * (mr - R(1))) - scale<-3>(mr * mr - R(1)) * (mr * mr - R(1));
    wtr = scale<-2>(mr - R(1)) * (mr - R(1)) * (R(2) + mr) -
          alpha * mr * (mr * mr - R(1)) * (mr * mr - R(1));
  } else {
    mrm = scale<-1>(mr - mra);
    wtr = scale<-1>(R(1) - mr / mra);
  }
  R rf = scale<-1>(rl + rr);
  R sigmabar = R(1) - sigma * mbarsq;
  R mp = (-(kp * pos_part(sigmabar) * (pr - pl))) / (fa * rf * af * af);
  R pu = -(ku * wtl * wtr * fa * af * (rl + rr) * (qr - ql));
  R mf = mlp + mrm + mp, mfa = fabs(mf);
  R mfp = scale<-1>(mf + mfa), mfm = scale<-1>(mf - mfa);
  R pf = wtl * pl + wtr * pr + pu;
  const R vFracF = R(1);
  flx[0] = prod((af * vFracF * (mfp * rl + mfm * rr)), nm);
  flx[1] = prod((af * vFracF * (prod(mfp * rl, ul) + prod(mfm * rr, ur)) + prod(pf, nx)), nm);
  flx[2] = prod((af * vFracF * (prod(mfp * rl, vl) + prod(mfm * rr, vr)) + prod(pf, ny)), nm);
  flx[3] = prod((af * vFracF * (prod(mfp * rl, wl) + prod(mfm * rr, wr)) + prod(pf, nz)), nm);
  flx[4] = prod((af * vFracF * (prod(mfp * rl, Hl) + prod(mfm * rr, Hr)) + pf * fs), nm);
}

template <typename R>
__device__ __forceinline__ R entropy_fix(R l, R d) {  // RFLU_ModEntropyFixes.F90:95-106
  return (l > d) ? l : (l * l + d * d) / scale<1>(d);
}

// Roe with the Harten-Hyman entropy fix (modflu/RFLU_ModRoeFlux.F90:2725-2855)
template <typename R>
__device__ __forceinline__ void roe_flux(const Phys &ph, const R L[5], const R Rt[5], R nx,
                                         R ny, R nz, R nm, R flx[5]) {
  const PC<R> k{ph};
  const R cp = k.cp(), g = k.g(), gc = k.gc(), fs = R(0);
  R rl = L[0], ul = L[1], vl = L[2], wl = L[3], pl = L[4];
  R rr = Rt[0], ur = Rt[1], vr = Rt[2], wr = Rt[3], pr = Rt[4];
  R tl = pl / (rl * gc);
  R Hl = cp * tl + scale<-1>(ul * ul + vl * vl + wl * wl) + R(0);
  R ql = prod(ul, nx) + prod(vl, ny) + prod(wl, nz) - fs;
  R tr = pr / (rr * gc);
  R Hr = cp * tr + scale<-1>(ur * ur + vr * vr + wr * wr) + R(0);
  R qr = prod(ur, nx) + prod(vr, ny) + prod(wr, nz) - fs;
  R rh = sqrt(rl * rr);
  R wt = rl / (rl + rh);
  R uh = wt * ul + (R(1) - wt) * ur;
  R vh = wt * vl + (R(1) - wt) * vr;
  R wh = wt * wl + (R(1) - wt) * wr;
  R Hh = wt * Hl + (R(1) - wt) * Hr;
  R qh = prod(uh, nx) + prod(vh, ny) + prod(wh, nz) - fs;
  R sh = scale<-1>(uh * uh + vh * vh + wh * wh);
  R ah = sqrt((g - R(1)) * (Hh - scale<-1>(scale<1>(sh))));
  R l1 = fabs(qh - ah), l2 = fabs(qh), l5 = fabs(qh + ah);
  R efc = k.eps() * l5;
  l1 = entropy_fix(l1, efc);
  l2 = entropy_fix(l2, efc);
  l5 = entropy_fix(l5, efc);
  R dr = rr - rl, du = ur - ul, de = vr - vl, dw = wr - wl, dp = pr - pl;
  R dq = prod(du, nx) + prod(de, ny) + prod(dw, nz);
  R dv1 = (dp - rh * ah * dq) / (scale<1>(ah) * ah);
  R dv5 = (dp + rh * ah * dq) / (scale<1>(ah) * ah);
  R dv2 = dr - dp / (ah * ah);
  R t1 = l1 * dv1, t2 = l2 * dv2, t3 = l2 * rh, t5 = l5 * dv5;
  R df = k.diss();
  flx[0] = prod(scale<-1>(ql * rl + qr * rr), nm) - R(0.5) * df * (t1 + t2 + t5) * nm;
  flx[1] = prod(scale<-1>(ql * rl * ul + prod(pl, nx) + qr * rr * ur + prod(pr, nx)), nm) -
           prod(scale<-1>(df) * (t1 * (uh - prod(ah, nx)) + t2 * uh + t3 * (du - prod(dq, nx)) + t5 * (uh + prod(ah, nx))), nm);
  flx[2] = prod(scale<-1>(ql * rl * vl + prod(pl, ny) + qr * rr * vr + prod(pr, ny)), nm) -
           prod(scale<-1>(df) * (t1 * (vh - prod(ah, ny)) + t2 * vh + t3 * (de - prod(dq, ny)) + t5 * (vh + prod(ah, ny))), nm);
  flx[3] = prod(scale<-1>(ql * rl * wl + prod(pl, nz) + qr * rr * wr + prod(pr, nz)), nm) -
           prod(scale<-1>(df) * (t1 * (wh - prod(ah, nz)) + t2 * wh + t3 * (dw - prod(dq, nz)) + t5 * (wh + prod(ah, nz))), nm);
  flx[4] = prod(scale<-1>(ql * rl * Hl + pl * fs + qr * rr * Hr + pr * fs), nm) -
           prod(scale<-1>(df) * (t1 * (Hh - qh * ah) + t2 * sh +
                                 t3 * (uh * du + vh * de + wh * dw - qh * dq) + t5 * (Hh + qh * ah)), nm);
}

// HLLC (modflu/RFLU_ModHLLCFlux.F90:2296-2409); irl/irr are the reciprocal
// cell densities before reconstruction, as the reference uses in Hl/Hr.
template <typename R>
__device__ __forceinline__ void hllc_flux(const Phys &ph, const R L[5], const R Rt[5], R irl,
                                          R irr, R nx, R ny, R nz, R nm, R flx[5]) {
  const R g = PC<R>{ph}.g(), fs = R(0);
  R rl = L[0], ul = L[1], vl = L[2], wl = L[3], pl = L[4];
  R rr = Rt[0], ur = Rt[1], vr = Rt[2], wr = Rt[3], pr = Rt[4];
  R el = eo_dgpuvw(rl, g, pl, ul, vl, wl);
  R al = sqrt(g * pl / rl);
  R ql = prod(ul, nx) + prod(vl, ny) + prod(wl, nz) - fs;
  R Hl = el + irl * pl;
  R er = eo_dgpuvw(rr, g, pr, ur, vr, wr);
  R ar = sqrt(g * pr / rr);
  R qr = prod(ur, nx) + prod(vr, ny) + prod(wr, nz) - fs;
  R Hr = er + irr * pr;
  R wt1 = sqrt(rr / rl);
  R wt2 = R(1) / (R(1) + wt1);
  R us = wt2 * (ul + wt1 * ur);
  R vs = wt2 * (vl + wt1 * vr);
  R ws = wt2 * (wl + wt1 * wr);
  R qs = wt2 * (ql + wt1 * qr);
  R Hs = wt2 * (Hl + wt1 * Hr);
  R Vms = us * us + vs * vs + ws * ws;
  R as = sqrt((g - R(1)) * (Hs - scale<-1>(Vms)));
  R sl = rmin(ql - al, qs - as);
  R sr = rmax(qr + ar, qs + as);
  if (unknown(sl) || unknown(sr)) {
    flx[0] = flx[1] = flx[2] = flx[3] = flx[4] = sl + sr;
  } else if (sl > R(0)) {
    flx[0] = ql * rl * nm;
    flx[1] = prod((ql * rl * ul + prod(pl, nx)), nm);
    flx[2] = prod((ql * rl * vl + prod(pl, ny)), nm);
    flx[3] = prod((ql * rl * wl + prod(pl, nz)), nm);
    flx[4] = prod((ql * (rl * el + pl) + pl * fs), nm);
  } else if (sr < R(0)) {
    flx[0] = qr * rr * nm;
    flx[1] = prod((qr * rr * ur + prod(pr, nx)), nm);
    flx[2] = prod((qr * rr * vr + prod(pr, ny)), nm);
    flx[3] = prod((qr * rr * wr + prod(pr, nz)), nm);
    flx[4] = prod((qr * (rr * er + pr) + pr * fs), nm);
  } else {
    R sm = (rr * qr * (sr - qr) - rl * ql * (sl - ql) - pr + pl) / (rr * (sr - qr) - rl * (sl - ql));
    R ps = pl + rl * (ql - sl) * (ql - sm);
    R rs, rus, rvs, rws, res, term;
    if (sm > R(0)) {
      term = R(1) / (sl - sm);
      rs = term * (sl - ql) * rl;
      rus = term * ((sl - ql) * rl * ul + (ps - pl) * nx);
      rvs = term * ((sl - ql) * rl * vl + (ps - pl) * ny);
      rws = term * ((sl - ql) * rl * wl + (ps - pl) * nz);
      res = term * ((sl - ql) * rl * el + (ps * sm - pl * ql));
    } else {
      term = R(1) / (sr - sm);
      rs = term * (sr - qr) * rr;
      rus = term * ((sr - qr) * rr * ur + (ps - pr) * nx);
      rvs = term * ((sr - qr) * rr * vr + (ps - pr) * ny);
      rws = term * ((sr - qr) * rr * wr + (ps - pr) * nz);
      res = term * ((sr - qr) * rr * er + (ps * sm - pr * qr));
    }
    flx[0] = sm * rs * nm;
    flx[1] = prod((sm * rus + prod(ps, nx)), nm);
    flx[2] = prod((sm * rvs + prod(ps, ny)), nm);
    flx[3] = prod((sm * rws + prod(ps, nz)), nm);
    flx[4] = prod((sm * (res + ps) - ps * fs), nm);
  }
}

// ---- vector access to AoS records --------------------------------------------
// Records are 32-byte aligned, so one record row of 8 floats (or 4 doubles) is
// a single 256-bit access: one request per warp touching each 32-byte sector
// once, where two 128-bit halves would issue two requests over the same
// sectors.  ld8/ld4 read through the non-coherent path and are for data no
// thread writes during the kernel; ld8_rw is the coherent form for a thread's
// own record that the same kernel rewrites.
// Read-once streams (per-face and per-cell arrays a pass reads exactly once):
// with H = 1 loaded L1::evict_first so L1 keeps the gathered records the pass
// reuses; H = 0 plain loads.  lds_rw is the coherent form for data the same
// kernel later overwrites (the thread's own state rows).
// Measured on the 128^3 tet box (mixed): update pass 0.650 -> 0.636 ms with
// its hint, gradient pass 1.928 -> 1.925 ms, face pass unchanged (0.636 ms;
// 0.631 ms with and without it once the gradient rows are prefetched), so the
// face pass keeps plain loads.
// Update face loop: the first RF_UPD_PRE face codes loaded together ahead of
// the flux gathers (measured: update pass 0.636 -> 0.596 ms with 4, 0.598 ms
// with 6).
#ifndef RF_UPD_PRE
#define RF_UPD_PRE 6
#endif
// RECONST 2 pass, mixed path: gradient rows gathered together per group and
// the weights from the hardware reciprocal.  Measured on the 128^3 tet box:
// exact division 4.95 ms (2 rows: 5.80, 4 rows: 6.62, the division code's
// registers), reciprocal 4.08 ms, with 2 rows 3.61 ms, with 4 rows 3.48 ms.
// The FP64 path keeps the IEEE division and one row at a time.
#ifndef RF_WENO_U
#define RF_WENO_U 4
#endif
#ifndef RF_WENO_FASTRCP
#define RF_WENO_FASTRCP 1
#endif
// Face pass: both cells' gradient rows prefetched into L1 as soon as the
// face's cells are known (measured 0.640 -> 0.631 ms).
#ifndef RF_FACE_PF
#define RF_FACE_PF 1
#endif
#ifndef RF_HINT_G
#define RF_HINT_G 1   // gradient pass: cell->face lists, WLSQ factor terms
#endif
#ifndef RF_HINT_F
#define RF_HINT_F 0   // face pass: f2c, normals, reconstruction offsets
#endif
#ifndef RF_HINT_U
#define RF_HINT_U 1   // update pass: face codes, state rows, increments, 1/vol
#endif
template <int H>
__device__ __forceinline__ int lds(const int *__restrict__ p) {
  if constexpr (H) {
    int v;
    asm("ld.global.nc.L1::evict_first.s32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
  } else {
    return *p;
  }
}
template <int H>
__device__ __forceinline__ float lds(const float *__restrict__ p) {
  if constexpr (H) {
    float v;
    asm("ld.global.nc.L1::evict_first.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
  } else {
    return *p;
  }
}
template <int H>
__device__ __forceinline__ double lds(const double *__restrict__ p) {
  if constexpr (H) {
    double v;
    asm("ld.global.nc.L1::evict_first.f64 %0, [%1];" : "=d"(v) : "l"(p));
    return v;
  } else {
    return *p;
  }
}
template <int H>
__device__ __forceinline__ float lds_rw(const float *p) {
  if constexpr (H) {
    float v;
    asm volatile("ld.global.L1::evict_first.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
  } else {
    return *p;
  }
}
template <int H>
__device__ __forceinline__ double lds_rw(const double *p) {
  if constexpr (H) {
    double v;
    asm volatile("ld.global.L1::evict_first.f64 %0, [%1];" : "=d"(v) : "l"(p));
    return v;
  } else {
    return *p;
  }
}

// The stencil-index stream of the mixed gradient pass: each index is read
// once, so it is loaded L1::evict_first and leaves L1 to the neighbour records
// the member gathers reuse (measured 1.955 -> 1.924 ms per pass on the
// 128^3 tet box; evict_last on the record gathers themselves changed nothing).
__device__ __forceinline__ int ld_index(const int *__restrict__ p) {
  int v;
  asm("ld.global.nc.L1::evict_first.s32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ void ld8(const float *__restrict__ p, float v[8]) {
  asm("ld.global.nc.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
      : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]),
        "=f"(v[7])
      : "l"(p));
}
__device__ __forceinline__ void ld4(const double *__restrict__ p, double v[4]) {
  asm("ld.global.nc.v4.f64 {%0,%1,%2,%3}, [%4];"
      : "=d"(v[0]), "=d"(v[1]), "=d"(v[2]), "=d"(v[3])
      : "l"(p));
}
__device__ __forceinline__ void ld8(const double *__restrict__ p, double v[8]) {
  ld4(p, v);
  ld4(p + 4, v + 4);
}
__device__ __forceinline__ void ld8_rw(const float *p, float v[8]) {
  asm volatile("ld.global.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]),
                 "=f"(v[6]), "=f"(v[7])
               : "l"(p)
               : "memory");
}
__device__ __forceinline__ void ld8_rw(const double *p, double v[8]) {
#pragma unroll
  for (int i = 0; i < 2; ++i)
    asm volatile("ld.global.v4.f64 {%0,%1,%2,%3}, [%4];"
                 : "=d"(v[4 * i]), "=d"(v[4 * i + 1]), "=d"(v[4 * i + 2]), "=d"(v[4 * i + 3])
                 : "l"(p + 4 * i)
                 : "memory");
}
__device__ __forceinline__ void ld4(const float *__restrict__ p, float v[4]) {
  float4 a = *reinterpret_cast<const float4 *>(p);
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
}
template <int H>
__device__ __forceinline__ void ld4s(const float *__restrict__ p, float v[4]) {
  if constexpr (H)
    asm("ld.global.nc.L1::evict_first.v4.f32 {%0,%1,%2,%3}, [%4];"
        : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]) : "l"(p));
  else
    ld4(p, v);
}
template <int H>
__device__ __forceinline__ void ld4s(const double *__restrict__ p, double v[4]) {
  if constexpr (H)
    asm("ld.global.nc.L1::evict_first.v4.f64 {%0,%1,%2,%3}, [%4];"
        : "=d"(v[0]), "=d"(v[1]), "=d"(v[2]), "=d"(v[3]) : "l"(p));
  else
    ld4(p, v);
}
__device__ __forceinline__ void st8(float *p, const float v[8]) {
  asm volatile("st.global.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "f"(v[0]), "f"(v[1]),
               "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7])
               : "memory");
}
__device__ __forceinline__ void st8(double *p, const double v[8]) {
#pragma unroll
  for (int i = 0; i < 2; ++i)
    asm volatile("st.global.v4.f64 [%0], {%1,%2,%3,%4};" ::"l"(p + 4 * i), "d"(v[4 * i]),
                 "d"(v[4 * i + 1]), "d"(v[4 * i + 2]), "d"(v[4 * i + 3])
                 : "memory");
}
template <typename R>
__device__ __forceinline__ void ld16(const R *__restrict__ p, R v[16]) {
  ld8(p, v);
  ld8(p + 8, v + 8);
}
template <typename R>
__device__ __forceinline__ void st16(R *p, const R v[16]) {
  st8(p, v);
  st8(p + 8, v + 8);
}

// Cell-centre values the *_ComputeFlux2_TCP loops start from: rho, u = rhou *
// (1/rho) with rhou the conserved momentum as CellGradientsMP's Prim2Cons
// left it (rho * u_prim; at first order the conserved momentum itself), p from
// dv.  On the FP64 path these velocities are the record's slots 5..7, formed
// once per cell with the record (trip_velocity) instead of at every face: two
// divisions and twelve products less per face.  On the mixed path the FP32
// primitive state is used directly.  rc = the cell's record; 1/rho where the
// scheme reads it (HLLC, AUSM+up).
template <typename R, typename A>
__device__ __forceinline__ void cell_values(const RegionDev<R> &g, const A rc[8], A S[5], A &ir) {
  constexpr int u = sizeof(R) == 8 ? 5 : 1;
  if (sizeof(R) == 4 || g.ph.spaceDiscr == 3 || g.ph.spaceDiscr == 5) ir = A(1) / rc[0];
  else ir = A(0);
  S[0] = rc[0];
  S[1] = rc[u];
  S[2] = rc[u + 1];
  S[3] = rc[u + 2];
  S[4] = rc[4];
}
__device__ __forceinline__ void trip_velocity(const Phys &ph, double ir, double r[8]) {
#pragma unroll
  for (int k = 1; k < 4; ++k) r[4 + k] = ph.spaceOrder > 1 ? (r[0] * r[k]) * ir : r[k];
}

template <typename R>
__device__ __forceinline__ void reconstruct(const R G[16], R dx, R dy, R dz, R S[5]) {
#pragma unroll
  for (int v = 0; v < 5; ++v)
    S[v] = S[v] + prod(G[3 * v], dx) + prod(G[3 * v + 1], dy) + prod(G[3 * v + 2], dz);
}

// One face term of RFLU_ComputeLimiterVenkat (modflu/RFLU_ModLimiters.F90:482-504).
// guard = 0 keeps the reference's denom + TINY; guard = 1 adds TINY with the
// sign of denom (for d2 < 0 the reference sum can cancel).
// Mixed path: the quotient is a times the hardware reciprocal of b, within
// 2^-23 + 2^-24 (12.6 M tets, gradient pass: IEEE division 1.838 ms, __fdividef
// 1.814; on the later kernel __fdividef 1.570, this 1.561); the FP64 path keeps
// IEEE division.
#ifndef RF_LIM_FASTDIV
#define RF_LIM_FASTDIV 1
#endif
// The hardware reciprocal: by the PTX manual a relative error of at most 2^-23,
// subnormal operands and results taken as zero.  The limiter's denominators are
// sums with a 1e-12, zero or normal; beyond 2^126 the reciprocal and the term
// are zero, as the programming guide has them for __fdividef.  WENO pass of 1.57
// M tets: __fdividef 0.396 ms, this 0.383.
__device__ __forceinline__ float rcp_ftz(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
template <typename R>
__device__ __forceinline__ R venkat_div(R a, R b) {
  if constexpr (sizeof(R) == 4 && RF_LIM_FASTDIV) return a * rcp_ftz(b);
  else return a / b;
}
// One Venkatakrishnan face term (modflu/RFLU_ModLimiters.F90:482-504): for d2 > 0
// the bound dmax = max - q and +TINY, for d2 < 0 the bound dmin = min - q and
// +TINY (the reference) or -TINY (guard 1, the signed extension); d2 = 0 or
// NaN leaves lim alone.  Written as one path with the bound and the TINY
// selected by the sign, not as two branches: the lanes of a warp whose d2
// differ in sign then run it once (gradient pass 1.803 -> 1.721 ms on the
// 128^3 tet box); every operation and its order is the reference's.
template <typename R>
__device__ __forceinline__ void venkat_term(R d2, R dmax, R dmin, R epsq, R &lim, int guard) {
  const R TINY = R(1.0e-12);
  if (d2 > R(0) || d2 < R(0)) {
    const bool pos = d2 > R(0);
    const R dm = pos ? dmax : dmin;
    R numer = (dm * dm + epsq) * d2 + R(2) * d2 * d2 * dm;
    R denom = d2 * (dm * dm + R(2) * d2 * d2 + dm * d2 + epsq);
    R term = venkat_div(numer, denom + ((pos || !guard) ? TINY : -TINY));
    lim = rmin(term, lim);
  }
}

// ---- kernels ------------------------------------------------------------------

// Bulk prefetch into L2 of the 16-byte-aligned part of [p, p + bytes): one
// instruction per contiguous range, issued by one lane.
__device__ __forceinline__ void prefetch_l1(const void *p) {
  asm volatile("prefetch.global.L1 [%0];" ::"l"(p));
}
__device__ __forceinline__ void prefetch_l2(const void *p, size_t bytes) {
  if (p == nullptr) return;  // an array this region does not hold
  const size_t a = ((size_t)p + 15) & ~(size_t)15, e = ((size_t)p + bytes) & ~(size_t)15;
  if (e > a)
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(a), "r"((unsigned)(e - a))
                 : "memory");
}

// Tile prefetches.  The streamed index and geometry arrays a tile reads
// (SELL slices of stencil members and cell->face lists, face tables, own-cell
// rows) are pulled into L2 in bulk, so the block does not wait on DRAM for
// each index before the gather it feeds can issue: the gradient pass at the
// start of its own tile, the face and update passes one wave of blocks
// ahead.  Lane 0 of each warp issues its 32-cell slice; thread 0 issues the
// per-tile face rows.
template <typename R>
__device__ __forceinline__ void prefetch_grad_slice(const RegionDev<R> &g, int sl, bool faces) {
  if ((threadIdx.x & 31) != 0 || sl * kSlice >= g.nCells) return;
  const long long s0 = g.stOff[sl], s1 = g.stOff[sl + 1];
  prefetch_l2(g.stIdx + s0, (size_t)(s1 - s0) * sizeof(int));
  if (sizeof(R) == 8)
    for (int k = 0; k < 3; ++k) prefetch_l2(g.stW + k * g.stTotal + s0, (size_t)(s1 - s0) * sizeof(R));
  if (faces) {
    const long long f0 = g.cfOff[sl], f1 = g.cfOff[sl + 1];
    const size_t nb = (size_t)(f1 - f0);
    prefetch_l2(g.cfCode + f0, nb * sizeof(int));
    prefetch_l2(g.cfNb + f0, nb * sizeof(int));
    for (int k = 0; k < 3; ++k) prefetch_l2(g.cfD + k * g.cfTotal + f0, nb * sizeof(R));
  }
}

template <typename R>
__device__ __forceinline__ void prefetch_face_tile(const RegionDev<R> &g, int first, int count) {
  if (threadIdx.x != 0) return;
  const int F = g.nFaces;
  if (first >= F) return;
  const size_t n = (size_t)(F - first < count ? F - first : count);
  prefetch_l2(g.f2c + first, n * sizeof(int));
  prefetch_l2(g.f2c + F + first, n * sizeof(int));
  prefetch_l2(g.fnA + 4 * (size_t)first, n * 4 * sizeof(R));
  for (int k = 0; k < 3; ++k) {
    prefetch_l2(g.fdl + (size_t)k * F + first, n * sizeof(R));
    prefetch_l2(g.fdr + (size_t)k * F + first, n * sizeof(R));
  }
}

// The update's per-slice ranges (17 on the mixed path) go out from as many
// lanes at once, lane j taking range j (its pointer picked by selects, so the
// warp runs the prefetch code once instead of once per range on one lane:
// update pass 0.600 -> 0.583 ms at config 2; the gradient and face passes,
// with 6 and 9 ranges, measured faster with one lane).
template <typename R>
__device__ __forceinline__ void prefetch_update_tile(const RegionDev<R> &g, int first) {
  const int N = g.nCells;
  const int j = threadIdx.x & 31;
  const int sl = (first >> 5) + (threadIdx.x >> 5);
  if (sl * kSlice >= N) return;
  const int c0 = sl * kSlice, nc = N - c0 < kSlice ? N - c0 : kSlice;
  // mixed: cvF rows 0-9, rhsSumF 10-14, 1/vol 15; split: cv rows 0-4, rhsSum
  // 5-9, 1/vol 10; FP64: cv rows 0-4; then the slice's cell->face codes
  const bool ff = sizeof(R) == 4 && g.cvF != nullptr;
  const int nrow = ff ? 16 : (sizeof(R) == 4 ? 11 : 5);
  if (j > nrow) return;
  const void *p;
  size_t bytes;
  if (j == nrow) {
    const long long f0 = g.cfOff[sl], f1 = g.cfOff[sl + 1];
    p = g.cfCode + f0;
    bytes = (size_t)(f1 - f0) * sizeof(int);
  } else if (ff) {
    const float *b = j < 10 ? g.cvF + (size_t)j * N : (j < 15 ? g.rhsSumF + (size_t)(j - 10) * N : g.ivolF);
    p = b + c0;
    bytes = (size_t)nc * sizeof(float);
  } else {
    const double *b = j < 5 ? g.cv + (size_t)j * N : (j < 10 ? g.rhsSum + (size_t)(j - 5) * N : g.ivol);
    p = b + c0;
    bytes = (size_t)nc * sizeof(double);
  }
  prefetch_l2(p, bytes);
}

// Calls pf(tile) for the tile a block works on now when it is in the first
// wave, and for the tile `dist` ahead (the one a block of the next wave, or
// this block in its next persistent iteration, will take).
template <typename PF>
__device__ __forceinline__ void prefetch_ahead(int t, int nTiles, int dist, PF pf) {
  if (t < dist) pf(t);
  if (t + dist < nTiles) pf(t + dist);
}

// Programmatic dependent launch.  A kernel of the step is set up while its
// predecessor's last blocks run, and waits, before it touches anything a
// predecessor writes, for the predecessor's completion; a kernel completes
// after its own wait, so the order is transitive.  Returns the block's index
// through the wait, so that every address computed from it (tile, region,
// cell) is known only afterwards; what a kernel reads at fixed addresses (the
// time step's scalars) it reads behind a branch on that index.  So no load can
// move ahead.  Measured, a
// residual of 512 cells 41.6 -> 35.3 us, a step of 10,000 tets 73.8 -> 70.8 us.
// Letting the successor's blocks in earlier (launch_dependents at the start)
// places them on SMs that are still busy: the 4,000-cell FP64 tube's step 131
// -> 147 us.
__device__ __forceinline__ int pdl_wait() {
  int b = blockIdx.x;
  asm volatile("griddepcontrol.wait;" : "+r"(b)::"memory");
  return b;
}

#define RF_TILE_LOOP(first, nTiles) \
  for (int t_ = (first); t_ < (nTiles); t_ += gridDim.x)

// Where a kernel finds its regions: a device table (batches), or, for a single
// region, its descriptor as a kernel parameter.  The descriptor's fields are
// then constant-bank operands instead of loads and of registers that hold
// them, and without a tile list (its tiles are consecutive) the two dependent
// loads of tile and descriptor ahead of a tile's own are gone.  Measured, mixed:
// 12.6 M tets gradient 1.72 -> 1.57 ms (20 bytes of spills gone), faces 0.628
// -> 0.548, WENO pass of 1.57 M tets 0.424 -> 0.396, a step of 10,000 tets 67.7
// -> 61.6 us.  FP64, bound by its pipe, gains 1 to 3%.
template <typename R> struct OneRegion {
  RegionDev<R> r;
  __device__ __forceinline__ const RegionDev<R> &operator[](int) const { return r; }
};
template <typename R>
__device__ __forceinline__ Tile tile_at(const RegionDev<R> *, const Tile *__restrict__ tiles, int t,
                                        int) {
  return tiles[t];
}
template <typename R>
__device__ __forceinline__ Tile tile_at(const OneRegion<R> &, const Tile *__restrict__ tiles, int t,
                                        int stride) {
  return tiles ? tiles[t] : Tile{0, t * stride};
}

// Cons2Prim (modflu/RFLU_ModConvertCv.F90:221-231) of one cell's FP64 state
// into its record, and optionally the EOS first (libflu/RFLU_SetDependentVars.F90:
// 256-287).  FP64 path: every slot of the record is written (trip_velocity).
template <typename R>
__device__ __forceinline__ void set_vars_cell(const RegionDev<R> &g, int c, int computeDv) {
  const int N = g.nCells;
  double q0 = g.cv[c], q1 = g.cv[N + c], q2 = g.cv[2 * N + c], q3 = g.cv[3 * N + c],
         q4 = g.cv[4 * N + c];
  double ir = 1.0 / q0;
  if (computeDv) {
    double gc = g.ph.gvR, gg = g.ph.gvG;
    double Eo = ir * q4;
    double Vm2 = ir * ir * (q1 * q1 + q2 * q2 + q3 * q3);
    double p = (gg - 1.0) * q0 * (Eo - 0.5 * Vm2 - 0.0);
    double T = p / (q0 * gc);
    g.dv[c] = p;
    g.dv[N + c] = T;
    g.dv[2 * N + c] = sqrt(gg * gc * T);
  }
  R r[8];
  if constexpr (sizeof(R) == 4) ld8_rw(g.rec + 8 * (size_t)c, r);
  r[0] = R(q0);
  r[1] = R(ir * q1);
  r[2] = R(ir * q2);
  r[3] = R(ir * q3);
  r[4] = R(g.dv[c]);
  if constexpr (sizeof(R) == 8) trip_velocity(g.ph, ir, r);
  st8(g.rec + 8 * (size_t)c, r);
}

// Mixed path: the record (rho, u, v, w, p) of a cell from its float-float
// conserved state, in FP32 (the total energy keeps its low part, so p loses
// only the kinetic term's rounding).  The one state-to-record map of the mixed
// path: the update, the upload and the border receive all use it.
__device__ __forceinline__ void record_from_pairs(const Phys &ph, const float qh[5],
                                                  const float ql[5], float r[5]) {
  const float rf = qh[0];
  const float irf = 1.0f / rf;
  r[0] = rf;
  r[1] = qh[1] * irf;
  r[2] = qh[2] * irf;
  r[3] = qh[3] * irf;
  const float kin = 0.5f * (qh[1] * qh[1] + qh[2] * qh[2] + qh[3] * qh[3]) * irf;
  r[4] = (ph.gvGF - 1.0f) * ((qh[4] - kin) + ql[4]);
}

// Pressure of RFLU_SetDependentVars (libflu/RFLU_SetDependentVars.F90:256-287,
// libfloflu/MixtPerf_P.F90:78) from an FP64 conserved vector, in the
// reference's operation order; ir = 1/rho is returned for the velocities.
__device__ __forceinline__ double eos_p(const Phys &ph, const double q[5], double &ir) {
  const double rr = q[0];
  ir = 1.0 / rr;
  const double Eo = ir * q[4];
  const double Vm2 = ir * ir * (q[1] * q[1] + q[2] * q[2] + q[3] * q[3]);
  return (ph.gvG - 1.0) * rr * (Eo - 0.5 * Vm2 - 0.0);
}

// The float nearest to a double (ties to even) assembled with integer
// operations: the conversion instruction runs on the FP64 pipe.  Magnitudes
// outside FP32's normal range, zeros among them, take the instruction.
__device__ __forceinline__ float nearest_f32(double x) {
  const unsigned h = (unsigned)__double2hiint(x), l = (unsigned)__double2loint(x);
  const unsigned t = (h & 0x7fffffffu) - (896u << 20);
  if (t - 0x00100000u >= 0x0fd00000u) return (float)x;  // exponents 897 .. 1149
  unsigned m = __funnelshift_l(l, t, 3);
  const unsigned rest = l << 3;
  m += (rest > 0x80000000u || (rest == 0x80000000u && (m & 1u))) ? 1u : 0u;
  return __uint_as_float((h & 0x80000000u) | m);
}
__device__ __forceinline__ bool finite_bits(double x) {
  return ((unsigned)__double2hiint(x) & 0x7ff00000u) != 0x7ff00000u;
}
// 0 < x < infinity and x normal, from the bits
__device__ __forceinline__ bool positive_bits(double x) {
  return (unsigned)__double2hiint(x) - 0x00100000u < 0x7fe00000u;
}

// Split path: the FP32 record of a cell from its FP64 conserved state and
// FP64 pressure (velocities u = (1/rho) rhou as Cons2Prim forms them).
__device__ __forceinline__ void record_from_fp64(const double q[5], double ir, double p,
                                                 float r[8]) {
  r[0] = nearest_f32(q[0]);
  r[1] = nearest_f32(ir * q[1]);
  r[2] = nearest_f32(ir * q[2]);
  r[3] = nearest_f32(ir * q[3]);
  r[4] = nearest_f32(p);
}

// Mixed path: a cell's state from an FP64 conserved vector (upload, border
// receive): float-float split, then the record from the pairs, with p from dv
// when given.  FP64 work is the split alone (GB300's FP64 rate bounds these
// conversions).  Split path (no pairs): the FP64 rows, and the record from
// the FP64 EOS (p from dv when given).
__device__ __forceinline__ void state_from_fp64_split(const RegionDev<float> &g, int c,
                                                      const double q[5], const double *pGiven) {
  const int N = g.nCells;
#pragma unroll
  for (int j = 0; j < 5; ++j) g.cv[(size_t)j * N + c] = q[j];
  double ir;
  const double p = eos_p(g.ph, q, ir);
  float r[8];
  ld8_rw(g.rec + 8 * (size_t)c, r);
  record_from_fp64(q, ir, pGiven ? *pGiven : p, r);
  st8(g.rec + 8 * (size_t)c, r);
}
__device__ __forceinline__ void state_from_fp64_ff(const RegionDev<float> &g, int c,
                                                   const double q[5], const double *pGiven) {
  const int N = g.nCells;
  float qh[5], ql[5];
#pragma unroll
  for (int j = 0; j < 5; ++j) {
    qh[j] = (float)q[j];
    ql[j] = (float)(q[j] - (double)qh[j]);
    g.cvF[(size_t)j * N + c] = qh[j];
    g.cvF[(size_t)(5 + j) * N + c] = ql[j];
  }
  float r[8];
  ld8_rw(g.rec + 8 * (size_t)c, r);
  record_from_pairs(g.ph, qh, ql, r);
  if (pGiven) r[4] = float(*pGiven);
  st8(g.rec + 8 * (size_t)c, r);
}
__device__ __forceinline__ void state_from_fp64(const RegionDev<float> &g, int c, const double q[5],
                                                const double *pGiven) {
  if (g.cvF)
    state_from_fp64_ff(g, c, q, pGiven);
  else
    state_from_fp64_split(g, c, q, pGiven);
}

// The double of a float (IEEE widening, always exact) assembled from its bit
// fields with integer operations: the download join is FP64-pipe bound on
// GB300, and this keeps the conversion off that pipe.  Zeros are assembled
// too; subnormals, infinities and NaNs take the conversion instruction.
__device__ __forceinline__ double widen_f32(float f) {
  const unsigned u = __float_as_uint(f);
  const unsigned e = (u >> 23) & 0xffu, m = u & 0x7fffffu;
  if (e == 0xffu || (e == 0u && m != 0u)) return (double)f;
  const unsigned long long s = (unsigned long long)(u & 0x80000000u) << 32;
  // exponent bias 127 -> 1023 (+896), 23 -> 52 fraction bits (<< 29)
  const unsigned long long b =
      e ? (s | ((unsigned long long)(e + 896u) << 52) | ((unsigned long long)m << 29)) : s;
  return __longlong_as_double((long long)b);
}

__device__ __forceinline__ double as_fp64(float f) { return widen_f32(f); }
__device__ __forceinline__ double as_fp64(double x) { return x; }
// Conserved state of a cell as FP64 (the float-float pair joined on the
// mixed path).
template <typename R>
__device__ __forceinline__ void cons_fp64(const RegionDev<R> &g, int c, double q[5]) {
  const int N = g.nCells;
  if (sizeof(R) == 4 && g.cvF) {
#pragma unroll
    for (int j = 0; j < 5; ++j)
      q[j] = (double)g.cvF[(size_t)j * N + c] + (double)g.cvF[(size_t)(5 + j) * N + c];
  } else {
#pragma unroll
    for (int j = 0; j < 5; ++j) q[j] = g.cv[(size_t)j * N + c];
  }
}

// Uploaded state -> records (and dv).
template <typename R>
__global__ void k_prim(const RegionDev<R> *__restrict__ regs, const Tile *__restrict__ tiles,
                       int nTiles, int computeDv) {
  RF_TILE_LOOP(blockIdx.x, nTiles) {
    const Tile tl = tiles[t_];
    const RegionDev<R> &g = regs[tl.region];
    const int c = tl.first + threadIdx.x;
    if (c >= g.nCells) continue;
    set_vars_cell(g, c, computeDv);
  }
}

// ---- halo exchange ---------------------------------------------------------------
// One received virtual cell: RFLU_MPI_CopyCellData (modflu/RFLU_ModMPI.F90:
// 332-390) of cv, then RFLU_SetVarsContWrapper of the cell
// (libfloflu/RungeKuttaMP.F90:381-396): FP64 path, dv and the record rebuilt
// from the copied cv with the EOS every cell uses; mixed path, the
// float-float pair and the sender's record slots copied (the record is a
// function of the pair and of the gas constants, which coupled regions share).
// The source cell's state is read through L2 (__ldcg): in a persistent stage
// launch other blocks updated it earlier in the same kernel.
template <typename R>
__device__ __forceinline__ void halo_cell(const RegionDev<R> &gs, int cs, const RegionDev<R> &gd,
                                          int cd) {
  const int Ns = gs.nCells, Nd = gd.nCells;
  if constexpr (sizeof(R) == 8) {
#pragma unroll
    for (int j = 0; j < 5; ++j) gd.cv[(size_t)j * Nd + cd] = __ldcg(gs.cv + (size_t)j * Ns + cs);
    set_vars_cell(gd, cd, 1);
  } else {
    if (gd.cvF) {
#pragma unroll
      for (int j = 0; j < 10; ++j) gd.cvF[(size_t)j * Nd + cd] = __ldcg(gs.cvF + (size_t)j * Ns + cs);
    } else {  // split path: the FP64 rows
#pragma unroll
      for (int j = 0; j < 5; ++j) gd.cv[(size_t)j * Nd + cd] = __ldcg(gs.cv + (size_t)j * Ns + cs);
    }
    R a[8], b[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) a[k] = __ldcg(gs.rec + 8 * (size_t)cs + k);
    ld8_rw(gd.rec + 8 * (size_t)cd, b);
#pragma unroll
    for (int k = 0; k < 5; ++k) b[k] = a[k];
    st8(gd.rec + 8 * (size_t)cd, b);
  }
}

template <typename R>
__global__ void k_halo(const RegionDev<R> *__restrict__ regs, const HaloLink *__restrict__ links,
                       int n) {
  const int i = pdl_wait() * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const HaloLink l = links[i];
  halo_cell(regs[l.srcRegion], l.srcCell, regs[l.dstRegion], l.dstCell);
}

template <typename R>
__global__ void k_halo_pair(const RegionDev<R> *__restrict__ src, const RegionDev<R> *__restrict__ dst,
                            const int *__restrict__ srcCells, const int *__restrict__ dstCells,
                            int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  halo_cell(*src, srcCells[i], *dst, dstCells[i]);
}

// sendBuff(5,n) = cv(:,cells) (RFLU_MPI_ISendWrapper's packing)
template <typename R>
__global__ void k_border_pack(const RegionDev<R> *__restrict__ gp, const int *__restrict__ cells,
                              int n, double *__restrict__ buf) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double q[5];
  cons_fp64(*gp, cells[i], q);
#pragma unroll
  for (int j = 0; j < 5; ++j) buf[5 * (size_t)i + j] = q[j];
}

// cv(:,cells) = recvBuff(5,n), then the cells' dv and records
// (RFLU_MPI_RecvWrapper + RFLU_SetVarsContWrapper(nCells+1,nCellsTot))
template <typename R>
__global__ void k_border_unpack(const RegionDev<R> *__restrict__ gp, const int *__restrict__ cells,
                                int n, const double *__restrict__ buf) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const RegionDev<R> &g = *gp;
  const int c = cells[i];
  double q[5];
#pragma unroll
  for (int j = 0; j < 5; ++j) q[j] = buf[5 * (size_t)i + j];
  if constexpr (sizeof(R) == 8) {
#pragma unroll
    for (int j = 0; j < 5; ++j) g.cv[(size_t)j * g.nCells + c] = q[j];
    set_vars_cell(g, c, 1);
  } else {
    state_from_fp64(g, c, q, nullptr);
  }
}

// WLSQ gradients of (rho,u,v,w,p) (RFLU_ComputeGradCellsFast_3D,
// modflu/RFLU_ModDifferentiationCells.F90:1021-1149) fused with the
// Venkatakrishnan limiter and RFLU_LimitGradCells (modflu/RFLU_ModLimiters.F90:
// 339-532, 707-760).  One thread per cell; stencil members in stored order
// (the reference's summation order).  The limiter of a cell needs only its own
// unlimited gradient and its face neighbours' values, and min/max and the MIN
// over faces do not depend on the face order, so the per-cell gather equals
// the reference's two face loops.  FP64 path: precomputed weights (bitwise the
// reference's); mixed path: weights rebuilt in FP32 from the records'
// centroids and the cell's WLSQ factor terms.
template <typename R>
__device__ __forceinline__ void dt_block_min(unsigned long long bits, unsigned long long *smin,
                                             unsigned long long *dst) {
  for (int o = 16; o > 0; o >>= 1) {
    unsigned long long x = __shfl_down_sync(0xffffffffu, bits, o);
    bits = x < bits ? x : bits;
  }
  if ((threadIdx.x & 31) == 0) smin[threadIdx.x >> 5] = bits;
  __syncthreads();
  if (threadIdx.x < 32) {
    unsigned long long v = threadIdx.x < (blockDim.x >> 5) ? smin[threadIdx.x] : 0x7FF0000000000000ull;
    for (int o = 16; o > 0; o >>= 1) {
      unsigned long long x = __shfl_down_sync(0xffffffffu, v, o);
      v = x < v ? x : v;
    }
    if (threadIdx.x == 0) atomicMin(dst, v);
  }
  __syncthreads();
}

// The per-face terms of cell_dt, shared with the gradient pass that folds the
// time step into its limiter face loop.
template <typename R>
__device__ __forceinline__ R dt_sound(const RegionDev<R> &g, int c, const R r[8]) {
  const R gg = PC<R>{g.ph}.gvG();
  return sizeof(R) == 8 ? R(g.dv[2 * g.nCells + c]) : R(sqrtf(float(gg * r[4] / r[0])));
}
template <typename R>
__device__ __forceinline__ void dt_interior_term(const RegionDev<R> &g, int code, const R r0[8],
                                                 R a0, int nb, const R rn[8], R &acc) {
  R nrm[4];
  ld4(g.fnA + 4 * (size_t)(code >> 1), nrm);
  const R an = dt_sound(g, nb, rn);
  // the face's c1 values first, as in the reference
  const bool first = (code & 1) == 0;
  const R u1 = first ? r0[1] : rn[1], u2 = first ? rn[1] : r0[1];
  const R v1 = first ? r0[2] : rn[2], v2 = first ? rn[2] : r0[2];
  const R w1 = first ? r0[3] : rn[3], w2 = first ? rn[3] : r0[3];
  const R a1 = first ? a0 : an, a2 = first ? an : a0;
  R vc = R(0.5) * ((u1 + u2) * nrm[0] + (v1 + v2) * nrm[1] + (w1 + w2) * nrm[2]);
  R as = R(0.5) * (a1 + a2);
  acc = acc + (fabs(vc - R(0)) + as) * nrm[3];
}
template <typename R>
__device__ __forceinline__ void dt_boundary_term(const RegionDev<R> &g, int code, const R r0[8],
                                                 R a0, R &acc) {
  R nrm[4];
  ld4(g.bfnA + 4 * (size_t)(-code - 1), nrm);
  R vc = r0[1] * nrm[0] + r0[2] * nrm[1] + r0[3] * nrm[2];
  acc = acc + (fabs(vc - R(0)) + a0) * nrm[3];
}
template <typename R>
__device__ __forceinline__ double dt_of(const RegionDev<R> &g, int c, R acc) {
  return sizeof(R) == 8 ? double(R(g.vol[c]) / acc) : double(float(g.vol[c]) / float(acc));
}

// Local time-step sum of RFLU_TimeStepInviscid (rocflu/RFLU_TimeStepInviscid.F90:
// 165-297) for one cell, as a gather over its faces in the reference order:
// sum of (|v_n| + a) * area with face-averaged velocity and sound speed
// (interior faces) or the cell's own (boundary faces).  u = rhou*(1/rho) is
// the record's velocity; a is dv(SOUN) on the FP64 path and sqrt(g p/rho) in
// FP32 on the mixed path.  Returns dt(c) = vol / sum.
template <typename R>
__device__ __forceinline__ double cell_dt(const RegionDev<R> &g, int c, const R r0[8]) {
  const R a0 = dt_sound(g, c, r0);
  R acc = R(0);
  const long long e0 = g.cfOff[c >> 5] + (c & 31);
  const int n = g.cfCnt[c];
  for (int k = 0; k < n; ++k) {
    const long long e = e0 + (long long)k * kSlice;
    const int code = g.cfCode[e];
    if (code >= 0) {
      const int nb = g.cfNb[e];
      R rn[8];
      ld8(g.rec + 8 * (size_t)nb, rn);
      dt_interior_term(g, code, r0, a0, nb, rn, acc);
    } else {
      dt_boundary_term(g, code, r0, a0, acc);
    }
  }
  return dt_of(g, c, acc);
}

// WLSQ gradients of (rho,u,v,w,p) (RFLU_ComputeGradCellsFast_3D,
// modflu/RFLU_ModDifferentiationCells.F90:1021-1149) fused with the
// Venkatakrishnan limiter and RFLU_LimitGradCells (modflu/RFLU_ModLimiters.F90:
// 339-532, 707-760).  One thread per cell; stencil members in stored order
// (the reference's summation order); the stencil indices are read from the
// SELL slice (coalesced across the warp) and the record gathers of
// consecutive members are issued together.  The limiter of a cell needs only its
// own unlimited gradient and its face neighbours' values, and min/max and the
// MIN over faces do not depend on the face order, so the per-cell gather
// equals the reference's two face loops.  FP64 path: precomputed weights
// (bitwise the reference's); mixed path: weights rebuilt in FP32 from the
// records' centroids and the cell's WLSQ factor terms.  With fuseDt the pass
// also reduces the time step (stage 1 of a step).
// Record gathers issued together in the mixed member loop (software-pipelined
// with the next group's index loads).  Measured on the 128^3 tet box: 4 ->
// 1.923 ms, 6 -> 1.893, 7 -> 1.897, 8 -> 1.880, 10 -> 2.033 (spills), 12 ->
// 2.052; without the index pipeline 8 -> 1.904, 12 -> 1.929.
// Limiter face loop: codes and neighbours of the first RF_LIM_PRE faces loaded
// ahead of the records (measured: gradient pass 1.881 -> 1.835 ms with 4,
// 1.830 ms with 6; keeping the six codes live for the second face loop instead
// of reading them again: 1.981 ms).
#ifndef RF_LIM_PRE
#define RF_LIM_PRE 6
#endif
#ifndef RF_GRAD_UNROLL
#define RF_GRAD_UNROLL 8
#endif
// Resident 128-thread blocks per SM requested for the gradient pass (mixed
// path).  Measured on the 128^3 tet box with the loop above: 7 -> 1.878 ms
// (72 registers), 8 -> 1.830 ms (64), 9 -> 2.075 ms (56, spills).
#ifndef RF_GRAD_MINB
#define RF_GRAD_MINB 8
#endif
#ifndef RF_GRAD_MINB_DT
#define RF_GRAD_MINB_DT 8  // the same for the stage-1 pass that also reduces the time step
#endif
// ---- FP64 gradient pass ------------------------------------------------------------
// Bound by the FP64 pipe (one warp operation per 64 cycles and SM quarter), so
// the pass keeps off it what has an exact equivalent elsewhere: the products
// of the member sum and of the limiter's d2 are integer products (soft_mul,
// the same bits), the min / max comparisons run on the bit patterns, and the
// limiter's quotients are first formed in FP32 to find the face that decides
// each variable's minimum, whose quotient alone is then formed in FP64.
// FP64 operations per tet cell with 40 members: about 975 against 2440.

// b < a for numbers that are neither infinite nor NaN.  (-0 counts as below
// +0; a zero's sign never reaches the limiter's result.)
__device__ __forceinline__ bool lt_bits(double b, double a) {
  long long kb = __double_as_longlong(b), ka = __double_as_longlong(a);
  kb ^= (kb >> 63) & 0x7fffffffffffffffll;
  ka ^= (ka >> 63) & 0x7fffffffffffffffll;
  return kb < ka;
}
// FP32 value of a double of magnitude in [2^-100, 2^40) (truncated); other
// values, zero apart, clear ok.
__device__ __forceinline__ float narrow_bits(double x, bool &ok) {
  const unsigned h = (unsigned)__double2hiint(x), l = (unsigned)__double2loint(x);
  const unsigned t = h & 0x7fffffffu;
  if ((t | l) == 0u) return 0.f;
  ok = ok && t - (923u << 20) < (140u << 20);
  return __uint_as_float((h & 0x80000000u) | __funnelshift_l(l, t - (896u << 20), 3));
}

// Screening of one variable's Venkatakrishnan terms.  In FP32 a term's
// numerator and denominator are sums of terms of one sign (d2 and its bound dm
// have the same sign), so its relative error stays below 3e-6 when nothing
// leaves FP32's normal range, the quotient included (at an extremum, dm = 0, it
// is epsq / 2 d2^2); two terms further apart than 1e-5 are then
// ordered as in FP64, and only the smallest one decides the limiter.  What the
// screen cannot order - two different d2 within 1e-5, magnitudes outside the
// ranges below, the reference's cancelling guard - is left to the FP64 loop.
struct VenkatScreen {
  float best, second;
  double d2;  // of the smallest term
};
__device__ __forceinline__ void venkat_screen(VenkatScreen &s, double d2, float mx, float mn,
                                              float e, int guard, bool &ok) {
  const float x = narrow_bits(d2, ok);
  if (soft_zero(d2)) return;  // the reference skips d2 = 0
  const bool pos = x > 0.f;
  const float m = pos ? mx : mn;
  const float a = fmaf(m, m, e), xm = x * m;
  const float num = x * fmaf(2.f, xm, a);
  const float den0 = x * (fmaf(2.f * x, x, a) + xm), mag = fabsf(den0);
  ok = ok && mag > 1e-30f && mag < 1e30f && (pos || guard || mag > 1e-6f);
  const float t = __fdividef(num, den0 + ((pos || !guard) ? 1e-12f : -1e-12f));
  ok = ok && t > 1e-36f;
  if (__double_as_longlong(d2) != __double_as_longlong(s.d2)) {  // an equal d2 has an equal term
    s.second = fminf(s.second, fmaxf(s.best, t));
    if (t < s.best) {
      s.best = t;
      s.d2 = d2;
    }
  }
}

// One variable v of one cell of the FP64 gradient pass.  Every sum and rounding
// is the reference's, in its order.  Returns the cell's local time step bits
// (FUSE_DT, first variable only).  RF_G64_U members' loads are issued ahead of
// their sums (64^3 tet box: 1 -> 3.26 ms, 2 -> 3.24, 4 -> 3.34).
#ifndef RF_G64_U
#define RF_G64_U 2
#endif
template <int FUSE_DT>
__device__ __forceinline__ unsigned long long grad_cell64(const RegionDev<double> &g, int c,
                                                          int v) {
  const double *__restrict__ rec = g.rec + v;
  const bool withDt = FUSE_DT && v == 0;
  unsigned long long dtbits = 0x7FF0000000000000ull;
  const double r0 = rec[8 * (size_t)c];
  const long long e0 = g.cfOff[c >> 5] + (c & 31);
  const int nf = g.cfCnt[c];
  double acc[3] = {0.0, 0.0, 0.0};
  {
    constexpr int U = RF_G64_U;
    const int n = g.stCnt[c];
    const long long base = g.stOff[c >> 5] + (c & 31), T = g.stTotal;
    const int *__restrict__ sidx = g.stIdx + base;
    const double *__restrict__ w0 = g.stW + base;
    auto member = [&](double q, const double w[3]) {
      q = q - r0;
      if (soft_ok(q) && soft_ok(w[0]) && soft_ok(w[1]) && soft_ok(w[2])) {
        const SoftB b = soft_b(q);
#pragma unroll
        for (int d = 0; d < 3; ++d) acc[d] = acc[d] + soft_mul(soft_a(w[d]), b);
      } else {
#pragma unroll
        for (int d = 0; d < 3; ++d) acc[d] = acc[d] + w[d] * q;
      }
    };
    int nx[U];
#pragma unroll
    for (int u = 0; u < U; ++u) nx[u] = u < n ? sidx[u * kSlice] : 0;
    for (int k = 0; k < n; k += U) {
      double q[U], w[U][3];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        q[u] = rec[8 * (size_t)nx[u]];
        const int kk = k + u < n ? k + u : k;
#pragma unroll
        for (int d = 0; d < 3; ++d) w[u][d] = w0[d * T + kk * kSlice];
      }
#pragma unroll
      for (int u = 0; u < U; ++u) nx[u] = k + U + u < n ? sidx[(k + U + u) * kSlice] : 0;
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (u == 0 || k + u < n) member(q[u], w[u]);
    }
  }
  if (g.ph.reconst == 11) {
    double vmin = r0, vmax = r0;
    const long long T = g.cfTotal;
    double dtacc = 0.0, a0 = 0.0, rc[8];
    if (withDt) {
      ld8(g.rec + 8 * (size_t)c, rc);
      a0 = dt_sound(g, c, rc);
    }
    const bool fin0 = finite_bits(r0);
    for (int k = 0; k < nf; ++k) {
      const long long ee = e0 + (long long)k * kSlice;
      const int code = g.cfCode[ee];
      if (code < 0) {
        if (withDt) dt_boundary_term(g, code, rc, a0, dtacc);
        continue;
      }
      const int nb = g.cfNb[ee];
      const double q = rec[8 * (size_t)nb];
      if (fin0 && finite_bits(q)) {
        if (lt_bits(q, vmin)) vmin = q;
        if (lt_bits(vmax, q)) vmax = q;
      } else {
        vmin = rmin(vmin, q);
        vmax = rmax(vmax, q);
      }
      if (withDt) {
        double rn[8];
        ld8(g.rec + 8 * (size_t)nb, rn);
        dt_interior_term(g, code, rc, a0, nb, rn, dtacc);
      }
    }
    if (withDt) {
      dtbits = (unsigned long long)__double_as_longlong(dt_of(g, c, dtacc));
      if (c >= g.nAct) dtbits = 0x7FF0000000000000ull;  // actual cells only
    }
    const double epsq = g.epsq[c];
    const int guard = g.ph.venkatGuard;
    vmax = vmax - r0;  // the bounds dmax, dmin
    vmin = vmin - r0;
    bool ok = epsq > 1e-25 && epsq < 1e12;
    const float ef = ok ? (float)epsq : 1.f;
    const float mx = narrow_bits(vmax, ok), mn = narrow_bits(vmin, ok);
    ok = ok && soft_ok(acc[0]) && soft_ok(acc[1]) && soft_ok(acc[2]);
    const SoftB bx = soft_b(acc[0]), by = soft_b(acc[1]), bz = soft_b(acc[2]);
    VenkatScreen sc = {3.0e38f, 3.0e38f, 0.0};
    for (int k = 0; k < nf; ++k) {
      const long long ee = e0 + (long long)k * kSlice;
      if (g.cfCode[ee] < 0) continue;
      const double dx = g.cfD[ee], dy = g.cfD[T + ee], dz = g.cfD[2 * T + ee];
      ok = ok && soft_ok(dx) && soft_ok(dy) && soft_ok(dz);
      if (ok) {
        const double d2 =
            soft_mul(soft_a(dx), bx) + soft_mul(soft_a(dy), by) + soft_mul(soft_a(dz), bz);
        venkat_screen(sc, d2, mx, mn, ef, guard, ok);
      }
    }
    double lim = 1.0;
    const float near = 1.00001f;
    if (ok && !(sc.best <= near && sc.second <= sc.best * near)) {
      if (sc.best <= near) venkat_term(sc.d2, vmax, vmin, epsq, lim, guard);
    } else {
      for (int k = 0; k < nf; ++k) {
        const long long ee = e0 + (long long)k * kSlice;
        if (g.cfCode[ee] < 0) continue;
        const double d2 = acc[0] * g.cfD[ee] + acc[1] * g.cfD[T + ee] + acc[2] * g.cfD[2 * T + ee];
        venkat_term(d2, vmax, vmin, epsq, lim, guard);
      }
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) acc[d] = lim * acc[d];
  }
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    if (!g.gradRaw) {
      g.grad[16 * (size_t)c + 3 * v + d] = acc[d];
    } else {
      // RECONST 2: the WENO weight of each component and its product, as
      // RFLU_WENOGradCellsXYZFast_3D forms them (same operations), once per
      // cell instead of once per stencil visit
      const double w = 1.0 / (acc[d] * acc[d] + 1.0E-15);
      g.gradRaw[32 * (size_t)c + 3 * v + d] = w;
      g.gradRaw[32 * (size_t)c + 16 + 3 * v + d] = w * acc[d];
    }
  }
  if (withDt && g.ph.reconst != 11) {  // no limiter face loop to ride on
    double rc[8];
    ld8(g.rec + 8 * (size_t)c, rc);
    dtbits = (unsigned long long)__double_as_longlong(cell_dt(g, c, rc));
    if (c >= g.nAct) dtbits = 0x7FF0000000000000ull;
  }
  return dtbits;
}

// BS threads per block (one cell each, a tile of BS cells); the requested
// residency keeps the same number of resident threads per SM for every BS.
// One tile of the gradient pass (every thread of the block, one cell each).
template <typename R, int FUSE_DT, typename RT>
__device__ __forceinline__ void grad_tile(const RT &regs, const Tile *__restrict__ tiles, int t_,
                                          unsigned long long *smin) {
  constexpr bool fuseDt = FUSE_DT != 0;
  {
    const Tile tl = tile_at(regs, tiles, t_, blockDim.x);
    const RegionDev<R> &g = regs[tl.region];
    const int c = tl.first + threadIdx.x;
    const int N = g.nCells;
    const bool valid = c < N;
    // own tile only: prefetching a wave ahead measured slower here (the
    // prefetched slices push the neighbour records the gathers reuse out of L2)
    prefetch_grad_slice(g, (tl.first >> 5) + (threadIdx.x >> 5), fuseDt || g.ph.reconst == 11);
    const long long base = valid ? g.stOff[c >> 5] + (c & 31) : 0;
    const int *__restrict__ sidx = g.stIdx + base;
    unsigned long long dtbits = 0x7FF0000000000000ull;
    if (valid) {
      const R *__restrict__ rec = g.rec;
      R r0[8];
      ld8(rec + 8 * (size_t)c, r0);
      R acc[15];
#pragma unroll
      for (int k = 0; k < 15; ++k) acc[k] = R(0);
      const int n = g.stCnt[c];
      {
        // The reference's weight of member m is w = A d/|d|^2 with d the
        // centroid offset and A the cell's symmetric inverse-moment matrix
        // built from its WLSQ factor (c11^2 + c12^2 c22^2 + c13^2 c33^2, ...).
        // A is the same for every member, so the member loop accumulates
        // S_v = sum (q_v,m - q_v,0) d/|d|^2 and the gradient is A S_v: the
        // reference's sum reassociated, about a quarter fewer operations per
        // member.
        auto member = [&](const R rn[8]) {
          R dx = rn[5] - r0[5], dy = rn[6] - r0[6], dz = rn[7] - r0[7];
          R t = rsqrtf(float(dx * dx + dy * dy + dz * dz));
          t = t * t;
          dx = t * dx;
          dy = t * dy;
          dz = t * dz;
#pragma unroll
          for (int v = 0; v < 5; ++v) {
            R dVar = rn[v] - r0[v];
            acc[3 * v] = acc[3 * v] + dx * dVar;
            acc[3 * v + 1] = acc[3 * v + 1] + dy * dVar;
            acc[3 * v + 2] = acc[3 * v + 2] + dz * dVar;
          }
        };
        // software pipeline: the next group's stencil indices are loaded while
        // this group's records are in flight (same members, same order)
        constexpr int U = RF_GRAD_UNROLL;
        const int nFull = n - n % U;
        int nx[U];
#pragma unroll
        for (int u = 0; u < U; ++u) nx[u] = u < n ? ld_index(sidx + u * kSlice) : 0;
        for (int k = 0; k < nFull; k += U) {
          R ra[U][8];
#pragma unroll
          for (int u = 0; u < U; ++u) ld8(rec + 8 * (size_t)nx[u], ra[u]);
#pragma unroll
          for (int u = 0; u < U; ++u)
            nx[u] = k + U + u < n ? ld_index(sidx + (k + U + u) * kSlice) : 0;
#pragma unroll
          for (int u = 0; u < U; ++u) member(ra[u]);
        }
#pragma unroll
        for (int u = 0; u < U - 1; ++u) {
          if (nFull + u < n) {
            R ra[8];
            ld8(rec + 8 * (size_t)nx[u], ra);
            member(ra);
          }
        }
        const R axx = lds<RF_HINT_G>(g.cwt + c), axy = lds<RF_HINT_G>(g.cwt + N + c),
                axz = lds<RF_HINT_G>(g.cwt + 2 * N + c);
        const R ayy = lds<RF_HINT_G>(g.cwt + 3 * N + c), ayz = lds<RF_HINT_G>(g.cwt + 4 * N + c),
                azz = lds<RF_HINT_G>(g.cwt + 5 * N + c);
#pragma unroll
        for (int v = 0; v < 5; ++v) {
          const R sx = acc[3 * v], sy = acc[3 * v + 1], sz = acc[3 * v + 2];
          acc[3 * v] = axx * sx + axy * sy + axz * sz;
          acc[3 * v + 1] = axy * sx + ayy * sy + ayz * sz;
          acc[3 * v + 2] = axz * sx + ayz * sy + azz * sz;
        }
      }
      if (g.ph.reconst == 11) {
        R vmin[5], vmax[5], lim[5];
#pragma unroll
        for (int v = 0; v < 5; ++v) {
          vmin[v] = r0[v];
          vmax[v] = r0[v];
          lim[v] = R(1);
        }
        const long long T = g.cfTotal;
        const long long e0 = g.cfOff[c >> 5] + (c & 31);
        const int nf = g.cfCnt[c];
        // stage 1: the time-step sum rides on this face loop (same faces, same
        // order and arithmetic as cell_dt)
        R dtacc = R(0), a0 = R(0);
        if constexpr (fuseDt) a0 = dt_sound(g, c, r0);
        auto face_minmax = [&](int code, int nb) {
          if (code < 0) {
            if constexpr (fuseDt) dt_boundary_term(g, code, r0, a0, dtacc);
            return;
          }
          R rn[8];
          ld8(rec + 8 * (size_t)nb, rn);
#pragma unroll
          for (int v = 0; v < 5; ++v) {
            vmin[v] = rmin(vmin[v], rn[v]);
            vmax[v] = rmax(vmax[v], rn[v]);
          }
          if constexpr (fuseDt) dt_interior_term(g, code, r0, a0, nb, rn, dtacc);
        };
        // the first faces' codes and neighbours are loaded together, ahead of
        // their records (same faces, same order); six covers every cell type
        constexpr int MF = RF_LIM_PRE;
        int cc[MF], nn[MF];
#pragma unroll
        for (int k = 0; k < MF; ++k) {
          const long long ee = e0 + (long long)k * kSlice;
          cc[k] = k < nf ? g.cfCode[ee] : -1;
          nn[k] = k < nf ? lds<RF_HINT_G>(g.cfNb + ee) : -1;
        }
#pragma unroll
        for (int k = 0; k < MF; ++k)
          if (k < nf) face_minmax(cc[k], nn[k]);
        for (int k = MF; k < nf; ++k) {
          const long long ee = e0 + (long long)k * kSlice;
          const int code = g.cfCode[ee];
          face_minmax(code, code < 0 ? -1 : lds<RF_HINT_G>(g.cfNb + ee));
        }
        if constexpr (fuseDt) {
          dtbits = (unsigned long long)__double_as_longlong(dt_of(g, c, dtacc));
          if (c >= g.nAct) dtbits = 0x7FF0000000000000ull;  // actual cells only
        }
        const R epsq = lds<RF_HINT_G>(g.epsq + c);
        const int guard = g.ph.venkatGuard;
        auto face_lim = [&](long long ee) {
          const R dx = lds<RF_HINT_G>(g.cfD + ee), dy = lds<RF_HINT_G>(g.cfD + T + ee),
                  dz = lds<RF_HINT_G>(g.cfD + 2 * T + ee);
#pragma unroll
          for (int v = 0; v < 5; ++v) {
            R d2 = acc[3 * v] * dx + acc[3 * v + 1] * dy + acc[3 * v + 2] * dz;
            venkat_term(d2, vmax[v] - r0[v], vmin[v] - r0[v], epsq, lim[v], guard);
          }
        };
        for (int k = 0; k < nf; ++k) {
          const long long ee = e0 + (long long)k * kSlice;
          if (lds<RF_HINT_G>(g.cfCode + ee) >= 0) face_lim(ee);  // its last read
        }
#pragma unroll
        for (int v = 0; v < 5; ++v)
#pragma unroll
          for (int d = 0; d < 3; ++d) acc[3 * v + d] = lim[v] * acc[3 * v + d];
      }
      R out[16];
#pragma unroll
      for (int k = 0; k < 15; ++k) out[k] = acc[k];
      out[15] = R(0);
      if (!g.gradRaw) {
        st16(g.grad + 16 * (size_t)c, out);
      } else {
        st16(g.gradRaw + 16 * (size_t)c, out);  // RECONST 2, mixed: weighted next
      }
      if constexpr (fuseDt) {
        if (g.ph.reconst != 11) {  // no limiter face loop to ride on
          dtbits = (unsigned long long)__double_as_longlong(cell_dt(g, c, r0));
          if (c >= g.nAct) dtbits = 0x7FF0000000000000ull;
        }
      }
    }
    if constexpr (fuseDt) dt_block_min<R>(dtbits, smin, g.dtBits);
  }
}

// FP64: one warp per 32 cells and variable, so that a region of a few thousand
// cells reaches every SM quarter's FP64 unit and a large one needs 64 registers
// a thread instead of 128.  Measured (pass with its launch): 512 cells 48.8 ->
// 22.8 us, 4,000 cells 49.0 -> 22.9, 64,000 cells 98 -> 66, 1.57 M cells 6.08
// -> 3.24 ms, about 975 FP64 operations per cell at 0.51 T/s (one thread per
// cell with all five variables: 67 us, 67 us, 84 us, 3.28 ms).  Residency
// asked for on 1.57 M cells: 4 blocks 3.63 ms, 5 3.26, 6 3.24, 7 3.21 (2 to 5%
// slower below 20,000 cells).
// The five warps of 32 cells form a block (blockDim.y = 5) and share the
// weights in L1 where there are slices enough to level the SM quarters out
// (kGrad64Rows; at 64,000 cells 67 against 64 us, the same from 235,000 on);
// otherwise they are five blocks (gridDim.y = 5).  per = 32-cell slices of a
// tile.
constexpr int kGrad64Rows = 4000;
// Slice i (32 cells) and variable v by one warp.
template <int FUSE_DT, typename RT>
__device__ __forceinline__ void grad64_slice(const RT &regs, const Tile *__restrict__ tiles, int i,
                                             int per, int v) {
  const int lane = threadIdx.x & 31;
  const Tile tl = tile_at(regs, tiles, i / per, per * 32);
  const RegionDev<double> &g = regs[tl.region];
  const int c = tl.first + i % per * 32 + lane;
  unsigned long long bits = 0x7FF0000000000000ull;
  if (c < g.nCells) bits = grad_cell64<FUSE_DT>(g, c, v);
  if (FUSE_DT && v == 0) {
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long x = __shfl_down_sync(0xffffffffu, bits, o);
      bits = x < bits ? x : bits;
    }
    if (lane == 0 && bits < __ldcg(g.dtBits)) atomicMin(g.dtBits, bits);
  }
}
template <int FUSE_DT, typename RT>
__device__ __forceinline__ void grad64_body(const RT &regs, const Tile *__restrict__ tiles,
                                            int nTiles, int per) {
  const int v = blockIdx.y * blockDim.y + threadIdx.y;
  for (int i = pdl_wait(); i < nTiles * per; i += gridDim.x)
    grad64_slice<FUSE_DT>(regs, tiles, i, per, v);
}
template <int FUSE_DT>
__global__ void __launch_bounds__(160, 6)
    k_grad_lim64(const RegionDev<double> *__restrict__ regs, const Tile *__restrict__ tiles,
                 int nTiles, int per) {
  grad64_body<FUSE_DT>(regs, tiles, nTiles, per);
}
template <int FUSE_DT>
__global__ void __launch_bounds__(160, 6)
    k_grad_lim64(const __grid_constant__ OneRegion<double> regs, const Tile *__restrict__ tiles,
                 int nTiles, int per) {
  grad64_body<FUSE_DT>(regs, tiles, nTiles, per);
}

// Small single regions, mixed path: latency bounds the pass, not the number of
// resident warps, so it takes 128 registers, which hold the eight gathers of a
// group in flight (64 serialise them), and blocks of 64 cells, which spread over
// the SMs.  A step of 3,000 / 10,000 / 25,000 / 48,000 tets: 61.4 / 61.5 / 65.6
// / 73.7 -> 54.7 / 55.3 / 59.4 / 71.0 us; at 105,000 tets the resident warps
// count again (108 -> 127 us).  Blocks of 32 and 128 measured the same within
// 2%, 20 gathers in flight slower.
constexpr int kFewBlock = 64, kFewTiles = 400;  // 128-cell tiles
template <typename R, int FUSE_DT>
__global__ void __launch_bounds__(kFewBlock, 8)
    k_grad_few(const __grid_constant__ OneRegion<R> regs, int nTiles) {
  __shared__ unsigned long long smin[32];
  RF_TILE_LOOP(pdl_wait(), nTiles) grad_tile<R, FUSE_DT>(regs, nullptr, t_, smin);
}

template <typename R, int FUSE_DT, int BS>
__global__ void __launch_bounds__(BS, ((sizeof(R) == 4) ? (FUSE_DT ? RF_GRAD_MINB_DT : RF_GRAD_MINB)
                                                        : 4) * 128 / BS)
    k_grad_lim(const RegionDev<R> *__restrict__ regs, const Tile *__restrict__ tiles, int nTiles) {
  __shared__ unsigned long long smin[32];
  RF_TILE_LOOP(pdl_wait(), nTiles) grad_tile<R, FUSE_DT>(regs, tiles, t_, smin);
}
template <typename R, int FUSE_DT, int BS>
__global__ void __launch_bounds__(BS, ((sizeof(R) == 4) ? (FUSE_DT ? RF_GRAD_MINB_DT : RF_GRAD_MINB)
                                                        : 4) * 128 / BS)
    k_grad_lim(const __grid_constant__ OneRegion<R> regs, const Tile *__restrict__ tiles, int nTiles) {
  __shared__ unsigned long long smin[32];
  RF_TILE_LOOP(pdl_wait(), nTiles) grad_tile<R, FUSE_DT>(regs, tiles, t_, smin);
}

// Riemann flux of one interior face on its (reconstructed) states, by DISCR.
// AUSM+up sets up H and a as its face loops do: at second order from the
// reconstructed state with refCp/refGamma (T = p/(rho R), a = sqrt(g R T),
// H = cp T + |v|^2/2; RFLU_AUSMPlusUp_ComputeFlux2_TCP :3255-3632), at first
// order from the cells (H = E/rho + p/rho, a = dv(SOUN); ComputeFlux1
// :894-1366, FP32 sound speed sqrt(g p/rho) on the mixed path).
template <typename R, typename A>
__device__ __forceinline__ void face_riemann(const RegionDev<R> &g, int c1, int c2, const A L[5],
                                             const A Rt[5], A irl, A irr, const A nrm[4],
                                             A flx[8]) {
  const int sd = g.ph.spaceDiscr;
  if (sd == 4) {
    ausm_flux(g.ph, L, Rt, nrm[0], nrm[1], nrm[2], nrm[3], flx);
  } else if (sd == 1) {
    roe_flux(g.ph, L, Rt, nrm[0], nrm[1], nrm[2], nrm[3], flx);
  } else if (sd == 5) {
    const PC<A> k{g.ph};
    A Hl, al, Hr, ar;
    if (g.ph.spaceOrder > 1) {
      const A cp = k.cp(), gm = k.g(), gc = k.gc();
      const A tl = L[4] / (L[0] * gc), tr = Rt[4] / (Rt[0] * gc);
      al = sqrt(gm * gc * tl);
      Hl = cp * tl + scale<-1>(L[1] * L[1] + L[2] * L[2] + L[3] * L[3]) + A(0);
      ar = sqrt(gm * gc * tr);
      Hr = cp * tr + scale<-1>(Rt[1] * Rt[1] + Rt[2] * Rt[2] + Rt[3] * Rt[3]) + A(0);
    } else if (sizeof(R) == 8) {
      const int N = g.nCells;
      al = A(g.dv[2 * N + c1]);
      Hl = A(g.cv[4 * N + c1]) * irl + L[4] / L[0];
      ar = A(g.dv[2 * N + c2]);
      Hr = A(g.cv[4 * N + c2]) * irr + Rt[4] / Rt[0];
    } else {
      const A gv = k.gvG();
      al = sqrt(gv * L[4] / L[0]);
      Hl = eo_dgpuvw(L[0], gv, L[4], L[1], L[2], L[3]) + L[4] / L[0];
      ar = sqrt(gv * Rt[4] / Rt[0]);
      Hr = eo_dgpuvw(Rt[0], gv, Rt[4], Rt[1], Rt[2], Rt[3]) + Rt[4] / Rt[0];
    }
    const A sig = sizeof(R) == 8 ? A(g.ph.ausmSigma) : A(g.ph.ausmSigmaF);
    const A kp = sizeof(R) == 8 ? A(g.ph.ausmKp) : A(g.ph.ausmKpF);
    const A ku = sizeof(R) == 8 ? A(g.ph.ausmKu) : A(g.ph.ausmKuF);
    ausmup_flux(sig, kp, ku, L, Rt, Hl, al, Hr, ar, nrm[0], nrm[1], nrm[2], nrm[3], flx);
  } else {
    hllc_flux(g.ph, L, Rt, irl, irr, nrm[0], nrm[1], nrm[2], nrm[3], flx);
  }
}

// Flux of one interior face in the arithmetic type A (R, or Sd for R = double).
template <typename A, typename R>
__device__ __forceinline__ void face_flux_in(const RegionDev<R> &g, int f, int c1, int c2,
                                             A flx[8]) {
  const int F = g.nFaces;
  auto num = [](const R *x, A *y, auto n) {
#pragma unroll
    for (int k = 0; k < decltype(n)::value; ++k) y[k] = A(x[k]);
  };
  R t4[4], t1[8], t2[8];
  ld4s<RF_HINT_F>(g.fnA + 4 * (size_t)f, t4);
  ld8(g.rec + 8 * (size_t)c1, t1);
  ld8(g.rec + 8 * (size_t)c2, t2);
  A nrm[4], r1[8], r2[8];
  num(t4, nrm, Int<4>());
  num(t1, r1, Int<8>());
  num(t2, r2, Int<8>());
  A L[5], Rt[5], irl, irr;
  cell_values(g, r1, L, irl);
  cell_values(g, r2, Rt, irr);
  if (g.ph.spaceOrder > 1) {
    R tg[16];
    A G[16];
    ld16(g.grad + 16 * (size_t)c1, tg);
    num(tg, G, Int<16>());
    reconstruct(G, A(lds<RF_HINT_F>(g.fdl + f)), A(lds<RF_HINT_F>(g.fdl + F + f)),
                A(lds<RF_HINT_F>(g.fdl + 2 * F + f)), L);
    ld16(g.grad + 16 * (size_t)c2, tg);
    num(tg, G, Int<16>());
    reconstruct(G, A(lds<RF_HINT_F>(g.fdr + f)), A(lds<RF_HINT_F>(g.fdr + F + f)),
                A(lds<RF_HINT_F>(g.fdr + 2 * F + f)), Rt);
  }
  face_riemann(g, c1, c2, L, Rt, irl, irr, nrm, flx);
}

// FP64: the products on the integer pipes (Sd); a face with an operand outside
// their range comes back as NaN and is evaluated again on plain doubles.
template <typename R>
__device__ __forceinline__ void face_flux_value(const RegionDev<R> &g, int f, int c1, int c2,
                                                R flx[8]) {
  if constexpr (sizeof(R) == 8) {
    Sd v[8];
    face_flux_in<Sd>(g, f, c1, c2, v);
    bool again = false;
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      flx[k] = v[k].v;
      again = again || unknown(v[k]);
    }
    if (again) face_flux_in<R>(g, f, c1, c2, flx);
  } else {
    face_flux_in<R>(g, f, c1, c2, flx);
  }
  flx[5] = flx[6] = flx[7] = R(0);
}

template <typename R>
__device__ __forceinline__ void face_flux_one(const RegionDev<R> &g, int f) {
  const int F = g.nFaces;
  {
    const int c1 = lds<RF_HINT_F>(g.f2c + f), c2 = lds<RF_HINT_F>(g.f2c + F + f);
#if RF_FACE_PF
    if (g.ph.spaceOrder > 1) {  // both gradient rows on their way while the records arrive
      prefetch_l1(g.grad + 16 * (size_t)c1);
      prefetch_l1(g.grad + 16 * (size_t)c2);
    }
#endif
    R flx[8];
    face_flux_value(g, f, c1, c2, flx);
    st8(g.flux + 8 * (size_t)f, flx);
  }
}

// Interior face fluxes, *_ComputeFlux2_TCP face loops (AUSM+ :2726-2846,
// Roe :2646-2855, HLLC :2239-2409), written to the face flux buffer.  A tile
// is BS * FPT consecutive faces; thread i of the block takes faces i, i + BS,
// ... of it (FPT faces per thread).
template <typename R, int BS, int FPT, typename RT>
__device__ __forceinline__ void face_tile(const RT &regs, const Tile *__restrict__ tiles,
                                          int nTiles, int t_, int dist) {
  const Tile tl = tile_at(regs, tiles, t_, BS * FPT);
  const RegionDev<R> &g = regs[tl.region];
  prefetch_ahead(t_, nTiles, dist, [&](int t) {
    const Tile tp = tile_at(regs, tiles, t, BS * FPT);
    prefetch_face_tile(regs[tp.region], tp.first, BS * FPT);
  });
#pragma unroll
  for (int k = 0; k < FPT; ++k) {
    const int f = tl.first + threadIdx.x + k * BS;
    if (f < g.nFaces) face_flux_one(g, f);
  }
}

// RFLU_MinimumTimeStep (rocflu/RFLU_MinimumTimeStep.F90:131-146,235-241) and the
// end-time clip of rocflu/RFLU_TimeStepping.F90:490-493 for one region, from
// the minimum local time step `raw` (bit pattern).
template <typename R>
__device__ __forceinline__ void dt_finalize_region(const RegionDev<R> &g, unsigned long long raw,
                                                   const DtArgs &a) {
  double dtMin = __longlong_as_double((long long)raw);
  const double t = a.useDeviceTime ? __ldcg(g.scal + 1) : a.timeHost;
  dtMin = a.cfl * dtMin;
  double wI = 0.0, wC = 0.0;
  if (t <= 1.0e-08) wI = 1.0; else wC = 1.0;
  dtMin = wI / a.dtImposed + wC / dtMin;
  dtMin = 1.0 / dtMin;
  if (dtMin <= 0.0) dtMin = 6.0e-12;
  dtMin = (a.dtMinLimit > dtMin) ? a.dtMinLimit : dtMin;
  double tNew = t + dtMin;
  if (a.endTime > 0.0 && t + dtMin > a.endTime) {
    dtMin = a.endTime - t;
    tNew = a.endTime;
  }
  if (a.endTime > 0.0 && t >= a.endTime) {  // finished: later stages leave cv as is
    dtMin = 0.0;
    tNew = t;
  }
  g.scal[0] = dtMin;
  g.scal[2] = dtMin;
  for (int i = 0; i < 5; ++i) g.scal[3 + i] = g.ph.ark[i] * dtMin;  // fac of RkUpdateGeneric
  if (a.useDeviceTime) g.scal[1] = tNew;
}

// The time-step finalisation of nRegions regions by one block.  Independent
// regions: one thread each.  Coupled regions: the minimum over all regions
// first, as the reference's MIN over local regions and MPI_Allreduce(MPI_MIN)
// (RFLU_MinimumTimeStep.F90:148-208), then every region finalizes it; the
// per-region steps of RFLU_MinimumTimeStep (cfl scaling, imposed/computed
// weighting, floor, dtMinLimit) are monotone non-decreasing, so applying them
// to the minimum gives the reference's minimum of the per-region results.  The
// raw minima are read through L2: in the persistent stage kernel other blocks
// reduced them earlier in the same launch.
template <typename R, typename RT>
__device__ __forceinline__ void dt_finalize_block(const RT &regs,
                                                  int nRegions, int coupled,
                                                  const DtArgs &a, unsigned long long *smin) {
  if (!coupled) {
    for (int r = threadIdx.x; r < nRegions; r += blockDim.x) {
      const RegionDev<R> &g = regs[r];
      const unsigned long long raw = __ldcg(g.dtBits);
      *g.dtBits = 0x7FF0000000000000ull;
      dt_finalize_region(g, raw, a);
    }
    return;
  }
  unsigned long long v = 0x7FF0000000000000ull;
  for (int r = threadIdx.x; r < nRegions; r += blockDim.x) {
    const unsigned long long x = __ldcg(regs[r].dtBits);
    v = x < v ? x : v;
  }
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long x = __shfl_down_sync(0xffffffffu, v, o);
    v = x < v ? x : v;
  }
  if ((threadIdx.x & 31) == 0) smin[threadIdx.x >> 5] = v;
  __syncthreads();
  unsigned long long raw = smin[0];
  for (int k = 1; k < (int)(blockDim.x >> 5); ++k) raw = smin[k] < raw ? smin[k] : raw;
  __syncthreads();
  for (int r = threadIdx.x; r < nRegions; r += blockDim.x) {
    *regs[r].dtBits = 0x7FF0000000000000ull;
    dt_finalize_region(regs[r], raw, a);
  }
}

// Farfield rind state, RFLU_SetRindStateFarfieldPerf
// (modflu/RFLU_ModRindStates.F90:249-421) without the airfoil lift
// correction; fd = (ri, pi, qi, ui, vi, wi, machInf) of the face, evaluated
// on the host.  Subsonic: characteristic combination of the interior and
// free-stream states; supersonic: free stream in, interior out.
template <typename R>
__device__ __forceinline__ void farfield_rind(const R *fd, R gGas, R nx, R ny, R nz, R rl, R rul,
                                              R rvl, R rwl, R rel, R &rr, R &rur, R &rvr, R &rwr,
                                              R &rer, R &pr) {
  const R ri = fd[0], pi = fd[1], qi = fd[2], ui = fd[3], vi = fd[4], wi = fd[5], machInf = fd[6];
  const R ul = rul / rl, vl = rvl / rl, wl = rwl / rl;
  const R ql = ul * nx + vl * ny + wl * nz;
  const R el = rel / rl;
  const R sl2 = ul * ul + vl * vl + wl * wl;
  const R pl = (gGas - R(1)) * rl * (el - R(0.5) * sl2 - R(0));
  if (machInf < R(1)) {
    const R al = sqrt(gGas * pl / rl);
    R pb, rb, ub, vb, wb;
    if (ql < R(0)) {
      pb = R(0.5) * (pi + pl - rl * al * ((ui - ul) * nx + (vi - vl) * ny + (wi - wl) * nz));
      rb = ri - (pi - pb) / (al * al);
      ub = ui - nx * (pi - pb) / (rl * al);
      vb = vi - ny * (pi - pb) / (rl * al);
      wb = wi - nz * (pi - pb) / (rl * al);
    } else {
      pb = pi;
      rb = rl - (pl - pi) / (al * al);
      ub = ul + nx * (pl - pi) / (rl * al);
      vb = vl + ny * (pl - pi) / (rl * al);
      wb = wl + nz * (pl - pi) / (rl * al);
    }
    rr = rb;
    rur = rb * ub;
    rvr = rb * vb;
    rwr = rb * wb;
    rer = rb * eo_dgpuvw(rb, gGas, pb, ub, vb, wb);
    pr = pb;
  } else if (ql < R(0)) {
    rr = ri;
    rur = ri * ui;
    rvr = ri * vi;
    rwr = ri * wi;
    rer = ri * (pi / (ri * (gGas - R(1))) + R(0.5) * qi * qi + R(0));  // MixtPerf_Eo_DGPVm
    pr = pi;
  } else {
    rr = rl;
    rur = rul;
    rvr = rvl;
    rwr = rwl;
    rer = rel;
    pr = pl;
  }
}

// Total-pressure / total-temperature inflow state, libfloflu/BcondInflowPerf.F90:
// 93-272 (ksg = 0).  d = (ptot, ttot, a02, cos betah, sin betah, cos betav,
// sin betav, fixed, supersonic-branch state rr, rur, rvr, rwr, rer, pr).  A
// SUBSONIC patch whose interior normal velocity is supersonic leaves the
// reference's outputs unset; the interior state is used here.
template <typename R>
__device__ __forceinline__ void inflow_totang(const R *d, int opt, R g, R rgas, R nx, R ny, R nz,
                                              R rl, R rul, R rvl, R rwl, R rel, R pl, R &rr,
                                              R &rur, R &rvr, R &rwr, R &rer, R &pr) {
  const R ptot = d[0], ttot = d[1], a02 = d[2], cbh = d[3], sbh = d[4], cbv = d[5], sbv = d[6];
  const bool fixed = d[7] != R(0);
  bool prescribed = opt == 0;  // BCOPT_SUPERSONIC
  if (!prescribed) {
    const R gm1 = g - R(1);
    const R ul = rul / rl, vl = rvl / rl, wl = rwl / rl;
    const R al = sqrt(a02 - R(0.5) * (g - R(1)) * (ul * ul + vl * vl + wl * wl));  // C_Co2GUVW
    const R ql = ul * nx + vl * ny + wl * nz;
    if (fabs(ql) < al) {
      const R sl = sqrt(ul * ul + vl * vl + wl * wl);
      R eta = R(-1);
      if (!fixed && sl > R(1.0e-6)) eta = ql / sl;
      const R Rm = al - R(0.5) * gm1 * ql;
      const R disc =
          R(0.5) * gm1 * (eta * eta) * (a02 / (Rm * Rm) * (R(1) + R(0.5) * gm1 * (eta * eta)) - R(1));
      R ar, tr, sr;
      if (disc < R(0)) {
        ar = sqrt(a02);
        tr = ttot;
        pr = ptot;
        sr = R(0);
      } else {
        ar = Rm / (R(1) + R(0.5) * gm1 * eta * eta) * (R(1) + sqrt(disc));
        tr = ar * ar / (g * rgas);                          // MixtPerf_T_CGR
        pr = ptot * pow(tr / ttot, g / (g - R(1)));         // MixtPerf_P_GPoTTo
        const R c2 = ar * ar;
        sr = a02 > c2 ? sqrt(R(2) / (g - R(1)) * (a02 - c2)) : R(0);  // MixtPerf_Vm_C2Co2G
      }
      rr = pr / (rgas * tr);
      const R ur = sr * cbh * cbv, vr = sr * sbh, wr = sr * cbh * sbv;
      rer = rr * (pr / (rr * (g - R(1))) + R(0.5) * sr * sr + R(0));  // MixtPerf_Eo_DGPVm
      rur = rr * ur;
      rvr = rr * vr;
      rwr = rr * wr;
      return;
    }
    prescribed = opt == 2;  // BCOPT_MIXED
  }
  if (prescribed) {
    rr = d[8];
    rur = d[9];
    rvr = d[10];
    rwr = d[11];
    rer = d[12];
    pr = d[13];
  } else {
    rr = rl;
    rur = rul;
    rvr = rvl;
    rwr = rwl;
    rer = rel;
    pr = pl;
  }
}

// Outflow boundary state, libfloflu/BcondOutflowPerf.F90:88-160 (ksg = 0).
template <typename R>
__device__ __forceinline__ void bcond_outflow(int bcOpt, R pout, R sxn, R syn, R szn, R gamma,
                                              R rho, R rhou, R rhov, R rhow, R rhoe, R press,
                                              R &rhob, R &rhoub, R &rhovb, R &rhowb, R &rhoeb) {
  R u = rhou / rho, v = rhov / rho, w = rhow / rho;
  R csound = sqrt(gamma * press / rho);
  R mach = sqrt(u * u + v * v + w * w) / csound;
  if (mach < R(1) && (bcOpt == 1 || bcOpt == 2)) {
    R rrhoc = R(1) / (rho * csound);
    R deltp = press - pout;
    rhob = rho - deltp / (csound * csound);
    R ub = u + sxn * deltp * rrhoc;
    R vb = v + syn * deltp * rrhoc;
    R wb = w + szn * deltp * rrhoc;
    R vnd = ub * sxn + vb * syn + wb * szn;
    if (vnd < R(0)) {
      ub = copysign(R(1), u) * rmax(fabs(ub), fabs(u));
      vb = copysign(R(1), v) * rmax(fabs(vb), fabs(v));
      wb = copysign(R(1), w) * rmax(fabs(wb), fabs(w));
    }
    rhoub = rhob * ub;
    rhovb = rhob * vb;
    rhowb = rhob * wb;
    rhoeb = rhob * eo_dgpuvw(rhob, gamma, pout, ub, vb, wb);
  } else {
    rhob = rho;
    rhoub = rhou;
    rhovb = rhov;
    rhowb = rhow;
    rhoeb = rhoe;
  }
}

// Boundary face fluxes: slip wall and outflow patches of
// rocflu/RFLU_CentralSecondPatch.F90:638-1013 (ORDER 2) and
// rocflu/RFLU_CentralFirstPatch.F90:575-946 (ORDER 1).  Slip walls store -0.0
// as mass flux, the exact additive identity, since the reference leaves the
// mass residual untouched there.
constexpr int kBTile = 128;  // boundary faces per tile and threads of the blocks that take it
template <typename R, typename RT>
__device__ __forceinline__ void bface_tile(const RT &regs, const Tile *__restrict__ tiles, int t_) {
  {
    const Tile tl = tile_at(regs, tiles, t_, kBTile);
    const RegionDev<R> &g = regs[tl.region];
    const int b = tl.first + threadIdx.x;
    const int B = g.nBFaces;
    if (b >= B) return;
    const int N = g.nCells;
    const int c = g.bf2c[b];
    const int kind = g.bkind[b];
    const int type = kind & 15, order = (kind >> 4) & 15, opt = kind >> 8;
    R nrm[4];
    ld4(g.bfnA + 4 * (size_t)b, nrm);
    const R nx = nrm[0], ny = nrm[1], nz = nrm[2], nm = nrm[3];
    const R fs = R(0);
    R flx[8];
    R rc[8];
    ld8(g.rec + 8 * (size_t)c, rc);
    R S[5], ir;
    cell_values(g, rc, S, ir);
    if (order == 2) {
      R G[16];
      ld16(g.grad + 16 * (size_t)c, G);
      reconstruct(G, g.bfd[b], g.bfd[B + b], g.bfd[2 * B + b], S);
    }
    const R gvG = PC<R>{g.ph}.gvG();
    if (type == BK_SLIP) {
      R pl = S[4];
      flx[0] = R(-0.0);
      flx[1] = pl * nx * nm;
      flx[2] = pl * ny * nm;
      flx[3] = pl * nz * nm;
      flx[4] = pl * fs * nm;
    } else if (type == BK_INJECTION && g.bdat[kBData * (size_t)b] > R(0)) {
      // burning surface (RFLU_CentralSecondPatch.F90:1237-1351 / FirstPatch
      // :1049-1133 with RFLU_SetRindStateInjectPerf, RFLU_ModRindStates.F90:460-505)
      const R minj = g.bdat[kBData * (size_t)b], tinj = g.bdat[kBData * (size_t)b + 1];
      const R rGas = R(g.ph.gvR), cpGas = R(g.ph.gvCp);
      const R pl = S[4];
      const R rl = pl / (rGas * tinj);
      const R ql = -minj / rl + fs;
      const R ul = ql * nx, vl = ql * ny, wl = ql * nz;
      const R Hl = cpGas * tinj + R(0.5) * (ul * ul + vl * vl + wl * wl) + R(0);
      flx[0] = -minj * nm;
      flx[1] = (-minj * ul + pl * nx) * nm;
      flx[2] = (-minj * vl + pl * ny) * nm;
      flx[3] = (-minj * wl + pl * nz) * nm;
      flx[4] = (-minj * Hl + pl * fs) * nm;
    } else {
      R rl, rul, rvl, rwl, rel, pl;
      if (order == 2) {
        rl = S[0];
        pl = S[4];
        rul = rl * S[1];
        rvl = rl * S[2];
        rwl = rl * S[3];
        rel = rl * eo_dgpuvw(rl, gvG, pl, S[1], S[2], S[3]);
      } else {
        rl = rc[0];
        pl = rc[4];
        if (sizeof(R) == 8 && g.ph.spaceOrder == 1) {  // no conversion round trip
          rul = R(g.cv[N + c]);
          rvl = R(g.cv[2 * N + c]);
          rwl = R(g.cv[3 * N + c]);
          rel = R(g.cv[4 * N + c]);
        } else {  // cv as CellGradientsMP's Prim2Cons left it
          R u = rc[1], v = rc[2], w = rc[3];
          rul = rl * u;
          rvl = rl * v;
          rwl = rl * w;
          rel = rl * eo_dgpuvw(rl, gvG, pl, u, v, w);
        }
      }
      if (type == BK_INJECTION) {
        // surface not burning: slip-wall rind pressure (RFLU_SetRindStateSlipWallPerf,
        // RFLU_ModRindStates.F90:539-588); the mass flux is a +0 contribution
        const R irl = R(1) / rl;
        const R ul = irl * rul, vl = irl * rvl, wl = irl * rwl;
        const R ql = ul * nx + vl * ny + wl * nz - fs;
        const R al = sqrt(gvG * pl / rl);
        if (ql < R(0)) {
          const R term = R(1) + R(0.5) * (gvG - R(1)) * ql / al;
          pl = pl * pow(term, R(2) * gvG / (gvG - R(1)));
        } else {
          const R term = (gvG + R(1)) / R(4);
          pl = pl + term * rl * ql * (ql + sqrt(al * al + term * term * ql * ql) / term);
        }
        flx[0] = R(0);
        flx[1] = pl * nx * nm;
        flx[2] = pl * ny * nm;
        flx[3] = pl * nz * nm;
        flx[4] = pl * fs * nm;
      } else {
        R pr, rr, rur, rvr, rwr, rer;
        if (type == BK_FARFIELD) {
          farfield_rind(g.bdat + kBData * (size_t)b, gvG, nx, ny, nz, rl, rul, rvl, rwl, rel, rr, rur,
                        rvr, rwr, rer, pr);
        } else if (type == BK_INFLOW_TA) {
          inflow_totang(g.bdat + kBData * (size_t)b, opt, gvG, R(g.ph.gvR), nx, ny, nz, rl, rul, rvl,
                        rwl, rel, pl, rr, rur, rvr, rwr, rer, pr);
        } else if (type == BK_INFLOW_VT) {
          const R *d = g.bdat + kBData * (size_t)b;
          const R ur = d[0], vr = d[1], wr = d[2], tr = d[3], rGas = R(g.ph.gvR);
          if (opt != 1) {  // BCOPT_SUBSONIC
            pr = d[4];
            rr = pr / (rGas * tr);  // MixtPerf_D_PRT
          } else {
            rr = rl;
            pr = rr * rGas * tr;    // MixtPerf_P_DRT
          }
          rer = rr * eo_dgpuvw(rr, gvG, pr, ur, vr, wr);
          rur = rr * ur;
          rvr = rr * vr;
          rwr = rr * wr;
        } else {
          pr = (opt != 0) ? R(g.bpout[b]) : pl;
          bcond_outflow(opt, pr, nx, ny, nz, gvG, rl, rul, rvl, rwl, rel, pl, rr, rur, rvr, rwr,
                        rer);
        }
        R ql = (rul * nx + rvl * ny + rwl * nz) / rl - fs;
        R qr = (rur * nx + rvr * ny + rwr * nz) / rr - fs;
        flx[0] = R(0.5) * (ql * rl + qr * rr) * nm;
        flx[1] = R(0.5) * (ql * rul + pl * nx + qr * rur + pr * nx) * nm;
        flx[2] = R(0.5) * (ql * rvl + pl * ny + qr * rvr + pr * ny) * nm;
        flx[3] = R(0.5) * (ql * rwl + pl * nz + qr * rwr + pr * nz) * nm;
        flx[4] = R(0.5) * (ql * (rel + pl) + pl * fs + qr * (rer + pr) + pr * fs) * nm;
      }
    }
    flx[5] = flx[6] = flx[7] = R(0);
    st8(g.bflux + 8 * (size_t)b, flx);
  }
}

// The flux pass of a stage: the interior-face tiles, behind the boundary-face
// tiles and (stage 1) one block that finalises the time step, all independent
// of one another; as launches of their own they followed one after another,
// each with its latency (4,000-cell tube, FP64: 16 + 15 us; 10,000 tets, mixed:
// 6.5 + 5.8 + 5 us).
struct FluxExtra {
  const Tile *bface;
  int nBFace;
  int dt, nRegions, coupled;
  DtArgs a;
};

template <typename R, int BS, int FPT>
__global__ void __launch_bounds__(BS)
    k_face_flux(const RegionDev<R> *__restrict__ regs, const Tile *__restrict__ tiles, int nTiles,
                int pfDist) {
  const int dist = (int)gridDim.x < nTiles ? (int)gridDim.x : pfDist;
  RF_TILE_LOOP(pdl_wait(), nTiles) face_tile<R, BS, FPT>(regs, tiles, nTiles, t_, dist);
}
template <typename R, int BS, int FPT>
__global__ void __launch_bounds__(BS)
    k_face_flux(const __grid_constant__ OneRegion<R> regs, const Tile *__restrict__ tiles,
                int nTiles, int pfDist) {
  const int dist = (int)gridDim.x < nTiles ? (int)gridDim.x : pfDist;
  RF_TILE_LOOP(pdl_wait(), nTiles) face_tile<R, BS, FPT>(regs, tiles, nTiles, t_, dist);
}

// FP64: one kernel for every launch shape, a tile of `stride` faces walked by
// its block.  Bound by the FP64 pipe; 128 registers asked for (168: the same
// time, 102: 1% slower).  64^3 tets AUSM+ 1.53 -> 1.11 ms, AUSM+up 1.76 ->
// 1.32, Roe 2.42 -> 1.83, HLLC 1.82 -> 1.44 with the reconstruction and prod()
// products on the integer pipes (the reconstruction alone: 1.32, 1.54, 2.14,
// 1.60), the exponent scalings, and the velocities kept per cell.
template <typename RT>
__device__ __forceinline__ void face64_body(const RT &regs, const Tile *__restrict__ tiles,
                                            int nTiles, int pfDist, int stride) {
  const int dist = (int)gridDim.x < nTiles ? (int)gridDim.x : pfDist;
  RF_TILE_LOOP(pdl_wait(), nTiles) {
    const Tile tl = tile_at(regs, tiles, t_, stride);
    const RegionDev<double> &g = regs[tl.region];
    prefetch_ahead(t_, nTiles, dist, [&](int t) {
      const Tile tp = tile_at(regs, tiles, t, stride);
      prefetch_face_tile(regs[tp.region], tp.first, stride);
    });
    const int last = tl.first + stride < g.nFaces ? tl.first + stride : g.nFaces;
    for (int f = tl.first + threadIdx.x; f < last; f += blockDim.x) face_flux_one(g, f);
  }
}
template <typename R>
__global__ void __launch_bounds__(128, 4)
    k_face_flux64(const RegionDev<double> *__restrict__ regs, const Tile *__restrict__ tiles,
                  int nTiles, int pfDist, int stride) {
  face64_body(regs, tiles, nTiles, pfDist, stride);
}
template <typename R>
__global__ void __launch_bounds__(128, 4)
    k_face_flux64(const __grid_constant__ OneRegion<double> regs, const Tile *__restrict__ tiles,
                  int nTiles, int pfDist, int stride) {
  face64_body(regs, tiles, nTiles, pfDist, stride);
}

template <typename R, typename RT>
__device__ __forceinline__ void flux_merged_body(const RT &regs, const Tile *__restrict__ tiles,
                                                 int nTiles, int pfDist, const FluxExtra &x,
                                                 unsigned long long *smin) {
  const int n0 = x.dt + x.nBFace;
  const int dist = (int)gridDim.x < nTiles + n0 ? (int)gridDim.x : pfDist;
  RF_TILE_LOOP(pdl_wait(), nTiles + n0) {
    if (t_ >= n0)
      face_tile<R, 128, 1>(regs, tiles, nTiles, t_ - n0, dist);
    else if (t_ >= x.dt)
      bface_tile<R>(regs, x.bface, t_ - x.dt);
    else
      dt_finalize_block<R>(regs, x.nRegions, x.coupled, x.a, smin);
  }
}
template <typename R>
__global__ void __launch_bounds__(128, (sizeof(R) == 4 ? 0 : 4))
    k_flux_merged(const RegionDev<R> *__restrict__ regs, const Tile *__restrict__ tiles, int nTiles,
                  int pfDist, const FluxExtra x) {
  __shared__ unsigned long long smin[32];
  flux_merged_body<R>(regs, tiles, nTiles, pfDist, x, smin);
}
template <typename R>
__global__ void __launch_bounds__(128, (sizeof(R) == 4 ? 0 : 4))
    k_flux_merged(const __grid_constant__ OneRegion<R> regs, const Tile *__restrict__ tiles, int nTiles,
                  int pfDist, const FluxExtra x) {
  __shared__ unsigned long long smin[32];
  flux_merged_body<R>(regs, tiles, nTiles, pfDist, x, smin);
}

template <typename R>
__global__ void __launch_bounds__(128) k_bface_flux(const RegionDev<R> *__restrict__ regs,
                                                    const Tile *__restrict__ tiles, int nTiles) {
  RF_TILE_LOOP(pdl_wait(), nTiles) bface_tile<R>(regs, tiles, t_);
}
template <typename R>
__global__ void __launch_bounds__(128) k_bface_flux(const __grid_constant__ OneRegion<R> regs,
                                                    const Tile *__restrict__ tiles, int nTiles) {
  RF_TILE_LOOP(pdl_wait(), nTiles) bface_tile<R>(regs, tiles, t_);
}

// AfterUpdateMP checks for one cell (libfloflu/AfterUpdateMP.F90:134-136):
// RFLU_CheckValidity, RFLU_EnforceBounds (libflu/RFLU_EnforceBounds.F90:163-232),
// RFLU_CheckPositivity (libflu/RFLU_CheckPositivity.F90).  Returns status bits.
__device__ __forceinline__ unsigned after_update(double gc, double gg, double q[5], double d[3]) {
  unsigned st = 0;
  {
    double rho = q[0], rrho = 1.0 / rho;
    double u = rrho * q[1], v = rrho * q[2], w = rrho * q[3];
    if (isnan(rho) || isnan(u) || isnan(v) || isnan(w) || isnan(d[0]) || isnan(d[1])) st |= 1u;
  }
  {
    const double pTol = 1.0e-12;
    double rr = q[0], ir = 1.0 / rr;
    double u = ir * q[1], v = ir * q[2], w = ir * q[3], Eo = ir * q[4];
    double Vm2 = u * u + v * v + w * w;
    double p = (gg - 1.0) * rr * (Eo - 0.5 * Vm2 - 0.0);
    if (p <= 0.0 && fabs(p) <= pTol) {
      p = pTol;
      q[4] = rr * (p / (rr * (gg - 1.0)) + 0.5 * (u * u + v * v + w * w) + 0.0);
      st |= 8u;
    }
  }
  {
    double rho = q[0], rrho = 1.0 / rho;
    double u = rrho * q[1], v = rrho * q[2], w = rrho * q[3];
    double Vm2 = u * u + v * v + w * w;
    double p = d[0];
    if (p <= 0.0) {
      double Eo = 1.0e4 + 0.5 * Vm2 + 0.0;
      p = (gg - 1.0) * rho * (Eo - 0.5 * Vm2 - 0.0);
      d[0] = p;
      d[1] = p / (rho * gc);
      q[4] = rho * Eo;
      st |= 4u;
    }
    if (rho <= 0.0 || p <= 0.0) st |= 2u;
  }
  return st;
}

// Whether after_update can change a cell or set a bit: not when density, energy
// and the EOS pressure p are positive and finite and p is no cancellation
// residue.  after_update forms the pressure again in another order of
// operations, and only beyond 2^-30 of the total energy are both sure to be
// positive.  Nothing is NaN then: an infinite or NaN momentum makes p -infinite
// or NaN, and finite ones over a normal density give no NaN.  One branch for
// all four tests: 197,000 tets, split update 35.7 us against 36.2 with a branch
// each.
__device__ __forceinline__ bool checks_can_act(const double q[5], double p) {
  const unsigned e = (unsigned)__double2hiint(q[4]), h = (unsigned)__double2hiint(p);
  return !(positive_bits(q[0]) & positive_bits(p) & positive_bits(q[4]) & (h + (30u << 20) >= e));
}

// Error-free transformation of a + b (Knuth's TwoSum); lo collects the
// rounding errors, so hi + lo carries about twice the FP32 significand.
__device__ __forceinline__ void two_sum_acc(float &hi, float &lo, float x) {
  float s = hi + x;
  float bb = s - hi;
  float err = (hi - (s - bb)) + (x - bb);
  hi = s;
  lo += err;
}

// (hi, lo) - d for a float-float pair: TwoSum of hi and -d, the low part and
// the rounding error added, then renormalised with TwoSum.  Additions only, so
// no contraction into FMA can change it.
__device__ __forceinline__ void ff_sub(float &hi, float &lo, float d) {
  const float s = hi - d;
  const float bb = s - hi;
  const float e = (hi - (s - bb)) + (-d - bb);
  const float t = lo + e;
  const float h2 = s + t;
  const float b2 = h2 - s;
  lo = (s - (h2 - b2)) + (t - b2);
  hi = h2;
}

// Mixed-path gather + update.  The FP32 face fluxes are summed with
// compensated (TwoSum) accumulation, so the residual is the FP32-rounded exact
// sum of the fluxes regardless of cancellation; the RK increment
// dU = a*dt/V (rhs - g rhsSum) is formed in FP32 and subtracted from the
// float-float conserved state exactly (ff_sub), so the state carries about 48
// significand bits without FP64 arithmetic (GB300's FP64 rate is a small
// fraction of its FP32 rate).  The pressure for the cell record is
// (g-1)((E_hi - |m|^2/(2 rho)) + E_lo) in FP32: the total energy keeps its low
// part and only the kinetic term is rounded.  Cells whose density or pressure
// is not clearly positive take the exact FP64 checks of AfterUpdateMP on the
// joined state.  dv (p, T, a) is evaluated in FP64 on download.
__device__ __forceinline__ void gather_update_mixed(const RegionDev<float> &g, int c,
                                                    const StepArgs &a) {
  const int N = g.nCells;
  const Phys &ph = g.ph;
  const int is = a.istage;
  const float *cvF = g.cvF;
  // own-cell loads first: they are independent of the flux gathers below
  float qh[5], ql[5];
  float rsOld[5];
  float r[8];
  float ivol = 0.f;
  if (a.update) {
#pragma unroll
    for (int j = 0; j < 5; ++j) {
      qh[j] = lds_rw<RF_HINT_U>(cvF + (size_t)j * N + c);
      ql[j] = lds_rw<RF_HINT_U>(cvF + (size_t)(5 + j) * N + c);
    }
#pragma unroll
    for (int j = 0; j < 5; ++j)
      rsOld[j] = (is > 1) ? lds_rw<RF_HINT_U>(g.rhsSumF + j * N + c) : 0.f;
    ld8_rw(g.rec + 8 * (size_t)c, r);  // the non-coherent path measured the same (0.598 ms)
    ivol = lds<RF_HINT_U>(g.ivolF + c);
  }
  float hi[5] = {0.f, 0.f, 0.f, 0.f, 0.f}, lo[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
  const long long e0 = g.cfOff[c >> 5] + (c & 31);
  const int n = g.cfCnt[c];
  auto face = [&](int code) {
    float fl[8];
    if (code >= 0) {
      ld8(g.flux + 8 * (size_t)(code >> 1), fl);
      const float sg = (code & 1) ? -1.f : 1.f;
#pragma unroll
      for (int j = 0; j < 5; ++j) two_sum_acc(hi[j], lo[j], sg * fl[j]);
    } else {
      ld8(g.bflux + 8 * (size_t)(-code - 1), fl);
#pragma unroll
      for (int j = 0; j < 5; ++j) two_sum_acc(hi[j], lo[j], fl[j]);
    }
  };
  // the first faces' codes loaded together, ahead of their flux gathers
  constexpr int MF = RF_UPD_PRE;
  int cc[MF];
#pragma unroll
  for (int k = 0; k < MF; ++k)
    cc[k] = k < n ? lds<RF_HINT_U>(g.cfCode + e0 + (long long)k * kSlice) : 0;
#pragma unroll
  for (int k = 0; k < MF; ++k)
    if (k < n) face(cc[k]);
  for (int k = MF; k < n; ++k) face(lds<RF_HINT_U>(g.cfCode + e0 + (long long)k * kSlice));
  if (a.writeRhs) {
#pragma unroll
    for (int j = 0; j < 5; ++j) g.rhs[j * N + c] = double(hi[j]) + double(lo[j]);
  }
  if (!a.update) return;
  float rhs[5];
#pragma unroll
  for (int j = 0; j < 5; ++j) rhs[j] = hi[j] + lo[j];
  // the device time step is read through L2 (__ldcg): in a persistent stage
  // launch another block wrote it earlier in the same kernel
  const float fac = a.useDeviceDt ? float(__ldcg(g.scal + 3 + is - 1)) : float(ph.ark[is - 1] * a.dtHost);
  const float adtv = fac * ivol;
  const float grk = ph.grkF[is - 1];
  float oh[5], ol[5];
  if (ph.rkScheme == 1) {
    if (is == 1) {
#pragma unroll
      for (int j = 0; j < 5; ++j) {
        oh[j] = qh[j];
        ol[j] = ql[j];
        g.cvOldF[(size_t)j * N + c] = qh[j];
        g.cvOldF[(size_t)(5 + j) * N + c] = ql[j];
      }
    } else {
#pragma unroll
      for (int j = 0; j < 5; ++j) {
        oh[j] = g.cvOldF[(size_t)j * N + c];
        ol[j] = g.cvOldF[(size_t)(5 + j) * N + c];
      }
    }
  } else {
#pragma unroll
    for (int j = 0; j < 5; ++j) {
      oh[j] = qh[j];
      ol[j] = ql[j];
    }
  }
  float *rs = g.rhsSumF;
#pragma unroll
  for (int j = 0; j < 5; ++j) {
    float dU;
    if (ph.rkScheme == 2) {
      if (is == 1) {
        dU = adtv * rhs[j];
        rs[j * N + c] = rhs[j];
      } else if (is == 2) {
        dU = adtv * (rhs[j] - grk * rsOld[j]);
        rs[j * N + c] = rhs[j];
      } else {
        dU = adtv * (rhs[j] - grk * rsOld[j]);
      }
    } else if (ph.rkScheme == 1) {
      if (is == 1) {
        dU = adtv * rhs[j];
        rs[j * N + c] = rhs[j];
      } else if (is == ph.nSteps) {
        dU = adtv * (rhs[j] + rsOld[j]);
      } else {
        dU = adtv * rhs[j];
        rs[j * N + c] = rsOld[j] + grk * rhs[j];
      }
    } else {
      dU = adtv * rhs[j];
    }
    qh[j] = oh[j];
    ql[j] = ol[j];
    ff_sub(qh[j], ql[j], dU);
  }
  // EOS of the new state in FP32 from the pairs
  float rr[5];
  record_from_pairs(ph, qh, ql, rr);
  const float rf = rr[0], uf = rr[1], vf = rr[2], wf = rr[3];
  float pf = rr[4];
  if (!(rf > 0.f) || !(pf > 1.0e-12f) || isnan(uf) || isnan(vf) || isnan(wf)) {
    // exact FP64 checks and bounds of AfterUpdateMP on the joined state
    const double gg = ph.gvG;
    double q[5];
#pragma unroll
    for (int j = 0; j < 5; ++j) q[j] = double(qh[j]) + double(ql[j]);
    const double m2 = fma(q[3], q[3], fma(q[2], q[2], q[1] * q[1]));
    double d[3];
    d[0] = (gg - 1.0) * (q[4] - 0.5 * m2 / q[0]);
    d[1] = d[0] / (q[0] * ph.gvR);
    d[2] = 0.0;
    unsigned st = after_update(ph.gvR, gg, q, d);
    if (st) atomicOr(g.status, st);
    pf = float(d[0]);
#pragma unroll
    for (int j = 0; j < 5; ++j) {
      qh[j] = float(q[j]);
      ql[j] = float(q[j] - double(qh[j]));
    }
  }
  float *cvW = g.cvF;
#pragma unroll
  for (int j = 0; j < 5; ++j) {
    cvW[(size_t)j * N + c] = qh[j];
    cvW[(size_t)(5 + j) * N + c] = ql[j];
  }
  r[0] = rf;
  r[1] = uf;
  r[2] = vf;
  r[3] = wf;
  r[4] = pf;
  st8(g.rec + 8 * (size_t)c, r);
}

// Flux row of a cell-to-face code and whether it counts negatively (the cell
// is the face's second cell).  One load and one addition for every kind of
// face: lanes whose faces differ in kind or side then run the FP64 sum once,
// not once per kind (a - x is a + (-x) exactly).  197,000 tets: split update
// 50.3 -> 38.2 us; 1.57 M tets: FP64 update 0.324 -> 0.284 ms.  The mixed
// update, bound by memory, is 5% slower this way and keeps its branches.
template <typename R>
__device__ __forceinline__ const R *flux_row(const RegionDev<R> &g, const R *flux, int code,
                                             bool &minus) {
  minus = code >= 0 && (code & 1);
  return code >= 0 ? flux + 8 * (size_t)(code >> 1) : g.bflux + 8 * (size_t)(-code - 1);
}

// FP64 sum of a cell's face fluxes in the reference accumulation order
// (ConvectiveFluxes' scatter restated as a gather: +flux where the cell is the
// face's first cell, -flux where it is the second, boundary faces added),
// starting from -0.0 as the FP64 path does.  The first RF_UPD_PRE face codes
// are loaded together ahead of the flux gathers.
template <typename R>
__device__ __forceinline__ void face_sum64(const RegionDev<R> &g, const R *__restrict__ flux,
                                           int c, double acc[5]) {
  const long long e0 = g.cfOff[c >> 5] + (c & 31);
  const int n = g.cfCnt[c];
#pragma unroll
  for (int j = 0; j < 5; ++j) acc[j] = -0.0;
  auto face = [&](int code) {
    R fl[8];
    bool minus;
    ld8(flux_row(g, flux, code, minus), fl);
#pragma unroll
    for (int j = 0; j < 5; ++j) acc[j] = acc[j] + as_fp64(minus ? -fl[j] : fl[j]);
  };
  constexpr int MF = RF_UPD_PRE;
  int cc[MF];
#pragma unroll
  for (int k = 0; k < MF; ++k)
    cc[k] = k < n ? lds<RF_HINT_U>(g.cfCode + e0 + (long long)k * kSlice) : 0;
#pragma unroll
  for (int k = 0; k < MF; ++k)
    if (k < n) face(cc[k]);
  for (int k = MF; k < n; ++k) face(lds<RF_HINT_U>(g.cfCode + e0 + (long long)k * kSlice));
}

// FP64 path: the update is bound by the FP64 pipe, so its products are integer
// products too and AfterUpdateMP's checks run only where they can act (1.57 M
// tets 0.48 -> 0.32 ms).  The split path's unit contracts into FMA, where a
// product costs nothing beside its sum; it keeps FP64 products.
// RK update of one cell (libfloflu/RkUpdateGeneric.F90:229-314) in the
// arithmetic type A: q = old - a dt/V (...), and the history row to store
// (rsNew; wr tells whether).
template <typename A>
__device__ __forceinline__ bool rk_cell(const Phys &ph, int is, double adtvD, const double rhsD[5],
                                        const double oldD[5], const double rsD[5], double q[5],
                                        double rsNew[5], bool &wr) {
  const A adtv(adtvD), grk(ph.grk[is - 1]);
  (void)grk;
  bool known = true;
  const bool wray = ph.rkScheme == 2, rk4 = ph.rkScheme == 1;
  wr = wray ? is < 3 : rk4 && is != ph.nSteps;
#pragma unroll
  for (int j = 0; j < 5; ++j) {
    const A rhs(rhsD[j]), old(oldD[j]), rs(rsD[j]);
    A d = rhs, r = rhs;
    if (wray) {
      if (is > 1) d = rhs - prod(grk, rs);
    } else if (rk4 && is > 1) {
      if (is == ph.nSteps) d = rhs + rs;
      else r = rs + prod(grk, rhs);
    }
    const A n = old - prod(adtv, d);
    known = known && !unknown(n) && !(wr && unknown(r));
    q[j] = value(n);
    rsNew[j] = value(r);
  }
  return known;
}
// The update with integer products, repeated on plain doubles where a product
// is outside their range.
__device__ __forceinline__ bool rk_cell64(const Phys &ph, int is, double adtv, const double rhs[5],
                                          const double old[5], const double rs[5], double q[5],
                                          double rsNew[5]) {
  bool wr;
  if (!rk_cell<Sd>(ph, is, adtv, rhs, old, rs, q, rsNew, wr))
    rk_cell<double>(ph, is, adtv, rhs, old, rs, q, rsNew, wr);
  return wr;
}
// 1/rho, the pressure (libflu/RFLU_SetDependentVars.F90:256-287 in the
// reference's operation order) and the velocities of a conserved vector.
template <typename A>
__device__ __forceinline__ bool eos_cell(const Phys &ph, const double qD[5], double &irD, double &pD,
                                         double vel[3]) {
  const A rr(qD[0]), ir = A(1) / rr;
  const A q1(qD[1]), q2(qD[2]), q3(qD[3]);
  const A Eo = prod(ir, A(qD[4]));
  const A Vm2 = prod(prod(ir, ir), prod(q1, q1) + prod(q2, q2) + prod(q3, q3));
  const A p = prod(prod(A(ph.gvG - 1.0), rr), Eo - scale<-1>(Vm2) - A(0));
  const A u = prod(ir, q1), v = prod(ir, q2), w = prod(ir, q3);
  irD = value(ir);
  pD = value(p);
  vel[0] = value(u);
  vel[1] = value(v);
  vel[2] = value(w);
  return !(unknown(ir) || unknown(p) || unknown(u) || unknown(v) || unknown(w));
}
__device__ __forceinline__ void eos_cell64(const Phys &ph, const double q[5], double &ir, double &p,
                                           double vel[3]) {
  if (!eos_cell<Sd>(ph, q, ir, p, vel)) eos_cell<double>(ph, q, ir, p, vel);
}

// Split-path gather + update: the FP32 face fluxes summed in FP64, the RK
// update of the FP64 conserved state (libfloflu/RkUpdateGeneric.F90:229-314)
// and the EOS (libflu/RFLU_SetDependentVars.F90:256-287) in FP64, with the
// reference's operation order except that a*dt/V is a*dt times the stored
// 1/V.  The FP32 record (rho, u, v, w, p) for the next stage's gathers is
// rounded from the FP64 values.  AfterUpdateMP's checks
// (libfloflu/AfterUpdateMP.F90:134-136) run only on cells they can act on
// (checks_can_act).
__device__ __forceinline__ void gather_update_split(const RegionDev<float> &g, int c,
                                                    const StepArgs &a) {
  const int N = g.nCells;
  const Phys &ph = g.ph;
  const int is = a.istage;
  double q[5], rsOld[5];
  float r[8];
  double ivol = 0.0;
  if (a.update) {  // own-cell loads first: independent of the flux gathers
#pragma unroll
    for (int j = 0; j < 5; ++j) q[j] = lds_rw<RF_HINT_U>(g.cv + (size_t)j * N + c);
    const bool hist = is > 1 && ph.rkScheme != 3;
#pragma unroll
    for (int j = 0; j < 5; ++j) rsOld[j] = hist ? lds_rw<RF_HINT_U>(g.rhsSum + (size_t)j * N + c) : 0.0;
    ld8_rw(g.rec + 8 * (size_t)c, r);
    ivol = lds<RF_HINT_U>(g.ivol + c);
  }
  double acc[5];
  face_sum64(g, g.flux, c, acc);
  if (a.writeRhs) {
#pragma unroll
    for (int j = 0; j < 5; ++j) g.rhs[(size_t)j * N + c] = acc[j];
  }
  if (!a.update) return;
  const double fac = a.useDeviceDt ? __ldcg(g.scal + 3 + is - 1) : ph.ark[is - 1] * a.dtHost;
  const double adtv = fac * ivol;
  const double grk = ph.grk[is - 1];
  double old[5];
  if (ph.rkScheme == 1) {  // RK4: cvOld saved at stage 1 only
#pragma unroll
    for (int j = 0; j < 5; ++j) {
      if (is == 1) {
        old[j] = q[j];
        g.cvOld[(size_t)j * N + c] = q[j];
      } else {
        old[j] = g.cvOld[(size_t)j * N + c];
      }
    }
  } else {  // Wray / Euler: cvOld = cv at every stage start
#pragma unroll
    for (int j = 0; j < 5; ++j) old[j] = q[j];
  }
  double *rs = g.rhsSum;
#pragma unroll
  for (int j = 0; j < 5; ++j) {
    const double rhs = acc[j];
    if (ph.rkScheme == 2) {
      if (is == 1) {
        q[j] = old[j] - adtv * rhs;
        rs[(size_t)j * N + c] = rhs;
      } else if (is == 2) {
        q[j] = old[j] - adtv * (rhs - grk * rsOld[j]);
        rs[(size_t)j * N + c] = rhs;
      } else {
        q[j] = old[j] - adtv * (rhs - grk * rsOld[j]);
      }
    } else if (ph.rkScheme == 1) {
      if (is == 1) {
        q[j] = old[j] - adtv * rhs;
        rs[(size_t)j * N + c] = rhs;
      } else if (is == ph.nSteps) {
        q[j] = old[j] - adtv * (rhs + rsOld[j]);
      } else {
        q[j] = old[j] - adtv * rhs;
        rs[(size_t)j * N + c] = rsOld[j] + grk * rhs;
      }
    } else {
      q[j] = old[j] - adtv * rhs;
    }
  }
  double ir;
  double p = eos_p(ph, q, ir);
  if (checks_can_act(q, p)) {
    double d[3];
    d[0] = p;
    d[1] = p / (q[0] * ph.gvR);
    d[2] = 0.0;
    const unsigned st = after_update(ph.gvR, ph.gvG, q, d);
    if (st) atomicOr(g.status, st);
    p = d[0];
    ir = 1.0 / q[0];
  }
#pragma unroll
  for (int j = 0; j < 5; ++j) g.cv[(size_t)j * N + c] = q[j];
  record_from_fp64(q, ir, p, r);
  st8(g.rec + 8 * (size_t)c, r);
}

// Face->cell residual gather in the reference accumulation order, then the
// RK update (libfloflu/RkUpdateGeneric.F90:229-314), EOS
// (libflu/RFLU_SetDependentVars.F90:256-287), AfterUpdate checks and
// Cons2Prim of the new state for the next stage.  With update = 0 only the
// residual is written (rfgpu_residual).
// SPLIT selects the split path's update at compile time (a run-time branch
// between the two FP32-flux updates costs the mixed path registers).
template <typename R, int SPLIT, typename RT>
__device__ __forceinline__ void update_tile(const RT &regs, const Tile *__restrict__ tiles,
                                            int nTiles, int t_, const StepArgs &a, int dist) {
  {
    const Tile tl = tile_at(regs, tiles, t_, blockDim.x);
    const RegionDev<R> &g = regs[tl.region];
    prefetch_ahead(t_, nTiles, dist, [&](int t) {
      const Tile tp = tile_at(regs, tiles, t, blockDim.x);
      prefetch_update_tile(regs[tp.region], tp.first);
    });
    const int c = tl.first + threadIdx.x;
    const int N = g.nCells;
    if (c >= N) return;
    if (c >= g.nAct) {  // virtual cell: ZeroDummyCellsMP, no update
      if (a.writeRhs) {
#pragma unroll
        for (int j = 0; j < 5; ++j) g.rhs[j * N + c] = 0.0;
      }
      return;
    }
    if constexpr (sizeof(R) == 4) {
      if constexpr (SPLIT)
        gather_update_split(g, c, a);
      else
        gather_update_mixed(g, c, a);
      return;
    }
    double acc[5];
    face_sum64(g, g.flux, c, acc);
    if (a.writeRhs) {
#pragma unroll
      for (int j = 0; j < 5; ++j) g.rhs[j * N + c] = acc[j];
    }
    if (!a.update) return;
    const Phys &ph = g.ph;
    const int is = a.istage;
    const double fac = a.useDeviceDt ? __ldcg(g.scal + 3 + is - 1) : ph.ark[is - 1] * a.dtHost;
    const double adtv = fac / g.vol[c];
    double q[5], old[5], rs[5];
    const bool hist = is > 1 && ph.rkScheme != 3;
#pragma unroll
    for (int j = 0; j < 5; ++j) {
      q[j] = g.cv[j * N + c];
      rs[j] = hist ? g.rhsSum[j * N + c] : 0.0;
    }
    if (ph.rkScheme == 1) {  // RK4: cvOld saved at stage 1 only
      if (is == 1) {
#pragma unroll
        for (int j = 0; j < 5; ++j) {
          old[j] = q[j];
          g.cvOld[j * N + c] = q[j];
        }
      } else {
#pragma unroll
        for (int j = 0; j < 5; ++j) old[j] = g.cvOld[j * N + c];
      }
    } else {  // Wray / Euler: cvOld = cv at every stage start
#pragma unroll
      for (int j = 0; j < 5; ++j) old[j] = q[j];
    }
    double rsNew[5];
    if (rk_cell64(ph, is, adtv, acc, old, rs, q, rsNew)) {
#pragma unroll
      for (int j = 0; j < 5; ++j) g.rhsSum[j * N + c] = rsNew[j];
    }
    // EOS
    const double gc = ph.gvR, gg = ph.gvG;
    double d[3], ir, vel[3];
    eos_cell64(ph, q, ir, d[0], vel);
    d[1] = d[0] / (q[0] * gc);
    d[2] = sqrt(gg * gc * d[1]);
    if (checks_can_act(q, d[0])) {
      const unsigned st = after_update(gc, gg, q, d);
      if (st) atomicOr(g.status, st);
    }
#pragma unroll
    for (int j = 0; j < 5; ++j) g.cv[j * N + c] = q[j];
    g.dv[c] = d[0];
    g.dv[N + c] = d[1];
    g.dv[2 * N + c] = d[2];
    if constexpr (sizeof(R) == 8) {
      double r[8] = {q[0], vel[0], vel[1], vel[2], d[0]};
      trip_velocity(ph, ir, r);
      st8(g.rec + 8 * (size_t)c, r);
    }
  }
}

template <typename R, int BS, int SPLIT>
__global__ void __launch_bounds__(BS) k_gather_update(const RegionDev<R> *__restrict__ regs,
                                                      const Tile *__restrict__ tiles,
                                                      int nTiles, StepArgs a, int pfDist) {
  const int dist = (int)gridDim.x < nTiles ? (int)gridDim.x : pfDist;
  RF_TILE_LOOP(pdl_wait(), nTiles) update_tile<R, SPLIT>(regs, tiles, nTiles, t_, a, dist);
}
// One region, mixed: 10 blocks of 128 asked for (48 registers).  Update pass of
// 12.6 M tets, 1.57 M tets and the 2.48 M-cell box: 0.591, 0.081, 0.100 ms; the
// compiler's 64 registers 0.601, 0.086, 0.122; 9 blocks 0.599, 0.081, 0.106; 11
// blocks 0.623, 0.084, 0.095; the table version 0.583, 0.084, 0.116.
template <typename R, int BS, int SPLIT>
__global__ void __launch_bounds__(BS, sizeof(R) == 4 && SPLIT == 0 ? 10 * 128 / BS : 0)
    k_gather_update(const __grid_constant__ OneRegion<R> regs, const Tile *__restrict__ tiles,
                    int nTiles, StepArgs a, int pfDist) {
  const int dist = (int)gridDim.x < nTiles ? (int)gridDim.x : pfDist;
  RF_TILE_LOOP(pdl_wait(), nTiles) update_tile<R, SPLIT>(regs, tiles, nTiles, t_, a, dist);
}

// Mixed path transfers: the host's Fortran images cv(5,N) / dv(3,N), copied
// by DMA into device staging buffers, are converted in one pass per direction
// and chunk, fusing the numbering, layout and precision conversions (upload:
// cons -> record with the EOS of k_prim, float-float split; download:
// float-float join, FP64 dv).  One thread per device cell of the chunk's list
// (its cells in ascending device order), so the device-side state is read and
// written coalesced and the Fortran images are addressed by host cell; one
// thread per host cell scattered the state's ten SoA rows instead.  Kernels
// reading or writing page-locked host memory directly over the CPU-GPU link
// were measured slower than the DMA copies (32 against 20 ms per end-to-end
// step).
template <typename R, int SPLIT>
__global__ void k_upload_list(const RegionDev<R> *__restrict__ regs, const int *__restrict__ list,
                              int n, const double *__restrict__ cvH, const double *__restrict__ dvH) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const RegionDev<R> &g = regs[0];
  const int c = list[i];
  const int h = g.cellOld ? g.cellOld[c] : c;
  double q[5];
#pragma unroll
  for (int j = 0; j < 5; ++j) q[j] = cvH[5 * (size_t)h + j];
  if constexpr (sizeof(R) == 4) {
    if constexpr (SPLIT)
      state_from_fp64_split(g, c, q, dvH ? dvH + 3 * (size_t)h : nullptr);
    else
      state_from_fp64_ff(g, c, q, dvH ? dvH + 3 * (size_t)h : nullptr);
  }
}

template <typename R, int SPLIT>
__global__ void k_download_list(const RegionDev<R> *__restrict__ regs, const int *__restrict__ list,
                                int n, double *__restrict__ cvH, double *__restrict__ dvH) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const RegionDev<R> &g = regs[0];
  const int c = list[i];
  const int h = g.cellOld ? g.cellOld[c] : c;
  const int N = g.nCells;
  double q[5];
  if constexpr (SPLIT) {
#pragma unroll
    for (int j = 0; j < 5; ++j) q[j] = g.cv[(size_t)j * N + c];
  } else {
#pragma unroll
    for (int j = 0; j < 5; ++j)
      q[j] = widen_f32(g.cvF[(size_t)j * N + c]) + widen_f32(g.cvF[(size_t)(5 + j) * N + c]);
  }
  if (cvH) {
#pragma unroll
    for (int j = 0; j < 5; ++j) cvH[5 * (size_t)h + j] = q[j];
  }
  if (dvH && SPLIT) {  // split path: the EOS of its update
    const double gc = g.ph.gvR, gg = g.ph.gvG;
    double ir;
    const double p = eos_p(g.ph, q, ir);
    const double T = p / (q[0] * gc);
    dvH[3 * (size_t)h] = p;
    dvH[3 * (size_t)h + 1] = T;
    dvH[3 * (size_t)h + 2] = sqrt(gg * gc * T);
  } else if (dvH) {
    // FP64 EOS of the joined pairs with one division (by rho) instead of two:
    // the conversion is FP64-pipe bound
    const double gc = g.ph.gvR, gg = g.ph.gvG;
    const double m2 = fma(q[3], q[3], fma(q[2], q[2], q[1] * q[1]));
    const double ir = 1.0 / q[0];
    const double p = (gg - 1.0) * (q[4] - 0.5 * m2 * ir);
    const double T = p * ir * g.ph.gvRinv;
    dvH[3 * (size_t)h] = p;
    dvH[3 * (size_t)h + 1] = T;
    dvH[3 * (size_t)h + 2] = sqrt(gg * gc * T);
  }
}

// ---- time step (standalone pass): per-cell gather of cell_dt, block minimum,
// then an atomic minimum on the bit pattern (dt > 0: the IEEE order equals
// the unsigned integer order).
template <typename R>
__global__ void __launch_bounds__(128) k_dt_cell(const RegionDev<R> *__restrict__ regs,
                                                 const Tile *__restrict__ tiles, int nTiles) {
  __shared__ unsigned long long smin[32];
  RF_TILE_LOOP(pdl_wait(), nTiles) {
    const Tile tl = tiles[t_];
    const RegionDev<R> &g = regs[tl.region];
    const int c = tl.first + threadIdx.x;
    unsigned long long bits = 0x7FF0000000000000ull;  // +inf
    if (c < g.nAct) {
      R r0[8];
      ld8(g.rec + 8 * (size_t)c, r0);
      bits = (unsigned long long)__double_as_longlong(cell_dt(g, c, r0));
    }
    dt_block_min<R>(bits, smin, g.dtBits);
  }
}

template <typename R>
__global__ void __launch_bounds__(128) k_dt_finalize(const RegionDev<R> *__restrict__ regs,
                                                     int nRegions, int coupled, DtArgs a) {
  __shared__ unsigned long long smin[32];
  if (pdl_wait() == 0) dt_finalize_block<R>(regs, nRegions, coupled, a, smin);
}
template <typename R>
void launch_dt_finalize(const RegionDev<R> *regs, const Work &w, const DtArgs &a,
                        cudaStream_t s) {
  launch_pdl(k_dt_finalize<R>, 1, 128, s, regs, w.nRegions, w.coupled, a);
}

// ---- launchers ----------------------------------------------------------------

template <typename R>
void launch_prim(const RegionDev<R> *regs, const Work &w, int computeDv, cudaStream_t s) {
  int grid = w.grid > 0 && w.grid < w.nCellTiles ? w.grid : w.nCellTiles;
  if (grid > 0) k_prim<R><<<grid, w.block, 0, s>>>(regs, w.cellTiles, w.nCellTiles, computeDv);
}

#define RF_MARK(kind, phase) \
  if (prof) prof->mark(prof->ctx, (kind), (phase), s)

inline int sm_count() {
  int dev = 0, n = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
  return n;
}

// Blocks of `kernel` (`threads` per block) resident on the whole device at
// once: the prefetch distance in tiles.
template <typename K>
int resident_blocks(K kernel, int threads = 128) {
  const int nsm = sm_count();
  int per = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, threads, 0);
  return per > 0 && nsm > 0 ? per * nsm : 1;
}

template <typename R>
void launch_weno_xyz(const RegionDev<R> *regs, const Work &w, cudaStream_t s);

// ---- tuned launches: block size (and faces per thread) picked at run time
// from the Work's launch shapes, one template instance per shape -------------
inline int grid_for(int cap, int nTiles) { return cap > 0 && cap < nTiles ? cap : nTiles; }

// A launch that may start while its predecessor in the stream runs (pdl_wait).
template <typename... P, typename... A>
void launch_pdl(void (*kernel)(P...), dim3 grid, dim3 block, cudaStream_t s, const A &...args) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c{};
  c.gridDim = grid;
  c.blockDim = block;
  c.stream = s;
  c.attrs = &at;
  c.numAttrs = 1;
  cudaLaunchKernelEx(&c, kernel, static_cast<P>(args)...);
}

// The region argument of a launch: the descriptor where the Work is one region
// (its own tile lists are then consecutive tiles), else the table.
template <bool ONE = true, typename R, typename F>
void with_regions(const RegionDev<R> *regs, const Work &w, const Tile *tiles, F f) {
  if constexpr (ONE) {  // other launch shapes than the default keep the table
    if (w.one) {
      const bool own = tiles == w.cellTiles || tiles == w.faceTiles || tiles == w.bfaceTiles;
      f(OneRegion<R>{*static_cast<const RegionDev<R> *>(w.one)}, own ? nullptr : tiles);
      return;
    }
  }
  f(regs, tiles);
}

template <typename R, int F, int BS>
void grad_launch(const RegionDev<R> *regs, const Work &w, const Tile *tiles, int nTiles, int cap,
                 cudaStream_t s) {
  if constexpr (sizeof(R) == 8) {
    const int per = BS / 32, n = grid_for(cap, nTiles * per);
    if (n <= 0) return;
    const bool five = n == nTiles * per && n < kGrad64Rows;
    with_regions(regs, w, tiles, [&](const auto &r, const Tile *t) {
      using RA = std::decay_t<decltype(r)>;
      launch_pdl(static_cast<void (*)(RA, const Tile *, int, int)>(k_grad_lim64<F>),
                 dim3(n, five ? 5 : 1), dim3(32, five ? 1 : 5), s, r, t, nTiles, per);
    });
  } else {
    const int grid = grid_for(cap, nTiles);
    if (grid <= 0) return;
    if constexpr (BS == 128) {
      if (w.one && tiles == w.cellTiles && cap == 0 && nTiles < kFewTiles) {
        const RegionDev<R> &d = *static_cast<const RegionDev<R> *>(w.one);
        const int n = (d.nCells + kFewBlock - 1) / kFewBlock;
        launch_pdl(k_grad_few<R, F>, n, kFewBlock, s, OneRegion<R>{d}, n);
        return;
      }
    }
    with_regions<BS == 128>(regs, w, tiles, [&](const auto &r, const Tile *t) {
      using RA = std::decay_t<decltype(r)>;
      launch_pdl(static_cast<void (*)(RA, const Tile *, int)>(k_grad_lim<R, F, BS>), grid, BS, s, r,
                 t, nTiles);
    });
  }
}

template <typename R>
void launch_grad_tuned(const RegionDev<R> *regs, const Work &w, int fuseDt, cudaStream_t s) {
  const bool tuned = w.gradTiles != nullptr;
  const Tile *t = tuned ? w.gradTiles : w.cellTiles;
  const int n = tuned ? w.nGradTiles : w.nCellTiles;
  const int bs = tuned ? w.gradBlock : 128;
  if (bs == 64) {
    if (fuseDt) grad_launch<R, 1, 64>(regs, w, t, n, w.grid, s);
    else grad_launch<R, 0, 64>(regs, w, t, n, w.grid, s);
  } else if (bs == 256) {
    if (fuseDt) grad_launch<R, 1, 256>(regs, w, t, n, w.grid, s);
    else grad_launch<R, 0, 256>(regs, w, t, n, w.grid, s);
  } else {
    if (fuseDt) grad_launch<R, 1, 128>(regs, w, t, n, w.grid, s);
    else grad_launch<R, 0, 128>(regs, w, t, n, w.grid, s);
  }
}

template <typename R>
void launch_face64(const RegionDev<R> *regs, const Work &w, const Tile *tiles, int nTiles, int grid,
                   int block, int stride, cudaStream_t s) {
  with_regions(regs, w, tiles, [&](const auto &r, const Tile *t) {
    using RA = std::decay_t<decltype(r)>;
    const auto k = static_cast<void (*)(RA, const Tile *, int, int, int)>(k_face_flux64<R>);
    static const int pf = resident_blocks(k, 128);
    launch_pdl(k, grid, block, s, r, t, nTiles, pf, stride);
  });
}

template <typename R, int BS, int FPT>
void face_launch(const RegionDev<R> *regs, const Work &w, const Tile *tiles, int nTiles,
                 cudaStream_t s) {
  const int grid = grid_for(w.grid, nTiles);
  if (grid <= 0) return;
  if constexpr (sizeof(R) == 8) {
    launch_face64<R>(regs, w, tiles, nTiles, grid, BS < 128 ? BS : 128, BS * FPT, s);
  } else {
    with_regions<BS == 128 && FPT == 1>(regs, w, tiles, [&](const auto &r, const Tile *t) {
      using RA = std::decay_t<decltype(r)>;
      const auto k = static_cast<void (*)(RA, const Tile *, int, int)>(k_face_flux<R, BS, FPT>);
      static const int pf = resident_blocks(k, BS);
      launch_pdl(k, grid, BS, s, r, t, nTiles, pf);
    });
  }
}

// The merged launch pays for single regions of every size (ms per step,
// separate -> merged: 512 cells 0.0457 -> 0.0353 a residual, 4,000-cell tube
// FP64 0.166 -> 0.131, 10,000 tets 0.082 -> 0.071, 197,000 tets 0.330 -> 0.313,
// 6.75 M tets 4.571 -> 4.547, split 6.130 -> 6.075, 12.6 M tets 8.099 -> 8.072,
// split 11.04 -> 10.95; FP64 8.4 M tets 81.52 -> 81.59, no difference) and for
// FP64 batches (1,500 face tiles 0.726 -> 0.687, 35,000 12.79 -> 12.71).  The
// FP32-flux kernel over a batch's table holds more registers, which costs large
// batches more than a launch: 35,000 tiles 1.635 -> 1.626, split 2.432 -> 2.424,
// but 71,000 tiles 3.127 -> 3.133, split 4.728 -> 4.744, and 314,000 tiles 14.37
// -> 14.69.
constexpr int kMergeBatchTiles = 50000;
template <typename R>
bool merge_pays(const Work &w) {
  return w.one || sizeof(R) == 8 || w.nFaceTiles < kMergeBatchTiles;
}
template <typename R>
void merged_launch(const RegionDev<R> *regs, const Work &w, FluxExtra x, cudaStream_t s) {
  const int grid = grid_for(w.grid, w.nFaceTiles + x.nBFace + x.dt);
  with_regions(regs, w, w.faceTiles, [&](const auto &r, const Tile *t) {
    using RA = std::decay_t<decltype(r)>;
    const auto k =
        static_cast<void (*)(RA, const Tile *, int, int, const FluxExtra)>(k_flux_merged<R>);
    static const int pf = resident_blocks(k, 128);
    if (!t) x.bface = nullptr;  // consecutive tiles as well
    launch_pdl(k, grid, 128, s, r, t, w.nFaceTiles, pf, x);
  });
}

template <typename R>
void launch_faces_tuned(const RegionDev<R> *regs, const Work &w, cudaStream_t s) {
  const int bs = w.faceBlock ? w.faceBlock : 128, fpt = w.facesPerThread ? w.facesPerThread : 1;
  if (bs == 64) {
    if (fpt == 2) face_launch<R, 64, 2>(regs, w, w.faceTiles, w.nFaceTiles, s);
    else face_launch<R, 64, 1>(regs, w, w.faceTiles, w.nFaceTiles, s);
  } else if (bs == 256) {
    if (fpt == 2) face_launch<R, 256, 2>(regs, w, w.faceTiles, w.nFaceTiles, s);
    else face_launch<R, 256, 1>(regs, w, w.faceTiles, w.nFaceTiles, s);
  } else {
    if (fpt == 2) face_launch<R, 128, 2>(regs, w, w.faceTiles, w.nFaceTiles, s);
    else face_launch<R, 128, 1>(regs, w, w.faceTiles, w.nFaceTiles, s);
  }
}

template <typename R, int BS, int SPLIT>
void update_launch_k(const RegionDev<R> *regs, const Work &w, const Tile *tiles, int nTiles,
                     const StepArgs &a, cudaStream_t s) {
  const int grid = grid_for(w.grid, nTiles);
  if (grid <= 0) return;
  with_regions<BS == 128>(regs, w, tiles, [&](const auto &r, const Tile *t) {
    using RA = std::decay_t<decltype(r)>;
    const auto k =
        static_cast<void (*)(RA, const Tile *, int, StepArgs, int)>(k_gather_update<R, BS, SPLIT>);
    static const int pf = resident_blocks(k, BS);
    launch_pdl(k, grid, BS, s, r, t, nTiles, a, pf);
  });
}
template <typename R, int BS>
void update_launch(const RegionDev<R> *regs, const Work &w, const Tile *tiles, int nTiles,
                   const StepArgs &a, cudaStream_t s) {
  if constexpr (sizeof(R) == 4) {
    if (w.split) return update_launch_k<R, BS, 1>(regs, w, tiles, nTiles, a, s);
  }
  update_launch_k<R, BS, 0>(regs, w, tiles, nTiles, a, s);
}

template <typename R>
void launch_update_tuned(const RegionDev<R> *regs, const Work &w, const StepArgs &a,
                         cudaStream_t s) {
  const bool tuned = w.updTiles != nullptr;
  const Tile *t = tuned ? w.updTiles : w.cellTiles;
  const int n = tuned ? w.nUpdTiles : w.nCellTiles;
  const int bs = tuned ? w.cellBlock : 128;
  if (bs == 64) update_launch<R, 64>(regs, w, t, n, a, s);
  else if (bs == 256) update_launch<R, 256>(regs, w, t, n, a, s);
  else update_launch<R, 128>(regs, w, t, n, a, s);
}

// ---- one launch per RK stage ---------------------------------------------------
template <typename R, typename RT>
__device__ __forceinline__ void weno_tile(const RT &regs, const Tile *__restrict__ tiles, int t_);

// Grid-wide barrier of the persistent stage kernel, a cooperative launch (so
// every block is resident).  Thread 0 of each block arrives; the last arrival
// clears the count and releases the others by advancing the generation.  Every
// wait is bounded by `spin` SM clock cycles: one that runs out sets bit 0 of
// err, and every block returns as soon as it sees err set after a barrier, so
// the kernel ends and the host reads RFGPU_ERR_TIMEOUT.
__device__ __forceinline__ bool grid_sync(GridBar *b, unsigned expect, long long spin) {
  __syncthreads();
  if (threadIdx.x == 0) {
    volatile unsigned *vgen = &b->gen;
    const unsigned g0 = *vgen;
    __threadfence();
    if (atomicAdd(&b->count, 1u) + 1u == expect) {
      atomicExch(&b->count, 0u);
      __threadfence();
      atomicAdd(&b->gen, 1u);
    } else {
      const long long t0 = clock64();
      while (*vgen == g0) {
        if (clock64() - t0 > spin) {
          atomicOr(&b->err, 1u);
          break;
        }
        __nanosleep(32);
      }
    }
    __threadfence();
  }
  __syncthreads();
  return *(volatile unsigned *)&b->err == 0;
}

// A whole RK stage of a Work (one region or a batch) in one launch: the
// gradient pass over every cell tile, the WENO-XYZ pass (RECONST 2), the
// time-step finalisation (stage 1 of a step), the interior and boundary face
// passes, the gather + update, and for a coupled batch the halo exchange,
// separated by grid-wide barriers.  The per-tile work is the device code the
// one-pass-per-launch kernels run.  Arrays one phase writes and a later one
// gathers through the read-only path (gradients, face fluxes) are first read
// after the barrier that follows their writes, so no stale copy can be cached;
// scalars and halo sources are read through L2.
#ifndef RF_COOP_MINB
#define RF_COOP_MINB 6  // resident blocks per SM requested for the persistent stage kernel
#endif
template <typename R, int SPLIT>
__global__ void __launch_bounds__(128, (sizeof(R) == 4) ? RF_COOP_MINB : 4)
    k_stage_coop(const RegionDev<R> *__restrict__ regs, Work w, StepArgs a, int grad, int weno) {
  __shared__ unsigned long long smin[32];
  const unsigned expect = gridDim.x + (unsigned)w.barExtra;
  GridBar *bar = w.bar;
  const long long spin = w.barSpin;
  if (grad) {
    if constexpr (sizeof(R) == 8) {
      // a warp per slice and variable, the next slice pulled into L2 meanwhile.
      // A step in persistent stages, a thread taking its cell's variables in
      // turn -> this: 4,000 cells 340 -> 215 us, 64,000 632 -> 604, 10,000
      // tets 532 -> 392, 663,000 tets 7.81 -> 6.99 ms.
      const int warps = gridDim.x * 4;  // 128-cell tiles: 4 slices of 5 variables each
      for (int i = blockIdx.x * 4 + (threadIdx.x >> 5); i < w.nCellTiles * 20; i += warps) {
        if ((i + warps) % 5 == 0 && i + warps < w.nCellTiles * 20) {
          const Tile tp = w.cellTiles[(i + warps) / 20];
          prefetch_grad_slice(regs[tp.region], (tp.first >> 5) + (i + warps) / 5 % 4, true);
        }
        if (a.fuseDt)
          grad64_slice<1>(regs, w.cellTiles, i / 5, 4, i % 5);
        else
          grad64_slice<0>(regs, w.cellTiles, i / 5, 4, i % 5);
      }
    } else {
      for (int t = blockIdx.x; t < w.nCellTiles; t += gridDim.x) {
        if (a.fuseDt)
          grad_tile<R, 1>(regs, w.cellTiles, t, smin);
        else
          grad_tile<R, 0>(regs, w.cellTiles, t, smin);
      }
    }
    if (!grid_sync(bar, expect, spin)) return;
    if (weno) {
      for (int t = blockIdx.x; t < w.nCellTiles; t += gridDim.x) weno_tile<R>(regs, w.cellTiles, t);
      if (!grid_sync(bar, expect, spin)) return;
    }
    if (a.fuseDt) {
      if (blockIdx.x == 0) dt_finalize_block<R>(regs, w.nRegions, w.coupled, a.dt, smin);
      if (!grid_sync(bar, expect, spin)) return;
    }
  }
  for (int t = blockIdx.x; t < w.nFaceTiles; t += gridDim.x)
    face_tile<R, 128, 1>(regs, w.faceTiles, w.nFaceTiles, t, gridDim.x);
  for (int t = blockIdx.x; t < w.nBFaceTiles; t += gridDim.x) bface_tile<R>(regs, w.bfaceTiles, t);
  if (!grid_sync(bar, expect, spin)) return;
  for (int t = blockIdx.x; t < w.nCellTiles; t += gridDim.x)
    update_tile<R, SPLIT>(regs, w.cellTiles, w.nCellTiles, t, a, gridDim.x);
  if (w.nHalo > 0 && a.update) {
    if (!grid_sync(bar, expect, spin)) return;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < w.nHalo; i += gridDim.x * blockDim.x) {
      const HaloLink l = w.halo[i];
      halo_cell(regs[l.srcRegion], l.srcCell, regs[l.dstRegion], l.dstCell);
    }
  }
}

template <typename R, int SPLIT>
void coop_launch(const RegionDev<R> *regs, const Work &w, const StepArgs &a, int grad, int weno,
                 cudaStream_t s) {
  static const int resident = resident_blocks(k_stage_coop<R, SPLIT>, 128);
  int grid = w.nCellTiles > w.nFaceTiles ? w.nCellTiles : w.nFaceTiles;
  // FP64: at least a block per SM while the gradient pass has slices and
  // variables for it.  4,000 cells, a block per tile and variable up to the
  // resident ones: 226 against 215 us, 385 against 305 with WENO, whose few
  // tiles then share SMs.
  if (sizeof(R) == 8 && grad) grid = std::max(grid, std::min(5 * w.nCellTiles, sm_count()));
  if (w.nBFaceTiles > grid) grid = w.nBFaceTiles;
  if (w.grid > 0 && w.grid < grid) grid = w.grid;
  if (grid > resident) grid = resident;
  if (grid < 1) grid = 1;
  cudaMemsetAsync(w.bar, 0, 2 * sizeof(unsigned), s);  // count and generation; err stays
  Work wc = w;
  StepArgs ac = a;
  void *args[] = {(void *)&regs, (void *)&wc, (void *)&ac, (void *)&grad, (void *)&weno};
  cudaLaunchCooperativeKernel((const void *)k_stage_coop<R, SPLIT>, dim3(grid), dim3(128), args, 0,
                              s);
}

template <typename R>
void launch_stage(const RegionDev<R> *regs, const Work &w, const StepArgs &a, cudaStream_t s,
                  long long *launches, int spaceOrder, int reconst, const Prof *prof,
                  int parts) {
  if (w.coop && parts == SP_ALL && w.bar) {
    const int grad = spaceOrder > 1 && w.nCellTiles > 0;
    const int weno = grad && reconst == 2;
    RF_MARK(KP_STAGE, 0);
    if constexpr (sizeof(R) == 4) {
      if (w.split)
        coop_launch<R, 1>(regs, w, a, grad, weno, s);
      else
        coop_launch<R, 0>(regs, w, a, grad, weno, s);
    } else {
      coop_launch<R, 0>(regs, w, a, grad, weno, s);
    }
    RF_MARK(KP_STAGE, 1);
    if (launches) *launches += 1;
    return;
  }
  long long n = 0;
  const bool hasGrad = spaceOrder > 1 && w.nCellTiles > 0;
  const bool grad = hasGrad && (parts & SP_GRADIENT);
  const bool flux = parts & SP_FLUX, upd = parts & SP_UPDATE;
  if (grad) {
    RF_MARK(KP_GRADIENT, 0);
    launch_grad_tuned<R>(regs, w, a.fuseDt, s);
    RF_MARK(KP_GRADIENT, 1);
    ++n;
  }
  if (hasGrad && flux && reconst == 2) {  // after every cell's gradient
    RF_MARK(KP_LIMITER, 0);
    launch_weno_xyz<R>(regs, w, s);
    RF_MARK(KP_LIMITER, 1);
    ++n;
  }
  // one launch for the independent flux passes; separate ones while the
  // profiler times each class, or when the caller launches the interior faces
  const bool dt = a.fuseDt && hasGrad && flux, bface = flux && w.nBFaceTiles > 0;
  const bool faces = flux && !(parts & SP_NOFACE) && w.nFaceTiles > 0;
  const bool tuned = w.faceBlock != 0 && (w.faceBlock != 128 || w.facesPerThread != 1);
  const bool merge = faces && !prof && !tuned && (dt || bface) && merge_pays<R>(w);
  if (dt && !merge) {
    RF_MARK(KP_DT_FINAL, 0);
    launch_dt_finalize<R>(regs, w, a.dt, s);
    RF_MARK(KP_DT_FINAL, 1);
    ++n;
  }
  if (faces) {
    RF_MARK(KP_FACE_FLUX, 0);
    if (merge)
      merged_launch<R>(regs, w, FluxExtra{w.bfaceTiles, bface ? w.nBFaceTiles : 0, dt, w.nRegions,
                                          w.coupled, a.dt}, s);
    else
      launch_faces_tuned<R>(regs, w, s);
    RF_MARK(KP_FACE_FLUX, 1);
    ++n;
  }
  if (bface && !merge) {
    RF_MARK(KP_BFACE_FLUX, 0);
    launch_bface_tiles<R>(regs, w, w.bfaceTiles, w.nBFaceTiles, s);
    RF_MARK(KP_BFACE_FLUX, 1);
    ++n;
  }
  if (upd && w.nCellTiles > 0) {
    RF_MARK(KP_GATHER_UPDATE, 0);
    launch_update_tuned<R>(regs, w, a, s);
    RF_MARK(KP_GATHER_UPDATE, 1);
    ++n;
  }
  if (upd && w.nHalo > 0 && a.update) {  // coupled regions: virtual cells from their owners
    RF_MARK(KP_HALO, 0);
    launch_pdl(k_halo<R>, (w.nHalo + 127) / 128, 128, s, regs, w.halo, w.nHalo);
    RF_MARK(KP_HALO, 1);
    ++n;
  }
  if (launches) *launches += n;
}

template <typename R>
void launch_dt(const RegionDev<R> *regs, const Work &w, const DtArgs &a, cudaStream_t s,
               long long *launches, const Prof *prof) {
  auto gsz = [&](int nt) { return w.grid > 0 && w.grid < nt ? w.grid : nt; };
  long long n = 0;
  if (w.nCellTiles > 0) {
    RF_MARK(KP_DT_CELL, 0);
    launch_pdl(k_dt_cell<R>, gsz(w.nCellTiles), w.block, s, regs, w.cellTiles, w.nCellTiles);
    RF_MARK(KP_DT_CELL, 1);
    ++n;
  }
  RF_MARK(KP_DT_FINAL, 0);
  launch_dt_finalize<R>(regs, w, a, s);
  RF_MARK(KP_DT_FINAL, 1);
  ++n;
  if (launches) *launches += n;
}

template <typename R>
void launch_step(const RegionDev<R> *regs, const Work &w, const DtArgs &da, int nStages,
                 cudaStream_t s, long long *launches, int spaceOrder, int reconst,
                 const Prof *prof) {
  const bool fuse = spaceOrder > 1 && w.nCellTiles > 0;
  if (!fuse) launch_dt<R>(regs, w, da, s, launches, prof);
  for (int is = 1; is <= nStages; ++is) {
    StepArgs sa{is, 1, 0.0, 0, 1, (fuse && is == 1) ? 1 : 0, da};
    launch_stage<R>(regs, w, sa, s, launches, spaceOrder, reconst, prof);
  }
}

// RECONST 2 (CellGradientsMP.F90:217-222): RFLU_WENOGradCellsXYZFast_3D
// (modflu/RFLU_ModWENO.F90:1402-1588, the 3-D branch of the wrapper at
// :1615-1668) then RFLU_LimitGradCellsSimple (modflu/RFLU_ModLimiters.F90:
// 793-921), one thread per cell.  Every gradient component becomes the
// average of the cell's and its stencil members' unweighted components
// (gradRaw) weighted by s = 1/(g^2 + 1e-15), the cell first and the members in
// stored order, sum(s g) / sum(s); then the gradient of density and pressure
// (the positive variables, libflu/RFLU_SetVarInfo.F90:140-144) is zeroed when
// var + grad . (fc - xc) is not positive at one of the cell's faces, interior
// or boundary (the result does not depend on the face order).  Regions that
// do not use RECONST 2 skip their tiles.
template <typename R, typename RT>
__device__ __forceinline__ void weno_tile(const RT &regs, const Tile *__restrict__ tiles, int t_) {
  {
    const Tile tl = tile_at(regs, tiles, t_, blockDim.x);
    const RegionDev<R> &g = regs[tl.region];
    if (!g.gradRaw) return;
    const int c = tl.first + threadIdx.x;
    if (c >= g.nCells) return;
    const R eps = R(1.0E-15);
    // the weight 1/(g^2 + 1e-15): IEEE division on the FP64 path; on the
    // mixed path optionally the hardware reciprocal (it only weights an average)
    auto weight = [&](R t) -> R {
      if constexpr (sizeof(R) == 4 && RF_WENO_FASTRCP) return rcp_ftz(t * t + eps);
      else return R(1) / (t * t + eps);
    };
    R ss[15], acc[15];
    const long long base = g.stOff[c >> 5] + (c & 31);
    const int n = g.stCnt[c];
    if constexpr (sizeof(R) == 8) {
      // weights and products precomputed by the gradient pass: sums only
      R w[16];
      ld16(g.gradRaw + 32 * (size_t)c, w);
#pragma unroll
      for (int k = 0; k < 15; ++k) ss[k] = w[k];
      ld16(g.gradRaw + 32 * (size_t)c + 16, w);
#pragma unroll
      for (int k = 0; k < 15; ++k) acc[k] = w[k];
      for (int m = 0; m < n; ++m) {
        const R *row = g.gradRaw + 32 * (size_t)g.stIdx[base + (long long)m * kSlice];
        ld16(row, w);
#pragma unroll
        for (int k = 0; k < 15; ++k) ss[k] = ss[k] + w[k];
        ld16(row + 16, w);
#pragma unroll
        for (int k = 0; k < 15; ++k) acc[k] = acc[k] + w[k];
      }
    } else {
      {
        R g0[16];
        ld16(g.gradRaw + 16 * (size_t)c, g0);
#pragma unroll
        for (int k = 0; k < 15; ++k) {
          const R t = g0[k];
          ss[k] = weight(t);
          acc[k] = ss[k] * t;
        }
      }
      auto member = [&](const R gm[16]) {
#pragma unroll
        for (int k = 0; k < 15; ++k) {
          const R t = gm[k];
          const R sm = weight(t);
          ss[k] = ss[k] + sm;
          acc[k] = acc[k] + sm * t;
        }
      };
      {
        // members in stored order, RF_WENO_U gathers issued together with the
        // next group's indices loaded while they are in flight
        constexpr int U = RF_WENO_U;
        const int nFull = n - n % U;
        int nx[U];
#pragma unroll
        for (int u = 0; u < U; ++u) nx[u] = u < n ? ld_index(g.stIdx + base + (long long)u * kSlice) : 0;
        for (int m = 0; m < nFull; m += U) {
          R gm[U][16];
#pragma unroll
          for (int u = 0; u < U; ++u) ld16(g.gradRaw + 16 * (size_t)nx[u], gm[u]);
#pragma unroll
          for (int u = 0; u < U; ++u)
            nx[u] = m + U + u < n ? ld_index(g.stIdx + base + (long long)(m + U + u) * kSlice) : 0;
#pragma unroll
          for (int u = 0; u < U; ++u) member(gm[u]);
        }
#pragma unroll
        for (int u = 0; u < U - 1; ++u) {
          if (nFull + u < n) {
            R gm[16];
            ld16(g.gradRaw + 16 * (size_t)nx[u], gm);
            member(gm);
          }
        }
      }
    }
    R out[16];
#pragma unroll
    for (int k = 0; k < 15; ++k) out[k] = acc[k] / ss[k];
    out[15] = R(0);
    // positivity of the face reconstructions of density (0) and pressure (4)
    R r0[8];
    ld8(g.rec + 8 * (size_t)c, r0);
    if (c >= g.nAct && g.vposOff) {  // a virtual cell of a partitioned region: all its faces
      const long long b0 = g.vposOff[c - g.nAct], b1 = g.vposOff[c - g.nAct + 1];
      const long long P = g.vposTotal;
#pragma unroll
      for (int v = 0; v < 5; v += 4) {
        for (long long e = b0; e < b1; ++e) {
          const R dx = g.vposD[e], dy = g.vposD[P + e], dz = g.vposD[2 * P + e];
          const R varf = r0[v] + out[3 * v] * dx + out[3 * v + 1] * dy + out[3 * v + 2] * dz;
          if (varf <= R(0)) {
            out[3 * v] = out[3 * v + 1] = out[3 * v + 2] = R(0);
            break;
          }
        }
      }
      st16(g.grad + 16 * (size_t)c, out);
      return;
    }
    const long long T = g.cfTotal;
    const long long e0 = g.cfOff[c >> 5] + (c & 31);
    const int nf = g.cfCnt[c];
    const int B = g.nBFaces;
#pragma unroll
    for (int v = 0; v < 5; v += 4) {
      for (int k = 0; k < nf; ++k) {
        const long long e = e0 + (long long)k * kSlice;
        const int code = g.cfCode[e];
        R dx, dy, dz;
        if (code >= 0) {  // the stored offset is xc - fc
          dx = -g.cfD[e];
          dy = -g.cfD[T + e];
          dz = -g.cfD[2 * T + e];
        } else {          // boundary: fc - xc
          const int b = -code - 1;
          dx = g.bfd[b];
          dy = g.bfd[B + b];
          dz = g.bfd[2 * B + b];
        }
        const R varf = r0[v] + out[3 * v] * dx + out[3 * v + 1] * dy + out[3 * v + 2] * dz;
        if (varf <= R(0)) {
          out[3 * v] = out[3 * v + 1] = out[3 * v + 2] = R(0);
          break;
        }
      }
    }
    st16(g.grad + 16 * (size_t)c, out);
  }
}

// The WENO-XYZ pass.  The mixed path's kernel asks for 6 resident blocks of
// 128 per SM: 0.381 ms per launch on 1.57 M tets, 7 blocks 0.383, 8 blocks
// 0.422 (spills).  The FP64 kernel keeps the compiler's choice.
#ifndef RF_WENO_MINB
#define RF_WENO_MINB 6
#endif
template <typename R>
__global__ void __launch_bounds__(128) k_weno_xyz(const RegionDev<R> *__restrict__ regs,
                                                  const Tile *__restrict__ tiles, int nTiles) {
  RF_TILE_LOOP(pdl_wait(), nTiles) weno_tile<R>(regs, tiles, t_);
}
template <typename R>
__global__ void __launch_bounds__(128) k_weno_xyz(const __grid_constant__ OneRegion<R> regs,
                                                  const Tile *__restrict__ tiles, int nTiles) {
  RF_TILE_LOOP(pdl_wait(), nTiles) weno_tile<R>(regs, tiles, t_);
}
template <int MINB>
__global__ void __launch_bounds__(128, MINB)
    k_weno_xyz_f32(const RegionDev<float> *__restrict__ regs, const Tile *__restrict__ tiles,
                   int nTiles) {
  RF_TILE_LOOP(pdl_wait(), nTiles) weno_tile<float>(regs, tiles, t_);
}
template <int MINB>
__global__ void __launch_bounds__(128, MINB)
    k_weno_xyz_f32(const __grid_constant__ OneRegion<float> regs, const Tile *__restrict__ tiles,
                   int nTiles) {
  RF_TILE_LOOP(pdl_wait(), nTiles) weno_tile<float>(regs, tiles, t_);
}

template <typename R>
void launch_weno_xyz(const RegionDev<R> *regs, const Work &w, cudaStream_t s) {
  if (w.nCellTiles <= 0) return;
  const int grid = w.grid > 0 && w.grid < w.nCellTiles ? w.grid : w.nCellTiles;
  with_regions(regs, w, w.cellTiles, [&](const auto &r, const Tile *t) {
    using K = void (*)(std::decay_t<decltype(r)>, const Tile *, int);
    if constexpr (sizeof(R) == 4)
      launch_pdl(static_cast<K>(k_weno_xyz_f32<RF_WENO_MINB>), grid, w.block, s, r, t, w.nCellTiles);
    else
      launch_pdl(static_cast<K>(k_weno_xyz<R>), grid, w.block, s, r, t, w.nCellTiles);
  });
}

template <typename R>
void launch_grad_tiles(const RegionDev<R> *regs, const Work &w, const Tile *tiles, int nTiles,
                       int fuseDt, cudaStream_t s) {
  // the phase tile lists hold 128-cell tiles
  if (fuseDt)
    grad_launch<R, 1, 128>(regs, w, tiles, nTiles, w.grid, s);
  else
    grad_launch<R, 0, 128>(regs, w, tiles, nTiles, w.grid, s);
}

template <typename R>
void launch_face_tiles(const RegionDev<R> *regs, const Work &w, const Tile *tiles, int nTiles,
                       cudaStream_t s) {
  // the phase lists hold 128-face tiles, one face per thread
  if (nTiles > 0) face_launch<R, 128, 1>(regs, w, tiles, nTiles, s);
}

template <typename R>
void launch_update_tiles(const RegionDev<R> *regs, const Work &w, const Tile *tiles, int nTiles,
                         const StepArgs &a, cudaStream_t s) {
  update_launch<R, 128>(regs, w, tiles, nTiles, a, s);  // 128-cell phase tiles
}

// The transfer chunk a host cell travels in.
__device__ __forceinline__ int host_chunk(const ChunkMap &m, int hostCell) {
  const int t = hostCell / m.block;
  int k = 0;
  while (k < m.nk - 1 && t >= m.tEnd[k]) ++k;
  return k;
}

// Per cell tile: the last chunk holding a record its gradient pass reads (the
// cell's own, its stencil members', its face neighbours') and the first chunk
// among its own cells.  Runs once per region.
template <typename R>
__global__ void k_tile_phases(const RegionDev<R> *__restrict__ regs, const Tile *__restrict__ tiles,
                              int nTiles, ChunkMap m, int *__restrict__ tileLast,
                              int *__restrict__ tileFirst) {
  RF_TILE_LOOP(blockIdx.x, nTiles) {
    const Tile tl = tiles[t_];
    const RegionDev<R> &g = regs[tl.region];
    const int c = tl.first + threadIdx.x;
    if (c >= g.nCells) continue;
    auto chunk = [&](int d) { return host_chunk(m, g.cellOld ? g.cellOld[d] : d); };
    const int own = chunk(c);
    int last = own;
    if (g.stOff) {
      const long long b = g.stOff[c >> 5] + (c & 31);
      const int n = g.stCnt[c];
      for (int k = 0; k < n; ++k) last = max(last, chunk(g.stIdx[b + (long long)k * kSlice]));
    }
    const long long e0 = g.cfOff[c >> 5] + (c & 31);
    const int nf = g.cfCnt[c];
    for (int k = 0; k < nf; ++k) {
      const long long e = e0 + (long long)k * kSlice;
      if (g.cfCode[e] >= 0) last = max(last, chunk(g.cfNb[e]));
    }
    atomicMax(tileLast + t_, last);
    atomicMin(tileFirst + t_, own);
  }
}

// The earliest phase any cell of a tile reads a record from: the minimum
// over its cells, their stencil members and face neighbours of the phase of
// the update tile (tilePhase, per 128-cell tile) that rewrites that record.
// A gradient tile of the last stage must run no later than that phase.
template <typename R>
__global__ void k_member_phase(const RegionDev<R> *__restrict__ regs, const Tile *__restrict__ tiles,
                               int nTiles, const int *__restrict__ tilePhase, int block,
                               int *__restrict__ out) {
  RF_TILE_LOOP(blockIdx.x, nTiles) {
    const Tile tl = tiles[t_];
    const RegionDev<R> &g = regs[tl.region];
    const int c = tl.first + threadIdx.x;
    if (c >= g.nCells) continue;
    int v = tilePhase[c / block];
    if (g.stOff) {
      const long long b = g.stOff[c >> 5] + (c & 31);
      const int n = g.stCnt[c];
      for (int k = 0; k < n; ++k) v = min(v, tilePhase[g.stIdx[b + (long long)k * kSlice] / block]);
    }
    const long long e0 = g.cfOff[c >> 5] + (c & 31);
    const int nf = g.cfCnt[c];
    for (int k = 0; k < nf; ++k) {
      const long long e = e0 + (long long)k * kSlice;
      if (g.cfCode[e] >= 0) v = min(v, tilePhase[g.cfNb[e] / block]);
    }
    atomicMin(out + t_, v);
  }
}

template <typename R>
void launch_member_phase(const RegionDev<R> *regs, const Work &w, const int *tilePhase, int *out,
                         cudaStream_t s) {
  if (w.nCellTiles > 0)
    k_member_phase<R><<<w.nCellTiles, w.block, 0, s>>>(regs, w.cellTiles, w.nCellTiles, tilePhase,
                                                       w.block, out);
}

template <typename R>
void launch_bface_tiles(const RegionDev<R> *regs, const Work &w, const Tile *tiles, int nTiles,
                        cudaStream_t s) {
  const int grid = grid_for(w.grid, nTiles);
  if (grid <= 0) return;
  with_regions(regs, w, tiles, [&](const auto &r, const Tile *t) {
    using RA = std::decay_t<decltype(r)>;
    launch_pdl(static_cast<void (*)(RA, const Tile *, int)>(k_bface_flux<R>), grid, w.block, s, r, t,
               nTiles);
  });
}

template <typename R>
void launch_tile_phases(const RegionDev<R> *regs, const Work &w, const ChunkMap &m,
                        int *tileLast, int *tileFirst, cudaStream_t s) {
  if (w.nCellTiles > 0)
    k_tile_phases<R><<<w.nCellTiles, w.block, 0, s>>>(regs, w.cellTiles, w.nCellTiles, m,
                                                       tileLast, tileFirst);
}

template <typename R>
void launch_upload_list(const RegionDev<R> *regs, const int *list, int n, const double *cvH,
                        const double *dvH, int split, cudaStream_t s) {
  if (n <= 0) return;
  if (split)
    k_upload_list<R, 1><<<(n + 255) / 256, 256, 0, s>>>(regs, list, n, cvH, dvH);
  else
    k_upload_list<R, 0><<<(n + 255) / 256, 256, 0, s>>>(regs, list, n, cvH, dvH);
}
template <typename R>
void launch_download_list(const RegionDev<R> *regs, const int *list, int n, double *cvH,
                          double *dvH, int split, cudaStream_t s) {
  if (n <= 0) return;
  if (split)
    k_download_list<R, 1><<<(n + 255) / 256, 256, 0, s>>>(regs, list, n, cvH, dvH);
  else
    k_download_list<R, 0><<<(n + 255) / 256, 256, 0, s>>>(regs, list, n, cvH, dvH);
}

// ---- residual without device allocation ---------------------------------------
// Variant of the face-flux and residual-gather passes for rfgpu_residual_noalloc:
// the face fluxes go to a caller-supplied scratch area (the library's static
// device array) and the residual to the same area, in the Fortran layout
// rhs(5,nCells), instead of the region's own buffers.  The region is passed by
// value, so no device-side descriptor has to be written.
template <typename R, bool PLAIN>
__global__ void __launch_bounds__(128) k_face_flux_scratch(const RegionDev<R> g,
                                                           R *__restrict__ flux) {
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  const int F = g.nFaces;
  if (f >= F) return;
  const int c1 = g.f2c[f], c2 = g.f2c[F + f];
  R flx[8];
  if constexpr (PLAIN) {
    face_flux_in<R>(g, f, c1, c2, flx);
    flx[5] = flx[6] = flx[7] = R(0);
  } else {
    face_flux_value(g, f, c1, c2, flx);
  }
  st8(flux + 8 * (size_t)f, flx);
}

template <typename R>
__global__ void __launch_bounds__(128) k_gather_rhs_scratch(const RegionDev<R> g,
                                                            const R *__restrict__ flux,
                                                            double *__restrict__ rhs) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= g.nCells) return;
  const long long e0 = g.cfOff[c >> 5] + (c & 31);
  const int n = g.cfCnt[c];
  const size_t hc = g.cellOld ? (size_t)g.cellOld[c] : (size_t)c;  // host numbering
  if (c >= g.nAct) {  // virtual cell: ZeroDummyCellsMP
#pragma unroll
    for (int j = 0; j < 5; ++j) rhs[5 * hc + j] = 0.0;
    return;
  }
  bool sum64 = true;  // FP64 and split paths: FP64 sums
  if constexpr (sizeof(R) == 4) sum64 = !g.cvF;
  if (sum64) {
    double acc[5];
    face_sum64(g, flux, c, acc);
#pragma unroll
    for (int j = 0; j < 5; ++j) rhs[5 * hc + j] = acc[j];
    return;
  }
  if constexpr (sizeof(R) == 4) {
    float hi[5] = {0.f, 0.f, 0.f, 0.f, 0.f}, lo[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
    for (int k = 0; k < n; ++k) {
      const int code = g.cfCode[e0 + (long long)k * kSlice];
      float fl[8];
      if (code >= 0) {
        ld8(flux + 8 * (size_t)(code >> 1), fl);
        const float sg = (code & 1) ? -1.f : 1.f;
#pragma unroll
        for (int j = 0; j < 5; ++j) two_sum_acc(hi[j], lo[j], sg * fl[j]);
      } else {
        ld8(g.bflux + 8 * (size_t)(-code - 1), fl);
#pragma unroll
        for (int j = 0; j < 5; ++j) two_sum_acc(hi[j], lo[j], fl[j]);
      }
    }
#pragma unroll
    for (int j = 0; j < 5; ++j) rhs[5 * hc + j] = double(hi[j]) + double(lo[j]);
  }
}

// Gradients (the region's own pass), face fluxes into `flux`, boundary fluxes,
// residual into `rhs`; all on stream s.
template <typename R>
void launch_residual_scratch(const RegionDev<R> *regs, const RegionDev<R> &g, const Work &w,
                             int spaceOrder, R *flux, double *rhs, cudaStream_t s) {
  if (spaceOrder > 1 && w.nCellTiles > 0) {
    grad_launch<R, 0, 128>(regs, w, w.cellTiles, w.nCellTiles, 0, s);
    if (g.gradRaw) launch_weno_xyz<R>(regs, w, s);
  }
  // FP64, first order: without a reconstruction, HLLC and AUSM+up have few
  // products to gain by, and FP64 ones are shorter in latency.  Integer and FP64
  // products, whole call: HLLC 94,000 tet faces 103.9 and 94.7 us, 96,000 tube
  // faces 114.6 and 105.2, 352,000 faces 242 and 256; AUSM+up 8,000 faces 53.8
  // and 51.1, 94,000 93.3 and 91.6, 352,000 207 and 221.  Roe and AUSM+ gain
  // at every size or lose nothing.
  auto faces = k_face_flux_scratch<R, false>;
  if constexpr (sizeof(R) == 8) {
    const int sd = g.ph.spaceDiscr;
    if (spaceOrder == 1 && (sd == 3 || sd == 5) && g.nFaces < 128000)
      faces = k_face_flux_scratch<R, true>;
  }
  if (g.nFaces > 0) faces<<<(g.nFaces + 127) / 128, 128, 0, s>>>(g, flux);
  if (w.nBFaceTiles > 0)
    launch_bface_tiles<R>(regs, w, w.bfaceTiles, w.nBFaceTiles, s);
  k_gather_rhs_scratch<R><<<(g.nCells + 127) / 128, 128, 0, s>>>(g, flux, rhs);
}

template <typename R>
void launch_halo(const RegionDev<R> *regs, const HaloLink *links, int n, cudaStream_t s) {
  if (n > 0) k_halo<R><<<(n + 127) / 128, 128, 0, s>>>(regs, links, n);
}
template <typename R>
void launch_halo_pair(const RegionDev<R> *src, const RegionDev<R> *dst, const int *srcCells,
                      const int *dstCells, int n, cudaStream_t s) {
  if (n > 0) k_halo_pair<R><<<(n + 127) / 128, 128, 0, s>>>(src, dst, srcCells, dstCells, n);
}
template <typename R>
void launch_border_pack(const RegionDev<R> *g, const int *cells, int n, double *buf,
                        cudaStream_t s) {
  if (n > 0) k_border_pack<R><<<(n + 127) / 128, 128, 0, s>>>(g, cells, n, buf);
}
template <typename R>
void launch_border_unpack(const RegionDev<R> *g, const int *cells, int n, const double *buf,
                          cudaStream_t s) {
  if (n > 0) k_border_unpack<R><<<(n + 127) / 128, 128, 0, s>>>(g, cells, n, buf);
}

#define RFGPU_INSTANTIATE(R)                                                                  \
  template void launch_prim<R>(const RegionDev<R> *, const Work &, int, cudaStream_t);        \
  template void launch_upload_list<R>(const RegionDev<R> *, const int *, int, const double *,  \
                                      const double *, int, cudaStream_t);                     \
  template void launch_download_list<R>(const RegionDev<R> *, const int *, int, double *,     \
                                        double *, int, cudaStream_t);                         \
  template void launch_residual_scratch<R>(const RegionDev<R> *, const RegionDev<R> &,         \
                                           const Work &, int, R *, double *, cudaStream_t);    \
  template void launch_stage<R>(const RegionDev<R> *, const Work &, const StepArgs &,         \
                                cudaStream_t, long long *, int, int, const Prof *, int);      \
  template void launch_tile_phases<R>(const RegionDev<R> *, const Work &, const ChunkMap &,   \
                                      int *, int *, cudaStream_t);                            \
  template void launch_grad_tiles<R>(const RegionDev<R> *, const Work &, const Tile *, int,   \
                                     int, cudaStream_t);                                      \
  template void launch_update_tiles<R>(const RegionDev<R> *, const Work &, const Tile *, int, \
                                       const StepArgs &, cudaStream_t);                       \
  template void launch_face_tiles<R>(const RegionDev<R> *, const Work &, const Tile *, int,   \
                                     cudaStream_t);                                           \
  template void launch_bface_tiles<R>(const RegionDev<R> *, const Work &, const Tile *, int,  \
                                      cudaStream_t);                                          \
  template void launch_member_phase<R>(const RegionDev<R> *, const Work &, const int *, int *, \
                                       cudaStream_t);                                         \
  template void launch_dt<R>(const RegionDev<R> *, const Work &, const DtArgs &, cudaStream_t, \
                             long long *, const Prof *);                                      \
  template void launch_step<R>(const RegionDev<R> *, const Work &, const DtArgs &, int,       \
                               cudaStream_t, long long *, int, int, const Prof *);            \
  template void launch_halo<R>(const RegionDev<R> *, const HaloLink *, int, cudaStream_t);    \
  template void launch_halo_pair<R>(const RegionDev<R> *, const RegionDev<R> *, const int *,  \
                                    const int *, int, cudaStream_t);                          \
  template void launch_border_pack<R>(const RegionDev<R> *, const int *, int, double *,       \
                                      cudaStream_t);                                          \
  template void launch_border_unpack<R>(const RegionDev<R> *, const int *, int,               \
                                        const double *, cudaStream_t);

}  // namespace rfgpu
