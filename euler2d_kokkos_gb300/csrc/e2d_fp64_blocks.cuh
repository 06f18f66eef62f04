// e2d_fp64_blocks.cuh -- the building blocks of the FP64 step, bit-identical
// to the reference's FP64 arithmetic (compile with --fmad=false; every
// expression keeps the reference's operation order): primitives, limited
// slopes, the half-step trace, the three Riemann solvers and the CFL term.
// Shared by the fused / two-launch step kernels (e2d_fp64.cu) and the
// implementation-1/2 orchestrations (e2d_impl12.cu).
#pragma once

#include "e2d_common.cuh"
#include "e2d_f64_exact.cuh"
#include "e2d_internal.h"

namespace e2d {
namespace {

using f64x::gt0;
using f64x::half;
using f64x::max_nn;
using f64x::max_pos;
using f64x::max_any;
using f64x::min_any;

__device__ __forceinline__ int src_lo_hi(int i, int n, int bc_lo, int bc_hi, bool &flip) {
  return ghost_source(i, n, bc_lo, bc_hi, flip);
}
__device__ __forceinline__ bool nonfinite(double x) { return (f64i::high(x) & 0x7ff00000u) == 0x7ff00000u; }

// ------------------------------------------------------------ numerics
using f64x::divisor;
using f64x::Divisor;
using f64x::Fp;
using f64x::quot;
using f64x::root;

// max(p, d * smallp), d > 0.  High words of positive doubles grow like 2^20
// times their logarithm (within 0.09 2^20), so p exceeds the product for
// certain when they differ by more than smallp's exponent plus two; only then
// is the product not formed (one FP64 instruction of the two each face state
// would take; every cell of an ordinary flow).
template <class F>
__device__ __forceinline__ double floor_pressure(const F &f, const KPhys<double> &ph, double p, double d) {
  const int lim = (int)(f64i::high(ph.smallp) & 0x7ff00000u) - (1020 << 20);  // (exponent + 3) 2^20
  const int hp = (int)f64i::high(p), hd = (int)f64i::high(d);
  if (hp >= 0x00100000 && hp - hd > lim) return p;
  return max_pos(p, f.mul(d, ph.smallp));
}

// src/HydroBaseFunctor.h:76-102 (computePrimitives) without the sound speed.
// `dv`: the density, ready as a divisor.
template <class F>
__device__ __forceinline__ void primitives(const F &f, const KPhys<double> &ph, double rho, double e, double mx,
                                           double my, double &d, double &p, double &ux, double &uy, Divisor &dv) {
  d = max_pos(rho, ph.smallr);
  dv = divisor(d);
  ux = quot(mx, dv);
  uy = quot(my, dv);
  const double eken = half(f.add(f.mul(ux, ux), f.mul(uy, uy)));
  const double ei = f.sub(quot(e, dv), eken);
  p = floor_pressure(f, ph, f.mul(f.mul(ph.gm1, d), ei), d);
}

// src/HydroBaseFunctor.h:475-516 for one variable and direction: slope_type
// 0 gives a zero slope, 1 and 2 the limited slope.  h: half of it.
template <class F>
__device__ __forceinline__ void slope(const F &f, int st_kind, double q, double qp, double qm, double &dq, double &h) {
  dq = h = 0.0;
  if (st_kind != 0) f64x::slope_limited(f, st_kind == 2, q, qp, qm, dq, h);
}
template <class F>
__device__ __forceinline__ double slope(const F &f, int st_kind, double q, double qp, double qm) {
  double dq, h;
  slope(f, st_kind, q, qp, qm, dq, h);
  return dq;
}

// Sources of trace_unsplit_2d_along_dir (src/HydroBaseFunctor.h:246-249).
template <class F>
__device__ __forceinline__ void trace_sources(const F &f, const KPhys<double> &ph, const double q[4],
                                              const double dqx[4], const double dqy[4], double s0[4]) {
  const double r = q[E2D_ID], p = q[E2D_IP], u = q[E2D_IU], v = q[E2D_IV];
  const Divisor dr = divisor(r);
  const double div = f.add(dqx[E2D_IU], dqy[E2D_IV]);
  const double nu = f.neg(u);
  auto advect = [&](int k) { return f.sub(f.xmul(nu, dqx[k]), f.xmul(v, dqy[k])); };  // -u*dqx - v*dqy
  s0[E2D_ID] = f.sub(advect(E2D_ID), f.mul(div, r));
  s0[E2D_IP] = f.sub(advect(E2D_IP), f.mul(f.mul(div, ph.gamma0), p));
  s0[E2D_IU] = f.sub(advect(E2D_IU), quot(dqx[E2D_IP], dr));
  s0[E2D_IV] = f.sub(advect(E2D_IV), quot(dqy[E2D_IP], dr));
}

// The two face states of one direction (src/HydroBaseFunctor.h:251-289):
// minus face q - dq/2 + s0*dtd/2, plus face q + dq/2 + s0*dtd/2, density
// clamped at smallr.  h = dq/2, hdtd = dtd/2.
template <class F>
__device__ __forceinline__ void face_pair(const F &f, const KPhys<double> &ph, int v, double q, double h,
                                          double s0, double dtd, double hdtd, double &fm, double &fp) {
  const double sx = f.half_product(s0, dtd, hdtd);
  fm = f.add(f.sub(q, h), sx);
  fp = f.add(f.add(q, h), sx);
  if (v == E2D_ID) {
    fm = max_pos(fm, ph.smallr);
    fp = max_pos(fp, ph.smallr);
  }
}

// src/HydroBaseFunctor.h:523-547.
template <class F>
__device__ __forceinline__ void cmpflx(const F &o, const KPhys<double> &ph, const double g[4], double f[4]) {
  f[E2D_ID] = o.mul(g[E2D_ID], g[E2D_IU]);
  f[E2D_IU] = o.add(o.mul(f[E2D_ID], g[E2D_IU]), g[E2D_IP]);
  f[E2D_IV] = o.mul(f[E2D_ID], g[E2D_IV]);
  const double ekin = o.mul(half(g[E2D_ID]), o.add(o.mul(g[E2D_IU], g[E2D_IU]), o.mul(g[E2D_IV], g[E2D_IV])));
  const double etot = o.add(o.mul(g[E2D_IP], ph.entho), ekin);
  f[E2D_IP] = o.mul(g[E2D_IU], o.add(etot, g[E2D_IP]));
}

// fmax of any two doubles, NaN dropped as fmax drops it, on the integer pipe.
__device__ __forceinline__ double fmax_any(double a, double b) {
  return f64x::is_nan(a) ? b : f64x::is_nan(b) ? a : max_any(a, b);
}

// src/HydroBaseFunctor.h:558-693 (riemann_approx).
template <class F>
__device__ __noinline__ void riemann_approx(const F &f, const KPhys<double> &ph, const double *ql,
                                            const double *qr, double *flux) {
  const double gamma0 = ph.gamma0, gamma6 = ph.gamma6;
  const double rl = fmax_any(ql[E2D_ID], ph.smallr), ul = ql[E2D_IU];
  const double pl = fmax_any(ql[E2D_IP], f.mul(rl, ph.smallp));
  const double rr = fmax_any(qr[E2D_ID], ph.smallr), ur = qr[E2D_IU];
  const double pr = fmax_any(qr[E2D_IP], f.mul(rr, ph.smallp));
  const double cl = f.mul(f.mul(gamma0, pl), rl);
  const double cr = f.mul(f.mul(gamma0, pr), rr);
  const Divisor dpl = divisor(pl), dpr = divisor(pr);
  // sqrt(c * (1 + gamma6 * (p - ps) / ps))
  auto wave = [&](double c, double p, double ps, const Divisor &dps) {
    return root(f.mul(c, f.add(f.one, quot(f.mul(gamma6, f.sub(p, ps)), dps))));
  };
  double wl = root(cl);
  double wr = root(cr);
  double pstar = fmax_any(quot(f.add(f.add(f.mul(wr, pl), f.mul(wl, pr)), f.mul(f.mul(wl, wr), f.sub(ul, ur))),
                               f.add(wl, wr)),
                          0.0);
  double pold = pstar;
  double conv = 1.0;
  for (int iter = 0; (iter < 10) && f64x::gt_pos(conv, 1e-6); ++iter) {
    const double wwl = wave(cl, pold, pl, dpl);
    const double wwr = wave(cr, pold, pr, dpr);
    const double w2l = f.mul(wwl, wwl), w2r = f.mul(wwr, wwr);
    // 2 w w w: the doubling is exact wherever it is applied (no overflow here)
    const double qxl = quot(f.mul(f64x::twice(w2l), wwl), f.add(w2l, cl));
    const double qxr = quot(f.mul(f64x::twice(w2r), wwr), f.add(w2r, cr));
    const double usl = f.sub(ul, quot(f.sub(pold, pl), wwl));
    const double usr = f.add(ur, quot(f.sub(pold, pr), wwr));
    const double delp = fmax_any(f.mul(quot(f.mul(qxr, qxl), f.add(qxr, qxl)), f.sub(usl, usr)), f.neg(pold));
    pold = f.add(pold, delp);
    // pold + smallpp is pold where that is 2^55 times the larger
    const int hs = (int)f64i::high(ph.smallpp);
    const bool far = hs >= 0 && (int)f64i::high(pold) - hs > 55 << 20;
    conv = f.abs(quot(delp, far ? pold : f.add(pold, ph.smallpp)));
  }
  pstar = pold;
  wl = wave(cl, pstar, pl, dpl);
  wr = wave(cr, pstar, pr, dpr);
  const double ustar =
      half(f.sub(f.add(f.add(ul, quot(f.sub(pl, pstar), wl)), ur), quot(f.sub(pr, pstar), wr)));
  const bool lft = f64x::sbits(ustar) >= 0;  // copysign(1, ustar) > 0
  auto signed_by = [&](double x) { return lft ? x : f.neg(x); };  // sgnm * x
  const double ro = lft ? rl : rr, uo = lft ? ul : ur, po = lft ? pl : pr, wo = lft ? wl : wr;
  const Divisor dro = divisor(ro);
  const double co = fmax_any(ph.smallc, root(f.abs(quot(f.mul(gamma0, po), dro))));
  const double rstar = fmax_any(
      quot(ro, f.add(f.one, quot(f.mul(ro, f.sub(po, pstar)), f.mul(wo, wo)))), ph.smallr);
  const double cstar = fmax_any(ph.smallc, root(f.abs(quot(f.mul(gamma0, pstar), rstar))));
  double spout = f.sub(co, signed_by(uo));
  double spin = f.sub(cstar, signed_by(ustar));
  const double ushock = f.sub(quot(wo, dro), signed_by(uo));
  if (f64x::okey(pstar) >= f64x::okey(po)) {
    spin = ushock;
    spout = ushock;
  }
  const double spsum = f.add(spout, spin);
  const double scr = fmax_any(f.sub(spout, spin), f.add(ph.smallc, f.abs(spsum)));
  double frac = half(f.add(f.one, quot(spsum, scr)));
  if (f64x::is_nan(frac))
    frac = 0.0;
  else
    frac = f64x::sbits(frac) >= f64x::sbits(1.0) ? 1.0 : f64x::le0(frac) ? 0.0 : frac;
  const double rest = f.sub(f.one, frac);
  double g[4];
  g[E2D_ID] = f.add(f.mul(frac, rstar), f.mul(rest, ro));
  g[E2D_IU] = f.add(f.mul(frac, ustar), f.mul(rest, uo));
  g[E2D_IP] = f.add(f.mul(frac, pstar), f.mul(rest, po));
  if (f64x::lt0(spout)) {
    g[E2D_ID] = ro;
    g[E2D_IU] = uo;
    g[E2D_IP] = po;
  }
  if (gt0(spin)) {
    g[E2D_ID] = rstar;
    g[E2D_IU] = ustar;
    g[E2D_IP] = pstar;
  }
  g[E2D_IV] = lft ? ql[E2D_IV] : qr[E2D_IV];
  cmpflx(f, ph, g, flux);
}

// src/HydroBaseFunctor.h:704-809 (riemann_hllc).  The reference builds the
// star states of both sides and keeps one; here only the total energy and the
// star state of the side that is read are built (SL > 0 reads the left state,
// else the contact selects), and the larger sound speed is the root of the
// larger square (a correctly rounded root is monotonic): the same values.
// S - us and rs (S - us) are, but for the sign, the differences and products
// that rcl and rcr are made of.
// Cut-offs, maxima, the 0.5 factors and the sign tests use the exact integer
// forms of e2d_f64_exact.cuh.
template <class F>
__device__ __forceinline__ void riemann_hllc(const F &f, const KPhys<double> &ph, const double *ql,
                                             const double *qr, double *flux) {
  const double rl = max_pos(ql[E2D_ID], ph.smallr);
  const double pl = floor_pressure(f, ph, ql[E2D_IP], rl);
  const double ul = ql[E2D_IU];
  const double rr = max_pos(qr[E2D_ID], ph.smallr);
  const double pr = floor_pressure(f, ph, qr[E2D_IP], rr);
  const double ur = qr[E2D_IU];
  const double c2l = max_pos(quot(f.mul(ph.gamma0, pl), rl), ph.smallc2);
  const double c2r = max_pos(quot(f.mul(ph.gamma0, pr), rr), ph.smallc2);
  const double cmax = root(max_nn(c2l, c2r));
  const double SL = f.sub(min_any(ul, ur), cmax);
  const double SR = f.add(max_any(ul, ur), cmax);
  const double dl = f.sub(ul, SL), dr = f.sub(SR, ur);
  const double rcl = f.mul(rl, dl);
  const double rcr = f.mul(rr, dr);
  const Divisor rc = divisor(f.add(rcr, rcl));
  const double ustar = quot(f.add(f.add(f.xmul(rcr, ur), f.xmul(rcl, ul)), f.sub(pl, pr)), rc);
  const double ptotstar =
      quot(f.add(f.add(f.xmul(rcr, pl), f.xmul(rcl, pr)), f.mul(f.mul(rcl, rcr), f.sub(ul, ur))), rc);
  const bool own_l = gt0(SL);
  const bool lft = own_l || gt0(ustar);
  const bool own = own_l || !(lft || gt0(SR));
  const double S = lft ? SL : SR;
  const double rs = lft ? rl : rr, us = lft ? ul : ur, ps = lft ? pl : pr, vs = lft ? ql[E2D_IV] : qr[E2D_IV];
  const double hrs = half(rs);
  const double es = f.add(f.xmul(ps, ph.entho), f.add(f.xmul(f.xmul(hrs, us), us), f.xmul(f.xmul(hrs, vs), vs)));
  const double sdu = lft ? f.reversed(dl) : dr, rsdu = lft ? f.reversed(rcl) : rcr;  // S - us, rs (S - us)
  const Divisor sds = divisor(f.sub(S, ustar));
  const double rstar = quot(rsdu, sds);
  const double etotstar = quot(f.add(f.sub(f.mul(sdu, es), f.mul(ps, us)), f.mul(ptotstar, ustar)), sds);
  const double ro = own ? rs : rstar, uo = own ? us : ustar, ptoto = own ? ps : ptotstar;
  const double etoto = own ? es : etotstar;
  flux[E2D_ID] = f.mul(ro, uo);
  flux[E2D_IU] = f.add(f.mul(flux[E2D_ID], uo), ptoto);
  flux[E2D_IP] = f.mul(f.add(etoto, ptoto), uo);
  flux[E2D_IV] = f.mul(flux[E2D_ID], gt0(flux[E2D_ID]) ? ql[E2D_IV] : qr[E2D_IV]);
}

static __device__ __noinline__ double etot_slow(double r, double p, double u, double v, double entho) {
  const double ecin = 0.5 * r * u * u;
  return p * entho + (ecin + 0.5 * r * v * v);
}

// HLL flux (Harten, Lax, van Leer; Toro, "Riemann Solvers and Numerical
// Methods for Fluid Dynamics", 3rd ed., eq. 10.21).  The reference declares
// RIEMANN_HLL but has no solver; this uses riemann_hllc's cut-offs and Davis
// wave speeds; the star flux multiplies by one reciprocal of SR - SL.
// Operation order matches the oracle's riemann_hll.
template <class F>
__device__ __forceinline__ void riemann_hll(const F &f, const KPhys<double> &ph, const double *ql,
                                            const double *qr, double *flux) {
  const double rl = max_pos(ql[E2D_ID], ph.smallr);
  const double pl = floor_pressure(f, ph, ql[E2D_IP], rl);
  const double ul = ql[E2D_IU], vl = ql[E2D_IV];
  const double rr = max_pos(qr[E2D_ID], ph.smallr);
  const double pr = floor_pressure(f, ph, qr[E2D_IP], rr);
  const double ur = qr[E2D_IU], vr = qr[E2D_IV];
  // r u, r v and r u u serve the state, the flux and the energy, whose factor
  // 0.5 is exact wherever it is applied, barring underflow, which the energy's
  // pressure term absorbs, and overflow of a product whose half is finite,
  // where the energies are formed as the oracle does (0.3 % of a step):
  // 12 products a cell fewer, 523 -> 495 us a
  // 1531x797 step, 488 with the last product on the integer pipes in the
  // room this leaves there (another 4 or 8 of a flux's: 492, 500).
  const double mxl = f.mul(rl, ul), myl = f.mul(rl, vl), mxul = f.mul(mxl, ul);
  const double mxr = f.mul(rr, ur), myr = f.mul(rr, vr), mxur = f.mul(mxr, ur);
  double etotl = f.add(f.xmul(pl, ph.entho), f.add(half(mxul), half(f.xmul(myl, vl))));
  double etotr = f.add(f.xmul(pr, ph.entho), f.add(half(mxur), half(f.xmul(myr, vr))));
  if (nonfinite(etotl) || nonfinite(etotr)) {
    etotl = etot_slow(rl, pl, ul, vl, ph.entho);
    etotr = etot_slow(rr, pr, ur, vr, ph.entho);
  }
  const double c2l = max_pos(quot(f.mul(ph.gamma0, pl), rl), ph.smallc2);
  const double c2r = max_pos(quot(f.mul(ph.gamma0, pr), rr), ph.smallc2);
  const double cmax = root(max_nn(c2l, c2r));
  const double SL = f.sub(min_any(ul, ur), cmax);
  const double SR = f.add(max_any(ul, ur), cmax);
  const double UL[4] = {rl, etotl, mxl, myl};
  const double UR[4] = {rr, etotr, mxr, myr};
  double FL[4], FR[4];
  FL[E2D_ID] = UL[E2D_IU];
  FL[E2D_IP] = f.xmul(f.add(etotl, pl), ul);
  FL[E2D_IU] = f.add(mxul, pl);
  FL[E2D_IV] = f.xmul(UL[E2D_IU], vl);
  FR[E2D_ID] = UR[E2D_IU];
  FR[E2D_IP] = f.xmul(f.add(etotr, pr), ur);
  FR[E2D_IU] = f.add(mxur, pr);
  FR[E2D_IV] = f.xmul(UR[E2D_IU], vr);
  if (gt0(SL)) {
#pragma unroll
    for (int v = 0; v < 4; ++v) flux[v] = FL[v];
  } else if (f64x::le0(SR)) {
#pragma unroll
    for (int v = 0; v < 4; ++v) flux[v] = FR[v];
  } else {
    // one division: the four star fluxes share the factor 1 / (SR - SL)
    const double sls = f.mul(SL, SR);
    const double rden = quot(f.one, f.sub(SR, SL));
#pragma unroll
    for (int v = 0; v < 4; ++v)
      flux[v] = f.xmul(f.add(f.sub(f.mul(SR, FL[v]), f.mul(SL, FR[v])), f.xmul(sls, f.sub(UR[v], UL[v]))), rden);
  }
}

template <int RS, class F>
__device__ __forceinline__ void riemann(const F &f, const KPhys<double> &ph, const double *ql, const double *qr,
                                        double *flux) {
  if (RS == E2D_RIEMANN_HLLC)
    riemann_hllc(f, ph, ql, qr, flux);
  else if (RS == E2D_RIEMANN_HLL)
    riemann_hll(f, ph, ql, qr, flux);
  else
    riemann_approx(f, ph, ql, qr, flux);
}

// CFL wave-speed term of a cell from its primitives (src/HydroRunFunctors.h:56-72):
// (c + |u|) / dx + (c + |v|) / dy, c = sqrt(gamma p / d); a division by a
// power-of-two dx, dy is the exact product by its reciprocal.
template <class F>
__device__ __forceinline__ double cfl_term(const F &f, const KPhys<double> &ph, const Divisor &dd, double p,
                                           double ux, double uy) {
  const double c = root(quot(f.mul(ph.gamma0, p), dd));
  const double vx = f.add(c, f.abs(ux));
  const double vy = f.add(c, f.abs(uy));
  const double tx = ph.inv_dx_pow2 != 0.0 ? f.mul(vx, ph.inv_dx_pow2) : quot(vx, ph.dx);
  const double ty = ph.inv_dy_pow2 != 0.0 ? f.mul(vy, ph.inv_dy_pow2) : quot(vy, ph.dy);
  return f.add(tx, ty);
}

// E2D_FLAG_* bits of a cell's conserved values.
__device__ __forceinline__ unsigned int state_flags(double rho, double e, double mx, double my) {
  unsigned int f = 0;
  if (nonfinite(rho) || nonfinite(e) || nonfinite(mx) || nonfinite(my)) f |= E2D_FLAG_NONFINITE;
  if (!f64i::positive(rho)) f |= E2D_FLAG_DENSITY;
  return f;
}


// ------------------------------------------------------------ fast forms
// The opt-in E2D_PRECISION_FP64_FAST step: the same formulas with a*b + c
// contracted into one FMA where it falls naturally (quotients and roots cost
// no FP64 instruction, so they stay as they are).  Results differ from the
// reference's by rounding (not bit-identical); the tests hold them to 1e-12
// on dt and 1e-10 relative L1.
template <class F>
__device__ __forceinline__ void primitives_fast(const F &f, const KPhys<double> &ph, double rho, double e,
                                                double mx, double my, double &d, double &p, double &ux, double &uy,
                                                Divisor &dv) {
  d = max_pos(rho, ph.smallr);
  dv = divisor(d);
  ux = quot(mx, dv);
  uy = quot(my, dv);
  const double ei = f.sub(quot(e, dv), half(fma(ux, ux, f.mul(uy, uy))));
  p = floor_pressure(f, ph, f.mul(f.mul(ph.gm1, d), ei), d);
}

template <class F>
__device__ __forceinline__ void trace_sources_fast(const F &f, const KPhys<double> &ph, const double q[4],
                                                   const double dqx[4], const double dqy[4], double s0[4]) {
  const double r = q[E2D_ID], p = q[E2D_IP], u = q[E2D_IU], v = q[E2D_IV];
  const Divisor dr = divisor(r);
  const double nu = f.neg(u), nv = f.neg(v), ndiv = f.neg(f.add(dqx[E2D_IU], dqy[E2D_IV]));
  s0[E2D_ID] = fma(nu, dqx[E2D_ID], fma(nv, dqy[E2D_ID], f.xmul(ndiv, r)));
  s0[E2D_IP] = fma(nu, dqx[E2D_IP], fma(nv, dqy[E2D_IP], f.xmul(f.xmul(ndiv, ph.gamma0), p)));
  s0[E2D_IU] = fma(nu, dqx[E2D_IU], fma(nv, dqy[E2D_IU], f.neg(quot(dqx[E2D_IP], dr))));
  s0[E2D_IV] = fma(nu, dqx[E2D_IV], fma(nv, dqy[E2D_IV], f.neg(quot(dqy[E2D_IP], dr))));
}

template <class F>
__device__ __forceinline__ void face_pair_fast(const F &f, const KPhys<double> &ph, int v, double q, double h,
                                               double s0, double hdtd, double &fm, double &fp) {
  const double qs = fma(s0, hdtd, q);
  fm = f.sub(qs, h);
  fp = f.add(qs, h);
  if (v == E2D_ID) {
    fm = max_pos(fm, ph.smallr);
    fp = max_pos(fp, ph.smallr);
  }
}

// riemann_hllc() with FMAs.
template <class F>
__device__ __forceinline__ void riemann_hllc_fast(const F &f, const KPhys<double> &ph, const double *ql,
                                                  const double *qr, double *flux) {
  const double rl = max_pos(ql[E2D_ID], ph.smallr);
  const double pl = floor_pressure(f, ph, ql[E2D_IP], rl);
  const double ul = ql[E2D_IU];
  const double rr = max_pos(qr[E2D_ID], ph.smallr);
  const double pr = floor_pressure(f, ph, qr[E2D_IP], rr);
  const double ur = qr[E2D_IU];
  const double c2l = max_pos(quot(f.mul(ph.gamma0, pl), rl), ph.smallc2);
  const double c2r = max_pos(quot(f.mul(ph.gamma0, pr), rr), ph.smallc2);
  const double cmax = root(max_nn(c2l, c2r));
  const double SL = f.sub(min_any(ul, ur), cmax);
  const double SR = f.add(max_any(ul, ur), cmax);
  const double dl = f.sub(ul, SL), dr = f.sub(SR, ur);
  const double rcl = f.mul(rl, dl);
  const double rcr = f.mul(rr, dr);
  const Divisor rc = divisor(f.add(rcr, rcl));
  const double ustar = quot(fma(rcr, ur, fma(rcl, ul, f.sub(pl, pr))), rc);
  const double ptotstar = quot(fma(rcr, pl, fma(rcl, pr, f.xmul(f.xmul(rcl, rcr), f.sub(ul, ur)))), rc);
  const bool own_l = gt0(SL);
  const bool lft = own_l || gt0(ustar);
  const bool own = own_l || !(lft || gt0(SR));
  const double S = lft ? SL : SR;
  const double rs = lft ? rl : rr, us = lft ? ul : ur, ps = lft ? pl : pr, vs = lft ? ql[E2D_IV] : qr[E2D_IV];
  const double es = fma(ps, ph.entho, f.xmul(half(rs), fma(us, us, f.xmul(vs, vs))));
  const double sdu = lft ? f.reversed(dl) : dr, rsdu = lft ? f.reversed(rcl) : rcr;  // S - us, rs (S - us)
  const Divisor sds = divisor(f.sub(S, ustar));
  const double rstar = quot(rsdu, sds);
  const double etotstar = quot(fma(sdu, es, fma(f.neg(ps), us, f.xmul(ptotstar, ustar))), sds);
  const double ro = own ? rs : rstar, uo = own ? us : ustar, ptoto = own ? ps : ptotstar;
  const double etoto = own ? es : etotstar;
  flux[E2D_ID] = f.xmul(ro, uo);
  flux[E2D_IU] = fma(flux[E2D_ID], uo, ptoto);
  flux[E2D_IP] = f.xmul(f.add(etoto, ptoto), uo);
  flux[E2D_IV] = f.xmul(flux[E2D_ID], gt0(flux[E2D_ID]) ? ql[E2D_IV] : qr[E2D_IV]);
}

// riemann_hll() with FMAs.
template <class F>
__device__ __forceinline__ void riemann_hll_fast(const F &f, const KPhys<double> &ph, const double *ql,
                                                 const double *qr, double *flux) {
  const double rl = max_pos(ql[E2D_ID], ph.smallr);
  const double pl = floor_pressure(f, ph, ql[E2D_IP], rl);
  const double ul = ql[E2D_IU], vl = ql[E2D_IV];
  const double rr = max_pos(qr[E2D_ID], ph.smallr);
  const double pr = floor_pressure(f, ph, qr[E2D_IP], rr);
  const double ur = qr[E2D_IU], vr = qr[E2D_IV];
  const double etotl = fma(pl, ph.entho, f.mul(half(rl), fma(ul, ul, f.mul(vl, vl))));
  const double etotr = fma(pr, ph.entho, f.mul(half(rr), fma(ur, ur, f.mul(vr, vr))));
  const double c2l = max_pos(quot(f.mul(ph.gamma0, pl), rl), ph.smallc2);
  const double c2r = max_pos(quot(f.mul(ph.gamma0, pr), rr), ph.smallc2);
  const double cmax = root(max_nn(c2l, c2r));
  const double SL = f.sub(min_any(ul, ur), cmax);
  const double SR = f.add(max_any(ul, ur), cmax);
  const double UL[4] = {rl, etotl, f.mul(rl, ul), f.mul(rl, vl)};
  const double UR[4] = {rr, etotr, f.mul(rr, ur), f.mul(rr, vr)};
  const double FL[4] = {UL[E2D_IU], f.mul(f.add(etotl, pl), ul), fma(UL[E2D_IU], ul, pl), f.mul(UL[E2D_IU], vl)};
  const double FR[4] = {UR[E2D_IU], f.mul(f.add(etotr, pr), ur), fma(UR[E2D_IU], ur, pr), f.mul(UR[E2D_IU], vr)};
  if (gt0(SL)) {
#pragma unroll
    for (int v = 0; v < 4; ++v) flux[v] = FL[v];
  } else if (f64x::le0(SR)) {
#pragma unroll
    for (int v = 0; v < 4; ++v) flux[v] = FR[v];
  } else {
    const double sls = f.mul(SL, SR);
    const double rden = quot(f.one, f.sub(SR, SL));
#pragma unroll
    for (int v = 0; v < 4; ++v)
      flux[v] = f.mul(fma(sls, f.sub(UR[v], UL[v]), fma(SR, FL[v], f.mul(f.neg(SL), FR[v]))), rden);
  }
}

template <int RS, bool FAST, class F>
__device__ __forceinline__ void riemann_sel(const F &f, const KPhys<double> &ph, const double *ql,
                                            const double *qr, double *flux) {
  if (FAST && RS == E2D_RIEMANN_HLLC)
    riemann_hllc_fast(f, ph, ql, qr, flux);
  else if (FAST && RS == E2D_RIEMANN_HLL)
    riemann_hll_fast(f, ph, ql, qr, flux);
  else
    riemann<RS>(f, ph, ql, qr, flux);
}

template <class F>
__device__ __forceinline__ double cfl_term_fast(const F &f, const KPhys<double> &ph, const Divisor &dd, double p,
                                                double ux, double uy) {
  const double c = root(quot(f.mul(ph.gamma0, p), dd));
  return fma(f.add(c, f.abs(ux)), ph.inv_dx, f.mul(f.add(c, f.abs(uy)), ph.inv_dy));
}

// dt of a step from the CFL maximum (src/main.cpp:128-134).
__device__ __forceinline__ double step_dt(const KPhys<double> &ph, unsigned long long invdt_bits, double t,
                                          double t_end) {
  const double inv_dt = __longlong_as_double((long long)invdt_bits);
  double dt = quot(ph.cfl, inv_dt);
  if (t + dt > t_end) dt = t_end - t;
  return dt;
}

}  // namespace
}  // namespace e2d
