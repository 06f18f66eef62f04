// e2d_fp64.cu -- FP64 kernels of the unsplit MUSCL-Hancock Godunov step,
// bit-identical to the reference (compiled with --fmad=false; every
// expression keeps the reference's operation order).
//
// The device time loop runs one fused launch per step (k_step_f64, after a
// prologue k_fill_f64 that folds the first step's CFL maximum and writes the
// primitives of the initial state), or many steps in one cooperative launch
// where the grid is small (k_loop_f64); FP64 batch instances run the same
// fused step in one launch per run call (k_batch_loop_f64).  The host-driven
// loop runs a step as two launches:
//   k_dt_f64           (compute_dt) primitives of every cell
//                      (ConvertToPrimitivesFunctor, src/HydroRunFunctors.h:84-143)
//                      and the CFL maximum of the interior
//                      (ComputeDtFunctor, src/HydroRunFunctors.h:17-79);
//                      k_fill_f64 writes the primitives where no compute_dt
//                      of the state came before;
//   k_flux_update_f64  (godunov_unsplit) per tile: limited slopes once per
//                      cell, the half-step trace once per cell and face, one
//                      Riemann solve per face, the conservative update
//                      (ComputeAndStoreFluxesFunctor + UpdateFunctor,
//                      src/HydroRunFunctors.h:412-723) and the ghost fill
//                      into both states (make_boundaries, deep_copy,
//                      src/HydroRun.h:388-399,302).
// The reference evaluates the slopes of a cell three times and the trace
// sources four times per cell; evaluating each once gives the same bits.
#include "e2d_fp64_blocks.cuh"
#include "e2d_tma.cuh"

#include <cudaTypedefs.h>

#include <cmath>
#include <cstdint>
#include <map>
#include <mutex>
#include <utility>

namespace e2d {
namespace {

constexpr int FILL_BX = 64, FILL_BY = 4;

// Shared memory of a tile of up to TX x TYM cells: primitives with a 2-cell
// halo, then XMIN/XMAX states of cells x in [-1, TX] and YMIN/YMAX states of
// cells y in [-1, TYM].
template <int TX, int TYM>
constexpr size_t flux_smem_bytes() {
  return sizeof(double) * (4 * (TYM + 4) * (TX + 4) + 2 * (4 * TYM * (TX + 2)) + 2 * (4 * (TYM + 2) * TX));
}

// The fused step's shared memory: the same tile + alignment slack of the
// TMA destination.
template <int TX, int TYM>
constexpr size_t step_smem_bytes() {
  return flux_smem_bytes<TX, TYM>() + 128;
}

// Ghost fill + primitives + CFL term of array cell (i, j) (see the file
// comment); `term`/`flags` receive its CFL term and E2D_FLAG_* bits.
__device__ __forceinline__ void fill_cell(const KParams64 &kp, double *__restrict__ u_in,
                                          double *__restrict__ u_out, double *__restrict__ q,
                                          const int mode, const int i, const int j, double &term,
                                          unsigned int &flags) {
  const KGeom &g = kp.g;
  const KPhys<double> &ph = kp.ph;
  if (i >= g.isize || j >= g.jsize) return;
  bool fu, fv;
  const int si = src_lo_hi(i, g.nx, g.bc_xmin, g.bc_xmax, fu);
  const int sj = src_lo_hi(j, g.ny, g.bc_ymin, g.bc_ymax, fv);
  const bool ghost = (si != i) || (sj != j);
  const size_t s = (size_t)si + (size_t)g.isize * sj;
  const double rho = u_in[s];
  const double e = u_in[s + g.plane];
  double mx = u_in[s + 2 * g.plane];
  double my = u_in[s + 3 * g.plane];
  if (fu) mx = -mx;
  if (fv) my = -my;
  const size_t d = (size_t)i + (size_t)g.isize * j;
  if (mode & FILL_COPY_OUT) {
    u_out[d] = rho;
    u_out[d + g.plane] = e;
    u_out[d + 2 * g.plane] = mx;
    u_out[d + 3 * g.plane] = my;
  }
  if (ghost) {
    if (mode & FILL_GHOSTS_IN) {
      u_in[d] = rho;
      u_in[d + g.plane] = e;
      u_in[d + 2 * g.plane] = mx;
      u_in[d + 3 * g.plane] = my;
    }
  }
  if (mode & (FILL_WRITE_Q | FILL_DT)) {
    const Fp f;
    double dd, p, ux, uy;
    Divisor dv;
    primitives(f, ph, rho, e, mx, my, dd, p, ux, uy, dv);
    if (mode & FILL_WRITE_Q) {
      q[d] = dd;
      q[d + g.plane] = p;
      q[d + 2 * g.plane] = ux;
      q[d + 3 * g.plane] = uy;
    }
    if ((mode & FILL_DT) && !ghost) {
      term = cfl_term(f, ph, dv, p, ux, uy);
      flags |= state_flags(rho, e, mx, my);
    }
  }
}

// Block maximum of the CFL term into *acc (fmax drops NaN like the
// reference's reducer; positive doubles order like their bit patterns) and
// the OR of the flags into *status.  Every thread of the block calls it.
__device__ __forceinline__ void fill_reduce(double term, unsigned int flags, unsigned long long *acc,
                                            unsigned int *status) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) term = fmax_any(term, __shfl_xor_sync(0xffffffffu, term, off));
  flags = __reduce_or_sync(0xffffffffu, flags);
  __shared__ double wmax[FILL_BX * FILL_BY / 32];
  __shared__ unsigned int wflags[FILL_BX * FILL_BY / 32];
  const int tid = threadIdx.y * FILL_BX + threadIdx.x;
  if ((tid & 31) == 0) {
    wmax[tid >> 5] = term;
    wflags[tid >> 5] = flags;
  }
  __syncthreads();
  if (tid == 0) {
    double m = wmax[0];
    unsigned int f = wflags[0];
    for (int w = 1; w < FILL_BX * FILL_BY / 32; ++w) {
      m = fmax_any(m, wmax[w]);
      f |= wflags[w];
    }
    if (gt0(m)) atomicMax(acc, (unsigned long long)__double_as_longlong(m));
    if (f) atomicOr(status, f);
  }
}

__global__ void __launch_bounds__(FILL_BX *FILL_BY)
    k_fill_f64(const KParams64 kp, double *__restrict__ u_in, double *__restrict__ u_out,
               double *__restrict__ q, DevClock *clk, const int mode, const int acc_slot) {
  if ((mode & FILL_DEVICE_CLOCK) && !(clk->t < clk->t_end)) return;
  double term = 0.0;
  unsigned int flags = 0;
  fill_cell(kp, u_in, u_out, q, mode, blockIdx.x * FILL_BX + threadIdx.x, blockIdx.y * FILL_BY + threadIdx.y,
            term, flags);
  if (mode & FILL_DT)
    fill_reduce(term, flags, acc_slot < 0 ? &clk->invdt_bits : &clk->acc[acc_slot & 1], &clk->status);
}

// compute_dt in one launch: the interior's primitives into q, its CFL maximum
// and flags by the last block to finish into *result (pinned host memory),
// and the accumulators cleared for the next call.
__global__ void __launch_bounds__(FILL_BX *FILL_BY)
    k_dt_f64(const KParams64 kp, double *__restrict__ u_in, double *__restrict__ q, DtAcc *acc, DtResult *result) {
  double term = 0.0;
  unsigned int flags = 0;
  fill_cell(kp, u_in, nullptr, q, q ? FILL_WRITE_Q | FILL_DT : FILL_DT, blockIdx.x * FILL_BX + threadIdx.x,
            blockIdx.y * FILL_BY + threadIdx.y, term, flags);
  fill_reduce(term, flags, &acc->bits, &acc->status);
  if (threadIdx.x == 0 && threadIdx.y == 0) {  // the thread that folded
    __threadfence();
    if (atomicAdd(&acc->done, 1u) == gridDim.x * gridDim.y - 1) {
      __threadfence();
      result->bits = __ldcg(&acc->bits);
      result->status = __ldcg(&acc->status);
      acc->bits = 0ull;
      acc->status = 0u;
      acc->done = 0u;
      __threadfence_system();
    }
  }
}

// ------------------------------------------------------------ kernel 2
// Tiles are TX x ty cells, ty <= TYM chosen at run time per grid (see
// choose_f64_tile); results do not depend on the shape.

// Shared memory of a tile: primitives with a 2-cell halo, then the face
// states (the scaled fluxes replace the XMIN / YMIN states in stage 3).  The
// primitives' planes are ty + 4 rows each (as a TMA copy writes them), the
// face states' planes TYM or TYM + 2.
template <int TX, int TYM>
struct TileSmem {
  static constexpr int QW = TX + 4;  // primitives tile width (2-cell halo)
  static constexpr int QH = TYM + 4;
  static constexpr int XW = TX + 2;  // x-face states: cells x in [-1, TX]
  static constexpr int YH = TYM + 2; // y-face states: cells y in [-1, TYM]
  double *sQ, *sXm, *sXp, *sYm, *sYp;
  __device__ explicit TileSmem(double *smem) {
    sQ = smem;                   // [4][ty + 4][QW]  primitives with halo
    sXm = sQ + 4 * QH * QW;      // [4][TYM][XW]  XMIN states, then x-fluxes
    sXp = sXm + 4 * TYM * XW;    // [4][TYM][XW]  XMAX states
    sYm = sXp + 4 * TYM * XW;    // [4][YH][TX]  YMIN states, then y-fluxes
    sYp = sYm + 4 * YH * TX;     // [4][YH][TX]  YMAX states
  }
};

// Stage 1 from the primitives of the interior cells (the fused step where its
// halo reaches ghost cells, the other steps throughout): the
// primitives of a ghost cell are those of its source cell with the normal
// velocity negated where the boundary reflects -- bit for bit the
// primitives of the reference's ghost-filled state (u = mx / d changes only
// its sign with mx; e, p and c depend on u^2).  Only interior cells of q are
// read.
template <int TX, int NT>
__device__ __forceinline__ void gather_qtile(const KGeom &g, const double *q, int i0, int j0, int ty,
                                             double *sQ) {
  constexpr int QW = TX + 4;
  const int n = (ty + 4) * QW;
  for (int k = threadIdx.x; k < n; k += NT) {
    const int y = k / QW, x = k - y * QW;
    const int gi = i0 + x, gj = j0 + y;
    if (gi < g.isize && gj < g.jsize) {
      bool fu, fv;
      const int si = src_lo_hi(gi, g.nx, g.bc_xmin, g.bc_xmax, fu);
      const int sj = src_lo_hi(gj, g.ny, g.bc_ymin, g.bc_ymax, fv);
      const size_t s = (size_t)si + (size_t)g.isize * sj;
      const double ux = __ldcg(q + s + 2 * g.plane), uy = __ldcg(q + s + 3 * g.plane);
      sQ[k] = __ldcg(q + s);
      sQ[n + k] = __ldcg(q + s + g.plane);
      sQ[2 * n + k] = fu ? Fp::neg(ux) : ux;
      sQ[3 * n + k] = fv ? Fp::neg(uy) : uy;
    } else {
#pragma unroll
      for (int v = 0; v < 4; ++v) sQ[v * n + k] = 1.0;
    }
  }
}

// Stage 2 of a tile whose primitives are in shared memory (the caller has
// synchronised after writing them): slopes, trace sources and face states of
// the tile cells and of the 1-cell ring (corners excluded) --
// src/HydroBaseFunctor.h:214-291.
template <int TX, int TYM, int NT, bool FAST, class F>
__device__ __forceinline__ void tile_faces(const F &fp64, const KPhys<double> &ph, const double dtdx,
                                           const double dtdy, const int ty, double *smem) {
  using T = TileSmem<TX, TYM>;
  constexpr int QW = T::QW, XW = T::XW, YH = T::YH;
  const T sm(smem);
  const double *sQ = sm.sQ;
  const int qs = QW * (ty + 4);
  // Items enumerate the tile and its 1-cell ring without the ring's four
  // corners, which carry no face.  The FP64 pipe takes as long for a warp
  // instruction with a few active lanes as for a full one, so a partial
  // round costs what its busiest scheduler's warps cost.
  const int st_kind = (ph.slope_type == 2.0) ? 2 : (ph.slope_type == 1.0) ? 1 : 0;
  const int ns2 = (ty + 2) * XW - 4;
  const double hdtdx = half(dtdx), hdtdy = half(dtdy);
  for (int k = threadIdx.x; k < ns2; k += NT) {
    int yy, xx;  // cell (xx-1, yy-1) of the tile
    if (k < TX) {
      yy = 0;
      xx = k + 1;
    } else if (k < TX + ty * XW) {
      const int r = k - TX;
      yy = 1 + r / XW;
      xx = r - (yy - 1) * XW;
    } else {
      yy = ty + 1;
      xx = k - (TX + ty * XW) + 1;
    }
    const bool xin = (xx >= 1) && (xx <= TX);
    const bool yin = (yy >= 1) && (yy <= ty);
    const int c = (yy + 1) * QW + (xx + 1);
    double qc[4], dqx[4], dqy[4], hx[4], hy[4];
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      const double *P = sQ + v * qs;
      qc[v] = P[c];
      slope(fp64, st_kind, qc[v], P[c + 1], P[c - 1], dqx[v], hx[v]);
      slope(fp64, st_kind, qc[v], P[c + QW], P[c - QW], dqy[v], hy[v]);
    }
    double s0[4];
    if (FAST)
      trace_sources_fast(fp64, ph, qc, dqx, dqy, s0);
    else
      trace_sources(fp64, ph, qc, dqx, dqy, s0);
    if (yin) {
      const int o = (yy - 1) * XW + xx;
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        double fm, fp;
        if (FAST)
          face_pair_fast(fp64, ph, v, qc[v], hx[v], s0[v], hdtdx, fm, fp);
        else
          face_pair(fp64, ph, v, qc[v], hx[v], s0[v], dtdx, hdtdx, fm, fp);
        if (xx >= 1) sm.sXm[v * TYM * XW + o] = fm;
        if (xx <= TX) sm.sXp[v * TYM * XW + o] = fp;
      }
    }
    if (xin) {
      const int o = yy * TX + (xx - 1);
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        double fm, fp;
        if (FAST)
          face_pair_fast(fp64, ph, v, qc[v], hy[v], s0[v], hdtdy, fm, fp);
        else
          face_pair(fp64, ph, v, qc[v], hy[v], s0[v], dtdy, hdtdy, fm, fp);
        if (yy >= 1) sm.sYm[v * YH * TX + o] = fm;
        if (yy <= ty) sm.sYp[v * YH * TX + o] = fp;
      }
    }
  }
}

// Stage 2 with a lane per cell and variable, for tiles so small that their
// cells do not fill the block's warps: a quarter of the instructions in each
// warp's chain (23 FP64 instead of 80; 21 % more of them in all).  The lanes
// of a cell exchange what the trace sources need of the other variables.
// Same operations, same bits.
template <int TX, int TYM, int NT, bool FAST, class F>
__device__ __forceinline__ void tile_faces_split(const F &f, const KPhys<double> &ph, const double dtdx,
                                                 const double dtdy, const int ty, double *smem) {
  using T = TileSmem<TX, TYM>;
  constexpr int QW = T::QW, XW = T::XW, YH = T::YH;
  const T sm(smem);
  const int qs = QW * (ty + 4);
  const int st_kind = (ph.slope_type == 2.0) ? 2 : (ph.slope_type == 1.0) ? 1 : 0;
  const int ns2 = (ty + 2) * XW - 4;
  const double hdtdx = half(dtdx), hdtdy = half(dtdy);
  const int v = threadIdx.x & 3;
  auto other = [](double x, int w) { return __shfl_sync(0xffffffffu, x, w, 4); };
  for (int k0 = threadIdx.x >> 2; (k0 & ~7) < ns2; k0 += NT / 4) {  // whole warps
    const int k = k0 < ns2 ? k0 : ns2 - 1;
    int yy, xx;  // cell (xx-1, yy-1) of the tile
    if (k < TX) {
      yy = 0;
      xx = k + 1;
    } else if (k < TX + ty * XW) {
      const int r = k - TX;
      yy = 1 + r / XW;
      xx = r - (yy - 1) * XW;
    } else {
      yy = ty + 1;
      xx = k - (TX + ty * XW) + 1;
    }
    const double *P = sm.sQ + v * qs + (yy + 1) * QW + (xx + 1);
    const double q = P[0];
    double dqx, dqy, hx, hy;
    slope(f, st_kind, q, P[1], P[-1], dqx, hx);
    slope(f, st_kind, q, P[QW], P[-QW], dqy, hy);
    const double r = other(q, E2D_ID), u = other(q, E2D_IU), w = other(q, E2D_IV);
    const double div = f.add(other(dqx, E2D_IU), other(dqy, E2D_IV));
    const double dpx = other(dqx, E2D_IP), dpy = other(dqy, E2D_IP);
    // the term of the variable's source beside its transport
    const double dg = f.mul(div, ph.gamma0);
    const double m = f.mul(v == E2D_IP ? dg : div, q), g = quot(v == E2D_IU ? dpx : dpy, r);
    const double ex = v < E2D_IU ? m : g;
    const double nu = f.neg(u);
    const double s0 = FAST ? fma(nu, dqx, fma(f.neg(w), dqy, f.neg(ex)))
                           : f.sub(f.sub(f.mul(nu, dqx), f.mul(w, dqy)), ex);
    double xm, xp, ym, yp;
    if (FAST) {
      face_pair_fast(f, ph, v, q, hx, s0, hdtdx, xm, xp);
      face_pair_fast(f, ph, v, q, hy, s0, hdtdy, ym, yp);
    } else {
      face_pair(f, ph, v, q, hx, s0, dtdx, hdtdx, xm, xp);
      face_pair(f, ph, v, q, hy, s0, dtdy, hdtdy, ym, yp);
    }
    if (k0 < ns2 && yy >= 1 && yy <= ty) {
      const int o = v * TYM * XW + (yy - 1) * XW + xx;
      if (xx >= 1) sm.sXm[o] = xm;
      if (xx <= TX) sm.sXp[o] = xp;
    }
    if (k0 < ns2 && xx >= 1 && xx <= TX) {
      const int o = v * YH * TX + yy * TX + (xx - 1);
      if (yy >= 1) sm.sYm[o] = ym;
      if (yy <= ty) sm.sYp[o] = yp;
    }
  }
}

// Stage 2 of a tile: by variable for the small tiles (which are the ones
// without integer products), else by cell.
template <int TX, int TYM, int NT, bool FAST, class F>
__device__ __forceinline__ void tile_stage2(const F &f, const KPhys<double> &ph, const double dtdx, const double dtdy,
                                            const int ty, double *smem) {
  if constexpr (TX <= 8)
    tile_faces_split<TX, TYM, NT, FAST>(f, ph, dtdx, dtdy, ty, smem);
  else
    tile_faces<TX, TYM, NT, FAST>(f, ph, dtdx, dtdy, ty, smem);
}

// Stage 3 (after a block barrier): one Riemann solve per face; the flux,
// scaled by dt/dx or dt/dy (the fast forms scale in the update), replaces
// the right-hand state, which no other face reads.
template <int RS, int TX, int TYM, int NT, bool FAST, class F>
__device__ __forceinline__ void tile_riemann(const F &fp64, const KPhys<double> &ph, const double dtdx,
                                             const double dtdy, const int ty, double *smem) {
  using T = TileSmem<TX, TYM>;
  constexpr int XW = T::XW, YH = T::YH;
  const T sm(smem);
  const int nxf = (TX + 1) * ty;
  const int nf = nxf + TX * (ty + 1);
  // one copy of the solver for both directions: the faces' states by
  // pointer, with the plane stride and the planes of the normal and the
  // tangential velocity (y: swapped, src/HydroRunFunctors.h:628-632)
  for (int k = threadIdx.x; k < nf; k += NT) {
    const bool xd = k < nxf;
    const int kk = xd ? k : k - nxf;
    const int w = xd ? TX + 1 : TX;
    const int y = xd ? kk / (TX + 1) : kk / TX, x = kk - y * w;
    const int ol = xd ? y * XW + x : kk;
    const int ps = xd ? TYM * XW : YH * TX;
    const double *pl = (xd ? sm.sXp : sm.sYp) + ol;
    double *pr = (xd ? sm.sXm + 1 : sm.sYm + TX) + ol;
    const int on = xd ? 2 * ps : 3 * ps, ot = xd ? 3 * ps : 2 * ps;
    const double ql[4] = {pl[0], pl[ps], pl[on], pl[ot]}, qr[4] = {pr[0], pr[ps], pr[on], pr[ot]};
    double f[4];
    riemann_sel<RS, FAST>(fp64, ph, ql, qr, f);
    if (!FAST) {
      const double dtd = xd ? dtdx : dtdy;
#pragma unroll
      for (int v = 0; v < 4; ++v) f[v] = fp64.xmul(f[v], dtd);
    }
    pr[0] = f[E2D_ID];
    pr[ps] = f[E2D_IP];
    pr[on] = f[E2D_IU];
    pr[ot] = f[E2D_IV];
  }
}

// The input values of a thread's cells of the tile, loaded before the
// Riemann solves so that the update does not wait for them.
template <int TX, int TYM, int NT>
struct TileCells {
  static constexpr int N = (TX * TYM + NT - 1) / NT;
  double u[N][4];
  // cell n of the thread: its offset in a plane, or -1
  static __device__ __forceinline__ long long offset(const KGeom &g, int i0, int j0, int ty, int n, int &x, int &y) {
    const int k = threadIdx.x + n * NT;
    y = k / TX;
    x = k - y * TX;
    const int gi = i0 + 2 + x, gj = j0 + 2 + y;
    return (y < ty && gi < g.nx + 2 && gj < g.ny + 2) ? gi + (long long)g.isize * gj : -1;
  }
  __device__ __forceinline__ void load(const KGeom &g, const double *u_in, int i0, int j0, int ty) {
#pragma unroll
    for (int n = 0; n < N; ++n) {
      int x, y;
      const long long s = offset(g, i0, j0, ty, n, x, y);
#pragma unroll
      for (int v = 0; v < 4; ++v) u[n][v] = s >= 0 ? __ldcg(u_in + s + v * g.plane) : 0.0;
    }
  }
};

// The conservative update of cell (x, y) of a tile in the reference's order
// (src/HydroRunFunctors.h:691-713): +Fx(i) -Fx(i+1) +Fy(j) -Fy(j+1).  The
// fast forms take unscaled fluxes: one difference and one FMA a direction.
template <int TX, int TYM, bool FAST, class F>
__device__ __forceinline__ double update_var(const F &f, const TileSmem<TX, TYM> &sm, int v, int x, int y,
                                             double uu, double dtdx, double dtdy) {
  using T = TileSmem<TX, TYM>;
  const double *fx = sm.sXm + v * TYM * T::XW + y * T::XW + x + 1;
  const double *fy = sm.sYm + v * T::YH * TX + (y + 1) * TX + x;
  if (FAST) return fma(f.sub(fx[0], fx[1]), dtdx, fma(f.sub(fy[0], fy[TX]), dtdy, uu));
  uu = f.add(uu, fx[0]);
  uu = f.sub(uu, fx[1]);
  uu = f.add(uu, fy[0]);
  uu = f.sub(uu, fy[TX]);
  return uu;
}

// The ghost cells next to a tile -- those whose nearest interior cell is in
// it -- receive the ghost fill of u_in in both states, read from interior
// cells of u_in only (no block writes those during a step).
template <int TX, int NT>
__device__ __forceinline__ void ghost_fill_tile(const KGeom &g, double *u_in, double *u_out,
                                                int i0, int j0, int ty, bool lo_x, bool hi_x, bool lo_y, bool hi_y) {
  if (!(lo_x || hi_x || lo_y || hi_y)) return;
  const int xa = lo_x ? 0 : i0 + 2, xb = hi_x ? g.isize : i0 + 2 + TX;
  const int ya = lo_y ? 0 : j0 + 2, yb = hi_y ? g.jsize : j0 + 2 + ty;
  const int w = xb - xa, n = w * (yb - ya);
  for (int k = threadIdx.x; k < n; k += NT) {
    const int j = ya + k / w, i = xa + k % w;
    if (i >= 2 && i < g.nx + 2 && j >= 2 && j < g.ny + 2) continue;
    bool fu, fv;
    const int si = src_lo_hi(i, g.nx, g.bc_xmin, g.bc_xmax, fu);
    const int sj = src_lo_hi(j, g.ny, g.bc_ymin, g.bc_ymax, fv);
    const size_t s = (size_t)si + (size_t)g.isize * sj, d = (size_t)i + (size_t)g.isize * j;
    double v4[4];
#pragma unroll
    for (int v = 0; v < 4; ++v) v4[v] = __ldcg(u_in + s + v * g.plane);
    if (fu) v4[E2D_IU] = -v4[E2D_IU];
    if (fv) v4[E2D_IV] = -v4[E2D_IV];
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      u_in[d + v * g.plane] = v4[v];
      u_out[d + v * g.plane] = v4[v];
    }
  }
}

// Stages 1-4 of the two-launch step for tile (bx, by) of a grid,
// block-wide; the caller provides dt/dx, dt/dy and the tile's shared memory.
template <int RS, int TX, int TYM, int NT, class F>
__device__ __forceinline__ void flux_tile(const KParams64 &kp, const double *q, double *u_in, double *u_out,
                                          const int bx, const int by, const int ty, const double dtdx,
                                          const double dtdy, double *smem) {
  const KGeom &g = kp.g;
  const int i0 = bx * TX;  // array column of the tile's first halo cell
  const int j0 = by * ty;
  const F f;
  gather_qtile<TX, NT>(g, q, i0, j0, ty, smem);
  __syncthreads();
  tile_stage2<TX, TYM, NT, false>(f, kp.ph, dtdx, dtdy, ty, smem);
  TileCells<TX, TYM, NT> cells;
  cells.load(g, u_in, i0, j0, ty);
  __syncthreads();
  tile_riemann<RS, TX, TYM, NT, false>(f, kp.ph, dtdx, dtdy, ty, smem);
  __syncthreads();
  const TileSmem<TX, TYM> sm(smem);
  // stage 4: conservative update
#pragma unroll
  for (int n = 0; n < cells.N; ++n) {
    int x, y;
    const long long s = cells.offset(g, i0, j0, ty, n, x, y);
    if (s >= 0) {
#pragma unroll
      for (int v = 0; v < 4; ++v)
        u_out[s + v * g.plane] = update_var<TX, TYM, false>(f, sm, v, x, y, cells.u[n][v], dtdx, dtdy);
    }
  }
  ghost_fill_tile<TX, NT>(g, u_in, u_out, i0, j0, ty, bx == 0, bx == (int)gridDim.x - 1, by == 0,
                          by == (int)gridDim.y - 1);
}

template <int RS, int TX, int TYM, int NT, int MINB, bool XMUL>
__global__ void __launch_bounds__(NT, MINB)
    k_flux_update_f64(const KParams64 kp, const double *q, double *u_in, double *u_out, DevClock *clk,
                      const int use_clock, const double host_dt, double *dt_trace) {
  extern __shared__ double smem[];
  const KPhys<double> &ph = kp.ph;
  const int tid = threadIdx.x;
  // dt of this step (the caller's, or src/main.cpp:128-134 on the device)
  // and dt/dx, dt/dy, computed once per block and broadcast: per-thread FP64
  // divisions here would cost ~2 divisions per cell on the FP64 pipe
  __shared__ double s_dt[3];
  __shared__ int s_run;
  if (tid == 0) {
    double dt = host_dt;
    int run = 1;
    if (use_clock) {
      run = clk->t < clk->t_end;
      dt = step_dt(ph, clk->invdt_bits, clk->t, clk->t_end);
    }
    s_dt[0] = dt;
    s_dt[1] = quot(dt, ph.dx);
    s_dt[2] = quot(dt, ph.dy);
    s_run = run;
  }
  __syncthreads();
  if (!s_run) return;
  const double dt = s_dt[0];
  flux_tile<RS, TX, TYM, NT, f64x::FpT<XMUL>>(kp, q, u_in, u_out, blockIdx.x, blockIdx.y, kp.ty, s_dt[1], s_dt[2], smem);

  if (!use_clock) return;
  // the last block to finish advances the loop state (src/main.cpp:139-143)
  __syncthreads();
  if (tid == 0) {
    __threadfence();
    const unsigned int nblocks = gridDim.x * gridDim.y;
    const unsigned int ticket = atomicAdd(&clk->done_blocks, 1u);
    if (ticket == nblocks - 1) {
      __threadfence();
      const int ns = clk->nstep;
      const int slot = ns - clk->trace_base;
      if (dt_trace && slot >= 0 && slot < clk->trace_cap) dt_trace[slot] = dt;
      if (!(dt > 0.0) || nonfinite(dt)) clk->status |= E2D_FLAG_BAD_DT;
      clk->dt = dt;
      clk->t = clk->t + dt;  // only this block writes t during the step
      clk->nstep = ns + 1;
      clk->invdt_bits = 0ull;
      clk->done_blocks = 0u;
      __threadfence();
    }
  }
}

// ------------------------------------------------------------ the fused step
// Block maximum of the CFL term into *acc and the OR of the flags into
// *status, one atomic of each per block (fmax drops NaN like the reference's
// reducer; positive doubles order like their bit patterns).
template <int NT>
__device__ __forceinline__ void block_fold(double term, unsigned int flags, unsigned long long *acc,
                                           unsigned int *status) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) term = fmax_any(term, __shfl_xor_sync(0xffffffffu, term, off));
  flags = __reduce_or_sync(0xffffffffu, flags);
  __shared__ double wmax[NT / 32];
  __shared__ unsigned int wflags[NT / 32];
  const int tid = threadIdx.x;
  if ((tid & 31) == 0) {
    wmax[tid >> 5] = term;
    wflags[tid >> 5] = flags;
  }
  __syncthreads();
  if (tid == 0) {
    double m = wmax[0];
    unsigned int f = wflags[0];
#pragma unroll
    for (int w = 1; w < NT / 32; ++w) {
      m = fmax_any(m, wmax[w]);
      f |= wflags[w];
    }
    if (gt0(m)) atomicMax(acc, (unsigned long long)__double_as_longlong(m));
    if (f) atomicOr(status, f);
  }
}

// A new cell of the fused step: its state and primitives, its CFL term into
// the running maximum and its flags.
template <bool FAST, class F>
__device__ __forceinline__ void finish_cell(const F &f, const KParams64 &kp, long long s, const double un[4],
                                            double *u_out, double *q_out, double &term, unsigned int &flags) {
  const KGeom &g = kp.g;
  const KPhys<double> &ph = kp.ph;
#pragma unroll
  for (int v = 0; v < 4; ++v) u_out[s + v * g.plane] = un[v];
  double dd, p, ux, uy;
  Divisor dv;
  if (FAST)
    primitives_fast(f, ph, un[E2D_ID], un[E2D_IP], un[E2D_IU], un[E2D_IV], dd, p, ux, uy, dv);
  else
    primitives(f, ph, un[E2D_ID], un[E2D_IP], un[E2D_IU], un[E2D_IV], dd, p, ux, uy, dv);
  q_out[s] = dd;
  q_out[s + g.plane] = p;
  q_out[s + 2 * g.plane] = ux;
  q_out[s + 3 * g.plane] = uy;
  term = fmax_any(term, FAST ? cfl_term_fast(f, ph, dv, p, ux, uy) : cfl_term(f, ph, dv, p, ux, uy));
  flags |= state_flags(un[E2D_ID], un[E2D_IP], un[E2D_IU], un[E2D_IV]);
}

// The last block to finish a step advances the loop state
// (src/main.cpp:139-143); one thread per block, after a block barrier.
__device__ __forceinline__ void finish_step64(DevClock *clk, const double dt, const int par, double *dt_trace) {
  __threadfence();
  const unsigned int ticket = atomicAdd(&clk->done_blocks, 1u);
  if (ticket != gridDim.x * gridDim.y - 1) return;
  __threadfence();
  const int ns = clk->nstep;
  const int slot = ns - clk->trace_base;
  if (dt_trace && slot >= 0 && slot < clk->trace_cap) dt_trace[slot] = dt;
  if (!(dt > 0.0) || nonfinite(dt)) clk->status |= E2D_FLAG_BAD_DT;
  clk->dt = dt;
  clk->t = clk->t + dt;  // only this block writes t during the step
  clk->nstep = ns + 1;
  clk->acc[par] = 0ull;  // read by this step; folded into by the next
  clk->done_blocks = 0u;
  __threadfence();
}

// The fused step's epilogue for the cells of a tile whose fluxes are in
// shared memory: the conservative update into u_out, the primitives of the
// new cells into q_out and the running maximum of their CFL terms and flags.
template <int TX, int TYM, int NT, bool FAST, class F>
__device__ __forceinline__ void step_epilogue(const F &f, const KParams64 &kp, const TileCells<TX, TYM, NT> &cells,
                                              double *u_out, double *q_out, int i0, int j0, int ty, double dtdx, double dtdy, double *smem, double &term,
                                              unsigned int &flags) {
  const KGeom &g = kp.g;
  const KPhys<double> &ph = kp.ph;
  const TileSmem<TX, TYM> sm(smem);
#pragma unroll
  for (int n = 0; n < cells.N; ++n) {
    int x, y;
    const long long s = cells.offset(g, i0, j0, ty, n, x, y);
    if (s >= 0) {
      double un[4];
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        un[v] = update_var<TX, TYM, FAST>(f, sm, v, x, y, cells.u[n][v], dtdx, dtdy);
      }
      finish_cell<FAST>(f, kp, s, un, u_out, q_out, term, flags);
    }
  }
}

// One whole time step of the device loop (src/main.cpp:128-143 around
// godunov_unsplit_impl, src/HydroRun.h:279-364), one TX x ty tile per block:
//  - dt from the CFL maximum of the input state, clock->acc[nstep & 1],
//    which the previous step (or the prologue fill) folded;
//  - stage 1: primitives of the tile and its 2-cell halo, from q_in (the
//    primitives of u_in's interior cells): one TMA copy of the box for tiles
//    whose halo is interior, else a gather through the boundary map;
//  - stages 2-3: slopes, trace, face states, one Riemann solve per face;
//  - epilogue: the conservative update into u_out, the primitives of the
//    new cells into q_out and their CFL term, folded into
//    clock->acc[(nstep + 1) & 1] with one atomic per block;
//  - boundary tiles write the ghost fill of u_in into the ghost cells of
//    both states (make_boundaries + deep_copy of the reference), reading
//    only interior cells of u_in, which no block writes;
//  - the last block to finish advances the loop state.
// Bit-identical to the two-launch step; FP64 work per cell is the same.
template <int RS, int TX, int TYM, int NT, int MINB, bool XMUL, bool FAST>
__global__ void __launch_bounds__(NT, MINB)
    k_step_f64(const KParams64 kp, const __grid_constant__ CUtensorMap tm_q, const int use_tma,
               const double *__restrict__ q_in, double *__restrict__ q_out, double *__restrict__ u_in,
               double *__restrict__ u_out, DevClock *clk, double *__restrict__ dt_trace) {
  extern __shared__ unsigned char smem_raw[];
  // a TMA destination must be 128-byte aligned
  double *smem = reinterpret_cast<double *>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~uintptr_t(127));
  __shared__ double s_dt[3];
  __shared__ int s_run, s_par;
  __shared__ __align__(8) unsigned long long s_bar;
  const KGeom &g = kp.g;
  const KPhys<double> &ph = kp.ph;
  const int tid = threadIdx.x;
  const int bx = blockIdx.x, by = blockIdx.y;
  const int ty = kp.ty;
  const int i0 = bx * TX, j0 = by * ty;  // array cell of the halo box's corner
  constexpr int QW = TX + 4;
  const bool tma_tile = use_tma && i0 >= 2 && j0 >= 2 && i0 + QW <= g.nx + 2 && j0 + ty + 4 <= g.ny + 2;
  if (tid == 0) {
    const int run = clk->t < clk->t_end;
    const int par = clk->nstep & 1;
    const double dt = step_dt(ph, clk->acc[par], clk->t, clk->t_end);
    s_dt[0] = dt;
    s_dt[1] = quot(dt, ph.dx);
    s_dt[2] = quot(dt, ph.dy);
    s_run = run;
    s_par = par;
    if (run && tma_tile) {
      mbar_init(&s_bar, 1u);
      mbar_init_fence();
      // wait_test: tile (1, 1) never copies, so its bounded wait runs out
      if (!(kp.wait_test == 1 && bx == 1 && by == 1)) {
        mbar_arrive_expect(&s_bar, (unsigned int)(sizeof(double) * 4 * QW) * (unsigned int)(ty + 4));
        tma_load_3d(smem, &tm_q, i0, j0, 0, &s_bar);
      }
    }
  }
  __syncthreads();
  if (!s_run) return;  // past t_end: no copy was issued
  const int par = s_par;
  bool ok = true;
  if (tma_tile) {
    ok = __syncthreads_and(mbar_wait(&s_bar, 0u));
    if (!ok) {
      // flag the step, then wait (bounded) for the copy that may still land
      // in this block's shared memory before leaving the tile
      if (tid == 0) atomicOr(&clk->status, E2D_FLAG_TIMEOUT);
      mbar_wait(&s_bar, 0u);
      __syncthreads();
    }
  } else {
    gather_qtile<TX, NT>(g, q_in, i0, j0, ty, smem);
    __syncthreads();
  }

  const f64x::FpT<XMUL> f;
  double term = 0.0;
  unsigned int flags = 0;
  if (ok) {
    const double dtdx = s_dt[1], dtdy = s_dt[2];
    tile_stage2<TX, TYM, NT, FAST>(f, ph, dtdx, dtdy, ty, smem);
    TileCells<TX, TYM, NT> cells;
    cells.load(g, u_in, i0, j0, ty);
    __syncthreads();
    tile_riemann<RS, TX, TYM, NT, FAST>(f, ph, dtdx, dtdy, ty, smem);
    __syncthreads();
    step_epilogue<TX, TYM, NT, FAST>(f, kp, cells, u_out, q_out, i0, j0, ty, dtdx, dtdy, smem, term, flags);
  }
  ghost_fill_tile<TX, NT>(g, u_in, u_out, i0, j0, ty, bx == 0, bx == (int)gridDim.x - 1, by == 0,
                          by == (int)gridDim.y - 1);

  block_fold<NT>(term, flags, &clk->acc[par ^ 1], &clk->status);

  __syncthreads();
  if (tid == 0) finish_step64(clk, s_dt[0], par, dt_trace);
}

// ------------------------------------------------------------ the march
// The fused step of a large grid: a block walks a segment of a 32-column
// strip upwards in chunks of CHUNK rows.  Each chunk traces its own rows
// once -- the face states, x- and y-fluxes of the last row stay in shared
// memory for the next chunk (16 rows of each, used as rings) -- so only the
// strip's two side columns are traced twice, where a tile traces a ring of
// cells around it.  15 rows make 16 warps of traced cells and 31 of Riemann
// solves, two and four full rounds of the block's 8 warps, which is what 13
// rows of a tile take.  The next chunk's primitives arrive by TMA (where the
// strip is away from the boundary) while this one is computed, and dt, the
// CFL fold and the block's launch are paid once a segment.
//
// Rows of a chunk are numbered 1 .. CHUNK (array rows r0 .. r0 + CHUNK - 1),
// row 0 is the last one of the chunk before; the chunk updates rows 0 ..
// CHUNK - 1, whose upper y-flux it has.  A segment of rows jb .. je starts at
// r0 = jb - 1 and ends once row je + 1 is traced.
constexpr int MTX = 32, CHUNK = 15, MNT = 256, MRING = 16;
constexpr int MQW = MTX + 4, MQH = CHUNK + 2, MXW = MTX + 2;
static_assert((MRING & (MRING - 1)) == 0 && MRING == CHUNK + 1, "row k of a chunk sits in slot (base + k) mod 16");
constexpr size_t kMarchQ = sizeof(double) * 4 * MQH * MQW;  // one chunk's primitives
static_assert(kMarchQ % 128 == 0, "a TMA destination is 128-byte aligned");
constexpr size_t march_smem_bytes() {
  return 2 * kMarchQ + sizeof(double) * (2 * 4 * MRING * MXW + 2 * 4 * MRING * MTX) + 128;
}

template <int RS, bool FAST>
__global__ void __launch_bounds__(MNT, 2)
    k_march_f64(const KParams64 kp, const __grid_constant__ CUtensorMap tm_q, const int use_tma, const double *q_in,
                double *q_out, double *u_in, double *u_out, DevClock *clk, double *dt_trace) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char *base_ptr = smem_raw + ((128u - (smem_u32(smem_raw) & 127u)) & 127u);
  double *sQ[2] = {reinterpret_cast<double *>(base_ptr), reinterpret_cast<double *>(base_ptr + kMarchQ)};
  double *sXm = reinterpret_cast<double *>(base_ptr + 2 * kMarchQ);  // [4][16][34] XMIN states, then x-fluxes
  double *sXp = sXm + 4 * MRING * MXW;                               // [4][16][34] XMAX states
  double *sYm = sXp + 4 * MRING * MXW;                               // [4][16][32] YMIN states, then y-fluxes
  double *sYp = sYm + 4 * MRING * MTX;                               // [4][16][32] YMAX states
  __shared__ double s_dt[3];
  __shared__ int s_run, s_par;
  __shared__ __align__(8) unsigned long long s_bar[2];
  const KGeom &g = kp.g;
  const KPhys<double> &ph = kp.ph;
  const int tid = threadIdx.x;
  const int bx = blockIdx.x, i0 = bx * MTX;
  const int jb = 2 + blockIdx.y * kp.march_rows, je = min(jb + kp.march_rows, g.ny + 2) - 1;
  const bool tma_x = use_tma && i0 >= 2 && i0 + MQW <= g.nx + 2;
  // primitives of rows r0 - 1 .. r0 + CHUNK of a chunk by one TMA copy
  auto by_tma = [&](int r0) { return tma_x && r0 - 1 >= 2 && r0 + CHUNK <= g.ny + 1; };
  auto issue = [&](int r0, int b) {
    // wait_test: block (1, 0)'s second chunk is never copied, so its wait runs out
    if (kp.wait_test == 1 && bx == 1 && blockIdx.y == 0 && b == 1) return;
    fence_proxy_async_smem();
    mbar_arrive_expect(&s_bar[b], (unsigned int)kMarchQ);
    tma_load_3d(sQ[b], &tm_q, i0, r0 - 1, 0, &s_bar[b]);
  };
  if (tid == 0) {
    mbar_init(&s_bar[0], 1u);
    mbar_init(&s_bar[1], 1u);
    mbar_init_fence();
    const int run = clk->t < clk->t_end;
    s_run = run;
    s_par = clk->nstep & 1;
    if (run && by_tma(jb - 1)) issue(jb - 1, 0);
    const double dt = step_dt(ph, clk->acc[clk->nstep & 1], clk->t, clk->t_end);
    s_dt[0] = dt;
    s_dt[1] = quot(dt, ph.dx);
    s_dt[2] = quot(dt, ph.dy);
  }
  __syncthreads();
  if (!s_run) return;  // past t_end: no copy was issued
  const int par = s_par;
  const double dtdx = s_dt[1], dtdy = s_dt[2];
  const double hdtdx = half(dtdx), hdtdy = half(dtdy);
  const int st_kind = (ph.slope_type == 2.0) ? 2 : (ph.slope_type == 1.0) ? 1 : 0;
  const Fp f;
  double term = 0.0;
  unsigned int flags = 0, phase = 0;
  bool ok = true;
  int base = 0, buf = 0;
  for (int r0 = jb - 1; r0 <= je + 1; r0 += CHUNK, buf ^= 1, base = (base + CHUNK) & (MRING - 1)) {
    auto slot = [&](int k) { return (base + k) & (MRING - 1); };
    // stage 1: this chunk's primitives; the next one's on their way (its
    // buffer was last read before the barriers of the previous chunk)
    if (by_tma(r0)) {
      ok = __syncthreads_and(mbar_wait(&s_bar[buf], (phase >> buf) & 1u));
      if (!ok) {
        // flag the step, then wait (bounded) for the copy that may still land
        // in this block's shared memory before leaving the segment
        if (tid == 0) atomicOr(&clk->status, E2D_FLAG_TIMEOUT);
        mbar_wait(&s_bar[buf], (phase >> buf) & 1u);
        __syncthreads();
        break;
      }
      phase ^= 1u << buf;
    } else {
      gather_qtile<MTX, MNT>(g, q_in, i0, r0 - 1, CHUNK - 2, sQ[buf]);
      __syncthreads();
    }
    if (tid == 0 && r0 + CHUNK <= je + 1 && by_tma(r0 + CHUNK)) issue(r0 + CHUNK, buf ^ 1);

    // stage 2: face states of rows 1 .. CHUNK, columns -1 .. 32
    for (int k = tid; k < CHUNK * MXW; k += MNT) {
      const int y = k / MXW, xx = k - y * MXW, sl = slot(y + 1);
      const double *P = sQ[buf] + (y + 1) * MQW + (xx + 1);
      double qc[4], dqx[4], dqy[4], hx[4], hy[4], s0[4];
#pragma unroll
      for (int v = 0; v < 4; ++v, P += MQH * MQW) {
        qc[v] = P[0];
        slope(f, st_kind, qc[v], P[1], P[-1], dqx[v], hx[v]);
        slope(f, st_kind, qc[v], P[MQW], P[-MQW], dqy[v], hy[v]);
      }
      if (FAST)
        trace_sources_fast(f, ph, qc, dqx, dqy, s0);
      else
        trace_sources(f, ph, qc, dqx, dqy, s0);
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        double fm, fp;
        if (FAST)
          face_pair_fast(f, ph, v, qc[v], hx[v], s0[v], hdtdx, fm, fp);
        else
          face_pair(f, ph, v, qc[v], hx[v], s0[v], dtdx, hdtdx, fm, fp);
        const int o = (v * MRING + sl) * MXW + xx;
        if (xx >= 1) sXm[o] = fm;
        if (xx <= MTX) sXp[o] = fp;
      }
      if (xx >= 1 && xx <= MTX) {
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          double fm, fp;
          if (FAST)
            face_pair_fast(f, ph, v, qc[v], hy[v], s0[v], hdtdy, fm, fp);
          else
            face_pair(f, ph, v, qc[v], hy[v], s0[v], dtdy, hdtdy, fm, fp);
          const int o = (v * MRING + sl) * MTX + xx - 1;
          sYm[o] = fm;
          sYp[o] = fp;
        }
      }
    }
    // the cells this chunk updates, loaded ahead of the Riemann solves
    constexpr int N = (MTX * CHUNK + MNT - 1) / MNT;
    double u[N][4];
    long long at[N];
#pragma unroll
    for (int n = 0; n < N; ++n) {
      const int k = tid + n * MNT, y = k / MTX, gi = i0 + 2 + (k - y * MTX), gj = r0 - 1 + y;
      at[n] = (y < CHUNK && gi < g.nx + 2 && gj >= jb && gj <= je) ? gi + (long long)g.isize * gj : -1;
#pragma unroll
      for (int v = 0; v < 4; ++v) u[n][v] = at[n] >= 0 ? __ldcg(u_in + at[n] + v * g.plane) : 0.0;
    }
    __syncthreads();

    // stage 3: x-faces of rows 1 .. CHUNK, y-faces below them
    constexpr int nxf = (MTX + 1) * CHUNK, nf = nxf + MTX * CHUNK;
    for (int k = tid; k < nf; k += MNT) {
      const bool xd = k < nxf;
      const int kk = xd ? k : k - nxf;
      const int y = xd ? kk / (MTX + 1) : kk / MTX, x = kk - y * (xd ? MTX + 1 : MTX);
      const int sl = slot(y + 1), sb = slot(y);
      const int ps = MRING * (xd ? MXW : MTX);
      const double *pl = xd ? sXp + sl * MXW + x : sYp + sb * MTX + x;
      double *pr = xd ? sXm + sl * MXW + x + 1 : sYm + sl * MTX + x;
      const int on = xd ? 2 * ps : 3 * ps, ot = xd ? 3 * ps : 2 * ps;
      const double ql[4] = {pl[0], pl[ps], pl[on], pl[ot]}, qr[4] = {pr[0], pr[ps], pr[on], pr[ot]};
      double fl[4];
      riemann_sel<RS, FAST>(f, ph, ql, qr, fl);
      if (!FAST) {
        const double dtd = xd ? dtdx : dtdy;
#pragma unroll
        for (int v = 0; v < 4; ++v) fl[v] = f.xmul(fl[v], dtd);
      }
      pr[0] = fl[E2D_ID];
      pr[ps] = fl[E2D_IP];
      pr[on] = fl[E2D_IU];
      pr[ot] = fl[E2D_IV];
    }
    __syncthreads();

    // stage 4: rows 0 .. CHUNK - 1
#pragma unroll
    for (int n = 0; n < N; ++n) {
      if (at[n] < 0) continue;
      const int k = tid + n * MNT, y = k / MTX, x = k - y * MTX;
      const double *fx = sXm + slot(y) * MXW + x + 1;
      const double *fy = sYm + slot(y) * MTX + x, *fz = sYm + slot(y + 1) * MTX + x;
      double un[4];
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        const int ox = v * MRING * MXW, oy = v * MRING * MTX;
        if (FAST)
          un[v] = fma(f.sub(fx[ox], fx[ox + 1]), dtdx, fma(f.sub(fy[oy], fz[oy]), dtdy, u[n][v]));
        else
          un[v] = f.sub(f.add(f.sub(f.add(u[n][v], fx[ox]), fx[ox + 1]), fy[oy]), fz[oy]);
      }
      finish_cell<FAST>(f, kp, at[n], un, u_out, q_out, term, flags);
    }
    // the rows this chunk read are rewritten two barriers from here at the
    // earliest, but for the slots stage 2 of the next chunk writes
    __syncthreads();
  }
  ghost_fill_tile<MTX, MNT>(g, u_in, u_out, i0, jb - 2, je - jb + 1, bx == 0, bx == (int)gridDim.x - 1,
                            blockIdx.y == 0, blockIdx.y == gridDim.y - 1);
  block_fold<MNT>(term, flags, &clk->acc[par ^ 1], &clk->status);
  __syncthreads();
  if (tid == 0) finish_step64(clk, s_dt[0], par, dt_trace);
}

// Up to `steps` steps of the device loop in one cooperative launch, a grid
// barrier between them: each block takes the same tiles in every step.  A
// launch per step costs a small grid about 4 us of it -- the drain, the next
// launch and instructions fetched anew -- and a barrier 1.5.  Tiles are
// gathered with L2 loads (what other blocks wrote in this launch must not
// come from an L1 line or the read-only path); arithmetic and bits are
// k_step_f64's.
template <int RS, int TX, int TYM, int NT, int MINB, bool XMUL, bool FAST>
__global__ void __launch_bounds__(NT, MINB)
    k_loop_f64(const KParams64 kp, double *q0, double *q1, double *u0, double *u1, DevClock *clk, double *dt_trace,
               const int steps) {
  extern __shared__ unsigned char smem_raw[];
  double *smem = reinterpret_cast<double *>(smem_raw);
  __shared__ double s_dt[3];
  const KGeom &g = kp.g;
  const KPhys<double> &ph = kp.ph;
  const int tid = threadIdx.x, ty = kp.ty;
  const int ntx = (g.nx + TX - 1) / TX, nty = (g.ny + ty - 1) / ty;
  const f64x::FpT<XMUL> f;
  LoopClock c = loop_begin(clk);
  int s = 0;
  for (; s < steps && c.t < c.t_end; ++s) {
    if (tid == 0) {
      const double dt = step_dt(ph, loop_cfl(clk, c, s), c.t, c.t_end);
      s_dt[0] = dt;
      s_dt[1] = quot(dt, ph.dx);
      s_dt[2] = quot(dt, ph.dy);
    }
    const bool odd = c.ns & 1;
    double *u_in = odd ? u1 : u0, *u_out = odd ? u0 : u1;
    const double *q_in = odd ? q1 : q0;
    double *q_out = odd ? q0 : q1;
    double term = 0.0;
    unsigned int flags = 0;
    for (int w = blockIdx.x; w < ntx * nty; w += gridDim.x) {
      const int by = w / ntx, bx = w - by * ntx;
      const int i0 = bx * TX, j0 = by * ty;
      gather_qtile<TX, NT>(g, q_in, i0, j0, ty, smem);
      __syncthreads();
      const double dtdx = s_dt[1], dtdy = s_dt[2];
      tile_stage2<TX, TYM, NT, FAST>(f, ph, dtdx, dtdy, ty, smem);
      TileCells<TX, TYM, NT> cells;
      cells.load(g, u_in, i0, j0, ty);
      __syncthreads();
      tile_riemann<RS, TX, TYM, NT, FAST>(f, ph, dtdx, dtdy, ty, smem);
      __syncthreads();
      step_epilogue<TX, TYM, NT, FAST>(f, kp, cells, u_out, q_out, i0, j0, ty, dtdx, dtdy, smem, term, flags);
      ghost_fill_tile<TX, NT>(g, u_in, u_out, i0, j0, ty, bx == 0, bx == ntx - 1, by == 0, by == nty - 1);
      __syncthreads();
    }
    block_fold<NT>(term, flags, &clk->acc3[(s + 1) % 3], &clk->status);
    const double dt = s_dt[0];
    if (blockIdx.x == 0 && tid == 0) loop_record(clk, c, s, dt, dt_trace);
    c.t = c.t + dt;
    c.ns += 1;
    // wait_test: a block more than there are, so the bounded wait runs out
    if (!grid_barrier(&clk->arrived, (unsigned)(s + 1) * gridDim.x + (kp.wait_test ? 1u : 0u))) {
      if (tid == 0) atomicOr(&clk->status, E2D_FLAG_TIMEOUT);
      return;
    }
  }
  if (blockIdx.x == 0 && tid == 0) loop_end(clk, c, s);
}

// ------------------------------------------------------------ batches
// Instance k of a work list with begin[k] <= w < begin[k + 1].
__device__ __forceinline__ int list_entry(const int *__restrict__ begin, int n, int w) {
  int lo = 0, hi = n;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (begin[mid] <= w)
      lo = mid;
    else
      hi = mid;
  }
  return lo;
}

// An admitted FP64 instance's first primitives and CFL maximum (the device
// loop's prologue): q[0] from u[0], the maximum into acc[0].
__global__ void __launch_bounds__(FILL_BX *FILL_BY) k_batch_prime_f64(BatchInst64 *__restrict__ I) {
  const int by = blockIdx.x / I->nbx, bx = blockIdx.x - by * I->nbx;
  double term = 0.0;
  unsigned int flags = 0;
  fill_cell(I->kp, I->u[0], nullptr, I->q[0], FILL_WRITE_Q | FILL_DT, bx * FILL_BX + threadIdx.x,
            by * FILL_BY + threadIdx.y, term, flags);
  fill_reduce(term, flags, &I->acc[0], &I->status);
}

// `iterations` steps of every listed FP64 instance in one cooperative launch,
// a grid barrier between them: each block takes the same TX x ty tiles of the
// work list (instance k's tiles are tile_begin[k] .. tile_begin[k+1]-1) in
// every iteration and runs the fused step on each with its instance's dt,
// primitives and ghost cells (tiles gathered); the instance's last tile of an
// iteration advances its loop state.  The tile is chosen for the whole list
// (choose_f64_tile), so the last few solves of a batch still use every SM:
// 32 x 32 tiles left a lone 256^2 solve on 64 of 152.
// A block whose barrier wait runs out stops its instances by a bit of their
// status and leaves; one that arrives after that may go on for a while, so
// one thread reads what steers a block (another block may be setting the bit
// meanwhile, and threads that disagree would part at the block's barriers),
// and nothing but the last tile writes `active`.
// late: blocks more than there are that the barriers wait for (tests).
// A launch of one iteration has no barrier and need not be cooperative.
template <int RS, int TX, int TYM, int NT, int MINB, bool XMUL>
__global__ void __launch_bounds__(NT, MINB)
    k_batch_loop_f64(BatchInst64 *insts, const int *__restrict__ list_slots, const int *__restrict__ tile_begin,
                     const int n_inst, const int total_tiles, const int ty, const int iterations,
                     unsigned int *arrived, const unsigned int late) {
  extern __shared__ unsigned char smem_raw[];
  double *smem = reinterpret_cast<double *>(smem_raw);
  __shared__ double s_dt[3];
  __shared__ int s_par;       // of the instance at hand, -1 if it is not to be stepped
  __shared__ KParams64 s_kp;  // of the instance at hand
  const int tid = threadIdx.x;
  const f64x::FpT<XMUL> f;
  const KParams64 &kp = s_kp;
  int held = -1;  // list entry whose parameters are in s_kp
  for (int it = 0; it < iterations; ++it) {
    for (int w = blockIdx.x; w < total_tiles; w += gridDim.x) {
      const int k = list_entry(tile_begin, n_inst, w);
      BatchInst64 &I = insts[list_slots[k]];
      int steer = -1;
      if (tid == 0) {
        const int active = __ldcg(&I.active), p = __ldcg(&I.par);
        if (active && !(__ldcg(&I.status) & E2D_FLAG_TIMEOUT)) steer = p;
      }
      __syncthreads();  // the previous tile is done with s_par, s_dt, s_kp and the shared tile
      if (tid == 0) s_par = steer;
      if (k != held) {
        static_assert(sizeof(KParams64) % 4 == 0, "copied by words");
        for (int j = tid; j < (int)(sizeof(KParams64) / 4); j += NT)
          reinterpret_cast<int *>(&s_kp)[j] = reinterpret_cast<const int *>(&I.kp)[j];
        held = k;
      }
      __syncthreads();
      const int par = s_par;
      if (par < 0) continue;
      if (tid == 0) {
        const double dt = step_dt(kp.ph, __ldcg(&I.acc[par]), __ldcg(&I.t), __ldcg(&I.t_end));
        s_dt[0] = dt;
        s_dt[1] = quot(dt, kp.ph.dx);
        s_dt[2] = quot(dt, kp.ph.dy);
      }
      const int ntx = (kp.g.nx + TX - 1) / TX, nty = (kp.g.ny + ty - 1) / ty;
      const int b = w - tile_begin[k];
      const int by = b / ntx, bx = b - by * ntx;
      const int i0 = bx * TX, j0 = by * ty;
      gather_qtile<TX, NT>(kp.g, I.q[par], i0, j0, ty, smem);
      __syncthreads();
      double term = 0.0;
      unsigned int flags = 0;
      const double dtdx = s_dt[1], dtdy = s_dt[2];
      tile_stage2<TX, TYM, NT, false>(f, kp.ph, dtdx, dtdy, ty, smem);
      TileCells<TX, TYM, NT> cells;
      cells.load(kp.g, I.u[par], i0, j0, ty);
      __syncthreads();
      tile_riemann<RS, TX, TYM, NT, false>(f, kp.ph, dtdx, dtdy, ty, smem);
      __syncthreads();
      step_epilogue<TX, TYM, NT, false>(f, kp, cells, I.u[par ^ 1], I.q[par ^ 1], i0, j0, ty, dtdx, dtdy, smem, term,
                                        flags);
      ghost_fill_tile<TX, NT>(kp.g, I.u[par], I.u[par ^ 1], i0, j0, ty, bx == 0, bx == ntx - 1, by == 0,
                              by == nty - 1);
      block_fold<NT>(term, flags, &I.acc[par ^ 1], &I.status);
      __syncthreads();
      if (tid == 0) {
        __threadfence();
        const unsigned int ticket = atomicAdd(&I.done, 1u);
        if (ticket == (unsigned)(ntx * nty) - 1u) {
          __threadfence();
          const double dt = s_dt[0];
          if (!(dt > 0.0) || nonfinite(dt)) atomicOr(&I.status, (unsigned)E2D_FLAG_BAD_DT);
          const double t = __ldcg(&I.t) + dt;
          I.dt = dt;
          I.t = t;
          I.nstep = __ldcg(&I.nstep) + 1;
          I.par = par ^ 1;
          I.acc[par] = 0ull;  // read by this step; folded into by the next
          I.done = 0u;
          I.active = (t < __ldcg(&I.t_end)) && !(__ldcg(&I.status) & (E2D_FLAG_NONFINITE | E2D_FLAG_BAD_DT));
          __threadfence();
        }
      }
    }
    if (it + 1 == iterations) return;
    if (!grid_barrier(arrived, (unsigned)(it + 1) * gridDim.x + late)) {
      // the states of this block's tiles are incomplete: their instances stop
      for (int w = blockIdx.x; tid == 0 && w < total_tiles; w += gridDim.x)
        atomicOr(&insts[list_slots[list_entry(tile_begin, n_inst, w)]].status, (unsigned)E2D_FLAG_TIMEOUT);
      return;
    }
  }
}

// ------------------------------------------------------------ building blocks
// One building block of the step per thread, with the exact device code the
// step kernels use (see e2d_eval_device in include/e2d.h for the layouts).
__global__ void k_eval_f64(const KParams64 kp, const int what, const int n,
                           const double *__restrict__ in, double *__restrict__ out, const double dtdx,
                           const double dtdy) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const KPhys<double> &ph = kp.ph;
  const Fp f;
  const int st_kind = (ph.slope_type == 2.0) ? 2 : (ph.slope_type == 1.0) ? 1 : 0;
  if (what == E2D_EVAL_PRIMITIVES) {
    const double *u = in + 4 * k;
    double d, p, ux, uy;
    Divisor dv;
    primitives(f, ph, u[E2D_ID], u[E2D_IP], u[E2D_IU], u[E2D_IV], d, p, ux, uy, dv);
    double *o = out + 5 * k;
    o[E2D_ID] = d;
    o[E2D_IP] = p;
    o[E2D_IU] = ux;
    o[E2D_IV] = uy;
    o[4] = root(quot(f.mul(ph.gamma0, p), dv));
  } else if (what == E2D_EVAL_SLOPES) {
    const double *s = in + 20 * k;  // q, q(+x), q(-x), q(+y), q(-y)
    double *o = out + 8 * k;
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      o[v] = slope(f, st_kind, s[v], s[4 + v], s[8 + v]);
      o[4 + v] = slope(f, st_kind, s[v], s[12 + v], s[16 + v]);
    }
  } else if (what >= E2D_EVAL_TRACE_XMIN && what <= E2D_EVAL_TRACE_YMAX) {
    const double *s = in + 12 * k;  // q, dqx, dqy
    double s0[4];
    trace_sources(f, ph, s, s + 4, s + 8, s0);
    const int face = what - E2D_EVAL_TRACE_XMIN;
    const bool xdir = face < 2;
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      double fm, fp;
      const double dtd = xdir ? dtdx : dtdy;
      face_pair(f, ph, v, s[v], half(xdir ? s[4 + v] : s[8 + v]), s0[v], dtd, half(dtd), fm, fp);
      out[4 * k + v] = (face == 0 || face == 2) ? fm : fp;
    }
  } else {
    const double *s = in + 8 * k;  // qleft, qright
    double *o = out + 4 * k;
    if (what == E2D_EVAL_RIEMANN_HLLC)
      riemann_hllc(f, ph, s, s + 4, o);
    else if (what == E2D_EVAL_RIEMANN_HLL)
      riemann_hll(f, ph, s, s + 4, o);
    else
      riemann_approx(f, ph, s, s + 4, o);
  }
}

// ------------------------------------------------------------ initial conditions
// src/HydroRunFunctors.h:1347-1827: cell centres x = xmin + dx/2 + (i-g)*dx.
__global__ void k_init_f64(const KParams64 kp, const e2d_params p, double *__restrict__ u,
                           const double blast_e_inside) {
  const KGeom &g = kp.g;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= g.isize || j >= g.jsize) return;
  const double gamma0 = p.gamma0;
  const double x = p.xmin + p.dx / 2 + (i - 2) * p.dx;
  const double y = p.ymin + p.dy / 2 + (j - 2) * p.dy;
  double d = 0, e = 0, mx = 0, my = 0;
  switch (p.problemType) {
    case E2D_PROBLEM_IMPLODE: {  // :1375-1401
      bool in;
      if (p.implode_shape == 0) {
        const double tmp = x + y * y;
        in = tmp > 0.5 && tmp < 1.5;
      } else {
        in = x + y > 0.5;
      }
      d = in ? 1.0 : 0.125;
      e = in ? 1.0 / (gamma0 - 1.0) : 0.14 / (gamma0 - 1.0);
      break;
    }
    case E2D_PROBLEM_BLAST: {  // :1451-1520
      const double r2 = p.blast_radius * p.blast_radius;
      const double d2 = (x - p.blast_center_x) * (x - p.blast_center_x) +
                        (y - p.blast_center_y) * (y - p.blast_center_y);
      const bool in = d2 < r2;
      d = in ? p.blast_density_in : p.blast_density_out;
      e = (in ? p.blast_pressure_in : p.blast_pressure_out) / (gamma0 - 1.0);
      if (in && blast_e_inside > 0.0) e = blast_e_inside;
      break;
    }
    case E2D_PROBLEM_FOUR_QUADRANT: {  // :1578-1665 (default states: Lax-Liu case 3)
      const int r = (x < p.fq_split_x) ? ((y < p.fq_split_y) ? 2 : 1) : ((y < p.fq_split_y) ? 3 : 0);
      const double rho = p.fq_state[r][0], pr = p.fq_state[r][1], uu = p.fq_state[r][2], vv = p.fq_state[r][3];
      d = rho;
      mx = uu * rho;
      my = vv * rho;
      e = pr / (gamma0 - 1.0) + rho * (uu * uu + vv * vv) * 0.5;
      break;
    }
    case E2D_PROBLEM_DISCONTINUITY: {  // :1697-1731
      if (x + y < 1) {
        d = 1.0 + x * x;
      } else {
        d = 0.25;
      }
      e = 1.0 / (gamma0 - 1.0);
      break;
    }
    default: {  // E2D_PROBLEM_SHOCKED_BUBBLE, :1761-1822
      if (x < p.shock_loc) {
        d = p.postshock_density;
        mx = p.postshock_density * p.postshock_velocity;
        my = 0.0;
        const double rho_eint = p.postshock_pressure / (gamma0 - 1);
        e = rho_eint + 0.5 * (mx * mx + my * my) / d;
      } else {
        const double rad = sqrt((x - p.bubble_center_x) * (x - p.bubble_center_x) +
                                (y - p.bubble_center_y) * (y - p.bubble_center_y));
        const bool in = rad < p.bubble_radius;
        d = in ? p.bubble_density : p.preshock_density;
        const double rho_eint = (in ? p.bubble_pressure : p.preshock_pressure) / (gamma0 - 1);
        e = rho_eint + 0.5 * (mx * mx + my * my) / d;
      }
      break;
    }
  }
  const size_t o = (size_t)i + (size_t)g.isize * j;
  u[o] = d;
  u[o + g.plane] = e;
  u[o + 2 * g.plane] = mx;
  u[o + 3 * g.plane] = my;
}

}  // namespace


cudaError_t launch_fill_f64(const KParams64 &kp, double *u_in, double *u_out, double *q,
                            DevClock *clk, int mode, cudaStream_t s, int acc_slot) {
  dim3 block(FILL_BX, FILL_BY);
  dim3 grid((kp.g.isize + FILL_BX - 1) / FILL_BX, (kp.g.jsize + FILL_BY - 1) / FILL_BY);
  k_fill_f64<<<grid, block, 0, s>>>(kp, u_in, u_out, q, clk, mode, acc_slot);
  return cudaGetLastError();
}

// Tile shapes of the fused step and of the two-launch step's flux kernel: TX
// columns, up to TYM rows, NT threads, MINB blocks on an SM; XMUL: see FpT.
template <int SHAPE>
struct Shape;
template <>
struct Shape<0> {
  static constexpr int TX = 32, TYM = 16, NT = 256, MINB = 2;
  static constexpr bool XMUL = true;
};
template <>
struct Shape<1> {
  static constexpr int TX = 16, TYM = 16, NT = 128, MINB = 4;
  static constexpr bool XMUL = true;
};
template <>
struct Shape<2> {
  static constexpr int TX = 8, TYM = 8, NT = 256, MINB = 2;
  static constexpr bool XMUL = false;
};
constexpr int kShapes = 3;
// Waves of tiles up to which a grid's steps run in one launch.
constexpr int LOOP_WAVES = 4;
// Waves of tiles up to which a batch's iterations run in one launch.  A
// barrier gives up after a second, so what a block does between two has to be
// bounded: a wave takes 0.25 ms with the slowest solver (the iterative one, a
// 600x401 grid), this many a quarter of a second, of which a block waits for
// the part by which others are slower.  A launch for each such iteration
// costs nothing beside it.
constexpr int BATCH_WAVES = 1024;
template <class F>
static void with_shape(int shape, F &&f) {
  switch (shape) {
    case 1: f(Shape<1>{}); break;
    case 2: f(Shape<2>{}); break;
    default: f(Shape<0>{}); break;
  }
}

// The tile of a grid, or of a batch's grids together: the shape and rows
// whose step a simple model of the launch puts lowest.  A tile's stages take
// whole warps of face-state cells (lanes of cell and variable for the 8-column
// shape), Riemann solves and updates (W2, W3, W4); one tile alone takes L, a
// latency per round of its block's warps; k tiles on an SM share the FP64
// pipe, k (80 W2 + 50 W3 + 34 W4) instructions (23 W2 by variable) at 5.07 ns;
// the two add with exponent 1.3; tiles beyond what is resident make further
// waves, which average out once there are four.  The constants are fitted to
// 300 timings (16 grids from 32x20 to 2048^2, every shape, 3 to 16 rows; 4 %
// rms), on which the model's choice is within a few percent of the fastest.
// What it buys (us a step, HLLC; before: 32 x 32 tiles for every grid):
// 64x48 71 -> 10.9 (8 x 3), 128^2 71 -> 15.1 (8 x 7), 256^2 72 -> 33.4
// (32 x 7), 500x300 128 -> 61 (32 x 16), 2048^2 1832 -> 1553 (32 x 13: the
// Riemann solves of 13 rows fill their last round of warps, those of 16 do
// not: 1580).  The fast forms' rounds are shorter and a tile's fixed part
// weighs more: with many waves they take the most rows (2048^2: 1236 us with
// 16, 1260 with 13).
void choose_f64_tile(const int (*dims)[2], int n, bool fast, int tile, int *shape, int *ty) {
  struct Info {
    int tx, most, warps, resident;
  };
  auto info = [](int sh) {
    Info i{};
    with_shape(sh, [&](auto s) {
      using S = decltype(s);
      i = Info{S::TX, S::TYM, S::NT / 32, S::MINB};
    });
    return i;
  };
  if (tile >= 0) {
    *shape = tile % 100 < kShapes ? tile % 100 : 0;
    const int m = info(*shape).most;
    *ty = tile >= 100 && tile / 100 < m ? tile / 100 : m;
    return;
  }
  static const double lat[kShapes][3] = {{4.77, 2.49, 1.83}, {3.93, 2.24, 3.95}, {1.62, 0.42, 5.36}};  // us
  constexpr double kSms = 152.0, kFixed = 2.7, kInst = 0.00507, kExp = 1.3;
  auto up = [](int a, int b) { return (a + b - 1) / b; };
  double best = 0.0;
  for (int sh = 0; sh < kShapes; ++sh) {
    const Info i = info(sh);
    for (int y = 3; y <= i.most; ++y) {
      const bool split = i.tx <= 8;  // tile_stage2
      const int w[3] = {up(((i.tx + 2) * (y + 2) - 4) * (split ? 4 : 1), 32),
                        up((i.tx + 1) * y + i.tx * (y + 1), 32), up(i.tx * y, 32)};
      const double inst = kInst * ((split ? 23 : 80) * w[0] + 50 * w[1] + 34 * w[2]);
      double alone = 0.0;
      for (int k = 0; k < 3; ++k) alone += up(w[k], i.warps) * lat[sh][k];
      auto wave = [&](double k) { return std::pow(std::pow(alone, kExp) + std::pow(k * inst, kExp), 1.0 / kExp); };
      double tiles = 0.0;
      for (int k = 0; k < n; ++k) tiles += (double)up(dims[k][0], i.tx) * up(dims[k][1], y);
      const double per_wave = kSms * i.resident;
      const double full = std::floor(tiles / per_wave), rest = tiles - full * per_wave;
      if (fast && full >= 4 && y < i.most) continue;
      const double t = full >= 4 ? wave(i.resident) * tiles / per_wave + 0.5 * wave(1)
                                 : full * wave(i.resident) + (rest > 0 ? wave(std::ceil(rest / kSms)) : 0.0);
      if (best == 0.0 || kFixed + t < best) {
        best = kFixed + t;
        *shape = sh;
        *ty = y;
      }
    }
  }
}

// Blocks of a kernel that are resident on the current device at once, 0 if
// it cannot launch cooperatively (kept per kernel and device: the occupancy
// query costs more than a launch).
int resident_blocks(const void *kernel, int threads, size_t smem) {
  static std::mutex mutex;
  static std::map<std::pair<const void *, int>, int> known;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  std::lock_guard<std::mutex> lock(mutex);
  auto it = known.find({kernel, dev});
  if (it != known.end()) return it->second;
  int sms = 0, per_sm = 0, coop = 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem) != cudaSuccess)
    return 0;
  return known[{kernel, dev}] = sms * per_sm;
}

template <int RS>
static cudaError_t launch_flux_t(const KParams64 &kp, const double *q, double *u_in,
                                 double *u_out, DevClock *clk, int use_clock, double host_dt,
                                 double *dt_trace, cudaStream_t s) {
  with_shape(kp.shape, [&](auto sh) {
    using S = decltype(sh);
    dim3 grid((kp.g.nx + S::TX - 1) / S::TX, (kp.g.ny + kp.ty - 1) / kp.ty);
    k_flux_update_f64<RS, S::TX, S::TYM, S::NT, S::MINB, S::XMUL><<<grid, S::NT, flux_smem_bytes<S::TX, S::TYM>(), s>>>(
        kp, q, u_in, u_out, clk, use_clock, host_dt, dt_trace);
  });
  return cudaGetLastError();
}

template <int RS>
static cudaError_t configure_rs() {
  constexpr auto kDyn = cudaFuncAttributeMaxDynamicSharedMemorySize;
  cudaError_t e = cudaFuncSetAttribute(k_march_f64<RS, false>, kDyn, (int)march_smem_bytes());
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_march_f64<RS, true>, kDyn, (int)march_smem_bytes());
  for (int k = 0; k < kShapes; ++k)
    with_shape(k, [&](auto sh) {
      using S = decltype(sh);
      constexpr int step = (int)step_smem_bytes<S::TX, S::TYM>(), flux = (int)flux_smem_bytes<S::TX, S::TYM>();
      constexpr auto attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
      if (e == cudaSuccess) e = cudaFuncSetAttribute(k_flux_update_f64<RS, S::TX, S::TYM, S::NT, S::MINB, S::XMUL>, attr, flux);
      if (e == cudaSuccess) e = cudaFuncSetAttribute(k_step_f64<RS, S::TX, S::TYM, S::NT, S::MINB, S::XMUL, false>, attr, step);
      if (e == cudaSuccess) e = cudaFuncSetAttribute(k_step_f64<RS, S::TX, S::TYM, S::NT, S::MINB, S::XMUL, true>, attr, step);
      if (e == cudaSuccess) e = cudaFuncSetAttribute(k_loop_f64<RS, S::TX, S::TYM, S::NT, S::MINB, S::XMUL, false>, attr, flux);
      if (e == cudaSuccess) e = cudaFuncSetAttribute(k_loop_f64<RS, S::TX, S::TYM, S::NT, S::MINB, S::XMUL, true>, attr, flux);
      if (e == cudaSuccess) e = cudaFuncSetAttribute(k_batch_loop_f64<RS, S::TX, S::TYM, S::NT, S::MINB, S::XMUL>, attr, flux);
    });
  return e;
}

cudaError_t configure_f64_kernels(int riemann) {
  static std::mutex mutex;
  static std::map<std::pair<int, int>, bool> done;  // per device and solver, for the life of the process
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> lock(mutex);
  bool &ready = done[{dev, riemann}];
  if (ready) return cudaSuccess;
  e = riemann == E2D_RIEMANN_HLLC  ? configure_rs<E2D_RIEMANN_HLLC>()
      : riemann == E2D_RIEMANN_HLL ? configure_rs<E2D_RIEMANN_HLL>()
                                   : configure_rs<E2D_RIEMANN_APPROX>();
  ready = e == cudaSuccess;
  return e;
}

void batch_f64_shape(const KParams64 &kp, int *nbx, int *nfill) {
  *nbx = (kp.g.isize + FILL_BX - 1) / FILL_BX;
  *nfill = *nbx * ((kp.g.jsize + FILL_BY - 1) / FILL_BY);
}

int f64_tiles(int nx, int ny, int shape, int ty) {
  int tx = 0;
  with_shape(shape, [&](auto sh) { tx = decltype(sh)::TX; });
  return ((nx + tx - 1) / tx) * ((ny + ty - 1) / ty);
}

cudaError_t launch_batch_prime_f64(BatchInst64 *inst, int nfill, cudaStream_t s) {
  k_batch_prime_f64<<<nfill, dim3(FILL_BX, FILL_BY), 0, s>>>(inst);
  return cudaGetLastError();
}

template <int RS>
static cudaError_t launch_batch_t(BatchInst64 *insts, const int *list_slots, const int *tile_begin, int n_inst,
                                  int total_tiles, int shape, int ty, int iterations, unsigned int *arrived,
                                  unsigned int late, bool loop, cudaStream_t s) {
  cudaError_t e = cudaMemsetAsync(arrived, 0, sizeof(unsigned int), s);
  with_shape(shape, [&](auto sh) {
    using S = decltype(sh);
    auto kernel = k_batch_loop_f64<RS, S::TX, S::TYM, S::NT, S::MINB, S::XMUL>;
    constexpr size_t sm = flux_smem_bytes<S::TX, S::TYM>();
    const int resident = resident_blocks(reinterpret_cast<const void *>(kernel), S::NT, sm);
    if (loop && resident > 0 && total_tiles <= (long long)resident * BATCH_WAVES) {
      const int grid = total_tiles < resident ? total_tiles : resident;
      void *args[] = {&insts, &list_slots, &tile_begin, &n_inst, &total_tiles, &ty, &iterations, &arrived, &late};
      if (e == cudaSuccess)
        e = cudaLaunchCooperativeKernel(reinterpret_cast<const void *>(kernel), dim3(grid), dim3(S::NT), args, sm, s);
      return;
    }
    // as many blocks as are resident take the tiles, where that is known
    const int grid = resident > 0 && resident < total_tiles ? resident : total_tiles;
    for (int it = 0; it < iterations && e == cudaSuccess; ++it) {
      kernel<<<grid, S::NT, sm, s>>>(insts, list_slots, tile_begin, n_inst, total_tiles, ty, 1, arrived, 0u);
      e = cudaGetLastError();
    }
  });
  return e;
}

cudaError_t launch_batch_f64(int riemann, BatchInst64 *insts, const int *list_slots, const int *tile_begin,
                             int n_inst, int total_tiles, int shape, int ty, int iterations, unsigned int *arrived,
                             unsigned int late, bool loop, cudaStream_t s) {
  if (n_inst <= 0 || total_tiles <= 0 || iterations <= 0) return cudaSuccess;
  switch (riemann) {
    case E2D_RIEMANN_HLLC:
      return launch_batch_t<E2D_RIEMANN_HLLC>(insts, list_slots, tile_begin, n_inst, total_tiles, shape, ty, iterations,
                                              arrived, late, loop, s);
    case E2D_RIEMANN_HLL:
      return launch_batch_t<E2D_RIEMANN_HLL>(insts, list_slots, tile_begin, n_inst, total_tiles, shape, ty, iterations,
                                             arrived, late, loop, s);
    default:
      return launch_batch_t<E2D_RIEMANN_APPROX>(insts, list_slots, tile_begin, n_inst, total_tiles, shape, ty,
                                                iterations, arrived, late, loop, s);
  }
}

cudaError_t launch_flux_update_f64(const KParams64 &kp, int riemann, const double *q,
                                   double *u_in, double *u_out, DevClock *clk,
                                   int use_clock, double host_dt, double *dt_trace,
                                   cudaStream_t s) {
  switch (riemann) {
    case E2D_RIEMANN_HLLC:
      return launch_flux_t<E2D_RIEMANN_HLLC>(kp, q, u_in, u_out, clk, use_clock, host_dt, dt_trace, s);
    case E2D_RIEMANN_HLL:
      return launch_flux_t<E2D_RIEMANN_HLL>(kp, q, u_in, u_out, clk, use_clock, host_dt, dt_trace, s);
    default:
      return launch_flux_t<E2D_RIEMANN_APPROX>(kp, q, u_in, u_out, clk, use_clock, host_dt, dt_trace, s);
  }
}

// Rows of a march's segments (0: tiles).  Grids march from 100 rows a
// resident block on (two blocks an SM): 1024^2, 108 rows, takes 399 us a step
// against 408 with tiles, 1531x797 HLL 526 against 547 (both before HLL shared its products; now 488), 2048^2 1445 against
// 1561, 4096^2 5535 against 6143 -- but 700^2, 51 rows, 205 against 197.  The
// segment is the number of chunks whose waves of blocks take the fewest
// chunks, a last wave with at most one block an SM counting 0.62 of a full
// one (measured within 4 % over 10 segment lengths on 3000x1700; at 2048^2 and
// 4096^2 the choice is within 2 % of the best of 13).
int choose_f64_march(int nx, int ny, int rows) {
  if (rows > 0) return rows;
  constexpr double kSlots = 152.0 * 2, kMinRows = 100.0;
  const double cols = (nx + MTX - 1) / MTX;
  if (cols * ny < kMinRows * kSlots) return 0;
  int best = 0;
  double cost = 0.0;
  for (int n = 4; n <= 20; ++n) {
    const int h = CHUNK * n - 2;
    const double waves = cols * std::ceil((double)ny / h) / kSlots, full = std::floor(waves), rest = waves - full;
    // 0.3: a segment's start (dt, the first copy) and end (the fold)
    const double c = (n + 0.3) * (full + (rest == 0.0 ? 0.0 : rest <= 0.5 ? 0.62 : 1.0));
    if (best == 0 || c < cost) best = h, cost = c;
  }
  return best;
}

template <int RS>
static cudaError_t launch_step_t(const KParams64 &kp, const CUtensorMap &tm_q, int use_tma, const double *q_in,
                                 double *q_out, double *u_in, double *u_out, DevClock *clk, double *dt_trace,
                                 cudaStream_t s) {
  if (kp.march_rows > 0) {
    dim3 grid((kp.g.nx + MTX - 1) / MTX, (kp.g.ny + kp.march_rows - 1) / kp.march_rows);
    if (kp.fast)
      k_march_f64<RS, true><<<grid, MNT, march_smem_bytes(), s>>>(kp, tm_q, use_tma, q_in, q_out, u_in, u_out, clk,
                                                                  dt_trace);
    else
      k_march_f64<RS, false><<<grid, MNT, march_smem_bytes(), s>>>(kp, tm_q, use_tma, q_in, q_out, u_in, u_out, clk,
                                                                   dt_trace);
    return cudaGetLastError();
  }
  with_shape(kp.shape, [&](auto sh) {
    using S = decltype(sh);
    dim3 grid((kp.g.nx + S::TX - 1) / S::TX, (kp.g.ny + kp.ty - 1) / kp.ty);
    constexpr size_t sm = step_smem_bytes<S::TX, S::TYM>();
    if (kp.fast)
      k_step_f64<RS, S::TX, S::TYM, S::NT, S::MINB, S::XMUL, true>
          <<<grid, S::NT, sm, s>>>(kp, tm_q, use_tma, q_in, q_out, u_in, u_out, clk, dt_trace);
    else
      k_step_f64<RS, S::TX, S::TYM, S::NT, S::MINB, S::XMUL, false>
          <<<grid, S::NT, sm, s>>>(kp, tm_q, use_tma, q_in, q_out, u_in, u_out, clk, dt_trace);
  });
  return cudaGetLastError();
}

cudaError_t launch_dt_f64(const KParams64 &kp, double *u, double *q, DtAcc *acc, DtResult *result, cudaStream_t s) {
  dim3 block(FILL_BX, FILL_BY);
  dim3 grid((kp.g.isize + FILL_BX - 1) / FILL_BX, (kp.g.jsize + FILL_BY - 1) / FILL_BY);
  k_dt_f64<<<grid, block, 0, s>>>(kp, u, q, acc, result);
  return cudaGetLastError();
}

template <int RS, class F>
static void with_loop(const KParams64 &kp, F &&f) {
  with_shape(kp.shape, [&](auto sh) {
    using S = decltype(sh);
    constexpr size_t sm = flux_smem_bytes<S::TX, S::TYM>();
    const int tiles = ((kp.g.nx + S::TX - 1) / S::TX) * ((kp.g.ny + kp.ty - 1) / kp.ty);
    if (kp.fast)
      f(k_loop_f64<RS, S::TX, S::TYM, S::NT, S::MINB, S::XMUL, true>, S::NT, sm, tiles);
    else
      f(k_loop_f64<RS, S::TX, S::TYM, S::NT, S::MINB, S::XMUL, false>, S::NT, sm, tiles);
  });
}
template <class F>
static void with_loop(int riemann, const KParams64 &kp, F &&f) {
  switch (riemann) {
    case E2D_RIEMANN_HLLC: with_loop<E2D_RIEMANN_HLLC>(kp, f); break;
    case E2D_RIEMANN_HLL: with_loop<E2D_RIEMANN_HLL>(kp, f); break;
    default: with_loop<E2D_RIEMANN_APPROX>(kp, f); break;
  }
}

int f64_loop_blocks(const KParams64 &kp, int riemann) {
  if (kp.march_rows > 0) return 0;
  int blocks = 0;
  with_loop(riemann, kp, [&](auto kernel, int threads, size_t sm, int tiles) {
    const int resident = resident_blocks(reinterpret_cast<const void *>(kernel), threads, sm);
    if (tiles <= resident * LOOP_WAVES) blocks = tiles < resident ? tiles : resident;
  });
  return blocks;
}

cudaError_t launch_loop_f64(const KParams64 &kp, int riemann, int blocks, double *const u[2], double *const q[2],
                            DevClock *clk, double *dt_trace, int steps, cudaStream_t s) {
  cudaError_t e = cudaSuccess;
  with_loop(riemann, kp, [&](auto kernel, int threads, size_t sm, int) {
    KParams64 p = kp;
    double *q0 = q[0], *q1 = q[1], *u0 = u[0], *u1 = u[1];
    void *args[] = {&p, &q0, &q1, &u0, &u1, &clk, &dt_trace, &steps};
    e = cudaLaunchCooperativeKernel(reinterpret_cast<const void *>(kernel), dim3(blocks), dim3(threads), args, sm, s);
  });
  return e;
}

cudaError_t launch_step_f64(const KParams64 &kp, int riemann, const CUtensorMap &tm_q, int use_tma,
                            const double *q_in, double *q_out, double *u_in, double *u_out, DevClock *clk,
                            double *dt_trace, cudaStream_t s) {
  switch (riemann) {
    case E2D_RIEMANN_HLLC:
      return launch_step_t<E2D_RIEMANN_HLLC>(kp, tm_q, use_tma, q_in, q_out, u_in, u_out, clk, dt_trace, s);
    case E2D_RIEMANN_HLL:
      return launch_step_t<E2D_RIEMANN_HLL>(kp, tm_q, use_tma, q_in, q_out, u_in, u_out, clk, dt_trace, s);
    default:
      return launch_step_t<E2D_RIEMANN_APPROX>(kp, tm_q, use_tma, q_in, q_out, u_in, u_out, clk, dt_trace, s);
  }
}

// The box of the fused step's primitives tile for the tile shape of kp:
// dimensions (isize, jsize, 4 planes), box (TX + 4) x (ty + 4) x 4.  Row and
// plane strides must be multiples of 16 bytes, so isize must be even; false
// (tiles are then gathered) otherwise or if the driver cannot encode it.
bool encode_q_map(CUtensorMap *map, const double *q, const KParams64 &kp) {
  static const PFN_cuTensorMapEncodeTiled_v12000 encode = []() -> PFN_cuTensorMapEncodeTiled_v12000 {
    void *fn = nullptr;
    cudaDriverEntryPointQueryResult qr;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &qr) != cudaSuccess ||
        qr != cudaDriverEntryPointSuccess)
      return nullptr;
    return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
  }();
  if (!encode || (kp.g.isize & 1) || (reinterpret_cast<uintptr_t>(q) & 15u)) return false;
  const cuuint64_t dims[3] = {(cuuint64_t)kp.g.isize, (cuuint64_t)kp.g.jsize, 4};
  const cuuint64_t strides[2] = {(cuuint64_t)kp.g.isize * sizeof(double), (cuuint64_t)kp.g.plane * sizeof(double)};
  int tx = 0;
  with_shape(kp.shape, [&](auto sh) { tx = decltype(sh)::TX; });
  const cuuint32_t box[3] = {(cuuint32_t)(kp.march_rows > 0 ? MQW : tx + 4),
                             (cuuint32_t)(kp.march_rows > 0 ? MQH : kp.ty + 4), 4};
  const cuuint32_t estr[3] = {1, 1, 1};
  return encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 3, const_cast<double *>(q), dims, strides, box, estr,
                CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

cudaError_t launch_eval_f64(const KParams64 &kp, int what, int n, const double *in, double *out,
                            double dtdx, double dtdy, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  k_eval_f64<<<(n + 127) / 128, 128, 0, s>>>(kp, what, n, in, out, dtdx, dtdy);
  return cudaGetLastError();
}

cudaError_t launch_init_f64(const KParams64 &kp, const e2d_params &p, double *u, cudaStream_t s) {
  // Sedov variant (src/HydroRunFunctors.h:1425-1447, :1496-1547): the
  // inside energy is total_energy_inside / (inside cell count * dx * dy).
  double e_inside = 0.0;
  if (p.problemType == E2D_PROBLEM_BLAST && p.blast_total_energy_inside > 0) {
    long long count = 0;
    const double r2 = p.blast_radius * p.blast_radius;
    for (int j = 0; j < kp.g.jsize; ++j)
      for (int i = 0; i < kp.g.isize; ++i) {
        const double x = p.xmin + p.dx / 2 + (i - 2) * p.dx;
        const double y = p.ymin + p.dy / 2 + (j - 2) * p.dy;
        const double d2 = (x - p.blast_center_x) * (x - p.blast_center_x) +
                          (y - p.blast_center_y) * (y - p.blast_center_y);
        if (d2 < r2) count++;
      }
    if (count > 0) e_inside = p.blast_total_energy_inside / ((double)count * (p.dx * p.dy));
  }
  dim3 block(64, 4);
  dim3 grid((kp.g.isize + 63) / 64, (kp.g.jsize + 3) / 4);
  k_init_f64<<<grid, block, 0, s>>>(kp, p, u, e_inside);
  return cudaGetLastError();
}

}  // namespace e2d
