// grhd_evolve.cu -- GRHD evolution in the Cowling approximation on a cubed
// shell: DG elements (LGL points) with LLF faces, finite-volume elements on
// nf equally spaced points (WENO-reconstructed primitives, LLF midpoint
// fluxes), con2prim with atmosphere every stage, the DG <-> finite-volume
// switch with the reference's data transfer (PARENT_2n_P_UNIFORM,
// src/main/evolve/trouble.c:162-183, src/main/basis/gridpoints.c:158-200),
// RK4 stages with the update fused into each kernel, graph-captured steps.
//
// The reference has no GRHD (its physics lives in external repositories),
// so the physics and the finite-volume form are parity unpinned; they are
// restated step by step in the oracle (oracle/nmo_grhd.c), which the tests
// hold this file to.  From the reference come the DG strong form with the
// chain rule (src/main/coordinates/derivs.c:102-181,756-815), the LLF flux
// (src/main/dg/numflux1d.c:85-112), the lift (src/main/dg/dg.c:30-151), the
// WENO reconstructions (src/main/dg/rec1d.c, weno.cuh), the root finder
// newton1d_brak (grhd.cuh) and RK4 (src/main/evolve/RungeKutta.c:19-82).
//
// Device layout: DG states [E][5][n^3] for every element (rows of
// finite-volume elements unused), finite-volume states [slot][5][nf^3] for
// the elements in finite-volume mode (slots in ascending element order),
// per DG node the background (alpha, psi, d alpha, d psi) [E][8][n^3], per
// finite-volume slot the geometry of its points and midpoints
// [slot][kGeo][nf^3] computed on the device from the shell map, and per
// DG / finite-volume face a trace slot of primitives [5][max(n,nf)^2].
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <new>
#include <string>
#include <vector>

#include "../../include/nmg.h"
#include "mesh.h"
#include "fp64_fast.cuh"
#include "tc_device.cuh"
#include "weno_cell.cuh"

namespace {

using nmgk::fast_div;
using nmgk::fast_rcp;
using nmgk::fast_rsqrt;
using nmgk::fast_sqrt;
using nmgk::positive_finite;

#include "grhd.cuh"

constexpr int NF = 5;
constexpr int kMaxN = 10;   // DG points per direction
constexpr int kMaxNF = 16;  // finite-volume points per direction
// per finite-volume point: det(dXb/dx), background (8), per direction the
// unit normal and J |grad Xb^a| (4 x 3), per direction at the midpoint right
// of the point: unit normal, J |grad Xb^a|, alpha, psi^2 (6 x 3)
constexpr int kGeo = 39;
constexpr int kNT = 256;

// the equation of state as the kernels use it: rho h = rho + p hfac
struct GrEos {
  double gamma, hfac;  // hfac = gamma / (gamma - 1)
  double tau_atm;      // rho h - p of the atmosphere
};

struct ShellMap {
  int dom[6];
  double s0[6], s1[6], xc[3];
};

// x and dXb/dx-free dX/dx of the CubedShell map (constant radii s0 < s1),
// the operation order of the reference's xyz_of_lamAB_CubSph /
// dlamAB_dxyz_CubSph (src/main/coordinates/coordtrans_CubedSphere.c:37-118,
// 257-509) for dom / 2 = dir
__device__ void shell_map(const ShellMap &S, int p, const double X[3], double x[3],
                          double J[3][3]) {
  const double lam = X[0], A = X[1], B = X[2];
  const int dom = S.dom[p], dir = dom / 2;
  const int ia = dir == 1 ? 0 : 1, ib = dir == 2 ? 0 : 2;
  const double pm = 2 * (dom % 2) - 1;
  const double sq = sqrt(1.0 + A * A + B * B);
  const double a0 = pm * S.s0[p] / sq, a1 = pm * S.s1[p] / sq;
  const double rR = (a1 - a0) * lam + a0;
  x[dir] = S.xc[dir] + rR;
  x[ia] = S.xc[ia] + A * rR;
  x[ib] = S.xc[ib] + B * rR;
  double r[3];
  for (int c = 0; c < 3; c++) r[c] = (c == dir) ? rR : x[c] - S.xc[c];
  const double rc2 = r[0] * r[0] + r[1] * r[1] + r[2] * r[2];
  const double rR2 = r[dir] * r[dir];
  for (int c = 0; c < 3; c++) {
    const double m = (c == dir) ? (1.0 / rR - rR / rc2) : (-r[c] / rc2);
    const double da0 = a0 * m, da1 = a1 * m;
    J[0][c] = ((c == dir ? 1.0 : 0.0) - da0 - (da1 - da0) * lam) / (a1 - a0);
    J[1][c] = 0.;
    J[2][c] = 0.;
  }
  J[1][dir] = -r[ia] / rR2;
  J[1][ia] = 1.0 / rR;
  J[2][dir] = -r[ib] / rR2;
  J[2][ib] = J[1][ia];
}

__host__ __device__ inline void background(double mass, const double x[3], double bg[8]) {
  const double r2 = x[0] * x[0] + x[1] * x[1] + x[2] * x[2];
  const double r = sqrt(r2);
  const double a = 0.5 * mass / r;
  const double ps = 1. + a;
  const double c1 = 2. * a / (r2 * (ps * ps)), c2 = -a / r2;
  bg[0] = (1. - a) / (1. + a);
  bg[1] = ps;
  for (int i = 0; i < 3; i++) {
    bg[2 + i] = c1 * x[i];
    bg[5 + i] = c2 * x[i];
  }
}

// flux along x^i
__device__ __forceinline__ void flux_i(const double *U, const double *P, int i, double al,
                                       double ps, double F[NF]) {
  const double ps2 = ps * ps, ps6 = ps2 * ps2 * ps2;
  const double v = i == 0 ? P[1] : (i == 1 ? P[2] : P[3]);
  const double av = al * v, ap = al * ps6 * P[4];
  F[0] = av * U[0];
  F[1] = av * U[1] + (i == 0 ? ap : 0.);
  F[2] = av * U[2] + (i == 1 ? ap : 0.);
  F[3] = av * U[3] + (i == 2 ? ap : 0.);
  F[4] = av * U[4] + ap * v;
}

__device__ __forceinline__ void sources(const GrEos &g, const double *P, const double *bg,
                                        int bstride, double S[NF]) {
  const double al = bg[0], ps = bg[bstride];
  const double ps2 = ps * ps, ps4 = ps2 * ps2, ps6 = ps4 * ps2;
  const double p = P[4];
  const double v2 = ps4 * (P[1] * P[1] + P[2] * P[2] + P[3] * P[3]);
  const double rhW2 = fma(p, g.hfac, P[0]) * fast_rcp(1. - v2);
  const double E = rhW2 - p;
  const double c = 2. * al * fast_rcp(ps) * fma(3., p, rhW2 * v2);
  double vda = 0.;
  S[0] = 0.;
  for (int j = 0; j < 3; j++) {
    const double da = bg[(2 + j) * bstride], dp = bg[(5 + j) * bstride];
    S[1 + j] = ps6 * (c * dp - E * da);
    vda += P[1 + j] * da;
  }
  S[4] = -ps6 * rhW2 * vda;
}

// What the fluxes and speeds of one side need of its primitives P along a
// covector m (v . m = vm, psi^4 v^2 = v2): rho h, and the numerator and
// denominator of the largest |characteristic speed| along m,
//   alpha (|vm| (1 - cs^2) + cs sqrt((1 - v^2)(|m|^2 (1 - v^2 cs^2) - vm^2 (1 - cs^2))))
//     / (1 - v^2 cs^2),   cs^2 = gamma p / (rho h),
// multiplied through by rho h (no division here; m2 = |m|^2 = g^ij m_i m_j).
struct Side {
  double v2, vm, w, num, den;
};

__device__ __forceinline__ void side(const GrEos &g, const double *P, const double m[3],
                                     double ps4, double m2, Side &s) {
  s.v2 = ps4 * (P[1] * P[1] + P[2] * P[2] + P[3] * P[3]);
  s.vm = P[1] * m[0] + P[2] * m[1] + P[3] * m[2];
  s.w = fma(P[4], g.hfac, P[0]);
  const double gp = g.gamma * P[4], A = s.w - gp, om = 1. - s.v2;
  const double den = fma(-s.v2, gp, s.w);
  const double disc = om * gp * fma(m2, den, -(s.vm * s.vm) * A);
  s.num = fma(fabs(s.vm), fabs(A), fast_sqrt(disc));
  s.den = fabs(den);
  // cs^2 < 0 (an interpolated trace with p < 0): no sound speed, the other
  // side's speed counts
  if ((__double2hiint(gp) ^ __double2hiint(s.w)) < 0) {
    s.num = 0.;
    s.den = 1.;
  }
}

// the larger of the two sides' speeds (without the factor alpha)
__device__ __forceinline__ double larger_speed(const Side &a, const Side &b) {
  const bool first = a.num * b.den > b.num * a.den;
  return (first ? a.num : b.num) * fast_rcp(first ? a.den : b.den);
}

// conserved state without the factor psi^6
__device__ __forceinline__ void side_con(const double *P, const Side &s, double ps4, double U[NF]) {
  const double W = fast_rsqrt(1. - s.v2), rhW2 = s.w * (W * W), q = rhW2 * ps4;
  U[0] = P[0] * W;
  U[1] = q * P[1];
  U[2] = q * P[2];
  U[3] = q * P[3];
  U[4] = (rhW2 - P[4]) - U[0];
}

__host__ __device__ __forceinline__ int face_ijk(int n, int f, int a, int b) {
  const int d = f >> 1, q = (f & 1) * (n - 1);
  return d == 0 ? q + n * (a + n * b) : d == 1 ? a + n * (q + n * b) : a + n * (b + n * q);
}

__device__ __forceinline__ void orient_ab(int n, int o, int a, int b, int *a2, int *b2) {
  int aa = (o & 1) ? b : a, bb = (o & 1) ? a : b;
  if (o & 2) aa = n - 1 - aa;
  if (o & 4) bb = n - 1 - bb;
  *a2 = aa;
  *b2 = bb;
}

__device__ __forceinline__ double det3(const double M[3][3]) {
  return M[0][0] * (M[1][1] * M[2][2] - M[1][2] * M[2][1]) -
         M[0][1] * (M[1][0] * M[2][2] - M[1][2] * M[2][0]) +
         M[0][2] * (M[1][0] * M[2][1] - M[1][1] * M[2][0]);
}

// parameters of every stage kernel
struct GrP {
  int n, np, nn, nf, npf, nnf, tpts;
  int ndg, nfv;
  nmg_grhd_params g;
  GrEos eos;
  double mass;
  int rec;
  const int *dglist;     // [ndg] DG elements
  const int *slotelem;   // [nfv] element of each finite-volume slot
  const int *fvslot;     // [E] slot, -1: DG
  const int *nb, *code;  // [E][6]
  const int *tslot;      // [E][6] trace slot of a DG / FV face, -1: none
  const int *tface;      // [ntr][2] element, face of each trace slot
  int ntr;
  const double *dXbdx;   // [E][9][np] dXb^a/dx^i
  const int *mmask;      // [E] bit 3 a + i: dXb^a/dx^i is not zero on the whole element
  const double *bgd;     // [E][8][np]
  const double *bbox;    // [E][6]
  const double *basis;   // D [n*n], wl [n], xl [n], xu [nf]
  const double *geo;     // [slot][kGeo][npf]
  double *trace;         // [ntr][5][tpts]
  // stage buffers
  const double *win_d, *win_f, *u0_d, *u0_f;
  double *acc_d, *acc_f, *wout_d, *wout_f;
  const double *prim_d, *prim_f;
  double *rbuf;          // [3][slot][5][npf] divergence part of each direction
  int mode;              // 0: r into acc; 1..4: RK4 stage s
  double cacc, cw;
};

__device__ __forceinline__ void epilogue(const GrP &P, double r, size_t idx, const double *u0,
                                         double *acc, double *wout) {
  if (P.mode == 0) {
    acc[idx] = r;
  } else if (P.mode == 1) {
    const double u = u0[idx];
    acc[idx] = u + P.cacc * r;
    wout[idx] = u + P.cw * r;
  } else if (P.mode <= 3) {
    acc[idx] += P.cacc * r;
    wout[idx] = u0[idx] + P.cw * r;
  } else {
    acc[idx] += P.cacc * r;
  }
}

// c2p_point (grhd.cuh) for the stage kernels, which the FP64 pipe bounds:
// * with E = tau + D + p and v^2 = S^2/E^2 the pressure function is
//     f = (gamma - 1) (tau - W^2 v^2 (D / (W + 1) + p)) (1 - v^2) - p
//   (D (W - 1) = D W^2 v^2 / (W + 1)): two reciprocals and a reciprocal
//   square root instead of four divisions and a square root, and no
//   cancellation in W - 1; the Newton step multiplies f' = v^2 cs^2 - 1
//   through by the denominator of cs^2;
// * the signs at the ends of the bracket follow from the data where
//   S <= tau + D: f(0) >= 0 is tau (tau + 2 D) >= S^2, and at
//   (gamma - 1)(tau + D) f <= -(gamma - 1) D < 0;
// * a point that no pressure of the bracket lifts above rho_atm (a falling
//   atmosphere) is reset before the root is looked for.
// Bracket, acceptance and the atmosphere are c2p_point's.  Where rho comes
// within 1e-12 of rho_atm it is formed by c2p_point's own sequence of operations:
// the points of the atmosphere sit exactly there, and whether they are reset may
// not hang on the last bit of another formula.  fast_div and the root corrected by its
// residual round to nearest but where the exact value lies within about 2^-52 units of
// the last place of a rounding boundary; the compiler's division in their place, and for D,
// took con2prim 5.2 -> 5.4 ms a step and reset the same points.
// FP64 pipe 85 % busy; 5.0 -> 1.3 ms per stage on 9331 elements of 7^3 and 1037
// of 13^3 points (43 % of them atmosphere), 95 -> 36 us on 345 of 5^3 and 38
// of 10^3 points.

// a < b for b >= 0 (a not a number: false) and v == +-0, on the integer pipe
// (an FP64 comparison costs as much as a multiplication)
__device__ __forceinline__ bool less_bits(double a, double b) {
  return __double_as_longlong(a) < __double_as_longlong(b);
}
__device__ __forceinline__ bool zero_bits(double v) {
  return (__double_as_longlong(v) << 1) == 0;
}

struct PressureF {
  double D, tau, S2, tD, gm1, gam;
  double v2, W, om, num;  // of the last p

  __device__ __forceinline__ double operator()(double p) {
    const double y = fast_rcp(tD + p);
    v2 = S2 * (y * y);
    om = 1. - v2;
    W = fast_rsqrt(om);
    num = fma(-(W * W) * v2, fma(D, fast_rcp(W + 1.), p), tau);
    return fma(gm1 * num, om, -p);
  }
};

__device__ __forceinline__ int c2p_fast(const nmg_grhd_params &g, double tau_atm, double ps,
                                        double U[5], double P[5]) {
  const double ps4 = ps * ps * ps * ps, ps6 = ps4 * ps * ps;
  const double i6 = fast_rcp(ps6), i4 = i6 * (ps * ps);
  const double D = fast_div(U[0], ps6, i6);
  int rc = -1;
  if (!less_bits(D, g.rho_atm)) {  // D >= rho_atm, or not a number (refused below)
    const double Sx = U[1] * i6, Sy = U[2] * i6, Sz = U[3] * i6;
    PressureF q;
    q.D = D;
    q.tau = U[4] * i6;
    q.S2 = (Sx * Sx + Sy * Sy + Sz * Sz) * i4;
    q.tD = q.tau + D;
    q.gm1 = g.gamma - 1.;
    q.gam = g.gamma;
    double p = P[4], plo = 0., phi = q.gm1 * q.tD, flo, fhi;
    bool ok = isfinite(q.tD) && isfinite(q.S2);
    if (positive_finite(q.tD) && !less_bits(q.tD * q.tD, q.S2) && less_bits(q.tD, 1e10 * D)) {
      flo = fma(q.tau, fma(2., D, q.tau), -q.S2);
      fhi = -1.;
      // no p in the bracket gives rho >= rho_atm: W is at least its value at
      // p = phi, rho at most D / W (the margin covers the rounding of both)
      const double E = q.tD + phi, E2 = E * E;
      ok = ok && !less_bits((D * D) * (E2 - q.S2), (1. - 1e-12) * (g.rho_atm * g.rho_atm) * E2);
    } else if (ok) {
      plo = fast_sqrt(q.S2) - q.tau - D;
      plo = plo > 0. ? plo * (1. + 1e-14) : 0.;
      if (phi < plo) phi = 2. * plo;
      if (phi <= 0.) phi = 1e-300;
      fhi = q(phi);
      for (int k = 0; k < 200 && !(fhi < 0.); k++) fhi = q(phi *= 2.);
      flo = q(plo);
      ok = isfinite(plo) && isfinite(phi);
    }
    const double xacc = g.tol * phi;
    // newton1d_brak on [plo, phi] (src/utility/numerics/newton1d_brak.c:20-121)
    if (!ok || !((flo <= 0. && fhi >= 0.) || (flo >= 0. && fhi <= 0.))) {
      rc = -1;
    } else if (flo == 0. || fhi == 0.) {
      p = flo == 0. ? plo : phi;
      rc = 0;
    } else {
      double x = !less_bits(p, plo) && !less_bits(phi, p) ? p : 0.5 * (plo + phi);
      double xl = flo < 0. ? plo : phi, xh = flo < 0. ? phi : plo;
      double dxold = fabs(phi - plo), dx = dxold;
      rc = g.maxits + 1;
      for (int j = 1; j <= g.maxits; j++) {
        const double f = q(x);
        if (!isfinite(f)) { rc = -j; break; }
        if (zero_bits(f)) { rc = j; break; }
        if (__double2hiint(f) < 0) xl = x;
        else xh = x;
        // f' = v2 cs2 - 1 = h / den
        const double den = fma(q.gam, q.num, D * q.W);
        const double h = fma(q.v2, q.gam * q.gm1 * q.num, -den), fd = f * den;
        bool bisect = !isfinite(h) || less_bits(fabs(dxold * h), fabs(2. * fd));
        if (!bisect) {
          const double step = fd * fast_rcp(h), nx = x - step, a = nx - xh, b = nx - xl;
          const bool out = (__double2hiint(a) ^ __double2hiint(b)) >= 0 && !zero_bits(a) &&
                           !zero_bits(b);
          if (out || !isfinite(step)) {
            bisect = true;
          } else if (less_bits(fabs(step), xacc)) {
            // converged; tested before the step is found to be lost in x
            // (which newton1d_brak answers with a bisection of the bracket,
            // and so up to 25 more iterations to come back to the same x)
            x = nx;
            rc = j;
            break;
          } else if (zero_bits(nx - x)) {
            bisect = true;
          } else {
            dxold = dx;
            dx = step;
            x = nx;
          }
        }
        if (bisect) {
          dxold = dx;
          dx = 0.5 * (xh - xl);
          x = xl + dx;
          if (xl == x || less_bits(fabs(dx), xacc)) { rc = j; break; }
        }
      }
      p = x;
    }
    if (rc >= 0) {
      const double y = fast_rcp(q.tD + p), om = 1. - q.S2 * (y * y);
      double W = fast_rsqrt(om), rho = D * (om * W);
      if (fabs(rho - g.rho_atm) < 1e-12 * g.rho_atm) {
        const double sx = fast_div(U[1], ps6, i6), sy = fast_div(U[2], ps6, i6);
        const double sz = fast_div(U[3], ps6, i6);
        const double E = fast_div(U[4], ps6, i6) + D + p, E2 = E * E;
        const double v2 = fast_div(fast_div(sx * sx + sy * sy + sz * sz, ps4, i4), E2, y * y);
        const double r = fast_sqrt(1. - v2), w = fast_rcp(r);
        W = fma(fma(-r, w, 1.), w, w);
        rho = fast_div(D, W, r);
      }
      if (!positive_finite(rho) || less_bits(rho, g.rho_atm) || !positive_finite(p) || !isfinite(W)) {
        rc = -1;
      } else {
        const double fac = y * i4;
        P[0] = rho;
        P[1] = Sx * fac;
        P[2] = Sy * fac;
        P[3] = Sz * fac;
        P[4] = p;
      }
    }
  }
  if (rc < 0) {
    P[0] = g.rho_atm;
    P[1] = P[2] = P[3] = 0.;
    P[4] = g.p_atm;
    const double Da = ps6 * g.rho_atm;
    U[0] = Da;
    U[1] = U[2] = U[3] = 0.;
    U[4] = ps6 * tau_atm - Da;
  }
  return rc;
}

// con2prim of the stage input on every point in use, atmosphere fixes
// written back; stats[0] += iterations, stats[1] += atmosphere points
__global__ void c2p_kernel(GrP P, double *w_d, double *w_f, double *prim_d, double *prim_f,
                           unsigned long long *stats) {
  const int64_t nd = (int64_t)P.ndg * P.np, tot = nd + (int64_t)P.nfv * P.npf;
  unsigned long long it = 0, atm = 0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < tot;
       i += (int64_t)gridDim.x * blockDim.x) {
    double *W, *PP, ps;
    int64_t npts, q;
    if (i < nd) {
      const int e = P.dglist[i / P.np];
      q = i % P.np;
      npts = P.np;
      W = w_d + (size_t)e * NF * P.np;
      PP = prim_d + (size_t)e * NF * P.np;
      ps = P.bgd[((size_t)e * 8 + 1) * P.np + q];
    } else {
      const int64_t j = i - nd;
      const int s = (int)(j / P.npf);
      q = j % P.npf;
      npts = P.npf;
      W = w_f + (size_t)s * NF * P.npf;
      PP = prim_f + (size_t)s * NF * P.npf;
      ps = P.geo[((size_t)s * kGeo + 2) * P.npf + q];
    }
    double U[NF], Pq[NF];
    for (int f = 0; f < NF; f++) {
      U[f] = W[f * npts + q];
      Pq[f] = PP[f * npts + q];
    }
    const int rc = c2p_fast(P.g, P.eos.tau_atm, ps, U, Pq);
    for (int f = 0; f < NF; f++) {
      W[f * npts + q] = U[f];
      PP[f * npts + q] = Pq[f];
    }
    if (rc < 0) atm++;
    else it += rc;
  }
  // one atomic per warp
  for (int o = 16; o > 0; o >>= 1) {
    it += __shfl_down_sync(0xffffffffu, it, o);
    atm += __shfl_down_sync(0xffffffffu, atm, o);
  }
  if ((threadIdx.x & 31) == 0 && (it || atm)) {
    atomicAdd(stats, it);
    atomicAdd(stats + 1, atm);
  }
}

// Primitives across every DG / finite-volume face at this face's points:
// piecewise linear in each in-plane direction from a finite-volume
// neighbour, Lagrange interpolation of a DG neighbour's face plane (with
// transfer matrix Pm, one direction after the other through shared memory).
// One CTA per trace slot: n^2 nf + n nf^2 products a field instead of
// (n^2 + n) nf^2 and the Lagrange weights of every point (1.02 -> 0.15 ms per
// stage, 11,000 slots at n = 7, nf = 13).
constexpr int kNTT = 128;
__global__ void __launch_bounds__(kNTT) trace_kernel(GrP P, const double *Pm, const double *prim_d,
                                                     const double *prim_f) {
  __shared__ double sU[NF][kMaxN * kMaxN], sV[NF][kMaxNF * kMaxN], sM[kMaxNF * kMaxN];
  const int t = blockIdx.x, n = P.n, nf = P.nf;
  const int e = P.tface[2 * t], f = P.tface[2 * t + 1];
  const bool fv = P.fvslot[e] >= 0;
  const int mine = fv ? nf : n, pts = mine * mine;
  const int e2 = P.nb[6 * e + f], f2 = P.code[6 * e + f] & 7, o = (P.code[6 * e + f] >> 3) & 7;
  double *out = P.trace + (size_t)t * NF * P.tpts;
  if (fv) {
    for (int i = threadIdx.x; i < NF * n * n; i += kNTT) {
      const int q = i / (n * n), ab = i - q * n * n;
      sU[q][ab] = prim_d[((size_t)e2 * NF + q) * P.np + face_ijk(n, f2, ab % n, ab / n)];
    }
    for (int i = threadIdx.x; i < nf * n; i += kNTT) sM[i] = Pm[i];
    __syncthreads();
    for (int i = threadIdx.x; i < NF * nf * n; i += kNTT) {  // sV[q][j][a] along the first axis
      const int q = i / (nf * n), r = i - q * nf * n, a = r % nf, j = r / nf;
      double v = 0.;
      for (int k = 0; k < n; k++) v = fma(sM[a * n + k], sU[q][k + n * j], v);
      sV[q][a + nf * j] = v;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < NF * pts; i += kNTT) {
      const int q = i / pts, ab = i - q * pts, a = ab % nf, b = ab / nf;
      int a2, b2;  // this point's place on the neighbour's face
      orient_ab(nf, o, a, b, &a2, &b2);
      double v = 0.;
      for (int k = 0; k < n; k++) v = fma(sM[b2 * n + k], sV[q][a2 + nf * k], v);
      out[q * P.tpts + ab] = v;
    }
    return;
  }
  const double *xl = P.basis + n * n + n, *xu = xl + n;
  const double *src0 = prim_f + (size_t)P.fvslot[e2] * NF * P.npf;
  for (int ab = threadIdx.x; ab < pts; ab += kNTT) {
    const int a = ab % n, b = ab / n;
    double x = (o & 1) ? xl[b] : xl[a], u = (o & 1) ? xl[a] : xl[b];
    if (o & 2) x = -x;
    if (o & 4) u = -u;
    int ka = (int)floor((x + 1.) * 0.5 * (nf - 1)), kb = (int)floor((u + 1.) * 0.5 * (nf - 1));
    ka = min(max(ka, 0), nf - 2);
    kb = min(max(kb, 0), nf - 2);
    const double wa1 = (x - xu[ka]) / (xu[ka + 1] - xu[ka]), wa0 = 1. - wa1;
    const double wb1 = (u - xu[kb]) / (xu[kb + 1] - xu[kb]), wb0 = 1. - wb1;
    for (int q = 0; q < NF; q++) {
      const double *src = src0 + (size_t)q * P.npf;
      const double v0 = wa0 * src[face_ijk(nf, f2, ka, kb)] + wa1 * src[face_ijk(nf, f2, ka + 1, kb)];
      const double v1 =
          wa0 * src[face_ijk(nf, f2, ka, kb + 1)] + wa1 * src[face_ijk(nf, f2, ka + 1, kb + 1)];
      out[q * P.tpts + ab] = wb0 * v0 + wb1 * v1;
    }
  }
}

// exterior state of face node (a, b) of face f of element e; false: outer
// face.  Same-type neighbours are read at the coincident point, the others
// from the trace slot (primitives; U from prim2con at psi ps).
__device__ bool exterior(const GrP &P, int e, int f, int a, int b, double ps, double Uo[NF],
                         double Po[NF]) {
  const int e2 = P.nb[6 * e + f];
  if (e2 < 0) return false;
  const bool fv = P.fvslot[e] >= 0, fv2 = P.fvslot[e2] >= 0;
  if (fv == fv2) {
    const int nn = fv ? P.nf : P.n, npts = fv ? P.npf : P.np;
    const int f2 = P.code[6 * e + f] & 7, o = (P.code[6 * e + f] >> 3) & 7;
    int a2, b2;
    orient_ab(nn, o, a, b, &a2, &b2);
    const int idx = face_ijk(nn, f2, a2, b2);
    const size_t row = fv ? (size_t)P.fvslot[e2] : (size_t)e2;
    const double *W = fv ? P.win_f : P.win_d, *PP = fv ? P.prim_f : P.prim_d;
    for (int q = 0; q < NF; q++) {
      Uo[q] = W[(row * NF + q) * npts + idx];
      Po[q] = PP[(row * NF + q) * npts + idx];
    }
    return true;
  }
  const int t = P.tslot[6 * e + f];
  const int mine = fv ? P.nf : P.n;
  const double *tr = P.trace + (size_t)t * NF * P.tpts;
  for (int q = 0; q < NF; q++) Po[q] = tr[q * P.tpts + a + mine * b];
  const double ps2 = ps * ps, ps4 = ps2 * ps2, ps6 = ps4 * ps2;
  Side s;
  s.v2 = ps4 * (Po[1] * Po[1] + Po[2] * Po[2] + Po[3] * Po[3]);
  s.w = fma(Po[4], P.eos.hfac, Po[0]);
  side_con(Po, s, ps4, Uo);
  for (int q = 0; q < NF; q++) Uo[q] *= ps6;
  return true;
}

// DG faces (LLF with the fluid's characteristic speeds, lifted with
// |grad Xb^d| / w_end), one direction at a time (its two faces are
// disjoint), then the stage update of the element's r (shared by the DG
// kernels).  The flux and the speed are taken along the covector
// grad Xb^d itself, so that its length needs no square root and no division:
// |grad Xb^d| (f* - f_in) = (F_out - F_in) . m / 2 - a_m (U_out - U_in) / 2;
// one reciprocal and two square roots a node instead of ~14 divisions and
// five square roots.
__device__ __forceinline__ void dg_faces_epilogue(const GrP &P, int e, double *sR,
                                                  const double *Pg, const double *Ug,
                                                  const double *M, const double *bg,
                                                  double w_end) {
  const int n = P.n, np = P.np, nn = P.nn;
  const double hw = 0.5 / w_end;
  for (int d = 0; d < 3; d++) {
    for (int task = threadIdx.x; task < 2 * nn; task += blockDim.x) {
      const int sd = task / nn, ab = task - sd * nn, a = ab % n, b = ab / n;
      const int f = 2 * d + sd, q2 = face_ijk(n, f, a, b);
      const double al = bg[q2], ps = bg[np + q2];
      double Ui[NF], Pi[NF], Uo[NF], Po[NF];
      if (!exterior(P, e, f, a, b, ps, Uo, Po)) continue;
      for (int q = 0; q < NF; q++) {
        Ui[q] = Ug[q * np + q2];
        Pi[q] = Pg[q * np + q2];
      }
      const double m[3] = {M[(d * 3 + 0) * np + q2], M[(d * 3 + 1) * np + q2],
                           M[(d * 3 + 2) * np + q2]};
      const double ps2 = ps * ps, ps4 = ps2 * ps2;
      const double m2 = (m[0] * m[0] + m[1] * m[1] + m[2] * m[2]) * fast_rcp(ps4);
      Side si, so;
      side(P.eos, Pi, m, ps4, m2, si);
      side(P.eos, Po, m, ps4, m2, so);
      const double am = larger_speed(si, so), sg = sd ? 1. : -1.;
      // outward: the covector is sd ? m : -m
      const double vi = sg * si.vm, vo = sg * so.vm;
      const double ap = sg * (ps4 * ps2) * (Po[4] - Pi[4]);
      const double g = hw * al;
      double *r = sR + q2;
      r[0] -= g * ((vo * Uo[0] - vi * Ui[0]) - am * (Uo[0] - Ui[0]));
      r[np] -= g * ((vo * Uo[1] - vi * Ui[1]) + (ap * m[0] - am * (Uo[1] - Ui[1])));
      r[2 * np] -= g * ((vo * Uo[2] - vi * Ui[2]) + (ap * m[1] - am * (Uo[2] - Ui[2])));
      r[3 * np] -= g * ((vo * Uo[3] - vi * Ui[3]) + (ap * m[2] - am * (Uo[3] - Ui[3])));
      r[4 * np] -= g * ((vo * Uo[4] - vi * Ui[4]) +
                        ((ps4 * ps2) * (vo * Po[4] - vi * Pi[4]) - am * (Uo[4] - Ui[4])));
    }
    __syncthreads();
  }
  for (int i = threadIdx.x; i < NF * np; i += blockDim.x)
    epilogue(P, sR[i], (size_t)e * NF * np + i, P.u0_d, P.acc_d, P.wout_d);
}

// DG elements: one CTA per element
__global__ void __launch_bounds__(kNT) dg_kernel(GrP P) {
  extern __shared__ double sm[];
  const int n = P.n, np = P.np, nn = P.nn;
  double *sF = sm, *sR = sF + 15 * np, *sD = sR + NF * np;
  const int e = P.dglist[blockIdx.x];
  const double *Pg = P.prim_d + (size_t)e * NF * np, *Ug = P.win_d + (size_t)e * NF * np;
  const double *M = P.dXbdx + (size_t)e * 9 * np, *bg = P.bgd + (size_t)e * 8 * np;
  const int mask = P.mmask[e];
  const double w_end = P.basis[n * n];
  for (int i = threadIdx.x; i < n * n; i += blockDim.x) sD[i] = P.basis[i];
  __syncthreads();
  for (int q = threadIdx.x; q < np; q += blockDim.x) {
    double Uq[NF], Pq[NF], Fq[NF];
    for (int f = 0; f < NF; f++) {
      Uq[f] = Ug[f * np + q];
      Pq[f] = Pg[f * np + q];
    }
    const double al = bg[q], ps = bg[np + q];
    for (int i = 0; i < 3; i++) {
      flux_i(Uq, Pq, i, al, ps, Fq);
      for (int f = 0; f < NF; f++) sF[(i * NF + f) * np + q] = Fq[f];
    }
    sources(P.eos, Pq, bg + q, np, Fq);
    for (int f = 0; f < NF; f++) sR[f * np + q] = Fq[f];
  }
  __syncthreads();
  // strong-form divergence with the chain rule
  for (int task = threadIdx.x; task < NF * np; task += blockDim.x) {
    const int f = task / np, q = task - f * np;
    const int ijk[3] = {q % n, (q / n) % n, q / nn};
    const int str[3] = {1, n, nn};
    double div = 0.;
    for (int i = 0; i < 3; i++) {
      const double *Fi = sF + (i * NF + f) * np;
      for (int a = 0; a < 3; a++) {
        if (!((mask >> (3 * a + i)) & 1)) continue;
        const int base = q - ijk[a] * str[a];
        const double *Dr = sD + ijk[a] * n;
        double ds = 0.;
        for (int k = 0; k < n; k++) ds += Dr[k] * Fi[base + k * str[a]];
        div += M[(a * 3 + i) * np + q] * ds;
      }
    }
    sR[f * np + q] -= div;
  }
  __syncthreads();
  dg_faces_epilogue(P, e, sR, Pg, Ug, M, bg, w_end);
}

// DG elements with the divergence's line derivatives on the tensor cores
// (n = 7, 8, 9; the exact integer digit products of stage_tc.cu): the fluxes
// F^i along x^i are formed one i at a time for the five fields, split into
// digits, and D applied along every direction a by 16-line MMA tiles (the
// line left over at odd n in FP64); the chain rule M[a][i] D_a F^i with
// M = dXb/dx (whose entries that vanish on the element, two of nine on a
// cubed shell, are left out with their derivatives), the sources, the faces
// and the update are dg_kernel's FP64 code.  The primitives are read from
// global memory (L1), which leaves 55 KB of shared memory an element at n = 7.
// FP64 pipe 72 % busy; 4.4 -> 2.15 ms per stage on 9331 elements at n = 7
// (2.38 with three CTAs on an SM instead of four).
// Threads and CTAs per SM: a pass has 5 fields x (3, 4, 5) tiles at n = 7, 8, 9
// and an element 55, 82, 117 KB, so five warps four times, ten twice,
// thirteen once.
template <int N>
constexpr int dg_tc_threads() {
  return N == 7 ? 160 : (N == 8 ? 320 : 416);
}
template <int N>
constexpr int dg_tc_ctas() {
  return N == 7 ? 4 : (N == 8 ? 2 : 1);
}
template <int N>
constexpr size_t dg_tc_smem() {
  return sizeof(double) * 2 * NF * N * N * N + sizeof(uint4) * NF * N * N * N;
}

template <int N>
__global__ void __launch_bounds__(dg_tc_threads<N>(), dg_tc_ctas<N>()) dg_tc_kernel(GrP P) {
  using S = nmgk::TcShape<N>;
  constexpr int np = S::NP, nn = S::NN, TILES = S::TILES, kNTD = dg_tc_threads<N>(),
                NWARP = kNTD / 32;
  extern __shared__ __align__(16) unsigned char gsm[];
  // the digits first: ldmatrix rows and uint4 stores want 16-byte addresses,
  // and 10 np doubles are not a multiple of 16 bytes at odd np
  uint4 *sDig = reinterpret_cast<uint4 *>(gsm);                 // [5][np] digits of sF
  double *sR = reinterpret_cast<double *>(sDig + NF * np);      // [5][np] r
  double *sF = sR + NF * np;                                    // [5][np] fluxes along x^i
  __shared__ int sEmax[3][NF];
  const int e = P.dglist[blockIdx.x];
  const double *Pg = P.prim_d + (size_t)e * NF * np, *Ug = P.win_d + (size_t)e * NF * np;
  const double *M = P.dXbdx + (size_t)e * 9 * np, *bg = P.bgd + (size_t)e * 8 * np;
  const int mask = P.mmask[e];
  const double w_end = P.basis[N * N];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, tq = lane & 3;
  if (tid < 3 * NF) sEmax[tid / NF][tid % NF] = 0;
  for (int q = tid; q < np; q += kNTD) {
    double Pq[NF], Fq[NF];
    for (int f = 0; f < NF; f++) Pq[f] = Pg[f * np + q];
    sources(P.eos, Pq, bg + q, np, Fq);
    for (int f = 0; f < NF; f++) sR[f * np + q] = Fq[f];
  }
  const uint32_t digbase = (uint32_t)__cvta_generic_to_shared(sDig);
  const int fd0 = nmgk::cTcRowExp[N - 7][tq], fd1 = nmgk::cTcRowExp[N - 7][min(tq + 4, 8)];
  const int fd8 = nmgk::cTcRowExp[N - 7][8];
  const uint4 *gB = &nmgk::gTcB[N - 7][0][0][0];
  const double *gD = nmgk::gTcD[N - 7];
  __syncthreads();  // sEmax
#pragma unroll 1
  for (int i = 0; i < 3; i++) {
    {
      // the fluxes along x^i and each field's largest exponent
      int em[NF] = {0, 0, 0, 0, 0};
      for (int q = tid; q < np; q += kNTD) {
        double Uq[NF], Pq[NF], Fq[NF];
        for (int f = 0; f < NF; f++) {
          Uq[f] = Ug[f * np + q];
          Pq[f] = Pg[f * np + q];
        }
        flux_i(Uq, Pq, i, bg[q], bg[np + q], Fq);
        for (int f = 0; f < NF; f++) {
          sF[f * np + q] = Fq[f];
          em[f] = max(em[f], (int)((unsigned long long)__double_as_longlong(Fq[f]) >> 52) & 0x7FF);
        }
      }
#pragma unroll
      for (int f = 0; f < NF; f++) {
        const unsigned m = __reduce_max_sync(0xffffffffu, (unsigned)em[f]);
        if (lane == 0) atomicMax(&sEmax[i][f], (int)m);
      }
    }
    __syncthreads();
    for (int q = tid; q < NF * np; q += kNTD) sDig[q] = nmgk::tc_digits(sF[q], sEmax[i][q / np]);
    __syncthreads();
#pragma unroll 1
    for (int a = 0; a < 3; a++) {
      if (!((mask >> (3 * a + i)) & 1)) continue;
      const double *Mai = M + (a * 3 + i) * np;
#pragma unroll 1
      for (int task = warp; task < NF * TILES; task += NWARP) {
        const int f = task / TILES, tile = task - f * TILES;
        const int Lr = min(tile * 16 + (lane & 15), nn - 1), chunk = lane >> 4;
        const int ps = a == 0 ? 1 : (a == 1 ? N : nn);
        const int nb = a == 0 ? N * Lr : (a == 1 ? (Lr % N) + nn * (Lr / N) : Lr);
        // owned output slots as in stage_tc.cu's kernel, and M[a][i] there
        int nodeS[5];
        bool okS[5];
        double mS[5];
#pragma unroll
        for (int sl = 0; sl < 5; sl++) {
          const int L = tile * 16 + g + (sl < 4 ? (sl >> 1) * 8 : tq * 8);
          const int io = sl < 4 ? tq + (sl & 1) * 4 : N - 1;
          okS[sl] = L < nn && io < N && (sl < 4 ? true : (N == 9 && tq < 2));
          nodeS[sl] = okS[sl] ? nmgk::tc_node<N>(a, L, io) : 0;
          mS[sl] = okS[sl] ? Mai[nodeS[sl]] : 0.;
        }
        double dv[5];
        nmgk::tc_derivs<N>(gB, digbase + (uint32_t)(f * np + nb) * 16u, (uint32_t)ps * 16u,
                           chunk, lane, tq, sEmax[i][f], fd0, fd1, fd8, dv);
#pragma unroll
        for (int sl = 0; sl < 5; sl++)
          if (okS[sl]) sR[f * np + nodeS[sl]] -= mS[sl] * dv[sl];
      }
      if (S::LAST) {
        // the line left over (l0 = l1 = n - 1) in FP64
        for (int t = tid; t < NF * N; t += kNTD) {
          const int f = t / N, io = t - f * N, L = nn - 1;
          double d = 0.;
          for (int p = 0; p < N; p++)
            d = fma(__ldg(gD + io * N + p), sF[f * np + nmgk::tc_node<N>(a, L, p)], d);
          const int node = nmgk::tc_node<N>(a, L, io);
          sR[f * np + node] -= Mai[node] * d;
        }
      }
      __syncthreads();
    }
  }
  dg_faces_epilogue(P, e, sR, Pg, Ug, M, bg, w_end);
}

// Finite-volume elements: one CTA per (slot, direction a, plane of nf
// pencils along a).  (1) per cell and field both face values of the cell's
// reconstruction, walked by stencil class so that warps do not diverge,
// (2) per midpoint the LLF flux of the two states meeting there and, in the
// warps after those, the outward flux of the pencils' ends, (3) per point
// the flux difference into the direction's part of rbuf, which
// fv_update_kernel gathers.  Bound by the FP64 pipe.  A plane of
// pencils wants 28 KB at nf = 13, so that several CTAs share an SM and their
// phases overlap, and 3 nf CTAs an element fill the chip when few elements
// are finite volume (one CTA an element took 205 KB and 512 threads).  FP64
// pipe 87 % busy; 17.5 -> 4.65 ms per stage (with fv_update_kernel) on 1037
// elements at nf = 13, 1.2 -> 0.11 ms on 38 at nf = 10, of which the
// instructions saved (fp64_fast.cuh, weno_cell.cuh, struct Side) account for
// a factor of 3.
__host__ __device__ __forceinline__ int fv_threads(int nf) {
  return ((nf * (nf - 1) + 31) / 32 + (2 * nf + 31) / 32) * 32;
}
__host__ __device__ __forceinline__ size_t fv_smem(int nf) {
  return sizeof(double) * NF * ((size_t)3 * nf * nf + (size_t)nf * (nf + 1));
}

template <int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB) fv_flux_kernel(GrP P) {
  extern __shared__ double sm[];
  const int nf = P.nf, npf = P.npf, nnf = P.nnf, nt = blockDim.x;
  const int plane = blockIdx.x % nf, a = (blockIdx.x / nf) % 3, slot = blockIdx.x / (3 * nf);
  const int e = P.slotelem[slot];
  double *sP = sm, *sQ = sP + NF * nnf;  // sQ: [2: left, right face][5][nnf]
  double *sG = sQ + 2 * NF * nnf;        // [5][nf (nf + 1)] fluxes: midpoints, then both ends
  const double *Pg = P.prim_f + (size_t)slot * NF * npf, *Ug = P.win_f + (size_t)slot * NF * npf;
  const double *G = P.geo + (size_t)slot * kGeo * npf;
  const int gst = nf * (nf + 1);
  // point t of pencil k: memory index, and index in shared memory; the
  // faster of the two runs along x where one of them does
  const int sa = a == 0 ? 1 : (a == 1 ? nf : nnf);             // along the pencil
  const int sk = a == 0 ? nf : 1;                              // from pencil to pencil
  const int off = plane * (a == 2 ? nf : nnf);
  const int ca = a == 0 ? 1 : nf, ck = a == 0 ? nf : 1;        // the same in shared memory
  for (int i = threadIdx.x; i < NF * nnf; i += nt) {
    const int f = i / nnf, r = i - f * nnf, t = (r / ca) % nf, k = (r / ck) % nf;
    sP[i] = Pg[f * npf + off + t * sa + k * sk];
  }
  __syncthreads();
  for (int i = threadIdx.x; i < NF * nnf; i += nt) {
    // i = ((class position) * 5 + field) * nf + pencil
    const int k = i % nf, r = i / nf, f = r % NF, c = nmgk::class_cell(P.rec, nf, r / NF);
    double lft, rgt;
    nmgk::cell_faces(P.rec, nf, sP + f * nnf + k * ck, ca, c, 2., &lft, &rgt);
    sQ[f * nnf + k * ck + c * ca] = lft;
    sQ[(NF + f) * nnf + k * ck + c * ca] = rgt;
  }
  __syncthreads();
  const int nmid = nf * (nf - 1), midw = (nmid + 31) / 32 * 32;
  if (threadIdx.x < midw) {
    const int i = threadIdx.x;
    if (i < nmid) {
      // midpoint t (between points t and t + 1) of pencil k
      const int t = a == 0 ? i % (nf - 1) : i / nf, k = a == 0 ? i / (nf - 1) : i % nf;
      const int qm = off + t * sa + k * sk, qs = t * ca + k * ck;
      const double *gm = G + (21 + 6 * a) * npf + qm;
      const double nr[3] = {gm[0], gm[npf], gm[2 * npf]};
      const double jg = gm[3 * npf], al = gm[4 * npf], ps2 = gm[5 * npf];
      const double ps4 = ps2 * ps2, ip4 = fast_rcp(ps4);
      double PL[NF], PR[NF], UL[NF], UR[NF];
      Side L, R;
      for (int f = 0; f < NF; f++) {
        PL[f] = sQ[(NF + f) * nnf + qs];  // right face of cell t
        PR[f] = sQ[f * nnf + qs + ca];    // left face of cell t + 1
      }
      // first order where a reconstructed state is unphysical (v^2 >= 1 or not
      // a number shows in the sign and exponent of 1 - v^2)
      side(P.eos, PL, nr, ps4, ip4, L);
      side(P.eos, PR, nr, ps4, ip4, R);
      if (!positive_finite(PL[0]) || !positive_finite(PL[4]) || !positive_finite(1. - L.v2)) {
        for (int f = 0; f < NF; f++) PL[f] = sP[f * nnf + qs];
        side(P.eos, PL, nr, ps4, ip4, L);
      }
      if (!positive_finite(PR[0]) || !positive_finite(PR[4]) || !positive_finite(1. - R.v2)) {
        for (int f = 0; f < NF; f++) PR[f] = sP[f * nnf + qs + ca];
        side(P.eos, PR, nr, ps4, ip4, R);
      }
      side_con(PL, L, ps4, UL);
      side_con(PR, R, ps4, UR);
      const double am = larger_speed(L, R);
      const double g = 0.5 * jg * al * (ps4 * ps2), ps = PL[4] + PR[4];
      double F[NF];
      for (int f = 0; f < NF; f++)
        F[f] = fma(L.vm, UL[f], fma(R.vm, UR[f], -am * (UR[f] - UL[f])));
      for (int j = 0; j < 3; j++) F[1 + j] = fma(ps, nr[j], F[1 + j]);
      F[4] = fma(PL[4], L.vm, fma(PR[4], R.vm, F[4]));
      for (int f = 0; f < NF; f++) sG[f * gst + k * (nf + 1) + t] = g * F[f];
    }
  } else if (threadIdx.x - midw < 2 * nf) {
    // end of pencil k on side sd: outward flux
    const int i = threadIdx.x - midw, sd = i / nf, k = i - sd * nf, t = sd ? nf - 1 : 0;
    const int qq = off + t * sa + k * sk, qs = t * ca + k * ck;
    // in-plane coordinates of the face point: (o1, o2) = (k, plane), o1 < o2
    const double sg = sd ? 1. : -1.;
    const double *gq = G + (9 + 4 * a) * npf + qq;
    const double nr[3] = {sg * gq[0], sg * gq[npf], sg * gq[2 * npf]};
    const double jg = gq[3 * npf], al = G[npf + qq], ps = G[2 * npf + qq];
    const double ps2 = ps * ps, ps4 = ps2 * ps2, ps6 = ps4 * ps2;
    double Ui[NF], Pi[NF], Uo[NF], Po[NF], F[NF];
    for (int f = 0; f < NF; f++) {
      Ui[f] = Ug[f * npf + qq];
      Pi[f] = sP[f * nnf + qs];
    }
    if (exterior(P, e, 2 * a + sd, k, plane, ps, Uo, Po)) {
      const double ip4 = fast_rcp(ps4);
      Side si, so;
      side(P.eos, Pi, nr, ps4, ip4, si);
      side(P.eos, Po, nr, ps4, ip4, so);
      const double am = larger_speed(si, so), ap = ps6 * (Pi[4] + Po[4]);
      for (int f = 0; f < NF; f++)
        F[f] = fma(si.vm, Ui[f], fma(so.vm, Uo[f], -am * (Uo[f] - Ui[f])));
      for (int j = 0; j < 3; j++) F[1 + j] = fma(ap, nr[j], F[1 + j]);
      F[4] = fma(ps6, fma(Pi[4], si.vm, Po[4] * so.vm), F[4]);
      for (int f = 0; f < NF; f++) F[f] *= 0.5;
    } else {
      const double vn = Pi[1] * nr[0] + Pi[2] * nr[1] + Pi[3] * nr[2], ap = ps6 * Pi[4];
      for (int f = 0; f < NF; f++) F[f] = vn * Ui[f];
      for (int j = 0; j < 3; j++) F[1 + j] = fma(ap, nr[j], F[1 + j]);
      F[4] = fma(ap, vn, F[4]);
    }
    for (int f = 0; f < NF; f++) sG[f * gst + k * (nf + 1) + nf - 1 + sd] = jg * al * F[f];
  }
  __syncthreads();
  double *R = P.rbuf + ((size_t)a * P.nfv + slot) * NF * npf;
  const double ih = (nf - 1) / 2.;  // 1/h, h = 2/(nf - 1)
  for (int i = threadIdx.x; i < nnf; i += nt) {
    const int t = (i / ca) % nf, k = (i / ck) % nf, qq = off + t * sa + k * sk;
    // det / h (det / (h/2) at the pencil ends) times the flux difference
    const double dh = G[qq] * ((t == 0 || t == nf - 1) ? 2. * ih : ih);
    for (int f = 0; f < NF; f++) {
      const double *g0 = sG + f * gst + k * (nf + 1);
      double df;
      if (t == 0) df = g0[0] + g0[nf - 1];
      else if (t == nf - 1) df = g0[nf] - g0[nf - 2];
      else df = g0[t] - g0[t - 1];
      R[f * npf + qq] = dh * df;
    }
  }
}

// sources minus the divergence of the three directions, and the stage update
__global__ void __launch_bounds__(kNT) fv_update_kernel(GrP P) {
  const int npf = P.npf;
  const int64_t tot = (int64_t)P.nfv * npf;
  const size_t dst = (size_t)P.nfv * NF * npf;  // from direction to direction
  for (int64_t i = blockIdx.x * (int64_t)kNT + threadIdx.x; i < tot; i += (int64_t)gridDim.x * kNT) {
    const int slot = (int)(i / npf), q = (int)(i - (int64_t)slot * npf);
    const size_t base = (size_t)slot * NF * npf + q;
    double Pq[NF], S[NF];
    for (int f = 0; f < NF; f++) Pq[f] = P.prim_f[base + (size_t)f * npf];
    sources(P.eos, Pq, P.geo + ((size_t)slot * kGeo + 1) * npf + q, npf, S);
    for (int f = 0; f < NF; f++) {
      const size_t idx = base + (size_t)f * npf;
      const double r = ((S[f] - P.rbuf[idx]) - P.rbuf[dst + idx]) - P.rbuf[2 * dst + idx];
      epilogue(P, r, idx, P.u0_f, P.acc_f, P.wout_f);
    }
  }
}

// dX/dx of every DG element to dXb/dx (times 2/dX^a), in place, and the
// mask of the entries that do not vanish on the whole element
__global__ void metric_kernel(int np, const double *bbox, double *M, int *mask) {
  const int e = blockIdx.x;
  int bits = 0;
  for (int k = 0; k < 9; k++) {
    const double *bb = bbox + 6 * (size_t)e + 2 * (k / 3), sc = 2. / (bb[1] - bb[0]);
    double *row = M + ((size_t)e * 9 + k) * np;
    int any = 0;
    for (int q = threadIdx.x; q < np; q += blockDim.x) {
      any |= row[q] != 0.;
      row[q] *= sc;
    }
    if (__syncthreads_or(any)) bits |= 1 << k;
  }
  if (threadIdx.x == 0) mask[e] = bits;
}

// geometry of the finite-volume slots (points and midpoints) from the map
__global__ void fvgeo_kernel(GrP P, ShellMap S, const int *pat, double *geo) {
  const int nf = P.nf, npf = P.npf;
  const double *xu = P.basis + P.n * P.n + 2 * P.n;
  const int64_t tot = (int64_t)P.nfv * npf;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < tot;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int slot = (int)(i / npf), q = (int)(i % npf), e = P.slotelem[slot];
    const int id[3] = {q % nf, (q / nf) % nf, q / (nf * nf)};
    const double *bb = P.bbox + 6 * (size_t)e;
    double *G = geo + (size_t)slot * kGeo * npf + q;
    auto eval = [&](const double Xb[3], double x[3], double Mb[3][3]) {
      double X[3], J[3][3];
      for (int d = 0; d < 3; d++)
        X[d] = 0.5 * ((bb[2 * d + 1] - bb[2 * d]) * Xb[d] + (bb[2 * d + 1] + bb[2 * d]));
      shell_map(S, pat[e], X, x, J);
      for (int d = 0; d < 3; d++)
        for (int c = 0; c < 3; c++) Mb[d][c] = (2. / (bb[2 * d + 1] - bb[2 * d])) * J[d][c];
    };
    double Xb[3] = {xu[id[0]], xu[id[1]], xu[id[2]]}, x[3], Mb[3][3], bgv[8];
    eval(Xb, x, Mb);
    const double det = det3(Mb);
    background(P.mass, x, bgv);
    G[0] = det;
    for (int k = 0; k < 8; k++) G[(1 + k) * npf] = bgv[k];
    for (int a = 0; a < 3; a++) {
      const double nm = sqrt(Mb[a][0] * Mb[a][0] + Mb[a][1] * Mb[a][1] + Mb[a][2] * Mb[a][2]);
      for (int c = 0; c < 3; c++) G[(9 + 4 * a + c) * npf] = Mb[a][c] / nm;
      G[(12 + 4 * a) * npf] = nm / det;
    }
    for (int a = 0; a < 3; a++) {
      double *Gm = G + (21 + 6 * a) * npf;
      if (id[a] >= nf - 1) {
        for (int k = 0; k < 6; k++) Gm[k * npf] = 0.;
        continue;
      }
      double Xm[3] = {Xb[0], Xb[1], Xb[2]}, xm[3], Mm[3][3], bm[8];
      Xm[a] = 0.5 * (xu[id[a]] + xu[id[a] + 1]);
      eval(Xm, xm, Mm);
      background(P.mass, xm, bm);
      const double nm = sqrt(Mm[a][0] * Mm[a][0] + Mm[a][1] * Mm[a][1] + Mm[a][2] * Mm[a][2]);
      for (int c = 0; c < 3; c++) Gm[c * npf] = Mm[a][c] / nm;
      Gm[3 * npf] = nm / det3(Mm);
      Gm[4 * npf] = bm[0];
      Gm[5 * npf] = bm[1] * bm[1];
    }
  }
}

// out = (A x A x A) in for every field of the listed elements, A (no x ni);
// src/dst rows given per element (in row isrc[k], out row idst[k])
__global__ void convert_kernel(const double *A, int ni, int no, const int *isrc,
                               const int *idst, const double *src, double *dst) {
  extern __shared__ double sm[];
  const int ni3 = ni * ni * ni, no3 = no * no * no;
  double *sIn = sm, *t1 = sIn + ni3, *t2 = t1 + no * ni * ni, *sA = t2 + no * no * ni;
  const int k = blockIdx.x;
  for (int i = threadIdx.x; i < no * ni; i += blockDim.x) sA[i] = A[i];
  for (int f = 0; f < NF; f++) {
    const double *in = src + ((size_t)isrc[k] * NF + f) * ni3;
    double *out = dst + ((size_t)idst[k] * NF + f) * no3;
    __syncthreads();
    for (int i = threadIdx.x; i < ni3; i += blockDim.x) sIn[i] = in[i];
    __syncthreads();
    for (int t = threadIdx.x; t < no * ni * ni; t += blockDim.x) {
      const int i = t % no, jk = t / no;
      double s = 0.;
      for (int m = 0; m < ni; m++) s += sA[i * ni + m] * sIn[m + ni * jk];
      t1[t] = s;
    }
    __syncthreads();
    for (int t = threadIdx.x; t < no * no * ni; t += blockDim.x) {
      const int i = t % no, j = (t / no) % no, kk = t / (no * no);
      double s = 0.;
      for (int m = 0; m < ni; m++) s += sA[j * ni + m] * t1[i + no * (m + ni * kk)];
      t2[t] = s;
    }
    __syncthreads();
    for (int t = threadIdx.x; t < no3; t += blockDim.x) {
      const int i = t % no, j = (t / no) % no, kk = t / (no * no);
      double s = 0.;
      for (int m = 0; m < ni; m++) s += sA[kk * ni + m] * t2[i + no * (j + no * m)];
      out[t] = s;
    }
  }
}

// copy rows (element states of 5 fields) between slot layouts
__global__ void copy_rows_kernel(int64_t rowlen, const int *isrc, const int *idst,
                                 const double *src, double *dst) {
  const int k = blockIdx.y;
  const double *in = src + (size_t)isrc[k] * rowlen;
  double *out = dst + (size_t)idst[k] * rowlen;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < rowlen;
       i += (int64_t)gridDim.x * blockDim.x)
    out[i] = in[i];
}

// Persson's modal indicator of D (field 0) per element (the reference's
// evolve_Persson_array_indicator, src/main/evolve/trouble.c:505-564): the
// LGL nodal values (a finite-volume element's projected back by R x R x R)
// analysed into normalised Legendre coefficients c by A x A x A, then
// log10(sum of c^2 over the modes of highest degree in some direction /
// sum of all c^2).  One CTA per element.
__global__ void persson_kernel(GrP P, const double *u_d, const double *u_f, const double *A,
                               const double *R, double *ind) {
  extern __shared__ double sm[];
  const int n = P.n, np = P.np, nf = P.nf;
  const int e = blockIdx.x, slot = P.fvslot[e];
  double *sU = sm, *t1 = sU + max(np, P.npf), *t2 = t1 + max(n * nf * nf, np);
  double *sC = t2 + max(n * n * nf, np), *red = sC + np;
  // nodal values of D on the LGL points
  if (slot < 0) {
    for (int q = threadIdx.x; q < np; q += blockDim.x) sU[q] = u_d[(size_t)e * NF * np + q];
  } else {
    const int npf = P.npf;
    for (int q = threadIdx.x; q < npf; q += blockDim.x) sU[q] = u_f[(size_t)slot * NF * npf + q];
    __syncthreads();
    for (int t = threadIdx.x; t < n * nf * nf; t += blockDim.x) {
      const int i = t % n, jk = t / n;
      double s = 0.;
      for (int m = 0; m < nf; m++) s += R[i * nf + m] * sU[m + nf * jk];
      t1[t] = s;
    }
    __syncthreads();
    for (int t = threadIdx.x; t < n * n * nf; t += blockDim.x) {
      const int i = t % n, j = (t / n) % n, k = t / (n * n);
      double s = 0.;
      for (int m = 0; m < nf; m++) s += R[j * nf + m] * t1[i + n * (m + nf * k)];
      t2[t] = s;
    }
    __syncthreads();
    for (int t = threadIdx.x; t < np; t += blockDim.x) {
      const int i = t % n, j = (t / n) % n, k = t / (n * n);
      double s = 0.;
      for (int m = 0; m < nf; m++) s += R[k * nf + m] * t2[i + n * (j + n * m)];
      sC[t] = s;
    }
    __syncthreads();
    for (int t = threadIdx.x; t < np; t += blockDim.x) sU[t] = sC[t];
  }
  __syncthreads();
  // modal analysis, one direction at a time (as nmo_persson)
  for (int d = 0; d < 3; d++) {
    const int st = d == 0 ? 1 : (d == 1 ? n : n * n);
    for (int k = threadIdx.x; k < np; k += blockDim.x) {
      const int ii = d == 0 ? k % n : (d == 1 ? (k / n) % n : k / (n * n));
      const double *line = sU + k - ii * st;
      double sum = 0.;
      for (int l = 0; l < n; l++) sum += A[ii * n + l] * line[l * st];
      sC[k] = sum;
    }
    __syncthreads();
    for (int k = threadIdx.x; k < np; k += blockDim.x) sU[k] = sC[k];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    double all = 0., hi = 0.;
    for (int k = 0; k < n; k++)
      for (int j = 0; j < n; j++)
        for (int i = 0; i < n; i++) {
          const double co = sU[i + n * (j + n * k)];
          all += co * co;
          if (i == n - 1 || j == n - 1 || k == n - 1) hi += co * co;
        }
    ind[e] = log10(hi / (all + 2.2250738585072014e-308) + 1e-50);
  }
  (void)red;
}

__global__ void p2c_kernel(nmg_grhd_params g, int64_t nrows, int npts, const double *psi_rows,
                           int psi_stride, const int *psi_row_of, const double *prim,
                           double *cons) {
  const int64_t tot = nrows * npts;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < tot;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = i / npts, q = i % npts;
    const int pr = psi_row_of ? psi_row_of[r] : (int)r;
    const double ps = psi_rows[(size_t)pr * psi_stride + q];
    double P[NF], U[NF];
    for (int f = 0; f < NF; f++) P[f] = prim[(r * NF + f) * npts + q];
    p2c_point(g, ps, P, U);
    for (int f = 0; f < NF; f++) cons[(r * NF + f) * npts + q] = U[f];
  }
}


}  // namespace

// ---------------------------------------------------------------------------
// context
// ---------------------------------------------------------------------------
struct nmg_grhd_ctx {
  std::string err;
  int device = -1;
  cudaStream_t stream = nullptr, fv_stream = nullptr;
  cudaEvent_t fork_ev = nullptr, join_ev = nullptr;  // fv_stream branches off and joins
  nmg_grhd_evolve_params prm{};
  int n = 0, np = 0, nn = 0, nf = 0, npf = 0, nnf = 0, tpts = 0;
  int64_t E = 0;
  ShellMap shell{};
  std::vector<int32_t> h_nb, h_code, h_fv, h_slot;
  std::vector<double> h_bbox;
  // device mesh
  int *d_nb = nullptr, *d_code = nullptr, *d_pat = nullptr;
  int *d_mmask = nullptr;
  double *d_dXbdx = nullptr, *d_bgd = nullptr, *d_bbox = nullptr, *d_basis = nullptr;
  double *d_Pm = nullptr, *d_Rm = nullptr, *d_A = nullptr, *d_ind = nullptr;
  // DG states and guesses
  double *d_ud[4] = {nullptr, nullptr, nullptr, nullptr};
  double *d_pd = nullptr;
  // finite-volume slots
  int nfv = 0, cap = 0;
  double *d_uf[4] = {nullptr, nullptr, nullptr, nullptr};
  double *d_pf = nullptr, *d_rbuf = nullptr, *d_geo = nullptr;
  int *d_slotelem = nullptr, *d_fvslot = nullptr, *d_dglist = nullptr;
  int ndg = 0;
  // DG / finite-volume faces
  int ntr = 0;
  int *d_tslot = nullptr, *d_tface = nullptr;
  double *d_trace = nullptr;
  int cur = 0;
  unsigned long long *d_stats = nullptr;
  cudaGraphExec_t graph[2] = {nullptr, nullptr};
  double graph_dt = 0.;
  int64_t launches = 0, graph_launches = 0;
  size_t smem_dg = 0, smem_fv = 0;
  bool dg_tc = false;  // DG divergence on the tensor cores (n = 7, 8, 9)
};

namespace {

int gset(nmg_grhd_ctx *c, int code, const std::string &msg) {
  if (c) c->err = msg;
  return code;
}

#define GCK(call)                                                                        \
  do {                                                                                   \
    cudaError_t e_ = (call);                                                             \
    if (e_ != cudaSuccess)                                                               \
      return gset(c, NMG_ECUDA, std::string(#call) + ": " + cudaGetErrorString(e_));     \
  } while (0)

template <class T>
int dalloc(nmg_grhd_ctx *c, T **p, size_t count) {
  if (*p) cudaFree(*p);
  *p = nullptr;
  if (count == 0) return NMG_OK;
  if (cudaMalloc((void **)p, count * sizeof(T)) != cudaSuccess) {
    cudaGetLastError();
    return gset(c, NMG_ENOMEM, "nmg_grhd: device allocation failed");
  }
  return NMG_OK;
}

template <class T>
int upload(nmg_grhd_ctx *c, T **p, const std::vector<T> &v) {
  int rc = dalloc(c, p, v.size());
  if (rc || v.empty()) return rc;
  GCK(cudaMemcpyAsync(*p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice, c->stream));
  return NMG_OK;
}

void drop_graphs(nmg_grhd_ctx *c) {
  for (auto &g : c->graph)
    if (g) {
      cudaGraphExecDestroy(g);
      g = nullptr;
    }
}

// LGL -> equally spaced interpolation P (nf x n) and its pseudo-inverse
// R = (P^T P)^-1 P^T (n x nf), in long double (gridpoints.c:158-200 with
// Inverse_InterpMatT_pseudo)
void transfer_matrices(int n, int nf, const std::vector<double> &xl, const std::vector<double> &xu,
                       std::vector<double> &Pm, std::vector<double> &Rm) {
  std::vector<long double> Pl((size_t)nf * n), A((size_t)n * (n + nf));
  Pm.assign((size_t)nf * n, 0.);
  Rm.assign((size_t)n * nf, 0.);
  for (int q = 0; q < nf; q++)
    for (int i = 0; i < n; i++) {
      long double v = 1.L;
      for (int j = 0; j < n; j++)
        if (j != i) v *= ((long double)xu[q] - xl[j]) / ((long double)xl[i] - xl[j]);
      Pl[(size_t)q * n + i] = v;
      Pm[(size_t)q * n + i] = (double)v;
    }
  const int w = n + nf;
  for (int i = 0; i < n; i++) {
    for (int j = 0; j < n; j++) {
      long double s = 0.L;
      for (int q = 0; q < nf; q++) s += Pl[(size_t)q * n + i] * Pl[(size_t)q * n + j];
      A[(size_t)i * w + j] = s;
    }
    for (int q = 0; q < nf; q++) A[(size_t)i * w + n + q] = Pl[(size_t)q * n + i];
  }
  for (int k = 0; k < n; k++) {
    int piv = k;
    for (int i = k + 1; i < n; i++)
      if (fabsl(A[(size_t)i * w + k]) > fabsl(A[(size_t)piv * w + k])) piv = i;
    if (piv != k)
      for (int j = 0; j < w; j++) std::swap(A[(size_t)k * w + j], A[(size_t)piv * w + j]);
    const long double d = A[(size_t)k * w + k];
    for (int j = 0; j < w; j++) A[(size_t)k * w + j] /= d;
    for (int i = 0; i < n; i++)
      if (i != k) {
        const long double f = A[(size_t)i * w + k];
        for (int j = 0; j < w; j++) A[(size_t)i * w + j] -= f * A[(size_t)k * w + j];
      }
  }
  for (int i = 0; i < n; i++)
    for (int q = 0; q < nf; q++) Rm[(size_t)i * nf + q] = (double)A[(size_t)i * w + n + q];
}

// normalised Legendre analysis of n LGL points: A[i][j] = w_j P_i(x_j)
// sqrt(c_i), c_i = (2i+1)/2 and n/2-1/2 ... (N/2 for the top mode), as the
// reference's LGL_AT_ST_matrices (src/main/basis/Legendre.c:277-310)
std::vector<double> analysis_matrix(const std::vector<double> &x, const std::vector<double> &w) {
  const int n = (int)x.size(), N = n - 1;
  std::vector<double> A((size_t)n * n);
  for (int i = 0; i < n; i++) {
    double ooci = 0.5 * (2 * i + 1);
    if (i == N && N != 0) ooci = 0.5 * i;
    const double oosci = std::sqrt(ooci);
    for (int j = 0; j < n; j++) {
      double Pk = 0., P0 = 1.0, P1 = x[j], Pi;
      if (i == 0) Pi = P0;
      else if (i == 1) Pi = P1;
      else {
        for (int k = 2; k <= i; k++) {
          Pk = (x[j] * (2 * k - 1) * P1 - (k - 1) * P0) / k;
          P0 = P1;
          P1 = Pk;
        }
        Pi = Pk;
      }
      A[(size_t)i * n + j] = w[j] * (Pi * oosci);
    }
  }
  return A;
}

GrP base_params(nmg_grhd_ctx *c) {
  GrP P;
  std::memset(&P, 0, sizeof(P));
  P.n = c->n; P.np = c->np; P.nn = c->nn;
  P.nf = c->nf; P.npf = c->npf; P.nnf = c->nnf; P.tpts = c->tpts;
  P.ndg = c->ndg; P.nfv = c->nfv;
  P.g = c->prm.eos;
  P.eos.gamma = c->prm.eos.gamma;
  P.eos.hfac = c->prm.eos.gamma / (c->prm.eos.gamma - 1.);
  {
    const nmg_grhd_params &g = c->prm.eos;
    const double eps = g.p_atm / ((g.gamma - 1.) * g.rho_atm);
    P.eos.tau_atm = g.rho_atm * (1. + eps + g.p_atm / g.rho_atm) - g.p_atm;
  }
  P.mass = c->prm.mass;
  P.rec = c->prm.rec;
  P.dglist = c->d_dglist; P.slotelem = c->d_slotelem; P.fvslot = c->d_fvslot;
  P.nb = c->d_nb; P.code = c->d_code; P.tslot = c->d_tslot; P.tface = c->d_tface;
  P.ntr = c->ntr;
  P.dXbdx = c->d_dXbdx; P.mmask = c->d_mmask; P.bgd = c->d_bgd; P.bbox = c->d_bbox; P.basis = c->d_basis;
  P.geo = c->d_geo; P.trace = c->d_trace; P.rbuf = c->d_rbuf;
  return P;
}

int grid_for(int64_t work) {
  return (int)std::max<int64_t>(1, std::min<int64_t>((work + kNT - 1) / kNT, 152 * 16));
}

// one stage: con2prim of the input (in place), traces, DG and FV kernels;
// with ev (8 events), each kernel class is bracketed by a pair of events
int enqueue_stage(nmg_grhd_ctx *c, GrP P, double *win_d, double *win_f,
                  cudaEvent_t *ev = nullptr) {
  P.win_d = win_d;
  P.win_f = win_f;
  P.prim_d = c->d_pd;
  P.prim_f = c->d_pf;
  auto mark = [&](int k) {
    if (ev) cudaEventRecord(ev[k], c->stream);
  };
  const int64_t work = (int64_t)c->ndg * c->np + (int64_t)c->nfv * c->npf;
  mark(0);
  if (work > 0) {
    c2p_kernel<<<grid_for(work), kNT, 0, c->stream>>>(P, win_d, win_f, c->d_pd, c->d_pf,
                                                      c->d_stats);
    GCK(cudaGetLastError());
    c->launches++;
  }
  mark(1);
  mark(2);
  if (c->ntr > 0) {
    trace_kernel<<<c->ntr, kNTT, 0, c->stream>>>(P, c->d_Pm, c->d_pd, c->d_pf);
    GCK(cudaGetLastError());
    c->launches++;
  }
  mark(3);
  // the finite-volume and the DG elements side by side: each reads what con2prim and
  // the traces wrote and writes its own (383 elements at n = 5: a stage 216 -> 199 us;
  // 10368 at n = 7, where either fills the chip, 1 %)
  const bool beside = !ev && c->ndg > 0 && c->nfv > 0;
  cudaStream_t fs = beside ? c->fv_stream : c->stream;
  if (beside) {
    GCK(cudaEventRecord(c->fork_ev, c->stream));
    GCK(cudaStreamWaitEvent(fs, c->fork_ev, 0));
  }
  mark(6);
  if (c->nfv > 0) {
    const int grid = 3 * c->nf * c->nfv;
    const int nt = fv_threads(c->nf);
    if (nt <= 192) fv_flux_kernel<192, 4><<<grid, nt, c->smem_fv, fs>>>(P);
    else fv_flux_kernel<288, 2><<<grid, nt, c->smem_fv, fs>>>(P);
    GCK(cudaGetLastError());
    fv_update_kernel<<<grid_for((int64_t)c->nfv * c->npf), kNT, 0, fs>>>(P);
    GCK(cudaGetLastError());
    c->launches += 2;
  }
  mark(7);
  mark(4);
  if (c->ndg > 0) {
    if (!c->dg_tc)
      dg_kernel<<<c->ndg, kNT, c->smem_dg, c->stream>>>(P);
    else if (c->n == 7)
      dg_tc_kernel<7><<<c->ndg, dg_tc_threads<7>(), dg_tc_smem<7>(), c->stream>>>(P);
    else if (c->n == 8)
      dg_tc_kernel<8><<<c->ndg, dg_tc_threads<8>(), dg_tc_smem<8>(), c->stream>>>(P);
    else
      dg_tc_kernel<9><<<c->ndg, dg_tc_threads<9>(), dg_tc_smem<9>(), c->stream>>>(P);
    GCK(cudaGetLastError());
    c->launches++;
  }
  mark(5);
  if (beside) {
    GCK(cudaEventRecord(c->join_ev, fs));
    GCK(cudaStreamWaitEvent(c->stream, c->join_ev, 0));
  }
  return NMG_OK;
}

// one RK4 step of the state in buffer cur (the result goes to 1 - cur);
// with ms, the step runs stage by stage and ms[k] accumulates the time of
// kernel class k (con2prim, traces, DG, finite volume)
int enqueue_step(nmg_grhd_ctx *c, int cur, double dt, double *ms = nullptr) {
  cudaEvent_t ev[8];
  if (ms)
    for (int k = 0; k < 8; k++) GCK(cudaEventCreate(&ev[k]));
  double *Ud = c->d_ud[cur], *Ad = c->d_ud[1 - cur], *WAd = c->d_ud[2], *WBd = c->d_ud[3];
  double *Uf = c->d_uf[cur], *Af = c->d_uf[1 - cur], *WAf = c->d_uf[2], *WBf = c->d_uf[3];
  const double cacc[4] = {dt / 6., dt / 3., dt / 3., dt / 6.};
  const double cw[4] = {dt / 2., dt / 2., dt, 0.};
  double *wind[4] = {Ud, WAd, WBd, WAd}, *winf[4] = {Uf, WAf, WBf, WAf};
  double *woutd[4] = {WAd, WBd, WAd, nullptr}, *woutf[4] = {WAf, WBf, WAf, nullptr};
  for (int s = 0; s < 4; s++) {
    GrP P = base_params(c);
    P.u0_d = Ud; P.u0_f = Uf;
    P.acc_d = Ad; P.acc_f = Af;
    P.wout_d = woutd[s]; P.wout_f = woutf[s];
    P.mode = s + 1;
    P.cacc = cacc[s];
    P.cw = cw[s];
    int rc = enqueue_stage(c, P, wind[s], winf[s], ms ? ev : nullptr);
    if (rc) return rc;
    if (ms) {
      GCK(cudaStreamSynchronize(c->stream));
      for (int k = 0; k < 4; k++) {
        float t = 0.f;
        GCK(cudaEventElapsedTime(&t, ev[2 * k], ev[2 * k + 1]));
        ms[k] += t;
      }
    }
  }
  if (ms)
    for (int k = 0; k < 8; k++) cudaEventDestroy(ev[k]);
  return NMG_OK;
}

// the element types: slots, lists, traces (host tables to the device)
int upload_types(nmg_grhd_ctx *c) {
  const int64_t E = c->E;
  std::vector<int> dgl, slotelem, fvslot(E, -1), tslot(E * 6, -1), tface;
  for (int64_t e = 0; e < E; e++) {
    if (c->h_fv[e]) {
      fvslot[e] = (int)slotelem.size();
      slotelem.push_back((int)e);
    } else {
      dgl.push_back((int)e);
    }
  }
  for (int64_t e = 0; e < E; e++)
    for (int f = 0; f < 6; f++) {
      const int e2 = c->h_nb[e * 6 + f];
      if (e2 >= 0 && (c->h_fv[e] != 0) != (c->h_fv[e2] != 0)) {
        tslot[e * 6 + f] = (int)(tface.size() / 2);
        tface.push_back((int)e);
        tface.push_back(f);
      }
    }
  c->ndg = (int)dgl.size();
  c->nfv = (int)slotelem.size();
  c->ntr = (int)(tface.size() / 2);
  c->h_slot = fvslot;
  int rc;
  if ((rc = upload(c, &c->d_dglist, dgl)) || (rc = upload(c, &c->d_slotelem, slotelem)) ||
      (rc = upload(c, &c->d_fvslot, fvslot)) || (rc = upload(c, &c->d_tslot, tslot)) ||
      (rc = upload(c, &c->d_tface, tface)))
    return rc;
  return dalloc(c, &c->d_trace, (size_t)c->ntr * NF * c->tpts);
}

}  // namespace

extern "C" {

int nmg_grhd_create(const nmg_mesh *m, const nmg_grhd_evolve_params *p, nmg_grhd_ctx **out) {
  if (!m || !p || !out) return NMG_EINVAL;
  *out = nullptr;
  nmg_grhd_ctx *c = new (std::nothrow) nmg_grhd_ctx;
  if (!c) return NMG_ENOMEM;
  *out = c;
  c->prm = *p;
  const nmg_grhd_params &g = p->eos;
  if (!(g.gamma > 1.) || !(g.rho_atm > 0.) || !(g.p_atm > 0.) || !(g.tol > 0.) || g.maxits <= 0 ||
      g.maxits > 100000 || !(p->mass >= 0.))
    return gset(c, NMG_EINVAL, "nmg_grhd_create: bad physical parameters");
  if (p->rec < NMG_FV_REC_1 || p->rec > NMG_FV_REC_WENOMZ_2)
    return gset(c, NMG_EINVAL, "nmg_grhd_create: unknown reconstruction");
  if (m->patches.size() != 6)
    return gset(c, NMG_EUNSUP, "nmg_grhd_create: the mesh must be NMG_MESH_CUBEDSHELL6");
  for (int q = 0; q < 6; q++) {
    const nmg::Patch &P = m->patches[q];
    if (!P.cubed || !P.shell) return gset(c, NMG_EUNSUP, "nmg_grhd_create: not a cubed shell");
    c->shell.dom[q] = P.dom;
    c->shell.s0[q] = P.s0;
    c->shell.s1[q] = P.s1;
  }
  for (int d = 0; d < 3; d++) c->shell.xc[d] = m->patches[0].xc[d];
  if (!m->fv.empty()) return gset(c, NMG_EUNSUP, "nmg_grhd_create: DG mesh expected");
  c->n = m->n;
  c->nf = p->nf > 0 ? p->nf : 2 * m->n;
  if (c->n < 3 || c->n > kMaxN)
    return gset(c, NMG_EUNSUP, "nmg_grhd_create: n must be in [3,10]");
  if (c->nf < 4 || c->nf > kMaxNF)
    return gset(c, NMG_EUNSUP, "nmg_grhd_create: nf must be in [4,16]");
  c->np = c->n * c->n * c->n;
  c->nn = c->n * c->n;
  c->npf = c->nf * c->nf * c->nf;
  c->nnf = c->nf * c->nf;
  c->tpts = std::max(c->nn, c->nnf);
  c->E = m->nelem;
  cudaError_t ce = cudaGetDevice(&c->device);
  if (ce != cudaSuccess) return gset(c, NMG_ECUDA, cudaGetErrorString(ce));
  GCK(cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking));
  GCK(cudaStreamCreateWithFlags(&c->fv_stream, cudaStreamNonBlocking));
  GCK(cudaEventCreateWithFlags(&c->fork_ev, cudaEventDisableTiming));
  GCK(cudaEventCreateWithFlags(&c->join_ev, cudaEventDisableTiming));
  // shared memory of the kernels
  c->smem_dg = sizeof(double) * ((size_t)20 * c->np + c->nn);
  c->smem_fv = fv_smem(c->nf);
  int optin = 0;
  GCK(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, c->device));
  if (c->smem_fv > (size_t)optin || c->smem_dg > (size_t)optin)
    return gset(c, NMG_EUNSUP, "nmg_grhd_create: element too large for shared memory");
  GCK(cudaFuncSetAttribute(dg_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)c->smem_dg));
  GCK(cudaFuncSetAttribute(fv_flux_kernel<192, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)c->smem_fv));
  GCK(cudaFuncSetAttribute(fv_flux_kernel<288, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)c->smem_fv));
  // the tensor-core DG kernel at n = 7, 8, 9 (NMG_GRHD_DG=fp64 keeps the FP64 one)
  {
    const char *ev = std::getenv("NMG_GRHD_DG");
    c->dg_tc = c->n >= 7 && c->n <= 9 && !(ev && std::strcmp(ev, "fp64") == 0);
  }
  if (c->dg_tc) {
    GCK(nmgk::tc_upload_tables(c->n, m->D.data(), false));
    if (c->n == 7)
      GCK(cudaFuncSetAttribute(dg_tc_kernel<7>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)dg_tc_smem<7>()));
    else if (c->n == 8)
      GCK(cudaFuncSetAttribute(dg_tc_kernel<8>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)dg_tc_smem<8>()));
    else
      GCK(cudaFuncSetAttribute(dg_tc_kernel<9>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)dg_tc_smem<9>()));
  }
  // mesh tables
  const int64_t E = c->E;
  c->h_nb.assign(m->nb.begin(), m->nb.end());
  c->h_code.resize(E * 6);
  for (int64_t i = 0; i < E * 6; i++) c->h_code[i] = m->code[i] & 63;
  c->h_bbox = m->bbox;
  c->h_fv.assign(E, 0);
  std::vector<double> bgd((size_t)E * 8 * c->np);
  for (int64_t e = 0; e < E; e++)
    for (int q = 0; q < c->np; q++) {
      double x[3], b[8];
      for (int d = 0; d < 3; d++) x[d] = m->xyz[((size_t)e * 3 + d) * c->np + q];
      background(p->mass, x, b);
      for (int k = 0; k < 8; k++) bgd[((size_t)e * 8 + k) * c->np + q] = b[k];
    }
  std::vector<double> basis;
  basis.insert(basis.end(), m->D.begin(), m->D.end());
  basis.insert(basis.end(), m->w.begin(), m->w.end());
  basis.insert(basis.end(), m->x.begin(), m->x.end());
  std::vector<double> xu(c->nf);
  {
    std::vector<double> wu(c->nf), Du((size_t)c->nf * c->nf);
    nmg::uniform_basis(c->nf, xu.data(), wu.data(), Du.data());
  }
  basis.insert(basis.end(), xu.begin(), xu.end());
  std::vector<double> Pm, Rm;
  transfer_matrices(c->n, c->nf, m->x, xu, Pm, Rm);
  int rc;
  if ((rc = upload(c, &c->d_nb, c->h_nb)) || (rc = upload(c, &c->d_code, c->h_code)) ||
      (rc = upload(c, &c->d_pat, m->pat)) || (rc = upload(c, &c->d_dXbdx, m->dXdx)) || (rc = dalloc(c, &c->d_mmask, (size_t)E)) ||
      (rc = upload(c, &c->d_bgd, bgd)) || (rc = upload(c, &c->d_bbox, m->bbox)) ||
      (rc = upload(c, &c->d_basis, basis)) || (rc = upload(c, &c->d_Pm, Pm)) ||
      (rc = upload(c, &c->d_Rm, Rm)) || (rc = upload(c, &c->d_A, analysis_matrix(m->x, m->w))) ||
      (rc = dalloc(c, &c->d_ind, (size_t)m->nelem)))
    return rc;
  metric_kernel<<<(unsigned)E, kNT, 0, c->stream>>>(c->np, c->d_bbox, c->d_dXbdx, c->d_mmask);
  GCK(cudaGetLastError());
  const size_t ld = (size_t)E * NF * c->np;
  for (int b = 0; b < 4; b++)
    if ((rc = dalloc(c, &c->d_ud[b], ld))) return rc;
  if ((rc = dalloc(c, &c->d_pd, ld)) || (rc = dalloc(c, &c->d_stats, 2))) return rc;
  GCK(cudaMemsetAsync(c->d_ud[0], 0, ld * sizeof(double), c->stream));
  GCK(cudaMemsetAsync(c->d_pd, 0, ld * sizeof(double), c->stream));
  GCK(cudaMemsetAsync(c->d_stats, 0, 2 * sizeof(unsigned long long), c->stream));
  if ((rc = upload_types(c))) return rc;
  GCK(cudaStreamSynchronize(c->stream));
  return NMG_OK;
}

void nmg_grhd_destroy(nmg_grhd_ctx *c) {
  if (!c) return;
  drop_graphs(c);
  if (c->stream) cudaStreamSynchronize(c->stream);
  void *ptrs[] = {c->d_nb, c->d_code, c->d_pat, c->d_mmask, c->d_dXbdx, c->d_bgd, c->d_bbox, c->d_basis,
                  c->d_Pm, c->d_Rm, c->d_A, c->d_ind, c->d_ud[0], c->d_ud[1], c->d_ud[2], c->d_ud[3], c->d_pd,
                  c->d_uf[0], c->d_uf[1], c->d_uf[2], c->d_uf[3], c->d_pf, c->d_rbuf, c->d_geo,
                  c->d_slotelem, c->d_fvslot, c->d_dglist, c->d_tslot, c->d_tface, c->d_trace,
                  c->d_stats};
  for (void *p : ptrs)
    if (p) cudaFree(p);
  if (c->fork_ev) cudaEventDestroy(c->fork_ev);
  if (c->join_ev) cudaEventDestroy(c->join_ev);
  if (c->fv_stream) cudaStreamDestroy(c->fv_stream);
  if (c->stream) cudaStreamDestroy(c->stream);
  delete c;
}

const char *nmg_grhd_last_error(const nmg_grhd_ctx *c) { return c ? c->err.c_str() : "null context"; }

int64_t nmg_grhd_fv_count(const nmg_grhd_ctx *c) { return c ? c->nfv : -1; }

int nmg_grhd_sizes(const nmg_grhd_ctx *c, int32_t *n, int32_t *nf, int64_t *nelem) {
  if (!c) return NMG_EINVAL;
  if (n) *n = c->n;
  if (nf) *nf = c->nf;
  if (nelem) *nelem = c->E;
  return NMG_OK;
}

int nmg_grhd_set_fv_elements(nmg_grhd_ctx *c, const int32_t *fv) {
  if (!c || !fv) return gset(c, NMG_EINVAL, "nmg_grhd_set_fv_elements: null argument");
  const int64_t E = c->E;
  std::vector<int32_t> nfv(E);
  for (int64_t e = 0; e < E; e++) nfv[e] = fv[e] ? 1 : 0;
  if (nfv == c->h_fv) return NMG_OK;
  // new slots: ascending elements
  std::vector<int> old_slot = c->h_slot, new_slot(E, -1);
  int count = 0;
  for (int64_t e = 0; e < E; e++)
    if (nfv[e]) new_slot[e] = count++;
  std::vector<int> keep_src, keep_dst, tofv_e, tofv_s, todg_s, todg_e;
  for (int64_t e = 0; e < E; e++) {
    if (nfv[e] && c->h_fv[e]) {
      keep_src.push_back(old_slot[e]);
      keep_dst.push_back(new_slot[e]);
    } else if (nfv[e]) {
      tofv_e.push_back((int)e);
      tofv_s.push_back(new_slot[e]);
    } else if (c->h_fv[e]) {
      todg_s.push_back(old_slot[e]);
      todg_e.push_back((int)e);
    }
  }
  const size_t lf = (size_t)count * NF * c->npf;
  double *nu = nullptr, *np_ = nullptr;
  int rc;
  if ((rc = dalloc(c, &nu, lf)) || (rc = dalloc(c, &np_, lf))) return rc;
  int *d_lists = nullptr;
  std::vector<int> all;
  auto put = [&](const std::vector<int> &v) {
    const size_t off = all.size();
    all.insert(all.end(), v.begin(), v.end());
    return off;
  };
  const size_t o_ks = put(keep_src), o_kd = put(keep_dst), o_fe = put(tofv_e), o_fs = put(tofv_s),
               o_ds = put(todg_s), o_de = put(todg_e);
  if ((rc = upload(c, &d_lists, all))) return rc;
  double *U = c->d_ud[c->cur], *Uf = c->d_uf[c->cur];
  if (!keep_src.empty()) {
    dim3 grid(8, (unsigned)keep_src.size());
    copy_rows_kernel<<<grid, kNT, 0, c->stream>>>((int64_t)NF * c->npf, d_lists + o_ks,
                                                  d_lists + o_kd, Uf, nu);
    copy_rows_kernel<<<grid, kNT, 0, c->stream>>>((int64_t)NF * c->npf, d_lists + o_ks,
                                                  d_lists + o_kd, c->d_pf, np_);
    GCK(cudaGetLastError());
  }
  const size_t sm_to = sizeof(double) * ((size_t)c->np + (size_t)c->nf * c->nn +
                                         (size_t)c->nf * c->nf * c->n + (size_t)c->nf * c->n);
  const size_t sm_back = sizeof(double) * ((size_t)c->npf + (size_t)c->n * c->nnf +
                                           (size_t)c->n * c->n * c->nf + (size_t)c->nf * c->n);
  GCK(cudaFuncSetAttribute(convert_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)std::max(sm_to, sm_back)));
  if (!tofv_e.empty()) {
    convert_kernel<<<(unsigned)tofv_e.size(), kNT, sm_to, c->stream>>>(
        c->d_Pm, c->n, c->nf, d_lists + o_fe, d_lists + o_fs, U, nu);
    convert_kernel<<<(unsigned)tofv_e.size(), kNT, sm_to, c->stream>>>(
        c->d_Pm, c->n, c->nf, d_lists + o_fe, d_lists + o_fs, c->d_pd, np_);
    GCK(cudaGetLastError());
  }
  if (!todg_s.empty()) {
    convert_kernel<<<(unsigned)todg_s.size(), kNT, sm_back, c->stream>>>(
        c->d_Rm, c->nf, c->n, d_lists + o_ds, d_lists + o_de, Uf, U);
    convert_kernel<<<(unsigned)todg_s.size(), kNT, sm_back, c->stream>>>(
        c->d_Rm, c->nf, c->n, d_lists + o_ds, d_lists + o_de, c->d_pf, c->d_pd);
    GCK(cudaGetLastError());
  }
  GCK(cudaStreamSynchronize(c->stream));
  cudaFree(d_lists);
  // swap in the new slot arrays
  for (int b = 0; b < 4; b++) {
    if (c->d_uf[b]) cudaFree(c->d_uf[b]);
    c->d_uf[b] = nullptr;
  }
  if (c->d_pf) cudaFree(c->d_pf);
  c->d_uf[c->cur] = nu;
  c->d_pf = np_;
  for (int b = 0; b < 4; b++)
    if (b != c->cur && (rc = dalloc(c, &c->d_uf[b], lf))) return rc;
  if ((rc = dalloc(c, &c->d_rbuf, 3 * lf)) || (rc = dalloc(c, &c->d_geo, (size_t)count * kGeo * c->npf)))
    return rc;
  c->h_fv = nfv;
  if ((rc = upload_types(c))) return rc;
  if (c->nfv > 0) {
    GrP P = base_params(c);
    fvgeo_kernel<<<grid_for((int64_t)c->nfv * c->npf), kNT, 0, c->stream>>>(P, c->shell, c->d_pat,
                                                                          c->d_geo);
    GCK(cudaGetLastError());
  }
  GCK(cudaStreamSynchronize(c->stream));
  drop_graphs(c);
  return NMG_OK;
}

int nmg_grhd_trouble_indicators(nmg_grhd_ctx *c, double *ind) {
  if (!c || !ind) return gset(c, NMG_EINVAL, "nmg_grhd_trouble_indicators: null argument");
  const int n = c->n, nf = c->nf, np = c->np;
  const size_t smem = sizeof(double) * ((size_t)std::max(np, c->npf) +
                                        std::max(n * nf * nf, np) + std::max(n * n * nf, np) + np);
  GCK(cudaFuncSetAttribute(persson_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  GrP P = base_params(c);
  persson_kernel<<<(unsigned)c->E, kNT, smem, c->stream>>>(P, c->d_ud[c->cur], c->d_uf[c->cur],
                                                          c->d_A, c->d_Rm, c->d_ind);
  GCK(cudaGetLastError());
  GCK(cudaMemcpyAsync(ind, c->d_ind, sizeof(double) * c->E, cudaMemcpyDeviceToHost, c->stream));
  GCK(cudaStreamSynchronize(c->stream));
  return NMG_OK;
}

int nmg_grhd_update_troubled(nmg_grhd_ctx *c, double persson_max, double back_margin,
                             int32_t *switched) {
  if (!c || !(back_margin >= 0.))
    return gset(c, NMG_EINVAL, "nmg_grhd_update_troubled: bad argument");
  std::vector<double> ind(c->E);
  int rc = nmg_grhd_trouble_indicators(c, ind.data());
  if (rc) return rc;
  std::vector<int32_t> fv = c->h_fv;
  int to_fv = 0, to_dg = 0;
  for (int64_t e = 0; e < c->E; e++) {
    if (!fv[e] && ind[e] > persson_max) {
      fv[e] = 1;
      to_fv++;
    } else if (fv[e] && ind[e] < persson_max - back_margin) {
      fv[e] = 0;
      to_dg++;
    }
  }
  if (switched) {
    switched[0] = to_fv;
    switched[1] = to_dg;
  }
  return (to_fv || to_dg) ? nmg_grhd_set_fv_elements(c, fv.data()) : NMG_OK;
}

int nmg_grhd_get_fv_elements(nmg_grhd_ctx *c, int32_t *fv) {
  if (!c || !fv) return gset(c, NMG_EINVAL, "nmg_grhd_get_fv_elements: null argument");
  std::memcpy(fv, c->h_fv.data(), sizeof(int32_t) * c->E);
  return NMG_OK;
}

// host layouts: DG [E][5][n^3] (rows of finite-volume elements ignored or
// zero), finite volume [nfv][5][nf^3] in ascending element order
int nmg_grhd_set_prim(nmg_grhd_ctx *c, const double *prim_dg, const double *prim_fv) {
  if (!c || !prim_dg || (c->nfv > 0 && !prim_fv))
    return gset(c, NMG_EINVAL, "nmg_grhd_set_prim: null argument");
  const size_t ld = (size_t)c->E * NF * c->np, lf = (size_t)c->nfv * NF * c->npf;
  GCK(cudaMemcpyAsync(c->d_pd, prim_dg, ld * sizeof(double), cudaMemcpyHostToDevice, c->stream));
  p2c_kernel<<<grid_for((int64_t)c->E * c->np), kNT, 0, c->stream>>>(
      c->prm.eos, c->E, c->np, c->d_bgd + c->np, 8 * c->np, nullptr, c->d_pd, c->d_ud[c->cur]);
  GCK(cudaGetLastError());
  if (lf) {
    GCK(cudaMemcpyAsync(c->d_pf, prim_fv, lf * sizeof(double), cudaMemcpyHostToDevice, c->stream));
    p2c_kernel<<<grid_for((int64_t)c->nfv * c->npf), kNT, 0, c->stream>>>(
        c->prm.eos, c->nfv, c->npf, c->d_geo + 2 * c->npf, kGeo * c->npf, nullptr, c->d_pf,
        c->d_uf[c->cur]);
    GCK(cudaGetLastError());
  }
  GCK(cudaStreamSynchronize(c->stream));
  return NMG_OK;
}

int nmg_grhd_set_state(nmg_grhd_ctx *c, const double *u_dg, const double *u_fv,
                       const double *prim_dg, const double *prim_fv) {
  if (!c || !u_dg || (c->nfv > 0 && !u_fv))
    return gset(c, NMG_EINVAL, "nmg_grhd_set_state: null argument");
  const size_t ld = (size_t)c->E * NF * c->np, lf = (size_t)c->nfv * NF * c->npf;
  GCK(cudaMemcpyAsync(c->d_ud[c->cur], u_dg, ld * sizeof(double), cudaMemcpyHostToDevice,
                      c->stream));
  if (prim_dg)
    GCK(cudaMemcpyAsync(c->d_pd, prim_dg, ld * sizeof(double), cudaMemcpyHostToDevice, c->stream));
  if (lf) {
    GCK(cudaMemcpyAsync(c->d_uf[c->cur], u_fv, lf * sizeof(double), cudaMemcpyHostToDevice,
                        c->stream));
    if (prim_fv)
      GCK(cudaMemcpyAsync(c->d_pf, prim_fv, lf * sizeof(double), cudaMemcpyHostToDevice,
                          c->stream));
  }
  GCK(cudaStreamSynchronize(c->stream));
  return NMG_OK;
}

int nmg_grhd_get_state(nmg_grhd_ctx *c, double *u_dg, double *u_fv, double *prim_dg,
                       double *prim_fv) {
  if (!c) return NMG_EINVAL;
  const size_t ld = (size_t)c->E * NF * c->np, lf = (size_t)c->nfv * NF * c->npf;
  if (u_dg)
    GCK(cudaMemcpyAsync(u_dg, c->d_ud[c->cur], ld * sizeof(double), cudaMemcpyDeviceToHost,
                        c->stream));
  if (prim_dg)
    GCK(cudaMemcpyAsync(prim_dg, c->d_pd, ld * sizeof(double), cudaMemcpyDeviceToHost, c->stream));
  if (lf && u_fv)
    GCK(cudaMemcpyAsync(u_fv, c->d_uf[c->cur], lf * sizeof(double), cudaMemcpyDeviceToHost,
                        c->stream));
  if (lf && prim_fv)
    GCK(cudaMemcpyAsync(prim_fv, c->d_pf, lf * sizeof(double), cudaMemcpyDeviceToHost, c->stream));
  GCK(cudaStreamSynchronize(c->stream));
  return NMG_OK;
}

// r = RHS of the resident state after its con2prim (which, as in the first
// stage of a step, may reset atmosphere points of the state in place)
int nmg_grhd_rhs(nmg_grhd_ctx *c, double *r_dg, double *r_fv) {
  if (!c || !r_dg) return gset(c, NMG_EINVAL, "nmg_grhd_rhs: null argument");
  GrP P = base_params(c);
  P.acc_d = c->d_ud[1 - c->cur];
  P.acc_f = c->d_uf[1 - c->cur];
  P.mode = 0;
  int rc = enqueue_stage(c, P, c->d_ud[c->cur], c->d_uf[c->cur]);
  if (rc) return rc;
  const size_t ld = (size_t)c->E * NF * c->np, lf = (size_t)c->nfv * NF * c->npf;
  GCK(cudaMemcpyAsync(r_dg, c->d_ud[1 - c->cur], ld * sizeof(double), cudaMemcpyDeviceToHost,
                      c->stream));
  if (lf && r_fv)
    GCK(cudaMemcpyAsync(r_fv, c->d_uf[1 - c->cur], lf * sizeof(double), cudaMemcpyDeviceToHost,
                        c->stream));
  GCK(cudaStreamSynchronize(c->stream));
  return NMG_OK;
}

int nmg_grhd_rk4_steps(nmg_grhd_ctx *c, double dt, int32_t nsteps) {
  if (!c || nsteps < 0 || !(dt > 0.)) return gset(c, NMG_EINVAL, "nmg_grhd_rk4_steps: bad argument");
  if (nsteps == 0) return NMG_OK;
  if (dt != c->graph_dt) {
    drop_graphs(c);
    c->graph_dt = dt;
  }
  for (int g = 0; g < 2; g++) {
    if (c->graph[g]) continue;
    cudaGraph_t gr;
    GCK(cudaStreamBeginCapture(c->stream, cudaStreamCaptureModeThreadLocal));
    const int64_t l0 = c->launches;
    int rc = enqueue_step(c, g, dt);
    cudaGraph_t tmp = nullptr;
    cudaError_t e2 = cudaStreamEndCapture(c->stream, &tmp);
    gr = tmp;
    c->graph_launches = c->launches - l0;
    c->launches = l0;
    if (rc) {
      if (gr) cudaGraphDestroy(gr);
      return rc;
    }
    GCK(e2);
    cudaError_t e3 = cudaGraphInstantiate(&c->graph[g], gr, 0);
    cudaGraphDestroy(gr);
    GCK(e3);
  }
  for (int s = 0; s < nsteps; s++) {
    GCK(cudaGraphLaunch(c->graph[c->cur], c->stream));
    c->launches += c->graph_launches;
    c->cur = 1 - c->cur;
  }
  GCK(cudaStreamSynchronize(c->stream));
  return NMG_OK;
}

int nmg_grhd_profile_step(nmg_grhd_ctx *c, double dt, double *ms) {
  if (!c || !ms || !(dt > 0.)) return gset(c, NMG_EINVAL, "nmg_grhd_profile_step: bad argument");
  for (int k = 0; k < 4; k++) ms[k] = 0.;
  int rc = enqueue_step(c, c->cur, dt, ms);
  if (rc) return rc;
  c->cur = 1 - c->cur;
  GCK(cudaStreamSynchronize(c->stream));
  return NMG_OK;
}

int nmg_grhd_stats(nmg_grhd_ctx *c, int64_t *c2p_iterations, int64_t *atmosphere_points,
                   int64_t *launches) {
  if (!c) return NMG_EINVAL;
  unsigned long long h[2] = {0, 0};
  GCK(cudaMemcpyAsync(h, c->d_stats, sizeof(h), cudaMemcpyDeviceToHost, c->stream));
  GCK(cudaStreamSynchronize(c->stream));
  if (c2p_iterations) *c2p_iterations = (int64_t)h[0];
  if (atmosphere_points) *atmosphere_points = (int64_t)h[1];
  if (launches) *launches = c->launches;
  return NMG_OK;
}

int nmg_grhd_reset_stats(nmg_grhd_ctx *c) {
  if (!c) return NMG_EINVAL;
  GCK(cudaMemsetAsync(c->d_stats, 0, 2 * sizeof(unsigned long long), c->stream));
  GCK(cudaStreamSynchronize(c->stream));
  return NMG_OK;
}

void *nmg_grhd_stream(nmg_grhd_ctx *c) { return c ? (void *)c->stream : nullptr; }

}  // extern "C"
