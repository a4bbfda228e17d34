// stage_fvc.cu -- "fvc": the finite-volume RHS and RK stage of stage_fv.cu
// (whose header names the reference's routines) with the fewest FP64
// instructions, for the path that the FP64 pipe bounds.
//
// * One CTA per (element, direction, group of planes of pencils): (1) both
//   face values of every cell and field (weno_cell.cuh), the cells walked by
//   stencil class so that warps do not diverge, (2) per midpoint the flux times
//   J sqrtgdiag, and in the tasks after those the fluxes through the pencils'
//   ends, (3) per point the conservative difference, written to the direction's
//   part of a scratch array.  A second kernel adds the three directions and does
//   the stage update.  The planes of a CTA want 17 to 70 KB of shared memory
//   instead of an element's 230 KB, so that several CTAs share an SM (their
//   phases overlap, barriers cost little) and small meshes fill the chip.
// * The scratch (96 bytes a point) is bounded: larger meshes run in groups of
//   elements, which also keeps it within a few L2 sizes.
// * 1/J, 1/dX are multiplied by instead of divided by; in Cartesian elements, where
//   J sqrtgdiag 1/J is the scale of the direction, that alone.  The LLF and the upwind
//   flux are written out for the wave's characteristics (pi -+ c.n, speeds +-1;
//   the matrix products of scalarwave1_numflux1d_upwind reduce to that).  Error of the
//   right-hand side against 64 bits, mean of 12 states, 8 and 56 (64 and 448) elements, with
//   divisions and here: boxes n = 5 3.5e-16, 3.5e-16 (6.7, 6.4), n = 9 6.0, 4.9 (11.8, 9.3);
//   cubed spheres n = 5 7.35, 7.24 (14.9, 14.8), n = 9 13.8, 13.3 (26.3, 25.8).
//
// FP64 pipe 86 % busy (tex_throttle, short scoreboard: its queue); 7 x 8^3
// elements at n = 13, WENOm5_2: 10.45 ms a stage with 256 threads (10.86 with 128,
// 11.1 with 512), where one CTA an element with per-cell face values took
// 19.2 ms and stage_fv.cu's "fv" 22.2; 1536 elements at n = 7, WENOmZ_2: 1.17 -> 0.67 ms.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "stage.cuh"
#include "weno_cell.cuh"

namespace nmgk {
namespace {

constexpr int kGeo = 13;  // per-node geometry of curvilinear elements (stage_fv.cu)

// planes of pencils per CTA of nt threads: about one cell per thread, evenly
__host__ __device__ __forceinline__ int fvc_planes(int n, int nt) {
  int p = (nt + n * n - 1) / (n * n);
  p = p < 1 ? 1 : (p > n ? n : p);
  const int groups = (n + p - 1) / p;
  return (n + groups - 1) / groups;
}

__host__ __device__ __forceinline__ size_t fvc_smem(int n, int nt) {
  const size_t pen = (size_t)fvc_planes(n, nt) * n;
  return sizeof(double) * (12 * pen * n + 4 * pen * (n + 1) + n);
}

// numerical flux of (pi, c) along the unit normal nr
__device__ __forceinline__ void flux4(int kind, const double *ui, const double *ua,
                                      const double nr[3], double *fn) {
  const double s0 = ui[0] + ua[0], d0 = ua[0] - ui[0];
  if (kind == NMG_NUMFLUX_UPWIND) {
    const double ci = fma(ui[1], nr[0], fma(ui[2], nr[1], ui[3] * nr[2]));
    const double ca = fma(ua[1], nr[0], fma(ua[2], nr[1], ua[3] * nr[2]));
    const double h = -0.5 * (s0 + (ca - ci));
    fn[0] = -0.5 * ((ci + ca) + d0);
    fn[1] = h * nr[0];
    fn[2] = h * nr[1];
    fn[3] = h * nr[2];
  } else {
    const double c = fma(ui[1] + ua[1], nr[0],
                         fma(ui[2] + ua[2], nr[1], (ui[3] + ua[3]) * nr[2]));
    fn[0] = -0.5 * (c + d0);
    fn[1] = -0.5 * fma(s0, nr[0], ua[1] - ui[1]);
    fn[2] = -0.5 * fma(s0, nr[1], ua[2] - ui[2]);
    fn[3] = -0.5 * fma(s0, nr[2], ua[3] - ui[3]);
  }
}

// state on the other side of face f of element e at face point (a, b), whose
// own state is ui and outward normal nr (as face_fnum of stage_fv.cu)
__device__ __forceinline__ void other_side(const StageParams &P, int e, int f, int a, int b,
                                           const double *ui, const double nr[3], double t,
                                           double *ua) {
  const int n = P.n, nn = n * n, np = nn * n;
  const int nbe = __ldg(P.nb + e * 6 + f);
  if (nbe >= 0) {
    const int cd = __ldg(P.code + e * 6 + f), f2 = cd & 7, o = cd >> 3;
    if (cd & kCodeMixed) {
      const double *G = P.ghost + (size_t)__ldg(P.bslot + e * 6 + f) * 4 * nn + a + n * b;
      for (int l = 0; l < 4; l++) ua[l] = G[l * nn];
    } else {
      int aa = (o & 1) ? b : a, bb = (o & 1) ? a : b;
      if (o & 2) aa = n - 1 - aa;
      if (o & 4) bb = n - 1 - bb;
      const int d2 = f2 >> 1, p = (f2 & 1) * (n - 1);
      const int node = d2 == 0 ? p + n * (aa + n * bb)
                               : (d2 == 1 ? aa + n * (p + n * bb) : aa + n * (bb + n * p));
      const double *W = P.win + (size_t)nbe * NF * np + node;
      for (int l = 0; l < 4; l++) ua[l] = __ldg(W + l * np);
    }
    return;
  }
  const size_t ob = (size_t)__ldg(P.bslot + e * 6 + f) * 3 * nn + a + n * b;
  if (P.bc == NMG_BC_EXACT_PLANEWAVE) {
    const double *X = P.fvbxyz + ob;
    const double arg = P.k0 * X[0] + P.k1 * X[nn] + P.k2 * X[2 * nn] - P.om * t;
    double sn, cn;
    sincos(arg, &sn, &cn);
    ua[0] = -P.om * cn;
    ua[1] = P.k0 * cn;
    ua[2] = P.k1 * cn;
    ua[3] = P.k2 * cn;
  } else {
    // outgoing radiation: zero incoming characteristic pi + c.n
    const double cn = ui[1] * nr[0] + ui[2] * nr[1] + ui[3] * nr[2], wo = ui[0] - cn;
    ua[0] = 0.5 * wo;
    for (int l = 0; l < 3; l++) ua[1 + l] = ui[1 + l] + (-0.5 * wo - cn) * nr[l];
  }
}

template <int NT>
__global__ void __launch_bounds__(NT, 768 / NT) fvc_flux_kernel(const StageParams P, int k0,
                                                                int count) {
  extern __shared__ double sm[];
  const int n = P.n, nn = n * n, np = nn * n, tid = threadIdx.x;
  const int ppc = fvc_planes(n, NT), groups = (n + ppc - 1) / ppc;
  const int grp = blockIdx.x % groups, d = (blockIdx.x / groups) % 3;
  const int k = blockIdx.x / (groups * 3);  // element of this launch
  const int e = P.fvlist ? __ldg(P.fvlist + k0 + k) : P.ebase + k0 + k;
  const int z0 = grp * ppc, planes = min(ppc, n - z0);
  const int pen = planes * n, cells = pen * n;
  double *sW = sm, *sQ = sW + 4 * cells;  // sQ: [2: left, right face][4][cells]
  double *sF = sQ + 8 * cells;            // [4][pen (n + 1)]: midpoints, then both ends
  double *sIw = sF + 4 * pen * (n + 1);   // 1 / dXb of the points along the pencil
  const bool addsurf = P.fv_extrap == NMG_FV_EXTRAP_DNFN1;
  // Point t of pencil k (plane k / n): offset in the element and in shared memory.
  // The faster index of both runs along x where the direction has one.
  const int sa = d == 0 ? 1 : (d == 1 ? n : nn);
  const int s1 = d == 0 ? n : 1, s2 = d == 2 ? n : nn;     // in a plane, from plane to plane
  const int ca = d == 0 ? 1 : pen, ck = d == 0 ? n : 1;
  const double *Wg = P.win + (size_t)e * NF * np + z0 * s2;
  for (int i = tid; i < 4 * cells; i += NT) {
    const int f = i / cells, r = i - f * cells;
    const int t = d == 0 ? r % n : r / pen, q = d == 0 ? r / n : r % pen;
    sW[i] = __ldg(Wg + f * np + t * sa + (q % n) * s1 + (q / n) * s2);
  }
  if (tid < n)
    sIw[tid] = 1. / (tid == 0 ? __ldg(P.fvdist + e * 6 + 2 * d)
                              : (tid == n - 1 ? __ldg(P.fvdist + e * 6 + 2 * d + 1)
                                              : __ldg(P.fvdxb + tid)));
  const int cs = __ldg(P.cslot + e);
  const double *G = cs >= 0 ? P.fvgeo + (size_t)cs * kGeo * np : nullptr;
  const double *Gm = (cs >= 0 && P.fvmid) ? P.fvmid + (size_t)cs * 15 * np : nullptr;
  // Cartesian: 1/J J sqrtgdiag, the scale of the direction
  const double scd = __ldg(P.scale + e * 3 + d);
  __syncthreads();
  for (int i = tid; i < 4 * cells; i += NT) {
    // i = ((class position) * 4 + field) * pen + pencil
    const int q = i % pen, r = i / pen, f = r & 3, c = class_cell(P.fv_rec, n, r >> 2);
    double lft, rgt;
    cell_faces(P.fv_rec, n, sW + f * cells + q * ck, ca, c, P.fv_w3ratio, &lft, &rgt);
    sQ[f * cells + q * ck + c * ca] = lft;
    sQ[(4 + f) * cells + q * ck + c * ca] = rgt;
  }
  __syncthreads();
  const int nmid = pen * (n - 1), midw = (nmid + 31) / 32 * 32;
  for (int i = tid; i < midw + 2 * pen; i += NT) {
    double ui[4], ua[4], nr[3], fn[4], j;  // j: J sqrtgdiag
    int q, slot;
    if (i < midw) {
      if (i >= nmid) continue;
      // midpoint t (normal at its left point): the right face of cell t meets
      // the left face of cell t + 1
      const int t = d == 0 ? i % (n - 1) : i / pen;
      q = d == 0 ? i / (n - 1) : i % pen;
      slot = t;
      const int node = t * sa + (q % n) * s1 + (q / n + z0) * s2, qs = t * ca + q * ck;
#pragma unroll
      for (int l = 0; l < 4; l++) {
        ui[l] = sQ[(4 + l) * cells + qs];
        ua[l] = sQ[l * cells + qs + ca];
      }
      if (Gm) {
        const double *g = Gm + (size_t)d * 5 * np + node;
        j = __ldg(g) * fast_rcp(__ldg(g + np));
#pragma unroll
        for (int c = 0; c < 3; c++) nr[c] = __ldg(g + (2 + c) * np);
      } else if (G) {
        j = __ldg(G + (1 + d) * np + node) * fast_rcp(__ldg(G + node));
#pragma unroll
        for (int c = 0; c < 3; c++) nr[c] = __ldg(G + (4 + 3 * d + c) * np + node);
      }
    } else {
      const int sd = (i - midw) / pen, t = sd ? n - 1 : 0;
      q = i - midw - sd * pen;
      slot = n - 1 + sd;
      const int a = q % n, b = q / n + z0, node = t * sa + a * s1 + b * s2, qs = t * ca + q * ck;
      const double sg = sd ? 1. : -1.;
#pragma unroll
      for (int l = 0; l < 4; l++) ui[l] = sW[l * cells + qs];
      if (G) {
        j = __ldg(G + (1 + d) * np + node) * fast_rcp(__ldg(G + node));
#pragma unroll
        for (int c = 0; c < 3; c++) nr[c] = sg * __ldg(G + (4 + 3 * d + c) * np + node);
      } else {
#pragma unroll
        for (int c = 0; c < 3; c++) nr[c] = c == d ? sg : 0.;
      }
      other_side(P, e, 2 * d + sd, a, b, ui, nr, stage_time(P), ua);
    }
    if (!G) {
      j = 1.;  // of the element (in the factor of the difference)
      if (i < midw)
#pragma unroll
        for (int c = 0; c < 3; c++) nr[c] = c == d ? 1. : 0.;
    }
    flux4(P.numflux, ui, ua, nr, fn);
#pragma unroll
    for (int l = 0; l < 4; l++) sF[(l * pen + q) * (n + 1) + slot] = j * fn[l];
  }
  __syncthreads();
  // J sqrtgdiag / dXb flux difference, times 1/J.  At the ends: with
  // dnfn_extrap1 the face flux completes it and the end value is extrapolated
  // (4/3 of it minus 1/3 of its neighbour's); else the midpoint flux alone, plus
  // the face flux as a surface term.
  double *D = P.fvdiv + ((size_t)d * count + k) * 4 * np;
  for (int i = tid; i < cells; i += NT) {
    const int t = d == 0 ? i % n : i / pen, q = d == 0 ? i / n : i % pen;
    const int node = t * sa + (q % n) * s1 + (q / n + z0) * s2;
    const double oj = G ? __ldg(G + node) : scd;
    const bool end = t == 0 || t == n - 1;
    const double w = oj * sIw[t];
#pragma unroll
    for (int l = 0; l < 4; l++) {
      const double *F = sF + (l * pen + q) * (n + 1);
      double v;
      if (!end) {
        v = w * (F[t] - F[t - 1]);
      } else {
        // end value and its neighbour's; outward face flux at F[n - 1], F[n]
        const double face = t ? F[n] : F[n - 1], mid = t ? -F[n - 2] : F[0];
        v = w * (mid + face);
        if (addsurf && n > 2) {
          const int t1 = t ? n - 2 : 1;
          v = fma(4. / 3., v, (1. - 4. / 3.) * (oj * sIw[t1] * (F[t1] - F[t1 - 1])));
        }
      }
      D[l * np + node] = v;
    }
  }
}

// r = -(sum of the directions) (r_phi = pi) and the stage update
__global__ void __launch_bounds__(256) fvc_update_kernel(const StageParams P, int k0, int count) {
  const int np = P.n * P.n * P.n;
  const size_t dst = (size_t)count * 4 * np;
  const int64_t tot = (int64_t)count * NF * np;
  for (int64_t i = blockIdx.x * (int64_t)256 + threadIdx.x; i < tot;
       i += (int64_t)gridDim.x * 256) {
    const int k = (int)(i / (NF * np)), q = (int)(i - (int64_t)k * NF * np);
    const int e = P.fvlist ? __ldg(P.fvlist + k0 + k) : P.ebase + k0 + k;
    const size_t idx = (size_t)e * NF * np + q;
    double r;
    if (q < 4 * np) {
      const double *D = P.fvdiv + (size_t)k * 4 * np + q;
      r = -((D[0] + D[dst]) + D[2 * dst]);
    } else {
      r = __ldg(P.win + (size_t)e * NF * np + (q - 4 * np));
    }
    if (P.mode == 0) {
      P.rout[idx] = r;
    } else if (P.mode == 1) {
      const double u = __ldg(P.u0 + idx);
      P.acc[idx] = fma(P.cacc, r, u);
      P.wout[idx] = fma(P.cw, r, u);
    } else if (P.mode == 4) {
      P.acc[idx] = fma(P.cacc, r, P.acc[idx]);
    } else if (P.mode == 5) {
      P.acc[idx] = fma(P.cacc, r, __ldg(P.u0 + idx));
    } else if (P.mode == 6) {
      P.acc[idx] = fma(P.cacc, r, P.acc[idx]);
      P.wout[idx] = fma(0.25, fma(P.cw, r, __ldg(P.win + idx)), 0.75 * __ldg(P.u0 + idx));
    } else {
      P.acc[idx] = fma(P.cacc, r, P.acc[idx]);
      P.wout[idx] = fma(P.cw, r, __ldg(P.u0 + idx));
    }
  }
}

int fvc_elements(const StageParams &P) {
  return P.fvlist ? P.nfvel : (P.ecount > 0 ? P.ecount : P.nelem);
}

template <int NT>
cudaError_t launch_fvc(const StageParams &P, cudaStream_t st) {
  const size_t smem = fvc_smem(P.n, NT);
  if (P.nelem == 0) {
    size_t most = 0;
    for (int n = 2; n <= kFvMaxN; n++) most = std::max(most, fvc_smem(n, NT));
    return cudaFuncSetAttribute(fvc_flux_kernel<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)most);
  }
  const int total = fvc_elements(P), np = P.n * P.n * P.n, ppc = fvc_planes(P.n, NT);
  const int ctas = 3 * ((P.n + ppc - 1) / ppc);  // of an element
  for (int k0 = 0; k0 < total; k0 += P.fvdiv_cap) {
    const int count = std::min(P.fvdiv_cap, total - k0);
    fvc_flux_kernel<NT><<<count * ctas, NT, smem, st>>>(P, k0, count);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    const int64_t work = (int64_t)count * NF * np;
    fvc_update_kernel<<<(int)std::min<int64_t>((work + 255) / 256, 152 * 16), 256, 0, st>>>(
        P, k0, count);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace

int fvc_variants(int n, Variant *out, int cap) {
  if (n < 2 || n > kFvMaxN || cap < 3) return 0;
  out[0] = {"fvc", 1, 128, launch_fvc<128>};
  out[1] = {"fvc", 1, 256, launch_fvc<256>};
  out[2] = {"fvc", 1, 512, launch_fvc<512>};
  return 3;
}

int fvc_capacity(int n, int nelem) {
  const size_t per = sizeof(double) * 12 * (size_t)n * n * n;
  return (int)std::max<size_t>(1, std::min<size_t>((size_t)nelem, ((size_t)256 << 20) / per));
}

int fvc_launches(const StageParams &P) {
  return 2 * ((fvc_elements(P) + P.fvdiv_cap - 1) / P.fvdiv_cap);
}

}  // namespace nmgk
