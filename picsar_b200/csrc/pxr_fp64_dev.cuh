// Device code of the plain FP64 path shared by its per-particle kernels
// (pxr_fp64.cu) and its grouped ones (pxr_group.cu).
#pragma once
#include "pxr_common.cuh"

namespace pxrd {

// ---------------------------------------------------------------------------
// Esirkepov deposition with global FP64 atomics.  The old position is
// reconstructed as x - dt/dx*ux*gaminv (esirkepov_3d.F90:161-163); for the
// generic "_n" entry (reconstruct = 1) the new position is recomputed as
// xold + dt/dx*v as that routine does (:3566-3577).
// Currents are prefix sums of W along x (Jx), y (Jy), z (Jz) over the box.
// ---------------------------------------------------------------------------
struct DepParams {
  i64 np;
  const double *xp, *yp, *zp, *uxp, *uyp, *uzp, *gaminv, *w;
  double *jx, *jy, *jz;
  GridG G;
  double q, xmin, ymin, zmin, dxi, dyi, dzi, dtsdx, dtsdy, dtsdz;
  double invdtdx, invdtdy, invdtdz;
  int reconstruct;
  int* err;
};

template <int ORDER>
__device__ __forceinline__ void esir_axis(double x, double xold, EsirAxis<ORDER, double>& A,
                                          bool& ok) {
  int n0 = EsirAxis<ORDER, double>::node(x);
  int n1 = EsirAxis<ORDER, double>::node(xold);
  ok = A.set(n0, x - n0, n1, xold - n1) && ok;
}

// One particle's current by global atomics.
template <int ORDER>
__device__ __forceinline__ void deposit_one(const DepParams& p, i64 ip) {
  constexpr int M = ORDER + 2;
  const double onethird = 1.0 / 3.0;
  double x = (p.xp[ip] - p.xmin) * p.dxi, y = (p.yp[ip] - p.ymin) * p.dyi,
         z = (p.zp[ip] - p.zmin) * p.dzi;
  double gi = p.gaminv[ip];
  double vx = p.uxp[ip] * gi, vy = p.uyp[ip] * gi, vz = p.uzp[ip] * gi;
  double xold = x - p.dtsdx * vx, yold = y - p.dtsdy * vy, zold = z - p.dtsdz * vz;
  if (p.reconstruct) {
    x = xold + p.dtsdx * vx; y = yold + p.dtsdy * vy; z = zold + p.dtsdz * vz;
  }
  double wq = p.q * p.w[ip];
  double wqx = wq * p.invdtdx, wqy = wq * p.invdtdy, wqz = wq * p.invdtdz;
  EsirAxis<ORDER, double> X, Y, Z;
  bool ok = true;
  esir_axis<ORDER>(x, xold, X, ok);
  esir_axis<ORDER>(y, yold, Y, ok);
  esir_axis<ORDER>(z, zold, Z, ok);
  if (!ok) { atomicExch(p.err, 1); return; }
  // Jx: sweep x for every (j, k)
#pragma unroll
  for (int k = 0; k < M; ++k) {
    if (k >= Z.n) continue;
    double dsz = Z.s1[k] - Z.s0[k];
#pragma unroll
    for (int j = 0; j < M; ++j) {
      if (j >= Y.n) continue;
      double dsy = Y.s1[j] - Y.s0[j];
      double fyz = (Y.s0[j] + 0.5 * dsy) * Z.s0[k] + (0.5 * Y.s0[j] + onethird * dsy) * dsz;
      double acc = 0.0;
      double* row = p.jx + p.G.idx(X.i0, Y.i0 + j, Z.i0 + k);
#pragma unroll
      for (int i = 0; i < M - 1; ++i) {
        if (i >= X.n - 1) continue;
        acc = acc + wqx * (X.s1[i] - X.s0[i]) * fyz;
        atomicAdd(row + i, acc);
      }
    }
  }
  // Jy: sweep y for every (i, k)
#pragma unroll
  for (int k = 0; k < M; ++k) {
    if (k >= Z.n) continue;
    double dsz = Z.s1[k] - Z.s0[k];
#pragma unroll
    for (int i = 0; i < M; ++i) {
      if (i >= X.n) continue;
      double dsx = X.s1[i] - X.s0[i];
      double fzx = (Z.s0[k] + 0.5 * dsz) * X.s0[i] + (0.5 * Z.s0[k] + onethird * dsz) * dsx;
      double acc = 0.0;
      double* col = p.jy + p.G.idx(X.i0 + i, Y.i0, Z.i0 + k);
#pragma unroll
      for (int j = 0; j < M - 1; ++j) {
        if (j >= Y.n - 1) continue;
        acc = acc + wqy * (Y.s1[j] - Y.s0[j]) * fzx;
        atomicAdd(col + j * p.G.sx, acc);
      }
    }
  }
  // Jz: sweep z for every (i, j)
#pragma unroll
  for (int j = 0; j < M; ++j) {
    if (j >= Y.n) continue;
    double dsy = Y.s1[j] - Y.s0[j];
#pragma unroll
    for (int i = 0; i < M; ++i) {
      if (i >= X.n) continue;
      double dsx = X.s1[i] - X.s0[i];
      double fxy = (X.s0[i] + 0.5 * dsx) * Y.s0[j] + (0.5 * X.s0[i] + onethird * dsx) * dsy;
      double acc = 0.0;
      double* col = p.jz + p.G.idx(X.i0 + i, Y.i0 + j, Z.i0);
#pragma unroll
      for (int k = 0; k < M - 1; ++k) {
        if (k >= Z.n - 1) continue;
        acc = acc + wqz * (Z.s1[k] - Z.s0[k]) * fxy;
        atomicAdd(col + k * p.G.sy, acc);
      }
    }
  }
}

// Grouped form of the deposition and grouped order for the separate gather
// (pxr_group.cu).  group_fits, order_fits: the call is one that
// pxrb_group_scratch or pxrb_order_scratch asks scratch for, and this serves it.
bool group_fits(int order, i64 np, const GridG& G, const void* scratch, i64 bytes);
bool order_fits(int order, i64 np, const GridG& G, const void* scratch, i64 bytes);
// The order in which the separate gather (order 3) takes the call's particles:
// perm where *use (device), else as they come.
struct GatherOrder {
  const int *perm, *use;
};
int gather_order(i64 np, const double* xp, const double* yp, const double* zp, const double* lo,
                 const double* di, const GridG& G, void* scratch, cudaStream_t st,
                 GatherOrder& o);
int esirkepov_grouped(int order, const DepParams& p, void* scratch, cudaStream_t st);

}  // namespace pxrd
