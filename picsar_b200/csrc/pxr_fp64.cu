// Plain FP64 path: the drop-in kernels behind PICSAR's Forthon-exposed
// routines, on PICSAR's own guarded column-major FP64 arrays.  One thread per
// particle; without scratch the deposition uses global FP64 atomics (with it,
// pxr_group.cu).  This is also the "plain FP64 GPU" baseline every
// mixed-precision / tiled speed-up is stated against.
#include "pxr_fp64_dev.cuh"
#include "picsar_b200.h"

namespace {

using namespace pxrd;
constexpr int TPB = 256;

inline int nblocks(i64 n, int tpb = TPB) {
  i64 b = (n + tpb - 1) / tpb;
  return (int)(b < 1 ? 1 : (b > 2147483647 ? 2147483647 : b));
}

// ---------------------------------------------------------------------------
// Energy-conserving gather (accumulates) with the staggering of the fused
// kernels: E_c staggered along c, B_c staggered along the two other axes.
// Summation: for each z point, a = sum_y (sum_x s_x g) s_y; f += a s_z.
// ---------------------------------------------------------------------------
template <int NA, int NB, int NC>
__device__ __forceinline__ double gather_comp(const double* __restrict__ g, const GridG& G,
                                              int ia, const double* sa, int ib,
                                              const double* sb, int ic, const double* sc,
                                              double f) {
  const double* base = g + G.idx(ia, ib, ic);
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    double a = 0.0;
#pragma unroll
    for (int b = 0; b < NB; ++b) {
      const double* row = base + (G.sx * b + G.sy * c);
      double r = 0.0;
#pragma unroll
      for (int t = 0; t < NA; ++t) r = r + sa[t] * __ldg(row + t);
      a = a + r * sb[b];
    }
    f = f + a * sc[c];
  }
  return f;
}

template <int ORDER>
__device__ __forceinline__ void gather_eb(double x, double y, double z, const GridG& G,
                                          const double* exg, const double* eyg,
                                          const double* ezg, const double* bxg,
                                          const double* byg, const double* bzg, double& ex,
                                          double& ey, double& ez, double& bx, double& by,
                                          double& bz) {
  NodeShape<ORDER, double> nx, ny, nz;
  StagShape<ORDER, double> sx, sy, sz;
  nx.set(x); ny.set(y); nz.set(z);
  sx.set(x); sy.set(y); sz.set(z);
  constexpr int N = ORDER + 1, S = ORDER;
  ex = gather_comp<S, N, N>(exg, G, sx.i0, sx.s, ny.i0, ny.s, nz.i0, nz.s, ex);
  ey = gather_comp<N, S, N>(eyg, G, nx.i0, nx.s, sy.i0, sy.s, nz.i0, nz.s, ey);
  ez = gather_comp<N, N, S>(ezg, G, nx.i0, nx.s, ny.i0, ny.s, sz.i0, sz.s, ez);
  bx = gather_comp<N, S, S>(bxg, G, nx.i0, nx.s, sy.i0, sy.s, sz.i0, sz.s, bx);
  by = gather_comp<S, N, S>(byg, G, sx.i0, sx.s, ny.i0, ny.s, sz.i0, sz.s, by);
  bz = gather_comp<S, S, N>(bzg, G, sx.i0, sx.s, sy.i0, sy.s, nz.i0, nz.s, bz);
}

struct GPParams {
  i64 np;
  double *xp, *yp, *zp, *uxp, *uyp, *uzp, *gaminv;
  double *ex, *ey, *ez, *bx, *by, *bz;
  double xmin, ymin, zmin, dxi, dyi, dzi;
  const double *exg, *eyg, *ezg, *bxg, *byg, *bzg;
  GridG G;
  double q, m, dt, clight;
};

// field_gathering_plus_particle_pusher_{n}_{n}_{n}: gather (+=) into the
// particle field arrays, then Boris + set_gamma (pusher 0) or Vay (1), then
// pushxyz, all with the module time step dt.
// Blocks of 128 threads, as many per SM as the gather's registers allow: left
// to itself the compiler took 136 registers at order 3, one block of 256 per
// SM.  8.4 M particles in cell order, fused gather + push: order 3 2255 ->
// 1019 us, order 2 971 -> 712 us (order 1 keeps the 64 registers it had,
// 350 us); 5 or 6 blocks at order 3 spill (1067, 1114 us).
constexpr int GTPB = 128;
constexpr int gp_blocks(int order) { return order == 1 ? 8 : 4; }
// separate gather, same particles, lower / full shapes: order 3 1497 / 2304 ->
// 744 / 1288 us, order 2 814 / 901 -> 528 / 617 us
constexpr int geteb_blocks(int order, bool lower) { return order == 3 ? (lower ? 5 : 4) : 6; }

template <int ORDER, int PUSHER>
__global__ void __launch_bounds__(GTPB, gp_blocks(ORDER)) k_gather_push(GPParams p) {
  const double cst_b = p.q * p.dt * 0.5 / p.m;
  const double cst_v = p.q * p.dt / p.m;
  const double clghtisq = 1.0 / (p.clight * p.clight);
  for (i64 i = blockIdx.x * (i64)blockDim.x + threadIdx.x; i < p.np;
       i += (i64)gridDim.x * blockDim.x) {
    double x = (p.xp[i] - p.xmin) * p.dxi;
    double y = (p.yp[i] - p.ymin) * p.dyi;
    double z = (p.zp[i] - p.zmin) * p.dzi;
    double ex = p.ex[i], ey = p.ey[i], ez = p.ez[i];
    double bx = p.bx[i], by = p.by[i], bz = p.bz[i];
    gather_eb<ORDER>(x, y, z, p.G, p.exg, p.eyg, p.ezg, p.bxg, p.byg, p.bzg, ex, ey, ez, bx,
                     by, bz);
    p.ex[i] = ex; p.ey[i] = ey; p.ez[i] = ez;
    p.bx[i] = bx; p.by[i] = by; p.bz[i] = bz;
    double ux = p.uxp[i], uy = p.uyp[i], uz = p.uzp[i], gi = p.gaminv[i];
    if (PUSHER == 1) {
      vay_push(ux, uy, uz, gi, ex, ey, ez, bx, by, bz, cst_v, 1.0 / p.clight, clghtisq);
    } else {
      boris_push(ux, uy, uz, gi, ex, ey, ez, bx, by, bz, cst_b, clghtisq);
      set_gamma(ux, uy, uz, gi, clghtisq);
    }
    p.uxp[i] = ux; p.uyp[i] = uy; p.uzp[i] = uz; p.gaminv[i] = gi;
    p.xp[i] = p.xp[i] + ux * gi * p.dt;
    p.yp[i] = p.yp[i] + uy * gi * p.dt;
    p.zp[i] = p.zp[i] + uz * gi * p.dt;
  }
}

// Separate gather (geteb3d_energy_conserving), both l_lower_order_in_v
// branches and the nodal switch; accumulates.  One kernel per order and
// branch: with run-time orders the shapes sat in local memory and the point
// loops did not unroll.
//
// Staggered shape of degree DEG at x - ss (ss = 1/2, or 0 on the nodal grid):
// the scalar Fortran forms, field_gathering_o{1,2,3}_3d.F90.
template <int DEG> struct StagDeg {
  static constexpr int N = DEG + 1;
  int i0;
  double s[N];
  __device__ __forceinline__ void set(double x, double ss) {
    if (DEG == 0) {
      i0 = ffloor(x + 0.5 - ss); s[0] = 1.0;
    } else if (DEG == 1) {
      const int j0 = ffloor(x - ss);
      const double xi = x - ss - j0;
      i0 = j0; s[0] = 1.0 - xi; s[1] = xi;
    } else if (DEG == 2) {
      const int j0 = ffloor(x + 0.5 - ss);
      const double xi = x - ss - j0, xs = xi * xi;
      i0 = j0 - 1;
      s[0] = 0.5 * (0.5 - xi) * (0.5 - xi); s[1] = 0.75 - xs; s[2] = 0.5 * (0.5 + xi) * (0.5 + xi);
    } else {
      const int j0 = ffloor(x - ss);
      const double xi = x - ss - j0, ox = 1.0 - xi, xs = xi * xi, oxs = ox * ox;
      i0 = j0 - 1;
      s[0] = (1.0 / 6.0) * oxs * ox; s[1] = (2.0 / 3.0) - xs * (1.0 - xi * 0.5);
      s[2] = (2.0 / 3.0) - oxs * (1.0 - ox * 0.5); s[3] = (1.0 / 6.0) * xs * xi;
    }
  }
};

struct GEBParams {
  i64 np;
  const double *xp, *yp, *zp;
  double *ex, *ey, *ez, *bx, *by, *bz;
  double xmin, ymin, zmin, dxi, dyi, dzi;
  const double *exg, *eyg, *ezg, *bxg, *byg, *bzg;
  GridG G;
  double ss;
};

template <int ORDER, bool LOWER>
__global__ void __launch_bounds__(GTPB, geteb_blocks(ORDER, LOWER)) k_geteb(GEBParams p, GatherOrder order) {
  constexpr int N = ORDER + 1, DEG = LOWER ? ORDER - 1 : ORDER, S = DEG + 1;
  const i64 t = blockIdx.x * (i64)blockDim.x + threadIdx.x;
  if (t >= p.np) return;
  // asked for together with the flag that says whether it is the one to take
  double px = p.xp[t], py = p.yp[t], pz = p.zp[t];
  i64 i = t;
  if (order.use && *order.use) {
    i = order.perm[t];
    px = p.xp[i]; py = p.yp[i]; pz = p.zp[i];
  }
  const double x = (px - p.xmin) * p.dxi, y = (py - p.ymin) * p.dyi, z = (pz - p.zmin) * p.dzi;
  NodeShape<ORDER, double> nx, ny, nz;
  StagDeg<DEG> sx, sy, sz;
  nx.set(x); ny.set(y); nz.set(z);
  sx.set(x, p.ss); sy.set(y, p.ss); sz.set(z, p.ss);
  p.ex[i] = gather_comp<S, N, N>(p.exg, p.G, sx.i0, sx.s, ny.i0, ny.s, nz.i0, nz.s, p.ex[i]);
  p.ey[i] = gather_comp<N, S, N>(p.eyg, p.G, nx.i0, nx.s, sy.i0, sy.s, nz.i0, nz.s, p.ey[i]);
  p.ez[i] = gather_comp<N, N, S>(p.ezg, p.G, nx.i0, nx.s, ny.i0, ny.s, sz.i0, sz.s, p.ez[i]);
  p.bx[i] = gather_comp<N, S, S>(p.bxg, p.G, nx.i0, nx.s, sy.i0, sy.s, sz.i0, sz.s, p.bx[i]);
  p.by[i] = gather_comp<S, N, S>(p.byg, p.G, sx.i0, sx.s, ny.i0, ny.s, sz.i0, sz.s, p.by[i]);
  p.bz[i] = gather_comp<S, S, N>(p.bzg, p.G, sx.i0, sx.s, sy.i0, sy.s, nz.i0, nz.s, p.bz[i]);
}

// ---------------------------------------------------------------------------
// Stand-alone pushers.
// ---------------------------------------------------------------------------
struct PushParams {
  i64 np;
  double *ux, *uy, *uz, *gi;
  const double *ex, *ey, *ez, *bx, *by, *bz;
  double *x, *y, *z;
  double q, m, dt, clight;
  int which;
};

__global__ void k_boris(PushParams p) {
  const double cst = p.q * p.dt * 0.5 / p.m, c2i = 1.0 / (p.clight * p.clight);
  for (i64 i = blockIdx.x * (i64)blockDim.x + threadIdx.x; i < p.np;
       i += (i64)gridDim.x * blockDim.x) {
    double ux = p.ux[i], uy = p.uy[i], uz = p.uz[i], gi = p.gi[i];
    boris_push(ux, uy, uz, gi, p.ex[i], p.ey[i], p.ez[i], p.bx[i], p.by[i], p.bz[i], cst, c2i);
    p.ux[i] = ux; p.uy[i] = uy; p.uz[i] = uz; p.gi[i] = gi;
  }
}

__global__ void k_vay(PushParams p) {
  const double invc = 1.0 / p.clight, invc2 = 1.0 / (p.clight * p.clight);
  for (i64 i = blockIdx.x * (i64)blockDim.x + threadIdx.x; i < p.np;
       i += (i64)gridDim.x * blockDim.x) {
    double ux = p.ux[i], uy = p.uy[i], uz = p.uz[i], gi = p.gi[i];
    double ex = p.ex[i], ey = p.ey[i], ez = p.ez[i], bx = p.bx[i], by = p.by[i], bz = p.bz[i];
    if (p.which == 0) {
      vay_push(ux, uy, uz, gi, ex, ey, ez, bx, by, bz, p.q * p.dt / p.m, invc, invc2);
    } else if (p.which == 1) {
      const double cst = 0.5 * p.q * p.dt / p.m;
      double vx = ux * gi, vy = uy * gi, vz = uz * gi;
      ux = ux + cst * (ex + vy * bz - vz * by);
      uy = uy + cst * (ey + vz * bx - vx * bz);
      uz = uz + cst * (ez + vx * by - vy * bx);
      gi = 1.0 / sqrt(1.0 + (ux * ux + uy * uy + uz * uz) * invc2);
    } else {
      const double cst = 0.5 * p.q * p.dt / p.m, bconst = cst;
      double uxpr = ux + cst * ex, uypr = uy + cst * ey, uzpr = uz + cst * ez;
      double gprsq = (1.0 + (uxpr * uxpr + uypr * uypr + uzpr * uzpr) * invc2);
      double taux = bconst * bx, tauy = bconst * by, tauz = bconst * bz;
      double tausq = taux * taux + tauy * tauy + tauz * tauz;
      double ust = (uxpr * taux + uypr * tauy + uzpr * tauz) * invc;
      double sigma = gprsq - tausq;
      double gisq = 2.0 / (sigma + sqrt(sigma * sigma + 4.0 * (tausq + ust * ust)));
      gi = sqrt(gisq);
      double bg = bconst * gi, tx = bg * bx, ty = bg * by, tz = bg * bz;
      double s = 1.0 / (1.0 + tausq * gisq);
      double tu = tx * uxpr + ty * uypr + tz * uzpr;
      ux = s * (uxpr + tx * tu + uypr * tz - uzpr * ty);
      uy = s * (uypr + ty * tu + uzpr * tx - uxpr * tz);
      uz = s * (uzpr + tz * tu + uxpr * ty - uypr * tx);
    }
    p.ux[i] = ux; p.uy[i] = uy; p.uz[i] = uz; p.gi[i] = gi;
  }
}

__global__ void k_set_gamma(PushParams p) {
  const double c2i = 1.0 / (p.clight * p.clight);
  for (i64 i = blockIdx.x * (i64)blockDim.x + threadIdx.x; i < p.np;
       i += (i64)gridDim.x * blockDim.x) {
    double gi;
    set_gamma(p.ux[i], p.uy[i], p.uz[i], gi, c2i);
    p.gi[i] = gi;
  }
}

__global__ void k_pushxyz(PushParams p) {
  for (i64 i = blockIdx.x * (i64)blockDim.x + threadIdx.x; i < p.np;
       i += (i64)gridDim.x * blockDim.x) {
    double gi = p.gi[i];
    p.x[i] = p.x[i] + p.ux[i] * gi * p.dt;
    p.y[i] = p.y[i] + p.uy[i] * gi * p.dt;
    p.z[i] = p.z[i] + p.uz[i] * gi * p.dt;
  }
}

template <int ORDER>
__global__ void __launch_bounds__(TPB) k_esirkepov(DepParams p) {
  for (i64 ip = blockIdx.x * (i64)blockDim.x + threadIdx.x; ip < p.np;
       ip += (i64)gridDim.x * blockDim.x)
    deposit_one<ORDER>(p, ip);
}

// Node-centred charge deposition (charge_deposition_3d.F90:77-400).
struct RhoParams {
  i64 np;
  const double *xp, *yp, *zp, *w;
  double* rho;
  GridG G;
  double q, xmin, ymin, zmin, dxi, dyi, dzi, invvol;
};

template <int ORDER>
__global__ void __launch_bounds__(TPB) k_rho(RhoParams p) {
  for (i64 ip = blockIdx.x * (i64)blockDim.x + threadIdx.x; ip < p.np;
       ip += (i64)gridDim.x * blockDim.x) {
    double x = (p.xp[ip] - p.xmin) * p.dxi, y = (p.yp[ip] - p.ymin) * p.dyi,
           z = (p.zp[ip] - p.zmin) * p.dzi;
    double wq = p.q * p.w[ip] * p.invvol;
    NodeShape<ORDER, double> sx, sy, sz;
    sx.set(x); sy.set(y); sz.set(z);
#pragma unroll
    for (int c = 0; c < ORDER + 1; ++c)
#pragma unroll
      for (int b = 0; b < ORDER + 1; ++b)
#pragma unroll
        for (int a = 0; a < ORDER + 1; ++a)
          atomicAdd(p.rho + p.G.idx(sx.i0 + a, sy.i0 + b, sz.i0 + c),
                    sx.s[a] * sy.s[b] * sz.s[c] * wq);
  }
}

// ---------------------------------------------------------------------------
// Yee (yee.F90:637-740, :1258-1347).  Thread (j,k,l) over the union of the
// three component ranges; each component predicated on its own range.
// ---------------------------------------------------------------------------
struct YeeParams {
  double *ex, *ey, *ez, *bx, *by, *bz;
  const double *jx, *jy, *jz;
  GridG gex, gey, gez, gbx, gby, gbz, gjx, gjy, gjz;  // per-array bounds
  int lo[3][3], hi[3][3];   // per-component loop ranges
  int ulo[3], uhi[3];       // union
  double mudt, dtsdx, dtsdy, dtsdz;
};

__device__ __forceinline__ bool inr(const int* lo, const int* hi, int j, int k, int l) {
  return j >= lo[0] && j <= hi[0] && k >= lo[1] && k <= hi[1] && l >= lo[2] && l <= hi[2];
}

__global__ void k_yee_e(YeeParams p) {
  int j = p.ulo[0] + blockIdx.x * blockDim.x + threadIdx.x;
  int k = p.ulo[1] + blockIdx.y * blockDim.y + threadIdx.y;
  int l = p.ulo[2] + blockIdx.z;
  if (j > p.uhi[0] || k > p.uhi[1] || l > p.uhi[2]) return;
  if (inr(p.lo[0], p.hi[0], j, k, l)) {
    double* e = p.ex + p.gex.idx(j, k, l);
    *e = *e + p.dtsdy * (p.bz[p.gbz.idx(j, k, l)] - p.bz[p.gbz.idx(j, k - 1, l)]) -
         p.dtsdz * (p.by[p.gby.idx(j, k, l)] - p.by[p.gby.idx(j, k, l - 1)]) -
         p.mudt * p.jx[p.gjx.idx(j, k, l)];
  }
  if (inr(p.lo[1], p.hi[1], j, k, l)) {
    double* e = p.ey + p.gey.idx(j, k, l);
    *e = *e - p.dtsdx * (p.bz[p.gbz.idx(j, k, l)] - p.bz[p.gbz.idx(j - 1, k, l)]) +
         p.dtsdz * (p.bx[p.gbx.idx(j, k, l)] - p.bx[p.gbx.idx(j, k, l - 1)]) -
         p.mudt * p.jy[p.gjy.idx(j, k, l)];
  }
  if (inr(p.lo[2], p.hi[2], j, k, l)) {
    double* e = p.ez + p.gez.idx(j, k, l);
    *e = *e + p.dtsdx * (p.by[p.gby.idx(j, k, l)] - p.by[p.gby.idx(j - 1, k, l)]) -
         p.dtsdy * (p.bx[p.gbx.idx(j, k, l)] - p.bx[p.gbx.idx(j, k - 1, l)]) -
         p.mudt * p.jz[p.gjz.idx(j, k, l)];
  }
}

__global__ void k_yee_b(YeeParams p) {
  int j = p.ulo[0] + blockIdx.x * blockDim.x + threadIdx.x;
  int k = p.ulo[1] + blockIdx.y * blockDim.y + threadIdx.y;
  int l = p.ulo[2] + blockIdx.z;
  if (j > p.uhi[0] || k > p.uhi[1] || l > p.uhi[2]) return;
  if (inr(p.lo[0], p.hi[0], j, k, l)) {
    double* b = p.bx + p.gbx.idx(j, k, l);
    *b = *b - p.dtsdy * (p.ez[p.gez.idx(j, k + 1, l)] - p.ez[p.gez.idx(j, k, l)]) +
         p.dtsdz * (p.ey[p.gey.idx(j, k, l + 1)] - p.ey[p.gey.idx(j, k, l)]);
  }
  if (inr(p.lo[1], p.hi[1], j, k, l)) {
    double* b = p.by + p.gby.idx(j, k, l);
    *b = *b + p.dtsdx * (p.ez[p.gez.idx(j + 1, k, l)] - p.ez[p.gez.idx(j, k, l)]) -
         p.dtsdz * (p.ex[p.gex.idx(j, k, l + 1)] - p.ex[p.gex.idx(j, k, l)]);
  }
  if (inr(p.lo[2], p.hi[2], j, k, l)) {
    double* b = p.bz + p.gbz.idx(j, k, l);
    *b = *b - p.dtsdx * (p.ey[p.gey.idx(j + 1, k, l)] - p.ey[p.gey.idx(j, k, l)]) +
         p.dtsdy * (p.ex[p.gex.idx(j, k + 1, l)] - p.ex[p.gex.idx(j, k, l)]);
  }
}

// ---------------------------------------------------------------------------
// Periodic single-domain guard exchanges (field_boundaries.F90:107-269 and
// :403-503).  The reference exchanges slabs axis by axis; with n > g per axis
// the outcome has a closed form, so one launch serves all axes and arrays:
//   field_bc:  every node outside [0, n) takes its periodic image;
//   summation: an inner node within g of a side adds the outer nodes that
//              fold onto it, x inside y inside z, each as
//              (A[i] + A[n+i]) + A[i-n] - the order of the slab sums - and
//              the outer nodes then take their images.
// A fold reads its own node and outer nodes only, and writes its own: no two
// threads meet.  One warp per row.  (A launch per axis with a thread per line
// was a serial chain of 4 (g+1) accesses: 10 us each, 15 a step, 0.15 of the
// 0.17 ms of device time of a small step.)
// ---------------------------------------------------------------------------
struct BcParams {
  double* a[3];
  i64 n[3], g[3];
  i64 sy, sz;                // row and plane strides
};

__device__ __forceinline__ i64 image(i64 i, i64 n) { return i < 0 ? i + n : (i >= n ? i - n : i); }

constexpr int BC_ROWS = TPB / 32;

__global__ void __launch_bounds__(TPB) k_bc_fill(BcParams p) {
  const i64 ey = p.n[1] + 1 + 2 * p.g[1], ez = p.n[2] + 1 + 2 * p.g[2];
  const i64 j = blockIdx.x * (i64)BC_ROWS + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (j >= ey) return;
  double* A = p.a[blockIdx.z];
  const i64 n = p.n[0], g = p.g[0];
  for (i64 k = blockIdx.y; k < ez; k += gridDim.y) {
    const i64 y = j - p.g[1], z = k - p.g[2];
    const i64 sy = image(y, p.n[1]), sz = image(z, p.n[2]);
    double* row = A + p.sy * j + p.sz * k + g;
    if (sy == y && sz == z) {                 // inner row: its two ends
      for (i64 t = lane; t < 2 * g + 1; t += 32) {
        const i64 x = t < g ? t - g : n + t - g;
        row[x] = row[image(x, n)];
      }
    } else {
      const double* src = A + p.sy * (sy + p.g[1]) + p.sz * (sz + p.g[2]) + g;
      for (i64 x = lane - g; x <= n + g; x += 32) row[x] = src[image(x, n)];
    }
  }
}

// value of an inner column i of a row with the outer columns folded in
__device__ __forceinline__ double fold_x(const double* row, i64 i, i64 n, i64 g) {
  double v = row[i];
  if (n == 0) return v;
  if (i <= g) v = v + row[n + i];
  if (i >= n - g) v = v + row[i - n];
  return v;
}
__device__ __forceinline__ double fold_xy(const BcParams& p, const double* plane, i64 i, i64 j) {
  const i64 n = p.n[1], g = p.g[1];
  double v = fold_x(plane + p.sy * j, i, p.n[0], p.g[0]);
  if (n == 0) return v;
  if (j <= g) v = v + fold_x(plane + p.sy * (n + j), i, p.n[0], p.g[0]);
  if (j >= n - g) v = v + fold_x(plane + p.sy * (j - n), i, p.n[0], p.g[0]);
  return v;
}

__global__ void __launch_bounds__(TPB) k_bc_fold(BcParams p) {
  const i64 j = blockIdx.x * (i64)BC_ROWS + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  const i64 nx = p.n[0], ny = p.n[1], nz = p.n[2], g = p.g[0];
  if (j >= max(ny, (i64)1)) return;
  double* o = p.a[blockIdx.z] + p.g[0] + p.sy * p.g[1] + p.sz * p.g[2];      // node (0, 0, 0)
  for (i64 k = blockIdx.y; k < max(nz, (i64)1); k += gridDim.y) {
    auto fold = [&](i64 i) {
      double v = fold_xy(p, o + p.sz * k, i, j);
      if (nz > 0) {
        if (k <= p.g[2]) v = v + fold_xy(p, o + p.sz * (nz + k), i, j);
        if (k >= nz - p.g[2]) v = v + fold_xy(p, o + p.sz * (k - nz), i, j);
      }
      o[i + p.sy * j + p.sz * k] = v;
    };
    const bool edge = (ny > 0 && (j <= p.g[1] || j >= ny - p.g[1])) ||
                      (nz > 0 && (k <= p.g[2] || k >= nz - p.g[2]));
    if (edge || nx <= 2 * g + 1) {
      for (i64 i = lane; i < max(nx, (i64)1); i += 32) fold(i);
    } else {                                  // the row's ends: [0, g] and [n - g, n)
      for (i64 t = lane; t < 2 * g + 1; t += 32) fold(t <= g ? t : nx - 1 - (t - g - 1));
    }
  }
}

// Periodic particle wrap (particle_boundaries.F90:1109-1300, pbound = 0).
struct WrapParams {
  i64 np;
  double *x, *y, *z;
  double lo[3], hi[3];
};

__global__ void k_wrap(WrapParams p) {
  double len[3] = {p.hi[0] - p.lo[0], p.hi[1] - p.lo[1], p.hi[2] - p.lo[2]};
  for (i64 i = blockIdx.x * (i64)blockDim.x + threadIdx.x; i < p.np;
       i += (i64)gridDim.x * blockDim.x) {
    double* c[3] = {p.x + i, p.y + i, p.z + i};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      double v = *c[a];
      if (v < p.lo[a]) *c[a] = v + len[a];
      else if (v >= p.hi[a]) *c[a] = v - len[a];
    }
  }
}

inline int grid_stride_blocks(i64 n) {
  // enough CTAs to fill 148 SMs several times over, capped by the work
  i64 b = (n + TPB - 1) / TPB;
  const i64 cap = 148 * 16;
  return (int)(b < 1 ? 1 : (b > cap ? cap : b));
}

bool bad_ptr(const void* p) { return p == nullptr; }

// ---------------------------------------------------------------------------
// 2D (x-z) path on PICSAR's 2-D arrays (-g:n+g) in x and z, Fortran order:
// the separate energy-conserving gather (field_gathering_o{1,2,3}_2d.F90),
// Esirkepov deposition (esirkepov_2d.F90:452-1082) with global FP64 atomics,
// the order-2 Yee update (yee.F90:216-310, :912-994) and pxr_pushxz.
// ---------------------------------------------------------------------------
struct G2 {
  i64 gx, gz, sx;
  __device__ __forceinline__ i64 idx(i64 i, i64 k) const { return (i + gx) + sx * (k + gz); }
};

template <int NA, int NC>
__device__ __forceinline__ double gather2(const double* __restrict__ g, const G2& G, int ia,
                                          const double* sa, int ic, const double* sc, double f) {
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    const double* row = g + G.idx(ia, ic + c);
    double r = 0.0;
#pragma unroll
    for (int t = 0; t < NA; ++t) r = r + sa[t] * __ldg(row + t);
    f = f + r * sc[c];
  }
  return f;
}

struct GEB2Params {
  i64 np;
  const double *xp, *zp;
  double *ex, *ey, *ez, *bx, *by, *bz;
  double xmin, zmin, dxi, dzi;
  const double *exg, *eyg, *ezg, *bxg, *byg, *bzg;
  G2 G;
  double ss;
};

template <int ORDER, bool LOWER>
__global__ void __launch_bounds__(TPB) k_geteb2d(GEB2Params p) {
  constexpr int N = ORDER + 1, DEG = LOWER ? ORDER - 1 : ORDER, S = DEG + 1;
  const i64 i = blockIdx.x * (i64)blockDim.x + threadIdx.x;
  if (i >= p.np) return;
  const double x = (p.xp[i] - p.xmin) * p.dxi, z = (p.zp[i] - p.zmin) * p.dzi;
  NodeShape<ORDER, double> nx, nz;
  StagDeg<DEG> sx, sz;
  nx.set(x); nz.set(z);
  sx.set(x, p.ss); sz.set(z, p.ss);
  p.ex[i] = gather2<S, N>(p.exg, p.G, sx.i0, sx.s, nz.i0, nz.s, p.ex[i]);
  p.ey[i] = gather2<N, N>(p.eyg, p.G, nx.i0, nx.s, nz.i0, nz.s, p.ey[i]);
  p.ez[i] = gather2<N, S>(p.ezg, p.G, nx.i0, nx.s, sz.i0, sz.s, p.ez[i]);
  p.bx[i] = gather2<N, S>(p.bxg, p.G, nx.i0, nx.s, sz.i0, sz.s, p.bx[i]);
  p.by[i] = gather2<S, S>(p.byg, p.G, sx.i0, sx.s, sz.i0, sz.s, p.by[i]);
  p.bz[i] = gather2<S, N>(p.bzg, p.G, sx.i0, sx.s, nz.i0, nz.s, p.bz[i]);
}

struct Dep2Params {
  i64 np;
  double *jx, *jy, *jz;
  const double *xp, *zp, *uxp, *uyp, *uzp, *gaminv, *w;
  double q, xmin, zmin, dt, dx, dz;
  G2 G;
};

// The reference's 2-D shapes: order 3 with its default-real (single
// precision) constants 1/6 and 2/3.
template <int ORDER> __device__ __forceinline__ void shape2d(double xint, double* s) {
  if (ORDER == 1) {
    s[0] = 1.0 - xint; s[1] = xint;
  } else if (ORDER == 2) {
    const double xs = xint * xint;
    s[0] = 0.5 * (0.5 - xint) * (0.5 - xint);
    s[1] = 0.75 - xs;
    s[2] = 0.5 * (0.5 + xint) * (0.5 + xint);
  } else {
    const double onesixth = (double)(1.0f / 6.0f), twothird = (double)(2.0f / 3.0f);
    const double ox = 1.0 - xint, xs = xint * xint, oxs = ox * ox;
    s[0] = onesixth * oxs * ox;
    s[1] = twothird - xs * (1.0 - xint * 0.5);
    s[2] = twothird - oxs * (1.0 - ox * 0.5);
    s[3] = onesixth * xs * xint;
  }
}

// One axis: the new (s0) and old (s1) shapes on the common box of their
// nodes, every index a compile-time constant (with shape arrays indexed by
// the run-time shift the kernel worked out of local memory).
template <int ORDER> struct Box2 {
  static constexpr int M = ORDER + 2;
  i64 i0;                   // first node of the box
  int n;
  double s0[M], d[M];       // new shape; old minus new
  __device__ __forceinline__ void set(double x, double xold) {
    const i64 n0 = ORDER == 2 ? (i64)round(x) : (i64)floor(x);
    const i64 n1 = ORDER == 2 ? (i64)round(xold) : (i64)floor(xold);
    double t0[ORDER + 1], t1[ORDER + 1];
    shape2d<ORDER>(x - n0, t0);
    shape2d<ORDER>(xold - n1, t1);
    // a move of more than one cell per step (beyond the CFL limit) would
    // leave the box: clamp, as no valid input reaches it
    int s = (int)(n1 - n0);
    s = s < -1 ? -1 : (s > 1 ? 1 : s);
    const bool up0 = s < 0, up1 = s > 0;
    i0 = n0 - ORDER / 2 - (up0 ? 1 : 0);
    n = ORDER + 1 + (s != 0 ? 1 : 0);
#pragma unroll
    for (int r = 0; r < M; ++r) {
      const double a0 = r <= ORDER ? t0[r <= ORDER ? r : 0] : 0.0, b0 = r ? t0[r ? r - 1 : 0] : 0.0;
      const double a1 = r <= ORDER ? t1[r <= ORDER ? r : 0] : 0.0, b1 = r ? t1[r ? r - 1 : 0] : 0.0;
      s0[r] = up0 ? b0 : a0;
      d[r] = (up1 ? b1 : a1) - s0[r];
    }
  }
};

// A warp takes particles SPREAD apart: neighbours in memory are mostly in one
// cell, and atomics of many lanes to one address go one by one.
template <int ORDER>
__global__ void __launch_bounds__(TPB) k_esirkepov2d(Dep2Params p) {
  constexpr int M = ORDER + 2, SPREAD = TPB / 32;
  const double onethird = (double)(1.0f / 3.0f);
  const double dxi = 1.0 / p.dx, dzi = 1.0 / p.dz;
  const double dtsdx0 = p.dt * dxi, dtsdz0 = p.dt * dzi;
  const double invvol = 1.0 / (p.dx * p.dz), invdtdx = 1.0 / (p.dt * p.dz),
               invdtdz = 1.0 / (p.dt * p.dx);
  const i64 ip = blockIdx.x * (i64)TPB + (threadIdx.x & 31) * SPREAD + (threadIdx.x >> 5);
  if (ip >= p.np) return;
  const double x = (p.xp[ip] - p.xmin) * dxi, z = (p.zp[ip] - p.zmin) * dzi;
  const double gi = p.gaminv[ip];
  const double vx = p.uxp[ip] * gi, vy = p.uyp[ip] * gi, vz = p.uzp[ip] * gi;
  const double wq = p.q * p.w[ip], wqx = wq * invdtdx, wqz = wq * invdtdz;
  Box2<ORDER> X, Z;
  X.set(x, x - dtsdx0 * vx);
  Z.set(z, z - dtsdz0 * vz);
  const i64 c0 = p.G.idx(X.i0, Z.i0);
  double cz[M];
#pragma unroll
  for (int i = 0; i < M; ++i) cz[i] = 0.0;
#pragma unroll
  for (int k = 0; k < M; ++k) {
    if (k >= Z.n) continue;
    double cx = 0.0;
#pragma unroll
    for (int i = 0; i < M; ++i) {
      if (i >= X.n) continue;
      const i64 c = c0 + i + p.G.sx * k;
      if (i < X.n - 1) {
        cx = cx + wqx * X.d[i] * (Z.s0[k] + 0.5 * Z.d[k]);
        atomicAdd(p.jx + c, cx);
      }
      atomicAdd(p.jy + c, wq * vy * invvol * ((Z.s0[k] + 0.5 * Z.d[k]) * X.s0[i] +
                                              (0.5 * Z.s0[k] + onethird * Z.d[k]) * X.d[i]));
      if (k < Z.n - 1) {
        cz[i] = cz[i] + wqz * Z.d[k] * (X.s0[i] + 0.5 * X.d[i]);
        atomicAdd(p.jz + c, cz[i]);
      }
    }
  }
}

struct Yee2Params {
  double *ex, *ey, *ez, *bx, *by, *bz;
  const double *jx, *jy, *jz;
  G2 gex, gey, gez, gbx, gby, gbz, gjx, gjy, gjz;
  int lo[3][2], hi[3][2];
  int ulo[2], uhi[2];
  double mudt, dtsdx, dtsdz;
};

__device__ __forceinline__ bool inr2(const int* lo, const int* hi, int j, int k) {
  return j >= lo[0] && j <= hi[0] && k >= lo[1] && k <= hi[1];
}

__global__ void k_yee2d_e(Yee2Params p) {
  const int j = p.ulo[0] + blockIdx.x * blockDim.x + threadIdx.x;
  const int k = p.ulo[1] + blockIdx.y * blockDim.y + threadIdx.y;
  if (j > p.uhi[0] || k > p.uhi[1]) return;
  if (inr2(p.lo[0], p.hi[0], j, k)) {
    double* e = p.ex + p.gex.idx(j, k);
    *e = *e - p.dtsdz * (p.by[p.gby.idx(j, k)] - p.by[p.gby.idx(j, k - 1)]) -
         p.mudt * p.jx[p.gjx.idx(j, k)];
  }
  if (inr2(p.lo[1], p.hi[1], j, k)) {
    double* e = p.ey + p.gey.idx(j, k);
    *e = *e - p.dtsdx * (p.bz[p.gbz.idx(j, k)] - p.bz[p.gbz.idx(j - 1, k)]) +
         p.dtsdz * (p.bx[p.gbx.idx(j, k)] - p.bx[p.gbx.idx(j, k - 1)]) -
         p.mudt * p.jy[p.gjy.idx(j, k)];
  }
  if (inr2(p.lo[2], p.hi[2], j, k)) {
    double* e = p.ez + p.gez.idx(j, k);
    *e = *e + p.dtsdx * (p.by[p.gby.idx(j, k)] - p.by[p.gby.idx(j - 1, k)]) -
         p.mudt * p.jz[p.gjz.idx(j, k)];
  }
}

__global__ void k_yee2d_b(Yee2Params p) {
  const int j = p.ulo[0] + blockIdx.x * blockDim.x + threadIdx.x;
  const int k = p.ulo[1] + blockIdx.y * blockDim.y + threadIdx.y;
  if (j > p.uhi[0] || k > p.uhi[1]) return;
  if (inr2(p.lo[0], p.hi[0], j, k)) {
    double* b = p.bx + p.gbx.idx(j, k);
    *b = *b + p.dtsdz * (p.ey[p.gey.idx(j, k + 1)] - p.ey[p.gey.idx(j, k)]);
  }
  if (inr2(p.lo[1], p.hi[1], j, k)) {
    double* b = p.by + p.gby.idx(j, k);
    *b = *b + p.dtsdx * (p.ez[p.gez.idx(j + 1, k)] - p.ez[p.gez.idx(j, k)]) -
         p.dtsdz * (p.ex[p.gex.idx(j, k + 1)] - p.ex[p.gex.idx(j, k)]);
  }
  if (inr2(p.lo[2], p.hi[2], j, k)) {
    double* b = p.bz + p.gbz.idx(j, k);
    *b = *b - p.dtsdx * (p.ey[p.gey.idx(j + 1, k)] - p.ey[p.gey.idx(j, k)]);
  }
}

__global__ void k_pushxz(i64 np, double* xp, double* zp, const double* uxp, const double* uzp,
                         const double* gaminv, double dt) {
  for (i64 i = blockIdx.x * (i64)blockDim.x + threadIdx.x; i < np;
       i += (i64)gridDim.x * blockDim.x) {
    xp[i] = xp[i] + uxp[i] * gaminv[i] * dt;
    zp[i] = zp[i] + uzp[i] * gaminv[i] * dt;
  }
}

inline G2 g2_lohi(const int64_t* lo, const int64_t* hi) {
  G2 g;
  g.gx = -lo[0]; g.gz = -lo[1];
  g.sx = hi[0] - lo[0] + 1;
  return g;
}

}  // namespace

// ===========================================================================
// extern "C" entry points
// ===========================================================================
extern "C" {

int pxrb_field_gathering_plus_particle_pusher(
    int64_t order, int64_t np, double* xp, double* yp, double* zp, double* uxp, double* uyp,
    double* uzp, double* gaminv, double* ex, double* ey, double* ez, double* bx, double* by,
    double* bz, double xmin, double ymin, double zmin, double dx, double dy, double dz,
    double dtt, int64_t nx, int64_t ny, int64_t nz, int64_t nxguard, int64_t nyguard,
    int64_t nzguard, const double* exg, const double* eyg, const double* ezg,
    const double* bxg, const double* byg, const double* bzg, double q, double m,
    int64_t lvect, int64_t l_lower_order_in_v, double dt, int64_t particle_pusher,
    double clight, void* stream) {
  (void)dtt; (void)lvect;
  if (np < 0 || nx < 0 || ny < 0 || nz < 0) return PXRB_EINVAL;
  if (np == 0) return PXRB_OK;
  if (order < 1 || order > 3 || !l_lower_order_in_v) return PXRB_EUNSUPPORTED;
  const void* ptrs[] = {xp, yp, zp, uxp, uyp, uzp, gaminv, ex, ey, ez, bx, by, bz,
                        exg, eyg, ezg, bxg, byg, bzg};
  for (const void* p : ptrs) if (bad_ptr(p)) return PXRB_EINVAL;
  GPParams p;
  p.np = np; p.xp = xp; p.yp = yp; p.zp = zp; p.uxp = uxp; p.uyp = uyp; p.uzp = uzp;
  p.gaminv = gaminv; p.ex = ex; p.ey = ey; p.ez = ez; p.bx = bx; p.by = by; p.bz = bz;
  p.xmin = xmin; p.ymin = ymin; p.zmin = zmin;
  p.dxi = 1.0 / dx; p.dyi = 1.0 / dy; p.dzi = 1.0 / dz;
  p.exg = exg; p.eyg = eyg; p.ezg = ezg; p.bxg = bxg; p.byg = byg; p.bzg = bzg;
  p.G = make_grid(nx, ny, nz, nxguard, nyguard, nzguard);
  p.q = q; p.m = m; p.dt = dt; p.clight = clight;
  cudaStream_t s = (cudaStream_t)stream;
  int nb = nblocks(np, GTPB);
  int vay = particle_pusher == 1;
#define LAUNCH_GP(O)                                                                   \
  if (vay) k_gather_push<O, 1><<<nb, GTPB, 0, s>>>(p);                                  \
  else k_gather_push<O, 0><<<nb, GTPB, 0, s>>>(p);
  if (order == 1) { LAUNCH_GP(1) }
  else if (order == 2) { LAUNCH_GP(2) }
  else { LAUNCH_GP(3) }
#undef LAUNCH_GP
  PXRB_CHECK_LAUNCH();
  return PXRB_OK;
}

#define PXRB_FGP_N(O)                                                                   \
  int pxrb_field_gathering_plus_particle_pusher_##O##_##O##_##O(                          \
      int64_t np, double* xp, double* yp, double* zp, double* uxp, double* uyp,           \
      double* uzp, double* gaminv, double* ex, double* ey, double* ez, double* bx,        \
      double* by, double* bz, double xmin, double ymin, double zmin, double dx, double dy, \
      double dz, double dtt, int64_t nx, int64_t ny, int64_t nz, int64_t nxguard,         \
      int64_t nyguard, int64_t nzguard, const double* exg, const double* eyg,             \
      const double* ezg, const double* bxg, const double* byg, const double* bzg,         \
      double q, double m, int64_t lvect, int64_t l_lower_order_in_v, double dt,           \
      int64_t particle_pusher, double clight, void* stream) {                             \
    return pxrb_field_gathering_plus_particle_pusher(                                     \
        O, np, xp, yp, zp, uxp, uyp, uzp, gaminv, ex, ey, ez, bx, by, bz, xmin, ymin,     \
        zmin, dx, dy, dz, dtt, nx, ny, nz, nxguard, nyguard, nzguard, exg, eyg, ezg, bxg, \
        byg, bzg, q, m, lvect, l_lower_order_in_v, dt, particle_pusher, clight, stream);  \
  }
PXRB_FGP_N(1)
PXRB_FGP_N(2)
PXRB_FGP_N(3)
#undef PXRB_FGP_N

int pxrb_geteb3d_energy_conserving_ws(
    int64_t np, const double* xp, const double* yp, const double* zp, double* ex, double* ey,
    double* ez, double* bx, double* by, double* bz, double xmin, double ymin, double zmin,
    double dx, double dy, double dz, int64_t nx, int64_t ny, int64_t nz, int64_t nxguard,
    int64_t nyguard, int64_t nzguard, int64_t nox, int64_t noy, int64_t noz,
    const double* exg, const double* eyg, const double* ezg, const double* bxg,
    const double* byg, const double* bzg, int64_t ll4symtry, int64_t l_lower_order_in_v,
    int64_t lvect, int64_t field_gathe_algo, int64_t l_nodal, void* scratch,
    int64_t scratch_bytes, void* stream) {
  (void)lvect; (void)field_gathe_algo;
  if (np < 0) return PXRB_EINVAL;
  if (np == 0) return PXRB_OK;
  if (nox != noy || noy != noz || nox < 1 || nox > 3 || ll4symtry) return PXRB_EUNSUPPORTED;
  const void* ptrs[] = {xp, yp, zp, ex, ey, ez, bx, by, bz, exg, eyg, ezg, bxg, byg, bzg};
  for (const void* p : ptrs) if (bad_ptr(p)) return PXRB_EINVAL;
  GEBParams p;
  p.np = np; p.xp = xp; p.yp = yp; p.zp = zp;
  p.ex = ex; p.ey = ey; p.ez = ez; p.bx = bx; p.by = by; p.bz = bz;
  p.xmin = xmin; p.ymin = ymin; p.zmin = zmin;
  p.dxi = 1.0 / dx; p.dyi = 1.0 / dy; p.dzi = 1.0 / dz;
  p.exg = exg; p.eyg = eyg; p.ezg = ezg; p.bxg = bxg; p.byg = byg; p.bzg = bzg;
  p.G = make_grid(nx, ny, nz, nxguard, nyguard, nzguard);
  p.ss = l_nodal ? 0.0 : 0.5;
  cudaStream_t s = (cudaStream_t)stream;
  const int nb = nblocks(np, GTPB);
  GatherOrder by_key = {nullptr, nullptr};
  if (order_fits((int)nox, np, p.G, scratch, scratch_bytes)) {
    const double lo[3] = {xmin, ymin, zmin}, di[3] = {p.dxi, p.dyi, p.dzi};
    const int rc = gather_order(np, xp, yp, zp, lo, di, p.G, scratch, s, by_key);
    if (rc) return rc;
  }
#define PXRB_GEB(O_)                                                  \
  if (l_lower_order_in_v) k_geteb<O_, true><<<nb, GTPB, 0, s>>>(p, by_key);    \
  else k_geteb<O_, false><<<nb, GTPB, 0, s>>>(p, by_key);
  if (nox == 1) { PXRB_GEB(1) } else if (nox == 2) { PXRB_GEB(2) } else { PXRB_GEB(3) }
#undef PXRB_GEB
  PXRB_CHECK_LAUNCH();
  return PXRB_OK;
}

int pxrb_geteb3d_energy_conserving(
    int64_t np, const double* xp, const double* yp, const double* zp, double* ex, double* ey,
    double* ez, double* bx, double* by, double* bz, double xmin, double ymin, double zmin,
    double dx, double dy, double dz, int64_t nx, int64_t ny, int64_t nz, int64_t nxguard,
    int64_t nyguard, int64_t nzguard, int64_t nox, int64_t noy, int64_t noz,
    const double* exg, const double* eyg, const double* ezg, const double* bxg,
    const double* byg, const double* bzg, int64_t ll4symtry, int64_t l_lower_order_in_v,
    int64_t lvect, int64_t field_gathe_algo, int64_t l_nodal, void* stream) {
  return pxrb_geteb3d_energy_conserving_ws(
      np, xp, yp, zp, ex, ey, ez, bx, by, bz, xmin, ymin, zmin, dx, dy, dz, nx, ny, nz, nxguard,
      nyguard, nzguard, nox, noy, noz, exg, eyg, ezg, bxg, byg, bzg, ll4symtry,
      l_lower_order_in_v, lvect, field_gathe_algo, l_nodal, nullptr, 0, stream);
}

static int launch_push(int kind, int64_t np, double* ux, double* uy, double* uz, double* gi,
                       const double* ex, const double* ey, const double* ez,
                       const double* bx, const double* by, const double* bz, double* x,
                       double* y, double* z, double q, double m, double dt, double clight,
                       int which, void* stream) {
  if (np < 0) return PXRB_EINVAL;
  if (np == 0) return PXRB_OK;
  PushParams p;
  p.np = np; p.ux = ux; p.uy = uy; p.uz = uz; p.gi = gi;
  p.ex = ex; p.ey = ey; p.ez = ez; p.bx = bx; p.by = by; p.bz = bz;
  p.x = x; p.y = y; p.z = z; p.q = q; p.m = m; p.dt = dt; p.clight = clight; p.which = which;
  cudaStream_t s = (cudaStream_t)stream;
  int nb = grid_stride_blocks(np);
  switch (kind) {
    case 0: k_boris<<<nb, TPB, 0, s>>>(p); break;
    case 1: k_vay<<<nb, TPB, 0, s>>>(p); break;
    case 2: k_set_gamma<<<nb, TPB, 0, s>>>(p); break;
    case 3: k_pushxyz<<<nb, TPB, 0, s>>>(p); break;
  }
  PXRB_CHECK_LAUNCH();
  return PXRB_OK;
}

int pxrb_boris_push_u_3d(int64_t np, double* uxp, double* uyp, double* uzp, double* gaminv,
                         const double* ex, const double* ey, const double* ez,
                         const double* bx, const double* by, const double* bz, double q,
                         double m, double dt, double clight, void* stream) {
  if (np > 0 && (!uxp || !uyp || !uzp || !gaminv || !ex || !ey || !ez || !bx || !by || !bz))
    return PXRB_EINVAL;
  return launch_push(0, np, uxp, uyp, uzp, gaminv, ex, ey, ez, bx, by, bz, nullptr, nullptr,
                     nullptr, q, m, dt, clight, 0, stream);
}

int pxrb_ebcancelpush3d(int64_t np, double* uxp, double* uyp, double* uzp, double* gi,
                        const double* ex, const double* ey, const double* ez,
                        const double* bx, const double* by, const double* bz, double q,
                        double m, double dt, int64_t which, double clight, void* stream) {
  if (which < 0 || which > 2) return PXRB_EUNSUPPORTED;
  if (np > 0 && (!uxp || !uyp || !uzp || !gi || !ex || !ey || !ez || !bx || !by || !bz))
    return PXRB_EINVAL;
  return launch_push(1, np, uxp, uyp, uzp, gi, ex, ey, ez, bx, by, bz, nullptr, nullptr,
                     nullptr, q, m, dt, clight, (int)which, stream);
}

int pxrb_set_gamma(int64_t np, const double* uxp, const double* uyp, const double* uzp,
                   double* gaminv, double clight, void* stream) {
  if (np > 0 && (!uxp || !uyp || !uzp || !gaminv)) return PXRB_EINVAL;
  return launch_push(2, np, const_cast<double*>(uxp), const_cast<double*>(uyp),
                     const_cast<double*>(uzp), gaminv, nullptr, nullptr, nullptr, nullptr,
                     nullptr, nullptr, nullptr, nullptr, nullptr, 0, 1, 0, clight, 0, stream);
}

int pxrb_pushxyz(int64_t np, double* xp, double* yp, double* zp, const double* uxp,
                 const double* uyp, const double* uzp, const double* gaminv, double dt,
                 void* stream) {
  if (np > 0 && (!xp || !yp || !zp || !uxp || !uyp || !uzp || !gaminv)) return PXRB_EINVAL;
  return launch_push(3, np, const_cast<double*>(uxp), const_cast<double*>(uyp),
                     const_cast<double*>(uzp), const_cast<double*>(gaminv), nullptr, nullptr,
                     nullptr, nullptr, nullptr, nullptr, xp, yp, zp, 0, 1, dt, 1, 0, stream);
}

int pxrb_depose_jxjyjz_ws(double* jx, double* jy, double* jz, int64_t np, const double* xp,
                       const double* yp, const double* zp, const double* uxp,
                       const double* uyp, const double* uzp, const double* gaminv,
                       const double* w, double q, double xmin, double ymin, double zmin,
                       double dt, double dx, double dy, double dz, int64_t nx, int64_t ny,
                       int64_t nz, int64_t nxguard, int64_t nyguard, int64_t nzguard,
                       int64_t nox, int64_t noy, int64_t noz, int64_t current_depo_algo,
                       int* err_flag, void* scratch, int64_t scratch_bytes, void* stream) {
  if (np < 0) return PXRB_EINVAL;
  if (np == 0) return PXRB_OK;
  if (nox != noy || noy != noz || nox < 1 || nox > 3) return PXRB_EUNSUPPORTED;
  if (current_depo_algo != 0 && current_depo_algo != 1) return PXRB_EUNSUPPORTED;
  const void* ptrs[] = {jx, jy, jz, xp, yp, zp, uxp, uyp, uzp, gaminv, w, err_flag};
  for (const void* p : ptrs) if (bad_ptr(p)) return PXRB_EINVAL;
  DepParams p;
  p.np = np; p.xp = xp; p.yp = yp; p.zp = zp; p.uxp = uxp; p.uyp = uyp; p.uzp = uzp;
  p.gaminv = gaminv; p.w = w; p.jx = jx; p.jy = jy; p.jz = jz;
  p.G = make_grid(nx, ny, nz, nxguard, nyguard, nzguard);
  p.q = q; p.xmin = xmin; p.ymin = ymin; p.zmin = zmin;
  p.dxi = 1.0 / dx; p.dyi = 1.0 / dy; p.dzi = 1.0 / dz;
  p.dtsdx = dt * p.dxi; p.dtsdy = dt * p.dyi; p.dtsdz = dt * p.dzi;
  p.invdtdx = 1.0 / (dt * dy * dz); p.invdtdy = 1.0 / (dt * dx * dz);
  p.invdtdz = 1.0 / (dt * dx * dy);
  p.reconstruct = current_depo_algo == 1;
  p.err = err_flag;
  cudaStream_t s = (cudaStream_t)stream;
  if (group_fits((int)nox, np, p.G, scratch, scratch_bytes))
    return esirkepov_grouped((int)nox, p, scratch, s);
  int nb = nblocks(np);
  if (nox == 1) k_esirkepov<1><<<nb, TPB, 0, s>>>(p);
  else if (nox == 2) k_esirkepov<2><<<nb, TPB, 0, s>>>(p);
  else k_esirkepov<3><<<nb, TPB, 0, s>>>(p);
  PXRB_CHECK_LAUNCH();
  return PXRB_OK;
}

int pxrb_depose_jxjyjz(double* jx, double* jy, double* jz, int64_t np, const double* xp,
                       const double* yp, const double* zp, const double* uxp,
                       const double* uyp, const double* uzp, const double* gaminv,
                       const double* w, double q, double xmin, double ymin, double zmin,
                       double dt, double dx, double dy, double dz, int64_t nx, int64_t ny,
                       int64_t nz, int64_t nxguard, int64_t nyguard, int64_t nzguard,
                       int64_t nox, int64_t noy, int64_t noz, int64_t current_depo_algo,
                       int* err_flag, void* stream) {
  return pxrb_depose_jxjyjz_ws(jx, jy, jz, np, xp, yp, zp, uxp, uyp, uzp, gaminv, w, q, xmin,
                               ymin, zmin, dt, dx, dy, dz, nx, ny, nz, nxguard, nyguard,
                               nzguard, nox, noy, noz, current_depo_algo, err_flag, nullptr, 0,
                               stream);
}

int pxrb_depose_rho(int64_t order, double* rho, int64_t np, const double* xp,
                    const double* yp, const double* zp, const double* w, double q,
                    double xmin, double ymin, double zmin, double dx, double dy, double dz,
                    int64_t nx, int64_t ny, int64_t nz, int64_t nxguard, int64_t nyguard,
                    int64_t nzguard, void* stream) {
  if (np < 0) return PXRB_EINVAL;
  if (np == 0) return PXRB_OK;
  if (order < 1 || order > 3) return PXRB_EUNSUPPORTED;
  if (!rho || !xp || !yp || !zp || !w) return PXRB_EINVAL;
  RhoParams p;
  p.np = np; p.xp = xp; p.yp = yp; p.zp = zp; p.w = w; p.rho = rho;
  p.G = make_grid(nx, ny, nz, nxguard, nyguard, nzguard);
  p.q = q; p.xmin = xmin; p.ymin = ymin; p.zmin = zmin;
  p.dxi = 1.0 / dx; p.dyi = 1.0 / dy; p.dzi = 1.0 / dz;
  p.invvol = p.dxi * p.dyi * p.dzi;
  cudaStream_t s = (cudaStream_t)stream;
  int nb = nblocks(np);
  if (order == 1) k_rho<1><<<nb, TPB, 0, s>>>(p);
  else if (order == 2) k_rho<2><<<nb, TPB, 0, s>>>(p);
  else k_rho<3><<<nb, TPB, 0, s>>>(p);
  PXRB_CHECK_LAUNCH();
  return PXRB_OK;
}

static GridG grid_lohi(const int64_t* lo, const int64_t* hi) {
  GridG g;
  // An array with Fortran bounds (lo:hi) per axis as a guarded grid: guards
  // gx = -lo, so that idx(i) = i - lo; and nx = hi + lo, so that the extent
  // nx + 1 + 2 gx equals hi - lo + 1.
  g.gx = -lo[0]; g.gy = -lo[1]; g.gz = -lo[2];
  g.nx = hi[0] + lo[0]; g.ny = hi[1] + lo[1]; g.nz = hi[2] + lo[2];
  g.sx = hi[0] - lo[0] + 1;
  g.sy = g.sx * (hi[1] - lo[1] + 1);
  return g;
}

static int yee_setup(YeeParams& p, const int64_t* xlo, const int64_t* xhi, const int64_t* ylo,
                     const int64_t* yhi, const int64_t* zlo, const int64_t* zhi) {
  const int64_t* L[3] = {xlo, ylo, zlo};
  const int64_t* H[3] = {xhi, yhi, zhi};
  for (int a = 0; a < 3; ++a) { p.ulo[a] = 1 << 30; p.uhi[a] = -(1 << 30); }
  for (int c = 0; c < 3; ++c)
    for (int a = 0; a < 3; ++a) {
      p.lo[c][a] = (int)L[c][a]; p.hi[c][a] = (int)H[c][a];
      p.ulo[a] = p.lo[c][a] < p.ulo[a] ? p.lo[c][a] : p.ulo[a];
      p.uhi[a] = p.hi[c][a] > p.uhi[a] ? p.hi[c][a] : p.uhi[a];
    }
  for (int a = 0; a < 3; ++a) if (p.uhi[a] < p.ulo[a]) return 1;
  return 0;
}

int pxrb_push_em3d_evec(const int64_t* xlo, const int64_t* xhi, const int64_t* ylo,
                        const int64_t* yhi, const int64_t* zlo, const int64_t* zhi,
                        double* ex, const int64_t* exlo, const int64_t* exhi, double* ey,
                        const int64_t* eylo, const int64_t* eyhi, double* ez,
                        const int64_t* ezlo, const int64_t* ezhi, const double* bx,
                        const int64_t* bxlo, const int64_t* bxhi, const double* by,
                        const int64_t* bylo, const int64_t* byhi, const double* bz,
                        const int64_t* bzlo, const int64_t* bzhi, const double* jx,
                        const int64_t* jxlo, const int64_t* jxhi, const double* jy,
                        const int64_t* jylo, const int64_t* jyhi, const double* jz,
                        const int64_t* jzlo, const int64_t* jzhi, double mudt, double dtsdx,
                        double dtsdy, double dtsdz, void* stream) {
  if (!ex || !ey || !ez || !bx || !by || !bz || !jx || !jy || !jz) return PXRB_EINVAL;
  YeeParams p;
  if (yee_setup(p, xlo, xhi, ylo, yhi, zlo, zhi)) return PXRB_OK;  // empty ranges
  p.ex = ex; p.ey = ey; p.ez = ez;
  p.bx = const_cast<double*>(bx); p.by = const_cast<double*>(by); p.bz = const_cast<double*>(bz);
  p.jx = jx; p.jy = jy; p.jz = jz;
  p.gex = grid_lohi(exlo, exhi); p.gey = grid_lohi(eylo, eyhi); p.gez = grid_lohi(ezlo, ezhi);
  p.gbx = grid_lohi(bxlo, bxhi); p.gby = grid_lohi(bylo, byhi); p.gbz = grid_lohi(bzlo, bzhi);
  p.gjx = grid_lohi(jxlo, jxhi); p.gjy = grid_lohi(jylo, jyhi); p.gjz = grid_lohi(jzlo, jzhi);
  p.mudt = mudt; p.dtsdx = dtsdx; p.dtsdy = dtsdy; p.dtsdz = dtsdz;
  dim3 blk(32, 8, 1);
  dim3 grd((p.uhi[0] - p.ulo[0] + 1 + 31) / 32, (p.uhi[1] - p.ulo[1] + 1 + 7) / 8,
           p.uhi[2] - p.ulo[2] + 1);
  k_yee_e<<<grd, blk, 0, (cudaStream_t)stream>>>(p);
  PXRB_CHECK_LAUNCH();
  return PXRB_OK;
}

int pxrb_push_em3d_bvec(const int64_t* xlo, const int64_t* xhi, const int64_t* ylo,
                        const int64_t* yhi, const int64_t* zlo, const int64_t* zhi,
                        const double* ex, const int64_t* exlo, const int64_t* exhi,
                        const double* ey, const int64_t* eylo, const int64_t* eyhi,
                        const double* ez, const int64_t* ezlo, const int64_t* ezhi,
                        double* bx, const int64_t* bxlo, const int64_t* bxhi, double* by,
                        const int64_t* bylo, const int64_t* byhi, double* bz,
                        const int64_t* bzlo, const int64_t* bzhi, double dtsdx, double dtsdy,
                        double dtsdz, void* stream) {
  if (!ex || !ey || !ez || !bx || !by || !bz) return PXRB_EINVAL;
  YeeParams p;
  if (yee_setup(p, xlo, xhi, ylo, yhi, zlo, zhi)) return PXRB_OK;
  p.ex = const_cast<double*>(ex); p.ey = const_cast<double*>(ey); p.ez = const_cast<double*>(ez);
  p.bx = bx; p.by = by; p.bz = bz;
  p.jx = p.jy = p.jz = nullptr;
  p.gex = grid_lohi(exlo, exhi); p.gey = grid_lohi(eylo, eyhi); p.gez = grid_lohi(ezlo, ezhi);
  p.gbx = grid_lohi(bxlo, bxhi); p.gby = grid_lohi(bylo, byhi); p.gbz = grid_lohi(bzlo, bzhi);
  p.mudt = 0; p.dtsdx = dtsdx; p.dtsdy = dtsdy; p.dtsdz = dtsdz;
  dim3 blk(32, 8, 1);
  dim3 grd((p.uhi[0] - p.ulo[0] + 1 + 31) / 32, (p.uhi[1] - p.ulo[1] + 1 + 7) / 8,
           p.uhi[2] - p.ulo[2] + 1);
  k_yee_b<<<grd, blk, 0, (cudaStream_t)stream>>>(p);
  PXRB_CHECK_LAUNCH();
  return PXRB_OK;
}

static int bc_launch(double** arrs, int na, int64_t nx, int64_t ny, int64_t nz, int64_t nxg,
                     int64_t nyg, int64_t nzg, bool fold, void* stream) {
  if (na < 1 || na > 3) return PXRB_EINVAL;
  for (int q = 0; q < na; ++q) if (!arrs[q]) return PXRB_EINVAL;
  // an axis of no cells and no guards (ny = 0 of PICSAR's x-z grids) is skipped
  auto bad = [](int64_t n, int64_t g) { return g < 0 || (n <= g && !(n == 0 && g == 0)); };
  if (bad(nx, nxg) || bad(ny, nyg) || bad(nz, nzg)) return PXRB_ERANGE;
  const GridG G = make_grid(nx, ny, nz, nxg, nyg, nzg);
  const i64 ey = ny + 1 + 2 * nyg, ez = nz + 1 + 2 * nzg;
  BcParams p;
  for (int q = 0; q < 3; ++q) p.a[q] = q < na ? arrs[q] : nullptr;
  const int64_t nn[3] = {nx, ny, nz}, gg[3] = {nxg, nyg, nzg};
  for (int q = 0; q < 3; ++q) { p.n[q] = nn[q]; p.g[q] = gg[q]; }
  p.sy = G.sx; p.sz = G.sy;
  cudaStream_t s = (cudaStream_t)stream;
  auto grid = [na](i64 rows, i64 planes) {
    rows = rows > 0 ? rows : 1; planes = planes > 0 ? planes : 1;
    return dim3((unsigned)((rows + BC_ROWS - 1) / BC_ROWS),
                (unsigned)(planes < 65535 ? planes : 65535), na);
  };
  if (fold) k_bc_fold<<<grid(ny, nz), TPB, 0, s>>>(p);
  k_bc_fill<<<grid(ey, ez), TPB, 0, s>>>(p);
  PXRB_CHECK_LAUNCH();
  return PXRB_OK;
}

int pxrb_field_bc_periodic(double* f1, double* f2, double* f3, int64_t nx, int64_t ny,
                           int64_t nz, int64_t nxg, int64_t nyg, int64_t nzg, void* stream) {
  double* a[3] = {f1, f2, f3};
  int na = f3 ? 3 : (f2 ? 2 : 1);
  return bc_launch(a, na, nx, ny, nz, nxg, nyg, nzg, false, stream);
}

int pxrb_summation_bcs_periodic(double* f1, double* f2, double* f3, int64_t nx, int64_t ny,
                                int64_t nz, int64_t nxg, int64_t nyg, int64_t nzg,
                                void* stream) {
  double* a[3] = {f1, f2, f3};
  int na = f3 ? 3 : (f2 ? 2 : 1);
  return bc_launch(a, na, nx, ny, nz, nxg, nyg, nzg, true, stream);
}

int pxrb_geteb2dxz_energy_conserving(
    int64_t np, const double* xp, const double* yp, const double* zp, double* ex, double* ey,
    double* ez, double* bx, double* by, double* bz, double xmin, double ymin, double zmin,
    double dx, double dy, double dz, int64_t nx, int64_t ny, int64_t nz, int64_t nxguard,
    int64_t nyguard, int64_t nzguard, int64_t nox, int64_t noy, int64_t noz,
    const double* exg, const double* eyg, const double* ezg, const double* bxg,
    const double* byg, const double* bzg, int64_t l4symtry, int64_t l_lower_order_in_v,
    int64_t lvect, int64_t field_gathe_algo, int64_t l_nodal, void* stream) {
  (void)yp; (void)ymin; (void)dy; (void)ny; (void)nyguard; (void)noy; (void)lvect;
  (void)field_gathe_algo;
  if (np < 0) return PXRB_EINVAL;
  if (np == 0) return PXRB_OK;
  if (nox != noz || nox < 1 || nox > 3 || l4symtry) return PXRB_EUNSUPPORTED;
  if (!xp || !zp || !ex || !ey || !ez || !bx || !by || !bz || !exg || !eyg || !ezg || !bxg ||
      !byg || !bzg)
    return PXRB_EINVAL;
  GEB2Params p;
  p.np = np; p.xp = xp; p.zp = zp;
  p.ex = ex; p.ey = ey; p.ez = ez; p.bx = bx; p.by = by; p.bz = bz;
  p.xmin = xmin; p.zmin = zmin; p.dxi = 1.0 / dx; p.dzi = 1.0 / dz;
  p.exg = exg; p.eyg = eyg; p.ezg = ezg; p.bxg = bxg; p.byg = byg; p.bzg = bzg;
  p.G.gx = nxguard; p.G.gz = nzguard; p.G.sx = nx + 1 + 2 * nxguard;
  p.ss = l_nodal ? 0.0 : 0.5;
  cudaStream_t s = (cudaStream_t)stream;
  const int nb = nblocks(np);
#define PXRB_GEB(O_)                                                    \
  if (l_lower_order_in_v) k_geteb2d<O_, true><<<nb, TPB, 0, s>>>(p);    \
  else k_geteb2d<O_, false><<<nb, TPB, 0, s>>>(p);
  if (nox == 1) { PXRB_GEB(1) } else if (nox == 2) { PXRB_GEB(2) } else { PXRB_GEB(3) }
#undef PXRB_GEB
  PXRB_CHECK_LAUNCH();
  return PXRB_OK;
}

int pxrb_depose_jxjyjz_2d(double* jx, double* jy, double* jz, int64_t np, const double* xp,
                          const double* yp, const double* zp, const double* uxp,
                          const double* uyp, const double* uzp, const double* gaminv,
                          const double* w, double q, double xmin, double zmin, double dt,
                          double dx, double dz, int64_t nx, int64_t nz, int64_t nxguard,
                          int64_t nzguard, int64_t nox, int64_t noz, int64_t lvect,
                          void* stream) {
  (void)yp; (void)lvect;
  if (np < 0) return PXRB_EINVAL;
  if (np == 0) return PXRB_OK;
  if (nox != noz || nox < 1 || nox > 3) return PXRB_EUNSUPPORTED;
  if (!jx || !jy || !jz || !xp || !zp || !uxp || !uyp || !uzp || !gaminv || !w)
    return PXRB_EINVAL;
  Dep2Params p;
  p.np = np; p.jx = jx; p.jy = jy; p.jz = jz;
  p.xp = xp; p.zp = zp; p.uxp = uxp; p.uyp = uyp; p.uzp = uzp; p.gaminv = gaminv; p.w = w;
  p.q = q; p.xmin = xmin; p.zmin = zmin; p.dt = dt; p.dx = dx; p.dz = dz;
  p.G.gx = nxguard; p.G.gz = nzguard; p.G.sx = nx + 1 + 2 * nxguard;
  cudaStream_t s = (cudaStream_t)stream;
  if (nox == 1) k_esirkepov2d<1><<<nblocks(np), TPB, 0, s>>>(p);
  else if (nox == 2) k_esirkepov2d<2><<<nblocks(np), TPB, 0, s>>>(p);
  else k_esirkepov2d<3><<<nblocks(np), TPB, 0, s>>>(p);
  PXRB_CHECK_LAUNCH();
  return PXRB_OK;
}

static int yee2d_setup(Yee2Params& p, const int64_t* xlo, const int64_t* xhi, const int64_t* ylo,
                       const int64_t* yhi, const int64_t* zlo, const int64_t* zhi) {
  const int64_t* L[3] = {xlo, ylo, zlo};
  const int64_t* H[3] = {xhi, yhi, zhi};
  for (int a = 0; a < 2; ++a) { p.ulo[a] = 1 << 30; p.uhi[a] = -(1 << 30); }
  for (int c = 0; c < 3; ++c)
    for (int a = 0; a < 2; ++a) {
      p.lo[c][a] = (int)L[c][a]; p.hi[c][a] = (int)H[c][a];
      p.ulo[a] = p.lo[c][a] < p.ulo[a] ? p.lo[c][a] : p.ulo[a];
      p.uhi[a] = p.hi[c][a] > p.uhi[a] ? p.hi[c][a] : p.uhi[a];
    }
  for (int a = 0; a < 2; ++a) if (p.uhi[a] < p.ulo[a]) return 1;
  return 0;
}

int pxrb_push_em2d_evec(const int64_t* xlo, const int64_t* xhi, const int64_t* ylo,
                        const int64_t* yhi, const int64_t* zlo, const int64_t* zhi,
                        double* ex, const int64_t* exlo, const int64_t* exhi, double* ey,
                        const int64_t* eylo, const int64_t* eyhi, double* ez,
                        const int64_t* ezlo, const int64_t* ezhi, const double* bx,
                        const int64_t* bxlo, const int64_t* bxhi, const double* by,
                        const int64_t* bylo, const int64_t* byhi, const double* bz,
                        const int64_t* bzlo, const int64_t* bzhi, const double* jx,
                        const int64_t* jxlo, const int64_t* jxhi, const double* jy,
                        const int64_t* jylo, const int64_t* jyhi, const double* jz,
                        const int64_t* jzlo, const int64_t* jzhi, double mudt, double dtsdx,
                        double dtsdy, double dtsdz, void* stream) {
  (void)dtsdy;
  if (!ex || !ey || !ez || !bx || !by || !bz || !jx || !jy || !jz) return PXRB_EINVAL;
  Yee2Params p;
  if (yee2d_setup(p, xlo, xhi, ylo, yhi, zlo, zhi)) return PXRB_OK;
  p.ex = ex; p.ey = ey; p.ez = ez;
  p.bx = const_cast<double*>(bx); p.by = const_cast<double*>(by); p.bz = const_cast<double*>(bz);
  p.jx = jx; p.jy = jy; p.jz = jz;
  p.gex = g2_lohi(exlo, exhi); p.gey = g2_lohi(eylo, eyhi); p.gez = g2_lohi(ezlo, ezhi);
  p.gbx = g2_lohi(bxlo, bxhi); p.gby = g2_lohi(bylo, byhi); p.gbz = g2_lohi(bzlo, bzhi);
  p.gjx = g2_lohi(jxlo, jxhi); p.gjy = g2_lohi(jylo, jyhi); p.gjz = g2_lohi(jzlo, jzhi);
  p.mudt = mudt; p.dtsdx = dtsdx; p.dtsdz = dtsdz;
  dim3 blk(32, 8, 1);
  dim3 grd((p.uhi[0] - p.ulo[0] + 1 + 31) / 32, (p.uhi[1] - p.ulo[1] + 1 + 7) / 8, 1);
  k_yee2d_e<<<grd, blk, 0, (cudaStream_t)stream>>>(p);
  PXRB_CHECK_LAUNCH();
  return PXRB_OK;
}

int pxrb_push_em2d_bvec(const int64_t* xlo, const int64_t* xhi, const int64_t* ylo,
                        const int64_t* yhi, const int64_t* zlo, const int64_t* zhi,
                        const double* ex, const int64_t* exlo, const int64_t* exhi,
                        const double* ey, const int64_t* eylo, const int64_t* eyhi,
                        const double* ez, const int64_t* ezlo, const int64_t* ezhi,
                        double* bx, const int64_t* bxlo, const int64_t* bxhi, double* by,
                        const int64_t* bylo, const int64_t* byhi, double* bz,
                        const int64_t* bzlo, const int64_t* bzhi, double dtsdx, double dtsdy,
                        double dtsdz, void* stream) {
  (void)dtsdy;
  if (!ex || !ey || !ez || !bx || !by || !bz) return PXRB_EINVAL;
  Yee2Params p;
  if (yee2d_setup(p, xlo, xhi, ylo, yhi, zlo, zhi)) return PXRB_OK;
  p.ex = const_cast<double*>(ex); p.ey = const_cast<double*>(ey); p.ez = const_cast<double*>(ez);
  p.bx = bx; p.by = by; p.bz = bz;
  p.jx = p.jy = p.jz = nullptr;
  p.gex = g2_lohi(exlo, exhi); p.gey = g2_lohi(eylo, eyhi); p.gez = g2_lohi(ezlo, ezhi);
  p.gbx = g2_lohi(bxlo, bxhi); p.gby = g2_lohi(bylo, byhi); p.gbz = g2_lohi(bzlo, bzhi);
  p.mudt = 0; p.dtsdx = dtsdx; p.dtsdz = dtsdz;
  dim3 blk(32, 8, 1);
  dim3 grd((p.uhi[0] - p.ulo[0] + 1 + 31) / 32, (p.uhi[1] - p.ulo[1] + 1 + 7) / 8, 1);
  k_yee2d_b<<<grd, blk, 0, (cudaStream_t)stream>>>(p);
  PXRB_CHECK_LAUNCH();
  return PXRB_OK;
}

int pxrb_pushxz(int64_t np, double* xp, double* zp, const double* uxp, const double* uzp,
                const double* gaminv, double dt, void* stream) {
  if (np < 0) return PXRB_EINVAL;
  if (np == 0) return PXRB_OK;
  if (!xp || !zp || !uxp || !uzp || !gaminv) return PXRB_EINVAL;
  k_pushxz<<<nblocks(np), TPB, 0, (cudaStream_t)stream>>>(np, xp, zp, uxp, uzp, gaminv, dt);
  PXRB_CHECK_LAUNCH();
  return PXRB_OK;
}

int pxrb_particle_bcs_periodic(int64_t np, double* xp, double* yp, double* zp, double xmin,
                               double ymin, double zmin, double xmax, double ymax,
                               double zmax, void* stream) {
  if (np < 0) return PXRB_EINVAL;
  if (np == 0) return PXRB_OK;
  if (!xp || !yp || !zp) return PXRB_EINVAL;
  WrapParams p;
  p.np = np; p.x = xp; p.y = yp; p.z = zp;
  p.lo[0] = xmin; p.lo[1] = ymin; p.lo[2] = zmin;
  p.hi[0] = xmax; p.hi[1] = ymax; p.hi[2] = zmax;
  k_wrap<<<grid_stride_blocks(np), TPB, 0, (cudaStream_t)stream>>>(p);
  PXRB_CHECK_LAUNCH();
  return PXRB_OK;
}

}  // extern "C"
