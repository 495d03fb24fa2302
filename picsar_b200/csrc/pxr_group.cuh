// Warp-level Esirkepov deposit of FP64 particles on the FP64 matrix instruction
// (mma.sync m8n8k4.f64).
//
// Particles are taken in groups that share the y and z base cell and whose x
// base cells lie in one run of C = 8 - ORDER cells, so that every stencil of
// the group falls on the same 8 x nodes (the matrix's columns) and the same
// ORDER+1 y and z nodes.  The deposit is then a product over the particles
// with the x shapes spread over the 8 columns (zero outside a particle's own
// nodes):
//   Jx(i; j,k) += sum_p F_yz(j,k; p) C_x(i; p)
//   Jy(i; j,k) += sum_p [C_y(j) P_z(k)] s0_x(i) + [C_y(j) Q_z(k)] d_x(i)
//   Jz(i; j,k) += sum_p [C_z(k) P_y(j)] s0_x(i) + [C_z(k) Q_y(j)] d_x(i)
// with s0 / d the new shape and old minus new, C the prefix sums of d (the
// reference's W summed along the component's axis, esirkepov_3d.F90:198-233)
// and P = s0 + d/2, Q = s0/2 + d/3.  A group's currents are summed in the
// accumulators, so a particle costs no atomic of its own.
//
// At order 3 four particles take 8 products: 512 FMA per particle against
// about 200 useful ones, on a pipe that DMMA and DFMA share (37 TFLOP/s
// measured for either).  The same products for the gather (fields as the
// other operand, 19 per 8 particles) were slower than loads by one thread per
// particle: the fragments, their reduction over the columns and the trip back
// to the particle's own lane cost more than 252 cached loads.
#pragma once
#include "pxr_common.cuh"

namespace pxrg {

constexpr int COLS = 8;                       // x nodes of a group

template <int ORDER> struct Geom {
  static_assert(ORDER == 2 || ORDER == 3, "two or three staggered nodes per axis");
  static constexpr int N = ORDER + 1;         // node-centred support
  static constexpr int S = ORDER;             // staggered support (one order lower)
  static constexpr int A = ORDER / 2;         // first support node: base cell - A
  static constexpr int C = COLS - ORDER;      // x cells of a group
  static constexpr int XT = (N + 1) / 2;      // row tiles of Jx
  // a particle's record in 16-byte units: y and z (s0, d) pairs, x pairs on the
  // common box of N + 1 nodes, then the prefix sums.  An odd number of units:
  // the 16-byte stores of 8 lanes go to distinct banks (an even one made them
  // half of the shared-memory wavefronts), and 3 mod 8 leaves one conflict in
  // the 8 lanes' reads of 4 particles x 2 points.
  static constexpr int DU = 19;
  static constexpr int DZ = N, DX = 2 * N, DC = 2 * N + N + 1;    // unit offsets
  static constexpr int WARP_BYTES = 32 * DU * 16;
};

__device__ __forceinline__ void dmma(double* c, double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1},{%2},{%3},{%0,%1};"
      : "+d"(c[0]), "+d"(c[1])
      : "d"(a), "d"(b));
}

// Currents of a group, summed over its particles.
template <int ORDER> struct Currents {
  typedef Geom<ORDER> G;
  static constexpr int N = G::N, S = G::S;
  double jx[G::XT][2], ja[2], jb[2], jm[2];
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int m = 0; m < G::XT; ++m) jx[m][0] = jx[m][1] = 0.0;
    ja[0] = ja[1] = jb[0] = jb[1] = jm[0] = jm[1] = 0.0;
  }

  // Writes the shapes of the lane's particle for sub().  X: its new and old x
  // nodes on their common box; y and z: new and old shapes without a node
  // change (first node the group's); cx, cy, cz: charge factors (0: no
  // particle, with finite shapes).  buf: the warp's
  // Geom::WARP_BYTES bytes of shared memory, 16-byte aligned; a
  // __syncwarp follows.
  template <class AX>
  __device__ __forceinline__ static void stage(double* buf, const AX& X, const double* y0,
                                               const double* y1, const double* z0,
                                               const double* z1, double cx, double cy, double cz) {
    double2* o = reinterpret_cast<double2*>(buf) + (threadIdx.x & 31) * G::DU;
    double* c = reinterpret_cast<double*>(o + G::DC);      // Cy[S] Cz[S] Cx[N]
    double sy = 0.0, sz = 0.0, sx = 0.0;
#pragma unroll
    for (int u = 0; u < N; ++u) {
      const double dy = y1[u] - y0[u], dz = z1[u] - z0[u];
      o[u] = make_double2(y0[u], dy);
      o[G::DZ + u] = make_double2(z0[u], dz);
      if (u < S) {
        sy += dy; sz += dz;
        c[u] = sy * cy;
        c[S + u] = sz * cz;
      }
    }
#pragma unroll
    for (int u = 0; u < N + 1; ++u) {
      const double dx = X.s1[u] - X.s0[u];
      o[G::DX + u] = make_double2(X.s0[u], dx);
      if (u < N) {
        sx += dx;
        c[2 * S + u] = u < X.n - 1 ? sx * cx : 0.0;
      }
    }
  }

  // Adds the warp's particles 4 sub .. 4 sub + 3, all of this group.  xoff:
  // column of the lane's own particle's x box.
  __device__ __forceinline__ void sub(const double* buf, int sub, int xoff) {
    const int lane = threadIdx.x & 31, r = lane >> 2, t = r & 3, h = r >> 2;
    const int pp = sub * 4 + (lane & 3);
    const int xo = __shfl_sync(0xffffffffu, xoff, pp);
    const double third = 1.0 / 3.0;
    const double2* o = reinterpret_cast<const double2*>(buf) + pp * G::DU;
    const double* c = reinterpret_cast<const double*>(o + G::DC);
    // columns: the x values of the particle at node r
    const int ix = r - xo;
    const double bC = (unsigned)ix < (unsigned)N ? c[2 * S + ix] : 0.0;
    double2 bx = make_double2(0.0, 0.0);
    if ((unsigned)ix < (unsigned)(N + 1)) bx = o[G::DX + ix];
    double2 y = make_double2(0.0, 0.0), z = y;
    if (t < N) { y = o[t]; z = o[G::DZ + t]; }
    const double Py = y.x + 0.5 * y.y, Qy = 0.5 * y.x + third * y.y;
    const double Pz = z.x + 0.5 * z.y, Qz = 0.5 * z.x + third * z.y;
#pragma unroll
    for (int m = 0; m < G::XT; ++m) {
      const int k = h + 2 * m;
      double2 zk = make_double2(0.0, 0.0);
      if (2 * m + 1 < N || k < N) zk = o[G::DZ + k];
      dmma(jx[m], Py * zk.x + Qy * zk.y, bC);
    }
    const double cy = c[h], cz = c[S + h];
    dmma(ja, cy * Pz, bx.x);
    dmma(ja, cy * Qz, bx.y);
    dmma(jb, cz * Py, bx.x);
    dmma(jb, cz * Qy, bx.y);
    if (S & 1) {
      const double cm = c[h * S + S - 1];
      dmma(jm, cm * (h ? Py : Pz), bx.x);
      dmma(jm, cm * (h ? Qy : Qz), bx.y);
    }
  }

  // put(comp, i, j, k, v): v to component comp at column i and support
  // points j, k.
  template <class F> __device__ __forceinline__ void flush(const F& put) const {
    const int lane = threadIdx.x & 31, q = lane & 3, r = lane >> 2, t = r & 3, h = r >> 2;
    if (t >= N) return;
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int i = 2 * q + e;
#pragma unroll
      for (int m = 0; m < G::XT; ++m)
        if (2 * m + 1 < N || h + 2 * m < N) put(0, i, t, h + 2 * m, jx[m][e]);
      put(1, i, h, t, ja[e]);
      put(2, i, t, h, jb[e]);
      if (S & 1) {
        if (h) put(2, i, t, S - 1, jm[e]);
        else put(1, i, S - 1, t, jm[e]);
      }
    }
  }
};

}  // namespace pxrg
