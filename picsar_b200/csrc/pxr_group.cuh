// Warp-level gather and Esirkepov deposit of FP64 particles on the FP64 matrix
// instruction (mma.sync m8n8k4.f64).
//
// Particles are taken in groups that share the y and z base cell and whose x
// base cells lie in one run of C = 8 - ORDER cells, so that every stencil of
// the group falls on the same 8 x nodes (the matrix's columns) and the same
// ORDER+1 y and z nodes.  Both contractions are then small matrix products
// with the x shapes spread over the 8 columns (zero outside a particle's own
// nodes):
//   gather   T[p, i] = sum_(j,k) s_y(j) s_z(k) F(i, j, k),  E(p) = sum_i s_x(i) T[p, i]
//   deposit  Jx(i; j,k) += sum_p F_yz(j,k; p) C_x(i; p)
//            Jy(i; j,k) += sum_p [C_y(j) P_z(k)] s0_x(i) + [C_y(j) Q_z(k)] d_x(i)
//            Jz(i; j,k) += sum_p [C_z(k) P_y(j)] s0_x(i) + [C_z(k) Q_y(j)] d_x(i)
// with s0 / d the new shape and old minus new, C the prefix sums of d (the
// reference's W summed along the component's axis, esirkepov_3d.F90:198-233)
// and P = s0 + d/2, Q = s0/2 + d/3.  A group's field fragments stay in
// registers over all of its particles and its currents are summed in the
// accumulators, so a particle costs no window load and no atomic of its own.
//
// FP64 throughput bounds this: DMMA and DFMA share one pipe (37 TFLOP/s
// measured for either, and for both together).  At order 3 the gather takes
// 19 products of 8 particles and the deposit 8 products of 4: 608 + 512 FMA
// per particle, against about 400 useful ones; the alternative, one particle
// per thread, spends its time on 252 loads and 144 FP64 atomics instead.
#pragma once
#include "pxr_common.cuh"

namespace pxrg {

constexpr int COLS = 8;                       // x nodes of a group

template <int ORDER> struct Geom {
  static constexpr int N = ORDER + 1;         // node-centred support
  static constexpr int S = ORDER;             // staggered support (one order lower)
  static constexpr int A = ORDER / 2;         // first support node: base cell - A
  static constexpr int C = COLS - ORDER;      // x cells of a group
  static constexpr int FRAGS = N + 5 * S;     // field fragments of the gather
  static constexpr int XT = (N + 1) / 2;      // row tiles of Jx
  // gather record (doubles): y and z shapes, x shapes; odd, so that the 8-byte
  // stores of a half-warp go to distinct banks.
  static constexpr int GYZ = 17, GX = 9;
  // deposit record in 16-byte units: y and z (s0, d) pairs, x pairs on the
  // common box of N + 1 nodes, then the prefix sums.  An odd number of units:
  // the 16-byte stores of 8 lanes go to distinct banks (an even one made them
  // half of the shared-memory wavefronts), and 3 mod 8 leaves one conflict in
  // the 8 lanes' reads of 4 particles x 2 points.
  static constexpr int DU = ORDER == 1 ? 11 : 19;
  static constexpr int DZ = N, DX = 2 * N, DC = 2 * N + N + 1;    // unit offsets
  static constexpr int WARP_BYTES_GATHER = 32 * (GYZ + GX) * 8;
  static constexpr int WARP_BYTES_DEPOSIT = 32 * DU * 16;
  static constexpr int WARP_BYTES =
      WARP_BYTES_GATHER > WARP_BYTES_DEPOSIT ? WARP_BYTES_GATHER : WARP_BYTES_DEPOSIT;
};

__device__ __forceinline__ void dmma(double* c, double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1},{%2},{%3},{%0,%1};"
      : "+d"(c[0]), "+d"(c[1])
      : "d"(a), "d"(b));
}

// Field fragments of a group: at(comp, i, j, k) is the field at column i and
// support points j, k (0 where outside the array).
template <int ORDER> struct Frags {
  double ex[ORDER + 1], ey[ORDER], ez[ORDER], bx[ORDER], by[ORDER], bz[ORDER];
  template <class F> __device__ __forceinline__ void load(const F& at) {
    constexpr int N = ORDER + 1, S = ORDER;
    const int lane = threadIdx.x & 31, q = lane & 3, i = lane >> 2;
#pragma unroll
    for (int s = 0; s < N; ++s) ex[s] = q < N ? at(0, i, q, s) : 0.0;
#pragma unroll
    for (int s = 0; s < S; ++s) {
      ey[s] = q < N ? at(1, i, s, q) : 0.0;
      ez[s] = q < N ? at(2, i, q, s) : 0.0;
      bx[s] = q < S ? at(3, i, q, s) : 0.0;
      by[s] = q < N ? at(4, i, q, s) : 0.0;
      bz[s] = q < N ? at(5, i, s, q) : 0.0;
    }
  }
};

// E and B at the 32 particles of a warp (one per lane): shapes of the lane's
// particle, xo its x base cell within the group (0 .. C-1); the first
// 8 nsub lanes are served (the others get finite values).  buf: the warp's
// Geom::WARP_BYTES_GATHER bytes of shared memory.
template <int ORDER, class NS, class SS>
__device__ __forceinline__ void warp_gather(const Frags<ORDER>& f, double* buf, const NS& nx,
                                            const NS& ny, const NS& nz, const SS& sx,
                                            const SS& sy, const SS& sz, int xo, int nsub,
                                            double* eb) {
  typedef Geom<ORDER> G;
  constexpr int N = G::N, S = G::S;
  const int lane = threadIdx.x & 31, q = lane & 3;
  double* yz = buf;                           // [32][GYZ]: yN[4] zN[4] yS[3] zS[3]
  double* xw = buf + 32 * G::GYZ;             // [32][GX]:  xN[4] xS[4]
  {
    double* r = yz + lane * G::GYZ;
#pragma unroll
    for (int t = 0; t < N; ++t) { r[t] = ny.s[t]; r[4 + t] = nz.s[t]; }
#pragma unroll
    for (int t = 0; t < S; ++t) { r[8 + t] = sy.s[t]; r[12 + t] = sz.s[t]; }
    double* x = xw + lane * G::GX;
#pragma unroll
    for (int t = 0; t < N; ++t) x[t] = nx.s[t];
#pragma unroll
    for (int t = 0; t < S; ++t) x[4 + t] = sx.s[t];
  }
  __syncwarp();
#pragma unroll 1
  for (int sub = 0; sub < nsub; ++sub) {
    const int p = sub * 8 + (lane >> 2);
    const int xop = __shfl_sync(0xffffffffu, xo, p);
    const double* r = yz + p * G::GYZ;
    const double yq = q < N ? r[q] : 0.0, zq = q < N ? r[4 + q] : 0.0,
                 ysq = q < S ? r[8 + q] : 0.0;
    double c[6][2];
#pragma unroll
    for (int t = 0; t < 6; ++t) c[t][0] = c[t][1] = 0.0;
#pragma unroll
    for (int s = 0; s < N; ++s) dmma(c[0], yq * r[4 + s], f.ex[s]);
#pragma unroll
    for (int s = 0; s < S; ++s) {
      const double a = zq * r[8 + s], zs = r[12 + s], b = yq * zs;
      dmma(c[1], a, f.ey[s]);
      dmma(c[5], a, f.bz[s]);
      dmma(c[2], b, f.ez[s]);
      dmma(c[4], b, f.by[s]);
      dmma(c[3], ysq * zs, f.bx[s]);
    }
    // x weights of the columns 2q and 2q + 1
    const double* x = xw + p * G::GX;
    double wn[2], ws[2];
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      const int o = 2 * q + t - xop;
      wn[t] = (unsigned)o < (unsigned)N ? x[o] : 0.0;
      ws[t] = (unsigned)o < (unsigned)S ? x[4 + o] : 0.0;
    }
    const double e[3] = {c[0][0] * ws[0] + c[0][1] * ws[1], c[1][0] * wn[0] + c[1][1] * wn[1],
                         c[2][0] * wn[0] + c[2][1] * wn[1]};
    const double b[3] = {c[3][0] * wn[0] + c[3][1] * wn[1], c[4][0] * ws[0] + c[4][1] * ws[1],
                         c[5][0] * ws[0] + c[5][1] * ws[1]};
    // sum over the four lanes of a particle: even lanes keep E, odd ones B
    double k[3];
#pragma unroll
    for (int t = 0; t < 3; ++t) {
      const double mine = (q & 1) ? b[t] : e[t], other = (q & 1) ? e[t] : b[t];
      k[t] = mine + __shfl_xor_sync(0xffffffffu, other, 1);
      k[t] += __shfl_xor_sync(0xffffffffu, k[t], 2);
    }
    // the sub-batch's shapes have been read (the shuffles above follow the
    // reads of every lane): its records take the results
    if (q < 2) {
      double* o = yz + p * G::GYZ + 3 * q;
      o[0] = k[0]; o[1] = k[1]; o[2] = k[2];
    }
  }
  __syncwarp();
#pragma unroll
  for (int t = 0; t < 6; ++t) eb[t] = yz[lane * G::GYZ + t];
  __syncwarp();
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

  // Adds the warp's first 4 nsub particles.  X, Y, Z: the lane's particle on the common
  // box of its new and old nodes; y and z without a node change (box start at
  // the group's first node); xoff: column of X's box start; cx, cy, cz: the
  // particle's charge factors (0: no particle).  buf: the warp's
  // Geom::WARP_BYTES_DEPOSIT bytes of shared memory, 16-byte aligned.
  template <class AX>
  __device__ __forceinline__ void add(double* buf, const AX& X, const double* y0,
                                      const double* y1, const double* z0, const double* z1,
                                      int xoff, double cx, double cy, double cz,
                                      int nsub) {
    const int lane = threadIdx.x & 31, p = lane & 3, r = lane >> 2, t = r & 3, h = r >> 2;
    double2* rec = reinterpret_cast<double2*>(buf);
    {
      double2* o = rec + lane * G::DU;
      double* c = reinterpret_cast<double*>(o + G::DC);    // Cy[S] Cz[S] Cx[N]
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
    __syncwarp();
    const double third = 1.0 / 3.0;
#pragma unroll 1
    for (int sub = 0; sub < nsub; ++sub) {
      const int pp = sub * 4 + p;
      const int xo = __shfl_sync(0xffffffffu, xoff, pp);
      const double2* o = rec + pp * G::DU;
      const double* c = reinterpret_cast<const double*>(o + G::DC);
      // columns: the x values of particle p at node r
      const int ix = r - xo;
      const double bC = (unsigned)ix < (unsigned)N ? c[2 * S + ix] : 0.0;
      double2 bx = make_double2(0.0, 0.0);
      if ((unsigned)ix < (unsigned)(N + 1)) bx = o[G::DX + ix];
      const bool tv = t < N;
      double2 y = make_double2(0.0, 0.0), z = y;
      if (tv) { y = o[t]; z = o[G::DZ + t]; }
      const double Py = y.x + 0.5 * y.y, Qy = 0.5 * y.x + third * y.y;
      const double Pz = z.x + 0.5 * z.y, Qz = 0.5 * z.x + third * z.y;
#pragma unroll
      for (int m = 0; m < G::XT; ++m) {
        const int k = h + 2 * m;
        double2 zk = make_double2(0.0, 0.0);
        if (2 * m + 1 < N || k < N) zk = o[G::DZ + k];
        dmma(jx[m], Py * zk.x + Qy * zk.y, bC);
      }
      if (S >= 2) {
        const double cy = c[h], cz = c[S + h];
        dmma(ja, cy * Pz, bx.x);
        dmma(ja, cy * Qz, bx.y);
        dmma(jb, cz * Py, bx.x);
        dmma(jb, cz * Qy, bx.y);
      }
      if (S & 1) {
        const double cm = c[h * S + S - 1];
        dmma(jm, cm * (h ? Py : Pz), bx.x);
        dmma(jm, cm * (h ? Qy : Qz), bx.y);
      }
    }
    __syncwarp();
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
      if (S >= 2) {
        put(1, i, h, t, ja[e]);
        put(2, i, t, h, jb[e]);
      }
      if (S & 1) {
        if (h) put(2, i, t, S - 1, jm[e]);
        else put(1, i, S - 1, t, jm[e]);
      }
    }
  }
};

}  // namespace pxrg
