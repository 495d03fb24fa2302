// The FP64 engine's fused particle kernel: a tile's particles taken in group
// order, one thread each for gather, push and position, then the Esirkepov
// deposit by groups on the FP64 matrix instruction (pxr_group.cuh).
//
// The one-pass kernel (k_tile_step) makes 252 8-byte window loads (two
// wavefronts each) and 144 FP64 shared atomics (about five) per particle at
// order 3, which keep the shared-memory pipe 69 % busy.  Here a tile's
// particles are counted into groups every step (one y and z base cell, a run
// of x cells).  In that order the lanes of a warp read the same few window
// elements, one wavefront a load, and a group's currents are added to the
// tile's J window once per eight or more particles: 8.4 M particles at 8 per cell 3.73 ->
// 2.95 ms, at 2 per cell (2.1 M) 1.31 -> 1.07 ms; at 1 per cell, not grouped,
// 0.86 -> 0.68 ms.  What is left is latency: the warps' records leave room for
// one CTA of 512 threads per SM, whose phases do not overlap, and for 28 KB of
// L1, which particles outside their window miss (four fifths of them outside,
// 8 per cell at 64^3: 12.0 ms against the one-pass kernel's 9.1; a plasma that
// hot wants a shorter sort interval).
// Orders 1 and 2 stay with k_tile_step (0.66 and 1.73 ms against 1.43 and 2.6
// here): their 12 and 54 atomics cost less than the extra passes.
#pragma once
#include "pxr_tiled_kernel.cuh"
#include "pxr_group.cuh"

namespace pxrt {

template <int ORDER, int T, int D> struct TileGroups {
  typedef pxrg::Geom<ORDER> G;
  static constexpr int L = Reach<ORDER>::L, H = Reach<ORDER>::H;
  static constexpr int W = T + 2 * D + L + H, SY = win_sy(T, W), SZ = win_sz(T, W), V = SZ * W;
  static_assert(L == G::A, "the window starts at the first cell's first node");
  static constexpr int NB = T + 2 * D;                       // base cells per axis
  static constexpr int NG = (NB + G::C - 1) / G::C;          // groups along x
  static constexpr int NKEY = NG * NB * NB;                  // and one more: outside the window
  // Window particles per key below which a tile is not grouped.  Edge 8, margin
  // 1, 512 threads, particle by particle / grouped: 0.68 / 0.91 ms at 1 per
  // cell (2.6 per key), 1.21 / 1.08 ms at 2 (128x128x64 cells).  Edge 4 gains
  // from the groups at any density (1 per cell, 256 threads 1.79 / 1.45 ms).
  static constexpr int THIN = T == 8 ? 4 : 0;
  // the E/B window of the gather, then in its place the J window and a record
  // per lane of the launch's warps (edge 4 with 256 threads: 100,880 bytes, two
  // CTAs per SM; records for 16 warps in any launch left it one)
  static constexpr int OFF_WIN = (2 * (NKEY + 2) * 4 + 15) / 16 * 16;
  static constexpr int OFF_BUF = OFF_WIN + (3 * V * 8 + 15) / 16 * 16;
  static constexpr int END_F = OFF_WIN + 6 * V * 8;
  static constexpr int smem(int threads) {
    const int end_j = OFF_BUF + threads / 32 * G::WARP_BYTES;
    return end_j > END_F ? end_j : END_F;
  }
};

// The current of a move from cell (ci, cj, ck), offsets o, by s cells to
// offsets n, by global atomics (values only: arrays passed by address would
// keep the caller's in local memory).  A move of more than one node (a step
// beyond the CFL limit) sets the error flag.
template <int ORDER>
__device__ __noinline__ void deposit_outside(const Job& J, int ci, int cj, int ck, int sx, int sy,
                                             int sz, double ox, double oy, double oz, double nox,
                                             double noy, double noz, double wgt) {
  typedef double R;
  int r0, r1;
  R a0, a1;
  EsirAxis<ORDER, R> EX, EY, EZ;
  esir_node<ORDER, R>(nox, r0, a0); esir_node<ORDER, R>(ox, r1, a1);
  bool ok = EX.set(ci + sx + r0, a0, ci + r1, a1);
  esir_node<ORDER, R>(noy, r0, a0); esir_node<ORDER, R>(oy, r1, a1);
  ok = EY.set(cj + sy + r0, a0, cj + r1, a1) && ok;
  esir_node<ORDER, R>(noz, r0, a0); esir_node<ORDER, R>(oz, r1, a1);
  ok = EZ.set(ck + sz + r0, a0, ck + r1, a1) && ok;
  if (!ok) atomicExch(&J.counters[1], 1);
  dep_global<ORDER, R>(J, EX, EY, EZ, wgt * (J.q / (J.dt * J.dy * J.dz)),
                       wgt * (J.q / (J.dt * J.dx * J.dz)), wgt * (J.q / (J.dt * J.dx * J.dy)));
}

template <int ORDER, int T, int D>
__global__ void __launch_bounds__(MAX_THREADS_FP64, 1)
    k_tile_group(const Job* __restrict__ jobs, const int2* __restrict__ work, int nwork,
                 const int* __restrict__ nwork_dev, int* ctr) {
  typedef double R;
  typedef TileGroups<ORDER, T, D> TG;
  typedef pxrg::Geom<ORDER> GE;
  typedef EsirAxis<ORDER, R> AX;
  constexpr int SY = TG::SY, SZ = TG::SZ, V = TG::V, W = TG::W, NB = TG::NB, NG = TG::NG;
  constexpr int NKEY = TG::NKEY, C = GE::C, A = GE::A;
  static_assert(ORDER == 3, "a particle's base cell is the cell that holds it");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  int* start = reinterpret_cast<int*>(smem_raw);                   // counts, then starts
  int* first = start + NKEY + 2;                                   // first octet of a key
  double* Fs = reinterpret_cast<double*>(smem_raw + TG::OFF_WIN);
  double* Js = Fs;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  double* buf = reinterpret_cast<double*>(smem_raw + TG::OFF_BUF + wid * GE::WARP_BYTES);
  __shared__ Job sj;
  __shared__ int s_item, s_qn, s_key, s_grouped;
  __shared__ double s_red[MAX_WARPS];

  if (nwork_dev) nwork = min(nwork, *nwork_dev);
  for (;;) {
    if (threadIdx.x == 0) {
      s_item = atomicAdd(ctr, 1);
      s_qn = 0;
      s_key = 0;
    }
    __syncthreads();
    const int item = s_item;
    if (item >= nwork) break;
    const int2 wk = work[item];
    {
      const int nw = (int)(sizeof(Job) / sizeof(int));
      const int* src = reinterpret_cast<const int*>(jobs + wk.x);
      int* dst = reinterpret_cast<int*>(&sj);
      for (int t = threadIdx.x; t < nw; t += blockDim.x) dst[t] = src[t];
    }
    for (int e = threadIdx.x; e < NKEY + 2; e += blockDim.x) start[e] = 0;
    __syncthreads();
    const int nx = sj.nx, ny = sj.ny, nz = sj.nz, G = sj.g;
    const int tile = wk.y;
    const int ti = tile % sj.ntx, tj = (tile / sj.ntx) % sj.nty, tk = tile / (sj.ntx * sj.nty);
    const int c0x = ti * T, c0y = tj * T, c0z = tk * T;
    const int tex = min(T, nx - c0x), tey = min(T, ny - c0y), tez = min(T, nz - c0z);
    const int pbeg = sj.tile_off[tile], pend = sj.tile_off[tile + 1];
    uint32_t* cellp = sj.cell;
    R *oxp = (R*)sj.ox, *oyp = (R*)sj.oy, *ozp = (R*)sj.oz;
    // cell relative to the tile, periodic; false outside the window
    auto local = [&](uint32_t c, int& vx, int& vy, int& vz) {
      int ci, cj, ck;
      unpack_cell(c, ci, cj, ck);
      vx = ci - c0x; vy = cj - c0y; vz = ck - c0z;
      if (vx > tex - 1 + D) vx -= nx; else if (vx < -D) vx += nx;
      if (vy > tey - 1 + D) vy -= ny; else if (vy < -D) vy += ny;
      if (vz > tez - 1 + D) vz -= nz; else if (vz < -D) vz += nz;
      return vx >= -D && vx <= tex - 1 + D && vy >= -D && vy <= tey - 1 + D && vz >= -D &&
             vz <= tez - 1 + D;
    };
    // ---- stage the E/B window: asynchronous copies, in flight while the
    // particles are counted ------------------------------------------------------
    {
      const int pitch = sj.pitch_x, NYg = sj.pitch_y;
      const i64 base0 = (i64)(c0x - D - A + G) +
                        (i64)pitch * ((c0y - D - A + G) + (i64)NYg * (c0z - D - A + G));
#pragma unroll 1
      for (int comp = 0; comp < 6; ++comp) {
        const R* src = (const R*)(comp == 0 ? sj.ex : comp == 1 ? sj.ey : comp == 2 ? sj.ez
                                 : comp == 3 ? sj.bx : comp == 4 ? sj.by : sj.bz) + base0;
        const uint32_t dst = (uint32_t)__cvta_generic_to_shared(Fs + comp * V);
        for (int r = threadIdx.x; r < W * W * W; r += blockDim.x) {
          const int a = r % W, b = (r / W) % W, c = r / (W * W);
          const R* g = src + a + (i64)pitch * (b + (i64)NYg * c);
          const uint32_t d = dst + (uint32_t)((a + b * SY + c * SZ) * sizeof(R));
          asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(g));
        }
      }
      asm volatile("cp.async.commit_group;\n" ::);
    }
    // ---- groups: count (rank kept), prefix, placement; a thin tile and one
    // that many particles have left is taken in storage order, its deposit by
    // the queue ------------------------------------------------------------------
    // scratch free between sorts: rank_b (ranks, then the queue's list),
    // cell_b (keys, then the queue's boxes), perm (particles in group order)
    int *rank = sj.rank_b, *perm = sj.perm;
    uint32_t* keys = sj.cell_b;
    const bool dense = pend - pbeg >= TG::THIN * NKEY;
    for (int ip = pbeg + threadIdx.x; dense && ip < pend; ip += blockDim.x) {
      int vx, vy, vz, key = NKEY;
      if (local(cellp[ip], vx, vy, vz)) key = (vx + D) / C + NG * (vy + D + NB * (vz + D));
      keys[ip] = (uint32_t)key;
      rank[ip] = atomicAdd(start + key, 1);
    }
    __syncthreads();
    if (wid == 0) {
      // particles before a key, and its octets (the matrix products take eight
      // particles of one key; a batch holds four octets of any keys)
      int run = 0, oct = 0;
      for (int b = 0; b <= NKEY; b += 32) {
        const int k = b + lane, v = k <= NKEY ? start[k] : 0, w = k < NKEY ? (v + 7) >> 3 : 0;
        int inc = v, ino = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int u = __shfl_up_sync(0xffffffffu, inc, o);
          const int x = __shfl_up_sync(0xffffffffu, ino, o);
          if (lane >= o) { inc += u; ino += x; }
        }
        if (k <= NKEY) { start[k] = run + inc - v; first[k] = oct + ino - w; }
        run += __shfl_sync(0xffffffffu, inc, 31);
        oct += __shfl_sync(0xffffffffu, ino, 31);
      }
      __syncwarp();
      if (lane == 0) {
        // start[NKEY]: particles in the window.  Those outside read and add to
        // global memory, in storage order with better locality than in the
        // groups': with a quarter of them outside 16.8 / 15.6 ms (8 per cell,
        // 64^3), with a third 16.7 / 11.3, with a sixth 16.3 / 19
        s_grouped = dense && start[NKEY] >= TG::THIN * NKEY && 5 * start[NKEY] >= 4 * run;
        start[NKEY + 1] = run;
        first[NKEY] = s_grouped ? oct : 0;
      }
    }
    __syncthreads();
    for (int ip = pbeg + threadIdx.x; s_grouped && ip < pend; ip += blockDim.x)
      perm[pbeg + start[keys[ip]] + rank[ip]] = ip;
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    __syncthreads();
    // ---- particles -----------------------------------------------------------
    const R dtdx = sj.dt / sj.dx, dtdy = sj.dt / sj.dy, dtdz = sj.dt / sj.dz;
    const R clghtisq = 1.0 / (sj.clight * sj.clight);
    const R cst_b = sj.q * sj.dt * 0.5 / sj.m, cst_v = sj.q * sj.dt / sj.m;
    const R qdx = sj.q / (sj.dt * sj.dy * sj.dz), qdy = sj.q / (sj.dt * sj.dx * sj.dz),
            qdz = sj.q / (sj.dt * sj.dx * sj.dy);
    const bool vay = sj.pusher == 1;
    R *uxp = (R*)sj.ux, *uyp = (R*)sj.uy, *uzp = (R*)sj.uz;
    const R* wp = (const R*)sj.w;
    int* q_list = sj.rank_b;
    uint32_t* q_pk = sj.cell_b;
    R *q_ox = (R*)sj.ox_b, *q_oy = (R*)sj.oy_b, *q_oz = (R*)sj.oz_b;
    double ke = 0.0;
    int bad = 0;
    // gather, push, position, store.  A window particle's box and old offsets
    // stay in the scratch for the deposit (cell_b, ox_b .. oz_b); the others
    // deposit here and are marked done.
    constexpr unsigned DONE = 1u << 31;
    {
      for (int s = threadIdx.x; s < pend - pbeg; s += blockDim.x) {
        const int ip = s_grouped ? perm[pbeg + s] : pbeg + s;
        const uint32_t cell = cellp[ip];
        const R ox = oxp[ip], oy = oyp[ip], oz = ozp[ip];
        int ci, cj, ck, vx, vy, vz;
        unpack_cell(cell, ci, cj, ck);
        const bool in_old = local(cell, vx, vy, vz);
        R eb[6];
        if (in_old) {
          NodeCO<ORDER, R> nxs, nys, nzs;
          StagCO<ORDER, R> sxs, sys, szs;
          nxs.set(ox); nys.set(oy); nzs.set(oz);
          sxs.set(ox); sys.set(oy); szs.set(oz);
          constexpr int N = GE::N, S = GE::S;
          const R* F0 = Fs + (vx + D + A) + (vy + D + A) * SY + (vz + D + A) * SZ;
          eb[0] = gwin<S, N, N, SY, SZ>(F0 + sxs.r0 + nys.r0 * SY + nzs.r0 * SZ,
                            sxs.s, nys.s, nzs.s);
          eb[1] = gwin<N, S, N, SY, SZ>(F0 + V + nxs.r0 + sys.r0 * SY + nzs.r0 * SZ,
                            nxs.s, sys.s, nzs.s);
          eb[2] = gwin<N, N, S, SY, SZ>(F0 + 2 * V + nxs.r0 + nys.r0 * SY + szs.r0 * SZ,
                            nxs.s, nys.s, szs.s);
          eb[3] = gwin<N, S, S, SY, SZ>(F0 + 3 * V + nxs.r0 + sys.r0 * SY + szs.r0 * SZ,
                            nxs.s, sys.s, szs.s);
          eb[4] = gwin<S, N, S, SY, SZ>(F0 + 4 * V + sxs.r0 + nys.r0 * SY + szs.r0 * SZ,
                            sxs.s, nys.s, szs.s);
          eb[5] = gwin<S, S, N, SY, SZ>(F0 + 5 * V + sxs.r0 + sys.r0 * SY + nzs.r0 * SZ,
                            sxs.s, sys.s, nzs.s);
        } else {
          gather_global<ORDER, R>(sj, ci, cj, ck, ox, oy, oz, eb);
        }
        R ux = uxp[ip], uy = uyp[ip], uz = uzp[ip], gi;
        const R wgt = wp[ip];
        if (vay) {
          gi = inv_sqrt<R>(1.0 + (ux * ux + uy * uy + uz * uz) * clghtisq);
          vay_push(ux, uy, uz, gi, eb[0], eb[1], eb[2], eb[3], eb[4], eb[5], cst_v,
                   1.0 / sj.clight, clghtisq);
        } else {
          boris_push(ux, uy, uz, gi, eb[0], eb[1], eb[2], eb[3], eb[4], eb[5], cst_b, clghtisq);
        }
        R nox = ox, noy = oy, noz = oz;
        int sx = 0, sy = 0, sz = 0;
        cell_step(nox, sx, ux * gi * dtdx);
        cell_step(noy, sy, uy * gi * dtdy);
        cell_step(noz, sz, uz * gi * dtdz);
        cellp[ip] = pack_cell(GlobAcc::wrap(ci + sx, nx), GlobAcc::wrap(cj + sy, ny),
                              GlobAcc::wrap(ck + sz, nz));
        oxp[ip] = nox; oyp[ip] = noy; ozp[ip] = noz;
        uxp[ip] = ux; uyp[ip] = uy; uzp[ip] = uz;
        const R u2 = (ux * ux + uy * uy + uz * uz) * clghtisq;
        ke += u2 / (1.0 + sqrt(u2 + 1.0)) * wgt;
        const bool in_new = in_old && vx + sx >= -D && vx + sx <= tex - 1 + D && vy + sy >= -D &&
                            vy + sy <= tey - 1 + D && vz + sz >= -D && vz + sz <= tez - 1 + D;
        // the box word holds shifts of -1, 0 and 1: a longer move is deposited
        // here, which flags it
        const bool packs = sx >= -1 && sx <= 1 && sy >= -1 && sy <= 1 && sz >= -1 && sz <= 1;
        if (in_new && packs) {
          q_pk[ip] = (unsigned)(vx + D + A) | ((unsigned)(vy + D + A) << 8) |
                     ((unsigned)(vz + D + A) << 16) | ((unsigned)(sx + 1) << 24) |
                     ((unsigned)(sy + 1) << 26) | ((unsigned)(sz + 1) << 28);
          q_ox[ip] = ox; q_oy[ip] = oy; q_oz[ip] = oz;
          if (!s_grouped) q_list[pbeg + atomicAdd(&s_qn, 1)] = ip;
        } else {
          q_pk[ip] = DONE;
          if (!in_new) atomicAdd(&sj.counters[0], 1);
          // a window particle's cell counted from its tile: its nodes before
          // and after the move are then at most one period outside the grid
          deposit_outside<ORDER>(sj, in_new ? c0x + vx : ci, in_new ? c0y + vy : cj,
                                 in_new ? c0z + vz : ck, sx, sy, sz, ox, oy, oz, nox, noy, noz,
                                 wgt);
        }
      }
    }
    __syncthreads();
    for (int e = threadIdx.x; e < 3 * V; e += blockDim.x) Js[e] = 0.0;
    __syncthreads();
    // ---- deposit by groups: in the group unless the y or z node changes or
    // the x box leaves the group's columns -------------------------------------
    const int noct = first[NKEY];
    for (;;) {
      int batch = 0;
      if (lane == 0) batch = atomicAdd(&s_key, 1);
      batch = __shfl_sync(0xffffffffu, batch, 0);
      if (4 * batch >= noct) break;
      const int nsub = min(4, noct - 4 * batch);
      // the lane's octet, its key (the last whose first octet is not past it;
      // empty keys share their first octet with the next) and particle
      const int oct = min(4 * batch + (lane >> 3), noct - 1);
      int key = 0;
      {
        int hi = NKEY;
        while (hi - key > 1) {
          const int mid = (key + hi) >> 1;
          if (first[mid] <= oct) key = mid; else hi = mid;
        }
      }
      const int x0c = (key % NG) * C;
      const int at = start[key] + (oct - first[key]) * 8 + (lane & 7);
      const bool valid = (lane >> 3) < nsub && at < start[key + 1];
      const int ip = perm[pbeg + (valid ? at : start[key])];
      const unsigned pk = q_pk[ip];
      const R ox = q_ox[ip], oy = q_oy[ip], oz = q_oz[ip];
      const R nox = oxp[ip], noy = oyp[ip], noz = ozp[ip], wgt = wp[ip];
      const int sx = (int)((pk >> 24) & 3u) - 1, sy = (int)((pk >> 26) & 3u) - 1,
                sz = (int)((pk >> 28) & 3u) - 1;
      int r0x, r1x, r0y, r1y, r0z, r1z;
      R x0, x1, y0, y1, z0, z1;
      esir_node<ORDER, R>(nox, r0x, x0); esir_node<ORDER, R>(ox, r1x, x1);
      esir_node<ORDER, R>(noy, r0y, y0); esir_node<ORDER, R>(oy, r1y, y1);
      esir_node<ORDER, R>(noz, r0z, z0); esir_node<ORDER, R>(oz, r1z, z1);
      const int xo = (int)(pk & 255u) - A + r1x, xn = xo - r1x + sx + r0x;   // base cells
      AX X;
      const bool okx = X.set(xn, x0, xo, x1);
      const bool todo = valid && !(pk & DONE);
      // (what is not finite keeps to the particle's own nodes in the queue: the
      // products spread a group's operands over all of its nodes)
      const R cx = wgt * qdx, cy = wgt * qdy, cz = wgt * qdz;
      const bool fin = isfinite(x0 + x1 + y0 + y1 + z0 + z1) &&
                       isfinite(fabs(cx) + fabs(cy) + fabs(cz));
      const bool fast = todo && okx && fin && sy + r0y == r1y && sz + r0z == r1z &&
                        (unsigned)(xn - x0c) < (unsigned)C;
      if (todo && !fast) q_list[pbeg + atomicAdd(&s_qn, 1)] = ip;
      R sy0[GE::N], sy1[GE::N], sz0[GE::N], sz1[GE::N];
      AX::shape(y0, sy0); AX::shape(y1, sy1);
      AX::shape(z0, sz0); AX::shape(z1, sz1);
      if (!fast) {
        // no contribution: finite shapes times zero charge
#pragma unroll
        for (int t = 0; t < GE::N; ++t) sy0[t] = sy1[t] = sz0[t] = sz1[t] = 0.0;
#pragma unroll
        for (int t = 0; t < GE::N + 1; ++t) X.s0[t] = X.s1[t] = 0.0;
      }
      pxrg::Currents<ORDER> J;
      J.stage(buf, X, sy0, sy1, sz0, sz1, fast ? cx : 0.0, fast ? cy : 0.0, fast ? cz : 0.0);
      __syncwarp();
      const int xoff = X.i0 + A - x0c;
      J.clear();
#pragma unroll 1
      for (int sub = 0; sub < 2 * nsub; ++sub) {
        J.sub(buf, sub, xoff);
        const int k = __shfl_sync(0xffffffffu, key, sub * 4);
        const int kn = __shfl_sync(0xffffffffu, key, min(sub * 4 + 4, 31));
        if (sub == 2 * nsub - 1 || kn != k) {
          const int col = (k % NG) * C;
          double* base = Js + col + ((k / NG) % NB) * SY + (k / (NG * NB)) * SZ;
          J.flush([&](int c, int i, int j, int l, double v) {
            if (v != 0.0 && col + i < W) atomicAdd(base + c * V + i + j * SY + l * SZ, v);
          });
          J.clear();
        }
      }
      __syncwarp();
    }
    __syncthreads();
    // ---- window particles with a node change ---------------------------------
    for (int q = threadIdx.x; q < s_qn; q += blockDim.x) {
      const int ip = q_list[pbeg + q];
      const unsigned pk = q_pk[ip];
      const int bx = pk & 255u, by = (pk >> 8) & 255u, bz = (pk >> 16) & 255u;
      const int sx = (int)((pk >> 24) & 3u) - 1, sy = (int)((pk >> 26) & 3u) - 1,
                sz = (int)((pk >> 28) & 3u) - 1;
      const R ox = q_ox[ip], oy = q_oy[ip], oz = q_oz[ip];
      const R nox = oxp[ip], noy = oyp[ip], noz = ozp[ip], wq = wp[ip];
      int r0, r1;
      R a0, a1;
      AX EX, EY, EZ;
      esir_node<ORDER, R>(nox, r0, a0); esir_node<ORDER, R>(ox, r1, a1);
      bool ok = EX.set(bx + sx + r0, a0, bx + r1, a1);
      esir_node<ORDER, R>(noy, r0, a0); esir_node<ORDER, R>(oy, r1, a1);
      ok = EY.set(by + sy + r0, a0, by + r1, a1) && ok;
      esir_node<ORDER, R>(noz, r0, a0); esir_node<ORDER, R>(oz, r1, a1);
      ok = EZ.set(bz + sz + r0, a0, bz + r1, a1) && ok;
      if (!ok) bad = 1;
      dep_window<ORDER, R, 3, SY, SZ, V>(Js, EX, EY, EZ, wq * qdx, wq * qdy, wq * qdz);
    }
    __syncthreads();
    // ---- flush the J window: FP64 atomics into the periodic grid -------------
    {
      const int wox = c0x - D - A, woy = c0y - D - A, woz = c0z - D - A;
#pragma unroll 1
      for (int comp = 0; comp < 3; ++comp) {
        double* dst = comp == 0 ? sj.jx : comp == 1 ? sj.jy : sj.jz;
        const double* src = Js + comp * V;
        for (int r = threadIdx.x; r < V; r += blockDim.x) {
          const double v = src[r];
          if (v == 0.0) continue;               // includes the pitch padding
          const int c = r / SZ, b = (r - c * SZ) / SY, a = r - c * SZ - b * SY;
          const int gi = GlobAcc::wrap(wox + a, nx), gj = GlobAcc::wrap(woy + b, ny),
                    gk = GlobAcc::wrap(woz + c, nz);
          atomicAdd(dst + gi + (i64)nx * (gj + (i64)ny * gk), v);
        }
      }
    }
    // ---- kinetic energy of the tile ------------------------------------------
    {
      double v = ke;
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
      if (lane == 0) s_red[wid] = v;
      if (bad) atomicExch(&sj.counters[1], 1);
      __syncthreads();
      if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < nwarps; ++w) t += s_red[w];
        sj.ke_tile[tile] = t * sj.m * sj.clight * sj.clight;
      }
    }
    __syncthreads();
  }
}

template <int ORDER, int T, int D>
int launch_group(const Job* jobs, const int2* work, int nwork, const int* nwork_dev, int* ctr,
                 int threads, int ctas, size_t smem, cudaStream_t s) {
  auto kern = k_tile_group<ORDER, T, D>;
  typedef TileGroups<ORDER, T, D> TG;
  const int need = TG::smem(threads);
  if (smem < (size_t)need) return PXRB_EINVAL;
  // the limit of the largest launch, whatever this one needs: host threads that
  // launch other CTA sizes set the same
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           TG::smem(MAX_THREADS_FP64)) != cudaSuccess)
    return PXRB_EUNSUPPORTED;
  if (cudaMemsetAsync(ctr, 0, sizeof(int), s) != cudaSuccess) return PXRB_ELAUNCH;
  kern<<<ctas, threads, need, s>>>(jobs, work, nwork, nwork_dev, ctr);
  PXRB_CHECK_LAUNCH();
  return PXRB_OK;
}

}  // namespace pxrt
