// Plain FP64 path: the Esirkepov deposition on PICSAR's arrays with the
// particles of a call first put into groups (one y and z cell, a run of x
// cells, pxr_group.cuh), in whatever order they come.  A warp then works
// through a group on the FP64 matrix instruction and the group's currents
// leave once, by global FP64 atomics.
//
// One particle per thread makes 144 global FP64 atomics per particle at order
// 3 (0.19 T/s: 4.5 ms for 8.4 M particles at 8 per cell); a group of 40 makes
// 240 together.  The grouping moves 24 B of position and 16 B of key, rank
// and permutation per particle (0.10 ms of the 0.97 ms these 8.4 M take; 1.97 M
// particles in no order at 4 per cell: 1.27 -> 0.41 ms).  The shared-memory
// pipe is the busiest unit then (64 %: records written and read back by other
// lanes), with the FP64 pipe at half (31 % DMMA, 21 % DFMA).
#include "pxr_fp64_dev.cuh"
#include "pxr_group.cuh"
#include "picsar_b200.h"

namespace {

using namespace pxrd;
using namespace pxrg;

constexpr int TPB = 256, WARPS = TPB / 32;
constexpr int CHUNK = 2048;                   // keys per scan block
constexpr int SLOW_PAD = 32;                  // ints: the slow list's counter
constexpr int SEG = 256;                      // particles of a group one warp takes

// Group keys of a guarded grid: x groups fastest, then y and z base cells,
// over every cell from -guard to n + guard.
struct Keys {
  int gx, gy, gz;                             // guards (offsets of cell -g)
  int nx, ny, nz;                             // base cells per axis
  int nkx, nkeys;
};

// Scratch of one call.
struct Scratch {
  int *cnt;                                   // per key: count, then prefix in its chunk
  int *chunk;                                 // per chunk: prefix of the chunk totals
  int *key, *rank, *perm;                     // per particle
  int *slow;                                  // counter; the deposit's list is in `rank`
};

__device__ __forceinline__ int clampi(int v, int n) { return v < 0 ? 0 : (v >= n ? n - 1 : v); }

// base cell of a position in cells (the shapes' first node + ORDER / 2)
template <int ORDER> __device__ __forceinline__ int base_cell(double x) {
  return ORDER == 2 ? fnint(x) : ffloor(x);
}

template <int ORDER>
__device__ __forceinline__ int key_of(const Keys& K, double x, double y, double z) {
  const int i = clampi(base_cell<ORDER>(x) + K.gx, K.nx) / Geom<ORDER>::C;
  const int j = clampi(base_cell<ORDER>(y) + K.gy, K.ny);
  const int k = clampi(base_cell<ORDER>(z) + K.gz, K.nz);
  return i + K.nkx * (j + K.ny * k);
}

__device__ __forceinline__ int key_start(const Scratch& s, int key) {
  return s.cnt[key] + s.chunk[key / CHUNK];
}

struct PosParams {
  i64 np;
  const double *xp, *yp, *zp;
  double xmin, ymin, zmin, dxi, dyi, dzi;
};

// Whether a call's particles are in no useful order (the separate gather's
// question): of 256 neighbours in memory, spread over the call by the golden
// ratio (even steps can fall on row ends only), more than half lie further
// apart than eight cells in x or one in y or z.  Every block asks the same
// 256 pairs and clears its share of the counters if so.
__global__ void __launch_bounds__(TPB) k_order_probe(PosParams p, Keys K, Scratch s) {
  const double f = threadIdx.x * 0.6180339887498949;
  const i64 i = (i64)((f - floor(f)) * (double)(p.np - 1)), j = min(i + 1, p.np - 1);
  const double dx = floor((p.xp[j] - p.xmin) * p.dxi) - floor((p.xp[i] - p.xmin) * p.dxi);
  const double dy = floor((p.yp[j] - p.ymin) * p.dyi) - floor((p.yp[i] - p.ymin) * p.dyi);
  const double dz = floor((p.zp[j] - p.zmin) * p.dzi) - floor((p.zp[i] - p.zmin) * p.dzi);
  const bool near = fabs(dx) <= 8.0 && fabs(dy) <= 1.0 && fabs(dz) <= 1.0;
  const bool group = 2 * __syncthreads_count(!near) > TPB;
  if (blockIdx.x == 0 && threadIdx.x == 0) s.slow[1] = group;
  if (group)
    for (int k = blockIdx.x * TPB + threadIdx.x; k < K.nkeys; k += gridDim.x * TPB) s.cnt[k] = 0;
}

// COND: only if the probe found no order.
template <int ORDER, bool COND>
__global__ void __launch_bounds__(TPB) k_group_count(PosParams p, Keys K, Scratch s) {
  if (COND && !s.slow[1]) return;
  for (i64 i = blockIdx.x * (i64)TPB + threadIdx.x; i < p.np; i += (i64)gridDim.x * TPB) {
    const int key = key_of<ORDER>(K, (p.xp[i] - p.xmin) * p.dxi, (p.yp[i] - p.ymin) * p.dyi,
                                  (p.zp[i] - p.zmin) * p.dzi);
    // one atomic per warp and key: a crowded key's counter is one address.  (In
    // a warp whose first particle shares its key with no other, each on its
    // own: particles in no order mostly differ, and matching them costs more.)
    const unsigned act = __activemask();
    const int lane = threadIdx.x & 31, k0 = __shfl_sync(act, key, __ffs(act) - 1);
    const bool match = __popc(__ballot_sync(act, key == k0)) > 1;
    const unsigned peers = match ? __match_any_sync(act, key) : 1u << lane;
    const int lead = __ffs(peers) - 1;
    int base = 0;
    if (lane == lead) base = atomicAdd(s.cnt + key, __popc(peers));
    s.key[i] = key;
    s.rank[i] = __shfl_sync(act, base, lead) + __popc(peers & ((1u << lane) - 1u));
  }
}

__device__ __forceinline__ int block_exclusive(int v, int* sh, int& total) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  int inc = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += u;
  }
  if (lane == 31) sh[wid] = inc;
  __syncthreads();
  if (wid == 0) {
    int w = lane < nw ? sh[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += u;
    }
    sh[lane] = w;
  }
  __syncthreads();
  const int before = wid ? sh[wid - 1] : 0;
  total = sh[nw - 1];
  __syncthreads();
  return before + inc - v;
}

// counts -> exclusive prefixes within each chunk of keys, chunk totals
template <bool COND>
__global__ void __launch_bounds__(TPB) k_group_scan(Keys K, Scratch s) {
  if (COND && !s.slow[1]) return;
  __shared__ int sh[32];
  constexpr int PER = CHUNK / TPB;
  const int base = blockIdx.x * CHUNK + threadIdx.x * PER;
  int v[PER], sum = 0;
#pragma unroll
  for (int u = 0; u < PER; ++u) {
    v[u] = base + u < K.nkeys ? s.cnt[base + u] : 0;
    sum += v[u];
  }
  int total;
  int run = block_exclusive(sum, sh, total);
#pragma unroll
  for (int u = 0; u < PER; ++u) {
    if (base + u < K.nkeys) s.cnt[base + u] = run;
    run += v[u];
  }
  if (threadIdx.x == 0) s.chunk[blockIdx.x] = total;
}

// chunk totals -> exclusive prefixes (one block)
template <bool COND>
__global__ void __launch_bounds__(1024) k_group_scan_top(int nchunks, Scratch s) {
  if (COND && !s.slow[1]) return;
  __shared__ int sh[32];
  int carry = 0;
  for (int b = 0; b < nchunks; b += 1024) {
    const int i = b + threadIdx.x, v = i < nchunks ? s.chunk[i] : 0;
    int total;
    const int ex = block_exclusive(v, sh, total);
    if (i < nchunks) s.chunk[i] = carry + ex;
    carry += total;
  }
  if (threadIdx.x == 0) *s.slow = 0;
}

template <bool COND>
__global__ void __launch_bounds__(TPB) k_group_perm(i64 np, Scratch s) {
  if (COND && !s.slow[1]) return;
  for (i64 i = blockIdx.x * (i64)TPB + threadIdx.x; i < np; i += (i64)gridDim.x * TPB)
    s.perm[key_start(s, s.key[i]) + s.rank[i]] = (int)i;
}

// A group: its particles (range of the permutation), base cells of column 0
// and of y and z.
struct Group {
  int p0, p1, bx, by, bz;
};
template <int ORDER>
__device__ __forceinline__ void group_of(const Keys& K, const Scratch& s, i64 np, int key, Group& g) {
  g.p0 = key_start(s, key);
  g.p1 = key + 1 < K.nkeys ? key_start(s, key + 1) : (int)np;
  const int r = key / K.nkx;
  g.bx = (key - r * K.nkx) * Geom<ORDER>::C - K.gx;
  g.by = r % K.ny - K.gy;
  g.bz = r / K.ny - K.gz;
}

// One warp's deposit of particles g.p0 .. g.p1 - 1 of a group.  A particle whose
// y or z node changes, or whose x box leaves the group's columns, goes to a
// list that one-particle-per-thread code works off after (a few percent of a
// thermal plasma): inline it would cost its warp a whole general deposit.
template <int ORDER>
__device__ __forceinline__ void deposit_group(const DepParams& p, const Scratch& s, const Group& g,
                                              double* buf) {
  typedef Geom<ORDER> GE;
  typedef EsirAxis<ORDER, double> AX;
  const int lane = threadIdx.x & 31;
  Currents<ORDER> J;
  J.clear();
  for (int b = g.p0; b < g.p1; b += 32) {
    const int n = min(32, g.p1 - b);
    const bool valid = lane < n;
    const int ip = s.perm[b + (valid ? lane : 0)];
    double x = (p.xp[ip] - p.xmin) * p.dxi, y = (p.yp[ip] - p.ymin) * p.dyi,
           z = (p.zp[ip] - p.zmin) * p.dzi;
    const double gi = p.gaminv[ip];
    const double vx = p.uxp[ip] * gi, vy = p.uyp[ip] * gi, vz = p.uzp[ip] * gi;
    const double wq = p.q * p.w[ip];
    const double xold = x - p.dtsdx * vx, yold = y - p.dtsdy * vy, zold = z - p.dtsdz * vz;
    if (p.reconstruct) {
      x = xold + p.dtsdx * vx; y = yold + p.dtsdy * vy; z = zold + p.dtsdz * vz;
    }
    const int x0 = AX::node(x), x1 = AX::node(xold), y0 = AX::node(y), z0 = AX::node(z);
    const bool ok = (unsigned)(x0 - g.bx) < (unsigned)GE::C &&
                    (unsigned)(x1 - g.bx) < (unsigned)GE::C && y0 == g.by &&
                    AX::node(yold) == g.by && z0 == g.bz && AX::node(zold) == g.bz;
    AX X;
    const bool oneoff = X.set(x0, x - x0, x1, xold - x1);
    double sy0[GE::N], sy1[GE::N], sz0[GE::N], sz1[GE::N];
    AX::shape(y - y0, sy0); AX::shape(yold - y0, sy1);
    AX::shape(z - z0, sz0); AX::shape(zold - z0, sz1);
    // the products spread a group's operands over all of its nodes (0 times
    // them): what is not finite keeps to the particle's own nodes in the list
    const double cx = wq * p.invdtdx, cy = wq * p.invdtdy, cz = wq * p.invdtdz;
    const bool fin = isfinite(x + xold + y + yold + z + zold) &&
                     isfinite(fabs(cx) + fabs(cy) + fabs(cz));
    const bool fast = valid && ok && oneoff && fin;
    if (valid && !fast) s.rank[atomicAdd(s.slow, 1)] = ip;
    if (!fast) {
      // no contribution: finite shapes times zero charge
#pragma unroll
      for (int t = 0; t < GE::N; ++t) sy0[t] = sy1[t] = sz0[t] = sz1[t] = 0.0;
#pragma unroll
      for (int t = 0; t < GE::N + 1; ++t) X.s0[t] = X.s1[t] = 0.0;
    }
    J.stage(buf, X, sy0, sy1, sz0, sz1, fast ? cx : 0.0, fast ? cy : 0.0, fast ? cz : 0.0);
    __syncwarp();
#pragma unroll 1
    for (int t = 0; t < (n + 3) >> 2; ++t) J.sub(buf, t, X.i0 - (g.bx - GE::A));
    __syncwarp();
  }
  const GridG& G = p.G;
  const int nx0 = g.bx - GE::A, ny0 = g.by - GE::A, nz0 = g.bz - GE::A;
  J.flush([&](int c, int i, int j, int k, double v) {
    if (v == 0.0) return;                     // columns no particle reaches
    double* a = c == 0 ? p.jx : c == 1 ? p.jy : p.jz;
    atomicAdd(a + G.idx(nx0 + i, ny0 + j, nz0 + k), v);
  });
}

// A group of at most SEG particles is one warp's.  A larger one (a beam, a thin
// target: with a warp per group 2^20 particles in one cell took 77 ms, one
// particle per thread 10.6) is cut at multiples of SEG of the permutation:
// the first nseg warps each look at one such segment, which at most two large
// groups can reach, and leave small groups to the warps after them.
template <int ORDER>
__global__ void __launch_bounds__(TPB, 2) k_esirkepov_group(DepParams p, Keys K, Scratch s, int nseg) {
  extern __shared__ __align__(16) unsigned char smem[];
  double* buf = reinterpret_cast<double*>(smem + (threadIdx.x >> 5) * Geom<ORDER>::WARP_BYTES);
  const int w = blockIdx.x * WARPS + (threadIdx.x >> 5);
  const bool seg = w < nseg;
  int lo = 0, hi = (int)p.np, key = w - nseg, last = key;
  if (seg) {
    lo = w * SEG;
    hi = lo + min(hi - lo, SEG);
    key = s.key[s.perm[lo]];
    last = s.key[s.perm[hi - 1]];
  } else if (key >= K.nkeys) {
    return;                                                  // whole warp, as below
  }
#pragma unroll 1
  for (;;) {
    Group g;
    group_of<ORDER>(K, s, p.np, key, g);
    if (seg == (g.p1 - g.p0 > SEG) && g.p0 < g.p1) {
      g.p0 = max(g.p0, lo);
      g.p1 = min(g.p1, hi);
      deposit_group<ORDER>(p, s, g, buf);
    }
    if (key == last) return;
    key = last;
  }
}

template <int ORDER>
__global__ void __launch_bounds__(TPB) k_esirkepov_list(DepParams p, Scratch s) {
  const int n = *s.slow;
  for (int t = blockIdx.x * TPB + threadIdx.x; t < n; t += gridDim.x * TPB)
    deposit_one<ORDER>(p, s.rank[t]);
}

int grid_of(i64 n, int tpb) {
  const i64 b = (n + tpb - 1) / tpb, cap = 148 * 16;
  return (int)(b < 1 ? 1 : (b > cap ? cap : b));
}

bool make_keys(int order, i64 nx, i64 ny, i64 nz, i64 gx, i64 gy, i64 gz, Keys& K) {
  const i64 bx = nx + 1 + 2 * gx, by = ny + 1 + 2 * gy, bz = nz + 1 + 2 * gz;
  const i64 c = COLS - order, nkx = (bx + c - 1) / c, nk = nkx * by * bz;
  if (nk < 1 || nk > (1 << 30) || bx > (1 << 20) || by > (1 << 20) || bz > (1 << 20)) return false;
  K.gx = (int)gx; K.gy = (int)gy; K.gz = (int)gz;
  K.nx = (int)bx; K.ny = (int)by; K.nz = (int)bz;
  K.nkx = (int)nkx; K.nkeys = (int)nk;
  return true;
}

i64 scratch_ints(const Keys& K, i64 np) {
  const i64 nch = (K.nkeys + CHUNK - 1) / CHUNK;
  return (i64)K.nkeys + nch + SLOW_PAD + 3 * np;
}

Scratch carve(const Keys& K, i64 np, void* mem) {
  const i64 nch = (K.nkeys + CHUNK - 1) / CHUNK;
  Scratch s;
  int* m = static_cast<int*>(mem);
  s.slow = m; m += SLOW_PAD;
  s.cnt = m; m += K.nkeys;
  s.chunk = m; m += nch;
  s.key = m; m += np;
  s.rank = m; m += np;
  s.perm = m;
  return s;
}

template <int ORDER>
int group_particles(const PosParams& q, const Keys& K, const Scratch& s, cudaStream_t st) {
  const int nch = (K.nkeys + CHUNK - 1) / CHUNK;
  if (cudaMemsetAsync(s.cnt, 0, sizeof(int) * (size_t)K.nkeys, st) != cudaSuccess)
    return PXRB_ELAUNCH;
  k_group_count<ORDER, false><<<grid_of(q.np, TPB), TPB, 0, st>>>(q, K, s);
  k_group_scan<false><<<nch, TPB, 0, st>>>(K, s);
  k_group_scan_top<false><<<1, 1024, 0, st>>>(nch, s);
  k_group_perm<false><<<grid_of(q.np, TPB), TPB, 0, st>>>(q.np, s);
  return PXRB_OK;
}

// The same permutation for the separate gather, made only if the particles
// are in no order (slow[1]).
template <int ORDER>
int order_particles(const PosParams& q, const Keys& K, const Scratch& s, cudaStream_t st) {
  const int nch = (K.nkeys + CHUNK - 1) / CHUNK;
  k_order_probe<<<148, TPB, 0, st>>>(q, K, s);
  k_group_count<ORDER, true><<<grid_of(q.np, TPB), TPB, 0, st>>>(q, K, s);
  k_group_scan<true><<<nch, TPB, 0, st>>>(K, s);
  k_group_scan_top<true><<<1, 1024, 0, st>>>(nch, s);
  k_group_perm<true><<<grid_of(q.np, TPB), TPB, 0, st>>>(q.np, s);
  PXRB_CHECK_LAUNCH();
  return PXRB_OK;
}

template <class KERN> int big_smem(KERN k, int bytes) {
  return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) == cudaSuccess
             ? PXRB_OK : PXRB_ELAUNCH;
}

template <int ORDER>
int run_esirkepov(const DepParams& p, const Keys& K, const Scratch& s, cudaStream_t st) {
  PosParams q = {p.np, p.xp, p.yp, p.zp, p.xmin, p.ymin, p.zmin, p.dxi, p.dyi, p.dzi};
  const int smem = WARPS * Geom<ORDER>::WARP_BYTES;
  if (const int e = big_smem(k_esirkepov_group<ORDER>, smem)) return e;
  if (const int e = group_particles<ORDER>(q, K, s, st)) return e;
  const int nseg = (int)((p.np + SEG - 1) / SEG);
  const i64 warps = (i64)nseg + K.nkeys;
  k_esirkepov_group<ORDER><<<(int)((warps + WARPS - 1) / WARPS), TPB, smem, st>>>(p, K, s, nseg);
  k_esirkepov_list<ORDER><<<148 * 4, TPB, 0, st>>>(p, s);
  PXRB_CHECK_LAUNCH();
  return PXRB_OK;
}

}  // namespace

namespace pxrd {

static bool fits(i64 need, const void* scratch, i64 bytes) {
  return scratch && need > 0 && bytes >= need && (reinterpret_cast<uintptr_t>(scratch) & 3) == 0;
}
bool group_fits(int order, i64 np, const GridG& G, const void* scratch, i64 bytes) {
  return fits(pxrb_group_scratch(order, np, G.nx, G.ny, G.nz, G.gx, G.gy, G.gz), scratch, bytes);
}
bool order_fits(int order, i64 np, const GridG& G, const void* scratch, i64 bytes) {
  return fits(pxrb_order_scratch(order, np, G.nx, G.ny, G.nz, G.gx, G.gy, G.gz), scratch, bytes);
}

int gather_order(i64 np, const double* xp, const double* yp, const double* zp, const double* lo,
                 const double* di, const GridG& G, void* scratch, cudaStream_t st,
                 GatherOrder& o) {
  Keys K;
  if (!make_keys(3, G.nx, G.ny, G.nz, G.gx, G.gy, G.gz, K)) return PXRB_EINVAL;
  const Scratch s = carve(K, np, scratch);
  PosParams q = {np, xp, yp, zp, lo[0], lo[1], lo[2], di[0], di[1], di[2]};
  o.perm = s.perm;
  o.use = s.slow + 1;
  return order_particles<3>(q, K, s, st);
}

int esirkepov_grouped(int order, const DepParams& p, void* scratch, cudaStream_t st) {
  Keys K;
  if (!make_keys(order, p.G.nx, p.G.ny, p.G.nz, p.G.gx, p.G.gy, p.G.gz, K)) return PXRB_EINVAL;
  const Scratch s = carve(K, p.np, scratch);
  return order == 2 ? run_esirkepov<2>(p, K, s, st) : run_esirkepov<3>(p, K, s, st);
}

}  // namespace pxrd

extern "C" int64_t pxrb_order_scratch(int64_t order, int64_t np, int64_t nx, int64_t ny,
                                      int64_t nz, int64_t nxguard, int64_t nyguard,
                                      int64_t nzguard) {
  // Particles in no order, as they come -> by cell, microseconds, order 3:
  // 1.97 M 1016 -> 400 (lower shapes) and 1463 -> 501 (full), 1.21 M 625 -> 208,
  // 8.4 M 4342 -> 2755.  Order 2 gains up to 2 M (413 -> 337) and loses at 8.4 M
  // (1746 -> 2692: the particles' nine columns no longer fit L2 and come in
  // single sectors), order 1 always loses (133 -> 329).  Particles in order
  // pay the probe and four kernels that return at once, 17 us: from 2^20
  // particles on, where that is small.  (The fused gather + push moves 26
  // columns per particle and by cell lost as much as it gained: 432 -> 903 at
  // order 2, 1022 -> 955 at order 3, 1.97 M.)
  Keys K;
  if (order != 3 || np < (1 << 20) || np >= (1LL << 31) || nx < 0 || ny < 0 ||
      nz < 0 || nxguard < 0 || nyguard < 0 || nzguard < 0 ||
      !make_keys((int)order, nx, ny, nz, nxguard, nyguard, nzguard, K) || K.nkeys > np)
    return 0;
  return 4 * scratch_ints(K, np);
}

extern "C" int64_t pxrb_group_scratch(int64_t order, int64_t np, int64_t nx, int64_t ny,
                                      int64_t nz, int64_t nxguard, int64_t nyguard,
                                      int64_t nzguard) {
  // Where grouping pays (one particle per thread -> grouped, microseconds):
  // order 3 from 6 particles per group (6.9 in no order: 360 -> 169; in cell
  // order about even; 5.4 in order: 31 -> 66) and 65536 particles (110592 at
  // 16 per group: 84 -> 66); order 2 from 16 (17.7: 368 -> 267, 8.7: 138 ->
  // 127) and 131072 (110592: 39 -> 51); order 1, with 12 atomics per
  // particle, never (8.4 M: 362 -> 561).  These are cold plasmas.  In a hot one
  // a third to half of the particles (u_th 0.5, 2) change their y or z node and
  // are deposited on their own after all.  Order 3 in cell order 7.9 per group
  // 958 -> 992 and 1071 -> 1235, 15.9 per group 2115 -> 1541 and 2345 -> 2014,
  // in no order always faster; order 2 in cell order 18.5 per group 902 -> 906
  // and 992 -> 1108, 37 per group 2130 -> 1588 and 2361 -> 1987, in no order
  // 2087 -> 2233 and 2282 -> 2705.  (A probe of the momenta on the device that
  // left such calls alone cost every call 10 us.)  Particles in few cells, in
  // no order, 2^20 of them, order 3 / 2: one cell 10573 -> 286 / 7183 -> 239,
  // a thousand 800 -> 192 / 341 -> 161.
  Keys K;
  const i64 least = order == 3 ? 1 << 16 : 1 << 17, per_key = order == 3 ? 6 : 16;
  if (order < 2 || order > 3 || np < least || np >= (1LL << 31) || nx < 0 || ny < 0 ||
      nz < 0 || nxguard < 0 || nyguard < 0 || nzguard < 0 ||
      !make_keys((int)order, nx, ny, nz, nxguard, nyguard, nzguard, K) ||
      np < per_key * (i64)K.nkeys)
    return 0;
  return 4 * scratch_ints(K, np);
}
