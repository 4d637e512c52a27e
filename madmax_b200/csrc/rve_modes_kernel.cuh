// rve_modes_kernel.cuh -- the batched stencil solve, in FP32 corrections or in
// FP64, one load case of one RVE per CTA at a time, on the element-mode operator
// (rve_modes.cuh).
//
// The load cases of an RVE are independent systems.  Solved one by one, the
// search direction p and the product q = A p of an RVE of up to about 20^3
// elements stay in one SM's shared memory (6 load cases at once are 2.7 MB of
// vectors at n = 20, which stream from HBM in every CG iteration); r and x,
// 16 bytes a node component, stream from L2 once per iteration.  A load case
// leaves when it has converged, not when the slowest of its RVE has.
//
// What a CTA runs is the solve of rve_solve.cuh for K = 1: FP64 residual of
// u = eps.x + w (here marched in element modes too), FP32 Jacobi-PCG
// corrections as reliable updates, w += x in FP64, volume averages in FP64.
//
// The scalars that steer CG are products formed and added in FP64 (ModesType::
// dot): in FP32 they left the range with small strains, lengths or moduli.
//
// What bounds it: the march's serial chain over the planes, a barrier and the
// shared-memory exchange per plane, with its shuffles and packed FP32 work (592
// RVEs of n = 16: issue slots 48%, L1 data pipe 60%, FP64 pipe 8% busy, DRAM
// idle).  Small RVEs hide it with several CTAs per SM (classes at the end of
// this file), so a class is as small as threads and shared memory allow.
// Measured against the block stencil with all load cases in one CTA, solves to
// 1e-10: 4096 RVEs of n = 8..20 335 -> 121 ms, 1 RVE of n = 24 with 6 load cases
// 38.0 -> 5.9 ms (6 SMs instead of 1), periodic 256 RVEs of n = 9..17 34.6 -> 5.1
// ms, FP64 192 RVEs of n = 8..16 21.9 -> 5.0 ms, 74 RVEs of n = 32 (no vector on
// chip) 206 -> 63 ms.  (With the scalars in FP32: 117, 5.6, 5.0, 4.9 ms.)
#pragma once

#include "rve_batch_kernel.cuh"
#include "rve_modes.cuh"

namespace sp {

// Work spaces of a launch's CTAs
struct ModesBufs {
  double *ws_w;    // per CTA [3][wlen]
  void *ws_v;      // per CTA [3][ntot] 8-byte values each of r, x, (q in L2) q, (p too) p
  void *ws_e;      // per CTA (q in L2) shares that cross strips: 2 x [planes][nex][3] values
  size_t w_stride, v_stride, e_stride;  // v_stride: of one of them
  size_t v_cta;                         // ... of a CTA's
};

// When a load case's solve ends
struct ModesLimits {
  double rtol, inner_rtol;
  double rtol_refine;  // target once a refinement step has run (<= rtol)
  int max_outer, max_inner;
};

struct ModesParams {
  const BatchPlan *plans;
  const BatchRve *rves;
  const int *order;  // RVEs of this launch, largest first
  int ntask, nrhs;   // tasks: (RVE, load case)
  const uint8_t *etype;
  const double *strains;  // [nrve][nrhs][6]
  const double *mats;     // [nrve][4]
  double *out_stress, *out_strain;
  sp_solve_info *out_info;
  sp_solve_info *task_info;  // [nrve][nrhs]
  unsigned *done;            // [nrve] finished load cases (0 between launches)
  int *counter;
  ModesBufs buf;
  ModesLimits lim;
};

constexpr int SP_MODES_MAX_NEZ = 32;  // a column's materials are one 32-bit mask
constexpr int SP_MODES_MAX_COLS = 1024;
constexpr int SP_MODES_MAX_WARPS = 20;

// What the CTA shares while it solves one load case; the first thing in its
// dynamic shared memory.
struct ModesShared {
  double cd[2][MC_N];    // mode coefficients of the two materials
  float2 c32[4][MC_N];   // FP32 pairs: materials of the (lower, upper) layer
  double dl64[9][4];     // Jacobi diagonal by the number of fibre elements around a node
  float4 dl[9];          // ... in FP32
  double kd2[9];         // sum over components of the squared diagonal
  double A[9];           // first-order modes of eps.x: [component][axis]
  double E[9];           // eps as a 3x3 matrix
  double len[3], hx[3], a[3];  // box, element edges and their inverses
  double lame[2][2];     // lambda, mu of the two materials
  double red[2 * SP_MODES_MAX_WARPS * 10];
  double cc[2][CC_N];    // cube: lambda, mu, 2 mu, lambda/3, mu/3, (lambda + 4 mu)/9, times c0 a^2
  float2 c6[4][CC_N];    // ... as FP32 pairs: materials of the (lower, upper) layer
  unsigned col[SP_MODES_MAX_COLS];  // per column: bit e = material of layer e
  int nex, ney, nez, nface, mz, h, ntot, wlen, rows;  // rows: of a strip
  int job, rid, k, outer, inner, wcols, qoff, cntoff, pad[3];  // qoff, cntoff: bytes from p on
};
static_assert(sizeof(ModesShared) % 16 == 0, "vectors follow on a 16-byte boundary");

// Sizes of one RVE's march.  Affine conditions: the interior planes, a row's
// first node and a plane's first row being the boundary's zeros.  Periodic
// conditions: every node of the periodic grid, neighbours wrapped; a row's
// columns are preceded by a repetition of its last one, the left neighbour of
// its first.
// FP32 vectors have a slot for each pair of planes, FP64 ones for each plane;
// a value is 8 bytes either way.  `on`: the vectors in shared memory -- 2: p
// and q, 1: p, 0: neither.  Without q there (affine conditions) the columns
// are marched in strips of `rows` rows, 512 threads at most, one strip after
// another.
struct ModesGeo {
  int nex, ney, nez, nface, mz, h, ntot, per, on, rows;
  __host__ __device__ ModesGeo(int ex, int ey, int ez, bool periodic, bool f64, int onchip)
      : nex(ex), ney(ey), nez(ez), nface(ex * ey), mz(periodic ? ez : ez - 1),
        h(f64 ? mz : (mz + 1) / 2), ntot(h * ex * ey + (periodic ? 0 : ex + 2)), per(periodic),
        on(onchip), rows(ey) {
    if (on < 2 && !per) {
      const int fit = 16 * wcols() / rowlanes(), n = fit > 0 ? (ey + fit - 1) / fit : 0;
      rows = n > 0 ? (ey + n - 1) / n : 0;
    }
  }
  __host__ __device__ int wlen() const { return mz * nface + (per ? 0 : nex + 2); }
  // lanes of a row, of a strip's rows, and of a warp: 32 where rows start at
  // lane 0 (whose left neighbour is the boundary, or its own repetition),
  // else 31 and a repetition of the last lane of the previous warp
  __host__ __device__ int rowlanes() const { return per ? nex + 1 : nex; }
  __host__ __device__ int lanes() const { return rowlanes() * rows; }
  __host__ __device__ int wcols() const { return 32 % rowlanes() == 0 ? 32 : 31; }
  __host__ __device__ int warps() const { return (lanes() + wcols() - 1) / wcols(); }
  // Dynamic shared memory: tables, p, then q, whose place the FP64 residual's
  // face state and exchange planes take too, or (q in L2) two exchange planes,
  // with the state in p's place or after them; material counts.
  __host__ __device__ int state() const { return 32 * warps() * 8; }
  __host__ __device__ int pbytes() const {
    const int a = on >= 1 ? ntot * 24 : 0, b = on == 1 ? 25 * state() : 0;
    return a > b ? a : b;
  }
  __host__ __device__ int qbytes() const {
    const int a = on == 2 ? ntot * 24 : 0, b = 2 * nex * rows * 24 + (on == 1 ? 0 : 13 * state());
    return a > b ? a : b;
  }
  __host__ __device__ int smem() const {
    return (int)sizeof(ModesShared) + pbytes() + qbytes() + (h * nface + 15) / 16 * 16;
  }
};

// what the march of G reads from shared memory
__device__ __forceinline__ void modes_sizes(const ModesGeo &G, ModesShared &sh) {
  sh.nex = G.nex;
  sh.ney = G.ney;
  sh.nez = G.nez;
  sh.nface = G.nface;
  sh.mz = G.mz;
  sh.h = G.h;
  sh.ntot = G.ntot;
  sh.wlen = G.wlen();
  sh.wcols = G.wcols();
  sh.rows = G.rows;
  sh.qoff = G.pbytes();
  sh.cntoff = G.pbytes() + G.qbytes();
  sh.outer = sh.inner = 0;
}
// whether a CTA of the kernel's threads and dynamic shared memory holds it
__device__ __forceinline__ bool modes_fit(const ModesGeo &G) {
  return dynamic_smem_bytes() >= (unsigned)G.smem() && G.warps() * 32 <= (int)blockDim.x &&
         G.warps() <= SP_MODES_MAX_WARPS && G.rows >= 1 && !(G.per && G.on == 0) &&
         G.nez <= (G.per ? SP_MODES_MAX_NEZ - 2 : SP_MODES_MAX_NEZ) &&
         G.nface <= SP_MODES_MAX_COLS;
}

extern __shared__ __align__(16) unsigned char s_modes[];
__device__ __forceinline__ ModesShared &msh() { return *reinterpret_cast<ModesShared *>(s_modes); }
template <typename V>
__device__ __forceinline__ V *mp() {
  return reinterpret_cast<V *>(s_modes + sizeof(ModesShared));
}
// q, or the exchange planes
template <typename V>
__device__ __forceinline__ V *mq() {
  return reinterpret_cast<V *>(mp<char>() + msh().qoff);
}
__device__ __forceinline__ uint8_t *mcnt() { return mp<uint8_t>() + msh().cntoff; }

// FP32 pairs or FP64 values: their memory type and the type of their scalars.
// dot: the product(s) of a and b, formed and added in FP64 -- squares of FP32
// residuals leave FP32's range where the residuals do not.
template <typename V>
struct ModesType;
template <>
struct ModesType<F2> {
  static constexpr bool F64 = false;
  using Mem = float2;
  using S = float;
  __device__ static F2 ld(const float2 *a) { return F2{__ldcg(a)}; }
  __device__ static void st(float2 *a, F2 v) { __stcg(a, v.v); }
  __device__ static void add(float2 *a, F2 v) { atomicAdd(a, v.v); }
  __device__ static F2 splat(float s) { return mk2(s, s); }
  __device__ static double dot(F2 a, F2 b) {
    return fma((double)a.v.y, (double)b.v.y, (double)a.v.x * (double)b.v.x);
  }
  // sums of the squares of a[0..2], of the lower and of the upper planes
  __device__ static void squares(const F2 (&a)[3], double (&s)[2]) {
    const double x0 = a[0].v.x, x1 = a[1].v.x, x2 = a[2].v.x;
    const double y0 = a[0].v.y, y1 = a[1].v.y, y2 = a[2].v.y;
    s[0] = x0 * x0 + x1 * x1 + x2 * x2;
    s[1] = y0 * y0 + y1 * y1 + y2 * y2;
  }
};
template <>
struct ModesType<double> {
  static constexpr bool F64 = true;
  using Mem = double;
  using S = double;
  __device__ static double ld(const double *a) { return __ldcg(a); }
  __device__ static void st(double *a, double v) { __stcg(a, v); }
  __device__ static void add(double *a, double v) { atomicAdd(a, v); }
  __device__ static double splat(double s) { return s; }
  __device__ static double dot(double a, double b) { return a * b; }
  __device__ static void squares(const double (&a)[3], double (&s)[2]) {
    s[0] = a[0] * a[0] + a[1] * a[1] + a[2] * a[2];
    s[1] = 0.0;
  }
};

// Sum NV doubles over the CTA in a fixed order; every thread gets the
// totals.  One barrier: red holds two buffers, used in turn.
template <int NV>
__device__ __forceinline__ void cta_sum(double (&v)[NV], int &ph) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  double *r = msh().red + ph * (SP_MODES_MAX_WARPS * 10);
#pragma unroll
  for (int q = 0; q < NV; q++)
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v[q] += __shfl_xor_sync(0xffffffffu, v[q], off);
  if (lane == 0)
#pragma unroll
    for (int q = 0; q < NV; q++) r[warp * NV + q] = v[q];
  __syncthreads();
#pragma unroll
  for (int q = 0; q < NV; q++) {
    v[q] = lane < nw ? r[lane * NV + q] : 0.0;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v[q] += __shfl_xor_sync(0xffffffffu, v[q], off);
  }
  ph ^= 1;
}

// A thread's place in the march of a strip.  f: its element column (face);
// the repeated lanes and the padding threads of the last warp write nothing.
template <bool PER>
struct ModesLane {
  int f;
  int f0, f1;    // columns of the strip: [f0, f1)
  int dx, dy;    // from f to the columns at x + 1 and y + 1
  int threads;   // of the warps that have a column
  bool warp_on;  // the warp has a column
  bool column;   // the thread has one
  bool owner;    // ... and its node (ex, ey) is an unknown
  __device__ __forceinline__ explicit ModesLane(int y0 = 0) {
    const ModesShared &sh = msh();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, rep = 32 - sh.wcols;
    const int i = warp * sh.wcols + lane - rep, row = PER ? sh.nex + 1 : sh.nex;
    const int rows = min(sh.rows, sh.ney - y0);
    const int n = row * rows, ic = min(max(i, 0), n - 1);
    f0 = y0 * sh.nex;
    f1 = f0 + rows * sh.nex;
    warp_on = warp * sh.wcols < n;
    threads = (n + sh.wcols - 1) / sh.wcols * 32;
    column = lane >= rep && i < n;
    if (PER) {
      const int y = ic / row, v = ic - y * row, x = v ? v - 1 : sh.nex - 1;
      f = y * sh.nex + x;
      dx = x == sh.nex - 1 ? 1 - sh.nex : 1;
      dy = y == sh.ney - 1 ? sh.nex - sh.nface : sh.nex;
      column = column && v != 0;
      owner = column;
    } else {
      f = f0 + ic;
      dx = 1;
      dy = sh.nex;
      owner = column && f >= sh.nex && f % sh.nex != 0;
    }
  }
};

__device__ __forceinline__ unsigned shr32(unsigned m, int n) { return n < 32 ? m >> n : 0u; }

// the columns at x - 1 and y - 1 of an owner's column
template <bool PER>
__device__ __forceinline__ void modes_below(int f, int &left, int &down) {
  const ModesShared &sh = msh();
  left = PER && f % sh.nex == 0 ? sh.nex - 1 : -1;
  down = PER && f < sh.nex ? sh.nface - sh.nex : -sh.nex;
}

// Barrier over the warps that have columns
__device__ __forceinline__ void plane_sync(int threads) {
  __syncwarp();
  asm volatile("bar.sync 1, %0;" ::"r"(threads) : "memory");
}

// q = A p on the strip from row y0: p [slot][3] and q in shared memory, or q
// in qg ([3][ntot]), or p in pg and the shares for the next strip's first row
// in eg too; returns the thread's share of p.q.
template <typename V, bool CUBE, int ON, bool PER>
__device__ __noinline__ double march_apply(typename ModesType<V>::Mem *qg, const V *pg, V *eg,
                                           int y0) {
  using MT = ModesType<V>;
  constexpr bool F64 = MT::F64, QS = ON == 2, STRIPS = ON < 2 && !PER;
  // registers to spare for the next slot's values (FP64 has none)
  constexpr bool AHEAD = QS && !F64;
  const ModesShared &sh = msh();
  const ModesLane<PER> T(y0);
  const unsigned mats = sh.col[T.f];
  const int nface = sh.nface, nf3 = 3 * nface, h = sh.h, ntot = sh.ntot;
  const int right = PER ? 3 * T.dx : 3, up = 3 * T.dy;
  const V *pf = (ON ? mp<V>() : pg) + 3 * T.f;  // corner (0, 0) of slot 0
  V *const qf = mq<V>() + 3 * (T.f - T.f0);
  const int ex3 = QS ? nf3 : 3 * sh.rows * sh.nex;
  // the halves of eg: written by one strip, read by the next
  const int eread = STRIPS && !((y0 / sh.rows) & 1) ? 3 * sh.mz * sh.nex : 0;
  const int ewrite = STRIPS ? 3 * sh.mz * sh.nex - eread : 0;
  const bool odd = !F64 && (sh.mz & 1) != 0;
  V raw[3][4], Fa[3][4], Fb[3][4], acc[3][4];
  auto load = [&](const V *a) {
#pragma unroll
    for (int c = 0; c < 3; c++) {
      raw[c][0] = a[c];
      raw[c][1] = a[right + c];
      raw[c][2] = a[up + c];
      raw[c][3] = a[up + right + c];
    }
  };
  // values of step s: slot s; above slot h - 1 lies plane h (lower half) and
  // the boundary plane (upper half), or plane 0 under periodic conditions
  // (for an odd number of planes, already at slot h - 1)
  auto next = [&](int s) {
    load(s < h ? pf + s * nf3 : pf);
    if (s >= h && !(F64 && PER)) {
      __syncwarp();  // a branch: predicated, the moves would be issued every step
#pragma unroll
      for (int c = 0; c < 3; c++)
#pragma unroll
        for (int m = 0; m < 4; m++) {
          if constexpr (F64)
            raw[c][m] = 0.0;
          else
            raw[c][m] = mk2(raw[c][m].v.y, PER ? raw[c][m].v.x : 0.f);
        }
    }
    if constexpr (PER && !F64) {
      if (odd && s == h - 1) {
        __syncwarp();
#pragma unroll
        for (int c = 0; c < 3; c++) {
          raw[c][0].v.y = pf[c].v.x;
          raw[c][1].v.y = pf[right + c].v.x;
          raw[c][2].v.y = pf[up + c].v.x;
          raw[c][3].v.y = pf[up + right + c].v.x;
        }
      }
    }
  };
  if (T.warp_on) {
    // below slot 0: the boundary plane, or the last one (lower half); plane
    // h - 1 (upper half)
    if constexpr (F64) {
      if (PER) load(pf + (h - 1) * nf3);
#pragma unroll
      for (int c = 0; c < 3; c++)
#pragma unroll
        for (int m = 0; m < 4; m++) {
          if (!PER) raw[c][m] = 0.0;
          acc[c][m] = 0.0;
        }
    } else {
      if (PER) {
        load(pf + (odd ? h - 2 : h - 1) * nf3);
#pragma unroll
        for (int c = 0; c < 3; c++)
#pragma unroll
          for (int m = 0; m < 4; m++) acc[c][m].v.x = raw[c][m].v.y;
      }
      load(pf + (h - 1) * nf3);
#pragma unroll
      for (int c = 0; c < 3; c++)
#pragma unroll
        for (int m = 0; m < 4; m++) {
          raw[c][m] = mk2(PER ? acc[c][m].v.x : 0.f, raw[c][m].v.x);
          acc[c][m] = mk2(0.f, 0.f);
        }
    }
    face_modes(raw, Fa);
    if (AHEAD) next(0);
  }
  if (!T.warp_on) return 0.0;
  double pq = 0.0;
  // one step: F0 the modes of the face below, F1 takes those above (two steps
  // a trip, so that the faces change places without copies)
  auto step = [&](int s, V (&F0)[3][4], V (&F1)[3][4]) {
    V low[3], edge[3];
    if (T.warp_on) {
      V S[3][3], D[3][4], high[3];
      if (STRIPS) {
        if (ON == 0 && s + 1 < h) asm volatile("prefetch.global.L1 [%0];" ::"l"(pf + (s + 1) * nf3));
        if (s > 0 && T.f0 > 0 && T.f < T.f0 + sh.nex)
#pragma unroll
          for (int c = 0; c < 3; c++) edge[c] = eg[eread + 3 * ((s - 1) * sh.nex + T.f - T.f0) + c];
      }
      if (!AHEAD) next(s);
      face_modes(raw, F1);
      layer_modes(F0, F1, S, D);
      const unsigned ma = shr32(mats, s) & 1u;
      if constexpr (F64) {
        if constexpr (CUBE) {
          const double *ct = sh.cc[ma];
          modes_cube(S, D, [ct](int i) { return ct[i]; });
        } else {
          const double *ct = sh.cd[ma];
          modes_box(S, D, [ct](int i) { return ct[i]; });
        }
      } else {
        const unsigned mb = shr32(mats, s + h) & 1u;
        if constexpr (CUBE) {
          const float2 *ct = sh.c6[ma + 2 * mb];
          modes_cube(S, D, [ct](int i) { return F2{ct[i]}; });
        } else {
          const float2 *ct = sh.c32[ma + 2 * mb];
          modes_box(S, D, [ct](int i) { return F2{ct[i]}; });
        }
      }
      layer_back(S, D, acc, low, high);
      // the upper row's share waits where that row's q goes (QS), or in the
      // exchange planes in turn
      V *const e = qf + (QS ? (s - 1) : (s & 1)) * ex3 + up;
      if (T.column && s > 0) {
        if (PER || T.f + sh.nex < T.f1) {
#pragma unroll
          for (int c = 0; c < 3; c++) e[c] = high[c];
        } else if (STRIPS && T.f1 < nface) {
#pragma unroll
          for (int c = 0; c < 3; c++)
            eg[ewrite + 3 * ((s - 1) * sh.nex + T.f + sh.nex - T.f1) + c] = high[c];
        }
      }
      // the next slot's values before the barrier
      if (AHEAD) next(s + 1);
    }
    if (s > 0) {
      plane_sync(T.threads);
      if (T.owner) {
        V *const e = qf + (QS ? (s - 1) : (s & 1)) * ex3;
        const bool seam = STRIPS && T.f0 > 0 && T.f < T.f0 + sh.nex;
        const V *ps = pf + (s - 1) * nf3;
        double t[3];
#pragma unroll
        for (int c = 0; c < 3; c++) {
          low[c] = low[c] + (seam ? edge[c] : e[c]);
          if constexpr (F64) {
            if (PER && s == 1 && T.f == 0) low[c] = 0.0;  // the fixed node
          } else {
            if (odd && s == h) low[c].v.y = 0.f;  // no plane there
            if (PER && s == 1 && T.f == 0) low[c].v.x = 0.f;  // the fixed node
          }
          if constexpr (QS)
            e[c] = low[c];
          else
            MT::st(qg + (size_t)c * ntot + (s - 1) * nface + T.f, low[c]);
          t[c] = MT::dot(low[c], ps[c]);
        }
        pq += t[0] + t[1] + t[2];
      }
    }
  };
#pragma unroll 1
  for (int s = 0; s <= h; s++) {
    step(s, Fa, Fb);
#pragma unroll
    for (int c = 0; c < 3; c++)
#pragma unroll
      for (int m = 0; m < 4; m++) Fa[c][m] = Fb[c][m];
  }
  return pq;
}

// b = -K (eps.x + w) on the interior nodes in FP64: rounded to V into rv;
// returns the thread's shares of |b|^2 and r.z.  The running plane's forces
// (and, at 96 registers a thread, the face's modes) wait in shared memory
// between layers: in registers they spill, and a spill goes to L2, since the
// vectors leave L1 next to nothing (n = 20: 285k cycles an evaluation with
// spills, 80k without).
template <typename V, bool CUBE, int ON, bool PER>
__device__ __noinline__ double2 march_residual(const double *w, typename ModesType<V>::Mem *rv,
                                               double *eg, int y0) {
  constexpr bool QS = ON != 1, STRIPS = ON < 2 && !PER;  // QS: 128 registers a thread
  const ModesShared &sh = msh();
  const ModesLane<PER> T(y0);
  const unsigned mats = sh.col[T.f];
  const int nface = sh.nface, right = PER ? T.dx : 1, up = T.dy, wl = sh.wlen, mz = sh.mz, h = sh.h;
  constexpr bool F64 = ModesType<V>::F64;
  double *const ex = mq<double>();  // two exchange planes
  const uint8_t *const cnt = mcnt();
  const int eread = STRIPS && !((y0 / sh.rows) & 1) ? 3 * mz * sh.nex : 0;  // (see march_apply)
  const int ewrite = STRIPS ? 3 * mz * sh.nex - eread : 0;
  // [c][m] of the running forces at 4 c + m, of the face's modes 12 further;
  // an odd number of doubles a thread (no bank conflicts)
  double *const state = (QS ? ex + 6 * sh.rows * sh.nex : mp<double>()) +
                        (T.warp_on ? threadIdx.x : 0) * (QS ? 13 : 25);
  double n2 = 0.0, rz = 0.0;
  double F0[3][4] = {};  // (QS)
  double raw[3][4];
  auto load = [&](int pl) {
    const double *a = w + (pl * nface + T.f);
#pragma unroll
    for (int c = 0; c < 3; c++) {
      raw[c][0] = a[c * wl];
      raw[c][1] = a[c * wl + right];
      raw[c][2] = a[c * wl + up];
      raw[c][3] = a[c * wl + up + right];
    }
  };
  if (!T.warp_on) return make_double2(0.0, 0.0);
#pragma unroll
  for (int j = 0; j < (QS ? 12 : 24); j++) state[j] = 0.0;
  if (PER) {  // below plane 0 lies the last one
    load(mz - 1);
    double F[3][4];
    face_modes(raw, F);
#pragma unroll
    for (int c = 0; c < 3; c++)
#pragma unroll
      for (int m = 0; m < 4; m++) {
        if (QS)
          F0[c][m] = F[c][m];
        else
          state[12 + 4 * c + m] = F[c][m];
      }
  }
  load(0);
#pragma unroll 1
  for (int s = 0; s <= mz; s++) {
    double low[3], edge[3];
    double *const exs = ex + ((s & 1) * sh.rows * sh.nex + T.f - T.f0) * 3;
    if (T.warp_on) {
      if (STRIPS && s > 0 && T.f0 > 0 && T.f < T.f0 + sh.nex)
#pragma unroll
        for (int c = 0; c < 3; c++) edge[c] = eg[eread + 3 * ((s - 1) * sh.nex + T.f - T.f0) + c];
      double S[3][3], D[3][4];
#pragma unroll
      for (int c = 0; c < 3; c++) {
        const double s0 = raw[c][1] + raw[c][0], d0 = raw[c][1] - raw[c][0];
        const double s1 = raw[c][3] + raw[c][2], d1 = raw[c][3] - raw[c][2];
        const double F1[4] = {s1 + s0, d1 + d0, s1 - s0, d1 - d0};
#pragma unroll
        for (int m = 0; m < 4; m++) {
          const double v = QS ? F0[c][m] : state[12 + 4 * c + m];
          if (m > 0) S[c][m - 1] = F1[m] + v;
          D[c][m] = F1[m] - v;
          if (QS)
            F0[c][m] = F1[m];
          else
            state[12 + 4 * c + m] = F1[m];
        }
        S[c][0] += sh.A[3 * c];
        S[c][1] += sh.A[3 * c + 1];
        D[c][0] += sh.A[3 * c + 2];
      }
      if constexpr (CUBE) {
        const double *ct = sh.cc[shr32(mats, s) & 1u];
        modes_cube(S, D, [ct](int i) { return ct[i]; });
      } else {
        const double *ct = sh.cd[shr32(mats, s) & 1u];
        modes_box(S, D, [ct](int i) { return ct[i]; });
      }
      double *e = exs + 3 * up;
      bool put = T.column && (PER || T.f + up < T.f1);
      if (STRIPS && T.column && s > 0 && T.f + up >= T.f1 && T.f1 < nface) {
        e = eg + ewrite + 3 * ((s - 1) * sh.nex + T.f + up - T.f1);
        put = true;
      }
#pragma unroll
      for (int c = 0; c < 3; c++) {
        double *const ac = state + 4 * c;
        const double t0 = ac[0] - D[c][0];
        const double t1 = ac[1] + (S[c][0] - D[c][1]);
        const double t2 = ac[2] + (S[c][1] - D[c][2]);
        const double t3 = ac[3] + (S[c][2] - D[c][3]);
        ac[0] = D[c][0];
        ac[1] = S[c][0] + D[c][1];
        ac[2] = S[c][1] + D[c][2];
        ac[3] = S[c][2] + D[c][3];
        double high;
        plane_back(t0, t1, t2, t3, low[c], high);
        if (put) e[c] = high;
      }
    }
    if (PER || s + 1 < mz) {
      load(PER && s + 1 >= mz ? 0 : s + 1);
    } else {
      __syncwarp();
#pragma unroll
      for (int c = 0; c < 3; c++)
#pragma unroll
        for (int m = 0; m < 4; m++) raw[c][m] = 0.0;
    }
    if (s > 0) {
      plane_sync(T.threads);
      if (T.owner) {
        const bool seam = STRIPS && T.f0 > 0 && T.f < T.f0 + sh.nex;
        const bool hi = !F64 && s - 1 >= h;
        const int i = (hi ? s - 1 - h : s - 1) * nface + T.f;
        const unsigned cv = hi ? cnt[i] >> 4 : cnt[i] & 15u;
#pragma unroll
        for (int c = 0; c < 3; c++) {
          double b = -(low[c] + (seam ? edge[c] : exs[c]));
          if (PER && s == 1 && T.f == 0) b = 0.0;  // the fixed node
          n2 += b * b;
          if constexpr (F64) {
            rv[c * sh.ntot + i] = b;
            rz += b * (sh.dl64[cv][c] * b);
          } else {
            const float bf = (float)b;
            reinterpret_cast<float *>(rv + c * sh.ntot + i)[hi] = bf;
            rz += (double)bf * (double)(reinterpret_cast<const float *>(&sh.dl[cv])[c] * bf);
          }
        }
      }
    }
  }
  return make_double2(n2, rz);
}

// Integrals over the fibre elements of the fluctuation's gradient, up to the
// factor element volume / 4 and the edge lengths: m[3 c + d] = sum of the
// first-order mode along d of component c, as a sum over nodes -- a node's
// weight is the number of fibre elements below it along d less the number
// above.  (Over all elements the weights vanish: the mean strain is eps.)
// m[9]: the number of fibre elements.
// Summed over the CTA; thread 0 gets the totals.
template <bool PER>
__device__ __noinline__ int march_average(const double *w, int ph) {
  const ModesShared &sh = msh();
  double m[10];
#pragma unroll
  for (int q = 0; q < 10; q++) m[q] = 0.0;
#pragma unroll 1
  for (int y0 = 0; y0 < sh.ney; y0 += sh.rows) {
    const ModesLane<PER> T(y0);
    if (T.column) m[9] += (double)__popc(sh.col[T.f] & ~(PER ? (1u | 2u << sh.nez) : 0u));
    if (T.owner) {
      const int wl = sh.wlen, mz = sh.mz, nface = sh.nface;
      int left, down;
      modes_below<PER>(T.f, left, down);
      const unsigned c3 = sh.col[T.f], c2 = sh.col[T.f + left], c1 = sh.col[T.f + down],
                     c0 = sh.col[T.f + left + down];
#pragma unroll 4
      for (int pl = 0; pl < mz; pl++) {
        const unsigned b0 = (c0 >> pl) & 3u, b1 = (c1 >> pl) & 3u, b2 = (c2 >> pl) & 3u,
                       b3 = (c3 >> pl) & 3u;
        const int n0 = __popc(b0), n1 = __popc(b1), n2 = __popc(b2), n3 = __popc(b3);
        const int lower = (b0 & 1) + (b1 & 1) + (b2 & 1) + (b3 & 1);
        const double k[3] = {(double)(n0 + n2 - n1 - n3), (double)(n0 + n1 - n2 - n3),
                             (double)(2 * lower - (n0 + n1 + n2 + n3))};
#pragma unroll
        for (int c = 0; c < 3; c++) {
          const double v = w[c * wl + pl * nface + T.f];
#pragma unroll
          for (int d = 0; d < 3; d++) m[3 * c + d] = fma(k[d], v, m[3 * c + d]);
        }
      }
    }
  }
  cta_sum<10>(m, ph);
  __syncthreads();
  if (threadIdx.x == 0)
#pragma unroll
    for (int q = 0; q < 10; q++) msh().red[q] = m[q];  // for thread 0 alone
  return ph;
}

// Jacobi diagonal of a slot's nodes (in a cube the components' are equal)
template <bool CUBE>
__device__ __forceinline__ void slot_dinv(int i, F2 (&dz)[3]) {
  const ModesShared &sh = msh();
  const unsigned cv = mcnt()[i];
  if (CUBE) {
    dz[0] = dz[1] = dz[2] = mk2(sh.dl[cv & 15u].x, sh.dl[cv >> 4].x);
    return;
  }
  const float4 da = sh.dl[cv & 15u], db = sh.dl[cv >> 4];
  dz[0] = mk2(da.x, db.x);
  dz[1] = mk2(da.y, db.y);
  dz[2] = mk2(da.z, db.z);
}
template <bool CUBE>
__device__ __forceinline__ void slot_dinv(int i, double (&dz)[3]) {
  const double *d = msh().dl64[mcnt()[i] & 15u];
#pragma unroll
  for (int c = 0; c < 3; c++) dz[c] = d[CUBE ? 0 : c];
}

// One group of up to U slots of update_xr: all loads before the stores, one L2
// round trip for the group.
template <typename V, bool CUBE, int ON, int U>
__device__ __forceinline__ void xr_slots(int s0, int f, const V *pg, typename ModesType<V>::Mem *rg,
                                         typename ModesType<V>::Mem *xg,
                                         const typename ModesType<V>::Mem *qg, V al, V nal,
                                         bool first, double &vz, double &vr) {
  using MT = ModesType<V>;
  const ModesShared &sh = msh();
  const int nface = sh.nface, ntot = sh.ntot, h = sh.h;
  constexpr bool QS = ON == 2;
  V *const q_ = mp<V>() + 3 * ntot;  // (QS)
  const V *const p = ON ? mp<V>() : pg;
  V r[U][3], q[U][3];
#pragma unroll
  for (int j = 0; j < U; j++)
#pragma unroll
    for (int c = 0; c < 3; c++) {
      const int o = c * ntot + min(s0 + j, h - 1) * nface + f;
      r[j][c] = MT::ld(rg + o);
      if (!QS) q[j][c] = MT::ld(qg + o);
    }
#pragma unroll
  for (int j = 0; j < U; j++) {
    if (s0 + j >= h) break;
    const int i = (s0 + j) * nface + f;
    V rn[3], dz[3];
    if (!CUBE) slot_dinv<CUBE>(i, dz);
    double zr[3];
#pragma unroll
    for (int c = 0; c < 3; c++) {
      const int o = c * ntot + i;
      rn[c] = mad(nal, QS ? q_[3 * i + c] : q[j][c], r[j][c]);
      const V dx = al * p[3 * i + c];
      MT::st(rg + o, rn[c]);
      if (first)
        MT::st(xg + o, dx);
      else
        MT::add(xg + o, dx);  // (no value back: nothing waits for it)
      if constexpr (QS) q_[3 * i + c] = rn[c];
      if (!CUBE) zr[c] = MT::dot(dz[c] * rn[c], rn[c]);
    }
    double s2[2];  // r.r of the slot's one or two planes
    MT::squares(rn, s2);
    vr += s2[0] + s2[1];
    if (CUBE) {  // the components' diagonal is the same: r.z from the squares
      const unsigned cv = mcnt()[i];
      vz += sh.dl64[cv & 15u][0] * s2[0];
      if (!MT::F64) vz += sh.dl64[cv >> 4][0] * s2[1];
    } else {
      vz += zr[0] + zr[1] + zr[2];
    }
  }
}

// x += alpha p, r -= alpha q over the thread's column (x = alpha p in a
// correction's first step); returns its shares of r.z and r.r.  x is added to
// in L2: only this thread touches its entries.  q's slots take the new r for
// the direction update.
template <typename V, bool CUBE, int ON, bool PER>
__device__ __noinline__ double2 update_xr(const V *pg, typename ModesType<V>::Mem *rg,
                                          typename ModesType<V>::Mem *xg,
                                          const typename ModesType<V>::Mem *qg, double alpha,
                                          bool first) {
  const int h = msh().h;
  const typename ModesType<V>::S a = (typename ModesType<V>::S)alpha;
  const V al = ModesType<V>::splat(a), nal = ModesType<V>::splat(-a);
  double vz = 0.0, vr = 0.0;
  constexpr int U = ON == 2 ? 5 : 3;
#pragma unroll 1
  for (int y0 = 0; y0 < (ON == 2 ? 1 : msh().ney); y0 += msh().rows) {
    const ModesLane<PER> T(y0);
    if (T.owner)
#pragma unroll 1
      for (int s = 0; s < h; s += U)
        xr_slots<V, CUBE, ON, U>(s, T.f, pg, rg, xg, qg, al, nal, first, vz, vr);
  }
  return make_double2(vz, vr);
}

// p = D^-1 r + beta p over the thread's column; r in q's slots (LOCAL) or in
// rg.  beta = 0 starts afresh without reading p.
template <typename V, bool CUBE, bool LOCAL, int U>
__device__ __forceinline__ void p_slots(int s0, int f, V *p, const typename ModesType<V>::Mem *rg, V be,
                                        bool fresh) {
  const ModesShared &sh = msh();
  const int nface = sh.nface, ntot = sh.ntot, h = sh.h;
  V r[U][3], pv[U][3];
#pragma unroll
  for (int j = 0; j < U; j++)
#pragma unroll
    for (int c = 0; c < 3; c++) {
      const int i = min(s0 + j, h - 1) * nface + f;
      if constexpr (LOCAL)
        r[j][c] = p[3 * (ntot + i) + c];
      else
        r[j][c] = ModesType<V>::ld(rg + (c * ntot + i));
      pv[j][c] = p[3 * i + c];
    }
#pragma unroll
  for (int j = 0; j < U; j++) {
    if (s0 + j >= h) break;
    const int i = (s0 + j) * nface + f;
    V dz[3];
    slot_dinv<CUBE>(i, dz);
#pragma unroll
    for (int c = 0; c < 3; c++) {
      const V z = dz[c] * r[j][c];
      p[3 * i + c] = fresh ? z : mad(be, pv[j][c], z);
    }
  }
}

template <typename V, bool CUBE, int ON, bool LOCAL, bool PER>
__device__ __noinline__ void update_p(V *pg, const typename ModesType<V>::Mem *rg, double beta) {
  const int h = msh().h;
  const typename ModesType<V>::S b = (typename ModesType<V>::S)beta;
  const V be = ModesType<V>::splat(b);
  constexpr int U = LOCAL ? 3 : 5;
#pragma unroll 1
  for (int y0 = 0; y0 < (ON == 2 ? 1 : msh().ney); y0 += msh().rows) {
    const ModesLane<PER> T(y0);
    if (T.owner)
#pragma unroll 1
      for (int s = 0; s < h; s += U)
        p_slots<V, CUBE, LOCAL, U>(s, T.f, ON ? mp<V>() : pg, rg, be, b == 0);
  }
}

// w += x in FP64 over the thread's column
template <typename V, bool PER>
__device__ __noinline__ void update_w(const typename ModesType<V>::Mem *xg, double *w) {
  const ModesShared &sh = msh();
  const int nface = sh.nface, ntot = sh.ntot, h = sh.h, mz = sh.mz, wl = sh.wlen;
#pragma unroll 1
  for (int y0 = 0; y0 < sh.ney; y0 += sh.rows) {
    const ModesLane<PER> T(y0);
    if (!T.owner) continue;
#pragma unroll 1
    for (int s = 0; s < h; s++) {
      const int i = s * nface + T.f;
      V x[3];
      double w0[3], w1[3];
#pragma unroll
      for (int c = 0; c < 3; c++) {
        x[c] = ModesType<V>::ld(xg + (c * ntot + i));
        w0[c] = w[c * wl + i];
        w1[c] = s + h < mz ? w[c * wl + i + h * nface] : 0.0;
      }
#pragma unroll
      for (int c = 0; c < 3; c++) {
        if constexpr (ModesType<V>::F64) {
          w[c * wl + i] = w0[c] + x[c];
        } else {
          w[c * wl + i] = w0[c] + (double)x[c].v.x;
          if (s + h < mz) w[c * wl + i + h * nface] = w1[c] + (double)x[c].v.y;
        }
      }
    }
  }
}

// The residual's face state takes p's place when q is not in shared memory:
// every column's p waits in q's global work space meanwhile, the padding is
// zeroed anew.
template <typename V, bool PER>
__device__ __noinline__ void save_p(typename ModesType<V>::Mem *qg) {
  const ModesShared &sh = msh();
#pragma unroll 1
  for (int y0 = 0; y0 < sh.ney; y0 += sh.rows) {
    const ModesLane<PER> T(y0);
    if (!T.owner) continue;
    for (int s = 0; s < sh.h; s++)
#pragma unroll
      for (int c = 0; c < 3; c++) {
        const int i = s * sh.nface + T.f;
        ModesType<V>::st(qg + (c * sh.ntot + i), mp<V>()[3 * i + c]);
      }
  }
  __syncthreads();
}
template <typename V, bool PER>
__device__ __noinline__ void restore_p(const typename ModesType<V>::Mem *qg, bool saved) {
  const ModesShared &sh = msh();
  for (int i = threadIdx.x; i < 3 * sh.ntot; i += blockDim.x) mp<V>()[i] = zero_of(V());
  __syncthreads();
#pragma unroll 1
  for (int y0 = 0; saved && y0 < sh.ney; y0 += sh.rows) {
    const ModesLane<PER> T(y0);
    if (!T.owner) continue;
    for (int s = 0; s < sh.h; s++)
#pragma unroll
      for (int c = 0; c < 3; c++) {
        const int i = s * sh.nface + T.f;
        mp<V>()[3 * i + c] = ModesType<V>::ld(qg + (c * sh.ntot + i));
      }
  }
}

// p = 0 (its padding stays)
__device__ __noinline__ inline void zero_p(float4 *p) {
  const int n = 3 * msh().ntot;  // 8-byte values
  for (int i = threadIdx.x; i < n / 2; i += blockDim.x) p[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  if (threadIdx.x == 0) reinterpret_cast<float2 *>(p)[n - 1] = make_float2(0.f, 0.f);
  __syncthreads();
}

// the tables, materials and start vectors of one load case
template <bool F64, bool PER>
__device__ __noinline__ void modes_setup(const double *len, const double *mat,
                                         const uint8_t *etype, const double *eps, double *w,
                                         void *rv) {
  ModesShared &sh = msh();
  const int t = threadIdx.x;
  const int nface = sh.nface, nex = sh.nex, wl = sh.wlen;
  if (t < 3) {
    const int n = t == 0 ? sh.nex : (t == 1 ? sh.ney : sh.nez);
    sh.len[t] = len[t];
    sh.hx[t] = len[t] / n;
    sh.a[t] = n / len[t];
  }
  if (t < 2) {
    const double E = mat[2 * t], nu = mat[2 * t + 1];
    sh.lame[t][0] = E * nu / ((1.0 + nu) * (1.0 - 2.0 * nu));
    sh.lame[t][1] = E / (2.0 * (1.0 + nu));
  }
  if (t >= 3 && t < 12) {
    const int i = (t - 3) / 3, j = (t - 3) % 3;
    // Voigt entry of (i, j): xx yy zz xy yz xz, shears halved
    const int v = i == j ? i : (i + j == 1 ? 3 : (i + j == 3 ? 4 : 5));
    sh.E[t - 3] = i == j ? eps[v] : eps[v] / 2;
  }
#pragma unroll 1
  for (int y0 = 0; y0 < sh.ney; y0 += sh.rows) {
    const ModesLane<PER> T(y0);
    unsigned mats = 0;
    const uint8_t *et = etype + T.f;
    if (T.warp_on)
      for (int e = 0; e < sh.nez; e++) mats |= (unsigned)__ldg(et + e * nface) << e;
    // bit s: the layer below plane s.  Periodic: layer s - 1, and the first
    // ones again past the last
    if (PER) mats = mats << 1 | mats >> (sh.nez - 1) | (mats & 1u) << (sh.nez + 1);
    if (T.column) sh.col[T.f] = mats;
    // w's padding: the columns without an interior node (and below the row
    // past the end)
    if (T.column && (PER || !T.owner))
      for (int c = 0; c < 3; c++)
        for (int pl = 0; pl < sh.mz; pl++) w[c * wl + pl * nface + T.f] = 0.0;
  }
  if (!PER)
    for (int i = t; i < 3 * (nex + 2); i += blockDim.x)
      w[(i / (nex + 2)) * wl + sh.mz * nface + i % (nex + 2)] = 0.0;
  __syncthreads();
  for (int i = t; i < 2 * MC_N; i += blockDim.x)
    sh.cd[i / MC_N][i % MC_N] = mode_coef(i % MC_N, sh.lame[i / MC_N][0], sh.lame[i / MC_N][1],
                                          sh.hx[0] * sh.hx[1] * sh.hx[2] / 16.0, sh.a);
  if (t < 9) sh.A[t] = 4.0 * sh.hx[t % 3] * sh.E[t];
  // fibre elements around the column's nodes; affine conditions: start of the
  // right-hand side's own residual, w = -eps.x inside, i.e. u = 0 inside
#pragma unroll 1
  for (int y0 = 0; y0 < sh.ney; y0 += sh.rows) {
    const ModesLane<PER> T(y0);
    if (T.owner) {
      int left, down;
      modes_below<PER>(T.f, left, down);
      const unsigned m0 = sh.col[T.f], m1 = sh.col[T.f + left], m2 = sh.col[T.f + down],
                     m3 = sh.col[T.f + left + down];
      auto count = [&](int pl) {
        return __popc(shr32(m0, pl) & 3u) + __popc(shr32(m1, pl) & 3u) + __popc(shr32(m2, pl) & 3u) +
               __popc(shr32(m3, pl) & 3u);
      };
      for (int s = 0; s < sh.h; s++)
        mcnt()[s * nface + T.f] = (uint8_t)(count(s) | (F64 ? 0 : count(s + sh.h) << 4));
      const double X = (T.f % nex) * sh.hx[0], Y = (T.f / nex) * sh.hx[1];
#pragma unroll
      for (int c = 0; c < 3; c++) {
        const double xy = sh.E[3 * c] * X + sh.E[3 * c + 1] * Y, ez = sh.E[3 * c + 2] * sh.hx[2];
        if (!PER)
          for (int pl = 0; pl < sh.mz; pl++) w[c * wl + pl * nface + T.f] = -(xy + ez * (pl + 1));
        // a slot without an upper plane keeps a zero there
        static_cast<float2 *>(rv)[c * sh.ntot + (sh.h - 1) * nface + T.f] = make_float2(0.f, 0.f);
      }
    }
  }
  __syncthreads();
  if (t < 2) {
    const double *C = sh.cd[t];
    double *k = sh.cc[t];
    k[CC_LAM] = C[MC_BXY];
    k[CC_MU] = C[MC_MXX];
    k[CC_MU2] = 2.0 * C[MC_MXX];
    k[CC_LAM3] = C[MC_B3XY];
    k[CC_MU3] = C[MC_M3XY];
    k[CC_K9] = C[MC_U111];
  }
  for (int i = t; i < 4 * MC_N; i += blockDim.x) {
    const int m = i / MC_N, c = i % MC_N;
    sh.c32[m][c] = make_float2((float)sh.cd[m & 1][c], (float)sh.cd[m >> 1][c]);
  }
  __syncthreads();
  if (t < 24) {
    const int m = t / 6, i = t % 6;
    sh.c6[m][i] =
        make_float2((float)sh.cc[m & 1][i], (float)sh.cc[m >> 1][i]);
  }
  if (t < 9) {
    double s2 = 0.0, d[3];
#pragma unroll
    for (int c = 0; c < 3; c++) {
      d[c] = (8 - t) * mode_diag(sh.cd[0], c) + t * mode_diag(sh.cd[1], c);
      s2 += d[c] * d[c];
    }
#pragma unroll
    for (int c = 0; c < 3; c++) sh.dl64[t][c] = 1.0 / d[c];
    sh.dl[t] = make_float4((float)(1.0 / d[0]), (float)(1.0 / d[1]), (float)(1.0 / d[2]), 0.f);
    sh.kd2[t] = s2;
  }
  __syncthreads();
}

// Averages from the fibre's integrals m (march_average), by one thread:
// <strain> = eps, <stress> = D_0 eps + (D_1 - D_0) f, f = the strain's integral
// over the fibre / volume.
__device__ __noinline__ inline void modes_output(const double *m, double *stress, double *strain) {
  const ModesShared &sh = msh();
  const double nel = (double)sh.nface * sh.nez;
  const double sc = 0.25 / nel, vf = m[9] / nel;
  const double *a = sh.a, *E = sh.E;
  const double e[6] = {E[0], E[4], E[8], 2.0 * E[1], 2.0 * E[5], 2.0 * E[2]};
  const double f[6] = {vf * e[0] + sc * a[0] * m[0],
                       vf * e[1] + sc * a[1] * m[4],
                       vf * e[2] + sc * a[2] * m[8],
                       vf * e[3] + sc * (a[1] * m[1] + a[0] * m[3]),
                       vf * e[4] + sc * (a[2] * m[5] + a[1] * m[7]),
                       vf * e[5] + sc * (a[2] * m[2] + a[0] * m[6])};
  const double l0 = sh.lame[0][0], m0 = sh.lame[0][1], l1 = sh.lame[1][0], m1 = sh.lame[1][1];
  const double tf = f[0] + f[1] + f[2], tm = e[0] + e[1] + e[2] - tf;
#pragma unroll
  for (int i = 0; i < 6; i++) {
    const double g = e[i] - f[i];
    if (strain) strain[i] = e[i];
    stress[i] = i < 3 ? (l0 * tm + 2.0 * m0 * g) + (l1 * tf + 2.0 * m1 * f[i])
                      : m0 * g + m1 * f[i];
  }
}

// The CTA's work spaces.  Formed anew at every use (hidden from the
// compiler's view of the loop), so that no pointer holds registers across the
// marches.
template <typename V, int ON>
struct ModesSpace {
  double *w;
  typename ModesType<V>::Mem *r, *x, *q;  // q: in L2
  V *p, *e;                               // p in L2; strips
  __device__ __forceinline__ explicit ModesSpace(const ModesBufs &P) {
    unsigned b = blockIdx.x;
    asm volatile("" : "+r"(b));
    w = P.ws_w + (size_t)b * P.w_stride;
    r = static_cast<typename ModesType<V>::Mem *>(P.ws_v) + (size_t)b * P.v_cta;
    x = r + P.v_stride;
    q = ON == 2 ? nullptr : x + P.v_stride;
    p = ON ? nullptr : reinterpret_cast<V *>(q + P.v_stride);
    e = ON == 2 ? nullptr : static_cast<V *>(P.ws_e) + (size_t)b * P.e_stride;
  }
};

// march_residual over all strips
template <typename V, bool CUBE, int ON, bool PER>
__device__ __forceinline__ double2 residual_strips(const ModesSpace<V, ON> &ws) {
  double *const e = reinterpret_cast<double *>(ws.e);
  double2 d = march_residual<V, CUBE, ON, PER>(ws.w, ws.r, e, 0);
  if (ON < 2)
#pragma unroll 1
    for (int y0 = msh().rows; y0 < msh().ney; y0 += msh().rows) {
      __syncthreads();  // the strip below's shares
      const double2 n = march_residual<V, CUBE, ON, PER>(ws.w, ws.r, e, y0);
      d.x += n.x;
      d.y += n.y;
    }
  return d;
}

// Norm of the right-hand side from the thread's share of its square (affine
// conditions: of u = 0 inside, as modes_setup left w; periodic ones: of the
// zero fluctuation, w = 0); one at the round-off level of its own
// cancelling terms is zero, and its load case is solved with that.  Else
// w = 0: the affine field starts.
template <bool F64, bool PER>
__device__ __noinline__ double rhs_norm(double n2, double *w, int ph) {
  const ModesShared &sh = msh();
  double v[2] = {n2, 0.0};
  for (int y0 = 0; y0 < sh.ney; y0 += sh.rows) {
    const ModesLane<PER> T(y0);
    if (T.owner)
      for (int s = 0; s < sh.h; s++) {
        const unsigned cv = mcnt()[s * sh.nface + T.f];
        v[1] += sh.kd2[cv & 15u];
        if (!F64 && s + sh.h < sh.mz) v[1] += sh.kd2[cv >> 4];
      }
  }
  cta_sum<2>(v, ph);
  double um = 0.0;
#pragma unroll
  for (int c = 0; c < 3; c++)
    um = fmax(um, fabs(sh.E[3 * c]) * sh.len[0] + fabs(sh.E[3 * c + 1]) * sh.len[1] +
                      fabs(sh.E[3 * c + 2]) * sh.len[2]);
  double rn0 = sqrt(v[0]);
  if (rn0 <= SP_RHS_FLOOR * sqrt(v[1]) * um) rn0 = 0.0;
  if (!PER && rn0 > 0.0)
    for (int y0 = 0; y0 < sh.ney; y0 += sh.rows) {
      const ModesLane<PER> T(y0);
      if (T.owner)
        for (int c = 0; c < 3; c++)
          for (int pl = 0; pl < sh.mz; pl++) w[c * sh.wlen + pl * sh.nface + T.f] = 0.0;
    }
  __syncthreads();
  return rn0;
}

// The RVE's last load case to finish reports for all of them: the worst
// status and residual, the most refinement steps and CG iterations.  One
// thread.
__device__ __noinline__ inline void modes_report(const sp_solve_info &in, sp_solve_info *ti, int k,
                                                 int nrhs, unsigned *done, sp_solve_info *out) {
  ti[k] = in;
  __threadfence();
  if (atomicAdd(done, 1u) == (unsigned)nrhs - 1) {
    __threadfence();
    sp_solve_info all = {};
    for (int i = 0; i < nrhs; i++) {
      const volatile sp_solve_info *c = ti + i;
      if (c->status > all.status) all.status = c->status;
      if (c->outer_its > all.outer_its) all.outer_its = c->outer_its;
      if (c->inner_its > all.inner_its) all.inner_its = c->inner_its;
      const double r = c->relres;
      if (!isnan(all.relres) && !(r <= all.relres)) all.relres = r;  // (NaN is the worst)
    }
    *out = all;
    *done = 0;
  }
}

// Refinement from the start iterate in w, as solve_rve's loop: FP64 residual,
// CG corrections (reliable updates) in V, w += x, until the residual is at
// most rtol rn0 -- rtol_refine rn0 once a correction has run.  Returns the
// last relative residual; the counts are in shared memory.
template <typename V, bool CUBE, int ON, bool PER>
__device__ __forceinline__ double modes_refine(const ModesBufs &B, const ModesLimits &L, double rn0,
                                               int &ph) {
  constexpr bool QS = ON == 2;
  ModesShared &sh = msh();
  double rho = 0.0, relres;
  int outer = 0;
  for (;;) {
    double v[2];
    {
      const ModesSpace<V, ON> ws(B);
      if (ON == 1 && rho != 0.0) save_p<V, PER>(ws.q);
      const double2 d = residual_strips<V, CUBE, ON, PER>(ws);
      v[0] = d.x;
      v[1] = d.y;
      cta_sum<2>(v, ph);
    }
    relres = rn0 > 0.0 ? sqrt(v[0]) / rn0 : 0.0;
    const double target = outer == 0 ? L.rtol : L.rtol_refine;
    if (!(rn0 > 0.0 && sqrt(v[0]) > target * rn0) || outer >= L.max_outer) break;
    const double fin = SP_FINAL_MARGIN * L.rtol_refine * rn0;
    const double thr = fmax(L.inner_rtol * L.inner_rtol * v[0], fin * fin);
    // a reliable update: r is the true residual, the search direction goes
    // on with beta = r.z / rho of the last step
    {
      const ModesSpace<V, ON> ws(B);
      if (ON == 1)
        restore_p<V, PER>(ws.q, rho != 0.0);
      else if (rho == 0.0)
        zero_p(ON ? mp<float4>() : reinterpret_cast<float4 *>(ws.p));
      update_p<V, CUBE, ON, false, PER>(ws.p, ws.r, rho != 0.0 ? v[1] / rho : 0.0);
    }
    rho = v[1];
    __syncthreads();
    int it = 0;
    while (it < L.max_inner) {
      {
        const ModesSpace<V, ON> ws(B);
        v[0] = march_apply<V, CUBE, ON, PER>(ws.q, ws.p, ws.e, 0);
        if (ON < 2)
#pragma unroll 1
          for (int y0 = sh.rows; y0 < sh.ney; y0 += sh.rows) {
            __syncthreads();  // the strip below's shares
            v[0] += march_apply<V, CUBE, ON, PER>(ws.q, ws.p, ws.e, y0);
          }
      }
      double d[1] = {v[0]};
      cta_sum<1>(d, ph);
      {
        const ModesSpace<V, ON> ws(B);
        const double2 u = update_xr<V, CUBE, ON, PER>(ws.p, ws.r, ws.x, ws.q,
                                                      d[0] != 0.0 ? rho / d[0] : 0.0, it == 0);
        v[0] = u.x;
        v[1] = u.y;
      }
      cta_sum<2>(v, ph);
      it++;
      if (v[1] <= thr) break;
      {
        const ModesSpace<V, ON> ws(B);
        update_p<V, CUBE, ON, QS, PER>(ws.p, ws.r, rho != 0.0 ? v[0] / rho : 0.0);
      }
      rho = v[0];
      __syncthreads();
    }
    if (it > 0) {
      const ModesSpace<V, ON> ws(B);
      update_w<V, PER>(ws.x, ws.w);
    }
    outer++;
    if (threadIdx.x == 0) {
      sh.inner += it;
      sh.outer = outer;
    }
    __syncthreads();
  }
  return relres;
}

// V: FP32 pairs or FP64; NT threads at most, MINB CTAs per SM; CUBE: equal
// element edges; ON: vectors in shared memory (ModesGeo); PER: periodic
// conditions
template <typename V, int NT, int MINB, bool CUBE, int ON, bool PER>
__global__ void __launch_bounds__(NT, MINB) k_modes(ModesParams P) {
  constexpr bool F64 = ModesType<V>::F64;
  ModesShared &sh = msh();
  if (dynamic_smem_bytes() < sizeof(ModesShared)) return;
  int ph = 0;  // the reduction buffer in turn
  for (;;) {
    if (threadIdx.x == 0) {
      const int task = atomicAdd(P.counter, 1);
      sh.job = task < P.ntask ? 1 : 0;
      if (task < P.ntask) {
        sh.rid = P.order[task / P.nrhs];
        sh.k = task % P.nrhs;
        const MeshGeo &mg = P.plans[P.rves[sh.rid].plan].geo;
        const ModesGeo G(mg.nex, mg.ney, mg.nez, PER, F64, ON);
        if (!modes_fit(G)) sh.job = 2;  // launched with less than this RVE needs
        modes_sizes(G, sh);
      }
    }
    __syncthreads();
    if (sh.job == 0) break;
    double relres = 0.0;
    if (sh.job == 1) {
      // 1. tables
      {
        const ModesSpace<V, ON> ws(P.buf);
        const BatchRve &rv = P.rves[sh.rid];
        modes_setup<F64, PER>(rv.len, P.mats + (size_t)sh.rid * 4, P.etype + rv.etype_off,
                              P.strains + ((size_t)sh.rid * P.nrhs + sh.k) * 6, ws.w, ws.r);
      }
      // 2. the right-hand side's norm
      double rn0;
      {
        const ModesSpace<V, ON> ws(P.buf);
        rn0 = rhs_norm<F64, PER>(residual_strips<V, CUBE, ON, PER>(ws).x, ws.w, ph);
        ph ^= 1;
      }
      // 3. refinement
      relres = modes_refine<V, CUBE, ON, PER>(P.buf, P.lim, rn0, ph);
      // 4. averages
      {
        const ModesSpace<V, ON> ws(P.buf);
        ph = march_average<PER>(ws.w, ph);
      }
      if (threadIdx.x == 0) {
        const size_t o = ((size_t)sh.rid * P.nrhs + sh.k) * 6;
        modes_output(sh.red, P.out_stress + o, P.out_strain ? P.out_strain + o : nullptr);
      }
    }
    if (threadIdx.x == 0) {
      sp_solve_info in = {};
      in.relres = relres;
      in.status = sh.job != 1 ? SP_ERR_STATE : (relres <= P.lim.rtol ? SP_OK : SP_ERR_NOCONV);
      in.outer_its = sh.outer;
      in.inner_its = sh.inner;
      modes_report(in, P.task_info + (size_t)sh.rid * P.nrhs, sh.k, P.nrhs, P.done + sh.rid,
                   P.out_info + sh.rid);
    }
    __syncthreads();
  }
}

using ModesFn = void (*)(ModesParams);

// the instantiated classes (threads, CTAs per SM, vectors in shared memory):
// the largest blocks of which 8, 3, 2 and 1 fit an SM's register file at 128
// registers a thread; periodic conditions, which have no strips, also at 96
// registers for meshes of more columns, affine ones without any vector in
// shared memory
#define SP_MODES_CLASSES(X, V, PER) \
  X(V, 64, 8, 2, PER) X(V, 160, 3, 2, PER) X(V, 256, 2, 2, PER) X(V, 512, 1, 2, PER) \
  X(V, 512, 1, 1, PER)
#define SP_MODES_PERIODIC(X, V) X(V, 640, 1, 1, true)
#define SP_MODES_AFFINE(X, V) X(V, 512, 1, 0, false)
#define SP_MODES_EXTERN(V, NT, MINB, ON, PER) \
  extern template __global__ void k_modes<V, NT, MINB, true, ON, PER>(ModesParams); \
  extern template __global__ void k_modes<V, NT, MINB, false, ON, PER>(ModesParams);

}  // namespace sp
